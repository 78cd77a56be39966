"""The saved-arg adjoint on both sides of the rule that takes its strips or its tiles: many small planes (strips), few of
them (tiles), narrow ones, and the long full strips the 7x7 backward wants.  Bit-identical to the recomputing kernels."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [1, 2, 3])
@pytest.mark.parametrize("dilate", [True, False])
@pytest.mark.parametrize("shape", [(1, 33, 64), (2, 200, 8), (3000, 1, 4), (2500, 2, 60), (2100, 7, 64), (900, 17, 68), (1000, 9, 124),
                                   (500, 65, 132), (3000, 40, 8), (460, 255, 252)])
def test_equals_recomputed(r, dilate, shape):
    from poutre2_gb300 import autograd as ag
    g = torch.Generator(device="cuda").manual_seed(shape[0] + shape[2])
    x = torch.randn(shape, device="cuda", generator=g)
    u = torch.rand(shape, device="cuda", generator=g)
    x[u < 0.3] = 0.25  # ties
    x[u > 0.99] = float("inf")
    x[(u > 0.98) & (u < 0.99)] = float("-inf")
    gy = torch.randn(shape, device="cuda", generator=g)
    y, code = ag.flat_forward_arg(x, r, dilate)
    assert torch.equal(y, ag.flat_forward(x, r, dilate))
    assert torch.equal(ag.flat_backward_arg(code, gy, r), ag.flat_backward(x, gy, r, dilate))
