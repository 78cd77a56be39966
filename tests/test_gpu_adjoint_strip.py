"""The register-streaming saved-arg adjoint (rows of whole 16-byte vectors): segments of 64 columns, strips of 8 to 64
rows.  Values, codes and gradients are bit-identical to the recomputing kernels, ties and infinities included."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [1, 2, 3])
@pytest.mark.parametrize("dilate", [True, False])
@pytest.mark.parametrize("shape", [(1, 1, 4), (3, 2, 60), (2, 7, 64), (2, 8, 68), (1, 9, 124), (2, 65, 128), (1, 131, 132),
                                   (400, 63, 64), (700, 66, 8), (300, 129, 320)])
def test_strip_equals_recomputed(r, dilate, shape):
    from poutre2_gb300 import autograd as ag
    g = torch.Generator(device="cuda").manual_seed(shape[1] * 1000 + shape[2])
    for levels in (0, 3):
        x = torch.randint(0, levels, shape, device="cuda", generator=g).float() - 1 if levels else \
            torch.randn(shape, device="cuda", generator=g)
        if not levels:
            x[torch.rand(shape, device="cuda", generator=g) < 0.02] = float("inf")
            x[torch.rand(shape, device="cuda", generator=g) < 0.02] = float("-inf")
        gy = torch.randn(shape, device="cuda", generator=g)
        y, code = ag.flat_forward_arg(x, r, dilate)
        assert torch.equal(y, ag.flat_forward(x, r, dilate))
        assert torch.equal(ag.flat_backward_arg(code, gy, r), ag.flat_backward(x, gy, r, dilate))


def test_a_misaligned_tensor_takes_the_tile_kernels():
    from poutre2_gb300 import autograd as ag
    buf = torch.randn(2 * 40 * 64 + 1, device="cuda")
    x = buf[1:].view(2, 40, 64)
    y, code = ag.flat_forward_arg(x, 2, True)
    y2, code2 = ag.flat_forward_arg(x.clone(), 2, True)
    assert torch.equal(y, y2) and torch.equal(code, code2)
    gy = torch.randn_like(y2)
    assert torch.equal(ag.flat_backward_arg(code, gy, 2), ag.flat_backward(x, gy, 2, True))
