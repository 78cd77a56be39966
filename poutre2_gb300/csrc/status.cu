// status.cu -- results that come back to the host: the pinned words kernels write them to, and
// pg_check_device, which reads the status words of every kernel file.
//
// pg_check_device used to synchronise the stream and then copy seven device symbols one by one, each copy a
// round trip of about 9 us: 72 us after a 170 us reconstruction.  One warp now reads the seven words at the
// end of the stream, so that one synchronisation brings the answer (binary h-maxima 2048^2 u8 238 -> 177 us a call).
#include <atomic>
#include <mutex>

#include "common.cuh"

namespace pg {
namespace {

struct SlotPool {
  long long *host = nullptr;
  long long *device = nullptr;
  std::atomic<uint64_t> taken{0};
};

// Made on first use and kept for the life of the process (512 bytes); null where that fails, as it does while a
// stream capture of another thread forbids the allocation: the next caller tries again.
SlotPool *slots() {
  static SlotPool pool;
  static std::mutex mu;
  static std::atomic<bool> made{false};
  if (made.load()) return &pool;
  std::lock_guard<std::mutex> lk(mu);
  if (made.load()) return &pool;
  void *h = nullptr, *d = nullptr;
  if (cudaHostAlloc(&h, kHostSlots * sizeof(long long), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  if (cudaHostGetDevicePointer(&d, h, 0) != cudaSuccess) {
    (void)cudaGetLastError();
    cudaFreeHost(h);
    return nullptr;
  }
  pool.host = static_cast<long long *>(h);
  pool.device = static_cast<long long *>(d);
  made.store(true);
  return &pool;
}

constexpr int kWords = 7;
struct StatusWords {
  int *p[kWords];
};

// The first non-zero word (in order) goes back as index << 32 | code and is cleared; 0: none.
__global__ void k_read_status(StatusWords w, long long *result) {
  int st = 0;
  if (threadIdx.x < kWords) st = *(volatile int *)w.p[threadIdx.x];
  const unsigned any = __ballot_sync(0xffffffffu, st != 0);
  const int first = __ffs(any) - 1;
  if (any == 0u) {
    if (threadIdx.x == 0) *(volatile long long *)result = 0;
  } else if ((int)threadIdx.x == first) {
    *(volatile int *)w.p[first] = 0;
    *(volatile long long *)result = ((long long)first << 32) | (unsigned)st;
  }
  __threadfence_system();
}

}  // namespace

HostSlot::HostSlot(bool wanted) {
  SlotPool *pool = wanted ? slots() : nullptr;
  if (!pool) return;
  uint64_t t = pool->taken.load();
  while (t != ~0ull) {
    const int i = __builtin_ctzll(~t);
    if (pool->taken.compare_exchange_weak(t, t | (1ull << i))) {
      index_ = i;
      word = pool->device + i;
      break;
    }
  }
  static_assert(kHostSlots == 64, "one bit per word");
}
HostSlot::~HostSlot() {
  if (index_ >= 0) slots()->taken.fetch_and(~(1ull << index_));
}
long long HostSlot::value() const { return *const_cast<volatile long long *>(slots()->host + index_); }

}  // namespace pg

extern "C" {

// Synchronises `stream`, then returns and clears the first status that a kernel recorded since the last check
// (PG_ERR_NOT_CONVERGED if a reconstruction gave up, PG_ERR_CUDA if a bounded wait of a tile copy or a
// labelling loop ran out).
pg_status pg_check_device(pg_stream_t stream) {
  using namespace pg;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  static cudaError_t (*const word_of[kWords])(void **) = {recon_status_word, rect_status_word,       diag_status_word,
                                                          oct_status_word,   small_tile_status_word, open_status_word,
                                                          label_status_word};
  static const char *const text[kWords] = {
      "reconstruction did not converge within its round cap or wait limit",
      "a box tile load did not complete within its wait limit",
      "a segment tile load did not complete within its wait limit",
      "an octagon tile load did not complete within its wait limit",
      "a small-SE tile load did not complete within its wait limit",
      "an opening tile load did not complete within its wait limit",
      "a labelling union-find loop exceeded its iteration limit"};
  StatusWords w{};
  for (int k = 0; k < kWords; ++k) {
    void *p = nullptr;
    PG_CUDA_TRY(word_of[k](&p), "status word");
    w.p[k] = static_cast<int *>(p);
  }
  // a capturing stream cannot be synchronised: that call reports it, with nothing added to the graph
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) {
    (void)cudaGetLastError();
    capture = cudaStreamCaptureStatusActive;
  }
  HostSlot slot(capture == cudaStreamCaptureStatusNone);  // its pool's allocation would break a capture
  bool queued = false;
  if (slot.word) {
    // The launch's own result: cudaGetLastError would also return an error some earlier call left behind, and the
    // word that this kernel reads and clears would then be lost.
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(32);
    cfg.stream = s;
    queued = cudaLaunchKernelEx(&cfg, k_read_status, w, slot.word) == cudaSuccess;  // not on another device's stream
    if (!queued) (void)cudaGetLastError();
  }
  PG_CUDA_TRY(cudaStreamSynchronize(s), "stream synchronisation");
  if (queued) {
    const long long v = slot.value();
    if (v == 0) return PG_OK;
    return fail(static_cast<pg_status>((int)v), text[v >> 32]);
  }
  for (int k = 0; k < kWords; ++k) {
    int st = 0;
    PG_CUDA_TRY(cudaMemcpy(&st, w.p[k], sizeof(int), cudaMemcpyDeviceToHost), "read device status");
    if (st == 0) continue;
    const int zero = 0;
    PG_CUDA_TRY(cudaMemcpy(w.p[k], &zero, sizeof(int), cudaMemcpyHostToDevice), "clear device status");
    return fail(static_cast<pg_status>(st), text[k]);
  }
  return PG_OK;
}

}  // extern "C"
