// recon.cu -- geodesic reconstruction (by dilation / erosion) as one persistent kernel, and
// the filters built on it: h-extrema (marker made on the fly), low/high leveling (mask and
// final clip made on the fly), binary h-maxima (comparison fused), ragged batches.
//
// Reference: t_ReconstructionViewDispatcher (geodesy/details/mreconstruct_t.hpp:84-195), a
// sequential Vincent hybrid (raster scan, anti-raster scan, FIFO).  Its result is the
// least fixpoint rec = min(mask, dilate(rec)) above min(marker, mask) (dual for erosion),
// which is unique, so any order of monotone updates reaches the same image: the parallel
// scheme below is bit-exact with it.  Leveling (leveling_t.hpp:45-202) is the same fixpoint
// with mask max(marker, ref) (low) / min(marker, ref) (high) followed by a clip by ref.
//
// GPU design: tiles iterated to a tile-local fixpoint, scheduled until no tile changes.
//  * Single images of 1- or 2-byte pixels whose 32x32 tiles all fit on the GPU at once
//    (k_reconstruct_resident): every tile stays in its warp, neighbours exchange border pixels.
//  * Other images of pixels of at most 4 bytes (k_reconstruct_wl): 32x32 tiles, one warp per tile, the tile
//    in registers; directional sweep sets (down/up by warp shuffles, right/left after a
//    shared-memory transpose; two rows per register for 1- and 2-byte pixels) until a set
//    changes nothing.  The tiles are driven by a device worklist (a ticket ring and a state
//    per tile, below): a warp pops a tile, visits it, and queues the neighbours whose shared
//    border changed, until no tile is queued or running.
//  * 8-byte pixels, the allocation-free entry and one batch-plan configuration
//    (k_reconstruct): 64x64 (32x32) tiles staged in shared memory with a one-pixel halo and
//    swept by a CTA; rounds over the flagged tiles (round 0: all tiles, marker computed from
//    the inputs) separated by a grid barrier, until a round flags nothing.  Flags live in a
//    double-buffered device worklist; the "any flag" word is triple-buffered so no CTA resets
//    a word another may still read.
//  * Reads of other tiles' pixels bypass L1 (ld.global.cg): values only grow (shrink for
//    erosion), so a concurrently updated halo value is either the old or the new one, both
//    below the fixpoint; a tile that saw an old value is queued (flagged) again by its writer.
//  * Every wait is bounded (kBarrierTimeoutNs of %globaltimer on the grid barrier and on the
//    worklist; visit and round caps), recording PG_ERR_NOT_CONVERGED in a device status word.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "common.cuh"
#include "words.cuh"

namespace pg {

// tile side = threads per CTA: 64 (32 for 8-byte pixels, to keep the staged tile within the
// 48 KB static shared-memory limit)
__host__ __device__ constexpr int tile_side_for(int elem_bytes) { return elem_bytes == 8 ? 32 : 64; }
template <typename T> __host__ __device__ constexpr int tile_side() { return tile_side_for((int)sizeof(T)); }
static constexpr int kMaxSweeps = 512;
static constexpr int kVisitSweeps = 2;  // sweep sets per visit of a register tile (single calls)
static constexpr unsigned long long kBarrierTimeoutNs = 4000000000ull;  // 4 s

// Limits that a test may lower (pg_debug_set_limits): the device wait limit, passed to every launch
// and used by every bounded wait below, and a cap on the rounds (round kernel) / visits per tile
// (worklist kernel) that replaces the host's default when positive.
static std::atomic<unsigned long long> g_dbg_wait_ns{kBarrierTimeoutNs};
static std::atomic<int> g_dbg_max_rounds{0};

// Device-wide sticky status of the reconstruction kernels (0 = ok) and the round count of
// the last completed launch.
__device__ int g_recon_status = 0;
__device__ int g_recon_rounds = 0;

struct RImg {
  const void *marker;  // marker (INIT_MARKER and the leveling masks)
  const void *mask;    // mask, or the leveling reference
  void *rec;           // reconstruction buffer
  void *out;           // epilogue output (binary u8 image, or == rec)
  int64_t H, W;
  int tiles_x, tiles_y;
  int tile_begin;
  int pad;
};

struct RCtl {
  unsigned any[3];
  unsigned bar_count;
  unsigned bar_gen;
  int status;
  int rounds;
  int pad;
};

template <typename T> struct RParams {
  RImg single;        // used when nimg == 1
  const RImg *imgs;   // device table when nimg > 1
  int nimg;
  int ntiles;
  RCtl *ctl;
  unsigned *flags;    // 2 * ntiles
  int max_rounds;
  int max_sweeps = kMaxSweeps;  // sweep sets per tile visit before the tile yields (and re-flags itself)
  unsigned long long wait_ns = kBarrierTimeoutNs;  // limit of every bounded device wait
  int init, mask_mode, epi;
  T h;
};

// row pitch (in pixels) of a shared tile: a row spans an odd number of 32-bit words so that
// thread-per-row sweeps touch 32 distinct banks
template <typename T> __host__ __device__ constexpr int tile_pitch(int cols) {
  if constexpr (sizeof(T) <= 4) {
    int words = (cols * (int)sizeof(T) + 3) / 4;
    if (words % 2 == 0) ++words;
    return words * 4 / (int)sizeof(T);
  } else {
    return cols | 1;
  }
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}


__device__ __forceinline__ void set_status(RCtl *ctl, int code) {
  atomicCAS(&ctl->status, 0, code);
  atomicCAS(&g_recon_status, 0, code);
}

// Grid barrier with a bounded wait.  Returns false once any CTA recorded an error; thread 0
// reads the status for its whole CTA so that every thread takes the same branch afterwards.
__device__ bool grid_barrier(RCtl *ctl, unsigned long long wait_ns) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *genp = &ctl->bar_gen;
    const unsigned gen = *genp;
    __threadfence();
    const unsigned arrived = atomicAdd(&ctl->bar_count, 1u) + 1u;
    if (arrived == gridDim.x) {
      atomicExch(&ctl->bar_count, 0u);
      __threadfence();
      atomicAdd(&ctl->bar_gen, 1u);
    } else {
      const unsigned long long t0 = global_ns();
      unsigned ns = 32;
      while (*genp == gen) {
        __nanosleep(ns);
        if (ns < 1024) ns <<= 1;
        if (global_ns() - t0 > wait_ns) {
          set_status(ctl, PG_ERR_NOT_CONVERGED);
          break;
        }
      }
    }
    __threadfence();
    s_ok = *((volatile int *)&ctl->status) == 0;
  }
  __syncthreads();
  return s_ok != 0;
}

template <typename T, bool SUP>
__device__ __forceinline__ T sat_shift(T m, T h) {
  // marker of h-maxima (sat_sub) / h-minima (sat_add), op_Saturated_{Sub,Add}_Constant
  // (pixel_processing/details/arith_op_t.hpp:218-345), clamped to the pixel type's range
  if constexpr (std::is_integral_v<T>) {
    using Wide = std::conditional_t<(sizeof(T) < 4), int, std::conditional_t<(sizeof(T) < 8), long long, __int128>>;
    const Wide r = SUP ? (Wide)m - (Wide)h : (Wide)m + (Wide)h;
    if (r < (Wide)Lim<T>::lo()) return Lim<T>::lo();
    if (r > (Wide)Lim<T>::hi()) return Lim<T>::hi();
    return (T)r;
  } else {
    return SUP ? m - h : m + h;
  }
}

// Effective mask and initial value of a pixel from its loaded inputs -- `a` the mask (the
// leveling reference), `mk` the marker, loaded only when needs_marker() says so -- kept apart
// from the loads so that a caller can issue the loads of many pixels before it waits for the
// first.  Round 0 starts from select_marker: min(marker, mask) (max for erosion).
template <typename T>
__device__ __forceinline__ bool needs_marker(const RParams<T> &P, int round) {
  return P.init != INIT_SAT_CONST && (round == 0 || P.mask_mode != MASK_PLAIN);
}
template <typename T, bool SUP>
__device__ __forceinline__ void combine_init(const RParams<T> &P, T a, T mk, T &mask, T &init) {
  if (P.init == INIT_SAT_CONST) {
    mask = a;
    init = sat_shift<T, SUP>(a, P.h);
    return;
  }
  if (P.mask_mode == MASK_MAX_MARKER) mask = Op<T, true>::apply(mk, a);
  else if (P.mask_mode == MASK_MIN_MARKER) mask = Op<T, false>::apply(mk, a);
  else mask = a;
  init = Op<T, !SUP>::apply(mk, mask);
}
template <typename T>
__device__ __forceinline__ T combine_mask(const RParams<T> &P, T a, T mk) {
  if (P.init == INIT_SAT_CONST || P.mask_mode == MASK_PLAIN) return a;
  return P.mask_mode == MASK_MAX_MARKER ? Op<T, true>::apply(mk, a) : Op<T, false>::apply(mk, a);
}

template <typename T> __device__ __forceinline__ T ld_cg(const T *p) {
  if constexpr (sizeof(T) == 1) return (T)__ldcg(reinterpret_cast<const unsigned char *>(p));
  else if constexpr (sizeof(T) == 2) return (T)__ldcg(reinterpret_cast<const unsigned short *>(p));
  else if constexpr (std::is_same_v<T, int64_t>) return (T)__ldcg(reinterpret_cast<const long long *>(p));
  else return __ldcg(p);
}
template <typename T> __device__ __forceinline__ void st_cg(T *p, T v) {
  if constexpr (sizeof(T) == 1) __stcg(reinterpret_cast<unsigned char *>(p), (unsigned char)v);
  else if constexpr (sizeof(T) == 2) __stcg(reinterpret_cast<unsigned short *>(p), (unsigned short)v);
  else if constexpr (std::is_same_v<T, int64_t>) __stcg(reinterpret_cast<long long *>(p), (long long)v);
  else __stcg(p, v);
}

enum : int { B_N = 1, B_S = 2, B_W = 4, B_E = 8, B_NW = 16, B_NE = 32, B_SW = 64, B_SE = 128, B_SELF = 256 };  // B_x = 1 << direction

// Puts the tiles next to tile (tx, ty) whose shared border changed (f: B_* bits) on the next
// round's worklist, and the tile itself when it yielded before its local fixpoint.
template <bool CONN8>
__device__ void flag_neighbours(const RImg &im, unsigned *flags, int ntiles, RCtl *ctl, int round, int tx, int ty,
                                int f) {
  unsigned *fnext = flags + (size_t)((round + 1) & 1) * ntiles;
  auto flag = [&](int dx, int dy) {
    const int nx = tx + dx, ny = ty + dy;
    if (nx < 0 || ny < 0 || nx >= im.tiles_x || ny >= im.tiles_y) return;
    fnext[im.tile_begin + ny * im.tiles_x + nx] = 1u;
  };
  if (f & B_N) flag(0, -1);
  if (f & B_S) flag(0, 1);
  if (f & B_W) flag(-1, 0);
  if (f & B_E) flag(1, 0);
  if (CONN8) {
    if (f & B_NW) flag(-1, -1);
    if (f & B_NE) flag(1, -1);
    if (f & B_SW) flag(-1, 1);
    if (f & B_SE) flag(1, 1);
  }
  if (f & B_SELF) flag(0, 0);
  // a changed corner pixel is also on a changed edge, so the edge bits cover every flag.  A
  // plain store: the writer does not wait for it (an atomic exchange would return a value).
  if (f & (B_N | B_S | B_W | B_E | B_SELF)) *((volatile unsigned *)&ctl->any[(round + 1) % 3]) = 1u;
}

template <typename T, bool SUP, bool CONN8, int RT>
__device__ void process_tile(const RImg &im, const RParams<T> &P, int t_local, int round, T *s_out, T *s_mask,
                             int *s_flag) {
  constexpr int RTHREADS = RT;
  constexpr int PO = tile_pitch<T>(RT + 2);
  constexpr int PM = tile_pitch<T>(RT);
  const T NEU = Op<T, SUP>::neutral();
  const int tx = t_local % im.tiles_x, ty = t_local / im.tiles_x;
  const int64_t y0 = (int64_t)ty * RT, x0 = (int64_t)tx * RT;
  const T *rec_in = static_cast<const T *>(im.rec);

  // stage: current reconstruction (round 0: marker) with halo, effective mask.  Eight pixels
  // per thread at a time: their loads (at clamped, always valid addresses) are all issued
  // before the first shared-memory store.
  constexpr int NEL = (RT + 2) * (RT + 2);
  constexpr int ITER = (NEL + RTHREADS - 1) / RTHREADS;
  constexpr int CH = 8;
  const bool need_mk = needs_marker(P, round);
  const T *ms_in = static_cast<const T *>(im.mask);
  const T *mk_in = static_cast<const T *>(im.marker);
  for (int k0 = 0; k0 < ITER; k0 += CH) {
    T a[CH], b[CH], c[CH];
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const int i = (k0 + k) * RTHREADS + threadIdx.x;
      const int r = i / (RT + 2) - 1, cc = i % (RT + 2) - 1;
      const int64_t gy = y0 + r, gx = x0 + cc;
      const bool inside = i < NEL && gy >= 0 && gy < im.H && gx >= 0 && gx < im.W;
      const int64_t gi = inside ? gy * im.W + gx : 0;
      a[k] = ldg(ms_in + gi);
      b[k] = need_mk ? ldg(mk_in + gi) : a[k];
      c[k] = round > 0 ? ld_cg(rec_in + gi) : a[k];
    }
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const int i = (k0 + k) * RTHREADS + threadIdx.x;
      if (i >= NEL) break;
      const int r = i / (RT + 2) - 1, cc = i % (RT + 2) - 1;
      const int64_t gy = y0 + r, gx = x0 + cc;
      const bool inside = gy >= 0 && gy < im.H && gx >= 0 && gx < im.W;
      const bool interior = r >= 0 && r < RT && cc >= 0 && cc < RT;
      T v = NEU, m = NEU;
      if (inside) {
        if (round == 0) combine_init<T, SUP>(P, a[k], b[k], m, v);
        else {
          v = c[k];
          m = combine_mask(P, a[k], b[k]);
        }
      }
      s_out[(r + 1) * PO + (cc + 1)] = v;
      if (interior) s_mask[r * PM + cc] = m;
    }
  }
  if (threadIdx.x == 0) *s_flag = 0;
  __syncthreads();

  int bflags = 0;
  bool converged = false;
  // one update: v = sel(op(cur, nb), mask); values are monotone, so "changed" means "grew"
  auto upd = [&](int r, int c, T nb) -> bool {
    T *cell = s_out + (r + 1) * PO + (c + 1);
    const T cur = *cell;
    const T v = Op<T, !SUP>::apply(Op<T, SUP>::apply(cur, nb), s_mask[r * PM + c]);
    if (v != cur) {
      *cell = v;
      if (r == 0) bflags |= B_N;
      if (r == RT - 1) bflags |= B_S;
      if (c == 0) bflags |= B_W;
      if (c == RT - 1) bflags |= B_E;
      if (r == 0 && c == 0) bflags |= B_NW;
      if (r == 0 && c == RT - 1) bflags |= B_NE;
      if (r == RT - 1 && c == 0) bflags |= B_SW;
      if (r == RT - 1 && c == RT - 1) bflags |= B_SE;
      return true;
    }
    return false;
  };
  const int lane = threadIdx.x;  // column for vertical sweeps, row for horizontal ones
  bool changed = false;          // any pixel of the tile changed during this visit
  for (int sweep = 0; sweep < P.max_sweeps; ++sweep) {
    bool ch = false;
    // down: neighbours in the row above
    for (int r = 0; r < RT; ++r) {
      const T *up = s_out + r * PO + lane;  // (r-1, lane-1 .. lane+1) in interior coords
      T nb = up[1];
      if (CONN8) nb = Op<T, SUP>::apply(nb, Op<T, SUP>::apply(up[0], up[2]));
      ch |= upd(r, lane, nb);
      __syncwarp();
    }
    __syncthreads();
    // up: neighbours in the row below
    for (int r = RT - 1; r >= 0; --r) {
      const T *dn = s_out + (r + 2) * PO + lane;
      T nb = dn[1];
      if (CONN8) nb = Op<T, SUP>::apply(nb, Op<T, SUP>::apply(dn[0], dn[2]));
      ch |= upd(r, lane, nb);
      __syncwarp();
    }
    __syncthreads();
    // right: neighbours in the column to the left
    for (int c = 0; c < RT; ++c) {
      const T *lf = s_out + lane * PO + c;  // (lane-1 .. lane+1, c-1)
      T nb = lf[PO];
      if (CONN8) nb = Op<T, SUP>::apply(nb, Op<T, SUP>::apply(lf[0], lf[2 * PO]));
      ch |= upd(lane, c, nb);
      __syncwarp();
    }
    __syncthreads();
    // left: neighbours in the column to the right
    for (int c = RT - 1; c >= 0; --c) {
      const T *rt = s_out + lane * PO + c + 2;
      T nb = rt[PO];
      if (CONN8) nb = Op<T, SUP>::apply(nb, Op<T, SUP>::apply(rt[0], rt[2 * PO]));
      ch |= upd(lane, c, nb);
      __syncwarp();
    }
    if (!__syncthreads_or(ch)) {
      converged = true;
      break;
    }
    changed = true;
  }
  if (!converged) bflags |= B_SELF;
  if (bflags) atomicOr(s_flag, bflags);
  __syncthreads();
  const int f = *s_flag;

  // write back (round 0 always: the marker itself is new; later rounds whenever a pixel
  // changed -- an interior-only change happens when the previous visit yielded) and flag the
  // neighbours
  T *rec = static_cast<T *>(im.rec);
  if (round == 0 || changed) {
    for (int i = threadIdx.x; i < RT * RT; i += RTHREADS) {
      const int r = i / RT, c = i % RT;
      const int64_t gy = y0 + r, gx = x0 + c;
      if (gy < im.H && gx < im.W) st_cg(rec + gy * im.W + gx, s_out[(r + 1) * PO + (c + 1)]);
    }
  }
  if (threadIdx.x == 0 && f != 0) flag_neighbours<CONN8>(im, P.flags, P.ntiles, P.ctl, round, tx, ty, f);
  __syncthreads();
}

// The image that holds a tile, and the tile's index in it.  `begin`: the images' first tiles in shared memory,
// or null (the search then reads the device table, a dependent load per step).
template <typename T>
__device__ __forceinline__ const RImg &image_of(const RParams<T> &P, int tile, int &t_local, const int *begin = nullptr) {
  if (P.nimg == 1) { t_local = tile; return P.single; }
  int lo = 0, hi = P.nimg - 1;
  while (lo < hi) {  // last image whose tile_begin <= tile
    const int mid = (lo + hi + 1) >> 1;
    if ((begin ? begin[mid] : P.imgs[mid].tile_begin) <= tile) lo = mid; else hi = mid - 1;
  }
  t_local = tile - (begin ? begin[lo] : P.imgs[lo].tile_begin);
  return P.imgs[lo];
}

// The pixels of every image cut into as many runs as it has tiles, one warp per run (the images of a batch
// go side by side; image after image over the whole grid, each waited for its loads in turn: 0.9 of the
// 6.2 ms of a 512-image batch, twice): calls run(image, first pixel, end), runs on 16-pixel boundaries.
template <typename T, typename F>
__device__ __forceinline__ void for_pixel_runs(const RParams<T> &P, const int *begin, F run) {
  const int warps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); t < P.ntiles; t += warps) {
    int c = 0;
    const RImg &im = image_of(P, t, c, begin);
    const int64_t n = im.H * im.W, tiles = (int64_t)im.tiles_x * im.tiles_y;
    const int64_t len = ((n + tiles - 1) / tiles + 15) / 16 * 16, lo = c * len;
    if (lo < n) run(im, lo, min(lo + len, n));
  }
}

// Epilogue of pixels [lo, hi) of an image, by one warp, after the last round: the binary h-maxima comparison or
// the leveling clip by the reference.  Pure streaming: 16-byte vectors when the image's buffers allow it,
// otherwise EPI_UNROLL independent elements per lane per step, so that many loads are in flight.
static constexpr int EPI_UNROLL = 8;

template <typename T, bool SUP>
__device__ __forceinline__ uint8_t epi_binary(T ref, T rec) { return ref > rec ? 255 : 0; }

template <typename T, bool SUP>
__device__ __forceinline__ void epilogue_run(const RImg &im, int epi, int64_t lo, int64_t hi) {
  const int lane = threadIdx.x & 31;
  const T *rec = static_cast<const T *>(im.rec);
  const T *ref = static_cast<const T *>(im.mask);
  constexpr int VE = 16 / (int)sizeof(T);  // pixels per 16-byte vector
  const bool vec = ((reinterpret_cast<uintptr_t>(rec) | reinterpret_cast<uintptr_t>(ref) |
                     reinterpret_cast<uintptr_t>(im.out)) % 16 == 0);
  int64_t done = lo;
  if (epi == EPI_BINARY_SUP) {
    uint8_t *o = static_cast<uint8_t *>(im.out);
    if (vec && sizeof(T) == 1) {
      // 16 u8 pixels per lane and step: byte-wise unsigned compare gives 0xff / 0x00 directly
#pragma unroll 2
      for (int64_t j = lo / 16 + lane; j < hi / 16; j += 32) {
        const uint4 a = __ldg(reinterpret_cast<const uint4 *>(ref) + j);
        const uint4 b = __ldcg(reinterpret_cast<const uint4 *>(rec) + j);
        reinterpret_cast<uint4 *>(o)[j] =
            make_uint4(__vcmpgtu4(a.x, b.x), __vcmpgtu4(a.y, b.y), __vcmpgtu4(a.z, b.z), __vcmpgtu4(a.w, b.w));
      }
      done = hi / 16 * 16;
    }
    for (int64_t i0 = done + lane; i0 < hi; i0 += 32 * EPI_UNROLL) {
      T a[EPI_UNROLL], b[EPI_UNROLL];
#pragma unroll
      for (int u = 0; u < EPI_UNROLL; ++u) {
        const int64_t i = i0 + u * 32;
        a[u] = i < hi ? ldg(ref + i) : T(0);
        b[u] = i < hi ? ld_cg(rec + i) : T(0);
      }
#pragma unroll
      for (int u = 0; u < EPI_UNROLL; ++u) {
        const int64_t i = i0 + u * 32;
        if (i < hi) o[i] = epi_binary<T, SUP>(a[u], b[u]);
      }
    }
  } else {  // EPI_CLIP_REF: low leveling min(rec, ref), high leveling max(rec, ref)
    T *o = static_cast<T *>(im.out);
    if (vec) {
#pragma unroll 2
      for (int64_t j = lo / VE + lane; j < hi / VE; j += 32) {
        const Pack<T> a = Pack<T>::load_cg(rec + j * VE);
        const Pack<T> b = Pack<T>::load(ref + j * VE);
        Pack<T>::template op<!SUP>(a, b).store(o + j * VE);
      }
      done = hi / VE * VE;
    }
    for (int64_t i0 = done + lane; i0 < hi; i0 += 32 * EPI_UNROLL) {
      T a[EPI_UNROLL], b[EPI_UNROLL];
#pragma unroll
      for (int u = 0; u < EPI_UNROLL; ++u) {
        const int64_t i = i0 + u * 32;
        a[u] = i < hi ? ld_cg(rec + i) : T(0);
        b[u] = i < hi ? ldg(ref + i) : T(0);
      }
#pragma unroll
      for (int u = 0; u < EPI_UNROLL; ++u) {
        const int64_t i = i0 + u * 32;
        if (i < hi) o[i] = Op<T, !SUP>::apply(a[u], b[u]);
      }
    }
  }
}

template <typename T, bool SUP>
__device__ void recon_epilogue(const RParams<T> &P, const int *begin) {
  for_pixel_runs(P, begin, [&](const RImg &im, int64_t lo, int64_t hi) { epilogue_run<T, SUP>(im, P.epi, lo, hi); });
}

template <typename T, bool SUP, bool CONN8, int RT = tile_side<T>()>
__global__ void __launch_bounds__(RT) k_reconstruct(RParams<T> P) {
  constexpr int PO = tile_pitch<T>(RT + 2);
  constexpr int PM = tile_pitch<T>(RT);
  __shared__ __align__(16) T s_out[(RT + 2) * PO];
  __shared__ __align__(16) T s_mask[RT * PM];
  __shared__ int s_flag;
  __shared__ int s_active;
  RCtl *ctl = P.ctl;

  int round = 0;
  bool ok = true;
  for (;;) {
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->any[(round + 2) % 3] = 0u;
    unsigned *fcur = P.flags + (size_t)(round & 1) * P.ntiles;
    for (int t = blockIdx.x; t < P.ntiles; t += gridDim.x) {
      if (threadIdx.x == 0) {
        int a = 1;
        if (round > 0) {
          a = *((volatile unsigned *)(fcur + t)) != 0u;
          if (a) fcur[t] = 0u;
        }
        s_active = a;
      }
      __syncthreads();
      const bool active = s_active != 0;
      __syncthreads();
      if (active) {
        int tl = 0;
        const RImg &im = image_of(P, t, tl);
        process_tile<T, SUP, CONN8, RT>(im, P, tl, round, s_out, s_mask, &s_flag);
      }
    }
    if (!grid_barrier(ctl, P.wait_ns)) { ok = false; break; }
    const unsigned any = *((volatile unsigned *)&ctl->any[(round + 1) % 3]);
    ++round;
    if (!any) break;
    if (round >= P.max_rounds) {
      if (threadIdx.x == 0) set_status(ctl, PG_ERR_NOT_CONVERGED);
      ok = false;
      break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->rounds = round;
    g_recon_rounds = round;
  }
  if (!ok || P.epi == EPI_NONE) return;
  recon_epilogue<T, SUP>(P, nullptr);
}

// ------------------------------------------------------------------ register tiles
// For pixels of at most 4 bytes the tiles are 32x32 and one warp owns a tile with its values in
// registers: for the vertical sweeps lane c holds column c (v[r] = row r), for the horizontal
// ones the tile goes through shared memory once each way and lane r holds row r.
//  * down / up sweeps take the three pixels of the previous row (8-connected; the same column
//    4-connected), the neighbours' columns by warp shuffles;
//  * right / left sweeps take only the pixel before in the row, a chain inside each lane's
//    registers.  The diagonal relations inside the tile are all covered by the vertical sweeps,
//    and every halo pixel's relations by the one-off halo values below, so a sweep set that
//    changes nothing still means a local fixpoint of the full neighbourhood;
//  * the mask is read from shared memory in either layout (pitch 33 words: conflict-free).
// About one instruction per pixel and sweep set, against some seventy for the shared-memory
// tile above; a CTA holds kRegWarps independent warps.
static constexpr int kRegWarps = 4;
static constexpr int kRP = 33;  // pitch in words of the per-warp shared arrays


// Mask reads inside the sweeps: a volatile shared load is performed where it is written, so the
// compiler does not keep the whole 32x32 mask in registers across sweeps (which would cost 64
// registers per thread and most of the occupancy).
template <typename T> __device__ __forceinline__ T lds_mask(const T *p) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
  uint32_t r;
  asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(r) : "r"(addr));
  if constexpr (std::is_same_v<T, float>) return __uint_as_float(r);
  else return (T)r;
}

template <typename T> __device__ __forceinline__ T shfl_up1(T v) {
  if constexpr (sizeof(T) < 4) return (T)__shfl_up_sync(0xffffffffu, (unsigned)v, 1);
  else return __shfl_up_sync(0xffffffffu, v, 1);
}
template <typename T> __device__ __forceinline__ T shfl_dn1(T v) {
  if constexpr (sizeof(T) < 4) return (T)__shfl_down_sync(0xffffffffu, (unsigned)v, 1);
  else return __shfl_down_sync(0xffffffffu, v, 1);
}

// Tiles of 1- or 2-byte pixels hold two rows per 32-bit register: pair p holds row p (low half) and row 31 - p
// (high half) of the lane's column, so the two chains that the vertical sweeps run at once (down over the top
// half with up over the bottom half, then the reverse) advance together in one 2x16-bit min/max per step;
// after the transpose, pair c holds columns c and 31 - c of the lane's row and the horizontal chains pair up
// the same way.  The masks are packed the same way.
__device__ __forceinline__ uint32_t u16x2_max(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t u16x2_min(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t pk2(uint32_t lo, uint32_t hi) { return __byte_perm(lo, hi, 0x5410); }
__device__ __forceinline__ uint32_t swap2(uint32_t x) { return __byte_perm(x, 0, 0x1032); }

__device__ __forceinline__ uint32_t lds_u32(const uint32_t *p) {  // see lds_mask
  const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
  uint32_t r;
  asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(r) : "r"(addr));
  return r;
}


// Shared memory of a packed tile's warp.  Rows of TP pixels are an odd number of words, so that a lane per row
// and a lane per column both touch 32 banks.
template <typename T> struct PackedCore {
  static constexpr int TP = 32 + 4 / (int)sizeof(T);
  uint32_t ma[16 * kRP];  // mask pairs of the rows (lane = column)
  uint32_t mb[16 * kRP];  // mask pairs of the columns (lane = row)
  T val[32 * TP];         // staged values; transposes; write-back
};
template <typename T> struct PackedTile : PackedCore<T> {
  T mask[32 * PackedCore<T>::TP];  // staged mask
};

// eight bytes from address a on, those outside the image at img zero, one by one (tiles at a buffer's ends)
__device__ __noinline__ uint2 edge_bytes(uintptr_t a, const void *img, uintptr_t bytes) {
  const uintptr_t base = reinterpret_cast<uintptr_t>(img);
  uint32_t w[2] = {0u, 0u};
  for (int b = 0; b < 8; ++b)
    if (a + b >= base && a + b < base + bytes)
      w[b >> 2] |= (uint32_t)*reinterpret_cast<const volatile unsigned char *>(a + b) << (8 * (b & 3));
  return make_uint2(w[0], w[1]);
}

// One array of a tile in 8-byte pieces: pass k brings rows k * RI + lane / LR, piece lane % LR, at any
// alignment: whole aligned words and a funnel shift with the next lane's.
template <typename T, bool CG> struct TileRows {
  static constexpr int LR = 4 * (int)sizeof(T), RI = 32 / LR, PASSES = 32 / RI;
  const T *img;
  uintptr_t a;       // this lane's piece of pass 0
  intptr_t pitch;    // RI rows
  bool safe, pairs;  // every word of the tile in the buffer; pieces aligned to 8 bytes
  __device__ __forceinline__ TileRows(const void *img_, const RImg &im, int64_t y0, int64_t x0, int rows)
      : img(static_cast<const T *>(img_)) {
    const int lane = threadIdx.x & 31;
    const intptr_t row = (intptr_t)im.W * (int)sizeof(T);
    const uintptr_t base = reinterpret_cast<uintptr_t>(img), end = base + (uintptr_t)im.H * row;
    const uintptr_t t = base + (uintptr_t)y0 * row + (uintptr_t)x0 * sizeof(T);
    safe = (t & ~(uintptr_t)3) >= base && t + (rows - 1) * row + 8 * LR + 4 <= end;
    pairs = ((t | (uintptr_t)row) & 7) == 0;
    a = t + (lane / LR) * row + 8 * (lane % LR);
    pitch = RI * row;
  }
  __device__ __forceinline__ static uint32_t ld(uintptr_t p) {
    if constexpr (CG) return __ldcg(reinterpret_cast<const uint32_t *>(p));
    else return __ldg(reinterpret_cast<const uint32_t *>(p));
  }
  // raw words of pass k: the piece's two aligned words and, in a row's last lane, the word after
  __device__ __forceinline__ void load(int k, bool live, const RImg &im, uint32_t (&w)[3]) const {
    const uintptr_t p = a + k * pitch;
    w[0] = w[1] = w[2] = 0u;
    if (!live) return;
    if (!safe) {
      const uint2 v = edge_bytes(p, img, (uintptr_t)(im.H * im.W) * sizeof(T));
      w[0] = v.x;
      w[1] = v.y;
    } else if (pairs) {
      uint2 v;
      if constexpr (CG) v = __ldcg(reinterpret_cast<const uint2 *>(p));
      else v = __ldg(reinterpret_cast<const uint2 *>(p));
      w[0] = v.x;
      w[1] = v.y;
    } else {
      const uintptr_t q = p & ~(uintptr_t)3;
      w[0] = ld(q);
      w[1] = ld(q + 4);
      if ((threadIdx.x & 31) % LR == LR - 1) w[2] = ld(q + 8);
    }
  }
  // the piece's pixels from its raw words; called by the whole warp
  __device__ __forceinline__ uint2 pixels(int k, const uint32_t (&w)[3]) const {
    if (!safe || pairs) return make_uint2(w[0], w[1]);  // uniform
    const unsigned sh = (unsigned)((a + k * pitch) & 3u) * 8u;
    uint32_t n = __shfl_down_sync(0xffffffffu, w[0], 1);
    if ((threadIdx.x & 31) % LR == LR - 1) n = w[2];
    return make_uint2(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], n, sh));
  }
};

// Sweep sets of a packed tile until one changes nothing (returns true) or max_sweeps of them ran.  V: row pairs
// (lane = column), in and out; tb, lr: what the halo contributes to the first pair of each direction; end_lr:
// the outermost column pair (lane = row) at the end.  s.val is overwritten: where a set changed something it
// holds the last values by rows.
template <typename T, bool SUP, bool CONN8>
__device__ __forceinline__ bool packed_sweeps(uint32_t (&V)[16], PackedCore<T> &s, uint32_t tb, uint32_t lr, int max_sweeps,
                                              uint32_t &end_lr, bool &changed) {
  constexpr int TP = PackedCore<T>::TP;
  const int lane = threadIdx.x & 31;
  auto OS = [](uint32_t a, uint32_t b) { return SUP ? u16x2_max(a, b) : u16x2_min(a, b); };  // propagation
  auto OC = [](uint32_t a, uint32_t b) { return SUP ? u16x2_min(a, b) : u16x2_max(a, b); };  // clip by the mask
  auto nbrow = [&](uint32_t x) -> uint32_t {
    if (CONN8) {
      const uint32_t a = __shfl_up_sync(0xffffffffu, x, 1), b = __shfl_down_sync(0xffffffffu, x, 1);
      return OS(x, OS(a, b));
    }
    return x;
  };
  const uint32_t *MAs = s.ma + lane, *MBs = s.mb + lane;
  changed = false;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    uint32_t ch = 0;
    // vertical: pair k from pair k - 1 (k = 0: the halo rows), then pair 15 from itself swapped and pair q
    // from pair q + 1
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t nb = k == 0 ? tb : nbrow(V[k - 1]);  // the halo rows are already 3-wide
      const uint32_t nv = OC(OS(V[k], nb), lds_u32(MAs + k * kRP));
      ch |= nv ^ V[k];
      V[k] = nv;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int q = 15 - k;
      const uint32_t nb = nbrow(k == 0 ? swap2(V[15]) : V[q + 1]);
      const uint32_t nv = OC(OS(V[q], nb), lds_u32(MAs + q * kRP));
      ch |= nv ^ V[q];
      V[q] = nv;
    }
    // to lane = row
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      s.val[p * TP + lane] = (T)V[p];
      s.val[(31 - p) * TP + lane] = (T)(V[p] >> 16);
    }
    __syncwarp();
    uint32_t Q[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) Q[c] = pk2(s.val[lane * TP + c], s.val[lane * TP + 31 - c]);
    __syncwarp();
    // horizontal, the same pairing
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t nb = k == 0 ? lr : Q[k - 1];
      const uint32_t nv = OC(OS(Q[k], nb), lds_u32(MBs + k * kRP));
      ch |= nv ^ Q[k];
      Q[k] = nv;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int q = 15 - k;
      const uint32_t nb = k == 0 ? swap2(Q[15]) : Q[q + 1];
      const uint32_t nv = OC(OS(Q[q], nb), lds_u32(MBs + q * kRP));
      ch |= nv ^ Q[q];
      Q[q] = nv;
    }
    end_lr = Q[0];
    const bool any = __any_sync(0xffffffffu, ch != 0);
    changed |= any;
    // back to lane = column (where nothing moved, s.val still holds the values by rows)
    if (any) {
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        s.val[lane * TP + c] = (T)Q[c];
        s.val[lane * TP + 31 - c] = (T)(Q[c] >> 16);
      }
      __syncwarp();
    }
#pragma unroll
    for (int p = 0; p < 16; ++p) V[p] = pk2(s.val[p * TP + lane], s.val[(31 - p) * TP + lane]);
    __syncwarp();
    if (!any) return true;
  }
  return false;
}

// A halo pixel's contribution goes into one value per border pixel; 8-connected: of the three pixels beside it.
// h_top, h_bot: per column; h_l, h_r: per row; c_top, c_bot: the corners, left ones in lane 0, right in lane 31.
template <typename T, bool SUP>
__device__ __forceinline__ void fold_halo(T &h_top, T &h_bot, T &h_l, T &h_r, T c_top, T c_bot) {
  using OT = Op<T, SUP>;
  auto up1 = [](T v, T first) {
    const T n = (T)__shfl_up_sync(0xffffffffu, (unsigned)v, 1);
    return (threadIdx.x & 31) == 0 ? first : n;
  };
  auto dn1 = [](T v, T last) {
    const T n = (T)__shfl_down_sync(0xffffffffu, (unsigned)v, 1);
    return (threadIdx.x & 31) == 31 ? last : n;
  };
  const T bl = (T)__shfl_sync(0xffffffffu, (unsigned)c_bot, 0), tr = (T)__shfl_sync(0xffffffffu, (unsigned)c_top, 31);
  const T t3 = OT::apply(h_top, OT::apply(up1(h_top, c_top), dn1(h_top, c_top)));
  const T b3 = OT::apply(h_bot, OT::apply(up1(h_bot, c_bot), dn1(h_bot, c_bot)));
  const T l3 = OT::apply(h_l, OT::apply(up1(h_l, c_top), dn1(h_l, bl)));
  const T r3 = OT::apply(h_r, OT::apply(up1(h_r, tr), dn1(h_r, c_bot)));
  h_top = t3; h_bot = b3; h_l = l3; h_r = r3;
}

// two border pixels after their halo: the value, pulled by the halo's within the mask
template <bool SUP> __device__ __forceinline__ uint32_t pulled(uint32_t v, uint32_t halo, uint32_t mask) {
  return SUP ? u16x2_min(u16x2_max(v, halo), mask) : u16x2_max(u16x2_min(v, halo), mask);
}

// One visit of a packed tile: as process_tile_reg below, but the pixels stay in their own width in shared memory
// (6.5 KB a warp for u8, five CTAs per SM) and come in whole words at any alignment.  Rows of no whole 16-byte
// vectors were staged pixel by pixel before: 21500 of a visit's 37700 cycles in a 512-image batch (sweeps 8100),
// now 6600 of 22300; with the runs of for_pixel_runs and a search of the images in shared memory the batch of
// 512 u8 images of 64-1024 pixels a side takes 2.24 ms (before: 6.25), one 2048^2 u8 image 131 us a call (177).
// A visit is bound by latency: loads 6600 cycles, sweeps 7300, the fence, atomics and slot of its end 10300.
template <typename T, bool SUP, bool CONN8>
__device__ __forceinline__ int process_tile_packed(const RImg &im, const RParams<T> &P, int t_local, bool settled,
                                                   PackedTile<T> &s) {
  static_assert(sizeof(T) <= 2, "two pixels per register");
  constexpr int S = (int)sizeof(T), TP = PackedTile<T>::TP;
  using OT = Op<T, SUP>;
  constexpr int LR = TileRows<T, true>::LR, RI = TileRows<T, true>::RI, PASSES = TileRows<T, true>::PASSES;
  const int lane = threadIdx.x & 31;
  const T NEU = OT::neutral();
  const uint32_t NEUW = splat<T>(NEU);
  const int tx = t_local % im.tiles_x, ty = t_local / im.tiles_x;
  const int64_t y0 = (int64_t)ty * 32, x0 = (int64_t)tx * 32;
  const int rows = (int)min((int64_t)32, im.H - y0), cols = (int)min((int64_t)32, im.W - x0);
  const T *rec_in = static_cast<const T *>(im.rec);

  // Halo, fixed during the visit: the row above and below per column, the columns left and right per row, and
  // the four corners in lanes 0 (left) and 31 (right); outside the image the neutral value.
  T h_top = NEU, h_bot = NEU, h_l = NEU, h_r = NEU, c_top = NEU, c_bot = NEU;
  {
    const T *top = rec_in + (y0 - 1) * im.W + x0, *bot = rec_in + (y0 + 32) * im.W + x0;
    const T *left = rec_in + (y0 + lane) * im.W + x0 - 1;
    const bool up = ty > 0, down = ty + 1 < im.tiles_y, west = tx > 0, east = tx + 1 < im.tiles_x;
    if (up && lane < cols) h_top = ld_cg(top + lane);
    if (down && lane < cols) h_bot = ld_cg(bot + lane);
    if (west && lane < rows) h_l = ld_cg(left);
    if (east && lane < rows) h_r = ld_cg(left + 33);
    if (CONN8 && ((lane == 0 && west) || (lane == 31 && east))) {
      const int c = lane == 0 ? -1 : 32;
      if (up) c_top = ld_cg(top + c);
      if (down) c_bot = ld_cg(bot + c);
    }
  }
  // stage: the loads of four passes of both arrays go together
  const TileRows<T, true> r_rec(im.rec, im, y0, x0, rows);
  {
    const TileRows<T, false> r_mask(im.mask, im, y0, x0, rows);
#pragma unroll
    for (int k0 = 0; k0 < PASSES; k0 += 4) {
      uint32_t wm[4][3], wr[4][3];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool live = (k0 + k) * RI + lane / LR < rows;
        r_mask.load(k0 + k, live, im, wm[k]);
        r_rec.load(k0 + k, live, im, wr[k]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint2 m = r_mask.pixels(k0 + k, wm[k]), v = r_rec.pixels(k0 + k, wr[k]);
        const int row = (k0 + k) * RI + lane / LR;
        uint32_t *sm = reinterpret_cast<uint32_t *>(s.mask + row * TP) + 2 * (lane % LR);
        uint32_t *sv = reinterpret_cast<uint32_t *>(s.val + row * TP) + 2 * (lane % LR);
        sm[0] = m.x;
        sm[1] = m.y;
        sv[0] = v.x;
        sv[1] = v.y;
      }
    }
  }
  if (needs_marker(P, 1)) {  // leveling: the effective mask
    const TileRows<T, false> r_mark(im.marker, im, y0, x0, rows);
#pragma unroll
    for (int k0 = 0; k0 < PASSES; k0 += 4) {
      uint32_t wk[4][3];
#pragma unroll
      for (int k = 0; k < 4; ++k) r_mark.load(k0 + k, (k0 + k) * RI + lane / LR < rows, im, wk[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint2 b = r_mark.pixels(k0 + k, wk[k]);
        uint32_t *sm = reinterpret_cast<uint32_t *>(s.mask + ((k0 + k) * RI + lane / LR) * TP) + 2 * (lane % LR);
        if (P.mask_mode == MASK_MAX_MARKER) {
          sm[0] = wop<T, true>(sm[0], b.x);
          sm[1] = wop<T, true>(sm[1], b.y);
        } else {
          sm[0] = wop<T, false>(sm[0], b.x);
          sm[1] = wop<T, false>(sm[1], b.y);
        }
      }
    }
  }
  if (rows < 32 || cols < 32) {  // uniform: pixels outside the image are neutral
#pragma unroll 1
    for (int k = 0; k < PASSES; ++k) {
      const int row = k * RI + lane / LR;
      const int nb = row < rows ? min(max(cols * S - 8 * (lane % LR), 0), 8) : 0;
      const unsigned long long in_m = nb == 8 ? ~0ull : (1ull << (8 * nb)) - 1ull;
      uint32_t *sm = reinterpret_cast<uint32_t *>(s.mask + row * TP) + 2 * (lane % LR);
      uint32_t *sv = reinterpret_cast<uint32_t *>(s.val + row * TP) + 2 * (lane % LR);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const uint32_t m = (uint32_t)(in_m >> (32 * j));
        sm[j] = (sm[j] & m) | (NEUW & ~m);
        sv[j] = (sv[j] & m) | (NEUW & ~m);
      }
    }
  }
  __syncwarp();
  uint32_t V[16];
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    V[p] = pk2(s.val[p * TP + lane], s.val[(31 - p) * TP + lane]);
    s.ma[p * kRP + lane] = pk2(s.mask[p * TP + lane], s.mask[(31 - p) * TP + lane]);
    s.mb[p * kRP + lane] = pk2(s.mask[lane * TP + p], s.mask[lane * TP + 31 - p]);
  }
  // staged borders, to tell afterwards which neighbours must be revisited
  const uint32_t init_tb = V[0], init_lr = pk2(s.val[lane * TP], s.val[lane * TP + 31]);
  __syncwarp();
  if (CONN8) fold_halo<T, SUP>(h_top, h_bot, h_l, h_r, c_top, c_bot);
  const uint32_t tb = pk2(h_top, h_bot), lr = pk2(h_l, h_r);
  // A settled tile whose halo moves nothing is done.  512 u8 images of 64-1024 pixels 2356 -> 2238 us, leveling 4096^2
  // u8 793 -> 766; u16 has no register left for it (leveling 3000 x 4001 911 -> 948), nor have the 4-byte tiles
  // (binary h-maxima 2048^2 f32 198 -> 211).
  if constexpr (sizeof(T) == 1) {
    if (settled && !__any_sync(0xffffffffu, pulled<SUP>(V[0], tb, s.ma[lane]) != V[0] ||
                                                pulled<SUP>(init_lr, lr, s.mb[lane]) != init_lr))
      return 0;
  }

  uint32_t end_lr = init_lr;
  bool changed = false;
  const bool converged = packed_sweeps<T, SUP, CONN8>(V, s, tb, lr, P.max_sweeps, end_lr, changed);

  const uint32_t d_tb = V[0] ^ init_tb, d_lr = end_lr ^ init_lr;
  const unsigned bN = __ballot_sync(0xffffffffu, (d_tb & 0xffffu) != 0u), bS = __ballot_sync(0xffffffffu, (d_tb >> 16) != 0u);
  const unsigned bW = __ballot_sync(0xffffffffu, (d_lr & 0xffffu) != 0u), bE = __ballot_sync(0xffffffffu, (d_lr >> 16) != 0u);
  int f = converged ? 0 : B_SELF;
  if (bN) f |= B_N;
  if (bS) f |= B_S;
  if (bW) f |= B_W;
  if (bE) f |= B_E;
  if (bN & 1u) f |= B_NW;
  if (bN >> 31) f |= B_NE;
  if (bS & 1u) f |= B_SW;
  if (bS >> 31) f |= B_SE;

  if (changed) {
    T *rec = static_cast<T *>(im.rec);
    if (r_rec.pairs && cols == 32) {
      // s.val holds the last values by rows (the transposes leave them there): 8-byte pieces out
#pragma unroll
      for (int k = 0; k < PASSES; ++k) {
        const int row = k * RI + lane / LR;
        const uint32_t *sv = reinterpret_cast<const uint32_t *>(s.val + row * TP) + 2 * (lane % LR);
        if (row < rows) __stcg(reinterpret_cast<uint2 *>(r_rec.a + k * r_rec.pitch), make_uint2(sv[0], sv[1]));
      }
    } else if (lane < cols) {
      T *p = rec + y0 * im.W + x0 + lane;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        if (r < rows) st_cg(p + r * im.W, (T)(r < 16 ? V[r] : V[31 - r] >> 16));
      }
    }
    __syncwarp();
  }
  return f;
}

// One visit of a register tile: stage it from the reconstruction buffer (which the worklist
// kernel's first phase set to the marker), iterate sweep sets to the tile-local fixpoint (or
// P.max_sweeps), write it back if anything changed.  Returns the B_* bits of the borders that
// changed (the neighbours to revisit) and B_SELF when the tile yielded.  Warp-uniform.
template <typename T, bool SUP, bool CONN8>
__device__ int process_tile_reg(const RImg &im, const RParams<T> &P, int t_local, T *s_m, T *s_t) {
  using OS = Op<T, SUP>;   // propagation
  using OC = Op<T, !SUP>;  // clip by the mask
  const int lane = threadIdx.x & 31;
  const T NEU = OS::neutral();
  const int tx = t_local % im.tiles_x, ty = t_local / im.tiles_x;
  const int64_t y0 = (int64_t)ty * 32, x0 = (int64_t)tx * 32;
  const T *rec_in = static_cast<const T *>(im.rec);
  const int64_t gx = x0 + lane;
  const bool colin = gx < im.W;

  // Halo loads first (they stay in flight during the stage).  Its values stay fixed during the
  // visit, so each halo pixel's contribution is folded into one value per border pixel:
  // `top`/`bot` per column (lane = column: the three pixels above / below), `hl`/`hr` per row
  // (lane = row: the three pixels left / right; one in 4-connectivity).  The sweeps apply them
  // at the tile's first/last row and column.  Addresses outside the image are clamped to pixel
  // 0 and the values replaced by the neutral element.
  constexpr int NH = CONN8 ? 12 : 4;
  const int64_t hy[12] = {y0 - 1, y0 + 32, y0 + lane, y0 + lane, y0 - 1, y0 - 1, y0 + 32, y0 + 32,
                          y0 + lane - 1, y0 + lane + 1, y0 + lane - 1, y0 + lane + 1};
  const int64_t hx[12] = {gx, gx, x0 - 1, x0 + 32, gx - 1, gx + 1, gx - 1, gx + 1, x0 - 1, x0 - 1, x0 + 32, x0 + 32};
  T hv[NH];
#pragma unroll
  for (int k = 0; k < NH; ++k) {
    const bool in = hy[k] >= 0 && hy[k] < im.H && hx[k] >= 0 && hx[k] < im.W;
    hv[k] = ld_cg(rec_in + (in ? hy[k] * im.W + hx[k] : 0));
    if (!in) hv[k] = NEU;  // applied after the load returns; the load itself is unconditional
  }

  // stage, lane = column: tile values and mask (pixels outside the image: neutral, fixed).
  const T *mk_in = static_cast<const T *>(im.marker);
  const T *ms_in = static_cast<const T *>(im.mask);
  const bool need_mk = needs_marker(P, 1);
  T v[32];
  // loads come first, 16 rows at a time, so that they are all in flight together
#pragma unroll
  for (int h = 0; h < 32; h += 16) {
    T a[16], b[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const int64_t gy = y0 + h + r;
      const int64_t gi = (colin && gy < im.H) ? gy * im.W + gx : 0;
      a[r] = ldg(ms_in + gi);
      b[r] = need_mk ? ldg(mk_in + gi) : a[r];
      v[h + r] = ld_cg(rec_in + gi);
    }
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      const bool ok = colin && y0 + h + r < im.H;
      T m = combine_mask(P, a[r], b[r]);
      if (!ok) {
        m = NEU;
        v[h + r] = NEU;
      }
      s_m[(h + r) * kRP + lane] = m;
    }
  }
  T top = hv[0], bot = hv[1], hl = hv[2], hr = hv[3];
  if (CONN8) {
    top = OS::apply(top, OS::apply(hv[4], hv[5]));
    bot = OS::apply(bot, OS::apply(hv[6], hv[7]));
    hl = OS::apply(hl, OS::apply(hv[8], hv[9]));
    hr = OS::apply(hr, OS::apply(hv[10], hv[11]));
  }
  // staged borders, to tell afterwards which neighbours must be revisited
#pragma unroll
  for (int r = 0; r < 32; ++r) s_t[r * kRP + lane] = v[r];
  __syncwarp();
  const T initL = (T)s_t[lane * kRP], initR = (T)s_t[lane * kRP + 31];
  const T initT = v[0], initB = v[31];
  __syncwarp();

  bool converged = false, changed = false, wch = false, ech = false;
  for (int sweep = 0; sweep < P.max_sweeps; ++sweep) {
    bool ch = false;
    auto vstep = [&](int r, T nb) {
      const T nv = OC::apply(OS::apply(v[r], nb), lds_mask<T>(s_m + r * kRP + lane));
      ch |= nv != v[r];
      v[r] = nv;
    };
    // the three pixels of a row seen from the row below / above (lanes 0 and 31 get their own
    // value back from the shuffle: the pixels beyond the tile's sides are halo, applied by the
    // horizontal sweeps)
    auto nbrow = [&](T p) -> T {
      if (CONN8) return OS::apply(p, OS::apply(shfl_up1(p), shfl_dn1(p)));
      return p;
    };
    // vertical, two independent chains at once: down over the top half with up over the
    // bottom half, then down over the bottom half with up over the top half.  A value still
    // travels the whole column in one direction per sweep set.
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const T nd = (k == 0) ? top : nbrow(v[k - 1]);
      const T nu = (k == 0) ? bot : nbrow(v[32 - k]);
      vstep(k, nd);
      vstep(31 - k, nu);
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const T nd = nbrow(v[15 + k]);
      const T nu = nbrow(v[16 - k]);
      vstep(16 + k, nd);
      vstep(15 - k, nu);
    }
    // to lane = row
#pragma unroll
    for (int r = 0; r < 32; ++r) s_t[r * kRP + lane] = v[r];
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 32; ++c) v[c] = (T)s_t[lane * kRP + c];
    __syncwarp();
    // horizontal (the pixel on the left / on the right), two chains at once in the same way
    auto hstep = [&](int c, T nb) {
      const T nv = OC::apply(OS::apply(v[c], nb), lds_mask<T>(s_m + lane * kRP + c));
      ch |= nv != v[c];
      v[c] = nv;
    };
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      hstep(k, k == 0 ? hl : v[k - 1]);
      hstep(31 - k, k == 0 ? hr : v[32 - k]);
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      hstep(16 + k, v[15 + k]);
      hstep(15 - k, v[16 - k]);
    }
    wch = v[0] != initL;
    ech = v[31] != initR;
    // back to lane = column
#pragma unroll
    for (int c = 0; c < 32; ++c) s_t[lane * kRP + c] = v[c];
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 32; ++r) v[r] = (T)s_t[r * kRP + lane];
    __syncwarp();
    if (!__any_sync(0xffffffffu, ch)) {
      converged = true;
      break;
    }
    changed = true;
  }

  const unsigned bN = __ballot_sync(0xffffffffu, v[0] != initT);
  const unsigned bS = __ballot_sync(0xffffffffu, v[31] != initB);
  const unsigned bW = __ballot_sync(0xffffffffu, wch);
  const unsigned bE = __ballot_sync(0xffffffffu, ech);
  int f = converged ? 0 : B_SELF;
  if (bN) f |= B_N;
  if (bS) f |= B_S;
  if (bW) f |= B_W;
  if (bE) f |= B_E;
  if (bN & 1u) f |= B_NW;
  if (bN >> 31) f |= B_NE;
  if (bS & 1u) f |= B_SW;
  if (bS >> 31) f |= B_SE;

  if (changed) {
    // the row stride goes through a shuffle so that the compiler recomputes these addresses
    // here instead of keeping the stage's 32 row addresses alive across the sweeps
    const long long Wd = __shfl_sync(0xffffffffu, (long long)im.W, 0);
    T *p = static_cast<T *>(im.rec) + (y0 * Wd + gx);
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      if (colin && y0 + r < im.H) st_cg(p, v[r]);
      p += Wd;
    }
  }
  return f;
}

// ------------------------------------------------------------------ tile worklist
// The register-tile kernel has no rounds.  Every tile is queued once at the start; a warp pops
// a tile, visits it, and queues the neighbours whose shared border changed.  The kernel ends
// when no tile is queued or being visited (`pending` == 0).  A tile is visited by one warp at a
// time, through its state:
//   IDLE --queue--> QUEUED --pop--> RUNNING --done--> IDLE (or QUEUED again if it yielded)
//   RUNNING --a neighbour changed its border meanwhile--> DIRTY --done--> QUEUED
// The queue is a ring of 64-bit slots (position tag << 32 | kSettled | tile + 1), a multi-producer multi-
// consumer ring with sequence numbers: a popper takes a ticket with one atomicAdd on `head`
// and waits for its slot to carry its position; a pusher takes positions with one atomicAdd
// on `tail` and waits until the slot's previous lap was consumed (tag = position - cap, tile
// field 0).  No compare-and-swap retries on the shared counters.
enum : unsigned { TS_IDLE = 0, TS_QUEUED = 1, TS_RUNNING = 2, TS_DIRTY = 3 };

// `tail` (next position to push, low 32 bits) and `pending` (tiles queued or being visited, high
// 32 bits) share one 64-bit word, so that a warp counts the tiles it pushes and reserves their
// positions in one atomic: a tile cannot be popped and finished (pending - 1) before its own
// pending + 1 is performed.
struct RQueue {                // each counter on its own 128-byte line
  unsigned head, pad0[31];     // next ticket to pop
  unsigned long long tp;       // pending << 32 | tail
  unsigned pad1[30];
  unsigned pad2[64];
};
__device__ __forceinline__ unsigned tp_tail(unsigned long long tp) { return (unsigned)tp; }
__device__ __forceinline__ int tp_pending(unsigned long long tp) { return (int)(tp >> 32); }
static_assert(sizeof(RQueue) == 512, "RQueue layout");

template <typename T> struct WorkList {
  RQueue *q;
  unsigned *state;             // ntiles
  unsigned long long *ring;    // cap slots
  unsigned cap;
  unsigned long long wait_ns;  // limit of every bounded wait
};

__device__ __forceinline__ bool wait_expired(RCtl *ctl, unsigned long long t0, unsigned long long wait_ns) {
  if (global_ns() - t0 > wait_ns) {
    set_status(ctl, PG_ERR_NOT_CONVERGED);
    return true;
  }
  return false;
}

__device__ __forceinline__ unsigned long long slot_val(unsigned pos, unsigned tile1) {
  return ((unsigned long long)pos << 32) | tile1;
}

// In a slot's tile field: the tile's last visit ended at its local fixpoint (it was idle when a neighbour queued
// it, or it was dirtied during that visit), so it moves only if its new halo moves a border pixel.  u8 tiles look.
template <typename T> constexpr unsigned kSettled = sizeof(T) == 1 ? 0x80000000u : 0u;

// Lane 0 pops ticket `pos`: the slot's tile field (tile + 1 and kSettled), or 0 when the work is done or an error was
// recorded.  A waiting
// warp polls its own slot only (every idle warp polling the shared counters as well slowed the atomics on
// them): the warp that ends the last visit fills the slots of the tickets still out with kExit, and a warp that
// takes its ticket later sees `pending` at zero on its first poll.
static constexpr unsigned kExit = 0xffffffffu;

template <typename T>
__device__ unsigned wl_pop(const WorkList<T> &wl, RCtl *ctl, unsigned pos, long long max_tickets) {
  if ((long long)pos >= max_tickets) {  // runaway guard: far more visits than any input needs
    set_status(ctl, PG_ERR_NOT_CONVERGED);
    return 0u;
  }
  volatile unsigned long long *slot = wl.ring + pos % wl.cap;
  const unsigned long long t0 = global_ns();
  unsigned long long v;
  for (unsigned polls = 0;; ++polls) {
    v = *slot;
    unsigned long long tp = ~0ull;
    if (polls % 16 == 0) tp = *((volatile unsigned long long *)&wl.q->tp);  // with the slot: one round trip
    if ((unsigned)(v >> 32) == pos && (unsigned)v != 0u) break;
    if (tp_pending(tp) == 0) return 0u;
    if (polls % 16 == 15) {
      if (*((volatile int *)&ctl->status) != 0) return 0u;
      if (wait_expired(ctl, t0, wl.wait_ns)) return 0u;
    }
    __nanosleep(polls < 8 ? 40 : 200);
  }
  if ((unsigned)v == kExit) return 0u;
  *slot = slot_val(pos, 0u);  // consumed: the next lap's pusher may write
  const unsigned tile = ((unsigned)v & ~kSettled<T>) - 1u;
  *((volatile unsigned *)(wl.state + tile)) = TS_RUNNING;  // QUEUED until now: nobody else moves it
  __threadfence();  // the neighbours' pixels written before they queued this tile
  return (unsigned)v;
}

// Retry limit of the state-change loops below: a retry means another warp changed the same
// word in between, which happens a bounded number of times; the limit only guards the kernel.
static constexpr int kCasRetries = 1 << 20;

// Warp-wide end of a visit: lanes 0..7 queue the neighbours whose shared border changed (one
// lane each, in parallel), lane 8 releases the tile (or queues it again), and the queued tiles
// are pushed with one position reservation for the warp.  Called by the whole warp.
// (Keeping one queued neighbour as the warp's next visit, past the ring, was measured: it
// shortens long propagations but makes tiles of short ones -- the h-extrema -- be revisited
// more often, so every queued tile goes through the ring.)
template <typename T, bool CONN8>
__device__ void wl_finish(const WorkList<T> &wl, RCtl *ctl, const RImg &im, int tile, int t_local, int f) {
  const int lane = threadIdx.x & 31;
  const int tx = t_local % im.tiles_x, ty = t_local / im.tiles_x;
  // lane d < 8 handles direction d = N S W E NW NE SW SE, whose B_* bit is 1 << d
  int cand = -1;
  bool push = false;
  if (lane < (CONN8 ? 8 : 4) && (f & (1 << lane))) {
    const int dx = lane < 2 ? 0 : ((lane & 1) ? 1 : -1);
    const int dy = lane < 2 ? (lane ? 1 : -1) : lane < 4 ? 0 : (lane < 6 ? -1 : 1);
    const int nx = tx + dx, ny = ty + dy;
    if (nx >= 0 && ny >= 0 && nx < im.tiles_x && ny < im.tiles_y) cand = im.tile_begin + ny * im.tiles_x + nx;
  }
  // Every lane's expected transition in one compare-and-swap, all in flight together; what another warp moved
  // in between is settled after.
  const bool self = lane == 8, yielded = (f & B_SELF) != 0;
  if (self) cand = tile;
  if (cand >= 0) {
    unsigned want = self ? TS_RUNNING : TS_IDLE, to = self && !yielded ? TS_IDLE : TS_QUEUED;
    bool done = false;
    for (int it = 0; it < kCasRetries && !done; ++it) {
      const unsigned s = atomicCAS(wl.state + cand, want, to);
      if (s == want) {
        push = to == TS_QUEUED;
        done = true;
      } else if (self) {  // DIRTY: a neighbour changed its border meanwhile; only we move it out
        want = s;
        to = TS_QUEUED;
      } else if (s == TS_RUNNING) {
        want = TS_RUNNING;
        to = TS_DIRTY;
      } else if (s == TS_IDLE) {
        want = TS_IDLE;
        to = TS_QUEUED;
      } else {
        done = true;  // already queued, or already marked for another visit
      }
    }
    if (!done) set_status(ctl, PG_ERR_NOT_CONVERGED);
  }
  const unsigned pm = __ballot_sync(0xffffffffu, push);
  // One atomic reserves the pushed tiles' positions, counts them and takes this visit off `pending`: a tile
  // cannot be popped and finished before it is counted, so `pending` is zero only when all work is done.
  const int n = __popc(pm);
  unsigned base = 0, left = 0;
  if (lane == 0) {
    const unsigned long long add = ((unsigned long long)(unsigned)(n - 1) << 32) + (unsigned)n;
    const unsigned long long tp = atomicAdd(&wl.q->tp, add);
    base = tp_tail(tp);
    left = (unsigned)tp_pending(tp + add);
  }
  base = __shfl_sync(0xffffffffu, base, 0);
  left = __shfl_sync(0xffffffffu, left, 0);
  if (push) {
    const unsigned pos = base + __popc(pm & ((1u << lane) - 1u));
    volatile unsigned long long *slot = wl.ring + pos % wl.cap;
    const unsigned long long want = slot_val(pos - wl.cap, 0u);  // previous lap consumed
    // the first lap's slots were set to `want` before the grid barrier of phase 0: no need to look
    if (pos >= wl.cap) {
      const unsigned long long t0 = global_ns();
      while (*slot != want) {
        __nanosleep(64);
        if (wait_expired(ctl, t0, wl.wait_ns)) break;
      }
    }
    // a neighbour pushed here was idle: its last visit had settled; this tile settled unless it yielded
    *slot = slot_val(pos, ((unsigned)cand + 1u) | (self && yielded ? 0u : kSettled<T>));
  }
  if (left == 0) {  // the last visit: release the warps that wait (tickets from the tail on)
    unsigned head = 0;
    if (lane == 0) {
      __threadfence();  // a ticket taken after this read finds `pending` at zero
      head = atomicAdd(&wl.q->head, 0u);
    }
    head = __shfl_sync(0xffffffffu, head, 0);
    for (unsigned pos = base + (unsigned)n + lane; (int)(head - pos) > 0; pos += 32)
      *((volatile unsigned long long *)(wl.ring + pos % wl.cap)) = slot_val(pos, kExit);
  }
}

// first phase: every reconstruction buffer starts at the marker (select_marker, or the saturated shift of the
// h-extrema)
template <typename T, bool SUP>
__device__ void init_rec(const RParams<T> &P, const int *begin) {
  const bool need_mk = needs_marker(P, 0);
  const int lane = threadIdx.x & 31;
  for_pixel_runs(P, begin, [&](const RImg &im, int64_t lo, int64_t hi) {
    const T *ms = static_cast<const T *>(im.mask);
    const T *mk = need_mk ? static_cast<const T *>(im.marker) : ms;
    T *rec = static_cast<T *>(im.rec);
    constexpr int VE = Pack<T>::N;
    int64_t done = lo;
    if ((reinterpret_cast<uintptr_t>(ms) | reinterpret_cast<uintptr_t>(mk) | reinterpret_cast<uintptr_t>(rec)) % 16 == 0) {
#pragma unroll 2
      for (int64_t j = lo / VE + lane; j < hi / VE; j += 32) {
        const Pack<T> a = Pack<T>::load(ms + j * VE), b = need_mk ? Pack<T>::load(mk + j * VE) : a;
        Pack<T> r;
#pragma unroll
        for (int e = 0; e < VE; ++e) {
          T m;
          combine_init<T, SUP>(P, a.e[e], b.e[e], m, r.e[e]);
        }
        __stcg(reinterpret_cast<uint4 *>(rec + j * VE), r.v);
      }
      done = hi / VE * VE;
    }
    for (int64_t i0 = done + lane; i0 < hi; i0 += 32 * EPI_UNROLL) {
      T a[EPI_UNROLL], b[EPI_UNROLL];
#pragma unroll
      for (int u = 0; u < EPI_UNROLL; ++u) {
        const int64_t i = i0 + u * 32;
        a[u] = i < hi ? ldg(ms + i) : T(0);
        b[u] = (need_mk && i < hi) ? ldg(mk + i) : a[u];
      }
#pragma unroll
      for (int u = 0; u < EPI_UNROLL; ++u) {
        const int64_t i = i0 + u * 32;
        T m, v;
        combine_init<T, SUP>(P, a[u], b[u], m, v);
        if (i < hi) st_cg(rec + i, v);
      }
    }
  });
}

__device__ long long g_recon_visits = 0;

template <typename T> struct TileSmem {
  static constexpr size_t bytes = 2 * 32 * kRP * sizeof(T);  // process_tile_reg's two arrays
};
template <> struct TileSmem<uint8_t> { static constexpr size_t bytes = (sizeof(PackedTile<uint8_t>) + 15) / 16 * 16; };
template <> struct TileSmem<uint16_t> { static constexpr size_t bytes = (sizeof(PackedTile<uint16_t>) + 15) / 16 * 16; };
constexpr int kBeginMax = 1024;  // images whose first tiles are kept in shared memory

template <typename T, bool SUP, bool CONN8>
__global__ void __launch_bounds__(kRegWarps * 32, sizeof(T) <= 2 ? 5 : 4) k_reconstruct_wl(const __grid_constant__ RParams<T> P,
                                                                                          const WorkList<T> wl) {
  static_assert(sizeof(T) <= 4, "register tiles hold pixels of at most 4 bytes");
  __shared__ __align__(16) unsigned char s_raw[kRegWarps][TileSmem<T>::bytes];
  __shared__ int s_begin[kBeginMax];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  RCtl *ctl = P.ctl;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nth = (int64_t)gridDim.x * blockDim.x;

  // the images' first tiles, for the searches of image_of
  const int *begin = P.nimg > 1 && P.nimg <= kBeginMax ? s_begin : nullptr;
  if (begin) {
    for (int k = threadIdx.x; k < P.nimg; k += blockDim.x) s_begin[k] = P.imgs[k].tile_begin;
    __syncthreads();
  }
  // phase 0: marker into the reconstruction buffers, every tile queued once
  init_rec<T, SUP>(P, begin);
  for (int64_t i = tid; i < (int64_t)wl.cap; i += nth) {
    // positions 0..ntiles-1 hold the tiles; the others wait for their first lap
    wl.ring[i] = i < P.ntiles ? slot_val((unsigned)i, (unsigned)i + 1u) : slot_val((unsigned)i - wl.cap, 0u);
    if (i < P.ntiles) wl.state[i] = TS_QUEUED;
  }
  const unsigned warps = (unsigned)(nth >> 5);
  if (tid == 0) {
    wl.q->tp = ((unsigned long long)P.ntiles << 32) | (unsigned long long)P.ntiles;
    wl.q->head = warps;  // every warp starts with the ticket of its number
  }
  if (!grid_barrier(ctl, P.wait_ns)) return;

  // phase 1: visits until no tile is queued or running
  // runaway guard on the tickets (visits plus idle pops), also below the wrap of the 32-bit ring
  // positions
  const long long max_tickets = std::min<long long>((long long)P.ntiles * P.max_rounds, (1ll << 31) - 2ll * P.ntiles);
  for (unsigned ticket = (unsigned)(tid >> 5);;) {
    unsigned popped = 0u;
    if (lane == 0) popped = wl_pop(wl, ctl, ticket, max_tickets);
    popped = __shfl_sync(0xffffffffu, popped, 0);
    if (popped == 0u) break;
    const int t = (int)((popped & ~kSettled<T>) - 1u);
    const bool settled = (popped & kSettled<T>) != 0u;
    int tl = 0;
    const RImg &im = image_of(P, t, tl, begin);
    int f;
    if constexpr (sizeof(T) <= 2) {
      f = process_tile_packed<T, SUP, CONN8>(im, P, tl, settled, *reinterpret_cast<PackedTile<T> *>(s_raw[warp]));
    } else {
      T *s_m = reinterpret_cast<T *>(s_raw[warp]);
      f = process_tile_reg<T, SUP, CONN8>(im, P, tl, s_m, s_m + 32 * kRP);
    }
    __threadfence();  // this tile's pixels, before any neighbour is queued
    __syncwarp();
    wl_finish<T, CONN8>(wl, ctl, im, t, tl, f);
    if (lane == 0) ticket = atomicAdd(&wl.q->head, 1u);
    __syncwarp();
  }
  if (!grid_barrier(ctl, P.wait_ns)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const long long visits = (long long)tp_tail(*((volatile unsigned long long *)&wl.q->tp));  // every pushed tile was visited
    g_recon_visits = visits;
    g_recon_rounds = (int)((visits + P.ntiles - 1) / P.ntiles);
    ctl->rounds = g_recon_rounds;
  }
  if (P.epi == EPI_NONE) return;
  recon_epilogue<T, SUP>(P, begin);
}

// ------------------------------------------------------------------ resident tiles
// Images of 1- or 2-byte pixels whose tiles all fit on the GPU at once (32 warps per SM: 4864 tiles of 32 x 32,
// 5 Mpixel) keep every tile in one warp from start to end: the values in registers, the mask in shared memory.
// No tile is staged again, nothing is queued: a visit reads its neighbours' border pixels, sweeps, publishes its
// own changed borders (32 contiguous pixels each) and marks the neighbours beside them; a warp with nothing to do
// polls its tile's state word.  A value crosses a tile in the time of one border load, the sweeps, one fence and
// one atomic, where the worklist also pops, stages, writes back and queues.
//
// State of a tile: RS_IDLE, RS_RUNNING (its warp is visiting), RS_DIRTY (a border beside it changed since the
// visit read its halo).  `pending` counts the tiles that are not idle.  A warp adds the neighbours it may wake
// before it marks them and takes off the ones that were awake already, and itself when it falls idle,
// afterwards: `pending` never reads zero early, and the warp that brings it to zero ends the kernel.
// Bound: the chain of dependent visits (border load, two sweep sets, fence, atomic: about 4 us a hop).  Kernel
// alone, by ncu: binary h-maxima 2048^2 u8 110 -> 71 us, one half of the leveling of 1537 x 1805 u16 250 -> 78 us;
// calls 131 -> 93 and 555 -> 192 us.  One to 64 sweep sets per visit: 93-101 us, two kept.
enum : unsigned { RS_IDLE = 0, RS_RUNNING = 1, RS_DIRTY = 2 };
static constexpr int kResidentWarps = 32;

// `pending` (low half of `work`) shares its word with a count of the visits that woke a tile or fell idle (high
// half), so that a waiting tile can tell a long propagation elsewhere from one that stands still.
struct ResCtl {  // in the work area, cleared before the launch
  unsigned long long work;
  int pad0[30];
  int done, pad1[31];
};
static_assert(sizeof(ResCtl) == 256, "ResCtl layout");
__device__ __forceinline__ unsigned res_progress(const ResCtl *res) {
  return (unsigned)(*((volatile const unsigned long long *)&res->work) >> 32);
}

template <typename T> struct ResTiles {
  ResCtl *ctl;
  unsigned *state;  // ntiles
  T *border;        // ntiles x 4 x 32 pixels: rows top and bottom, columns left and right
};

__device__ __forceinline__ unsigned exch_acquire(unsigned *p, unsigned v) {
  unsigned old;
  asm volatile("atom.acquire.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

// End of a resident visit, by the whole warp: marks neighbour nb of every lane with `wake` (the changed borders are
// stored), lets tile t fall idle if it has converged and nothing beside it changed, and waits until there is
// work.  Returns 0: visit again (the state is RS_RUNNING), 1: all tiles are idle, 2: an error was recorded.
// The wait gives up when its limit passes with no progress anywhere; a tile that a front reaches late may have to
// wait longer than that (the limit alone, counted from falling idle, refused paths of more than 4 s).
__device__ __forceinline__ int resident_rest(ResCtl *res, RCtl *ctl, unsigned *state, int t, int nb, bool wake,
                                             bool converged, unsigned long long wait_ns) {
  const int lane = threadIdx.x & 31;
  const int n_wake = __popc(__ballot_sync(0xffffffffu, wake));
  int off = 0;  // tiles to take off `pending` again
  if (n_wake) {
    if (lane == 0) atomicAdd(&res->work, (1ull << 32) + (unsigned)n_wake);
    __threadfence();  // the borders and the count before the marks
    __syncwarp();
    const bool awake = wake && atomicExch(state + nb, RS_DIRTY) != RS_IDLE;
    off = __popc(__ballot_sync(0xffffffffu, awake));
  }
  // ---- back to idle, or on with another visit
  unsigned again = 1;
  if (lane == 0) {
    if (converged && atomicCAS(state + t, RS_RUNNING, RS_IDLE) == RS_RUNNING) {
      again = 0;
      ++off;
    }
    // less `off` in the low half carries one into the high half
    if (off && (unsigned)atomicAdd(&res->work, (1ull << 32) - (unsigned)off) == (unsigned)off) *((volatile int *)&res->done) = 1;
  }
  again = __shfl_sync(0xffffffffu, again, 0);
  int stop = 0;
  if (lane == 0) {
    if (!again) {
      unsigned long long t0 = global_ns();
      unsigned seen = ~0u;
      for (unsigned polls = 0;; ++polls) {
        if (*((volatile unsigned *)(state + t)) == RS_DIRTY) break;
        if (polls % 8 == 7) {
          if (*((volatile int *)&res->done)) { stop = 1; break; }
          if (*((volatile int *)&ctl->status)) { stop = 2; break; }
          if (global_ns() - t0 > wait_ns) {
            const unsigned now = res_progress(res);  // looked at once a limit: idle polls leave the counter's line alone
            if (now == seen) {
              set_status(ctl, PG_ERR_NOT_CONVERGED);
              stop = 2;
              break;
            }
            seen = now;
            t0 = global_ns();
          }
        }
        __nanosleep(polls < 16 ? 20 : 100);
      }
    } else if (*((volatile int *)&ctl->status)) {
      stop = 2;
    }
    if (!stop) exch_acquire(state + t, RS_RUNNING);  // before the halo is read: what changes later marks again
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, stop, 0);
}

template <typename T, bool SUP, bool CONN8>
__global__ void __launch_bounds__(kResidentWarps * 32, 1) k_reconstruct_resident(const __grid_constant__ RParams<T> P,
                                                                                const ResTiles<T> rt) {
  static_assert(sizeof(T) <= 2, "packed tiles");
  using OT = Op<T, SUP>;
  constexpr int TP = PackedCore<T>::TP;
  constexpr int LR = TileRows<T, true>::LR, RI = TileRows<T, true>::RI, PASSES = TileRows<T, true>::PASSES;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  PackedCore<T> &s = reinterpret_cast<PackedCore<T> *>(s_dyn)[warp];
  RCtl *ctl = P.ctl;
  const T NEU = OT::neutral();
  // tiles are dealt over the SMs, so that a front of active tiles is spread over all of them
  const int t = (int)(blockIdx.x + gridDim.x * (unsigned)warp);
  const bool have = t < P.ntiles;
  int tl = 0;
  const RImg &im = image_of(P, have ? t : 0, tl);
  const int tx = tl % im.tiles_x, ty = tl / im.tiles_x;
  const int64_t y0 = (int64_t)ty * 32, x0 = (int64_t)tx * 32;
  const int rows = (int)min((int64_t)32, im.H - y0), cols = (int)min((int64_t)32, im.W - x0);
  T *mine = rt.border + (size_t)t * 128;
  uint32_t V[16], pub_lr = 0;

  if (have) {
    // the reference (or mask), then the marker, through s.val into registers: effective mask and initial value
    auto stage = [&](const void *img) {
      const TileRows<T, false> r(img, im, y0, x0, rows);
#pragma unroll
      for (int k0 = 0; k0 < PASSES; k0 += 4) {
        uint32_t w[4][3];
#pragma unroll
        for (int k = 0; k < 4; ++k) r.load(k0 + k, (k0 + k) * RI + lane / LR < rows, im, w[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint2 v = r.pixels(k0 + k, w[k]);
          uint32_t *d = reinterpret_cast<uint32_t *>(s.val + ((k0 + k) * RI + lane / LR) * TP) + 2 * (lane % LR);
          d[0] = v.x;
          d[1] = v.y;
        }
      }
      __syncwarp();
    };
    uint32_t M[16];
    stage(im.mask);
#pragma unroll
    for (int p = 0; p < 16; ++p) M[p] = pk2(s.val[p * TP + lane], s.val[(31 - p) * TP + lane]);
    if (P.init != INIT_SAT_CONST) {
      __syncwarp();
      stage(im.marker);
    }
    auto pixel = [&](int r, uint32_t ref, T &m, T &v) {  // pixel (r, lane)
      m = v = NEU;
      if (r < rows && lane < cols) combine_init<T, SUP>(P, (T)ref, s.val[r * TP + lane], m, v);
    };
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      T m0, m1, v0, v1;
      pixel(p, M[p], m0, v0);
      pixel(31 - p, M[p] >> 16, m1, v1);
      M[p] = pk2(m0, m1);
      V[p] = pk2(v0, v1);
    }
    // both by rows, for the column pairs
    auto by_rows = [&](const uint32_t (&x)[16]) {
      __syncwarp();
#pragma unroll
      for (int p = 0; p < 16; ++p) {
        s.val[p * TP + lane] = (T)x[p];
        s.val[(31 - p) * TP + lane] = (T)(x[p] >> 16);
      }
      __syncwarp();
    };
    by_rows(M);
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      s.ma[p * kRP + lane] = M[p];
      s.mb[p * kRP + lane] = pk2(s.val[lane * TP + p], s.val[lane * TP + 31 - p]);
    }
    by_rows(V);
    pub_lr = pk2(s.val[lane * TP], s.val[lane * TP + 31]);
    st_cg(mine + lane, (T)V[0]);
    st_cg(mine + 32 + lane, (T)(V[0] >> 16));
    st_cg(mine + 64 + lane, (T)pub_lr);
    st_cg(mine + 96 + lane, (T)(pub_lr >> 16));
    if (lane == 0) rt.state[t] = RS_RUNNING;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    rt.ctl->work = (unsigned)P.ntiles;
    g_recon_rounds = 0;
  }
  if (!grid_barrier(ctl, P.wait_ns)) return;
  if (!have) return;

  // lane d < 8 looks after the neighbour in direction d = N S W E NW NE SW SE (B_x = 1 << d)
  int nb = -1;
  if (lane < (CONN8 ? 8 : 4)) {
    const int dx = lane < 2 ? 0 : ((lane & 1) ? 1 : -1);
    const int dy = lane < 2 ? (lane ? 1 : -1) : lane < 4 ? 0 : (lane < 6 ? -1 : 1);
    const int nx = tx + dx, ny = ty + dy;
    if (nx >= 0 && ny >= 0 && nx < im.tiles_x && ny < im.tiles_y) nb = t + dy * im.tiles_x + dx;
  }
  const bool up = ty > 0, down = ty + 1 < im.tiles_y, west = tx > 0, east = tx + 1 < im.tiles_x;
  int visits = 0;
  bool settled = false;  // at the local fixpoint of the last halo
  for (;;) {
    // ---- visit: the halo from the neighbours' borders
    if (++visits > P.max_rounds) {
      if (lane == 0) set_status(ctl, PG_ERR_NOT_CONVERGED);
      return;
    }
    T h_top = NEU, h_bot = NEU, h_l = NEU, h_r = NEU, c_top = NEU, c_bot = NEU;
    {
      const T *b = rt.border + (size_t)t * 128 + lane;
      const int down_row = im.tiles_x * 128;
      if (up) h_top = ld_cg(b - down_row + 32);
      if (down) h_bot = ld_cg(b + down_row);
      if (west) h_l = ld_cg(b - 128 + 96);
      if (east) h_r = ld_cg(b + 128 + 64);
      if (CONN8 && ((lane == 0 && west) || (lane == 31 && east))) {
        const T *c = lane == 0 ? b - 128 + 31 : b + 128 - 31;  // the last / first pixel of that neighbour's rows
        if (up) c_top = ld_cg(c - down_row + 32);
        if (down) c_bot = ld_cg(c + down_row);
      }
    }
    if (CONN8) fold_halo<T, SUP>(h_top, h_bot, h_l, h_r, c_top, c_bot);
    const uint32_t init_tb = V[0], tb = pk2(h_top, h_bot), lr = pk2(h_l, h_r);
    uint32_t end_lr = pub_lr;
    bool changed = false;
    // A tile at its local fixpoint moves only if its new halo moves a border pixel: most wakes end here.
    if (!settled || __any_sync(0xffffffffu, pulled<SUP>(V[0], tb, s.ma[lane]) != V[0] ||
                                                pulled<SUP>(pub_lr, lr, s.mb[lane]) != pub_lr))
      settled = packed_sweeps<T, SUP, CONN8>(V, s, tb, lr, P.max_sweeps, end_lr, changed);

    // ---- the borders that changed, and the neighbours beside them
    const uint32_t d_tb = V[0] ^ init_tb, d_lr = end_lr ^ pub_lr;
    const unsigned bN = __ballot_sync(0xffffffffu, (d_tb & 0xffffu) != 0u), bS = __ballot_sync(0xffffffffu, (d_tb >> 16) != 0u);
    const unsigned bW = __ballot_sync(0xffffffffu, (d_lr & 0xffffu) != 0u), bE = __ballot_sync(0xffffffffu, (d_lr >> 16) != 0u);
    pub_lr = end_lr;
    if (bN) st_cg(mine + lane, (T)V[0]);
    if (bS) st_cg(mine + 32 + lane, (T)(V[0] >> 16));
    if (bW) st_cg(mine + 64 + lane, (T)pub_lr);
    if (bE) st_cg(mine + 96 + lane, (T)(pub_lr >> 16));
    bool wake = false;
    if (nb >= 0) {
      const unsigned of = lane == 0 ? bN : lane == 1 ? bS : lane == 2 ? bW : lane == 3 ? bE
                          : lane == 4 ? (bN & 1u) : lane == 5 ? (bN >> 31) : lane == 6 ? (bS & 1u) : (bS >> 31);
      wake = of != 0u;
    }
    const int stop = resident_rest(rt.ctl, ctl, rt.state, t, nb, wake, settled, P.wait_ns);
    if (stop == 2) return;
    if (stop == 1) break;
  }
  if (lane == 0) atomicMax(&g_recon_rounds, visits);

  // ---- result: the values by rows in shared memory, then the epilogue's function of them and the reference
  __syncwarp();
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    s.val[p * TP + lane] = (T)V[p];
    s.val[(31 - p) * TP + lane] = (T)(V[p] >> 16);
  }
  __syncwarp();
  if (P.epi == EPI_BINARY_SUP) {  // the mask here is the reference itself
    uint8_t *o = static_cast<uint8_t *>(im.out) + y0 * im.W + x0 + lane;
    if (lane < cols)
#pragma unroll 8
      for (int r = 0; r < rows; ++r) {
        const T ref = (T)(r < 16 ? s.ma[r * kRP + lane] : s.ma[(31 - r) * kRP + lane] >> 16);
        o[r * im.W] = epi_binary<T, SUP>(ref, s.val[r * TP + lane]);
      }
    return;
  }
  const TileRows<T, true> ro(im.out, im, y0, x0, rows);
  if (P.epi == EPI_CLIP_REF) {
    const TileRows<T, false> rr(im.mask, im, y0, x0, rows);
#pragma unroll
    for (int k0 = 0; k0 < PASSES; k0 += 4) {
      uint32_t w[4][3];
#pragma unroll
      for (int k = 0; k < 4; ++k) rr.load(k0 + k, (k0 + k) * RI + lane / LR < rows, im, w[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint2 v = rr.pixels(k0 + k, w[k]);
        uint32_t *d = reinterpret_cast<uint32_t *>(s.val + ((k0 + k) * RI + lane / LR) * TP) + 2 * (lane % LR);
        d[0] = wop<T, !SUP>(d[0], v.x);
        d[1] = wop<T, !SUP>(d[1], v.y);
      }
    }
    __syncwarp();
  }
  if (ro.pairs && cols == 32) {
#pragma unroll
    for (int k = 0; k < PASSES; ++k) {
      const int row = k * RI + lane / LR;
      const uint32_t *d = reinterpret_cast<const uint32_t *>(s.val + row * TP) + 2 * (lane % LR);
      if (row < rows) *reinterpret_cast<uint2 *>(ro.a + k * ro.pitch) = make_uint2(d[0], d[1]);
    }
  } else if (lane < cols) {
    T *o = static_cast<T *>(im.out) + y0 * im.W + x0 + lane;
#pragma unroll 8
    for (int r = 0; r < rows; ++r) o[r * im.W] = s.val[r * TP + lane];
  }
}

// ------------------------------------------------------------------ host side
// Scratch work area of one launch: control block (256 B) | worklist counters (512 B) | per-tile
// words: the double-buffered flags of the round kernel, or the tile states and the ring of the
// worklist.  The work area is cleared before the launch.
static constexpr size_t kWorkHead = 256 + sizeof(RQueue);

// Rounds (round kernel) or visits per tile (worklist kernel) before a launch gives up: far more than
// any input needs (a tile is revisited only when a neighbour changed its border), unless a test set
// a cap through pg_debug_set_limits.
static int max_rounds_for(int64_t ntiles) {
  const int cap = g_dbg_max_rounds.load();
  if (cap > 0) return cap;
  return (int)std::min<int64_t>(INT32_MAX / 2, 1024 + 64 * ntiles);
}
static unsigned ring_cap(int64_t ntiles) { return (unsigned)(2 * ntiles + 4096); }
static size_t ring_offset(int64_t ntiles) { return ((4 * (size_t)ntiles + 255) / 256) * 256; }
static size_t work_bytes(int64_t ntiles) {
  return kWorkHead + ring_offset(ntiles) + ((8 * (size_t)ring_cap(ntiles) + 255) / 256) * 256;
}

// Launches the reconstruction kernel for tile side RT: the worklist kernel on register tiles
// for 32-pixel tiles of pixels up to 4 bytes, the round kernel on shared-memory tiles otherwise.
// P's images, tiles and modes are set by the caller; `work` is a cleared work area.
template <typename T, bool SUP, bool CONN8, int RT>
static pg_status launch_recon(RParams<T> &P, char *work, cudaStream_t s, int *grid_out) {
  constexpr bool REG = RT == 32 && sizeof(T) <= 4;
  constexpr int THREADS = REG ? kRegWarps * 32 : RT;
  constexpr int TILES_PER_CTA = REG ? kRegWarps : 1;
  P.ctl = reinterpret_cast<RCtl *>(work);
  P.flags = reinterpret_cast<unsigned *>(work + kWorkHead);
  P.max_rounds = max_rounds_for(P.ntiles);
  P.wait_ns = g_dbg_wait_ns.load();
  WorkList<T> wl{};
  wl.wait_ns = P.wait_ns;
  wl.q = reinterpret_cast<RQueue *>(work + 256);
  wl.state = P.flags;
  wl.ring = reinterpret_cast<unsigned long long *>(work + kWorkHead + ring_offset(P.ntiles));
  wl.cap = ring_cap(P.ntiles);
  void *kern = nullptr;
  if constexpr (REG) kern = reinterpret_cast<void *>(k_reconstruct_wl<T, SUP, CONN8>);
  else kern = reinterpret_cast<void *>(k_reconstruct<T, SUP, CONN8, RT>);
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  static std::mutex mu;
  static std::vector<int> cached;  // blocks per SM, per device
  int per_sm = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    if ((size_t)dev >= cached.size()) cached.resize((size_t)dev + 1, 0);
    if (cached[(size_t)dev] == 0)
      PG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cached[(size_t)dev], kern, THREADS, 0), "occupancy");
    per_sm = cached[(size_t)dev];
  }
  if (per_sm < 1) return fail(PG_ERR_CUDA, "reconstruction kernel cannot be resident");
  int grid = per_sm * num_sms();
  if (grid > ceil_div(P.ntiles, TILES_PER_CTA)) grid = (int)ceil_div(P.ntiles, TILES_PER_CTA);
  if (grid_out) *grid_out = grid;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if constexpr (REG) PG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_reconstruct_wl<T, SUP, CONN8>, P, wl), "cooperative reconstruction launch");
  else PG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_reconstruct<T, SUP, CONN8, RT>, P), "cooperative reconstruction launch");
  return PG_OK;
}

// Whether the resident kernel holds this many tiles, and its launch.  `work` is a cleared work area of
// resident_bytes().
static size_t resident_bytes(int64_t ntiles, size_t elem_bytes) {
  return 256 + sizeof(ResCtl) + (4 * (size_t)ntiles + 255) / 256 * 256 + 128 * (size_t)ntiles * elem_bytes;
}
static bool resident_fits(int64_t ntiles) { return ntiles <= (int64_t)kResidentWarps * num_sms(); }

template <typename T, bool SUP, bool CONN8>
static pg_status launch_resident(RParams<T> &P, char *work, cudaStream_t s) {
  static_assert(sizeof(PackedCore<T>) * kResidentWarps <= 227 * 1024, "a CTA's tiles fit in shared memory");
  P.ctl = reinterpret_cast<RCtl *>(work);
  P.max_rounds = max_rounds_for(P.ntiles);
  P.wait_ns = g_dbg_wait_ns.load();
  ResTiles<T> rt{};
  rt.ctl = reinterpret_cast<ResCtl *>(work + 256);
  rt.state = reinterpret_cast<unsigned *>(work + 256 + sizeof(ResCtl));
  rt.border = reinterpret_cast<T *>(work + 256 + sizeof(ResCtl) + (4 * (size_t)P.ntiles + 255) / 256 * 256);
  const int grid = std::min(num_sms(), P.ntiles);
  const int warps = (int)ceil_div(P.ntiles, grid);
  const size_t smem = sizeof(PackedCore<T>) * (size_t)warps;
  static std::atomic<uint64_t> attr_devices{0};  // the opt-in shared-memory size, once per device
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  const uint64_t bit = 1ull << (dev & 63);
  if (!(attr_devices.load() & bit)) {
    PG_CUDA_TRY(cudaFuncSetAttribute(k_reconstruct_resident<T, SUP, CONN8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(sizeof(PackedCore<T>) * kResidentWarps)),
                "resident reconstruction smem attribute");
    attr_devices.fetch_or(bit);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)warps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_reconstruct_resident<T, SUP, CONN8>, P, rt), "cooperative reconstruction launch");
  return PG_OK;
}

template <typename T, bool SUP, bool CONN8>
static pg_status run_t(std::vector<RImg> &imgs, const ReconRequest &rq, bool binary, cudaStream_t s) {
  // register tiles (32x32, a warp each) up to 4-byte pixels, shared-memory tiles for 8-byte ones
  constexpr int RT = sizeof(T) <= 4 ? 32 : tile_side<T>();
  int ntiles = 0;
  size_t rec_bytes = 0;
  for (auto &im : imgs) {
    im.tiles_x = (int)ceil_div(im.W, RT);
    im.tiles_y = (int)ceil_div(im.H, RT);
    im.tile_begin = ntiles;
    ntiles += im.tiles_x * im.tiles_y;
    if (binary) rec_bytes += (sizeof(T) * (size_t)(im.H * im.W) + 15) / 16 * 16;  // 16-byte aligned slots
  }
  if (ntiles == 0) return PG_OK;
  const int nimg = (int)imgs.size();
  if constexpr (sizeof(T) <= 2) {
    if (nimg == 1 && resident_fits(ntiles)) {
      Scratch work;
      PG_TRY(work.alloc(resident_bytes(ntiles, sizeof(T)), s));
      // control words and states; the borders are written before they are read
      PG_CUDA_TRY(cudaMemsetAsync(work.ptr, 0, 256 + sizeof(ResCtl) + 4 * (size_t)ntiles, s), "clear reconstruction work area");
      RParams<T> P{};
      P.single = imgs[0];
      P.nimg = 1;
      P.ntiles = ntiles;
      P.init = rq.init;
      P.mask_mode = rq.mask_mode;
      P.epi = rq.epi;
      P.h = scalar_as<T>(rq.h);
      P.max_sweeps = kVisitSweeps;
      return launch_resident<T, SUP, CONN8>(P, work.as<char>(), s);
    }
  }
  // scratch: work area | image table | reconstruction buffers (binary mode)
  const size_t off_tab = work_bytes(ntiles);
  const size_t off_rec = off_tab + ((sizeof(RImg) * (size_t)(nimg > 1 ? nimg : 0) + 255) / 256) * 256;
  const size_t total = off_rec + rec_bytes + 256;
  Scratch scr;
  PG_TRY(scr.alloc(total, s));
  char *base = scr.as<char>();
  if (binary) {
    size_t off = off_rec;
    for (auto &im : imgs) {
      im.rec = base + off;
      off += sizeof(T) * (size_t)(im.H * im.W);
      off = (off + 15) / 16 * 16;
    }
  }
  PG_CUDA_TRY(cudaMemsetAsync(base, 0, off_tab, s), "clear reconstruction work area");
  std::vector<RImg> table;
  if (nimg > 1) {
    table = imgs;
    PG_CUDA_TRY(cudaMemcpyAsync(base + off_tab, table.data(), sizeof(RImg) * (size_t)nimg, cudaMemcpyHostToDevice, s),
                "upload image table");
  }
  RParams<T> P{};
  P.single = imgs[0];
  P.imgs = reinterpret_cast<const RImg *>(base + off_tab);
  P.nimg = nimg;
  P.ntiles = ntiles;
  P.init = rq.init;
  P.mask_mode = rq.mask_mode;
  P.epi = rq.epi;
  P.h = scalar_as<T>(rq.h);
  // register tiles yield after kVisitSweeps sweep sets and are revisited: measured as fast or faster
  // than sweeping each visit to its local fixpoint (h-maxima 4096^2 -2 %, a long propagation -6 %)
  if constexpr (RT == 32 && sizeof(T) <= 4) P.max_sweeps = kVisitSweeps;
  return launch_recon<T, SUP, CONN8, RT>(P, base, s, nullptr);
}

template <typename T>
static pg_status run_dispatch(std::vector<RImg> &imgs, const ReconRequest &rq, cudaStream_t s) {
  const bool binary = rq.epi == EPI_BINARY_SUP;
  if (rq.dilate) return rq.conn8 ? run_t<T, true, true>(imgs, rq, binary, s) : run_t<T, true, false>(imgs, rq, binary, s);
  return rq.conn8 ? run_t<T, false, true>(imgs, rq, binary, s) : run_t<T, false, false>(imgs, rq, binary, s);
}

pg_status launch_reconstruction(const pg_image *markers, const pg_image *masks, const pg_image *outs, int n_images,
                                const ReconRequest &rq, cudaStream_t s) {
  if (n_images < 1) return PG_OK;
  if (masks[0].rank == 3) {  // volumes: the iterated geodesic step of recon3d.cu, one volume at a time
    for (int i = 0; i < n_images; ++i)
      PG_TRY(launch_reconstruction3d(markers ? &markers[i] : nullptr, masks[i], outs[i], rq, s));
    return PG_OK;
  }
  std::vector<RImg> imgs((size_t)n_images);
  for (int i = 0; i < n_images; ++i) {
    const Dims d = dims_of(masks[i]);
    RImg &im = imgs[(size_t)i];
    im = RImg{};
    im.marker = markers ? markers[i].data : nullptr;
    im.mask = masks[i].data;
    im.rec = outs[i].data;
    im.out = outs[i].data;
    im.H = d.nz * d.ny;  // rank 1: one row
    im.W = d.nx;
  }
  PG_DISPATCH_PTYPE(masks[0].ptype, T, { return run_dispatch<T>(imgs, rq, s); });
  return PG_OK;
}

// ------------------------------------------------------------------ batch plans + autotuner
// A plan keeps a ragged batch's image tables, worklist and reconstruction buffers on the device
// so that each run is one memset and one cooperative launch (both capturable in a CUDA graph).
// The autotuner times the candidate configurations -- tile side (32: register tiles, 64: shared-
// memory tiles) x sweep sets per tile visit before the tile yields to the next global round
// (4, 16, unbounded) -- on the plan's own batch and keeps the fastest; the choice is cached per
// (pixel type, connectivity, batch size class).
struct PlanCfg {
  int rt = 64;
  int sweeps = kMaxSweeps;
};

struct PlanTable {  // one tile decomposition of the batch
  int ntiles = 0;
  RImg *d_imgs = nullptr;  // device table
  std::vector<RImg> imgs;  // host copy
};

}  // namespace pg

struct pg_batch_plan {
  int device = 0;
  int ptype = 0;
  bool conn8 = true;
  pg_scalar h{};
  void *scratch = nullptr;  // control block | flags (sized for the finest tiling) | recon buffers
  size_t clear_bytes = 0;
  pg::PlanTable t64, t32;
  pg::PlanCfg cfg;
  int grid = 0;
};

namespace pg {

template <int RT> static PlanTable &plan_table(pg_batch_plan &p) { return RT == 64 ? p.t64 : p.t32; }

template <typename T, bool CONN8, int RT>
static pg_status plan_launch_t(pg_batch_plan &p, int sweeps, cudaStream_t s, int *grid_out) {
  PlanTable &tb = plan_table<RT>(p);
  RParams<T> P{};
  P.single = tb.imgs[0];
  P.imgs = tb.d_imgs;
  P.nimg = (int)tb.imgs.size();
  P.ntiles = tb.ntiles;
  P.max_sweeps = sweeps;
  P.init = INIT_SAT_CONST;
  P.mask_mode = MASK_PLAIN;
  P.epi = EPI_BINARY_SUP;
  P.h = scalar_as<T>(p.h);
  PG_CUDA_TRY(cudaMemsetAsync(p.scratch, 0, p.clear_bytes, s), "clear batch work area");
  return launch_recon<T, true, CONN8, RT>(P, static_cast<char *>(p.scratch), s, grid_out);
}

template <typename T>
static pg_status plan_launch(pg_batch_plan &p, const PlanCfg &c, cudaStream_t s, int *grid_out) {
  if constexpr (sizeof(T) == 8) {
    return p.conn8 ? plan_launch_t<T, true, 32>(p, c.sweeps, s, grid_out) : plan_launch_t<T, false, 32>(p, c.sweeps, s, grid_out);
  } else {
    if (c.rt == 64)
      return p.conn8 ? plan_launch_t<T, true, 64>(p, c.sweeps, s, grid_out) : plan_launch_t<T, false, 64>(p, c.sweeps, s, grid_out);
    return p.conn8 ? plan_launch_t<T, true, 32>(p, c.sweeps, s, grid_out) : plan_launch_t<T, false, 32>(p, c.sweeps, s, grid_out);
  }
}

static pg_status plan_run(pg_batch_plan &p, const PlanCfg &c, cudaStream_t s, int *grid_out) {
  PG_DISPATCH_PTYPE(p.ptype, T, { return plan_launch<T>(p, c, s, grid_out); });
  return PG_OK;
}

static void plan_tables(pg_batch_plan &p, const std::vector<RImg> &base, int rt, PlanTable &tb) {
  tb.imgs = base;
  int ntiles = 0;
  for (auto &im : tb.imgs) {
    im.tiles_x = (int)ceil_div(im.W, rt);
    im.tiles_y = (int)ceil_div(im.H, rt);
    im.tile_begin = ntiles;
    ntiles += im.tiles_x * im.tiles_y;
  }
  tb.ntiles = ntiles;
}

struct TuneKey {
  int ptype, conn8, size_class, count_class;
  bool operator<(const TuneKey &o) const {
    return std::tie(ptype, conn8, size_class, count_class) < std::tie(o.ptype, o.conn8, o.size_class, o.count_class);
  }
};

pg_status create_batch_plan(const pg_image *ins, const pg_image *outs, int n, const pg_scalar &h, bool conn8, bool autotune,
                            cudaStream_t s, pg_batch_plan **out_plan) {
  auto plan = std::make_unique<pg_batch_plan>();
  PG_CUDA_TRY(cudaGetDevice(&plan->device), "cudaGetDevice");
  plan->ptype = ins[0].ptype;
  plan->conn8 = conn8;
  plan->h = h;
  const size_t es = (size_t)elem_size(plan->ptype);
  std::vector<RImg> base((size_t)n);
  int64_t pixels = 0;
  for (int i = 0; i < n; ++i) {
    const Dims d = dims_of(ins[i]);
    RImg &im = base[(size_t)i];
    im = RImg{};
    im.mask = ins[i].data;
    im.out = outs[i].data;
    im.H = d.nz * d.ny;
    im.W = d.nx;
    pixels += im.H * im.W;
  }
  plan_tables(*plan, base, 64, plan->t64);
  plan_tables(*plan, base, 32, plan->t32);
  const int max_tiles = std::max(plan->t64.ntiles, plan->t32.ntiles);
  const size_t off_tab64 = work_bytes(max_tiles);
  const size_t tab_bytes = ((sizeof(RImg) * (size_t)n + 255) / 256) * 256;
  const size_t off_tab32 = off_tab64 + tab_bytes;
  size_t off_rec = off_tab32 + tab_bytes;
  size_t rec_bytes = 0;
  for (auto &im : base) rec_bytes += (es * (size_t)(im.H * im.W) + 255) / 256 * 256;
  PG_CUDA_TRY(cudaMalloc(&plan->scratch, off_rec + rec_bytes + 256), "batch plan allocation");
  plan->clear_bytes = off_tab64;
  // reconstruction buffers, then device copies of both tile tables
  char *b = static_cast<char *>(plan->scratch);
  size_t off = off_rec;
  for (size_t i = 0; i < base.size(); ++i) {
    plan->t64.imgs[i].rec = b + off;
    plan->t32.imgs[i].rec = b + off;
    off += (es * (size_t)(base[i].H * base[i].W) + 255) / 256 * 256;
  }
  plan->t64.d_imgs = reinterpret_cast<RImg *>(b + off_tab64);
  plan->t32.d_imgs = reinterpret_cast<RImg *>(b + off_tab32);
  cudaError_t e = cudaMemcpy(plan->t64.d_imgs, plan->t64.imgs.data(), sizeof(RImg) * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(plan->t32.d_imgs, plan->t32.imgs.data(), sizeof(RImg) * (size_t)n, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(plan->scratch);
    return cuda_status(e, "upload batch tile tables");
  }

  static std::mutex mu;
  static std::map<TuneKey, PlanCfg> cache;
  const TuneKey key{plan->ptype, conn8 ? 1 : 0, (int)std::log2((double)std::max<int64_t>(pixels, 1)),
                    (int)std::log2((double)std::max(n, 1))};
  bool cached = false;
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) { plan->cfg = it->second; cached = true; }
  }
  if (autotune && !cached) {
    std::vector<PlanCfg> cands;
    for (int rt : {64, 32}) {
      if (es == 8 && rt == 64) continue;
      for (int sw : {kVisitSweeps, 4, 16, kMaxSweeps}) cands.push_back(PlanCfg{rt, sw});
    }
    cudaEvent_t a, z;
    PG_CUDA_TRY(cudaEventCreate(&a), "event");
    PG_CUDA_TRY(cudaEventCreate(&z), "event");
    float best = 1e30f;
    for (const PlanCfg &c : cands) {
      pg_status st = plan_run(*plan, c, s, nullptr);  // warm
      if (st != PG_OK) { cudaEventDestroy(a); cudaEventDestroy(z); cudaFree(plan->scratch); return st; }
      float tot = 0.f;
      for (int r = 0; r < 2; ++r) {
        cudaEventRecord(a, s);
        plan_run(*plan, c, s, nullptr);
        cudaEventRecord(z, s);
        cudaEventSynchronize(z);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, a, z);
        tot += ms;
      }
      if (tot < best) { best = tot; plan->cfg = c; }
    }
    cudaEventDestroy(a);
    cudaEventDestroy(z);
    std::lock_guard<std::mutex> lk(mu);
    cache[key] = plan->cfg;
  } else if (!cached) {
    plan->cfg = PlanCfg{32, kMaxSweeps};
  }
  *out_plan = plan.release();
  return PG_OK;
}

pg_status run_batch_plan(pg_batch_plan *p, cudaStream_t s) {
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev != p->device) return fail(PG_ERR_INVALID_ARGUMENT, "batch plan used on another device");
  return plan_run(*p, p->cfg, s, &p->grid);
}

void destroy_batch_plan(pg_batch_plan *p) {
  if (!p) return;
  if (p->scratch) cudaFree(p->scratch);
  delete p;
}

cudaError_t recon_status_word(void **p) { return cudaGetSymbolAddress(p, g_recon_status); }

// ------------------------------------------------------------------ allocation-free variant
// For callers that must not touch the device allocator (see pg_reconstruction_noalloc in
// include/poutre_gb300.h).  Its only scratch -- the control block and the tile worklist --
// lives in this file-scope array, which every GPU that loads the library holds until exit.
static constexpr size_t kNoAllocScratchBytes = PG_NOALLOC_SCRATCH_BYTES;
static constexpr size_t kNoAllocFlagsOffset = 256;  // RCtl fits below
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

static_assert(sizeof(RCtl) <= kNoAllocFlagsOffset, "control block must fit below the flags");

// Tiles of an H x W image in the no-alloc kernel (tile_side<T>() squares: 64, or 32 for 8-byte
// pixels) and the most the fixed scratch holds (two flag words per tile above the control block).
// The one place both numbers are computed: the entry point's shape check and the launch use it.
static void noalloc_tiles(int elem_bytes, int64_t H, int64_t W, int64_t &ntiles, int64_t &max_tiles) {
  const int64_t rt = tile_side_for(elem_bytes);
  ntiles = ceil_div(H, rt) * ceil_div(W, rt);
  max_tiles = (int64_t)((kNoAllocScratchBytes - kNoAllocFlagsOffset) / (2 * sizeof(unsigned)));
}

// Device address of g_noalloc_scratch, looked up once per device with that device current.
// In host code the symbol name is only a host-side stand-in, so the kernel is given this
// address instead.  The address is kept for the life of the process: after cudaDeviceReset
// (which destroys the context holding the array) this entry point must not be called again.
static pg_status noalloc_scratch(void **out) {
  static std::mutex mu;
  static std::vector<void *> addr;  // indexed by device ordinal
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lk(mu);
  if ((size_t)dev >= addr.size()) addr.resize((size_t)dev + 1, nullptr);
  if (!addr[(size_t)dev]) {
    void *p = nullptr;
    PG_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress(no-alloc scratch)");
    addr[(size_t)dev] = p;
  }
  *out = addr[(size_t)dev];
  return PG_OK;
}

template <typename T, bool SUP, bool CONN8>
static pg_status run_noalloc_t(RImg im, cudaStream_t s) {
  constexpr int RT = tile_side<T>(), RTHREADS = RT;
  im.tiles_x = (int)ceil_div(im.W, RT);
  im.tiles_y = (int)ceil_div(im.H, RT);
  im.tile_begin = 0;
  int64_t ntiles = 0, max_tiles = 0;
  noalloc_tiles((int)sizeof(T), im.H, im.W, ntiles, max_tiles);
  if (ntiles == 0) return PG_OK;
  if (ntiles > max_tiles)
    return fail(PG_ERR_INVALID_ARGUMENT, "pg_reconstruction_noalloc: the image needs " + std::to_string(ntiles) +
                                             " tiles of " + std::to_string(RT) + "x" + std::to_string(RT) +
                                             " pixels; the fixed scratch holds at most " + std::to_string(max_tiles));
  void *base = nullptr;
  PG_TRY(noalloc_scratch(&base));
  // the control block and both flag buffers must start at zero; the array keeps the
  // previous call's contents
  const size_t used = kNoAllocFlagsOffset + 2 * sizeof(unsigned) * (size_t)ntiles;
  PG_CUDA_TRY(cudaMemsetAsync(base, 0, used, s), "clear no-alloc scratch");
  RParams<T> P{};
  P.single = im;
  P.imgs = nullptr;
  P.nimg = 1;
  P.ntiles = (int)ntiles;
  P.ctl = static_cast<RCtl *>(base);
  P.flags = reinterpret_cast<unsigned *>(static_cast<char *>(base) + kNoAllocFlagsOffset);
  P.max_rounds = max_rounds_for(ntiles);
  P.wait_ns = g_dbg_wait_ns.load();
  P.init = INIT_MARKER;
  P.mask_mode = MASK_PLAIN;
  P.epi = EPI_NONE;
  P.h = static_cast<T>(0);
  auto kern = k_reconstruct<T, SUP, CONN8>;
  int per_sm = 0;
  PG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RTHREADS, 0), "occupancy");
  if (per_sm < 1) return fail(PG_ERR_CUDA, "reconstruction kernel cannot be resident");
  int64_t grid = (int64_t)per_sm * num_sms();
  if (grid > ntiles) grid = ntiles;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(RTHREADS);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, P), "cooperative reconstruction launch (no-alloc)");
  return PG_OK;
}

static pg_status reconstruction_noalloc(bool dilate, bool conn8, const pg_image &marker, const pg_image &mask,
                                        const pg_image &out, cudaStream_t s) {
  const Dims d = dims_of(mask);
  RImg im{};
  im.marker = marker.data;
  im.mask = mask.data;
  im.rec = out.data;
  im.out = out.data;
  im.H = d.nz * d.ny;
  im.W = d.nx;
  PG_DISPATCH_PTYPE(mask.ptype, T, {
    if (dilate) return conn8 ? run_noalloc_t<T, true, true>(im, s) : run_noalloc_t<T, true, false>(im, s);
    return conn8 ? run_noalloc_t<T, false, true>(im, s) : run_noalloc_t<T, false, false>(im, s);
  });
  return PG_OK;
}

}  // namespace pg

#include "recon3d_resident.cuh"

extern "C" {

// Test hooks: lower the reconstruction's round / visit cap and its device wait limit so that a test
// can make a bounded wait run out and read PG_ERR_NOT_CONVERGED back; 0 restores the defaults.
pg_status pg_debug_set_limits(int32_t max_rounds, int64_t wait_ns) {
  if (max_rounds < 0 || wait_ns < 0) return pg::fail(PG_ERR_INVALID_ARGUMENT, "pg_debug_set_limits: negative limit");
  pg::g_dbg_max_rounds.store(max_rounds);
  pg::g_dbg_wait_ns.store(wait_ns > 0 ? (unsigned long long)wait_ns : pg::kBarrierTimeoutNs);
  return PG_OK;
}

int32_t pg_last_reconstruction_rounds(void) {
  int r = -1;
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  if (cudaMemcpyFromSymbol(&r, pg::g_recon_rounds, sizeof(int)) != cudaSuccess) return -1;
  return r;
}

// Reconstruction that allocates nothing: same checks and result as pg_reconstruction, scratch
// taken from g_noalloc_scratch.  The first call on a device looks up that array's device
// address; make it before any stream capture.
pg_status pg_reconstruction_noalloc(int32_t type, const pg_image *marker, const pg_image *mask, int32_t se,
                                    const pg_image *out, pg_stream_t stream) {
  // the checks of pg_reconstruction, in its order
  PG_TRY(pg::check_in_out(marker, out, "t_Reconstruct"));
  PG_TRY(pg::check_in_out(mask, out, "t_Reconstruct"));
  if (type != PG_RECONSTRUCT_ERODE && type != PG_RECONSTRUCT_DILATE)
    return pg::fail(PG_ERR_INVALID_ARGUMENT, "t_ReconstructionDispatchRectType unsupported reconstruction_type");
  bool conn8 = true;
  PG_TRY(pg::recon_se(se, mask->rank, conn8));
  // then the limits of this entry point
  if (mask->rank == 3)
    return pg::fail(PG_ERR_UNSUPPORTED_SE, "pg_reconstruction_noalloc: 1D and 2D images only (volumes need "
                                           "pg_reconstruction)");
  const pg::Dims d = pg::dims_of(*mask);
  int64_t ntiles = 0, max_tiles = 0;
  pg::noalloc_tiles(pg::elem_size(mask->ptype), d.nz * d.ny, d.nx, ntiles, max_tiles);
  if (ntiles > max_tiles)
    return pg::fail(PG_ERR_INVALID_ARGUMENT, "pg_reconstruction_noalloc: the image needs " + std::to_string(ntiles) +
                                                 " tiles; the fixed scratch holds at most " + std::to_string(max_tiles));
  return pg::reconstruction_noalloc(type == PG_RECONSTRUCT_DILATE, conn8, *marker, *mask, *out,
                                    reinterpret_cast<cudaStream_t>(stream));
}

pg_status pg_batch_plan_set_config(pg_batch_plan *plan, int32_t tile, int32_t sweeps) {
  if (!plan) return pg::fail(PG_ERR_INVALID_ARGUMENT, "null plan");
  if (tile != 32 && tile != 64) return pg::fail(PG_ERR_INVALID_ARGUMENT, "batch plan tile side must be 32 or 64");
  if (tile == 64 && pg::elem_size(plan->ptype) == 8)
    return pg::fail(PG_ERR_INVALID_ARGUMENT, "batch plan tile side 64 needs pixels of at most 4 bytes");
  if (sweeps < 1) return pg::fail(PG_ERR_INVALID_ARGUMENT, "batch plan sweeps per visit must be >= 1");
  plan->cfg = pg::PlanCfg{tile, sweeps};
  return PG_OK;
}

pg_status pg_batch_plan_config(const pg_batch_plan *plan, int32_t *tile, int32_t *sweeps, int32_t *grid) {
  if (!plan) return pg::fail(PG_ERR_INVALID_ARGUMENT, "null plan");
  if (tile) *tile = plan->cfg.rt;
  if (sweeps) *sweeps = plan->cfg.sweeps;
  if (grid) *grid = plan->grid;
  return PG_OK;
}

}  // extern "C"
