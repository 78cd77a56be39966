// label.cu -- connected-component labelling: poutre::label::label_binary and label_flat_zones
// (src/label/label_binary.cpp, src/label/label_flat_zones.cpp; algorithm in
// include/poutre/label/details/label_t.hpp:132-247).
//
// The reference scans in raster order: an accepted pixel joins the provisional labels of its
// related upper-half neighbours (disjoint sets, the smaller root wins) or opens a new one; the
// roots are then numbered 1.. in creation order and every accepted pixel takes its root's number.
// A component's root is the provisional label of its first pixel in raster order (that pixel has no
// related earlier neighbour), so the result is: components numbered by the raster position of their
// first pixel.  The GPU builds the same components with a union-find over pixel indices (parent[]
// only ever points to a smaller index; a root hangs under the smaller root), so each component's
// root is its first pixel, and numbers the roots in raster order:
//   tile     -- a CTA labels a tile of 8192 pixels in shared memory.  A warp turns 32 pixels of a row
//               into bit masks (one ballot per kind of edge); a thread then owns those 32 pixels as
//               runs: each run hangs under the first run above that it touches, pointer jumping flattens
//               these trees, and the few edges left (runs that touch several above) are united.  It
//               writes every pixel's tile root and a bitmap of the tile roots;
//   border   -- the edges between tiles (and, in a volume, between slices) are united in global memory;
//   flatten  -- the tile roots find their component's root; the bitmap keeps the components' roots;
//   number   -- the roots take their number from the bitmap, in raster order;
//   resolve  -- every pixel takes its root's number, at most three loads away.
// The global union-find that did all edges before (one thread per pixel, every edge an atomic) spent
// 0.80 ms on a thresholded 2048^2 u8 image, nearly all of it in long chains of dependent loads
// contending for the same few roots; a tile's chains are in shared memory, and one pixel in forty
// reaches global memory.  2048^2 u8 binary: tile 25 us,
// border 11, flatten 6, number 5, resolve 11; 75 us a call with the count's read back, against 800.  Where
// nearly every pixel is a component of its own there are no such chains, and small images of that kind
// are what the tiles cost most on: flat zones of 512^2 noise 56 us against 53, of 605 x 216 textured by
// threes 71 against 42 (512^2 blobs 52 against 188).
// The floor (input read, labels written) is 5.6 us; the tile pass is bound by the dependent shared-memory
// loads of the runs (40 % of the issue slots), border and flatten by the L2 latency of their chains.
//
// An edge that follows from other edges is skipped: with L / U / UL / UR the edges of pixel x to its
// left / upper / upper-left / upper-right neighbour and L' those of the row above,
//   U(x)  follows from L(x), U(x-1), L'(x);
//   UL(x) follows from L(x), U(x-1) or from U(x), L'(x);
//   UR(x) follows from U(x), L'(x+1) or from L(x+1), U(x+1).
// U depends only on edges further left and UL, UR only on U, so no edge is dropped in a circle; one
// union per pair of touching runs remains.
//
// Edges are the reference's: pixel p and its upper-half neighbour q (earlier in raster order) of the
// SE are joined when p is accepted and q is related -- binary: p != 0 and q > 0 (a negative pixel is
// accepted but joins no later pixel), flat zones: p == q.  Binary labelling of float images is not
// on this path (the reference's background test |v| > 1e-10 and its neighbour test v > 0 disagree on
// (0, 1e-10], where it reads an unset label), nor is SESquare3D (its upper half in the reference is
// not the raster-earlier half).
//
// Every find / union loop is bounded (kLabelIters); exceeding it records PG_ERR_CUDA in
// g_label_status, read by pg_check_device.
#include <algorithm>

#include "common.cuh"

namespace pg {

__device__ int g_label_status = 0;

namespace {

constexpr int kLabelIters = 1 << 24;
constexpr int kLThreads = 256;
constexpr int kLTile = 32 * kLThreads;             // pixels of a tile: one 32-pixel chunk of a row per thread
constexpr int kLSegments = 2048;                   // most bitmap segments of the numbering pass

// which neighbours of the SE's raster-earlier half exist
enum : unsigned { E_L = 1, E_U = 2, E_UL = 4, E_UR = 8, E_Z = 16 };

struct LabelGeom {
  int64_t nx, ny, nz;
  int64_t tiles_x, tiles_y;  // tiles per slice
  int slices;                // slices of a tile, one under the other (more than one only where tiles_y == 1)
  int64_t words_x;           // bitmap words per row (32 pixels each, rows padded)
  int log_tw;                // tile width (a multiple of 32); the height is kLTile >> log_tw
  unsigned edges;
};

template <typename T, bool FLAT> __device__ __forceinline__ bool accepted(T v) { return FLAT || v != T(0); }
template <typename T, bool FLAT> __device__ __forceinline__ bool joined(T p, T q) {
  return FLAT ? p == q : (p != T(0) && q > T(0));
}

__device__ __forceinline__ void label_gave_up() { atomicCAS(&g_label_status, 0, (int)PG_ERR_CUDA); }

// Loads go past L1 (other CTAs write).  A parent replaced by its own parent stays an ancestor, so later walks through
// the same tile roots are short (border unions of 2048^2 blobs: 20 -> 14 us).  A background pixel (parent < 0) is never
// reached: only accepted pixels are joined.
__device__ __forceinline__ int32_t find_halving(int32_t *par, int32_t x) {
  for (int it = 0; it < kLabelIters; ++it) {
    const int32_t p = __ldcg(par + x);
    if (p == x) return x;
    if (p < 0) break;
    const int32_t q = __ldcg(par + p);
    if (q == p) return p;
    if (q < 0) break;
    __stcg(par + x, q);
    x = q;
  }
  label_gave_up();
  return x;
}

__device__ __forceinline__ void unite(int32_t *par, int32_t a, int32_t b) {
  for (int it = 0; it < kLabelIters; ++it) {
    a = find_halving(par, a);
    b = find_halving(par, b);
    if (a == b) return;
    if (a < b) { const int32_t t = a; a = b; b = t; }  // hang the larger root under the smaller
    const int32_t old = atomicCAS(par + a, a, b);
    if (old == a) return;
    a = old;
  }
  label_gave_up();
}

// ------------------------------------------------------------------ tile
template <typename T> __device__ __forceinline__ T shfl_dn(T v, int d) {
  if constexpr (sizeof(T) < 4) return (T)__shfl_down_sync(0xffffffffu, (unsigned)v, d);
  else if constexpr (std::is_same_v<T, int64_t>) return (T)__shfl_down_sync(0xffffffffu, (long long)v, d);
  else return __shfl_down_sync(0xffffffffu, v, d);
}
template <typename T> __device__ __forceinline__ T shfl_up(T v, int d) {
  if constexpr (sizeof(T) < 4) return (T)__shfl_up_sync(0xffffffffu, (unsigned)v, d);
  else if constexpr (std::is_same_v<T, int64_t>) return (T)__shfl_up_sync(0xffffffffu, (long long)v, d);
  else return __shfl_up_sync(0xffffffffu, v, d);
}

// A pixel as its row's equalities are tested.  Doubles as integers, for the double-precision pipe compares 32 of them in
// 16 cycles or more (flat zones of 334 x 1120 f64: 22000 of a tile's 80000 cycles): equal bits mean equal values but for
// the two zeros, which become one, and NaN, which equals nothing (key_nan).
template <typename T> struct KeyOf { using type = T; };
template <> struct KeyOf<double> { using type = int64_t; };
template <typename T> using Key = typename KeyOf<T>::type;
template <typename T> __device__ __forceinline__ Key<T> key_of(T v) {
  if constexpr (std::is_same_v<T, double>) {
    const int64_t b = __double_as_longlong(v);
    return (b & 0x7fffffffffffffffll) == 0 ? 0 : b;
  } else {
    return v;
  }
}
template <typename T> __device__ __forceinline__ bool key_nan(Key<T> k) {
  if constexpr (std::is_same_v<T, double>) return (k & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
  else return false;
}

// FULL: the form that waits less -- many runs of a chunk (noise, vertical segments) are handled four at a time, and the
// pointer jumping ends with the first turn that moves nothing -- and that takes several slices a tile.  Where there
// are tiles enough to hide the waits its longer code costs 3 % (binary 2048^2: 75 us without it, 77 with; flat zones
// of 512^2 100 without, 86 with; 28 x 3 x 199 along z 100, 51).
template <typename T, bool FLAT, bool FULL>
__global__ void __launch_bounds__(kLThreads) k_label_tile(const T *__restrict__ in, int32_t *__restrict__ par,
                                                          unsigned *__restrict__ roots, LabelGeom g) {
  // masks of the chunks: chunk id = chunk column * tile rows + row, so the chunk above is id - 1.
  // Flat zones: the four kinds of edge.  Binary: pixels != 0 and pixels > 0; the edges follow from them.
  __shared__ unsigned s_m[FLAT ? 4 : 2][kLThreads];
  __shared__ unsigned s_l[kLThreads], s_u[kLThreads];  // left and upper edges, for the neighbour chunks
  __shared__ unsigned s_start[kLThreads], s_acc[kLThreads];
  __shared__ int32_t s_p[kLTile];  // parents of the run starts
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int log_th = 13 - g.log_tw, tw = 1 << g.log_tw, th = 1 << log_th;
  static_assert(kLTile == 1 << 13, "tile geometry");
  const uint32_t tile = blockIdx.x, tiles_x = (uint32_t)g.tiles_x, tiles_y = (uint32_t)g.tiles_y;
  const int nx = (int)g.nx;  // the image has less than 2^31 pixels: its indices are 32-bit
  const int x0 = (int)(tile % tiles_x) << g.log_tw, y0 = (int)(tile / tiles_x % tiles_y) << log_th;
  const int ny = (int)g.ny, z0 = (int)(tile / tiles_x / tiles_y) * (FULL ? g.slices : 1);
  const int row0 = z0 * ny + y0;  // first row, slices stacked
  const int w = min(tw, nx - x0);  // the tile inside the image
  const int h = FULL && g.slices > 1 ? min(g.slices, (int)g.nz - z0) * ny : min(th, ny - y0);
  const int base = row0 * nx + x0;
  const T *src = in + base;
  const bool hor = (g.edges & E_L) != 0, ver = (g.edges & E_U) != 0, eul = (g.edges & E_UL) != 0,
             eur = (g.edges & E_UR) != 0;

  // pixel c of row r, and (lanes 0 and 31) the pixel beside the chunk, if in the tile
  auto load = [&](int r, int c, Key<T> &v, Key<T> &e) {
    const int ce = lane == 0 ? c - 1 : c + 1;
    const T *q = src + r * nx;
    const bool row = r < h;
    v = (row && c < w) ? key_of(q[c]) : Key<T>(0);
    e = (FLAT && row && (lane == 0 || lane == 31) && (unsigned)ce < (unsigned)w) ? key_of(q[ce]) : Key<T>(0);
  };
  // ---- masks: a warp walks down its chunks
  constexpr int AT = FLAT ? 8 : 16;        // chunks whose loads go together
  Key<T> pv = 0, pe = 0, nv[AT], ne[AT];  // pv, pe: the row above
  if (FLAT && ((warp * 32) & (th - 1)) != 0)
    load(((warp * 32) & (th - 1)) - 1, ((warp * 32) >> log_th) * 32 + lane, pv, pe);
#pragma unroll 1
  for (int k0 = 0; k0 < 32; k0 += AT) {
#pragma unroll
    for (int k = 0; k < AT; ++k) {
      const int id = warp * 32 + k0 + k;
      load(id & (th - 1), (id >> log_th) * 32 + lane, nv[k], ne[k]);
    }
#pragma unroll
    for (int k = 0; k < AT; ++k) {
      const int id = warp * 32 + k0 + k;
      const Key<T> v = nv[k], e = ne[k];
      unsigned m0, m1, m2 = 0u, m3 = 0u;
      if constexpr (FLAT) {
        Key<T> vl = shfl_up(v, 1), ul = shfl_up(pv, 1), ur = shfl_dn(pv, 1);
        if (lane == 0) { vl = e; ul = pe; }
        if (lane == 31) ur = pe;
        m0 = __ballot_sync(0xffffffffu, v == vl);
        m1 = __ballot_sync(0xffffffffu, v == pv);
        m2 = __ballot_sync(0xffffffffu, v == ul);
        m3 = __ballot_sync(0xffffffffu, v == ur);
        if constexpr (std::is_same_v<T, double>) {
          const unsigned num = ~__ballot_sync(0xffffffffu, key_nan<T>(v));
          m0 &= num;
          m1 &= num;
          m2 &= num;
          m3 &= num;
        }
        pv = v;
        pe = e;
      } else {
        m0 = __ballot_sync(0xffffffffu, v != T(0));
        m1 = std::is_unsigned_v<T> ? m0 : __ballot_sync(0xffffffffu, v > T(0));
      }
      if (lane == 0) {
        s_m[0][id] = m0;
        if (FLAT || !std::is_unsigned_v<T>) s_m[1][id] = m1;
        if constexpr (FLAT) {
          s_m[2][id] = m2;
          s_m[3][id] = m3;
        }
      }
    }
  }
  __syncthreads();

  // ---- runs: thread t owns chunk t
  const int id = threadIdx.x, r = id & (th - 1), cx = id >> log_th;
  const bool has_left = cx > 0, has_right = (cx + 1) * 32 < tw;      // neighbour chunks of the tile
  const bool has_up = FULL ? (unsigned)r % (unsigned)ny != 0u : r > 0;  // no edge up from a slice's first row
  const int l0 = (r << g.log_tw) + cx * 32;  // local raster index of the chunk's first pixel
  unsigned L, U = 0u, UL = 0u, UR = 0u, acc;
  {
    // pixels of the chunk inside the image, and of those the ones with a neighbour on the left / right
    const int wc = w - cx * 32;
    const unsigned in_m = r >= h || wc <= 0 ? 0u : wc >= 32 ? 0xffffffffu : (1u << wc) - 1u;
    const unsigned left_m = has_left ? in_m : in_m & ~1u, right_m = wc > 32 ? in_m : in_m & (in_m >> 1);
    if constexpr (FLAT) {
      acc = in_m;
      L = s_m[0][id];
      if (has_up) { U = s_m[1][id]; UL = s_m[2][id]; UR = s_m[3][id]; }
    } else {
      constexpr int POS = std::is_unsigned_v<T> ? 0 : 1;  // unsigned pixels: > 0 is != 0
      acc = s_m[0][id] & in_m;
      L = (s_m[POS][id] << 1) | (has_left ? s_m[POS][id - th] >> 31 : 0u);
      if (has_up) {
        U = s_m[POS][id - 1];
        UL = (U << 1) | (has_left ? s_m[POS][id - 1 - th] >> 31 : 0u);
        UR = (U >> 1) | (has_right ? s_m[POS][id - 1 + th] << 31 : 0u);
      }
    }
    L = hor ? L & acc & left_m : 0u;
    U = ver ? U & acc : 0u;
    UL = eul ? UL & acc & left_m : 0u;
    UR = eur ? UR & acc & right_m : 0u;
  }
  const unsigned starts = acc & ~(L & ~1u);  // a chunk's first pixel always starts a run
  s_l[id] = L;
  s_u[id] = U;
  s_start[id] = starts;
  s_acc[id] = acc;
  __syncthreads();
  // parents are stored with the row folded into the bank, or a column of runs would share one bank
  auto ph = [&](int l) { return l ^ ((l >> g.log_tw) & 31); };
  auto run_of = [&](int i, int x) {  // start (local index) of the run that holds pixel x of chunk i
    const int ri = i & (th - 1), ci = i >> log_th;
    return (ri << g.log_tw) + ci * 32 + 31 - __clz(s_start[i] & (0xffffffffu >> (31 - x)));
  };
  auto above = [&](int x) {  // the run that holds the pixel above x, x in [-1, 32]
    return x < 0 ? run_of(id - 1 - th, 31) : x > 31 ? run_of(id - 1 + th, 0) : run_of(id - 1, x);
  };
  {
    const unsigned Lu = has_up ? s_l[id - 1] : 0u;  // left edges of the row above
    const unsigned Ul = (U << 1) | (has_left ? s_u[id - th] >> 31 : 0u);
    const unsigned Lur = (Lu >> 1) | (has_up && has_right ? s_l[id - 1 + th] << 31 : 0u);
    const unsigned Lr = (L >> 1) | (has_right ? s_l[id + th] << 31 : 0u);
    const unsigned Ur = (U >> 1) | (has_right ? s_u[id + th] << 31 : 0u);
    UR &= ~(U & Lur) & ~(Lr & Ur);
    UL &= ~(L & Ul) & ~(U & Lu);
    U &= ~(L & Ul & Lu);
    L &= 1u;  // inside a chunk the run holds it
  }
  unsigned hang = 0u;  // runs that hang under another
  for (unsigned todo = starts; todo; todo &= todo - 1) {
    const unsigned bit = todo & (0u - todo), later = todo ^ bit;
    const unsigned run = ~(bit - 1) & (later ? (later & (0u - later)) - 1u : 0xffffffffu);
    const unsigned e = (U | UL | UR) & run;
    const int l = l0 + __ffs(bit) - 1;
    int to = l;
    if (e) {
      const unsigned f = e & (0u - e);
      const int x = __ffs(f) - 1;
      if (U & f) { U ^= f; to = above(x); }
      else if (UL & f) { UL ^= f; to = above(x - 1); }
      else { UR ^= f; to = above(x + 1); }
    } else if (bit & L) {
      L = 0u;
      to = run_of(id - th, 31);
    }
    s_p[ph(l)] = to;
    if (to != l) hang |= bit;
  }
  __syncthreads();
  // pointer jumping: a link goes up a row or left a chunk, so six doublings flatten the usual tree
  // (what is deeper still is walked by find).  Roots stay where they are (in noise nearly every run is one).
  volatile int32_t *vp = s_p;
#pragma unroll 1
  for (int it = 0; it < 6; ++it) {
    bool moved = false;
    unsigned todo = hang;
    // many runs in a chunk (vertical segments, noise): the loads of four go together
    while (FULL && __popc(todo) > 6) {
      int i[4], p[4];
#pragma unroll
      for (int k = 0; k < 4; ++k, todo &= todo - 1) {
        i[k] = ph(l0 + __ffs(todo) - 1);
        p[k] = vp[i[k]];
      }
      int q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = vp[ph(p[k])];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        moved |= q[k] != p[k];
        vp[i[k]] = q[k];
      }
    }
    for (; todo; todo &= todo - 1) {
      const int i = ph(l0 + __ffs(todo) - 1), p = vp[i], q = vp[ph(p)];
      if (FULL) moved |= q != p;
      vp[i] = q;
    }
    if constexpr (FULL) {
      if (!__syncthreads_or(moved)) break;
    } else {
      __syncthreads();
    }
  }
  // the edges left
  auto find = [&](int x) {
    for (int it = 0; it < kLabelIters; ++it) {
      const int p = vp[ph(x)];
      if (p == x) return x;
      x = p;
    }
    label_gave_up();
    return x;
  };
  auto join = [&](int a, int b) {
    for (int it = 0; it < kLabelIters; ++it) {
      a = find(a);
      b = find(b);
      if (a == b) return;
      if (a < b) { const int t = a; a = b; b = t; }  // hang the larger root under the smaller
      const int old = atomicCAS(s_p + ph(a), a, b);
      if (old == a) return;
      a = old;
    }
    label_gave_up();
  };
  for (unsigned todo = U | UL | UR; todo; todo &= todo - 1) {
    const unsigned f = todo & (0u - todo);
    const int x = __ffs(f) - 1, me = run_of(id, x);
    if (U & f) join(me, above(x));
    if (UL & f) join(me, above(x - 1));
    if (UR & f) join(me, above(x + 1));
  }
  if (L) join(l0, run_of(id - th, 31));
  __syncthreads();
  unsigned root_m = 0u, todo4 = starts;
  while (FULL && __popc(todo4) > 6) {  // as above
    int i[4], p[4];
    unsigned bit[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      bit[k] = todo4 & (0u - todo4);
      todo4 ^= bit[k];
      i[k] = p[k] = l0 + __ffs(bit[k]) - 1;
    }
    bool more = true;
    for (int it = 0; more; ++it) {
      int q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = vp[ph(p[k])];
      more = false;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        more |= q[k] != p[k];
        p[k] = q[k];
      }
      if (more && it == kLabelIters) {
        label_gave_up();
        break;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      vp[ph(i[k])] = p[k];
      if (p[k] == i[k]) root_m |= bit[k];
    }
  }
  for (unsigned todo = todo4; todo; todo &= todo - 1) {
    const int l = l0 + __ffs(todo) - 1, p = find(l);
    vp[ph(l)] = p;
    if (p == l) root_m |= todo & (0u - todo);
  }
  if (r < h && cx * 32 < w) roots[(int64_t)(row0 + r) * g.words_x + (x0 >> 5) + cx] = root_m;
  __syncthreads();  // every tree is flat and no thread reads another's runs any more
  for (unsigned todo = starts; todo; todo &= todo - 1) {
    const int i = ph(l0 + __ffs(todo) - 1), p = vp[i];
    vp[i] = base + (p >> g.log_tw) * nx + (p & (tw - 1));  // the root's index in the image
  }
  __syncthreads();

  // ---- output: a warp per chunk again
#pragma unroll 8
  for (int k = 0; k < 32; ++k) {
    const int i = warp * 32 + k, ri = i & (th - 1), c = (i >> log_th) * 32 + lane;
    if (ri < h && c < w) {
      const bool a = (s_acc[i] >> lane) & 1u;
      const int b = a ? 31 - __clz(s_start[i] & (0xffffffffu >> (31 - lane))) : lane;
      const int q = (ri << g.log_tw) + c - lane + b;
      const int32_t root = s_p[ph(q)];  // not a parent where the pixel is background: any word is read
      par[base + ri * nx + c] = a ? root : -1;
    }
  }
}

// ------------------------------------------------------------------ borders
// Work items: the pixels of the rows that start a tile row (edges up), the pixels that start a tile in
// their row (left edge, and the two diagonals that cross the border inside a tile row), and in a volume
// every pixel (the edge to the slice before).
template <typename T, bool FLAT>
__global__ void __launch_bounds__(kLThreads) k_label_border(const T *__restrict__ in, int32_t *par, LabelGeom g,
                                                            int64_t n_rows, int64_t n_cols, int64_t n_z) {
  const int th = kLTile >> g.log_tw;
  const bool hor = (g.edges & E_L) != 0, ver = (g.edges & E_U) != 0;
  const int64_t items = n_rows + n_cols + n_z;
  for (int64_t t = (int64_t)blockIdx.x * kLThreads + threadIdx.x; t < items; t += (int64_t)gridDim.x * kLThreads) {
    if (t < n_rows) {
      // every count below is less than 2^31: 32-bit divisions
      const uint32_t q = (uint32_t)t / (uint32_t)g.nx, x = (uint32_t)t % (uint32_t)g.nx, ty = (uint32_t)g.tiles_y - 1;
      const int64_t y = (int64_t)(q % ty + 1) * th, z = q / ty;
      const int64_t p = (z * g.ny + y) * g.nx + x, u = p - g.nx;
      const bool has_l = x > 0, has_r = x + 1 < g.nx;
      const T vc = in[p], uc = in[u];
      const T vl = has_l ? in[p - 1] : T(0), ul = has_l ? in[u - 1] : T(0);
      const T vr = has_r ? in[p + 1] : T(0), ur = has_r ? in[u + 1] : T(0);
      const bool L = hor && has_l && joined<T, FLAT>(vc, vl), Lu = hor && has_l && joined<T, FLAT>(uc, ul);
      const bool U = ver && joined<T, FLAT>(vc, uc), Ul = ver && has_l && joined<T, FLAT>(vl, ul);
      if (U && !(L && Ul && Lu)) unite(par, (int32_t)p, (int32_t)u);
      if ((g.edges & E_UL) && has_l && joined<T, FLAT>(vc, ul) && !(L && Ul) && !(U && Lu))
        unite(par, (int32_t)p, (int32_t)u - 1);
      if ((g.edges & E_UR) && has_r && joined<T, FLAT>(vc, ur)) {
        const bool Lur = hor && joined<T, FLAT>(ur, uc), Lr = hor && joined<T, FLAT>(vr, vc);
        const bool Ur = ver && joined<T, FLAT>(vr, ur);
        if (!(U && Lur) && !(Lr && Ur)) unite(par, (int32_t)p, (int32_t)u + 1);
      }
    } else if (t < n_rows + n_cols) {
      const uint32_t c = (uint32_t)(t - n_rows), tx = (uint32_t)g.tiles_x - 1, row = c / tx;
      const int64_t x = (int64_t)(c % tx + 1) << g.log_tw;
      const int64_t y = row % (uint32_t)g.ny, p = (int64_t)row * g.nx + x;
      const T vc = in[p], vl = in[p - 1];
      const bool L = hor && joined<T, FLAT>(vc, vl);
      if (y % th == 0) {  // no row above in this tile row: its diagonals are among the row items
        if (L) unite(par, (int32_t)p, (int32_t)p - 1);
        continue;
      }
      const int64_t u = p - g.nx;
      const T uc = in[u], ul = in[u - 1];
      const bool U = ver && joined<T, FLAT>(vc, uc), Ul = ver && joined<T, FLAT>(vl, ul);
      const bool Lu = hor && joined<T, FLAT>(uc, ul);
      // the left edge follows from the one of the row above and both upper edges
      if (L && !(U && Ul && Lu)) unite(par, (int32_t)p, (int32_t)p - 1);
      if ((g.edges & E_UL) && joined<T, FLAT>(vc, ul) && !(L && Ul) && !(U && Lu)) unite(par, (int32_t)p, (int32_t)u - 1);
      // the upper-right edge of the pixel on the left of the border
      if ((g.edges & E_UR) && joined<T, FLAT>(vl, uc) && !(Ul && Lu) && !(L && U)) unite(par, (int32_t)p - 1, (int32_t)u);
    } else {
      const int64_t i = t - n_rows - n_cols, plane = g.nx * g.ny, p = i + plane;
      const T vc = in[p], zc = in[i];
      if (!joined<T, FLAT>(vc, zc)) continue;
      if (hor && (uint32_t)p % (uint32_t)g.nx != 0) {
        const T vl = in[p - 1], zl = in[i - 1];
        if (joined<T, FLAT>(vc, vl) && joined<T, FLAT>(vl, zl) && joined<T, FLAT>(zc, zl)) continue;
      }
      unite(par, (int32_t)p, (int32_t)i);
    }
  }
}

// ------------------------------------------------------------------ numbering
// Tile roots find their component's root; the bitmap keeps the components' roots, counted per segment.
// PARTS threads a word, whose roots are followed four at a time: noise and the columns of vertical segments have up to
// 32 tile roots a word, each a chain of L2 loads (12 x 10 x 363 along z: 40 us with a thread a word and one root after
// the other, 12 with four threads; with few roots a word one thread is 1 us faster on 2048^2).
template <int PARTS>
__global__ void __launch_bounds__(kLThreads) k_label_flatten(int32_t *par, unsigned *__restrict__ roots,
                                                             int32_t *__restrict__ cnt, LabelGeom g, int64_t words,
                                                             int log_seg) {
  const int64_t t = (int64_t)blockIdx.x * kLThreads + threadIdx.x, wi = t / PARTS;
  const unsigned which = (unsigned)t % PARTS, part = PARTS == 1 ? ~0u : 0xffu << (8 * which);
  const unsigned m = wi < words ? roots[wi] : 0u;
  unsigned gone = 0u;
  if (m & part) {
    const int64_t row = (uint32_t)wi / (uint32_t)g.words_x;
    const int32_t i0 = (int32_t)(row * g.nx + (wi - row * g.words_x) * 32);
    for (unsigned todo = m & part; todo;) {
      unsigned bit[4];
      int32_t p[4];  // the pixel, then its ancestors; -1: no root here
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        bit[k] = todo & (0u - todo);
        todo ^= bit[k];
        p[k] = bit[k] ? i0 + __ffs(bit[k]) - 1 : -1;
      }
      bool more = true;
      for (int it = 0; more; ++it) {
        int32_t q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = p[k] >= 0 ? __ldcg(par + p[k]) : -1;
        more = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (q[k] < 0 || q[k] == p[k]) continue;
          p[k] = q[k];
          more = true;
        }
        if (more && it == kLabelIters) {
          label_gave_up();
          break;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int32_t i = i0 + __ffs(bit[k]) - 1;
        if (p[k] < 0 || p[k] == i) continue;
        gone |= bit[k];
        __stcg(par + i, p[k]);
      }
    }
  }
  if constexpr (PARTS == 4) {
    gone |= __shfl_xor_sync(0xffffffffu, gone, 1);
    gone |= __shfl_xor_sync(0xffffffffu, gone, 2);
  }
  if (gone != 0u && which == 0) roots[wi] = m & ~gone;
  int32_t own = __popc(m & ~gone & part);
  // a segment is a whole number of CTAs' words
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) own += __shfl_xor_sync(0xffffffffu, own, o);
  if ((threadIdx.x & 31) == 0 && own) atomicAdd(cnt + (wi >> log_seg), own);
}

// CTA b numbers the roots of bitmap segment b: the roots before it are the sum of the earlier segments'
// counts.  A root's parent word becomes -1 - number (numbers start at 1; -1 stays the background).  A thread scans
// WPT words at a time: four, or one where the image is so small that four would leave most SMs without a segment.
// A word with more than kLDense roots is written by its warp, a lane per pixel (whole lines), others by their thread.
// (flat zones of 512^2 noise, nearly every pixel a root: 20 us with four words a thread and no whole lines, now 7).
constexpr int kLDense = 16;
template <int WPT>
__global__ void __launch_bounds__(kLThreads) k_label_number(int32_t *__restrict__ par, const unsigned *__restrict__ roots,
                                                            const int32_t *__restrict__ cnt, LabelGeom g, int64_t words,
                                                            int log_seg, long long *__restrict__ total) {
  __shared__ int32_t s_w[2][kLThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t before = 0;
  for (int j = threadIdx.x; j < (int)blockIdx.x; j += kLThreads) before += cnt[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 0) s_w[0][warp] = before;
  __syncthreads();
  int32_t base = 0;
#pragma unroll
  for (int w = 0; w < kLThreads / 32; ++w) base += s_w[0][w];
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    *(volatile long long *)total = (long long)base + cnt[blockIdx.x];
    __threadfence_system();  // it may be host memory
  }
  if (cnt[blockIdx.x] == 0) return;
  const int64_t end = min(words, ((int64_t)blockIdx.x + 1) << log_seg);
  int buf = 1;
  for (int64_t w0 = (int64_t)blockIdx.x << log_seg; w0 < end; w0 += WPT * kLThreads, buf ^= 1) {
    const int64_t wi = w0 + threadIdx.x * WPT;
    unsigned mw[WPT];
    if constexpr (WPT == 4) {  // the bitmap is padded to whole vectors
      uint4 m = make_uint4(0u, 0u, 0u, 0u);
      if (wi < end) m = *reinterpret_cast<const uint4 *>(roots + wi);
      mw[0] = m.x;
      mw[1] = wi + 1 < end ? m.y : 0u;
      mw[2] = wi + 2 < end ? m.z : 0u;
      mw[3] = wi + 3 < end ? m.w : 0u;
    } else {
      mw[0] = wi < end ? roots[wi] : 0u;
    }
    int32_t own = 0;
#pragma unroll
    for (int j = 0; j < WPT; ++j) own += __popc(mw[j]);
    int32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s_w[buf][warp] = incl;
    __syncthreads();  // one barrier a turn: the other buffer is rewritten only after the next one
    int32_t pre = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kLThreads / 32; ++w) {
      const int32_t c = s_w[buf][w];
      if (w < warp) pre += c;
      all += c;
    }
    int32_t code = -1 - (base + pre + incl - own);
#pragma unroll
    for (int j = 0; j < WPT; ++j) {
      const unsigned m = mw[j];
      const int64_t row = (uint32_t)(wi + j) / (uint32_t)g.words_x;
      const int32_t i0 = (int32_t)(row * g.nx + (wi + j - row * g.words_x) * 32);
      const bool dense = __popc(m) > kLDense;
      for (unsigned todo = __ballot_sync(0xffffffffu, dense); todo; todo &= todo - 1) {
        const int w = __ffs(todo) - 1;
        const unsigned mo = __shfl_sync(0xffffffffu, m, w);
        const int32_t first = __shfl_sync(0xffffffffu, i0, w), c = __shfl_sync(0xffffffffu, code, w);
        if ((mo >> lane) & 1u) par[first + lane] = c - 1 - __popc(mo & ((1u << lane) - 1u));
      }
      if (dense) code -= __popc(m);
      else
        for (unsigned todo = m; todo; todo &= todo - 1) par[i0 + __ffs(todo) - 1] = --code;
    }
    base += all;
  }
}

// Every pixel takes its root's number: its own word, its tile root's, or the component root's.  The four
// pixels of a thread go together, so that their loads overlap.
template <bool VEC>
__global__ void __launch_bounds__(kLThreads) k_label_resolve(const int32_t *__restrict__ par, int64_t n,
                                                             int64_t *__restrict__ out) {
  const int64_t i = ((int64_t)blockIdx.x * kLThreads + threadIdx.x) * 4;
  if (i >= n) return;
  const int4 v = *reinterpret_cast<const int4 *>(par + i);  // par is padded to whole vectors
  int32_t p[4] = {v.x, i + 1 < n ? v.y : -1, i + 2 < n ? v.z : -1, i + 3 < n ? v.w : -1};
#pragma unroll
  for (int hop = 0; hop < 2; ++hop) {
    if (p[0] < 0 && p[1] < 0 && p[2] < 0 && p[3] < 0) break;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (p[j] >= 0) p[j] = __ldg(par + p[j]);
  }
  if (VEC && i + 3 < n) {
    __stcs(reinterpret_cast<longlong2 *>(out + i), make_longlong2(-1 - (int64_t)p[0], -1 - (int64_t)p[1]));
    __stcs(reinterpret_cast<longlong2 *>(out + i) + 1, make_longlong2(-1 - (int64_t)p[2], -1 - (int64_t)p[3]));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i + j < n) out[i + j] = -1 - (int64_t)p[j];
  }
}

// the raster-earlier half of the SE
bool upper_edges(int se, unsigned *e) {
  switch (se) {
    case PG_SE_SEGMENT_X_1D: case PG_SE_SEGMENT_X_2D: case PG_SE_SEGMENT_X_3D: *e = E_L; return true;
    case PG_SE_SEGMENT_Y_2D: case PG_SE_SEGMENT_Y_3D: *e = E_U; return true;
    case PG_SE_SEGMENT_Z_3D: *e = E_Z; return true;
    case PG_SE_SQUARE_2D: *e = E_L | E_U | E_UL | E_UR; return true;
    case PG_SE_CROSS_2D: *e = E_L | E_U; return true;
    case PG_SE_CROSS_3D: *e = E_L | E_U | E_Z; return true;
    default: return false;
  }
}

template <typename T, bool FLAT>
pg_status label_t(const pg_image &in, const pg_image &out, unsigned edges, int64_t *count, cudaStream_t s) {
  Dims d = dims_of(in);
  const int64_t n = d.count();
  // Axes of length 1 are dropped, so that what is left lies along rows: a column is a row whose edges up are edges
  // left (300000 pixels: 78 us as a column, 57 as a row)
  if (d.nx == 1) {
    edges = (edges & E_U ? E_L : 0u) | (edges & E_Z ? E_U : 0u);
    d.nx = d.ny; d.ny = d.nz; d.nz = 1;
  }
  if (d.ny == 1 && d.nz > 1) {
    edges = (edges & E_L) | (edges & E_Z ? E_U : 0u);
    d.ny = d.nz; d.nz = 1;
  }
  if (d.nx == 1) {  // only the slices were many
    edges = edges & E_U ? E_L : 0u;
    d.nx = d.ny; d.ny = 1;
  }
  LabelGeom g{};
  g.nx = d.nx; g.ny = d.ny; g.nz = d.nz;
  g.edges = edges;
  // Tiles of 128 x 64 pixels (1 pixel in 43 on a border).  So that a tile is not mostly outside the image, images of
  // up to 32 columns take 32 x 256, images of a few rows wider ones, and a tile holds as many slices of a volume as
  // fit (a tile 128 pixels wide per slice: 20000 binary slices of 8 x 8 333 us, now 89; 60000 x 32 flat 81, now 63).
  g.log_tw = d.nx <= 32 ? 5 : 7;
  while (g.log_tw < 13 && (kLTile >> g.log_tw) / 2 >= d.ny * d.nz) ++g.log_tw;
  const int64_t tw = 1ll << g.log_tw, th = kLTile >> g.log_tw;
  g.tiles_x = ceil_div(d.nx, tw);
  g.tiles_y = ceil_div(d.ny, th);
  // (one slice a tile while that gives no more than two tiles an SM: 64^3 62 us, 72 with two slices)
  g.slices = g.tiles_x * g.tiles_y * d.nz <= 2 * num_sms() ? 1 : (int)std::max<int64_t>(std::min(th / d.ny, d.nz), 1);
  g.words_x = ceil_div(d.nx, 32);
  const int64_t words = g.words_x * d.ny * d.nz, tiles = g.tiles_x * g.tiles_y * ceil_div(d.nz, (int64_t)g.slices);
  // bitmap segments: whole chunks of the numbering pass (kLThreads words of one or four a thread), kLSegments of them
  // at most (a segment's CTA sums the counts before it)
  static_assert(kLThreads == 1 << 8, "a segment holds whole chunks");
  int log_seg = ceil_div(words, kLThreads) <= 4 * num_sms() ? 8 : 10;
  while (ceil_div(words, 1ll << log_seg) > kLSegments) ++log_seg;
  const int64_t nseg = ceil_div(words, 1ll << log_seg);
  const size_t par_bytes = (sizeof(int32_t) * (size_t)n + 255) / 256 * 256;
  const size_t root_bytes = (sizeof(unsigned) * (size_t)words + 255) / 256 * 256;
  Scratch work;
  PG_TRY(work.alloc(par_bytes + root_bytes + sizeof(int32_t) * kLSegments + sizeof(int64_t), s));
  int32_t *par = work.as<int32_t>();
  unsigned *roots = reinterpret_cast<unsigned *>(work.as<char>() + par_bytes);
  int32_t *cnt = reinterpret_cast<int32_t *>(work.as<char>() + par_bytes + root_bytes);
  // the count goes straight to the host, where one waits for it (without one the call can be captured)
  HostSlot slot(count != nullptr);
  long long *device_total = reinterpret_cast<long long *>(cnt + kLSegments);
  long long *total = slot.word ? slot.word : device_total;
  int64_t *o = static_cast<int64_t *>(out.data);
  const T *src = static_cast<const T *>(in.data);
  PG_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (size_t)nseg, s), "clear label counts");
  // the forms that wait less for flat zones of few tiles and for columns of runs
  const bool full = g.slices > 1 || (FLAT && tiles <= 2 * num_sms()) || !(edges & E_L);
  if (full) k_label_tile<T, FLAT, true><<<(unsigned)tiles, kLThreads, 0, s>>>(src, par, roots, g);
  else k_label_tile<T, FLAT, false><<<(unsigned)tiles, kLThreads, 0, s>>>(src, par, roots, g);
  const int64_t n_rows = (edges & (E_U | E_UL | E_UR)) ? d.nz * (g.tiles_y - 1) * d.nx : 0;
  const int64_t n_cols = (edges & (E_L | E_UL | E_UR)) ? d.nz * d.ny * (g.tiles_x - 1) : 0;
  const int64_t n_z = (edges & E_Z) ? (d.nz - 1) * d.ny * d.nx : 0;
  const int64_t items = n_rows + n_cols + n_z, cap = (int64_t)num_sms() * 8;
  if (items > 0)
    k_label_border<T, FLAT><<<(unsigned)std::min<int64_t>(ceil_div(items, kLThreads), cap), kLThreads, 0, s>>>(
        src, par, g, n_rows, n_cols, n_z);
  if (full) k_label_flatten<4><<<(unsigned)ceil_div(4 * words, kLThreads), kLThreads, 0, s>>>(par, roots, cnt, g, words, log_seg);
  else k_label_flatten<1><<<(unsigned)ceil_div(words, kLThreads), kLThreads, 0, s>>>(par, roots, cnt, g, words, log_seg);
  if (log_seg < 10) k_label_number<1><<<(unsigned)nseg, kLThreads, 0, s>>>(par, roots, cnt, g, words, log_seg, total);
  else k_label_number<4><<<(unsigned)nseg, kLThreads, 0, s>>>(par, roots, cnt, g, words, log_seg, total);
  const unsigned rg = (unsigned)ceil_div(n, 4 * kLThreads);
  if (reinterpret_cast<uintptr_t>(o) % 16 == 0) k_label_resolve<true><<<rg, kLThreads, 0, s>>>(par, n, o);
  else k_label_resolve<false><<<rg, kLThreads, 0, s>>>(par, n, o);
  const pg_status launched = cuda_status(cudaGetLastError(), "labelling kernels launch");
  if (launched != PG_OK) {
    // the kernels that were launched may still write the word: it goes back to the pool after them
    if (total != device_total) (void)cudaStreamSynchronize(s);
    return launched;
  }
  if (count) {
    if (total == device_total)
      PG_CUDA_TRY(cudaMemcpyAsync(count, total, sizeof(int64_t), cudaMemcpyDeviceToHost, s), "label count copy");
    PG_CUDA_TRY(cudaStreamSynchronize(s), "label count synchronisation");
    if (total != device_total) *count = slot.value();
  }
  return PG_OK;
}

}  // namespace

pg_status launch_label(const pg_image &in, int se, const pg_image &out, bool flat, int64_t *count, cudaStream_t s) {
  unsigned up = 0;
  if (!upper_edges(se, &up))
    return fail(PG_ERR_UNSUPPORTED_SE, flat ? "t_label_flat_zonesDispatch unsupported nl_static on the GPU path"
                                            : "t_label_binaryDispatch unsupported nl_static on the GPU path");
  const Dims d = dims_of(in);
  const int64_t n = d.count();
  if (n > (int64_t)INT32_MAX) return fail(PG_ERR_INVALID_ARGUMENT, "labelling: image larger than 2^31 - 1 pixels");
  if (n == 0) {
    if (count) *count = 0;
    return PG_OK;
  }
  if (!flat && (in.ptype == PG_PTYPE_F32 || in.ptype == PG_PTYPE_F64))
    return fail(PG_ERR_UNSUPPORTED_PTYPE, "label_binary of a float image is not on the GPU path");
  PG_DISPATCH_PTYPE(in.ptype, T, {
    return flat ? label_t<T, true>(in, out, up, count, s) : label_t<T, false>(in, out, up, count, s);
  });
  return PG_OK;
}

cudaError_t label_status_word(void **p) { return cudaGetSymbolAddress(p, g_label_status); }

}  // namespace pg
