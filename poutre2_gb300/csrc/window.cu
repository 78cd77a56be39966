// window.cu -- erosion / dilation of 2D images by a (2hy+1) x (2hx+1) box or by a vertical / 45- / 135-degree
// segment of any half length, for 1-, 2- and 4-byte pixels, rows of any length and alignment, in one pass.
//
// Same result as line.cu / line_w.cu (X then Y van Herk passes, ero_dil_line_se_t.hpp:50-89, clipped
// windows; the diagonals are the runtime neighbour-list segments); the half lengths are run-time values.
// The window extremum is built from windows of fixed lengths (along rows powers of two, each from two of half
// the length): a handful of steps whatever the window, none of which needs its length at compile time, where
// a van Herk scan keeps a window of registers per thread.
//
// A CTA (8 warps) owns a tile of up to 120 32-bit words (E = 4 / sizeof(T) pixels each) x TH rows:
//   rows    -- a warp takes a row of 128 words (a lane 4 consecutive words).  The row starts hx pixels left
//              of the tile at any byte: aligned words are loaded and funnel-shifted.  Forward windows of
//              length 2hx + 1 are put together in registers along the binary expansion of the length; the
//              shifts are powers of two, inside a lane's words or whole lanes (shuffles).  u8 pixels are
//              kept as even / odd pixels on 16-bit lanes (two max.u16x2 per word; the packed 4 x 8-bit
//              instruction is an emulated sequence on this GPU).  The result goes to shared memory.
//   columns -- a thread walks up its word column and replaces each word by the window of 3 or 9 rows
//              (delay lines in registers, one shared load and store per word; three values meet in one
//              instruction); then
//   output  -- every output is the extremum of ceil((2hy+1) / 9) of those, and is shifted to the
//              alignment of its row in memory by one shuffle, so that stores are whole aligned words.
// A diagonal segment is a column of a sheared tile: row y of the tile starts lean * (y - y0) pixels further
// right, which the unaligned loads and stores absorb.
//
// Bound: the ALU pipe (min / max, shifts and byte permutes all issue there at half rate; 54 % busy at 2999 x
// 4001 u8, 21x21) and the waits of the 24 warps an image of that size gives an SM; the input is read from
// DRAM once, the halo from L2.  2999 x 4001 u8: 21x21 120 -> 26 us, 45-degree segment of 21 90 -> 19 us (pixel-
// wise van Herk in shared memory before: rows of no whole words); f32 4096^2 45 degrees of 21 104 -> 43 us.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "words.cuh"

namespace pg {
namespace {

constexpr int kWThreads = 256, kWWarps = kWThreads / 32;
constexpr int kWRow = 128;                       // words of a tile row
constexpr int kWOut = 4 * 31;                    // words the four warps of a column pass put out (lane 0 lends)
constexpr size_t kWSmemMax = 227 * 1024;

// A word as the operands of the min / max instructions: u8 words as two words whose 16-bit lanes hold the
// even / odd pixels in their high byte (the low byte only breaks ties), others as they are.
template <typename T, bool SUP> struct Acc {
  static constexpr bool B8 = sizeof(T) == 1;
  uint32_t a, b;
  __device__ __forceinline__ static uint32_t op16(uint32_t x, uint32_t y) { return wop<uint16_t, SUP>(x, y); }
  __device__ __forceinline__ static Acc of(uint32_t w) {
    if constexpr (B8) return Acc{w << 8, w};
    else return Acc{w, 0u};
  }
  __device__ __forceinline__ Acc with(const Acc &o) const {
    if constexpr (B8) return Acc{op16(a, o.a), op16(b, o.b)};
    else return Acc{wop<T, SUP>(a, o.a), 0u};
  }
  __device__ __forceinline__ uint32_t word() const {
    if constexpr (B8) return __byte_perm(a, b, 0x7351);
    else return a;
  }
};

// A lane's four words of a row in registers, as NR registers of two 16-bit lanes or one 32-bit pixel:
// u8: r[2j] = even, r[2j + 1] = odd pixels of word j (in the high bytes, as Acc); others: r[j] = word j.
template <typename T> struct RowRegs {
  static constexpr int NR = sizeof(T) == 1 ? 8 : 4;
  uint32_t r[NR];
  __device__ __forceinline__ static RowRegs of(const uint32_t (&w)[4]) {
    RowRegs o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (sizeof(T) == 1) {
        o.r[2 * j] = w[j] << 8;
        o.r[2 * j + 1] = w[j];
      } else {
        o.r[j] = w[j];
      }
    }
    return o;
  }
  __device__ __forceinline__ uint4 words() const {
    if constexpr (sizeof(T) == 1)
      return make_uint4(__byte_perm(r[0], r[1], 0x7351), __byte_perm(r[2], r[3], 0x7351),
                        __byte_perm(r[4], r[5], 0x7351), __byte_perm(r[6], r[7], 0x7351));
    else
      return make_uint4(r[0], r[1], r[2], r[3]);
  }
};

__device__ __forceinline__ uint32_t from_lane(uint32_t v, int ahead) { return __shfl_down_sync(0xffffffffu, v, ahead); }

// the row moved left by S pixels (a power of two): pixel i takes pixel i + S.  The last lanes take
// anything; they feed no output.
template <typename T, int S> __device__ __forceinline__ RowRegs<T> ahead(const RowRegs<T> &x) {
  constexpr int E = 4 / (int)sizeof(T), LP = 4 * E, NR = RowRegs<T>::NR;  // pixels per word, per lane
  RowRegs<T> o;
  if constexpr (S >= LP) {
#pragma unroll
    for (int j = 0; j < NR; ++j) o.r[j] = from_lane(x.r[j], S / LP);
  } else if constexpr (S >= E) {  // whole words
    constexpr int D = S / E * (NR / 4);
#pragma unroll
    for (int j = 0; j < NR; ++j) o.r[j] = j + D < NR ? x.r[j + D] : from_lane(x.r[j + D - NR], 1);
  } else if constexpr (sizeof(T) == 2) {  // S = 1
    const uint32_t n = from_lane(x.r[0], 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) o.r[j] = __funnelshift_r(x.r[j], j < 3 ? x.r[j + 1] : n, 16);
  } else if constexpr (S == 1) {  // u8: the odd pixels, and the even ones from the next on
    const uint32_t n = from_lane(x.r[0], 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o.r[2 * j] = x.r[2 * j + 1];
      o.r[2 * j + 1] = __funnelshift_r(x.r[2 * j], j < 3 ? x.r[2 * j + 2] : n, 16);
    }
  } else {  // u8, S = 2
    const uint32_t n0 = from_lane(x.r[0], 1), n1 = from_lane(x.r[1], 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o.r[2 * j] = __funnelshift_r(x.r[2 * j], j < 3 ? x.r[2 * j + 2] : n0, 16);
      o.r[2 * j + 1] = __funnelshift_r(x.r[2 * j + 1], j < 3 ? x.r[2 * j + 3] : n1, 16);
    }
  }
  return o;
}
template <typename T, bool SUP> __device__ __forceinline__ RowRegs<T> both(const RowRegs<T> &x, const RowRegs<T> &y) {
  RowRegs<T> o;
#pragma unroll
  for (int j = 0; j < RowRegs<T>::NR; ++j)
    o.r[j] = sizeof(T) == 1 ? wop<uint16_t, SUP>(x.r[j], y.r[j]) : wop<T, SUP>(x.r[j], y.r[j]);
  return o;
}

// forward windows of w pixels (1 <= w < 2^7), along w's bits: m holds windows of 2^j, res those of the bits
// so far (w odd: it starts as the pixels themselves; w even: it is set at w's lowest bit)
template <typename T, bool SUP, int J>
__device__ __forceinline__ void row_steps(RowRegs<T> &m, RowRegs<T> &res, int w) {
  if (w >> J) {  // uniform; m: windows of 2^(J-1) -> 2^J
    m = both<T, SUP>(m, ahead<T, 1 << (J - 1)>(m));
    if ((w >> J) & 1) res = (w & ((1 << J) - 1)) ? both<T, SUP>(m, ahead<T, 1 << J>(res)) : m;
    if constexpr (J < 6) row_steps<T, SUP, J + 1>(m, res, w);
  }
}

struct WindowGeom {
  int64_t H, W;
  int hx;          // half width
  int hy;          // half height
  int lean;        // pixels a tile row starts further right than the row above: -1, 0, 1
  int th;          // output rows of a tile, a multiple of 8
  int half;        // half the rows of the tile's array in shared memory, a multiple of 6
  int vw;          // output words of a tile row
  int64_t u_first; // first pixel of tile column 0 at the tile's first output row
  int64_t tiles_x, tiles_y;
  double work;     // 64-row tiles of a 3-row window per SM that this costs
};

// Columns, in place: word of row i <- op over rows [i, i + N), N = 3 or 9 (the min / max of three values is
// one instruction).  Group [ga, ga + half) of the 2 * half rows of the tile's array, walking up (half a
// multiple of 6); the N - 1 rows below the first group prime its delay lines before any is overwritten.
// Rows past the tile's last only reach windows no output uses.
template <typename T, bool SUP, int N>
__device__ __forceinline__ void column_windows(uint32_t *col, int ga, int half) {
  using A = Acc<T, SUP>;
  constexpr int B = 6;  // steps per unrolled turn: every delay line's length divides it
  const A neu = A::of(splat<T>(Op<T, SUP>::neutral()));
  A d1[2] = {neu, neu}, d3[6] = {neu, neu, neu, neu, neu, neu};
  auto step = [&](A x, int i) -> A {
    A m = x.with(d1[0]).with(d1[1]);  // rows r .. r + 2
    d1[i % 2] = x;
    if constexpr (N == 9) {
      const A t = m.with(d3[i % 6]).with(d3[(i + 3) % 6]);  // the windows 6 and 3 rows below
      d3[i % 6] = m;
      m = t;
    }
    return m;
  };
  if (ga == 0) {
#pragma unroll
    for (int i = 0; i < N - 1; ++i) {
      const int r = half + N - 2 - i;
      step(r < 2 * half ? A::of(col[r * kWRow]) : neu, i % B);
    }
  }
  __syncthreads();
  for (int r0 = ga + half - B; r0 >= ga; r0 -= B) {
    uint32_t *q = col + r0 * kWRow, x[B];
#pragma unroll
    for (int i = 0; i < B; ++i) x[i] = q[(B - 1 - i) * kWRow];
#pragma unroll
    for (int i = 0; i < B; ++i) q[(B - 1 - i) * kWRow] = step(A::of(x[i]), (i + N - 1) % B).word();
  }
}

// Four words from aligned address p on, `step` bytes apart, of a row that may reach beyond the image's bytes
// [base, end): the bytes of a word across an end come one by one.
__device__ __noinline__ uint4 edge_words(uintptr_t p, int step, uintptr_t base, uintptr_t end) {
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uintptr_t pw = p + (uintptr_t)(step * j);
    w[j] = 0u;
    if (pw >= base && pw + 4 <= end) {
      w[j] = __ldg(reinterpret_cast<const uint32_t *>(pw));
    } else {
      for (int b = 0; b < 4; ++b)
        if (pw + b >= base && pw + b < end)
          w[j] |= (uint32_t)*reinterpret_cast<const unsigned char *>(pw + b) << (8 * b);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Stores a tile's output words, lane by lane word column c (c = -1 and lane 0 only lend): with its row's
// alignment word c covers the pixels from c * E - (pixels past an aligned word) on, so that every word is
// stored whole but at the image's sides.
template <typename T> struct TileStore {
  static constexpr int S = (int)sizeof(T), E = 4 / S;
  int64_t W, u0;
  int lean, c;
  bool inner, mine;
  __device__ __forceinline__ TileStore(int64_t W_, int64_t u0_, int lean_, int th, int vw, int c_)
      : W(W_), u0(u0_), lean(lean_), c(c_) {
    const int64_t x_end = u0 + (int64_t)lean * (th - 1);
    inner = min(u0, x_end) >= E && max(u0, x_end) + vw * E <= W;
    mine = (threadIdx.x & 31) != 0 && c < vw;
  }
  // word w of tile row y, whose pixel u0 + lean * y lies at byte address a; called by the whole warp
  __device__ __forceinline__ void put(uintptr_t a, int y, uint32_t w) const {
    const unsigned mis = S < 4 ? (unsigned)(a & 3u) : 0u;  // bytes past an aligned word
    if (mis) w = __funnelshift_l(__shfl_up_sync(0xffffffffu, w, 1), w, mis * 8u);
    if (!mine) return;
    T *dst = reinterpret_cast<T *>((a & ~(uintptr_t)3) + 4 * (intptr_t)c);
    if (inner) {
      *reinterpret_cast<uint32_t *>(dst) = w;
    } else {
      const int64_t x = u0 + (int64_t)lean * y + c * E - (int)mis / S;  // the word's first pixel
      if (x >= 0 && x + E <= W) {
        *reinterpret_cast<uint32_t *>(dst) = w;
      } else if (S < 4 && x + E > 0 && x < W) {
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (x + e >= 0 && x + e < W) dst[e] = (T)(w >> (8 * S * e));
      }
    }
  }
};

// Rows [0, rows) of a tile: row r starts at pixel x_top + lean * r of image row y_top + r; its words go to
// s_w[r][..] as forward windows of wlen pixels, those outside the image neutral.  Two rows at a time per warp,
// so that the loads of both are in flight.
// Lane l holds words 4l .. 4l + 3 of a row, where the windows' shifts are cheap; PLAIN (wlen == 1, nothing to
// shift) words l, l + 32, l + 64 and l + 96, whose loads and stores are one 128-byte line each at any alignment
// (3000 x 3500 f32, 45 degrees, 41 pixels: 37 -> 34 us a pass).
template <typename T, bool SUP, bool PLAIN>
__device__ __forceinline__ void window_rows_as(const T *in, int64_t H, int64_t W, int64_t y_top, int64_t x_top, int lean,
                                               int rows, int wlen, uint32_t *s_w) {
  constexpr int S = (int)sizeof(T), E = 4 / S;
  constexpr int LW = PLAIN ? 1 : 4, JW = PLAIN ? 32 : 1;  // word of (lane l, j): LW * l + JW * j
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t NEU = splat<T>(Op<T, SUP>::neutral());
  const intptr_t pitch = (intptr_t)(W + lean) * S;  // bytes from a tile row to the next
  // tile rows [r_lo, r_hi) are rows of the image
  const int r_lo = (int)min(max((int64_t)0, -y_top), (int64_t)rows), r_hi = (int)min((int64_t)rows, H - y_top);
  const int64_t x_bot = x_top + (int64_t)lean * (rows - 1);
  const uintptr_t a_top = reinterpret_cast<uintptr_t>(in) + (uintptr_t)((y_top * W + x_top) * S);
  uintptr_t a = a_top + warp * pitch;
  // some row holds pixels left / right of the image
  const bool clipped = min(x_top, x_bot) < 0 || max(x_top, x_bot) + kWRow * E > W;
  const uintptr_t base = reinterpret_cast<uintptr_t>(in), end = base + (uintptr_t)(H * W) * S;
  // every row of words lies in the image's buffer
  const bool safe = ((a_top + r_lo * pitch) & ~(uintptr_t)3) >= base && a_top + (r_hi - 1) * pitch + kWRow * 4 <= end;
  for (int r0 = warp; r0 < rows; r0 += 2 * kWWarps, a += 2 * kWWarps * pitch) {
    uint32_t w[2][4];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = r0 + q * kWWarps;
      const uintptr_t aq = a + q * kWWarps * pitch, seg = aq & ~(uintptr_t)3;
      if (r < r_lo || r >= r_hi) continue;
      if (safe || (seg >= base && seg + kWRow * 4 <= end)) {
        const uintptr_t p = seg + 4u * LW * lane;  // this lane's words
        if (!PLAIN && (aq & 12u) == 0) {
          const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
          w[q][0] = v.x; w[q][1] = v.y; w[q][2] = v.z; w[q][3] = v.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) w[q][j] = __ldg(reinterpret_cast<const uint32_t *>(p) + JW * j);
        }
      } else {
        const uint4 v = edge_words(seg + 4u * LW * lane, 4 * JW, base, end);
        w[q][0] = v.x; w[q][1] = v.y; w[q][2] = v.z; w[q][3] = v.w;
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = r0 + q * kWWarps;
      if (r >= rows) break;
      uint32_t *row = s_w + r * kWRow + LW * lane;
      auto store = [&](const uint4 &o) {
        if constexpr (PLAIN) {
          row[0] = o.x;
          row[JW] = o.y;
          row[2 * JW] = o.z;
          row[3 * JW] = o.w;
        } else {
          *reinterpret_cast<uint4 *>(row) = o;
        }
      };
      if (r < r_lo || r >= r_hi) {
        store(make_uint4(NEU, NEU, NEU, NEU));
        continue;
      }
      const unsigned sh = (unsigned)((a + q * kWWarps * pitch) & 3u) * 8u;
      if (S < 4 && sh) {
        // the row's last word lacks its upper pixels: no output of the tile needs them (vw)
        uint32_t n[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if constexpr (PLAIN) {
            n[j] = from_lane(w[q][j], 1);
            if (j < 3) {
              const uint32_t first = __shfl_sync(0xffffffffu, w[q][j + 1], 0);
              if (lane == 31) n[j] = first;
            }
          } else {
            n[j] = j < 3 ? w[q][j + 1] : from_lane(w[q][0], 1);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) w[q][j] = __funnelshift_r(w[q][j], n[j], sh);
      }
      if (clipped) {
        // pixels [lo, hi) of the row lie in the image
        const int64_t x = x_top + (int64_t)lean * r;
        const int lo = (int)min(max(-x, (int64_t)0), (int64_t)kWRow * E), hi = (int)min(max(W - x, (int64_t)0), (int64_t)kWRow * E);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int px = (LW * lane + JW * j) * E;
          const int l = min(max(lo - px, 0), E), k = min(max(hi - px, 0), E);  // of this word
          const uint32_t in_m = (uint32_t)(((1ull << (8 * S * k)) - 1ull) & ~((1ull << (8 * S * l)) - 1ull));
          w[q][j] = (w[q][j] & in_m) | (NEU & ~in_m);
        }
      }
      uint4 o = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
      if constexpr (!PLAIN) {
        RowRegs<T> m = RowRegs<T>::of(w[q]), res = m;
        row_steps<T, SUP, 1>(m, res, wlen);
        o = res.words();
      }
      store(o);
    }
  }
}
template <typename T, bool SUP>
__device__ __forceinline__ void window_rows(const T *in, int64_t H, int64_t W, int64_t y_top, int64_t x_top, int lean,
                                            int rows, int wlen, uint32_t *s_w) {
  if (wlen == 1) window_rows_as<T, SUP, true>(in, H, W, y_top, x_top, lean, rows, wlen, s_w);
  else window_rows_as<T, SUP, false>(in, H, W, y_top, x_top, lean, rows, wlen, s_w);
}

template <typename T, bool SUP>
__global__ void __launch_bounds__(kWThreads) k_window(const T *__restrict__ in, T *__restrict__ out, WindowGeom g) {
  constexpr int S = (int)sizeof(T), E = 4 / S;
  extern __shared__ __align__(16) uint32_t s_w[];  // [2 * half][kWRow]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t u0 = g.u_first + (int64_t)blockIdx.x * g.vw * E;  // the tile's first pixel in its first output row
  const int64_t y0 = (int64_t)blockIdx.y * g.th;
  const int rows = g.th + 2 * g.hy, half = g.half;
  const intptr_t pitch = (intptr_t)(g.W + g.lean) * S;  // bytes from a tile row to the next

  // ---- rows: from one word left of the tile, for the stores' shift
  window_rows<T, SUP>(in, g.H, g.W, y0 - g.hy, u0 - E - g.hx - (int64_t)g.lean * g.hy, g.lean, rows, 2 * g.hx + 1, s_w);
  __syncthreads();

  // ---- columns: four warps side by side, two groups of rows
  const int h = 2 * g.hy + 1;
  int n = 1;  // window length left in shared memory
  if (h >= 5) {
    uint32_t *mine = s_w + (threadIdx.x & (kWRow - 1));
    const int ga = (threadIdx.x >> 7) * half;
    if (h < 9) { column_windows<T, SUP, 3>(mine, ga, half); n = 3; }
    else { column_windows<T, SUP, 9>(mine, ga, half); n = 9; }
    __syncthreads();
  }
  // ---- output: th / 2 rows per group (a multiple of 4)
  using A = Acc<T, SUP>;
  // Word column c of the tile lies at array column c + 1; with its row's alignment it covers the pixels from
  // c * E - (pixels past an aligned word) on, so every word is stored whole but at the image's sides.
  const int c = (warp & 3) * 31 + lane - 1;  // lane 0 only lends its word to lane 1
  const int gh = g.th / 2, ya = (warp >> 2) * gh;
  const int yb = (int)min((int64_t)(ya + gh), g.H - y0);
  const TileStore<T> st(g.W, u0, g.lean, g.th, g.vw, c);
  const uint32_t *q = s_w + c + 1 + ya * kWRow;
  uintptr_t a = reinterpret_cast<uintptr_t>(out) + (uintptr_t)(((y0 + ya) * g.W + u0 + (int64_t)g.lean * ya) * S);
  constexpr int U = 4;
  for (int y = ya; y < yb; y += U, q += U * kWRow, a += U * pitch) {
    A v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) v[k] = A::of(q[k * kWRow]);
    if (h > n) {
      const uint32_t *qt = q + n * kWRow, *ql = q + (h - n) * kWRow;
      for (; qt + n * kWRow < ql; qt += 2 * n * kWRow)  // two windows at a time: one instruction takes both
#pragma unroll
        for (int k = 0; k < U; ++k) v[k] = v[k].with(A::of(qt[k * kWRow])).with(A::of(qt[(n + k) * kWRow]));
      if (qt < ql)
#pragma unroll
        for (int k = 0; k < U; ++k) v[k] = v[k].with(A::of(qt[k * kWRow])).with(A::of(ql[k * kWRow]));
      else
#pragma unroll
        for (int k = 0; k < U; ++k) v[k] = v[k].with(A::of(ql[k * kWRow]));
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (y + k >= yb) break;  // uniform
      st.put(a + k * pitch, y + k, v[k].word());
    }
  }
}

WindowGeom window_geom(const pg_image &in, const pg_image &out, int64_t hy, int64_t hx, int lean) {
  const int E = 4 / elem_size(in.ptype);
  const Dims d = dims_of(in);
  WindowGeom g{};
  g.H = d.ny;
  g.W = d.nx;
  // clipped windows reach no further than the image: on one column (row) they are the pixels themselves, with no
  // neutral value beside them to stand in for an infinity
  g.hx = (int)std::min(hx, d.nx - 1);
  g.hy = (int)std::min(hy, d.ny - 1);
  g.lean = lean;
  // valid words of a row (windows are forward), in whole 32-byte sectors: a misaligned load loses a word, the
  // stores' shift needs one left of the tile
  g.vw = std::min((kWRow * E - 2 * g.hx) / E - 2, kWOut) & ~7;
  // pixels a tile row has to reach beyond the image: the shear's, and a misaligned last word's
  const bool mis = E > 1 && (g.lean != 0 || (g.W % E) != 0 || reinterpret_cast<uintptr_t>(out.data) % 4 != 0);
  // 64 rows per tile, fewer (but no less than the halo's 2 hy) where the image would not give every SM four
  // CTAs: 2999 x 4001 u8 3x3 20.5 -> 18.9 us with 32 rows, 21x21 28.7 with both
  g.th = 64;
  const int64_t sms = num_sms();
  auto tiles_x = [&]() { return ceil_div(g.W + (g.lean ? g.th - 1 : 0) + (mis ? E - 1 : 0), (int64_t)g.vw * E); };
  while (g.th > 16 && g.th / 2 >= 2 * g.hy && tiles_x() * ceil_div(g.H, g.th) < 4 * sms) g.th /= 2;
  if (tiles_x() * ceil_div(g.H, g.th) < sms) g.th /= 2;  // 64, 32, 16 or 8: a group's rows are a multiple of 4
  g.tiles_x = tiles_x();
  g.tiles_y = ceil_div(g.H, g.th);
  g.work = (double)(g.tiles_x * g.tiles_y) * (g.th + 2 * g.hy) / (66. * (double)sms);
  g.u_first = g.lean > 0 ? -(int64_t)(g.th - 1) : 0;
  g.half = (g.th + 2 * g.hy + 11) / 12 * 6;
  return g;
}

template <typename T, bool SUP>
pg_status window_t(const pg_image &in, const pg_image &out, const WindowGeom &g, cudaStream_t s) {
  const size_t smem = (size_t)(2 * g.half) * kWRow * 4;
  static std::atomic<uint64_t> attr_devices{0};
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  const uint64_t bit = 1ull << (dev & 63);
  if (!(attr_devices.load() & bit)) {
    PG_CUDA_TRY(cudaFuncSetAttribute(k_window<T, SUP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWSmemMax),
                "window kernel smem attribute");
    attr_devices.fetch_or(bit);
  }
  const dim3 grid((unsigned)g.tiles_x, (unsigned)g.tiles_y);
  k_window<T, SUP><<<grid, kWThreads, smem, s>>>(static_cast<const T *>(in.data), static_cast<T *>(out.data), g);
  return cuda_status(cudaGetLastError(), "window kernel launch");
}

// ------------------------------------------------------------------ neighbour lists
// Erosion / dilation by an offset list (ero_dil_runtime_nl_se_t.hpp:129-193, clipped; like the gather kernel
// the extremum always holds the neutral value).  The list is cut into chords, runs of offsets along a row; the
// chords of one length, first column and slice form a group, whose row windows are formed once and serve
// all its rows: a disk of radius 7 has 149 offsets, 15 chords and 5 groups.  Per group the tile's rows go to
// shared memory as windows of the chord's length, moved by its first column (the loads take any alignment),
// and every thread adds the chords' rows to its R outputs, kept in registers.
// Bound: the ALU pipe, 4-5 instructions per chord and word of outputs plus a row pass per group.  2048^2 u8,
// radius 7: 905 us (149 bounds-checked loads per pixel, small_se.cu) -> 31 us; radius 2 f32 121 -> 25 us.
struct ChordGroup {
  int x0;                  // first column of the chords
  short dz, len;           // slice, pixels
  short dy_min, dy_max;    // rows
  short first, count;      // in ChordTable::dy
};
constexpr int kMaxGroups = 64, kMaxChords = 512, kMaxSpan = 96;
struct ChordTable {
  int n;
  ChordGroup g[kMaxGroups];
  short dy[kMaxChords];
};

template <typename T, bool SUP, int R>
__global__ void __launch_bounds__(kWThreads, sizeof(T) == 1 ? 3 : 4) k_chords(const T *__restrict__ in, T *__restrict__ out, int64_t D, int64_t H,
                                                      int64_t W, int vw, const __grid_constant__ ChordTable t) {
  constexpr int S = (int)sizeof(T), E = 4 / S, TH = 2 * R;
  extern __shared__ __align__(16) uint32_t s_w[];  // [TH + span of dy][kWRow]
  using A = Acc<T, SUP>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t u0 = (int64_t)blockIdx.x * vw * E, y0 = (int64_t)blockIdx.y * TH, z = blockIdx.z;
  const int c = (warp & 3) * 31 + lane - 1, ya = (warp >> 2) * R;  // as in k_window
  A acc[R];
#pragma unroll
  for (int i = 0; i < R; ++i) acc[i] = A::of(splat<T>(Op<T, SUP>::neutral()));
  for (int k = 0; k < t.n; ++k) {
    const ChordGroup &g = t.g[k];
    if (z + g.dz < 0 || z + g.dz >= D) continue;  // uniform
    __syncthreads();                              // the last group's windows have been read
    window_rows<T, SUP>(in + (z + g.dz) * H * W, H, W, y0 + g.dy_min, u0 - E + g.x0, 0, TH + g.dy_max - g.dy_min, g.len, s_w);
    __syncthreads();
    const uint32_t *q = s_w + c + 1 + (ya - g.dy_min) * kWRow;
    int j = g.first;
    const int end = g.first + g.count;
    for (; j + 1 < end; j += 2) {  // two chords at a time: one instruction takes both
      const uint32_t *p0 = q + t.dy[j] * kWRow, *p1 = q + t.dy[j + 1] * kWRow;
#pragma unroll
      for (int i = 0; i < R; ++i) acc[i] = acc[i].with(A::of(p0[i * kWRow])).with(A::of(p1[i * kWRow]));
    }
    if (j < end) {
      const uint32_t *p0 = q + t.dy[j] * kWRow;
#pragma unroll
      for (int i = 0; i < R; ++i) acc[i] = acc[i].with(A::of(p0[i * kWRow]));
    }
  }
  const TileStore<T> st(W, u0, 0, TH, vw, c);
  const intptr_t pitch = (intptr_t)W * S;
  const uintptr_t a = reinterpret_cast<uintptr_t>(out) + (uintptr_t)(((z * H + y0 + ya) * W + u0) * S);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (y0 + ya + i >= H) break;  // uniform
    st.put(a + i * pitch, ya + i, acc[i].word());
  }
}

// How an image is cut for k_chords.
struct ChordTiles {
  int vw;            // output words of a tile row, as in window_t
  int tiles_x;
  int rows;          // R, the rows a thread holds: half a tile's
  int64_t tiles;
};
// R is what three (u8, two registers a row) or four CTAs per SM leave room for (2048^2 u8, radius 5: 12 rows 29 us,
// 16 rows 35, 8 rows 34; f32: 16 rows 49, 12 rows 51, 8 rows 60); 4 where the image would not give every SM a tile.
constexpr int chord_rows(int es) { return es == 1 ? 12 : 16; }
ChordTiles chord_tiles(const pg_image &in, const pg_image &out, int max_len) {
  const int es = elem_size(in.ptype), E = 4 / es;
  const Dims d = dims_of(in);
  ChordTiles c{};
  c.vw = std::min((kWRow * E - (max_len - 1)) / E - 2, kWOut) & ~7;
  const bool mis = E > 1 && (d.nx % E != 0 || reinterpret_cast<uintptr_t>(out.data) % 4 != 0);
  c.tiles_x = (int)ceil_div(d.nx + (mis ? E - 1 : 0), (int64_t)c.vw * E);
  c.rows = chord_rows(es);
  if (c.tiles_x * ceil_div(d.ny, 2 * c.rows) * d.nz < num_sms()) c.rows = 4;
  c.tiles = c.tiles_x * ceil_div(d.ny, 2 * c.rows) * d.nz;
  return c;
}

// Whether the chords beat the gather of small_se.cu on this image, by the times of both in nanoseconds (fitted to
// 3200 lists and images, 6 % and 20 % off: the slower one by more than 8 % is taken on 64 of them).  A gather costs its loads; the groups of a tile go one after the other,
// which is what a small image waits for (61 offsets of two diagonals on 64^2 u8: 48 us, gathered 15), and a tile
// that an image fills only in part costs as much as a full one (a disk of 5 offsets on 200000 x 2 u8: 144 us, 11).
bool chords_win(const ChordTable &t, const ChordTiles &c, const Dims &d, int es, int n) {
  const double pixels = (double)d.count(), th = 2 * c.rows;
  double wait = 4200., rows = 0., adds = 0.;
  for (int k = 0; k < t.n; ++k) {
    const double r = th + t.g[k].dy_max - t.g[k].dy_min;  // rows of windows a tile makes, 16 at a time
    wait += 550. + 650. * (double)ceil_div((int64_t)r, 2 * kWWarps);
    rows += r;
    adds += t.g[k].count * th;
  }
  const double chords = wait + (double)c.tiles * (0.12 * rows + (es == 1 ? 0.028 : 0.014) * adds + 4.);
  const double gather = 6500. + 105. * n + 0.001 * (n + 4) * pixels;
  return chords < gather;
}

template <typename T, bool SUP, int R>
pg_status chords_r(const pg_image &in, const pg_image &out, const ChordTable &t, const ChordTiles &c, int span,
                   cudaStream_t s) {
  const Dims d = dims_of(in);
  static std::atomic<uint64_t> attr_devices{0};
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  const uint64_t bit = 1ull << (dev & 63);
  if (!(attr_devices.load() & bit)) {
    PG_CUDA_TRY(cudaFuncSetAttribute(k_chords<T, SUP, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWSmemMax),
                "neighbour-list kernel smem attribute");
    attr_devices.fetch_or(bit);
  }
  const dim3 grid((unsigned)c.tiles_x, (unsigned)ceil_div(d.ny, 2 * R), (unsigned)d.nz);
  k_chords<T, SUP, R><<<grid, kWThreads, (size_t)(2 * R + span) * kWRow * 4, s>>>(
      static_cast<const T *>(in.data), static_cast<T *>(out.data), d.nz, d.ny, d.nx, c.vw, t);
  return cuda_status(cudaGetLastError(), "neighbour-list kernel launch");
}

template <typename T, bool SUP>
pg_status chords_t(const pg_image &in, const pg_image &out, const ChordTable &t, const ChordTiles &c, int span, cudaStream_t s) {
  constexpr int R = chord_rows((int)sizeof(T));
  return c.rows == R ? chords_r<T, SUP, R>(in, out, t, c, span, s) : chords_r<T, SUP, 4>(in, out, t, c, span, s);
}

// The list as chords; false where it has too many, or where they are so short that gathering the offsets one
// by one costs less (per 32-bit word of outputs: 14 instructions per offset and pixel, against 50 per group and
// 5 per chord).
bool make_chords(const int32_t *offsets, int n, int rank, int pixels_per_word, int max_len, ChordTable &t, int &span,
                 int &longest) {
  // offsets and chords as one sortable word each (fields below 2^15, biased): dz, dy, dx and dz, x0, len, dy
  constexpr int kFar = 16383, kBias = 16384;
  uint64_t key[4096], chord[kMaxChords];
  if (n > 4096) return false;
  for (int k = 0; k < n; ++k) {
    uint64_t v = 0;
    for (int r = 0; r < 3; ++r) {
      const int o = r < 3 - rank ? 0 : offsets[k * rank + r - (3 - rank)];
      if (o < -kFar || o > kFar) return false;
      v = (v << 16) | (uint64_t)(o + kBias);
    }
    key[k] = v;
  }
  std::sort(key, key + n);
  n = (int)(std::unique(key, key + n) - key);
  int nc = 0;
  for (int i = 0, j; i < n; i = j) {
    // a run of a row: consecutive words (a column's neighbour never reaches the next field)
    for (j = i + 1; j < n && key[j] == key[j - 1] + 1 && j - i < max_len;) ++j;
    if (nc == kMaxChords) return false;
    const uint64_t dz = key[i] >> 32, dy = (key[i] >> 16) & 0xffff, dx = key[i] & 0xffff;
    chord[nc++] = (dz << 48) | (dx << 32) | ((uint64_t)(j - i) << 16) | dy;
  }
  std::sort(chord, chord + nc);
  auto row = [&](int i) { return (int)(chord[i] & 0xffff) - kBias; };
  t.n = 0;
  span = 0;
  longest = 1;
  for (int i = 0, j; i < nc; i = j) {
    if (t.n == kMaxGroups) return false;
    ChordGroup &g = t.g[t.n++];
    for (j = i; j < nc && (chord[j] >> 16) == (chord[i] >> 16) && row(j) - row(i) <= kMaxSpan; ++j) t.dy[j] = (short)row(j);
    g.dz = (short)((int)(chord[i] >> 48) - kBias);
    g.x0 = (int)((chord[i] >> 32) & 0xffff) - kBias;
    g.len = (short)((chord[i] >> 16) & 0xffff);
    g.dy_min = (short)row(i);
    g.dy_max = (short)row(j - 1);
    g.first = (short)i;
    g.count = (short)(j - i);
    span = std::max(span, (int)g.dy_max - g.dy_min);
    longest = std::max(longest, (int)g.len);
  }
  return 50 * t.n + 5 * nc <= 14 * n * pixels_per_word;
}

// A tile costs the same however little of its rows the image fills: where narrow images give the GPU more work than
// it has room for at once, the kernels that work in columns or narrow tiles are faster (us, window / other):
//   rectangles on whole-word rows of 1- and 2-byte pixels, and repeated 3x3 squares: u8 100000 x 8 5x5 58 / 13, 30000 x 64
//     21x21 31 / 24, u16 168033 x 5 5x5 78 / 15, but u8 1239 x 48 5x7 7 / 17, u16 11063 x 96 3x51 11 / 22;
//   vertical segments: whole-word rows up to 640 bytes (f32 k = 9 30068 x 144 25 / 21, 81041 x 128 54 / 35, 11734 x 338
//     17 / 18); ragged ones of a few pixels (u8 48833 x 21 k = 39 52 / 36, but 8461 x 18 k = 6 13 / 29);
//   45 / 135 degrees: u16 18835 x 6 k = 5 17 / 13;
//   one column: a row segment is a copy (u8 194408 x 1 115 / 4); others u8 182485 x 1 5 x 117 129 / 62.
bool window_narrow(const WindowGeom &g, int64_t hy, int64_t hx, int es, bool words) {
  const int64_t row = g.W * es;
  const double work = g.work;
  if (g.W == 1) return (g.hy == 0 && g.hx == 0) || work >= 4.;
  if (g.lean != 0) return words && es <= 2 && ((row <= 16 && work >= 3.) || (row <= 48 && work >= 8.));
  if (hx == 0) return words ? (row <= 640 && work >= 3.) || (row <= 48 && work >= 1.) : row <= 24 && work >= 5.;
  const bool squares = hy == hx && hy <= (es <= 2 ? 4 : 2);
  if (squares || (hx == 1 && hy <= 1)) return row <= 256 && work >= 4.;
  if (hy == 0 || es > 2 || !words) return false;
  return (row <= 256 && work >= 4.5) || (es == 1 && row <= 32 && work >= 1.2);
}

}  // namespace

bool window_ok(const pg_image &in, const pg_image &out, int64_t hy, int64_t hx, int lean) {
  const int es = elem_size(in.ptype);
  if (in.rank != 2 || (es != 1 && es != 2 && es != 4)) return false;
  if (hy < 0 || hx < 0 || hy > 63 || (hy == 0 && hx == 0) || (lean != 0 && hx != 0)) return false;
  // a row window needs its length below 2^7 and leaves at least half of a tile row's pixels
  if (hx > 63 || 4 * hx > kWRow * 4 / es) return false;
  const Dims d = dims_of(in);
  if (d.ny < 16 || d.nx < 1 || d.ny > (1 << 19) || d.nx > (1 << 30)) return false;
  const uintptr_t pixel = (uintptr_t)es - 1;
  if (((reinterpret_cast<uintptr_t>(in.data) | reinterpret_cast<uintptr_t>(out.data)) & pixel) != 0) return false;
  return !window_narrow(window_geom(in, out, hy, hx, lean), hy, hx, es, rows_aligned(in, out, 4));
}

bool try_window(const pg_image &in, const pg_image &out, int64_t hy, int64_t hx, int lean, bool dilate, cudaStream_t s,
                pg_status *st) {
  if (!window_ok(in, out, hy, hx, lean)) return false;
  const WindowGeom g = window_geom(in, out, hy, hx, lean);
  switch (in.ptype) {
    case PG_PTYPE_U8: *st = dilate ? window_t<uint8_t, true>(in, out, g, s) : window_t<uint8_t, false>(in, out, g, s); return true;
    case PG_PTYPE_U16: *st = dilate ? window_t<uint16_t, true>(in, out, g, s) : window_t<uint16_t, false>(in, out, g, s); return true;
    case PG_PTYPE_I32: *st = dilate ? window_t<int32_t, true>(in, out, g, s) : window_t<int32_t, false>(in, out, g, s); return true;
    case PG_PTYPE_F32: *st = dilate ? window_t<float, true>(in, out, g, s) : window_t<float, false>(in, out, g, s); return true;
    default: return false;
  }
}

static bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &status) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return status != cudaStreamCaptureStatusNone;
}

bool try_chords(const pg_image &in, const pg_image &out, const int32_t *offsets, int n, bool dilate, cudaStream_t s,
                pg_status *st) {
  const int es = elem_size(in.ptype);
  if (in.rank < 2 || (es != 1 && es != 2 && es != 4)) return false;
  const Dims d = dims_of(in);
  if (d.ny < 16 || d.nx < 1 || d.ny > (1 << 18) || d.nx > (1 << 30) || d.nz > 65535) return false;
  const uintptr_t pixel = (uintptr_t)es - 1;
  if ((reinterpret_cast<uintptr_t>(in.data) | reinterpret_cast<uintptr_t>(out.data)) & pixel) return false;
  ChordTable t;
  int span = 0, longest = 1;
  if (!make_chords(offsets, n, in.rank, 4 / es, es == 4 ? 32 : 64, t, span, longest)) return false;
  const ChordTiles c = chord_tiles(in, out, longest);
  // While the stream captures, the chords whatever they cost: their list goes by value into the graph, where a copy of
  // the gather's would read this call's host memory at every launch of the graph.
  if (!chords_win(t, c, d, es, n) && !capturing(s)) return false;
  switch (in.ptype) {
    case PG_PTYPE_U8: *st = dilate ? chords_t<uint8_t, true>(in, out, t, c, span, s) : chords_t<uint8_t, false>(in, out, t, c, span, s); return true;
    case PG_PTYPE_U16: *st = dilate ? chords_t<uint16_t, true>(in, out, t, c, span, s) : chords_t<uint16_t, false>(in, out, t, c, span, s); return true;
    case PG_PTYPE_I32: *st = dilate ? chords_t<int32_t, true>(in, out, t, c, span, s) : chords_t<int32_t, false>(in, out, t, c, span, s); return true;
    case PG_PTYPE_F32: *st = dilate ? chords_t<float, true>(in, out, t, c, span, s) : chords_t<float, false>(in, out, t, c, span, s); return true;
    default: return false;
  }
}

}  // namespace pg
