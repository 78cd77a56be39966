// recon3d_resident.cuh -- reconstruction of volumes (SECross3D) whose bricks all stay on the GPU from start to
// end: the 3D form of k_reconstruct_resident, included by recon.cu after it.
//
// A warp owns a brick of 32 x 8 x 8 voxels of 1 or 2 bytes (lane = x).  Pair (y, p) of its 32 registers holds
// voxels z = p (low half) and z = 7 - p (high half) of row y: the chains up and down z advance together in one
// 2x16-bit min/max, as the row pairs of the 2D tiles do.  A sweep set runs along z, along y (chains of whole
// registers), and, after a transpose through shared memory, along x (a lane two rows, columns c and 31 - c
// paired).  SECross3D has face neighbours only, so six faces are exchanged: a visit reads its neighbours' faces,
// sweeps, publishes the faces that changed and marks the bricks beside them.  States and the pending count are
// those of k_reconstruct_resident.
//
// Before, every brick was loaded, iterated and written by every launch, and the host read a flag back after
// every second one: 128 x 192 x 256 u8 h-maxima 12 launches of 33-60 us, 717 us a call; 163 us now,
// bound by the sweeps of the first visits (21 bricks per SM) and then by the chain of visits.
#pragma once

namespace pg {

// The mask pairs of a brick in shared memory: u8 pairs as two bytes.
template <typename T> struct MaskPair;
template <> struct MaskPair<uint8_t> {
  using Word = uint16_t;
  __device__ __forceinline__ static uint16_t put(uint32_t pair) { return (uint16_t)__byte_perm(pair, 0u, 0x4420); }
  __device__ __forceinline__ static uint32_t get(const uint16_t *p) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
    uint16_t r;
    asm volatile("ld.volatile.shared.u16 %0, [%1];" : "=h"(r) : "r"(addr));  // see lds_u32
    return __byte_perm((uint32_t)r, 0u, 0x4140);
  }
};
template <> struct MaskPair<uint16_t> {
  using Word = uint32_t;
  __device__ __forceinline__ static uint32_t put(uint32_t pair) { return pair; }
  __device__ __forceinline__ static uint32_t get(const uint32_t *p) { return lds_u32(p); }
};

template <typename T> struct Brick {
  static constexpr int TP = 32 + 4 / (int)sizeof(T);
  typename MaskPair<T>::Word mz[32 * 32];  // pair (y, p): [(4 y + p) * 32 + x]
  typename MaskPair<T>::Word mx[32 * 32];  // row set h, column pair c: [(16 h + c) * 32 + row % 32]
  T val[64 * TP];                          // rows 8 y + z
};
// faces in the exchange buffer: [y][x] planes z = 0 and 7, [z][x] planes y = 0 and 7, rows at x = 0 and 31
enum : int { F_ZM = 0, F_ZP = 256, F_YM = 512, F_YP = 768, F_XM = 1024, F_XP = 1088, F_SIZE = 1152 };
// warps per SM: what shared memory (227 KB) and a register budget of 80 leave room for
template <typename T> __host__ __device__ constexpr int brick_warps() { return sizeof(T) == 1 ? 24 : 18; }

// Sweep sets per visit: a set costs more than a halo here (128 x 192 x 256 u8: 1 set 163 us, 2 173, 4 201).
constexpr int kBrickSweeps = 1;

struct Vol {
  int D, H, W;
  int bz, by, bx;  // bricks
};

template <typename T> struct VolParams {
  Vol v;
  const T *ref, *marker;
  void *out;
  int bricks, init, mask_mode, epi, max_visits;
  T h;
  unsigned long long wait_ns;
  RCtl *ctl;
  ResCtl *res;
  unsigned *state;
  T *faces;
};

template <typename T, bool SUP>
__global__ void __launch_bounds__(brick_warps<T>() * 32, 1) k_r3_resident(const __grid_constant__ VolParams<T> P) {
  using OT = Op<T, SUP>;
  using MP = MaskPair<T>;
  constexpr int TP = Brick<T>::TP;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Brick<T> &s = reinterpret_cast<Brick<T> *>(s_dyn)[warp];
  RCtl *ctl = P.ctl;
  const T NEU = OT::neutral();
  auto OS = [](uint32_t a, uint32_t b) { return SUP ? u16x2_max(a, b) : u16x2_min(a, b); };
  auto OC = [](uint32_t a, uint32_t b) { return SUP ? u16x2_min(a, b) : u16x2_max(a, b); };
  const int t = (int)(blockIdx.x + gridDim.x * (unsigned)warp);  // bricks dealt over the SMs
  const bool have = t < P.bricks;
  const int tb = have ? t : 0, bx = tb % P.v.bx, by = tb / P.v.bx % P.v.by, bz = tb / P.v.bx / P.v.by;
  const int x = bx * 32 + lane, y0 = by * 8, z0 = bz * 8;
  T *mine = P.faces + (size_t)tb * F_SIZE;
  uint32_t V[32], end_x[2] = {0, 0};  // end_x: columns 0 and 31 of rows lane + 32 h
  // row r = 8 y + z of the brick: whether this lane's voxel is in the volume, and its index
  auto inside = [&](int r) { return x < P.v.W && y0 + r / 8 < P.v.H && z0 + r % 8 < P.v.D; };
  auto voxel = [&](int r) { return ((int64_t)(z0 + r % 8) * P.v.H + y0 + r / 8) * P.v.W + x; };
  auto from_rows = [&] {
#pragma unroll
    for (int y = 0; y < 8; ++y)
#pragma unroll
      for (int p = 0; p < 4; ++p)
        V[4 * y + p] = pk2(s.val[(8 * y + p) * TP + lane], s.val[(8 * y + 7 - p) * TP + lane]);
  };
  auto to_rows = [&] {  // V into s.val by rows
    __syncwarp();
#pragma unroll
    for (int y = 0; y < 8; ++y)
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        s.val[(8 * y + p) * TP + lane] = (T)V[4 * y + p];
        s.val[(8 * y + 7 - p) * TP + lane] = (T)(V[4 * y + p] >> 16);
      }
    __syncwarp();
  };

  if (have) {
    // effective mask by rows, then in both layouts
#pragma unroll 8
    for (int r = 0; r < 64; ++r) {
      T m = NEU;
      if (inside(r)) {
        const int64_t i = voxel(r);
        m = ldg(P.ref + i);
        if (P.init != INIT_SAT_CONST && P.mask_mode != MASK_PLAIN) {
          const T mk = ldg(P.marker + i);
          m = P.mask_mode == MASK_MAX_MARKER ? Op<T, true>::apply(mk, m) : Op<T, false>::apply(mk, m);
        }
      }
      s.val[r * TP + lane] = m;
    }
    __syncwarp();
    from_rows();
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      s.mz[k * 32 + lane] = MP::put(V[k]);
      const T *row = s.val + (lane + 32 * (k / 16)) * TP;
      s.mx[k * 32 + lane] = MP::put(pk2(row[k % 16], row[31 - k % 16]));
    }
    __syncwarp();
    // initial values
#pragma unroll 8
    for (int r = 0; r < 64; ++r) {
      T v = NEU;
      if (inside(r)) {
        const T m = s.val[r * TP + lane];
        v = P.init == INIT_SAT_CONST ? sat_shift<T, SUP>(m, P.h) : Op<T, !SUP>::apply(ldg(P.marker + voxel(r)), m);
      }
      s.val[r * TP + lane] = v;
    }
    __syncwarp();
    from_rows();
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      st_cg(mine + F_ZM + 32 * y + lane, (T)V[4 * y]);
      st_cg(mine + F_ZP + 32 * y + lane, (T)(V[4 * y] >> 16));
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      st_cg(mine + F_YM + 32 * p + lane, (T)V[p]);
      st_cg(mine + F_YM + 32 * (7 - p) + lane, (T)(V[p] >> 16));
      st_cg(mine + F_YP + 32 * p + lane, (T)V[28 + p]);
      st_cg(mine + F_YP + 32 * (7 - p) + lane, (T)(V[28 + p] >> 16));
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      end_x[h] = pk2(s.val[(lane + 32 * h) * TP], s.val[(lane + 32 * h) * TP + 31]);
      st_cg(mine + F_XM + 32 * h + lane, (T)end_x[h]);
      st_cg(mine + F_XP + 32 * h + lane, (T)(end_x[h] >> 16));
    }
    if (lane == 0) P.state[t] = RS_RUNNING;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.res->work = (unsigned)P.bricks;
    g_recon_rounds = 0;
  }
  if (!grid_barrier(ctl, P.wait_ns)) return;
  if (!have) return;

  // lane d < 6 looks after the neighbour in direction d = -z +z -y +y -x +x
  const bool has[6] = {bz > 0, bz + 1 < P.v.bz, by > 0, by + 1 < P.v.by, bx > 0, bx + 1 < P.v.bx};
  const int plane = P.v.bx * P.v.by;
  const int step[6] = {-plane, plane, -P.v.bx, P.v.bx, -1, 1};
  int nb = -1;
#pragma unroll
  for (int d = 0; d < 6; ++d)
    if (lane == d && has[d]) nb = t + step[d];
  int visits = 0;
  bool settled = false;  // at the local fixpoint of the last halo
  for (;;) {
    if (++visits > P.max_visits) {
      if (lane == 0) set_status(ctl, PG_ERR_NOT_CONVERGED);
      return;
    }
    // ---- halo: the six faces beside the brick
    uint32_t hz[8], hym[4], hyp[4], hx[2];
    {
      T zm[8], zp[8], ym[8], yp[8], xm[2], xp[2];
      const T *f = mine + lane;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        zm[k] = zp[k] = ym[k] = yp[k] = NEU;
        if (has[0]) zm[k] = ld_cg(f - (int64_t)plane * F_SIZE + F_ZP + 32 * k);
        if (has[1]) zp[k] = ld_cg(f + (int64_t)plane * F_SIZE + F_ZM + 32 * k);
        if (has[2]) ym[k] = ld_cg(f - (int64_t)P.v.bx * F_SIZE + F_YP + 32 * k);
        if (has[3]) yp[k] = ld_cg(f + (int64_t)P.v.bx * F_SIZE + F_YM + 32 * k);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        xm[h] = xp[h] = NEU;
        if (has[4]) xm[h] = ld_cg(f - F_SIZE + F_XP + 32 * h);
        if (has[5]) xp[h] = ld_cg(f + F_SIZE + F_XM + 32 * h);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) hz[k] = pk2(zm[k], zp[k]);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        hym[p] = pk2(ym[p], ym[7 - p]);
        hyp[p] = pk2(yp[p], yp[7 - p]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) hx[h] = pk2(xm[h], xp[h]);
    }
    // ---- sweep sets.  What changed on a face: d_z (low half z = 0, high half z = 7), d_ym, d_yp per lane = x; d_row
    // per lane = row (both row sets); d_x (low half x = 0, high half x = 31); d_any per lane = x.
    uint32_t d_z = 0, d_ym = 0, d_yp = 0, d_any = 0, d_row[2] = {0, 0}, d_x = 0;
    // A brick at its local fixpoint moves only if its new halo moves a voxel of a face: most wakes end here.
    bool move = !settled;
    if (settled) {
      auto pulled = [&](uint32_t v, uint32_t nbv, uint32_t m) { return OC(OS(v, nbv), m) ^ v; };
      uint32_t d = 0;
#pragma unroll
      for (int y = 0; y < 8; ++y) d |= pulled(V[4 * y], hz[y], MP::get(s.mz + 4 * y * 32 + lane));
#pragma unroll
      for (int p = 0; p < 4; ++p)
        d |= pulled(V[p], hym[p], MP::get(s.mz + p * 32 + lane)) | pulled(V[28 + p], hyp[p], MP::get(s.mz + (28 + p) * 32 + lane));
#pragma unroll
      for (int h = 0; h < 2; ++h) d |= pulled(end_x[h], hx[h], MP::get(s.mx + 16 * h * 32 + lane));
      move = __any_sync(0xffffffffu, d != 0);
    }
    for (int sweep = 0; move && sweep < kBrickSweeps; ++sweep) {
      settled = false;
      uint32_t ch = 0;
      auto update = [&](int y, int p, uint32_t nbv) {
        const int k = 4 * y + p;
        const uint32_t nv = OC(OS(V[k], nbv), MP::get(s.mz + k * 32 + lane)), d = nv ^ V[k];
        ch |= d;
        if (p == 0) d_z |= d;
        if (y == 0) d_ym |= d;
        if (y == 7) d_yp |= d;
        V[k] = nv;
      };
      // along z: pair p from pair p - 1 (p = 0: the faces), then pair 3 from itself swapped and back
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int y = 0; y < 8; ++y) update(y, p, p == 0 ? hz[y] : V[4 * y + p - 1]);
#pragma unroll
      for (int p = 3; p >= 0; --p)
#pragma unroll
        for (int y = 0; y < 8; ++y) update(y, p, p == 3 ? swap2(V[4 * y + 3]) : V[4 * y + p + 1]);
      // along y
#pragma unroll
      for (int y = 0; y < 8; ++y)
#pragma unroll
        for (int p = 0; p < 4; ++p) update(y, p, y == 0 ? hym[p] : V[4 * (y - 1) + p]);
#pragma unroll
      for (int y = 7; y >= 0; --y)
#pragma unroll
        for (int p = 0; p < 4; ++p) update(y, p, y == 7 ? hyp[p] : V[4 * (y + 1) + p]);
      d_any |= ch;
      // along x, lane = row: set h holds rows lane + 32 h, columns c and 31 - c paired
      to_rows();
      bool any_x = false;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        T *row = s.val + (lane + 32 * h) * TP;
        uint32_t Q[16], cx = 0;
#pragma unroll
        for (int c = 0; c < 16; ++c) Q[c] = pk2(row[c], row[31 - c]);
        auto step_x = [&](int c, uint32_t nbv) {
          const uint32_t nv = OC(OS(Q[c], nbv), MP::get(s.mx + (16 * h + c) * 32 + lane)), d = nv ^ Q[c];
          cx |= d;
          if (c == 0) d_x |= d;
          Q[c] = nv;
        };
#pragma unroll
        for (int c = 0; c < 16; ++c) step_x(c, c == 0 ? hx[h] : Q[c - 1]);
#pragma unroll
        for (int c = 15; c >= 0; --c) step_x(c, c == 15 ? swap2(Q[15]) : Q[c + 1]);
        d_row[h] |= cx;
        end_x[h] = Q[0];
        const bool any = __any_sync(0xffffffffu, cx != 0);
        any_x |= any;
        if (any) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            row[c] = (T)Q[c];
            row[31 - c] = (T)(Q[c] >> 16);
          }
        }
      }
      __syncwarp();
      from_rows();
      if (!any_x && !__any_sync(0xffffffffu, ch != 0)) {
        settled = true;
        break;
      }
    }
    // ---- the faces that changed (a row is 8 y + z: z = lane % 8, y = lane / 8 + 4 h)
    const uint32_t rows = d_row[0] | d_row[1];
    const unsigned edge_x = __ballot_sync(0xffffffffu, d_any != 0);
    const bool f_zm = __any_sync(0xffffffffu, (d_z & 0xffffu) != 0 || (rows != 0 && lane % 8 == 0));
    const bool f_zp = __any_sync(0xffffffffu, (d_z >> 16) != 0 || (rows != 0 && lane % 8 == 7));
    const bool f_ym = __any_sync(0xffffffffu, d_ym != 0 || (d_row[0] != 0 && lane < 8));
    const bool f_yp = __any_sync(0xffffffffu, d_yp != 0 || (d_row[1] != 0 && lane >= 24));
    const bool f_xm = __any_sync(0xffffffffu, (d_x & 0xffffu) != 0) || (edge_x & 1u);
    const bool f_xp = __any_sync(0xffffffffu, (d_x >> 16) != 0) || (edge_x >> 31);
    if (f_zm)
#pragma unroll
      for (int y = 0; y < 8; ++y) st_cg(mine + F_ZM + 32 * y + lane, (T)V[4 * y]);
    if (f_zp)
#pragma unroll
      for (int y = 0; y < 8; ++y) st_cg(mine + F_ZP + 32 * y + lane, (T)(V[4 * y] >> 16));
    if (f_ym)
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        st_cg(mine + F_YM + 32 * p + lane, (T)V[p]);
        st_cg(mine + F_YM + 32 * (7 - p) + lane, (T)(V[p] >> 16));
      }
    if (f_yp)
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        st_cg(mine + F_YP + 32 * p + lane, (T)V[28 + p]);
        st_cg(mine + F_YP + 32 * (7 - p) + lane, (T)(V[28 + p] >> 16));
      }
    if (f_xm)
#pragma unroll
      for (int h = 0; h < 2; ++h) st_cg(mine + F_XM + 32 * h + lane, (T)end_x[h]);
    if (f_xp)
#pragma unroll
      for (int h = 0; h < 2; ++h) st_cg(mine + F_XP + 32 * h + lane, (T)(end_x[h] >> 16));
    const unsigned faces = (f_zm ? 1u : 0u) | (f_zp ? 2u : 0u) | (f_ym ? 4u : 0u) | (f_yp ? 8u : 0u) | (f_xm ? 16u : 0u) |
                           (f_xp ? 32u : 0u);
    const int stop = resident_rest(P.res, ctl, P.state, t, nb, nb >= 0 && ((faces >> lane) & 1u), settled, P.wait_ns);
    if (stop == 2) return;
    if (stop == 1) break;
  }
  if (lane == 0) atomicMax(&g_recon_rounds, visits);

  // ---- result
  to_rows();
#pragma unroll 8
  for (int r = 0; r < 64; ++r) {
    if (!inside(r)) continue;
    const T v = s.val[r * TP + lane];
    const int64_t i = voxel(r);
    if (P.epi == EPI_NONE) {
      static_cast<T *>(P.out)[i] = v;
    } else {
      const T a = ldg(P.ref + i);
      if (P.epi == EPI_BINARY_SUP) static_cast<uint8_t *>(P.out)[i] = epi_binary<T, SUP>(a, v);
      else static_cast<T *>(P.out)[i] = Op<T, !SUP>::apply(v, a);
    }
  }
}

template <typename T, bool SUP>
static pg_status resident3d_t(const pg_image *marker, const pg_image &mask, const pg_image &out, const ReconRequest &rq,
                              const Vol &v, int bricks, cudaStream_t s) {
  static_assert(sizeof(Brick<T>) * brick_warps<T>() <= 227 * 1024, "an SM's bricks fit in shared memory");
  const size_t states = (4 * (size_t)bricks + 255) / 256 * 256, head = 256 + sizeof(ResCtl) + states;
  Scratch work;
  PG_TRY(work.alloc(head + sizeof(T) * F_SIZE * (size_t)bricks, s));
  PG_CUDA_TRY(cudaMemsetAsync(work.ptr, 0, head, s), "clear reconstruction work area");
  VolParams<T> P{};
  P.v = v;
  P.ref = static_cast<const T *>(mask.data);
  P.marker = marker ? static_cast<const T *>(marker->data) : nullptr;
  P.out = out.data;
  P.bricks = bricks;
  P.init = rq.init;
  P.mask_mode = rq.mask_mode;
  P.epi = rq.epi;
  P.max_visits = max_rounds_for(bricks);
  P.h = scalar_as<T>(rq.h);
  P.wait_ns = g_dbg_wait_ns.load();
  P.ctl = work.as<RCtl>();
  P.res = reinterpret_cast<ResCtl *>(work.as<char>() + 256);
  P.state = reinterpret_cast<unsigned *>(work.as<char>() + 256 + sizeof(ResCtl));
  P.faces = reinterpret_cast<T *>(work.as<char>() + head);
  const int grid = std::min(num_sms(), bricks), warps = (int)ceil_div(bricks, grid);
  static std::atomic<uint64_t> attr_devices{0};  // the opt-in shared-memory size, once per device
  int dev = 0;
  PG_CUDA_TRY(cudaGetDevice(&dev), "cudaGetDevice");
  const uint64_t bit = 1ull << (dev & 63);
  if (!(attr_devices.load() & bit)) {
    PG_CUDA_TRY(cudaFuncSetAttribute(k_r3_resident<T, SUP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(sizeof(Brick<T>) * brick_warps<T>())),
                "resident 3D reconstruction smem attribute");
    attr_devices.fetch_or(bit);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)warps * 32);
  cfg.dynamicSmemBytes = sizeof(Brick<T>) * (size_t)warps;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PG_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_r3_resident<T, SUP>, P), "cooperative 3D reconstruction launch");
  return PG_OK;
}

bool try_resident3d(const pg_image *marker, const pg_image &mask, const pg_image &out, const ReconRequest &rq, cudaStream_t s,
                    pg_status *st) {
  if (mask.ptype != PG_PTYPE_U8 && mask.ptype != PG_PTYPE_U16) return false;
  if (rq.init != INIT_SAT_CONST && !marker) return false;
  const Dims d = dims_of(mask);
  const int64_t bx = ceil_div(d.nx, 32), by = ceil_div(d.ny, 8), bz = ceil_div(d.nz, 8);
  const int64_t most = (int64_t)num_sms() * (mask.ptype == PG_PTYPE_U8 ? brick_warps<uint8_t>() : brick_warps<uint16_t>());
  if (d.count() == 0 || bx > most || by > most || bz > most || bx * by * bz > most) return false;
  const Vol v{(int)d.nz, (int)d.ny, (int)d.nx, (int)bz, (int)by, (int)bx};
  const int n = (int)(bx * by * bz);
  if (mask.ptype == PG_PTYPE_U8)
    *st = rq.dilate ? resident3d_t<uint8_t, true>(marker, mask, out, rq, v, n, s)
                    : resident3d_t<uint8_t, false>(marker, mask, out, rq, v, n, s);
  else
    *st = rq.dilate ? resident3d_t<uint16_t, true>(marker, mask, out, rq, v, n, s)
                    : resident3d_t<uint16_t, false>(marker, mask, out, rq, v, n, s);
  return true;
}

}  // namespace pg
