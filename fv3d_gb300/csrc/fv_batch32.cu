// fv_batch32.cu -- dispatch of the FP32-mixed 2-D kernels: the warp-marched
// form (fv_march32.cuh), which every mixed 2-D group takes, and the
// shared-memory block form below, which a forced schedule (FV3D_TILE with 32-
// or 64-wide blocks) selects; plus the mixed form's CFL reduction and its
// (hi, lo) pair conversions.  Built with
// fast-math (FP32 division / sqrt approximations, FMA contraction); the
// error-free pair arithmetic of fv_tile32.cuh is written with adds and _rn
// intrinsics, which contraction leaves alone.
#include "fv_march32.cuh"

namespace fv {

namespace {

// Work-item shapes (cells along a x rows along b) the autotuner starts
// from, each with the kernel that marches it: strip segments marched in
// blocks of 16 or 8 rows (cells per thread in the update: 32x16 -> 2,
// 64x16 -> 4, 32x8 -> 1, 64x8 -> 2), with the viscous fluxes fused per cell
// or split into a per-face pass (VF).  The rows of an item are a run-time
// value (BatchInst::tz), so shapes of one kernel differ only in their
// starting rows.
// march: the warp-marched form (0: the block form).
struct MixedKernel {
  int tx, block_rows, vface, march;
};
// Block rows of the two block heights (cells per thread in the update: 2 and
// 1 for 32-wide blocks).
#ifndef FV_MIXED_BR_A
#define FV_MIXED_BR_A 16
#endif
#ifndef FV_MIXED_BR_B
#define FV_MIXED_BR_B 8
#endif
constexpr int kBrA = FV_MIXED_BR_A, kBrB = FV_MIXED_BR_B;
constexpr MixedKernel kKernels32[] = {{32, kBrA, 0, 0}, {64, kBrA, 0, 0}, {32, kBrB, 0, 0}, {64, kBrB, 0, 0},
                                      {32, kBrA, 1, 0}, {64, kBrA, 1, 0}, {kMarchWidth, 0, 0, 1}};
constexpr TileShape kShapes32[] = {{32, 2 * kBrA}, {64, kBrA}, {32, kBrA},     {64, 2 * kBrA},        {32, 2 * kBrB},
                                   {64, kBrB},     {32, 2 * kBrA}, {64, kBrA}, {kMarchWidth, 32}};
constexpr int kKernelOf32[] = {0, 1, 0, 1, 2, 3, 4, 5, 6};
constexpr int kNumShapes32 = sizeof(kShapes32) / sizeof(kShapes32[0]);

// Copies the descriptor of the problem holding work item t to s_inst and
// returns its index (binary search over the first items).
__device__ __forceinline__ int fetch_inst32(const BatchInst* __restrict__ insts, int ninst, int t,
                                            BatchInst* s_inst) {
  int lo = 0, hi = ninst - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (insts[mid].tile0 <= t) lo = mid;
    else hi = mid - 1;
  }
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(insts + lo);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(s_inst);
  for (int w = threadIdx.x; w < (int)(sizeof(BatchInst) / 8); w += blockDim.x) dst[w] = src[w];
  return lo;
}

#if FV_MIXED_MIN_CTAS > 0
#define FV_MIXED_BOUNDS __launch_bounds__(kTileThreads, FV_MIXED_MIN_CTAS)
#else
#define FV_MIXED_BOUNDS __launch_bounds__(kTileThreads)
#endif

// One work item t (a strip segment of problem I) of one stage.  active / dt:
// the problem's step in flight; slot_next / err: its CFL maximum slot for the
// next step and its error flag (stages that end a step).  Every thread of
// the CTA calls it; s_inst holds I.
template <int PLANE, bool WACT, class TL, bool VF>
__device__ __forceinline__ void stage_item32(const BatchInst& I, int t, int kind, int flip, bool active, double dt_step,
                                             unsigned long long* slot_next, int* err, float* smem,
                                             unsigned long long* s_red) {
  const int lt = t - I.tile0;
  const int bx = lt % I.tiles_x, by = lt / I.tiles_x;
  MixedFields M;
  float2* src[5];
  float2* dst[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    M.un[v] = reinterpret_cast<float2*>(I.A.f[v]);
    M.us[v] = reinterpret_cast<float*>(I.B.f[v]);
    float2* a = reinterpret_cast<float2*>(I.A.f[v]);
    float2* b = reinterpret_cast<float2*>(I.B.f[v]);
    src[v] = (kind == STAGE_EULER && flip) ? b : a;
    dst[v] = (kind == STAGE_EULER && !flip) ? b : a;
  }
  const int x0 = bx * TL::TX, ya = by * I.tz;  // tz: rows per work item
  const int yb = ya + I.tz < I.G.nb ? ya + I.tz : I.G.nb;
  if (!active) {
    if (kind == STAGE_EULER) pass_on32<WACT, TL::TX>(I.G, src, dst, x0, ya, yb, threadIdx.x);
    return;
  }
  const float dt = (float)dt_step;  // the one FP64 -> FP32 conversion per item
  float red = 0.0f;
  bool bad = false;
  stage_segment32<PLANE, WACT, TL, VF>(I.G, M, src, dst, I.rs, kind, dt, x0, ya, yb, smem, red, bad);
  if (kind != STAGE_RK_1) {
    if (bad) atomicOr(err, 1);
    block_max_atomic((unsigned long long)__double_as_longlong((double)red), slot_next, s_red);
  }
}

template <int PLANE, bool WACT, class TL, bool VF>
__global__ void FV_MIXED_BOUNDS
batch_stage32(const BatchInst* __restrict__ insts, int ninst, int ntiles, unsigned* queue, int kind, int flip) {
  extern __shared__ float smem_f[];
  __shared__ unsigned long long s_red[kTileThreads / 32];
  __shared__ BatchInst s_inst;
  __shared__ int s_tile;
  pdl_wait();
  for (;;) {
    __syncthreads();  // the previous tile is finished with s_tile, s_inst and smem
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(queue, 1u);
    __syncthreads();
    const int t = s_tile;
    if (t >= ntiles) {
      pdl_trigger();  // no work left for this CTA
      break;
    }
    fetch_inst32(insts, ninst, t, &s_inst);
    __syncthreads();
    StepCtrl* ctrl = s_inst.ctrl;
    stage_item32<PLANE, WACT, TL, VF>(s_inst, t, kind, flip, ctrl->active != 0, ctrl->dt_cur,
                                  &ctrl->slot[ctrl->parity ^ 1], &ctrl->err, smem_f, s_red);
  }
}

template <int K>
using BlockOf32 = Tile<kKernels32[K].tx, kKernels32[K].block_rows>;

template <int PLANE, bool WACT, int K>
auto kernel_for() {
  return batch_stage32<PLANE, WACT, BlockOf32<K>, kKernels32[K].vface != 0>;
}

template <int K>
size_t smem_for(bool wact, bool tc) {
  if (kKernels32[K].vface && wact) return TileSmem<float, 5, BlockOf32<K>>::bytes_vface();
  return wact ? TileSmem<float, 5, BlockOf32<K>>::bytes(tc) : TileSmem<float, 4, BlockOf32<K>>::bytes(tc);
}

typedef void (*BatchKernel)(const BatchInst*, int, int, unsigned*, int, int);

MarchKernel march_kernel(int plane, bool wact, int kind, bool one) {
  return plane == PLANE_XY ? march_kernel_xy(wact, kind, one) : march_kernel_xz(wact, kind, one);
}

MarchMultiKernel march_multi_kernel(int plane, bool wact, bool one) {
  return plane == PLANE_XY ? march_multi_kernel_xy(wact, one) : march_multi_kernel_xz(wact, one);
}

// A parameter every launch passes: the descriptor of a one-problem group.
const BatchInst& one_or_empty(const BatchInst* one) {
  static const BatchInst empty{};
  return one ? *one : empty;
}

template <int PLANE, bool WACT>
BatchKernel pick(int shape) {
  switch (kKernelOf32[shape]) {
    case 0: return kernel_for<PLANE, WACT, 0>();
    case 1: return kernel_for<PLANE, WACT, 1>();
    case 2: return kernel_for<PLANE, WACT, 2>();
    case 3: return kernel_for<PLANE, WACT, 3>();
    case 4: return kernel_for<PLANE, WACT, 4>();
    default: return kernel_for<PLANE, WACT, 5>();
  }
}

BatchKernel pick_any(int plane, bool wact, int shape) {
  if (plane == PLANE_XY) return wact ? pick<PLANE_XY, true>(shape) : pick<PLANE_XY, false>(shape);
  return wact ? pick<PLANE_XZ, true>(shape) : pick<PLANE_XZ, false>(shape);
}

size_t smem_any(int shape, bool wact, bool tc) {
  switch (kKernelOf32[shape]) {
    case 0: return smem_for<0>(wact, tc);
    case 1: return smem_for<1>(wact, tc);
    case 2: return smem_for<2>(wact, tc);
    case 3: return smem_for<3>(wact, tc);
    case 4: return smem_for<4>(wact, tc);
    default: return smem_for<5>(wact, tc);
  }
}

cudaError_t prepare(int plane, bool wact, int shape) {
  static bool done[2][2][kNumShapes32] = {};
  bool& flag = done[plane == PLANE_XY ? 0 : 1][wact ? 1 : 0][shape];
  if (flag) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(pick_any(plane, wact, shape), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem_any(shape, wact, true));
  if (e == cudaSuccess) flag = true;
  return e;
}

int grid_for(long long n, int block) {
  long long b = (n + block - 1) / block;
  if (b > 152 * 16) b = 152 * 16;
  return b < 1 ? 1 : (int)b;
}

// CFL maximum of a state held as (hi, lo) pairs.
template <int PLANE, bool WACT>
__global__ void __launch_bounds__(256) reduce2d_mixed(const Grid G, const Fields pairs, StepCtrl* ctrl, int slot) {
  __shared__ unsigned long long s_red[8];
  float red = 0.0f;
  bool bad = false;
  const long long n = (long long)G.na * G.rows;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(c / G.na), x = (int)(c - (long long)y * G.na);
    const long long o = (long long)y * G.pitch + x;
    float2 w[5];
#pragma unroll
    for (int v = 0; v < 5; ++v)
      w[v] = (v == 3 && !WACT) ? make_float2(0.0f, 0.0f) : reinterpret_cast<const float2*>(pairs.f[v])[o];
    const float inv = inv_dt_hyp32<PLANE, WACT>(w, G);
    bad |= !(inv <= 3.0e38f);
    red = fmaxf(red, inv);
  }
  if (bad) atomicOr(&ctrl->err, 1);
  block_max_atomic((unsigned long long)__double_as_longlong((double)red), &ctrl->slot[slot], s_red);
}

// FP64 values -> (hi, lo) float pairs: hi = RN32(d), lo = RN32(d - hi).
__global__ void pairs_from_double(const Grid G, const Fields src, const Fields dst) {
  const long long n = (long long)G.na * G.rows;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(c / G.na), x = (int)(c - (long long)y * G.na);
    const long long o = (long long)y * G.pitch + x;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double d = src.f[v][o];
      const float hi = __double2float_rn(d);
      const float lo = __double2float_rn(d - (double)hi);
      reinterpret_cast<float2*>(dst.f[v])[o] = make_float2(hi, lo);
    }
  }
}

// (hi, lo) pairs -> FP64 values hi + lo (exact).
__global__ void double_from_pairs(const Grid G, const Fields src, const Fields dst) {
  const long long n = (long long)G.na * G.rows;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(c / G.na), x = (int)(c - (long long)y * G.na);
    const long long o = (long long)y * G.pitch + x;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float2 w = reinterpret_cast<const float2*>(src.f[v])[o];
      dst.f[v][o] = (double)w.x + (double)w.y;
    }
  }
}

// primToCons (States.h:20-31) of a caller's unpadded primitive arrays (a null
// field reads as zero), in FP64, split into pairs as pairs_from_double.
template <int PLANE>
__global__ void __launch_bounds__(256) prim_to_pairs_from(const Grid G, const Fields src, const Fields dst) {
  const long long n = (long long)G.na * G.rows;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(c / G.na), x = (int)(c - (long long)y * G.na);
    const long long o = (long long)y * G.pitch + x;
    double q[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) q[v] = src.f[v] ? src.f[v][c] : 0.0;
    const double r = q[0];
    const double ma = __dmul_rn(r, q[1]), mb = __dmul_rn(r, q[2]), mc = __dmul_rn(r, q[3]);
    const double mx = ma, my = PLANE == PLANE_XY ? mb : mc, mz = PLANE == PLANE_XY ? mc : mb;
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(mx, mx), __dmul_rn(my, my)), __dmul_rn(mz, mz));
    const double E = __dadd_rn(__ddiv_rn(__dmul_rn(0.5, s), r), __ddiv_rn(q[4], G.gm1));
    const double u[5] = {r, ma, mb, mc, E};
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float hi = __double2float_rn(u[v]);
      const float lo = __double2float_rn(u[v] - (double)hi);
      reinterpret_cast<float2*>(dst.f[v])[o] = make_float2(hi, lo);
    }
  }
}

// consToPrim (States.h:34-45) of pairs, in FP64, into a caller's unpadded
// arrays (a null one is skipped).
template <int PLANE, bool WACT>
__global__ void __launch_bounds__(256) pairs_to_prim_to(const Grid G, const Fields pairs, const Fields dst) {
  const long long n = (long long)G.na * G.rows;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(c / G.na), x = (int)(c - (long long)y * G.na);
    const long long o = (long long)y * G.pitch + x;
    double u[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float2 w = (WACT || v != 3) ? reinterpret_cast<const float2*>(pairs.f[v])[o] : make_float2(0.0f, 0.0f);
      u[v] = (double)w.x + (double)w.y;
    }
    const double r = u[0];
    const double va = __ddiv_rn(u[1], r), vb = __ddiv_rn(u[2], r), vc = WACT ? __ddiv_rn(u[3], r) : 0.0;
    const double vx = va, vy = PLANE == PLANE_XY ? vb : vc, vz = PLANE == PLANE_XY ? vc : vb;
    const double s = __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz));
    const double Ek = __dmul_rn(__dmul_rn(0.5, r), s);
    const double q[5] = {r, va, vb, vc, __dmul_rn(__dsub_rn(u[4], Ek), G.gm1)};
#pragma unroll
    for (int v = 0; v < 5; ++v)
      if (dst.f[v]) dst.f[v][c] = q[v];
  }
}

}  // namespace

int batch_tile_shapes32(const TileShape** shapes) {
  *shapes = kShapes32;
  return kNumShapes32;
}

int batch_shape_kernel32(int shape, int* block_rows, int* vface) {
  if (shape < 0 || shape >= kNumShapes32) return -1;
  const MixedKernel& k = kKernels32[kKernelOf32[shape]];
  if (block_rows) *block_rows = k.block_rows;
  if (vface) *vface = k.vface;
  return kKernelOf32[shape];
}

bool batch_shape_marched32(int shape) {
  return shape >= 0 && shape < kNumShapes32 && kKernels32[kKernelOf32[shape]].march;
}

int batch_items_per_cta32(int shape) { return batch_shape_marched32(shape) ? kMarchWarps : 1; }

int batch_stage_occupancy32(int plane, bool wact, int shape, bool tc, int kind,
                            bool one) {
  if (batch_shape_marched32(shape)) {
    int nb = 0;
    const MarchKernel k = march_kernel(plane, wact, kind, one);
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kMarchThreads, 0) == cudaSuccess ? nb : 0;
  }
  if (shape < 0 || shape >= kNumShapes32 || prepare(plane, wact, shape) != cudaSuccess) return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, pick_any(plane, wact, shape), kTileThreads,
                                                    smem_any(shape, wact, tc)) != cudaSuccess)
    return 0;
  return nb;
}

cudaError_t launch_batch_stage32(int plane, bool wact, int shape, const BatchInst* insts, int ninst, int ntiles,
                                 unsigned* queue, int kind, int flip, int grid, bool tc, cudaStream_t st,
                                 const BatchInst* one) {
  if (shape < 0 || shape >= kNumShapes32) return cudaErrorInvalidValue;
  if (batch_shape_marched32(shape)) {
    // With a warp for each item the queue is passed over: the atomics of all
    // warps on its counter took some 10 % of an Euler step (us a step of 100^2
    // PCM 5.8 -> 5.0, 512^2 11.9 -> 10.2, 16 of 64^2 9.5 -> 8.6).
    if (ntiles <= grid * kMarchWarps) queue = nullptr;
    const cudaError_t e = launch_pdl(march_kernel(plane, wact, kind, one != nullptr), dim3(grid), dim3(kMarchThreads),
                                     0, st, insts, ninst, ntiles, queue, flip, one_or_empty(one));
    return e != cudaSuccess ? e : cudaGetLastError();
  }
  cudaError_t e = prepare(plane, wact, shape);
  if (e != cudaSuccess) return e;
  e = launch_pdl(pick_any(plane, wact, shape), dim3(grid), dim3(kTileThreads), smem_any(shape, wact, tc), st, insts,
                 ninst, ntiles, queue, kind, flip);
  return e != cudaSuccess ? e : cudaGetLastError();
}

int batch_multi_problems32() { return kMultiMaxProblems; }

int batch_multi_occupancy32(int plane, bool wact, int shape, bool one) {
  if (!batch_shape_marched32(shape)) return 0;
  int nb = 0;
  const MarchMultiKernel k = march_multi_kernel(plane, wact, one);
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kMarchThreads, 0) == cudaSuccess ? nb : 0;
}

cudaError_t launch_batch_multi32(int plane, bool wact, int shape, const BatchInst* insts, int ninst, int ntiles,
                                 int nsteps, int mode_override, GridBarrier gb, int grid, cudaStream_t st,
                                 const BatchInst* one) {
  if (!batch_shape_marched32(shape) || ninst > kMultiMaxProblems) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kMarchThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // every CTA resident: the grid barriers need it
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, march_multi_kernel(plane, wact, one != nullptr), insts, ninst, ntiles,
                                           nsteps, mode_override, gb, one_or_empty(one));
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_reduce2d_mixed(const Grid& G, bool wact, Fields pairs, StepCtrl* ctrl, int slot,
                                  cudaStream_t st) {
  const int grid = grid_for((long long)G.na * G.rows, 256);
  if (G.plane == PLANE_XY) {
    if (wact) reduce2d_mixed<PLANE_XY, true><<<grid, 256, 0, st>>>(G, pairs, ctrl, slot);
    else reduce2d_mixed<PLANE_XY, false><<<grid, 256, 0, st>>>(G, pairs, ctrl, slot);
  } else {
    if (wact) reduce2d_mixed<PLANE_XZ, true><<<grid, 256, 0, st>>>(G, pairs, ctrl, slot);
    else reduce2d_mixed<PLANE_XZ, false><<<grid, 256, 0, st>>>(G, pairs, ctrl, slot);
  }
  return cudaGetLastError();
}

cudaError_t launch_pairs_from_double(const Grid& G, Fields src, Fields dst_pairs, cudaStream_t st) {
  pairs_from_double<<<grid_for((long long)G.na * G.rows, 256), 256, 0, st>>>(G, src, dst_pairs);
  return cudaGetLastError();
}

cudaError_t launch_prim_to_pairs_from(const Grid& G, Fields src, Fields dst_pairs, cudaStream_t st) {
  const int grid = grid_for((long long)G.na * G.rows, 128);
  if (G.plane == PLANE_XY) prim_to_pairs_from<PLANE_XY><<<grid, 128, 0, st>>>(G, src, dst_pairs);
  else prim_to_pairs_from<PLANE_XZ><<<grid, 128, 0, st>>>(G, src, dst_pairs);
  return cudaGetLastError();
}

cudaError_t launch_pairs_to_prim_to(const Grid& G, bool wact, Fields src_pairs, Fields dst, cudaStream_t st) {
  const int grid = grid_for((long long)G.na * G.rows, 128);
  if (G.plane == PLANE_XY) {
    if (wact) pairs_to_prim_to<PLANE_XY, true><<<grid, 128, 0, st>>>(G, src_pairs, dst);
    else pairs_to_prim_to<PLANE_XY, false><<<grid, 128, 0, st>>>(G, src_pairs, dst);
  } else {
    if (wact) pairs_to_prim_to<PLANE_XZ, true><<<grid, 128, 0, st>>>(G, src_pairs, dst);
    else pairs_to_prim_to<PLANE_XZ, false><<<grid, 128, 0, st>>>(G, src_pairs, dst);
  }
  return cudaGetLastError();
}

cudaError_t launch_double_from_pairs(const Grid& G, Fields src_pairs, Fields dst, cudaStream_t st) {
  double_from_pairs<<<grid_for((long long)G.na * G.rows, 256), 256, 0, st>>>(G, src_pairs, dst);
  return cudaGetLastError();
}

}  // namespace fv
