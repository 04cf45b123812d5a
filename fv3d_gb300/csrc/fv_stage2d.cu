// fv_stage2d.cu -- the FP64 fused stage kernel of one 2-D problem: 32-wide
// strips of cells marched in blocks of 32x16 cells (stage_strip64 in
// fv_tile64.cuh, compiled without FMA contraction, so it rounds exactly like
// the reference).  The strip rows are split evenly over as many CTAs as the
// GPU holds at once, so every SM gets the same FP64 work.
#include "fv_tile64.cuh"
#include <algorithm>
#include <cmath>
#include <cudaTypedefs.h>  // PFN_cuTensorMapEncodeTiled

namespace fv {

namespace {

using SingleTile = Tile<kTileX, kTileY>;

// Dynamic shared memory is over-allocated by this much and aligned up, so
// that tensor copies land on 128-byte boundaries.
constexpr size_t kSmemAlign = 128;

template <int PLANE, int RS, int KIND, bool WACT>
__global__ void __launch_bounds__(kTileThreads, WACT ? FV_FP64_MIN_CTAS_W : FV_FP64_MIN_CTAS)
stage2d_fp64(const __grid_constant__ Grid grid, const Fields uin, const Fields u0, const Fields uout, StepCtrl* __restrict__ ctrl,
             const Fields hout, int width, long long units, const __grid_constant__ TmaState tin, int use_tma, const Fields qin,
             const Fields qout, const __grid_constant__ TmaState tq, int use_tq) {
  extern __shared__ __align__(128) unsigned char smem_bytes[];
  __shared__ unsigned long long s_red[kTileThreads / 32];
  __shared__ __align__(8) unsigned long long s_mbar;
  __shared__ Grid s_grid;
  const Grid& G = s_grid;
  param_to_shared(grid, s_grid);
  opaque64_init();
  const unsigned sa = smem_u32(smem_bytes);
  double* smem = reinterpret_cast<double*>(smem_bytes + (((sa + kSmemAlign - 1) & ~(unsigned)(kSmemAlign - 1)) - sa));
  pdl_wait();
  if (use_tma || use_tq) {
    if (threadIdx.x == 0) {
      mbar_init(&s_mbar, 1);
      fence_mbar_init();
    }
  }
  __syncthreads();
  cell_div_init(G);
  __syncthreads();
  // the primitive copy of uin, when the last stage that wrote uin left one
  const bool prims = qin.f[0] != nullptr && ctrl->q_valid != 0;
  const Fields* qi = prims ? &qin : nullptr;
  const Fields* qo = qout.f[0] ? &qout : nullptr;
  const TmaState* tp = prims ? (use_tq ? &tq : nullptr) : (use_tma ? &tin : nullptr);
  const Fields* ho = hout.f[0] ? &hout : nullptr;
  const long long ub = units * blockIdx.x / gridDim.x, ue = units * (blockIdx.x + 1) / gridDim.x;
  stage_strip64<PLANE, WACT, SingleTile>(G, uin, u0, uout, ctrl, RS, KIND, width, ub, ue, smem, s_red, ho, tp,
                                         &s_mbar, qi, qo);
  pdl_trigger();
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      n = 1;
  }
  return n;
}

// The split of a plane into strips of `width` columns whose rows (units) are
// shared out evenly over `ctas` CTAs.
struct Strips {
  int width;
  long long units, ctas;
};

// The width and CTA count with the least estimated time of the busiest SM.
// Large grids take full strips on every CTA the GPU holds at once: the fewest
// faces solved twice.  On small grids that left SMs idle (a 64^2 grid made 32
// CTAs of 32 x 4 cells): narrower strips and fewer rows per CTA spread the
// FP64 work, which bounds an SM, over all of them.  The estimate counts FP64
// warp operations per phase (a warp with idle lanes costs a whole one) for the
// faces, conversions and cell updates of a CTA and divides the SM's sum by the
// share of the pipe its CTAs keep busy between their barriers: 60 % for one,
// 95 % for two against three (1024^2: 1,330, 850 and 813 us a step).
// On grids of less than a block of rows per CTA the latency of one segment is
// the step: a CTA whose rows end one strip and begin the next takes twice as
// long, so a whole number of CTAs per strip is tried first, and kept unless all
// there is room for are estimated faster (96x64 49.7 -> 31.2 us a step, 100^2
// 51.3 -> 32.5, 160^2 58.9 -> 40.6, 90x700 113 -> 102, x-z 64x192 with viscosity
// 86.7 -> 52.9; 200^2, 256^2 and larger choose as they did).
// On planes of less than half a block of rows a CTA's rows can span many strips,
// one started after the other, which a share of the rows alone does not show:
// they are counted, and one CTA per strip is tried too, more than there is room
// for at once (PLM RK2 9001x2 113 -> 40 us a step, 15000x5 181 -> 102, 4000x3 74
// -> 35, 60000x4 334 -> 306; from 8 rows on it gains and loses: 30000x8 265 ->
// 242, with conduction and viscosity 514 -> 534, 40000x12 441 -> 478).
Strips split_strips(const Grid& G, int rs, bool wact, int resident) {
  const int sms = sm_count();
  const bool visc = wact && G.visc;
  const double face = (rs == 0 ? 110 : 75) + (wact ? 12 : 0) + (visc ? 30 : 0);
  const double cell = 55 + (G.tc ? 20 : 0) + (visc ? 40 : 0), conv = 8;
  const double phase = 7000.0 / 16.0;  // latency of a block's phases, in FP64 warp operations
  const double busy[3] = {0.60, 0.95, 1.0};
  const bool low = G.nb < kTileY / 2;
  Strips best{};
  double best_t = 0.0;
  for (int w0 : {kTileX, 24, 16, 12, 8}) {
    const int n_strips = (G.na + w0 - 1) / w0;
    // strips of equal width; full ones where that saves none (they are staged by tensor copies)
    int w = (G.na + n_strips - 1) / n_strips;
    if (w0 == kTileX && G.na >= 8 * kTileX) w = kTileX;
    const long long units = (long long)n_strips * G.nb;
    auto warps = [](double lanes) { return std::ceil(lanes / 32.0); };
    auto segment = [&](double rows) {  // FP64 warp operations of `rows` rows of a strip
      return face * (warps((w + 1.0) * rows) + warps(w * (rows + 1.0))) + cell * warps(w * rows) +
             conv * warps((w + 4.0) * (rows + 4.0));
    };
    const int forms = 2 * resident + (low && n_strips > resident * sms);
    for (int k = 0; k < forms; ++k) {
      // a whole number of CTAs per strip, then all there is room for; at last, on low planes, one per strip
      const bool each = k == 2 * resident;
      const long long room = std::min(units, (long long)(k / 2 + 1) * sms), aligned = room / n_strips * n_strips;
      const bool cross = !each && k & 1;  // some CTA's rows end one strip and begin the next
      const long long ctas = each ? n_strips : (cross ? room : aligned);
      if (ctas == 0 || (cross && room == aligned)) continue;
      const long long rows = (units + ctas - 1) / ctas;  // of the busiest CTA
      const double blocks = std::ceil((double)rows / kTileY);
      const long long on_sm = (ctas + sms - 1) / sms;
      double t = std::max(segment((double)rows) * on_sm / busy[std::min(on_sm, 3LL) - 1], phase * blocks);
      // two segments one after the other; beyond one block the rest of the SM's work hides it
      if (cross && blocks == 1.0)
        t = std::max(t, std::max(2.0 * segment(0.5 * rows) / busy[0], phase * 2.0));
      // low planes: each start of a segment takes some three phases
      if (low && cross && rows > G.nb + 1) {
        const long long pieces = 2 + (rows - 2) / G.nb;
        t = std::max(t, std::max(pieces * segment((double)rows / pieces) * on_sm / busy[std::min(on_sm, 3LL) - 1],
                                 3.0 * phase * pieces));
      }
      if (each) t = std::max(t, 3.0 * phase * ((on_sm + resident - 1) / resident));
      if (best.ctas == 0 || t < best_t * 0.995) {
        best = Strips{w, units, ctas};
        best_t = t;
      }
    }
  }
  return best;
}

template <int PLANE, int RS, int KIND, bool WACT>
cudaError_t launch_one(const Grid& G, Fields uin, Fields u0, Fields uout, StepCtrl* ctrl, const Fields* hout,
                       const TmaState* tin, const PrimCopy& pc, cudaStream_t st) {
  using SM = TileSmem<double, WACT ? 5 : 4, SingleTile>;
  auto kern = stage2d_fp64<PLANE, RS, KIND, WACT>;
  static bool attr_set = false;  // per instantiation, once per process
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)((WACT ? SM::bytes_vface() : SM::bytes(true)) + kSmemAlign));
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  static int resident[3] = {0, 0, 0};  // CTAs per SM: plain / conduction / shared-face viscosity
  const int cfg = WACT && G.visc ? 2 : (G.tc != 0);
  const size_t smem = (cfg == 2 ? SM::bytes_vface() : SM::bytes(cfg == 1)) + kSmemAlign;
  if (!resident[cfg]) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident[cfg], kern, kTileThreads, smem);
    if (e != cudaSuccess) return e;
    if (resident[cfg] < 1) resident[cfg] = 1;
  }
  const Strips p = split_strips(G, RS, WACT, resident[cfg]);
  const Fields none{};
  static const TmaState no_tma{};
  const cudaError_t e = launch_pdl(kern, dim3((unsigned)p.ctas), dim3(kTileThreads), smem, st, G, uin, u0, uout, ctrl,
                                   hout ? *hout : none, p.width, p.units, tin ? *tin : no_tma, tin ? 1 : 0,
                                   pc.qin ? *pc.qin : none, pc.qout ? *pc.qout : none, pc.tq ? *pc.tq : no_tma,
                                   pc.tq ? 1 : 0);
  return e != cudaSuccess ? e : cudaGetLastError();
}

template <int PLANE, int RS, bool WACT>
cudaError_t launch_kind(const Grid& G, int kind, Fields uin, Fields u0, Fields uout, StepCtrl* ctrl,
                        const Fields* hout, const TmaState* tin, const PrimCopy& pc, cudaStream_t st) {
  switch (kind) {
    case STAGE_EULER: return launch_one<PLANE, RS, STAGE_EULER, WACT>(G, uin, u0, uout, ctrl, hout, tin, pc, st);
    case STAGE_RK_1: return launch_one<PLANE, RS, STAGE_RK_1, WACT>(G, uin, u0, uout, ctrl, nullptr, tin, pc, st);
    default: return launch_one<PLANE, RS, STAGE_RK_2, WACT>(G, uin, u0, uout, ctrl, hout, tin, pc, st);
  }
}

template <int PLANE, int RS>
cudaError_t launch_w(const Grid& G, int kind, bool wact, Fields uin, Fields u0, Fields uout, StepCtrl* ctrl,
                     const Fields* hout, const TmaState* tin, const PrimCopy& pc, cudaStream_t st) {
  return wact ? launch_kind<PLANE, RS, true>(G, kind, uin, u0, uout, ctrl, hout, tin, pc, st)
              : launch_kind<PLANE, RS, false>(G, kind, uin, u0, uout, ctrl, hout, tin, pc, st);
}

}  // namespace

cudaError_t launch_stage2d(const Grid& G, int riemann_solver, int kind, bool wact, Fields uin, Fields u0,
                           Fields uout, StepCtrl* ctrl, cudaStream_t st, const Fields* hout, const TmaState* tin,
                           const PrimCopy* prims) {
  static const PrimCopy no_prims{};
  const PrimCopy& pc = prims ? *prims : no_prims;
  if (G.plane == PLANE_XY)
    return riemann_solver == 0 ? launch_w<PLANE_XY, 0>(G, kind, wact, uin, u0, uout, ctrl, hout, tin, pc, st)
                               : launch_w<PLANE_XY, 1>(G, kind, wact, uin, u0, uout, ctrl, hout, tin, pc, st);
  return riemann_solver == 0 ? launch_w<PLANE_XZ, 0>(G, kind, wact, uin, u0, uout, ctrl, hout, tin, pc, st)
                             : launch_w<PLANE_XZ, 1>(G, kind, wact, uin, u0, uout, ctrl, hout, tin, pc, st);
}

bool encode_tma_state(const Grid& G, const Fields& u, TmaState* tin) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static bool looked = false;
  if (!looked) {
    looked = true;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  if (!encode || G.ndim != 2) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)G.na, (cuuint64_t)G.rows};
  const cuuint64_t strides[1] = {(cuuint64_t)G.pitch * sizeof(double)};  // bytes, a multiple of 128
  const cuuint32_t box[2] = {(cuuint32_t)(kTileX + 4), (cuuint32_t)kTmaRows};
  const cuuint32_t estr[2] = {1, 1};
  for (int v = 0; v < 5; ++v) {
    if (!u.f[v] || (reinterpret_cast<uintptr_t>(u.f[v]) & 15u)) return false;
    if (encode(&tin->m[v], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, u.f[v], dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  return true;
}

}  // namespace fv
