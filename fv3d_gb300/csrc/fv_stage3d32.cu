// fv_stage3d32.cu -- the block form of the FP32-mixed stage of 3-D problems.
//
// The same z-marching organisation as the FP64 3-D kernel (fv_stage3d.cu): a
// CTA owns a 16 x 16 block of columns and a chunk of z layers; a ring of four
// layers of primitives sits in shared memory (FP32 here: 51.6 KB with
// conduction, 4 CTAs per SM); the x and y faces of layer k are solved while
// layer k+2 is loaded; each thread solves the z face above its column and
// updates its cell.  The arithmetic is that of the 2-D mixed form
// (fv_tile32.cuh): U^n carried as an FP32 (hi, lo) pair, U* as FP32,
// primitives / slopes / Riemann solvers / conduction / viscosity in FP32,
// increments accumulated on the pairs with error-free sums, the CFL maximum
// turned into dt in FP64 by the control kernel.  Every reference feature of
// the 3-D FP64 kernel is kept: C91 ghosts, the well-balanced / C91 z-flux
// overrides, gravity, fixed-temperature / fixed-gradient conduction
// boundaries, viscosity with the reference's z-branch quirks, and the
// corrected physics as a template option (B02 conductivity runs on the FP64
// handle only).  Built with fast-math.
//
// Problems without z-boundary and corrected physics take a body of their own
// (stage3d_plain32): the operations of the z-marched form (fv_march3d32.cu) in
// its order, so that both forms give the same bits and the faster one can be
// chosen for a group of problems by their sizes.
#include "fv_march32.cuh"

namespace fv {

namespace {

// 1: RK2 stage 2 asks L1 for each cell's U^n before its z face and
// increments are formed (no registers held; the load comes where U^n is
// added): +2 % on random 160^3 and 192^3.
#ifndef FV_3D32_UN_PREFETCH
#define FV_3D32_UN_PREFETCH 1
#endif

constexpr int kTX = 16, kTY = 16;
constexpr int kThreads = kTX * kTY;
constexpr int kHX = kTX + 4, kHY = kTY + 4;
constexpr int kLayer = kHX * kHY;
constexpr int kRing = 4;
constexpr int kNFA = (kTX + 1) * kTY;
constexpr int kNFA_PAD = (kNFA + 31) / 32 * 32;
constexpr int kNFB = kTX * (kTY + 1);
static_assert(kThreads == kTileThreads, "one thread per column");

// Shared memory (floats): Q[ring][v][hy][hx], FA, FB of the current layer,
// TT[ring][hy][hx] (conduction only).  Every row is kRowPitch = 20 floats
// apart (FA and FB rows padded to it): a warp owns the columns of rows r and
// r + 4 (column_of), 80 floats = 16 banks apart, so its per-column accesses
// fall on disjoint banks.
constexpr int kRowPitch = kHX;
static_assert(kRowPitch >= kTX + 1 && (4 * kRowPitch) % 32 == 16, "rows r and r+4 on disjoint banks");
struct Smem3f {
  float* base;
  static constexpr int kFA = kRing * 5 * kLayer;
  static constexpr int kFB = kFA + 5 * kTY * kRowPitch;
  static constexpr int kT = kFB + 5 * (kTY + 1) * kRowPitch;
  static constexpr size_t bytes(bool tc) { return sizeof(float) * (size_t)(kT + (tc ? kRing * kLayer : 0)); }
  __device__ float& q(int s, int v, int hy, int hx) const { return base[((s * 5 + v) * kHY + hy) * kHX + hx]; }
  __device__ float& fa(int v, int fy, int fx) const { return base[kFA + (v * kTY + fy) * kRowPitch + fx]; }
  __device__ float& fb(int v, int fy, int fx) const { return base[kFB + (v * (kTY + 1) + fy) * kRowPitch + fx]; }
  __device__ float& temp(int s, int hy, int hx) const { return base[kT + (s * kHY + hy) * kHX + hx]; }
};

// The column (cx, cy) of the 16 x 16 block a thread owns: the two half-warps
// of warp w take rows r and r + 4 (r = (w & 3) + 8 * (w >> 2)).
__device__ __forceinline__ void column_of(int tid, int& cx, int& cy) {
  const int lane = tid & 31, w = tid >> 5;
  cx = lane & 15;
  cy = (w & 3) + ((w >> 2) << 3) + ((lane >> 4) << 2);
}

__device__ __forceinline__ int slot_of(int kg) { return (kg + 4) & 3; }

// The stage input of one stored cell: pairs (U^n) or U* values (internal
// energy in the energy slot).
struct MixedIn {
  const float2* const* pairs;  // src (STAGE_RK_1 / STAGE_EULER)
  const float* const* us;      // U* (STAGE_RK_2)
  bool in_pairs;
};

__device__ __forceinline__ void load_prim32(const MixedIn& in, unsigned o, float gm1, float q[5]) {
  if (in.in_pairs) {
    float2 w[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) w[v] = in.pairs[v][o];
    cons_to_prim_pairs<PLANE_XY, true>(w, gm1, q);
  } else {
    float u[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) u[v] = in.us[v][o];
    cons_to_prim_star<true>(u, gm1, q);
  }
}

// fillC91 (BoundaryConditions.h:87-134) in FP32, as the FP64 kernel's.
__device__ __forceinline__ void c91_ghost32(const Grid& G, const MixedIn& in, unsigned col, bool fa, bool fb, int kg,
                                            float res[5]) {
  const int kref = kg < 0 ? 0 : G.nc - 1;
  const int ksym = kg < 0 ? -kg - 1 : 2 * G.nc - kg - 1;
  float qref[5], qsym[5];
  const unsigned zs = (unsigned)G.nb * (unsigned)G.pitch;
  load_prim32(in, (unsigned)kref * zs + col, G.gm1_f, qref);
  load_prim32(in, (unsigned)ksym * zs + col, G.gm1_f, qsym);
  if (fa) {
    qref[1] = -qref[1];
    qsym[1] = -qsym[1];
  }
  if (fb) {
    qref[2] = -qref[2];
    qsym[2] = -qsym[2];
  }
  const float grav = G.gravity_flag ? 1.0f : 0.0f;
  const float posz = G.zmin_f + ((float)kg + 0.5f) * G.dz_f;
  if (kg < 0) {
    const float dz = posz - 0.5f * G.dz_f;
    const float T = 1.0f + posz * G.theta1_f;
    float p = qref[4] + dz * qref[0] * grav;
    float r = p / T;
    p = fmaxf(p, 1.0e-6f);
    r = fmaxf(r, 1.0e-6f);
    const float dratio = qsym[0] / r;
    res[0] = r;
    res[1] = qsym[1];
    res[2] = qsym[2];
    res[3] = -qsym[3] * dratio;
    res[4] = p;
  } else {
    const float Tref = qref[4] / qref[0];
    const float dz = posz - (1.0f - 0.5f * G.dz_f);
    const float T = Tref + dz * G.theta1_f;
    const float P = qref[4] + dz * qref[0] * grav;
    const float rho = P / T;
    res[4] = fmaxf(P, 1.0e-6f);
    res[0] = fmaxf(rho, 1.0e-6f);
    const float dratio = qsym[0] / rho;
    res[1] = qsym[1] * dratio;
    res[2] = qsym[2] * dratio;
    res[3] = -qsym[3] * dratio;
  }
}

__device__ __forceinline__ void load_layer32(const Grid& G, const MixedIn& in, int x0, int y0, int kg,
                                             const Smem3f& S, int tid) {
  const int s = slot_of(kg);
  const bool c91 = G.bc_c == DBC_C91 && (kg < 0 || kg >= G.nc);
  bool fz = false;
  const int sz = c91 ? 0 : bc_source(kg, G.nc, G.bc_c, fz);
  const unsigned zoff = (unsigned)sz * (unsigned)G.nb * (unsigned)G.pitch;
  for (int idx = tid; idx < kLayer; idx += kThreads) {
    const int hy = idx / kHX, hx = idx - hy * kHX;
    bool fa, fb;
    const int sa = bc_source(x0 + hx - 2, G.na, G.bc_a, fa);
    const int sb = bc_source(y0 + hy - 2, G.nb, G.bc_b, fb);
    const unsigned col = (unsigned)sb * (unsigned)G.pitch + (unsigned)sa;
    float q[5];
    if (!c91) {
      load_prim32(in, zoff + col, G.gm1_f, q);
      if (fa) q[1] = -q[1];
      if (fb) q[2] = -q[2];
      if (fz) q[3] = -q[3];
    } else {
      c91_ghost32(G, in, col, fa, fb, kg, q);
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) S.q(s, v, hy, hx) = q[v];
    if (G.tc) S.temp(s, hy, hx) = q[4] / q[0];
  }
}

template <int DIR>
__device__ __forceinline__ Slots<float> slots3f(const float q[5]) {
  Slots<float> s;
  s.r = q[0];
  s.p = q[4];
  s.un = DIR == 0 ? q[1] : (DIR == 1 ? q[2] : q[3]);
  s.t1 = DIR == 1 ? q[1] : q[2];
  s.t2 = DIR == 2 ? q[1] : q[3];
  return s;
}

template <int DIR>
__device__ __forceinline__ void unslot3f(const float f[5], float out[5]) {
  out[0] = f[0];
  out[4] = f[4];
  if (DIR == 0) {
    out[1] = f[1]; out[2] = f[2]; out[3] = f[3];
  } else if (DIR == 1) {
    out[2] = f[1]; out[1] = f[2]; out[3] = f[3];
  } else {
    out[3] = f[1]; out[2] = f[2]; out[1] = f[3];
  }
}

template <int DIR, bool CORR>
__device__ __forceinline__ void face3f(const float c[4][5], int rs, int recon, const Grid& G, float out[5],
                                       float* pout) {
  float qL[5], qR[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    if (recon == R_PLM) {
      const float d01 = c[1][v] - c[0][v], d12 = c[2][v] - c[1][v], d23 = c[3][v] - c[2][v];
      qL[v] = c[1][v] + minmod32(d01, d12) * 0.5f;
      qR[v] = c[2][v] - minmod32(d12, d23) * 0.5f;
    } else {
      qL[v] = c[1][v];
      qR[v] = c[2][v];
    }
  }
  if (DIR == 2 && recon == R_PCM_WB) {  // Update.h:27
    qL[4] = qL[4] + qL[0] * G.g_dz_f * 0.5f;
    qR[4] = qR[4] - qR[0] * G.g_dz_f * 0.5f;
  }
  const Slots<float> L = slots3f<DIR>(qL), R = slots3f<DIR>(qR);
  float f[5];
  if (rs == 0)
    hll32(L, R, G.gamma_f, G.inv_gm1_f, f, pout);
  else
    hllc32<CORR>(L, R, G.gamma_f, G.inv_gm1_f, f, pout);
  unslot3f<DIR>(f, out);
}

struct RingVelF {
  Smem3f S;
  int k, hy, hx;
  __device__ __forceinline__ float operator()(int dk, int dj, int di, int var) const {
    return S.q(slot_of(k + dk - 1), var, hy + dj - 1, hx + di - 1);
  }
};

// One mixed stage of the columns (bx, by), z chunk bz of tz layers (CORR:
// the corrected physics, as the FP64 kernel's).  Inputs
// per kind as the 2-D mixed tile: RK_1 reads U^n pairs and writes U*; RK_2
// reads U* and U^n and writes U^n+1 over U^n; Euler reads pairs `src` and
// writes pairs `dst`.
template <int RS, bool CORR>
__device__ __forceinline__ void stage3d_body32(const Grid& G, const MixedFields& M, float2* const src[5],
                                               float2* const dst[5], StepCtrl* ctrl, int kind, int bx, int by, int bz,
                                               int tz, float* smem, unsigned long long* s_red) {
  const Smem3f S{smem};
  const int tid = threadIdx.x;
  const int x0 = bx * kTX, y0 = by * kTY;
  const int k0 = bz * tz;
  const int k1 = min(k0 + tz, G.nc);
  int cx, cy;
  column_of(tid, cx, cy);
  const int x = x0 + cx, y = y0 + cy;
  const bool own = x < G.na && y < G.nb;
  // 32-bit offsets (the host keeps every field below 2^32 elements for the
  // mixed kernels).  Measured: 3-6% faster than 64-bit offsets here, while the
  // 2-D tile kernels keep 64-bit offsets, which spare them a register spill.
  const unsigned col = (unsigned)y * (unsigned)G.pitch + (unsigned)x;
  const unsigned zstride = (unsigned)G.nb * (unsigned)G.pitch;

  if (!ctrl->active) {
    if (kind == STAGE_EULER && own) {
      for (int k = k0; k < k1; ++k) {
        const unsigned o = (unsigned)k * zstride + col;
#pragma unroll
        for (int v = 0; v < 5; ++v) dst[v][o] = src[v][o];
      }
    }
    return;
  }
  const float dt = (float)ctrl->dt_cur;  // once per work item
  const int parity = ctrl->parity;
  const int recon = G.recon;
  const bool need_pout = G.wb_flux_z || G.bc_c == DBC_C91;
  const MixedIn in{src, M.us, kind != STAGE_RK_2};
  const float dtdx = dt * G.inv_dx_f, dtdy = dt * G.inv_dy_f, dtdz = dt * G.inv_dz_f;

  for (int kg = k0 - 2; kg <= k0 + 1; ++kg) load_layer32(G, in, x0, y0, kg, S, tid);
  __syncthreads();
  float fzL[5], poutL = 0.0f;
  if (own) {
    float c[4][5];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int v = 0; v < 5; ++v) c[m][v] = S.q(slot_of(k0 - 2 + m), v, cy + 2, cx + 2);
    face3f<2, CORR>(c, RS, recon, G, fzL, need_pout ? &poutL : nullptr);
  }
  __syncthreads();

  float red = 0.0f;
  bool bad = false;
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    load_layer32(G, in, x0, y0, k + 2, S, tid);
    const int sk = slot_of(k);
    for (int it = tid; it < kNFA_PAD + kNFB; it += kThreads) {
      float c[4][5], f[5];
      if (it < kNFA_PAD) {
        if (it >= kNFA) continue;
        const int fy = it / (kTX + 1), fx = it - fy * (kTX + 1);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v) c[m][v] = S.q(sk, v, fy + 2, fx + m);
        face3f<0, CORR>(c, RS, recon, G, f, nullptr);
#pragma unroll
        for (int v = 0; v < 5; ++v) S.fa(v, fy, fx) = f[v];
      } else {
        const int j = it - kNFA_PAD;
        const int fy = j / kTX, fx = j - fy * kTX;
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v) c[m][v] = S.q(sk, v, fy + m, fx + 2);
        face3f<1, CORR>(c, RS, recon, G, f, nullptr);
#pragma unroll
        for (int v = 0; v < 5; ++v) S.fb(v, fy, fx) = f[v];
      }
    }
    __syncthreads();

    if (own) {
#if FV_3D32_UN_PREFETCH
      if (kind == STAGE_RK_2) {  // U^n of the cell into L1 while the z face and increments are formed
        const unsigned o = (unsigned)k * zstride + col;
#pragma unroll
        for (int v = 0; v < 5; ++v) asm volatile("prefetch.global.L1 [%0];" ::"l"(M.un[v] + o));
      }
#endif
      float fzR[5], poutR = 0.0f;
      {
        float c[4][5];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v) c[m][v] = S.q(slot_of(k - 1 + m), v, cy + 2, cx + 2);
        face3f<2, CORR>(c, RS, recon, G, fzR, need_pout ? &poutR : nullptr);
      }
      const unsigned o = (unsigned)k * zstride + col;
      float fL[5], fR[5];
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        fL[v] = fzL[v];
        fR[v] = fzR[v];
      }
      const float rho_c = S.q(sk, 0, cy + 2, cx + 2);
      if (G.wb_flux_z && (k == 0 || k == G.nc - 1)) {  // Update.h:131-137
        if (k == 0) {
          fL[0] = 0.0f; fL[1] = 0.0f; fL[2] = 0.0f; fL[4] = 0.0f;
          fL[3] = poutR - rho_c * G.g_dz_f;
        } else {
          fR[0] = 0.0f; fR[1] = 0.0f; fR[2] = 0.0f; fR[4] = 0.0f;
          fR[3] = poutL + rho_c * G.g_dz_f;
        }
      } else if (G.bc_c == DBC_C91 && (k == 0 || k == G.nc - 1)) {  // Update.h:138-143
        if (k == 0) {
          fL[0] = 0.0f; fL[1] = 0.0f; fL[2] = 0.0f; fL[4] = 0.0f;
          fL[3] = poutL;
        } else {
          fR[0] = 0.0f; fR[1] = 0.0f; fR[2] = 0.0f; fR[4] = 0.0f;
          fR[3] = poutR;
        }
      }
      float du[5];
#pragma unroll
      for (int v = 0; v < 5; ++v)
        du[v] = (S.fa(v, cy, cx) - S.fa(v, cy, cx + 1)) * dtdx + (S.fb(v, cy, cx) - S.fb(v, cy + 1, cx)) * dtdy +
                (fL[v] - fR[v]) * dtdz;
      if (G.gravity) {
        du[3] += dt * rho_c * G.g_f;
        du[4] += dt * 0.5f * (fL[0] + fR[0]) * G.g_f;
      }
      float2 base[5];  // the stage input at this cell as pairs (U*: E* rebuilt, fv_tile32.cuh)
      if (in.in_pairs) {
#pragma unroll
        for (int v = 0; v < 5; ++v) base[v] = src[v][o];
      } else {
        float u[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) u[v] = M.us[v][o];
#pragma unroll
        for (int v = 0; v < 4; ++v) base[v] = make_float2(u[v], 0.0f);
        base[4] = pair_add(kinetic_star<true>(u), u[4]);
      }
      {  // density floor on the hydro update (Update.h:160)
        const float2 rho = pair_add(base[0], du[0]);
        if (rho.x + rho.y < 1.0e-6f) {
          base[0] = make_float2(1.0e-6f, 0.0f);
          du[0] = 0.0f;
        }
      }
      if (G.tc) {  // ThermalConduction.h:38-96
        const float kC = G.kappa_f, kF = G.kappa_f, kB = G.kappa_f;  // batches take constant kappa
        const int hy = cy + 2, hx = cx + 2;
        const float TC = S.temp(sk, hy, hx);
        const float FL = kC * (TC - S.temp(sk, hy, hx - 1)) * G.inv_dx_f;
        const float FR = kC * (S.temp(sk, hy, hx + 1) - TC) * G.inv_dx_f;
        const float FU = kC * (TC - S.temp(sk, hy - 1, hx)) * G.inv_dy_f;
        const float FD = kC * (S.temp(sk, hy + 1, hx) - TC) * G.inv_dy_f;
        float FF = kF * (TC - S.temp(slot_of(k - 1), hy, hx)) * G.inv_dz_f;
        float FB = kB * (S.temp(slot_of(k + 1), hy, hx) - TC) * G.inv_dz_f;
        if (k == 0 && G.bctc_zmin != 0)
          FF = G.bctc_zmin == 1 ? kF * 2.0f * (TC - G.bctc_zmin_value_f) * G.inv_dz_f : kF * G.bctc_zmin_value_f;
        if (k == G.nc - 1 && G.bctc_zmax != 0)
          FB = G.bctc_zmax == 1 ? kB * 2.0f * (G.bctc_zmax_value_f - TC) * G.inv_dz_f : kB * G.bctc_zmax_value_f;
        du[4] += dtdx * (FR - FL) + dtdy * (FD - FU) + dtdz * (FB - FF);
      }
      if (G.visc) {  // Viscosity.h:145-151
        const RingVelF P{S, k, cy + 2, cx + 2};
        float vf[3][5];
        viscous3d<CORR, float>(P, G.inv_dx_f, G.inv_dy_f, G.inv_dz_f, G.mu_f, vf);
        if (CORR) {  // the flux differences divided by the cell sizes
#pragma unroll
          for (int v = 1; v < 5; ++v)
            du[v] += (vf[0][v] * G.inv_dx_f + vf[1][v] * G.inv_dy_f + vf[2][v] * G.inv_dz_f) * dt;
        } else {
#pragma unroll
          for (int v = 1; v < 5; ++v) du[v] += (vf[0][v] + vf[1][v] + vf[2][v]) * dt;
        }
      }
      if (kind == STAGE_RK_1) {
        float us[5];
#pragma unroll
        for (int v = 0; v < 4; ++v) us[v] = base[v].x + (base[v].y + du[v]);
        us[4] = internal_energy(pair_add(base[4], du[4]), kinetic_star<true>(us));
#pragma unroll
        for (int v = 0; v < 5; ++v) M.us[v][o] = us[v];
      } else {
        float2 fin[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          float2 r;
          if (kind == STAGE_RK_2) {
            r = pair_add(pair_add(M.un[v][o], base[v]), du[v]);
            r = make_float2(0.5f * r.x, 0.5f * r.y);
          } else {
            r = pair_add(base[v], du[v]);
          }
          dst[v][o] = r;
          fin[v] = r;
        }
        const float inv = inv_dt_hyp32<PLANE_XY, true>(fin, G);
        bad |= !(inv <= 3.0e38f);
        red = fmaxf(red, inv);
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) fzL[v] = fzR[v];
      poutL = poutR;
    }
    __syncthreads();
  }
  if (kind != STAGE_RK_1) {
    if (bad) atomicOr(&ctrl->err, 1);
    block_max_atomic((unsigned long long)__double_as_longlong((double)red), &ctrl->slot[parity ^ 1], s_red);
  }
}

// ---- the arithmetic of the z-marched form -----------------------------------
//
// The marched form hides latency on small grids and keeps its lanes busy on
// planes that blocks of 30 x 15 columns fit; where those leave lanes idle,
// 16 x 16 blocks, four to an SM (three with viscosity), are the faster form
// (the choice: MarchedIsFaster in fv_batch.cpp).  Every operation below is one
// of march_block32, on the same operands: differences towards the higher index,
// face states, fluxes differenced as they are, the diffusive ones beside them,
// the increment's terms in the order x, gravity, lower z, y, upper z.
//
// Bound by instruction issue.  64 registers without spills (80 with viscosity);
// the diffusive fluxes of a face are formed once and shared, at the cost of the
// fourth CTA.  A step, the body of the z-boundary physics -> this one: PCM RK2
// 256^3 1,388 -> 1,071 us, PLM RK2 with conduction and viscosity 64 of 32^3
// 311 -> 297 (marched 638), 16 of 64^3 585 -> 537 (902), 32x16x2000 155 -> 150
// (380).

// Shared memory of the plain body: Smem3f and, with viscosity, four diffusive
// fluxes per face (three momenta, energy).
struct SmemPlain : Smem3f {
  static constexpr int kVA = kT + kRing * kLayer;
  static constexpr int kVB = kVA + 4 * kTY * kRowPitch;
  static constexpr int kEnd = kVB + 4 * (kTY + 1) * kRowPitch;
  static constexpr size_t plain_bytes(bool tc, bool visc) { return visc ? sizeof(float) * (size_t)kEnd : bytes(tc); }
  __device__ float& va(int v, int fy, int fx) const { return base[kVA + (v * kTY + fy) * kRowPitch + fx]; }
  __device__ float& vb(int v, int fy, int fx) const { return base[kVB + (v * (kTY + 1) + fy) * kRowPitch + fx]; }
};

// The flux of the face between cells c[1] and c[2] of four along an axis whose
// normal and transverse velocities are in slots UN, T1, T2.
template <int RS, int UN, int T1, int T2>
__device__ __forceinline__ void face_plain(const float c[4][5], bool plm, bool wb, const Grid& G, float f[5]) {
  using namespace m32;
  float L[5], R[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const float d = sub(c[2][v], c[1][v]);
    L[v] = fma_(0.5f, plm ? minmod(sub(c[1][v], c[0][v]), d) : 0.0f, c[1][v]);
    R[v] = fma_(-0.5f, plm ? minmod(d, sub(c[3][v], c[2][v])) : 0.0f, c[2][v]);
  }
  if (wb) {  // PCM_WB hydrostatic pressure (Update.h:27)
    L[4] = fma_(mul(L[0], G.g_dz_f), 0.5f, L[4]);
    R[4] = fma_(mul(R[0], G.g_dz_f), -0.5f, R[4]);
  }
  if (RS == 0) hll<UN, T1, T2, true>(L, R, G.gamma_f, G.inv_gm1_f, f);
  else hllc<UN, T1, T2, true>(L, R, G.gamma_f, G.inv_gm1_f, f);
}

template <int KIND>
__device__ __forceinline__ void load_layer_plain(const Grid& G, const char* in0, size_t fs, int x0, int y0, int kg,
                                                 const SmemPlain& S, int tid) {
  using namespace m32;
  constexpr bool STAR = KIND == STAGE_RK_2;
  const int s = slot_of(kg);
  bool mz;
  const unsigned zoff = (unsigned)bc_source(kg, G.nc, G.bc_c, mz) * ((unsigned)G.nb * (unsigned)G.pitch);
  for (int idx = tid; idx < kLayer; idx += kThreads) {
    const int hy = idx / kHX, hx = idx - hy * kHX;
    bool mx, my;
    const int sa = bc_source(x0 + hx - 2, G.na, G.bc_a, mx);
    const int sb = bc_source(y0 + hy - 2, G.nb, G.bc_b, my);
    const char* p = in0 + (size_t)(zoff + (unsigned)sb * (unsigned)G.pitch + (unsigned)sa) * (STAR ? 4 : 8);
    float2 c[5];
    float q[5];
#pragma unroll
    for (int v = 0; v < 5; ++v)
      c[v] = STAR ? make_float2(*reinterpret_cast<const float*>(p + v * fs), 0.0f)
                  : *reinterpret_cast<const float2*>(p + v * fs);
    const float r = STAR ? prim_of_star<true>(c, G.gm1_f, q) : prim_of_pairs<true>(c, G.gm1_f, q);
    S.q(s, 0, hy, hx) = q[0];
    S.q(s, 1, hy, hx) = mx ? -q[1] : q[1];
    S.q(s, 2, hy, hx) = my ? -q[2] : q[2];
    S.q(s, 3, hy, hx) = mz ? -q[3] : q[3];
    S.q(s, 4, hy, hx) = q[4];
    if (G.tc) S.temp(s, hy, hx) = mul(q[4], r);
  }
}

// Factors of a step that every cell shares.
struct PlainFactors {
  float dtdx, dtdy, dtdz, ktx, kty, ktz, vx1, vy1, vz1;
};

// Diffusive fluxes of the x face right of column (hy, hx - 1) and of the y face
// below row hy (Viscosity.h:163-213; conduction in the energy), layer slots
// D, P, U (below, at, above).
template <int DIR>
__device__ __forceinline__ void visc_face_plain(const SmemPlain& S, int sd, int sp, int su, int hy, int hx, bool tc,
                                                const PlainFactors& F, float g[4]) {
  using namespace m32;
  constexpr float k23 = 2.0f / 3.0f, k43 = 4.0f / 3.0f;
  const float cx = mul(0.25f, F.vx1), cy = mul(0.25f, F.vy1), cz = mul(0.25f, F.vz1);
  auto P = [&](int v, int dy, int dx) { return S.q(sp, v, hy + dy, hx + dx); };
  auto ez = [&](int v, int dy, int dx) { return sub(S.q(su, v, hy + dy, hx + dx), S.q(sd, v, hy + dy, hx + dx)); };
  if (DIR == 0) {  // columns hx - 1 and hx
    const float d1 = sub(P(1, 0, 0), P(1, 0, -1)), d2 = sub(P(2, 0, 0), P(2, 0, -1)), d3 = sub(P(3, 0, 0), P(3, 0, -1));
    auto sumy = [&](int v, int dx) {
      return add(sub(P(v, 0, dx), P(v, -1, dx)), sub(P(v, 1, dx), P(v, 0, dx)));
    };
    const float su_ = add(sumy(1, -1), sumy(1, 0)), sv = add(sumy(2, -1), sumy(2, 0));
    const float zu = add(ez(1, 0, -1), ez(1, 0, 0)), zw = add(ez(3, 0, -1), ez(3, 0, 0));
    const float txx = fma_(mul(k43, F.vx1), d1, -mul(k23, fma_(cy, sv, mul(cz, zw))));
    const float txy = fma_(F.vx1, d2, mul(cy, su_));
    const float txz = fma_(F.vx1, d3, mul(cz, zu));
    const float ma = fma_(0.5f, d1, P(1, 0, -1)), mb = fma_(0.5f, d2, P(2, 0, -1)), mc = fma_(0.5f, d3, P(3, 0, -1));
    const float ve = tc ? mul(F.ktx, sub(S.temp(sp, hy, hx), S.temp(sp, hy, hx - 1))) : 0.0f;
    g[0] = txx;
    g[1] = txy;
    g[2] = txz;
    g[3] = fma_(txx, ma, fma_(txy, mb, fma_(txz, mc, ve)));
  } else {  // rows hy - 1 and hy
    const float d1 = sub(P(1, 0, 0), P(1, -1, 0)), d2 = sub(P(2, 0, 0), P(2, -1, 0)), d3 = sub(P(3, 0, 0), P(3, -1, 0));
    auto sumx = [&](int v) {  // the row's two differences, and the row below's at once, as the marched form
      return add(add(sub(P(v, 0, 0), P(v, 0, -1)), sub(P(v, 0, 1), P(v, 0, 0))), sub(P(v, -1, 1), P(v, -1, -1)));
    };
    const float su_ = sumx(1), sv = sumx(2);
    const float zv = add(ez(2, 0, 0), ez(2, -1, 0)), zw = add(ez(3, 0, 0), ez(3, -1, 0));
    const float txy = fma_(F.vy1, d1, mul(cx, sv));
    const float tyy = fma_(mul(k43, F.vy1), d2, -mul(k23, fma_(cx, su_, mul(cz, zw))));
    const float tyz = fma_(F.vy1, d3, mul(cz, zv));
    const float ma = fma_(-0.5f, d1, P(1, 0, 0)), mb = fma_(-0.5f, d2, P(2, 0, 0)), mc = fma_(-0.5f, d3, P(3, 0, 0));
    const float ve = tc ? mul(F.kty, sub(S.temp(sp, hy, hx), S.temp(sp, hy - 1, hx))) : 0.0f;
    g[0] = txy;
    g[1] = tyy;
    g[2] = tyz;
    g[3] = fma_(txy, ma, fma_(tyy, mb, fma_(tyz, mc, ve)));
  }
}

// Diffusive fluxes of the z face between the cells of column (hy, hx) in layer
// slots sj (lower) and sm, with the reference's mix-ups (Viscosity.h:214-239):
// the lower cell's in up[4] (u, v, w, E), the upper cell's in low[4].
__device__ __forceinline__ void visc_z_plain(const SmemPlain& S, int sj, int sm, int hy, int hx, bool tc,
                                             const PlainFactors& F, float up[4], float low[4]) {
  using namespace m32;
  constexpr float k23 = 2.0f / 3.0f, k43 = 4.0f / 3.0f;
  const float cx = mul(0.25f, F.vx1), cz = mul(0.25f, F.vz1);
  auto J = [&](int v, int dy, int dx) { return S.q(sj, v, hy + dy, hx + dx); };
  auto M = [&](int v, int dy, int dx) { return S.q(sm, v, hy + dy, hx + dx); };
  auto right = [&](auto& C, int v) { return add(C(v, 0, 0), sub(C(v, 0, 1), C(v, 0, 0))); };
  // (a above) - (b below) of the cell
  auto updown = [&](auto& C, int a, int b) {
    return sub(add(C(a, 0, 0), sub(C(a, 1, 0), C(a, 0, 0))), sub(C(b, 0, 0), sub(C(b, 0, 0), C(b, -1, 0))));
  };
  const float d1 = sub(M(1, 0, 0), J(1, 0, 0)), d2 = sub(M(2, 0, 0), J(2, 0, 0)), d3 = sub(M(3, 0, 0), J(3, 0, 0));
  const float ma = fma_(0.5f, d1, J(1, 0, 0)), mb = fma_(0.5f, d2, J(2, 0, 0)), mc = fma_(0.5f, d3, J(3, 0, 0));
  const float ur = add(right(J, 1), right(M, 1)), vr = add(right(J, 2), right(M, 2));
  const float tzz = fma_(mul(k43, F.vz1), d3, -mul(k23, fma_(cx, ur, mul(cz, add(updown(J, 3, 2), updown(M, 3, 2))))));
  const float txz = fma_(F.vz1, d1, mul(cx, vr));
  const float tyz = fma_(F.vz1, d2, mul(cz, add(updown(J, 2, 3), updown(M, 2, 3))));
  const float ve = tc ? mul(F.ktz, sub(S.temp(sm, hy, hx), S.temp(sj, hy, hx))) : 0.0f;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    // left u and w of the cell, over its row and the one above (lower cell) or below (upper cell)
    const float ul = s == 0 ? add(sub(J(1, 0, 0), sub(J(1, 0, 0), J(1, 0, -1))), J(1, 1, -1)) : add(M(1, 0, -1), M(1, -1, -1));
    const float wl = s == 0 ? add(sub(J(3, 0, 0), sub(J(3, 0, 0), J(3, 0, -1))), J(3, 1, -1)) : add(M(3, 0, -1), M(3, -1, -1));
    float* V = s == 0 ? up : low;
    const float zz = fma_(mul(k23, cx), ul, tzz);
    const float xz = fma_(-cx, wl, txz);
    V[0] = xz;
    V[1] = tyz;
    V[2] = zz;
    V[3] = fma_(xz, ma, fma_(tyz, mb, fma_(zz, mc, ve)));
  }
}

// One stage of the columns (bx, by), z chunk bz; VISC: some problem of the
// group is viscous.
template <int RS, int KIND, bool VISC>
__device__ __forceinline__ void stage3d_plain32(const BatchInst& I, int flip, int bx, int by, int bz, float* smem,
                                                unsigned long long* s_red) {
  using namespace m32;
  constexpr bool STAR = KIND == STAGE_RK_2;
  const Grid& G = I.G;
  StepCtrl* ctrl = I.ctrl;
  const SmemPlain S{{smem}};
  const int tid = threadIdx.x;
  const int x0 = bx * kTX, y0 = by * kTY;
  const int k0 = bz * I.tz, k1 = min(k0 + I.tz, G.nc);
  int cx, cy;
  column_of(tid, cx, cy);
  const int hx = cx + 2, hy = cy + 2;
  const bool own = x0 + cx < G.na && y0 + cy < G.nb;
  const unsigned col = (unsigned)(y0 + cy) * (unsigned)G.pitch + (unsigned)(x0 + cx);
  const unsigned zstride = (unsigned)G.nb * (unsigned)G.pitch;
  const size_t fs = (size_t)G.fstride * 8;
  const char* in0 = reinterpret_cast<const char*>(STAR || (KIND == STAGE_EULER && flip) ? I.B.f[0] : I.A.f[0]);
  char* un0 = reinterpret_cast<char*>(I.A.f[0]);
  char* us0 = reinterpret_cast<char*>(I.B.f[0]);
  if (!ctrl->active) {
    if (KIND == STAGE_EULER && own) {
      char* out = flip ? un0 : us0;
      for (int k = k0; k < k1; ++k) {
        const size_t o = (size_t)((unsigned)k * zstride + col) * 8;
#pragma unroll
        for (int v = 0; v < 5; ++v)
          *reinterpret_cast<float2*>(out + o + v * fs) = *reinterpret_cast<const float2*>(in0 + o + v * fs);
      }
    }
    return;
  }
  const int parity = ctrl->parity;
  const bool plm = G.recon == R_PLM, wb_z = G.recon == R_PCM_WB;
  const bool tc = G.tc != 0, visc = VISC && G.visc != 0, grav = G.gravity != 0;
  const float2 dtp = ctrl->dt_pair;
  const float dt = dtp.x;
  PlainFactors F;
  F.dtdx = mul_to(dtp, I.inv_d[0]);
  F.dtdy = mul_to(dtp, I.inv_d[1]);
  F.dtdz = mul_to(dtp, I.inv_d[2]);
  F.ktx = tc ? mul_to(dtp, I.kappa_d2[0]) : 0.0f;
  F.kty = tc ? mul_to(dtp, I.kappa_d2[1]) : 0.0f;
  F.ktz = tc ? mul_to(dtp, I.kappa_d2[2]) : 0.0f;
  F.vx1 = visc ? mul_to(dtp, I.mu_d[0]) : 0.0f;
  F.vy1 = visc ? mul_to(dtp, I.mu_d[1]) : 0.0f;
  F.vz1 = visc ? mul_to(dtp, I.mu_d[2]) : 0.0f;

  for (int kg = k0 - 2; kg <= k0 + 1; ++kg) load_layer_plain<KIND>(G, in0, fs, x0, y0, kg, S, tid);
  __syncthreads();
  float fzL[5];                                  // flux of the z face below the cell
  float low[4] = {0.0f, 0.0f, 0.0f, 0.0f};       // its diffusive part
  auto z_face = [&](int k, float f[5]) {         // between layers k and k + 1
    float c[4][5];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int v = 0; v < 5; ++v) c[m][v] = S.q(slot_of(k - 1 + m), v, hy, hx);
    face_plain<RS, 3, 2, 1>(c, plm, wb_z, G, f);
  };
  if (own) {
    z_face(k0 - 1, fzL);
    if (visc) {
      float up[4];
      visc_z_plain(S, slot_of(k0 - 1), slot_of(k0), hy, hx, tc, F, up, low);
    }
  }
  __syncthreads();

  float red = 0.0f;
  bool bad = false;
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    load_layer_plain<KIND>(G, in0, fs, x0, y0, k + 2, S, tid);
    const int sd = slot_of(k - 1), sk = slot_of(k), su = slot_of(k + 1);
    for (int it = tid; it < kNFA_PAD + kNFB; it += kThreads) {
      float c[4][5], f[5], g[4];
      if (it < kNFA_PAD) {
        if (it >= kNFA) continue;
        const int fy = it / (kTX + 1), fx = it - fy * (kTX + 1);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v) c[m][v] = S.q(sk, v, fy + 2, fx + m);
        face_plain<RS, 1, 2, 3>(c, plm, false, G, f);
#pragma unroll
        for (int v = 0; v < 5; ++v) S.fa(v, fy, fx) = f[v];
        if (visc) {
          visc_face_plain<0>(S, sd, sk, su, fy + 2, fx + 2, tc, F, g);
#pragma unroll
          for (int v = 0; v < 4; ++v) S.va(v, fy, fx) = g[v];
        }
      } else {
        const int j = it - kNFA_PAD;
        const int fy = j / kTX, fx = j - fy * kTX;
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int v = 0; v < 5; ++v) c[m][v] = S.q(sk, v, fy + m, fx + 2);
        face_plain<RS, 2, 1, 3>(c, plm, false, G, f);
#pragma unroll
        for (int v = 0; v < 5; ++v) S.fb(v, fy, fx) = f[v];
        if (visc) {
          visc_face_plain<1>(S, sd, sk, su, fy + 2, fx + 2, tc, F, g);
#pragma unroll
          for (int v = 0; v < 4; ++v) S.vb(v, fy, fx) = g[v];
        }
      }
    }
    __syncthreads();

    if (own) {
      const size_t o = (size_t)((unsigned)k * zstride + col);
#if FV_3D32_UN_PREFETCH
      if (KIND == STAGE_RK_2) {  // U^n of the cell into L1 while the z face and increments are formed
#pragma unroll
        for (int v = 0; v < 5; ++v) asm volatile("prefetch.global.L1 [%0];" ::"l"(un0 + o * 8 + v * fs));
      }
#endif
      float fzR[5], up[4], next[4];
      z_face(k, fzR);
      if (visc) visc_z_plain(S, sk, su, hy, hx, tc, F, up, next);
      const float T = tc && !visc ? S.temp(sk, hy, hx) : 0.0f;
      float du[5];
#pragma unroll
      for (int v = 0; v < 5; ++v) du[v] = mul(F.dtdx, sub(S.fa(v, cy, cx), S.fa(v, cy, cx + 1)));
      if (visc) {
#pragma unroll
        for (int v = 1; v < 5; ++v) du[v] = add(du[v], sub(S.va(v - 1, cy, cx + 1), S.va(v - 1, cy, cx)));
      } else if (tc) {
        du[4] = add(du[4], sub(mul(F.ktx, sub(S.temp(sk, hy, hx + 1), T)), mul(F.ktx, sub(T, S.temp(sk, hy, hx - 1)))));
      }
      if (grav) du[3] = fma_(mul(dt, G.g_f), S.q(sk, 0, hy, hx), du[3]);
      if (visc) {
#pragma unroll
        for (int v = 1; v < 5; ++v) du[v] = sub(du[v], low[v - 1]);
      } else if (tc) {
        du[4] = sub(du[4], mul(F.ktz, sub(T, S.temp(sd, hy, hx))));
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        du[v] = fma_(F.dtdy, sub(S.fb(v, cy, cx), S.fb(v, cy + 1, cx)), du[v]);
        if (v > 0 && visc) du[v] = add(du[v], sub(S.vb(v - 1, cy + 1, cx), S.vb(v - 1, cy, cx)));
      }
      if (tc && !visc)
        du[4] = add(du[4], sub(mul(F.kty, sub(S.temp(sk, hy + 1, hx), T)), mul(F.kty, sub(T, S.temp(sk, hy - 1, hx)))));
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        du[v] = fma_(F.dtdz, sub(fzL[v], fzR[v]), du[v]);
        if (v > 0 && visc) du[v] = add(du[v], up[v - 1]);
      }
      if (tc && !visc) du[4] = add(du[4], mul(F.ktz, sub(S.temp(su, hy, hx), T)));
      if (grav)  // half the mass fluxes of both faces (Update.h:150)
        du[4] = fma_(mul(mul(0.5f, dt), G.g_f), add(fzL[0], fzR[0]), du[4]);
      float2 un[5];
      float us[5];
      {
        const char* p = (KIND == STAGE_RK_2 ? un0 : in0) + o * 8;
        const char* r = us0 + o * 4;
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          un[v] = *reinterpret_cast<const float2*>(p + v * fs);
          if (STAR) us[v] = *reinterpret_cast<const float*>(r + v * fs);
        }
      }
      // density floor on the hydro update (Update.h:160)
      const bool floored = (STAR ? add(us[0], du[0]) : add(add(un[0].x, du[0]), un[0].y)) < 1.0e-6f;
      if (floored) {
        if (!STAR) un[0] = make_float2(1.0e-6f, 0.0f);
        du[0] = 0.0f;
      }
      if (KIND == STAGE_RK_1) {
        float o5[5];
#pragma unroll
        for (int v = 0; v < 4; ++v) o5[v] = add(un[v].x, add(un[v].y, du[v]));
        // U* keeps its internal energy (fv_tile32.cuh)
        o5[4] = internal_energy(pair_add(un[4], du[4]), kinetic_star<true>(o5));
#pragma unroll
        for (int v = 0; v < 5; ++v) *reinterpret_cast<float*>(us0 + o * 4 + v * fs) = o5[v];
      } else {
        float2 fin[5];
        if (KIND == STAGE_RK_2) {  // 0.5 (U^n + U* + dU)
          const float2 ke = kinetic_star<true>(us);
          const float2 e = two_sum(ke.x, us[4]);
          if (floored) us[0] = 1.0e-6f;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            const float2 a = two_sum(un[v].x, v == 4 ? e.x : us[v]);
            const float2 b = two_sum(a.x, du[v]);
            const float lo = add(add(a.y, b.y), v == 4 ? add(un[v].y, add(e.y, ke.y)) : un[v].y);
            const float2 r = fast_two_sum(b.x, lo);
            fin[v] = make_float2(mul(0.5f, r.x), mul(0.5f, r.y));
          }
        } else {
#pragma unroll
          for (int v = 0; v < 5; ++v) fin[v] = pair_add(un[v], du[v]);
        }
        char* p = (KIND == STAGE_RK_2 || flip ? un0 : us0) + o * 8;
#pragma unroll
        for (int v = 0; v < 5; ++v) *reinterpret_cast<float2*>(p + v * fs) = fin[v];
        float q[5];
        const float r = prim_of_pairs<true>(fin, G.gm1_f, q);
        const float cs = sqrt_(mul(mul(q[4], G.gamma_f), r));
        const float inv = fma_(add(cs, fabsf(q[1])), G.inv_dx_f,
                               fma_(add(cs, fabsf(q[2])), G.inv_dy_f, mul(add(cs, fabsf(q[3])), G.inv_dz_f)));
        bad |= !(inv <= 3.0e38f);
        red = fmaxf(red, inv);
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) fzL[v] = fzR[v];
      if (visc) {
#pragma unroll
        for (int v = 0; v < 4; ++v) low[v] = next[v];
      }
    }
    __syncthreads();
  }
  if (KIND != STAGE_RK_1) {
    if (bad) atomicOr(&ctrl->err, 1);
    block_max_atomic((unsigned long long)__double_as_longlong((double)red), &ctrl->slot[parity ^ 1], s_red);
  }
}

static_assert(sizeof(BatchInst) % 8 == 0, "descriptor copied as 8-byte words");

// Work items of all problems of a group from the queue counter: item(I, bx, by, bz).
template <class Item>
__device__ __forceinline__ void each_item(const BatchInst* __restrict__ insts, int ninst, int ntiles, unsigned* queue,
                                          const Item& item) {
  __shared__ BatchInst s_inst;
  __shared__ int s_tile;
  pdl_wait();
  for (;;) {
    __syncthreads();  // the previous item is finished with s_tile, s_inst and smem
    if (threadIdx.x == 0) s_tile = (int)atomicAdd(queue, 1u);
    __syncthreads();
    const int t = s_tile;
    if (t >= ntiles) {
      pdl_trigger();  // no work left for this CTA
      break;
    }
    {
      int lo = 0, hi = ninst - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (insts[mid].tile0 <= t) lo = mid;
        else hi = mid - 1;
      }
      const unsigned long long* s = reinterpret_cast<const unsigned long long*>(insts + lo);
      unsigned long long* d = reinterpret_cast<unsigned long long*>(&s_inst);
      for (int w = threadIdx.x; w < (int)(sizeof(BatchInst) / 8); w += blockDim.x) d[w] = s[w];
    }
    __syncthreads();
    const BatchInst& I = s_inst;
    const int lt = t - I.tile0;
    const int per_layer = I.tiles_x * I.tiles_y;
    const int bz = lt / per_layer, rem = lt - bz * per_layer;
    const int by = rem / I.tiles_x, bx = rem - by * I.tiles_x;
    item(I, bx, by, bz);
  }
}

template <int RS, bool CORR>
__global__ void __launch_bounds__(kThreads, 4)
batch_stage3d32(const BatchInst* __restrict__ insts, int ninst, int ntiles, unsigned* queue, int kind, int flip) {
  extern __shared__ float smem_f[];
  __shared__ unsigned long long s_red[kThreads / 32];
  each_item(insts, ninst, ntiles, queue, [&](const BatchInst& I, int bx, int by, int bz) {
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
    stage3d_body32<RS, CORR>(I.G, M, src, dst, I.ctrl, kind, bx, by, bz, I.tz, smem_f, s_red);
  });
}

template <int RS, int KIND, bool VISC>
__global__ void __launch_bounds__(kThreads, VISC ? 3 : 4)
batch_plain3d32(const BatchInst* __restrict__ insts, int ninst, int ntiles, unsigned* queue, int, int flip) {
  extern __shared__ float smem_f[];
  __shared__ unsigned long long s_red[kThreads / 32];
  each_item(insts, ninst, ntiles, queue, [&](const BatchInst& I, int bx, int by, int bz) {
    stage3d_plain32<RS, KIND, VISC>(I, flip, bx, by, bz, smem_f, s_red);
  });
}

typedef void (*Batch3dKernel32)(const BatchInst*, int, int, unsigned*, int, int);

template <int RS, bool VISC>
Batch3dKernel32 plain_kernel(int kind) {
  switch (kind) {
    case STAGE_RK_1: return batch_plain3d32<RS, STAGE_RK_1, VISC>;
    case STAGE_RK_2: return batch_plain3d32<RS, STAGE_RK_2, VISC>;
    default: return batch_plain3d32<RS, STAGE_EULER, VISC>;
  }
}

// rs: the Riemann solver (bit 0), the corrected physics (bit 1) or the plain
// body (bit 2; then kind and visc too).
Batch3dKernel32 kernel32(int rs, int kind, bool visc) {
  switch (rs) {
    case 0: return batch_stage3d32<0, false>;
    case 1: return batch_stage3d32<1, false>;
    case 2: return batch_stage3d32<0, true>;
    case 3: return batch_stage3d32<1, true>;
    case 4: return visc ? plain_kernel<0, true>(kind) : plain_kernel<0, false>(kind);
    default: return visc ? plain_kernel<1, true>(kind) : plain_kernel<1, false>(kind);
  }
}

size_t smem32(int rs, bool tc, bool visc) { return rs >= 4 ? SmemPlain::plain_bytes(tc, visc) : Smem3f::bytes(tc); }

bool prepare32() {
  static bool done = false;
  if (done) return true;
  for (int rs = 0; rs < 6; ++rs)
    for (int kind : {STAGE_EULER, STAGE_RK_1, STAGE_RK_2})
      for (bool visc : {false, true})
        if (cudaFuncSetAttribute(kernel32(rs, kind, visc), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem32(rs, true, visc)) != cudaSuccess)
          return false;
  done = true;
  return true;
}

}  // namespace

int batch_stage3d_occupancy32(int rs, bool tc, bool visc, int kind) {
  if (!prepare32()) return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel32(rs, kind, visc), kThreads, smem32(rs, tc, visc)) !=
      cudaSuccess)
    return 0;
  return nb;
}

cudaError_t launch_batch_stage3d32(const BatchInst* insts, int ninst, int ntiles, unsigned* queue, int kind, int flip,
                                   int rs, int grid, bool tc, bool visc, cudaStream_t st) {
  if (!prepare32()) return cudaErrorInvalidConfiguration;
  const cudaError_t e = launch_pdl(kernel32(rs, kind, visc), dim3(grid), dim3(kThreads), smem32(rs, tc, visc), st, insts,
                                   ninst, ntiles, queue, kind, flip);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace fv
