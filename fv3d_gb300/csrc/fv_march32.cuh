// fv_march32.cuh -- one stage of a 2-D FP32-mixed problem, marched by warps.
//
// A work item is a strip of 28 columns and a run of rows; one warp owns it,
// each lane a column (two ghost columns on either side of the strip), and
// walks it row by row with the whole stencil in registers: the
// b-direction differences, face states and fluxes are carried from row to
// row, the a-direction neighbours come by warp shuffles.  Slopes are formed
// once per cell and direction and every face is solved once.  The conductive
// and viscous fluxes are carried beside the hydrodynamic ones and differenced
// on their own: added to a flux they would be rounded to the ulp of its
// pressure, and so would a flux scaled by dt/d before the difference (RT with
// conduction and viscosity 300x327, 64 steps: the error of w against FP64 was
// 1.8 times as large).  No shared memory, no barrier.
//
// Bound by instruction issue, as the block form (fv_tile32.cuh) it replaces,
// but with 21 (stage 1) and 26 (stage 2) warp instructions per cell with
// conduction and viscosity against 38 and 43: the block form forms each slope
// and reads each primitive of a face twice, evaluates every viscous face from
// both cells, and keeps the whole CTA at three barriers a block.  Four of 32
// lanes only serve their neighbours (a strip as wide as the warp needs its
// ghosts); two columns per lane (60 of 64 useful) took 255 registers and
// measured the same.  A step, block form -> this: shear 4096^2 1,259 -> 795 us
// (13.3 -> 21.1 G cell-updates/s), RT 512x1536 51.0 -> 41.1 us, 64 Sod / Sedov
// problems of 64^2..256^2 130.6 -> 91 us, Sedov 256^2 13.2 -> 12.8 us.
//
// The arithmetic is that of the mixed form (fv_tile32.cuh): U^n as (hi, lo)
// pairs, U* in FP32 with its internal energy, the pressure recovery in
// double-float, everything else FP32.  It is written with _rn intrinsics,
// which the compiler neither contracts nor reorders, so every kernel that
// includes it computes the same bits, however the rows are split.
#pragma once

#include "fv_control.cuh"
#include "fv_grid.cuh"
#include "fv_tile32.cuh"

namespace fv {

namespace m32 {

__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt_(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// a * b of (hi, lo) pairs, as a pair and rounded to FP32.
__device__ __forceinline__ float2 mul_pair(float2 a, float2 b) {
  const float p = mul(a.x, b.x);
  return make_float2(p, add(fma_(a.x, b.x, -p), fma_(a.x, b.y, mul(a.y, b.x))));
}
__device__ __forceinline__ float mul_to(float2 a, float2 b) {
  return fma_(a.x, b.x, fma_(a.x, b.y, mul(a.y, b.x)));
}

// minmod (Update.h:73-80) as the median of (a, b, 0): the argument of smaller
// magnitude when the signs agree, else 0.
__device__ __forceinline__ float minmod(float a, float b) {
  return fmaxf(fminf(a, b), fminf(fmaxf(a, b), 0.0f));
}

// HLLC of RiemannSolvers.h:39-112 (kinetic energy of the normal and first
// transverse velocity, as the reference) on states in storage order; UN, T1,
// T2: the slots of the normal and transverse velocities.  Each side has its own
// reciprocal of the density: products of two densities or of a density and a
// pressure leave the range of FP32 (rho above 9e18, p rho below 1.2e-38) where
// the quotients do not.
template <int UN, int T1, int T2, bool WACT>
__device__ __forceinline__ void hllc(const float L[5], const float R[5], float gamma, float inv_gm1, float f[5]) {
  constexpr bool H1 = WACT || T1 != 3, H2 = WACT || T2 != 3;
  const float rL = L[0], uL = L[UN], pL = L[4], rR = R[0], uR = R[UN], pR = R[4];
  const float cmax = sqrt_(mul(gamma, fmaxf(mul(pL, rcp(rL)), mul(pR, rcp(rR)))));
  const float SL = sub(fminf(uL, uR), cmax);
  const float SR = add(fmaxf(uL, uR), cmax);
  const float dL = sub(uL, SL), dR = sub(SR, uR);
  const float kL = mul(rL, dL), kR = mul(rR, dR);
  const float iD = rcp(add(kL, kR));
  const float uS = mul(fma_(kR, uR, fma_(kL, uL, sub(pL, pR))), iD);
  const float pS = mul(fma_(mul(kL, kR), sub(uL, uR), fma_(kR, pL, mul(kL, pR))), iD);
  const bool left = uS > 0.0f || SL > 0.0f;
  const bool outside = left ? SL > 0.0f : !(SR > 0.0f);
  const float r = left ? rL : rR, u = left ? uL : uR, p = left ? pL : pR;
  const float t1 = H1 ? (left ? L[T1] : R[T1]) : 0.0f;
  const float t2 = H2 ? (left ? L[T2] : R[T2]) : 0.0f;
  const float S = left ? SL : SR;
  const float m = left ? -dL : dR;   // S - u
  const float kS = left ? -kL : kR;  // r (S - u)
  float ke = mul(u, u);
  if (H1) ke = fma_(t1, t1, ke);
  const float E = fma_(mul(0.5f, r), ke, mul(p, inv_gm1));
  const float inv = rcp(sub(S, uS));
  const float sr = outside ? r : mul(kS, inv);
  const float sE = outside ? E : mul(fma_(m, E, fma_(pS, uS, -mul(p, u))), inv);
  const float su = outside ? u : uS;
  const float sp = outside ? p : pS;
  f[0] = mul(sr, su);
  f[UN] = fma_(f[0], su, sp);
  f[T1] = H1 ? mul(f[0], t1) : 0.0f;
  f[T2] = H2 ? mul(f[0], t2) : 0.0f;
  f[4] = mul(add(sE, sp), su);
}

// HLL with Davis wave speeds (RiemannSolvers.h:6-36).  The star flux
// (SR FL - SL FR + SL SR (UR - UL)) / (SR - SL) as a FL + b FR + c (UR - UL);
// a supersonic face takes (1, 0, 0) or (0, 1, 0), so its flux is exactly the
// upwind one.
template <int UN, int T1, int T2, bool WACT>
__device__ __forceinline__ void hll(const float L[5], const float R[5], float gamma, float inv_gm1, float f[5]) {
  constexpr bool H1 = WACT || T1 != 3, H2 = WACT || T2 != 3;
  const float cL = sqrt_(mul(mul(gamma, L[4]), rcp(L[0])));
  const float cR = sqrt_(mul(mul(gamma, R[4]), rcp(R[0])));
  const float SL = fminf(sub(L[UN], cL), sub(R[UN], cR));
  const float SR = fmaxf(add(L[UN], cL), add(R[UN], cR));
  const float inv = rcp(sub(SR, SL));
  float a = mul(SR, inv), b = -mul(SL, inv), c = mul(mul(SL, SR), inv);
  const bool up = SL >= 0.0f, dn = SR <= 0.0f;
  a = up ? 1.0f : (dn ? 0.0f : a);
  b = up ? 0.0f : (dn ? 1.0f : b);
  c = up || dn ? 0.0f : c;
  float kL = mul(L[UN], L[UN]), kR = mul(R[UN], R[UN]);
  if (H1) {
    kL = fma_(L[T1], L[T1], kL);
    kR = fma_(R[T1], R[T1], kR);
  }
  if (H2) {
    kL = fma_(L[T2], L[T2], kL);
    kR = fma_(R[T2], R[T2], kR);
  }
  const float EL = fma_(mul(0.5f, L[0]), kL, mul(L[4], inv_gm1));
  const float ER = fma_(mul(0.5f, R[0]), kR, mul(R[4], inv_gm1));
  const float mL = mul(L[0], L[UN]), mR = mul(R[0], R[UN]);
  f[0] = fma_(a, mL, fma_(b, mR, mul(c, sub(R[0], L[0]))));
  f[UN] = fma_(a, fma_(mL, L[UN], L[4]), fma_(b, fma_(mR, R[UN], R[4]), mul(c, sub(mR, mL))));
  f[T1] = H1 ? fma_(a, mul(mL, L[T1]), fma_(b, mul(mR, R[T1]), mul(c, fma_(R[0], R[T1], -mul(L[0], L[T1]))))) : 0.0f;
  f[T2] = H2 ? fma_(a, mul(mL, L[T2]), fma_(b, mul(mR, R[T2]), mul(c, fma_(R[0], R[T2], -mul(L[0], L[T2]))))) : 0.0f;
  f[4] = fma_(a, mul(add(L[4], EL), L[UN]), fma_(b, mul(add(R[4], ER), R[UN]), mul(c, sub(ER, EL))));
}

template <int PLANE, int DIR, bool WACT>
__device__ __forceinline__ void riemann(int rs, const float L[5], const float R[5], float gamma, float inv_gm1,
                                        float f[5]) {
  // storage slots of the sweep (to_slots in fv_tile64.cuh)
  constexpr int UN = DIR == 0 ? 1 : 2;
  constexpr int T1 = PLANE == PLANE_XY ? (DIR == 0 ? 2 : 1) : 3;
  constexpr int T2 = PLANE == PLANE_XY ? 3 : (DIR == 0 ? 2 : 1);
  if (rs == 0)
    hll<UN, T1, T2, WACT>(L, R, gamma, inv_gm1, f);
  else
    hllc<UN, T1, T2, WACT>(L, R, gamma, inv_gm1, f);
}

// consToPrim of a normalised pair state (hi = RN(hi + lo), which every writer
// of pairs leaves): as cons_to_prim_pairs, the density's reciprocal returned.
template <bool WACT>
__device__ __forceinline__ float prim_of_pairs(const float2 w[5], float gm1, float q[5]) {
  const float y = rcp(w[0].x);
  q[0] = w[0].x;
  q[1] = mul(w[1].x, y);
  q[2] = mul(w[2].x, y);
  q[3] = WACT ? mul(w[3].x, y) : 0.0f;
  const float2 k = kinetic_pair<WACT>(w[0], w[1], w[2], WACT ? w[3] : make_float2(0.0f, 0.0f));
  q[4] = mul(internal_energy(w[4], k), gm1);
  return y;
}

template <bool WACT>
__device__ __forceinline__ float prim_of_star(const float2 w[5], float gm1, float q[5]) {
  const float y = rcp(w[0].x);
  q[0] = w[0].x;
  q[1] = mul(w[1].x, y);
  q[2] = mul(w[2].x, y);
  q[3] = WACT ? mul(w[3].x, y) : 0.0f;
  q[4] = mul(w[4].x, gm1);
  return y;
}

}  // namespace m32

// Columns of a work item: a lane each, two ghost columns on either side.
constexpr int kMarchWidth = 28;

// Rows [ya, yb) of the strip whose first column is x0, by one warp (every
// lane calls it).  KIND: STAGE_RK_1 reads U^n pairs, writes U*; STAGE_RK_2
// reads U* and U^n, writes U^n+1 over U^n; STAGE_EULER reads the pairs of one
// buffer and writes the other's (flip: B -> A).  The CFL maximum and the
// non-finite flag of the result are folded into red / bad.
template <int PLANE, bool WACT, int KIND>
__device__ __forceinline__ void march_item32(const BatchInst& I, int flip, float2 dtp, int x0, int ya, int yb,
                                             float& red, bool& bad) {
  using namespace m32;
  constexpr bool STAR = KIND == STAGE_RK_2;  // the stage input is U*
  constexpr int kSz = STAR ? 4 : 8;          // bytes per input value
  constexpr unsigned kAll = 0xffffffffu;
  const Grid& G = I.G;
  const int lane = threadIdx.x & 31;
  const int rs = I.rs;
  const bool plm = G.recon == R_PLM, wb_z = PLANE == PLANE_XZ && G.recon == R_PCM_WB;
  const bool tc = G.tc != 0, visc = WACT && G.visc != 0, grav = PLANE == PLANE_XZ && G.gravity != 0;
  const float gamma = G.gamma_f, gm1 = G.gm1_f, inv_gm1 = G.inv_gm1_f;
  const float odx = G.inv_dx_f, odb = PLANE == PLANE_XY ? G.inv_dy_f : G.inv_dz_f;
  // the factors every cell shares are products of pairs, rounded once: their
  // errors, unlike a cell's, act the same way everywhere and in every step
  // (pairs, because the FP64 pipe takes 19 cycles a warp for each operation:
  // formed there they cost 8 us a step of 24^3)
  constexpr int B = PLANE == PLANE_XY ? 1 : 2;
  const float dt = dtp.x, dtdx = mul_to(dtp, I.inv_d[0]), dtdb = mul_to(dtp, I.inv_d[B]);

  const int x = x0 - 2 + lane;
  bool fa;
  const int sa = bc_source(x, G.na, G.bc_a, fa);
  const bool own = lane >= 2 && lane < 2 + kMarchWidth && x < G.na;
  const size_t fs = (size_t)G.fstride * 8;  // bytes between the fields of a state (pairs and U* alike)
  const char* in0 = reinterpret_cast<const char*>(STAR || (KIND == STAGE_EULER && flip) ? I.B.f[0] : I.A.f[0]);
  char* un0 = reinterpret_cast<char*>(I.A.f[0]);
  char* us0 = reinterpret_cast<char*>(I.B.f[0]);

#define FV_EACH_V(v) _Pragma("unroll") for (int v = 0; v < 5; ++v) if (WACT || v != 3)

  // the stored values of row r (a ghost row's source row; fb: its b velocity is mirrored)
  auto load_row = [&](int r, float2 w[5], bool& fb) {
    const int sb = bc_source(r, G.nb, G.bc_b, fb);
    const char* p = in0 + (size_t)((unsigned)sb * (unsigned)G.pitch + (unsigned)sa) * kSz;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      if (v == 3 && !WACT)
        w[v] = make_float2(0.0f, 0.0f);
      else if (STAR)
        w[v] = make_float2(*reinterpret_cast<const float*>(p + v * fs), 0.0f);
      else
        w[v] = *reinterpret_cast<const float2*>(p + v * fs);
    }
  };
  auto convert = [&](const float2 w[5], bool fb, float q[5], float& T) {
    const float y = STAR ? prim_of_star<WACT>(w, gm1, q) : prim_of_pairs<WACT>(w, gm1, q);
    if (fa) q[1] = -q[1];
    if (fb) q[2] = -q[2];
    T = mul(q[4], y);
  };

  float q0[5], q1[5];  // rows j, j+1
  float T0, T1;        // their temperatures
  float d[5];          // q1 - q0
  float Ls[5];         // face state of row j towards row j+1
  float Fb[5];         // hydrodynamic flux of face j-1/2
  float duA[5];        // increment of row j from the a faces, the diffusive flux of face j-1/2 and the per-cell terms
  float Fx[4];         // a-direction neighbour terms of row j (viscosity)
  bool fbn;
  float2 raw[5];
  {
    float2 r0[5], r1[5];
    bool fb0, fb1;
    load_row(ya - 2, r0, fb0);
    load_row(ya - 1, r1, fb1);
    load_row(ya, raw, fbn);
    convert(r0, fb0, q0, T0);
    convert(r1, fb1, q1, T1);
  }
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    if (WACT || v != 3) d[v] = sub(q1[v], q0[v]);
    Ls[v] = Fb[v] = duA[v] = 0.0f;
    if (v < 4) Fx[v] = 0.0f;
  }

  // viscous and conductive constants, dt, mu and kappa folded in
  float vx1 = 0.0f, vx43 = 0.0f, vb1 = 0.0f, vb43 = 0.0f, cx23 = 0.0f, cb23 = 0.0f, ktx = 0.0f, ktb = 0.0f;
  if (visc) {
    const float2 k43 = make_float2((float)(4.0 / 3.0), (float)(4.0 / 3.0 - (double)(float)(4.0 / 3.0)));
    const float2 k16 = make_float2((float)(1.0 / 6.0), (float)(1.0 / 6.0 - (double)(float)(1.0 / 6.0)));
    const float2 vx = mul_pair(dtp, I.mu_d[0]), vb = mul_pair(dtp, I.mu_d[B]);
    vx1 = add(vx.x, vx.y);
    vb1 = add(vb.x, vb.y);
    vx43 = mul_to(vx, k43);
    vb43 = mul_to(vb, k43);
    cx23 = mul_to(vx, k16);
    cb23 = mul_to(vb, k16);
  }
  const float cx = mul(0.25f, vx1), cb = mul(0.25f, vb1);
  if (tc) {
    ktx = mul_to(dtp, I.kappa_d2[0]);
    ktb = mul_to(dtp, I.kappa_d2[B]);
  }

  // one row: j - 2 .. ya - 1 only build up the carried state
#pragma unroll 1
  for (int j = ya - 2; j < yb; ++j) {
    // row j + 2 and the loads of row j + 3
    float qn[5], Tn;
    convert(raw, fbn, qn, Tn);
    if (j + 1 < yb) load_row(j + 3, raw, fbn);
    // row j: the cells' own values, used in the update at the end
    float2 un[5];
    float us[5];
    const size_t o = (size_t)((unsigned)j * (unsigned)G.pitch + (unsigned)sa);
    if (own && j >= ya) {
      const char* p = (KIND == STAGE_RK_2 ? un0 : in0) + o * 8;
      const char* r = us0 + o * 4;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        un[v] = (v == 3 && !WACT) ? make_float2(0.0f, 0.0f) : *reinterpret_cast<const float2*>(p + v * fs);
        if (STAR) us[v] = (v == 3 && !WACT) ? 0.0f : *reinterpret_cast<const float*>(r + v * fs);
      }
    }
    // slopes of row j + 1 along b, its a-direction differences to the right (dR) and left (dl) column
    float dn[5], m[5], dR[5], dl[5];
    FV_EACH_V(v) {
      dn[v] = sub(qn[v], q1[v]);
      dR[v] = sub(__shfl_down_sync(kAll, q1[v], 1), q1[v]);
      dl[v] = __shfl_up_sync(kAll, dR[v], 1);
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) m[v] = plm && (WACT || v != 3) ? minmod(d[v], dn[v]) : 0.0f;
    float FxN[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (WACT) {
      if (PLANE == PLANE_XY) {  // x differences of u, v across the cell, for the IY fluxes
        FxN[0] = add(dl[1], dR[1]);
        FxN[1] = add(dl[2], dR[2]);
      } else {  // right u, v (slots 1, 3) and left u, w (slots 1, 2) of the cell, for the IZ fluxes
        FxN[0] = add(q1[1], dR[1]);
        FxN[1] = add(q1[3], dR[3]);
        FxN[2] = sub(q1[1], dl[1]);
        FxN[3] = sub(q1[2], dl[2]);
      }
    }
    float duN[5], FbN[5], VbN[5], Vup[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) duN[v] = FbN[v] = VbN[v] = Vup[v] = 0.0f;
    if (j >= ya - 1) {
      // ---- a faces of row j + 1 (row yb is another item's): each lane the one right of its column
      if (j + 1 < yb) {
        float Fa[5], Va[5];
        {
          float L[5], R[5];
          FV_EACH_V(v) {
            const float s = plm ? minmod(dl[v], dR[v]) : 0.0f;
            L[v] = fma_(0.5f, s, q1[v]);
            R[v] = __shfl_down_sync(kAll, fma_(-0.5f, s, q1[v]), 1);
          }
          riemann<PLANE, 0, WACT>(rs, L, R, gamma, inv_gm1, Fa);
        }
        FV_EACH_V(v) duN[v] = mul(dtdx, sub(__shfl_up_sync(kAll, Fa[v], 1), Fa[v]));
        Va[4] = tc ? mul(ktx, sub(__shfl_down_sync(kAll, T1, 1), T1)) : 0.0f;
        float z1 = 0.0f, z3 = 0.0f;
        if (visc) {
          // e: difference over rows j, j+2 of the velocities; IX fluxes take the
          // in-plane pair (u, v) or (u, w) (slots 1, 2), the x-y IZ terms (u, w)
          const float e0 = sub(qn[1], q0[1]), e1 = sub(qn[2], q0[2]);
          const float s0 = add(e0, __shfl_down_sync(kAll, e0, 1));
          const float s1 = add(e1, __shfl_down_sync(kAll, e1, 1));
          Va[1] = fma_(vx43, dR[1], -mul(cb23, s1));
          Va[2] = fma_(vx1, dR[2], mul(cb, s0));
          Va[3] = mul(vx1, dR[3]);
          // the face's mean velocities: q + dR / 2
          const float ma = fma_(0.5f, dR[1], q1[1]), mb = fma_(0.5f, dR[2], q1[2]), mw = fma_(0.5f, dR[3], q1[3]);
          Va[4] = fma_(Va[1], ma, fma_(Va[2], mb, fma_(Va[3], mw, Va[4])));
#pragma unroll
          for (int v = 1; v < 4; ++v) duN[v] = add(duN[v], sub(Va[v], __shfl_up_sync(kAll, Va[v], 1)));
          if (PLANE == PLANE_XY) {
            // the IZ branch (Viscosity.h:214-239) in an x-y run: its two sides
            // differ only in the rows of the left column
            z1 = -mul(cx, __shfl_up_sync(kAll, sub(qn[3], q0[3]), 1));
            z3 = mul(cx23, __shfl_up_sync(kAll, e0, 1));
          }
        }
        if (tc || visc) duN[4] = add(duN[4], sub(Va[4], __shfl_up_sync(kAll, Va[4], 1)));
        if (PLANE == PLANE_XY && visc) {
          duN[1] = add(duN[1], z1);
          duN[3] = add(duN[3], z3);
          duN[4] = add(duN[4], fma_(z1, q1[1], mul(z3, q1[3])));
        }
        if (grav) duN[2] = fma_(mul(dt, G.g_f), q1[0], duN[2]);
      }
      // ---- b face between rows j and j + 1
      {
        float R[5];
        FV_EACH_V(v) R[v] = fma_(-0.5f, m[v], q1[v]);
        if (wb_z) {  // PCM_WB hydrostatic pressure in z (Update.h:27)
          Ls[4] = fma_(mul(Ls[0], G.g_dz_f), 0.5f, Ls[4]);
          R[4] = fma_(mul(R[0], G.g_dz_f), -0.5f, R[4]);
        }
        riemann<PLANE, 1, WACT>(rs, Ls, R, gamma, inv_gm1, FbN);
      }
      if (tc) VbN[4] = mul(ktb, sub(T1, T0));
      if (visc && PLANE == PLANE_XY) {  // IY (Viscosity.h:188-213)
        const float ma = fma_(0.5f, d[1], q0[1]), mb = fma_(0.5f, d[2], q0[2]), mw = fma_(0.5f, d[3], q0[3]);
        VbN[1] = fma_(vb1, d[1], mul(cx, add(Fx[1], FxN[1])));
        VbN[2] = fma_(vb43, d[2], -mul(cx23, add(Fx[0], FxN[0])));
        VbN[3] = mul(vb1, d[3]);
        VbN[4] = fma_(VbN[1], ma, fma_(VbN[2], mb, fma_(VbN[3], mw, VbN[4])));
      }
      FV_EACH_V(v) Vup[v] = VbN[v];
      if (visc && PLANE == PLANE_XZ) {
        // IZ with the reference's mix-ups: both cells of the face read their own left column
        const float ma = fma_(0.5f, d[1], q0[1]), mb = fma_(0.5f, d[2], q0[2]), mw = fma_(0.5f, d[3], q0[3]);
        const float wv = add(sub(q0[2], q0[3]), sub(q1[2], q1[3]));
        const float tzz = fma_(vb43, d[2], -fma_(cx23, add(Fx[0], FxN[0]), mul(cb23, wv)));
        const float txz = fma_(vb1, d[1], mul(cx, add(Fx[1], FxN[1])));
        const float tyz = fma_(vb1, d[3], -mul(cb, wv));
#pragma unroll
        for (int k = 0; k < 2; ++k) {  // cell j (its upper face), cell j + 1 (its lower face)
          float* V = k == 0 ? Vup : VbN;
          const float zz = fma_(add(cx23, cx23), k == 0 ? Fx[2] : FxN[2], tzz);
          const float xz = fma_(-add(cx, cx), k == 0 ? Fx[3] : FxN[3], txz);
          V[1] = xz;
          V[2] = zz;
          V[3] = tyz;
          V[4] = fma_(xz, ma, fma_(tyz, mw, fma_(zz, mb, V[4])));
        }
      }
      if (visc) {
#pragma unroll
        for (int v = 1; v < 4; ++v) duN[v] = sub(duN[v], VbN[v]);
      }
      if (tc || visc) duN[4] = sub(duN[4], VbN[4]);
    }
    // ---- row j: increments, accumulation on the pairs, CFL term
    if (own && j >= ya) {
      float du[5];
      FV_EACH_V(v) {
        du[v] = fma_(dtdb, sub(Fb[v], FbN[v]), duA[v]);
        if (v == 4 ? tc || visc : v > 0 && visc) du[v] = add(du[v], Vup[v]);
      }
      if (grav)  // half the mass fluxes of both faces (Update.h:150)
        du[4] = fma_(mul(mul(0.5f, dt), G.g_f), add(Fb[0], FbN[0]), du[4]);
      // density floor on the hydro update (Update.h:160)
      const bool low = (STAR ? add(us[0], du[0]) : add(add(un[0].x, du[0]), un[0].y)) < 1.0e-6f;
      if (KIND == STAGE_RK_1) {
        if (low) {
          un[0] = make_float2(1.0e-6f, 0.0f);
          du[0] = 0.0f;
        }
        float o5[5];
#pragma unroll
        for (int v = 0; v < 4; ++v) o5[v] = (v == 3 && !WACT) ? 0.0f : add(un[v].x, add(un[v].y, du[v]));
        // U* keeps its internal energy (fv_tile32.cuh)
        o5[4] = internal_energy(pair_add(un[4], du[4]), kinetic_star<WACT>(o5));
        char* r = us0 + o * 4;
        FV_EACH_V(v) *reinterpret_cast<float*>(r + v * fs) = o5[v];
      } else {
        float2 fin[5];
        if (KIND == STAGE_RK_2) {  // 0.5 (U^n + U* + dU)
          const float2 k = kinetic_star<WACT>(us);
          const float2 e = two_sum(k.x, us[4]);
          if (low) {
            us[0] = 1.0e-6f;
            du[0] = 0.0f;
          }
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            if (v == 3 && !WACT) {
              fin[v] = make_float2(0.0f, 0.0f);
              continue;
            }
            const float2 a = two_sum(un[v].x, v == 4 ? e.x : us[v]);
            const float2 b = two_sum(a.x, du[v]);
            const float lo = add(add(a.y, b.y), v == 4 ? add(un[v].y, add(e.y, k.y)) : un[v].y);
            const float2 r = fast_two_sum(b.x, lo);
            fin[v] = make_float2(mul(0.5f, r.x), mul(0.5f, r.y));
          }
        } else {
          if (low) {
            un[0] = make_float2(1.0e-6f, 0.0f);
            du[0] = 0.0f;
          }
#pragma unroll
          for (int v = 0; v < 5; ++v) fin[v] = (v == 3 && !WACT) ? make_float2(0.0f, 0.0f) : pair_add(un[v], du[v]);
        }
        char* p = (KIND == STAGE_RK_2 || flip ? un0 : us0) + o * 8;
        FV_EACH_V(v) *reinterpret_cast<float2*>(p + v * fs) = fin[v];
        float q[5];
        const float y = prim_of_pairs<WACT>(fin, gm1, q);
        const float cs = sqrt_(mul(mul(q[4], gamma), y));
        const float od2 = PLANE == PLANE_XY ? G.inv_dz_f : G.inv_dy_f;
        const float inv =
            fma_(add(cs, fabsf(q[1])), odx, fma_(add(cs, fabsf(q[2])), odb, mul(add(cs, fabsf(q[3])), od2)));
        bad |= !(inv <= 3.0e38f);  // NaN / inf: reported through the error flag
        red = fmaxf(red, inv);
      }
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      if (v == 3 && !WACT) continue;
      Ls[v] = fma_(0.5f, m[v], q1[v]);
      Fb[v] = FbN[v];
      duA[v] = duN[v];
      q0[v] = q1[v];
      q1[v] = qn[v];
      d[v] = dn[v];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) Fx[k] = FxN[k];
    T0 = T1;
    T1 = Tn;
  }
#undef FV_EACH_V
}

// ---- kernels ---------------------------------------------------------------

constexpr int kMarchWarps = 4;  // warps (work items in flight) per CTA
constexpr int kMarchThreads = 32 * kMarchWarps;
// Resident CTAs per SM asked of the register allocator: 4 (128 registers a
// thread, 16 warps per SM; five CTAs and 96 registers measured 824 us a step
// against 810 on shear 4096^2 and the same on RT 512x1536), but 3 where the x-z
// plane's viscous fluxes and a descriptor in shared memory come together: 4
// spill the row on its way, whose loads are then waited for at once (two RT
// 1024x3072 with conduction and viscosity 464 us a step against 374; x-y, two
// shear layers 2048^2, 456 against 471 with 3).
template <int PLANE, bool WACT, bool ONE>
constexpr int kMarchCtas = PLANE == PLANE_XZ && WACT && !ONE ? 3 : 4;

// The multi-step kernel holds both stages and spilled 20-100 bytes at 4: 3 gives
// four RT 128x384 with conduction and viscosity 23.7 us a step against 32.0, one
// 12.7 / 14.4, three shear layers 256^2 22.7 / 27.0, one 512^2 25.2 / 24.9; the
// hydro-only forms need no more than 128 registers and stay at 4 CTAs.
constexpr int kMultiCtas = 3;

// Copies the descriptor of the problem holding work item t to the warp's slot
// (binary search over the first items) unless it is there already.
__device__ __forceinline__ int march_fetch(const BatchInst* __restrict__ insts, int ninst, int t, int have,
                                           BatchInst* slot) {
  int lo = 0, hi = ninst - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (insts[mid].tile0 <= t) lo = mid;
    else hi = mid - 1;
  }
  if (lo != have) {
    __syncwarp();  // every lane is done with the previous descriptor
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(insts + lo);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(slot);
    for (int w = threadIdx.x & 31; w < (int)(sizeof(BatchInst) / 8); w += 32) dst[w] = src[w];
    __syncwarp();
  }
  return lo;
}

// One work item t (rows [by tz, by tz + tz) of strip bx of problem I) of one
// stage by the calling warp.  active / dt_step: the problem's step in flight;
// slot_next / err: its CFL maximum slot for the next step and its error flag.
template <int PLANE, bool WACT, int KIND>
__device__ __forceinline__ void march_stage_item(const BatchInst& I, int t, int flip, bool active, float2 dt_step,
                                                 unsigned long long* slot_next, int* err) {
  constexpr int W = kMarchWidth;
  const int lane = threadIdx.x & 31;
  const int lt = t - I.tile0;
  const int by = lt / I.tiles_x, bx = lt - by * I.tiles_x;
  const int x0 = bx * W, ya = by * I.tz;
  const int yb = min(ya + I.tz, I.G.nb);
  if (!active) {
    if (KIND == STAGE_EULER) {  // an inactive Euler step hands its state on
      for (int y = ya; y < yb; ++y)
        for (int x = x0 + lane; x < min(x0 + W, I.G.na); x += 32) {
          const long long o = (long long)y * I.G.pitch + x;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            if (v == 3 && !WACT) continue;
            float2* a = reinterpret_cast<float2*>(I.A.f[v]);
            float2* b = reinterpret_cast<float2*>(I.B.f[v]);
            if (flip) a[o] = b[o];
            else b[o] = a[o];
          }
        }
    }
    return;
  }
  float red = 0.0f;
  bool bad = false;
  march_item32<PLANE, WACT, KIND>(I, flip, dt_step, x0, ya, yb, red, bad);
  if (KIND != STAGE_RK_1) {
    // non-negative floats order like their bits
    const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(red));
    const bool any_bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
      if (any_bad) atomicOr(err, 1);
      atomicMax(slot_next, (unsigned long long)__double_as_longlong((double)__uint_as_float(m)));
    }
  }
}

// Persistent stage kernel: every warp pulls work items of all problems of a
// group from the queue counter, or, without one, takes the item of its own
// number (the caller's choice where the grid has a warp for each).
// That number waits in shared memory, so that the loop is the same for both: a
// test around it took up to 13 registers more, a fifth resident CTA for some.
// ONE: a group of one problem, whose descriptor `one` is read from the
// kernel's parameters (constant operands in place of registers and loads).
template <int PLANE, bool WACT, int KIND, bool ONE>
__global__ void __launch_bounds__(kMarchThreads, (kMarchCtas<PLANE, WACT, ONE>))
march_stage32(const BatchInst* __restrict__ insts, int ninst, int ntiles, unsigned* queue, int flip,
              const __grid_constant__ BatchInst one) {
  __shared__ BatchInst s_inst[ONE ? 1 : kMarchWarps];
  BatchInst& slot = s_inst[ONE ? 0 : threadIdx.x >> 5];
  const BatchInst& I = ONE ? one : slot;
  __shared__ int s_own[kMarchWarps];
  int have = -1;
  if ((threadIdx.x & 31) == 0) s_own[threadIdx.x >> 5] = blockIdx.x * kMarchWarps + (threadIdx.x >> 5);
  pdl_wait();
  for (;;) {
    int t = 0;
    if ((threadIdx.x & 31) == 0) {
      if (queue) {
        t = (int)atomicAdd(queue, 1u);
      } else {
        int* own = &s_own[threadIdx.x >> 5];
        t = *own;
        *own = ntiles;
      }
    }
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= ntiles) {
      pdl_trigger();  // no work left for this warp
      break;
    }
    if (!ONE) have = march_fetch(insts, ninst, t, have, &slot);
    StepCtrl* ctrl = I.ctrl;
    march_stage_item<PLANE, WACT, KIND>(I, t, flip, ctrl->active != 0, ctrl->dt_pair,
                                           &ctrl->slot[ctrl->parity ^ 1], &ctrl->err);
  }
}

// Problems a multi-step launch can carry (per-problem step state sits in
// shared memory).
constexpr int kMultiMaxProblems = 256;

// Several RK2 steps of a group in one cooperative launch (every CTA
// resident): per step, each CTA decides every problem's dt and active flag
// itself (step_decide on the reduced CFL maximum, the same arithmetic as the
// control kernel, so every CTA reaches the same values), then stage 1 over
// the work items of its warps (t = warp number, + warps of the grid, ...), a
// grid barrier, stage 2 (CFL maxima by atomics), a grid barrier.  Each work
// item runs the per-stage kernel's body, so the result is bit-identical to
// the per-stage launches.  The time and step counter of each problem are kept
// in shared memory during the launch and written back to the control blocks
// at its end by CTA 0; the CFL slot of the next step is zeroed by CTA 0.  A
// barrier wait that runs out sets bit 1 of every problem's error flag and
// the kernel returns.
template <int PLANE, bool WACT, bool ONE>
__global__ void __launch_bounds__(kMarchThreads, kMultiCtas)
march_multi32(const BatchInst* __restrict__ insts, int ninst, int ntiles, int nsteps, int mode_override,
              GridBarrier gb, const __grid_constant__ BatchInst one) {
  __shared__ BatchInst s_inst[ONE ? 1 : kMarchWarps];
  __shared__ double s_t[kMultiMaxProblems], s_dt[kMultiMaxProblems];
  __shared__ float2 s_dtp[kMultiMaxProblems];  // the same as pairs
  __shared__ long long s_step[kMultiMaxProblems];
  __shared__ int s_act[kMultiMaxProblems], s_par[kMultiMaxProblems], s_err[kMultiMaxProblems];
  __shared__ int s_any;
  BatchInst& slot = s_inst[ONE ? 0 : threadIdx.x >> 5];
  const BatchInst& I = ONE ? one : slot;
  const int warp0 = blockIdx.x * kMarchWarps + (threadIdx.x >> 5), nwarps = gridDim.x * kMarchWarps;
  int have = -1;
  auto timed_out = [&]() {
    if (threadIdx.x == 0)
      for (int m = 0; m < ninst; ++m) atomicOr(&insts[m].ctrl->err, 2);
  };
  for (int m = threadIdx.x; m < ninst; m += blockDim.x) {
    const StepCtrl* c = insts[m].ctrl;
    s_t[m] = c->t;
    s_step[m] = c->step;
    s_err[m] = 0;
  }
  __syncthreads();
  unsigned bar = 0;
  // every CTA has read the initial times before CTA 0 may write any control block
  if (!grid_sync(gb, bar++)) {
    timed_out();
    return;
  }
  bool decided = false;
  for (int k = 0; k < nsteps; ++k) {
    if (threadIdx.x == 0) s_any = 0;
    __syncthreads();
    for (int m = threadIdx.x; m < ninst; m += blockDim.x) {
      StepCtrl* c = insts[m].ctrl;
      double dt;
      int active;
      bool bad;
      step_decide(*c, s_t[m], s_step[m], c->err | s_err[m], mode_override, 0.0, dt, active, bad);
      const int p = (int)(s_step[m] & 1);
      if (bad) s_err[m] = 1;
      s_dt[m] = active ? dt : 0.0;
      s_dtp[m] = float_pair(s_dt[m]);
      s_act[m] = active;
      s_par[m] = p;
      if (blockIdx.x == 0) c->slot[p ^ 1] = 0ull;  // read by no CTA in this step
      if (active) {
        s_t[m] = __dadd_rn(s_t[m], dt);
        s_step[m] += 1;
        s_any = 1;
      }
    }
    __syncthreads();
    decided = true;
    if (!s_any) break;  // every CTA decides alike: no problem steps any more
    for (int t = warp0; t < ntiles; t += nwarps) {
      const int m = have = ONE ? 0 : march_fetch(insts, ninst, t, have, &slot);
      march_stage_item<PLANE, WACT, STAGE_RK_1>(I, t, 0, s_act[m] != 0, s_dtp[m], nullptr, nullptr);
    }
    if (!grid_sync(gb, bar++)) {
      timed_out();
      return;
    }
    for (int t = warp0; t < ntiles; t += nwarps) {
      const int m = have = ONE ? 0 : march_fetch(insts, ninst, t, have, &slot);
      StepCtrl* ctrl = I.ctrl;
      march_stage_item<PLANE, WACT, STAGE_RK_2>(I, t, 0, s_act[m] != 0, s_dtp[m], &ctrl->slot[s_par[m] ^ 1],
                                                   &ctrl->err);
    }
    if (!grid_sync(gb, bar++)) {
      timed_out();
      return;
    }
  }
  if (blockIdx.x == 0) {  // the control blocks as the per-stage launches leave them
    for (int m = threadIdx.x; m < ninst; m += blockDim.x) {
      StepCtrl* c = insts[m].ctrl;
      if (decided) {
        c->parity = s_par[m];
        c->active = s_act[m];
        c->dt_cur = s_dt[m];
        c->dt_pair = s_dtp[m];
      }
      c->t = s_t[m];
      c->step = s_step[m];
      if (s_err[m]) atomicOr(&c->err, 1);
    }
  }
}

typedef void (*MarchKernel)(const BatchInst*, int, int, unsigned*, int, BatchInst);
typedef void (*MarchMultiKernel)(const BatchInst*, int, int, int, int, GridBarrier, BatchInst);

// The kernels of one plane (fv_march32_xy.cu, fv_march32_xz.cu); one: a group of one problem.
MarchKernel march_kernel_xy(bool wact, int kind, bool one);
MarchKernel march_kernel_xz(bool wact, int kind, bool one);
MarchMultiKernel march_multi_kernel_xy(bool wact, bool one);
MarchMultiKernel march_multi_kernel_xz(bool wact, bool one);

template <int PLANE, bool WACT, bool ONE>
MarchKernel march_kernel_of(int kind) {
  switch (kind) {
    case STAGE_RK_1: return march_stage32<PLANE, WACT, STAGE_RK_1, ONE>;
    case STAGE_RK_2: return march_stage32<PLANE, WACT, STAGE_RK_2, ONE>;
    default: return march_stage32<PLANE, WACT, STAGE_EULER, ONE>;
  }
}

}  // namespace fv
