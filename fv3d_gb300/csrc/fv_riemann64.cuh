// fv_riemann64.cuh -- HLL and HLLC (RiemannSolvers.h) in FP64 with the
// reference's rounding and fewer FP64 instructions.
//
// States are in the slot order of the sweep (swap_component, States.h:104-111):
// r, normal velocity un, transverse t1, t2, p.  ZS names a transverse slot
// that is identically zero in a 2-D run without a third velocity (1: t1,
// 2: t2, 0: none); its terms are exact zeros in the reference arithmetic and
// are dropped.  Cheaper-but-identical steps, each returning the same bits:
//   - quotients and square roots by FP32-seeded two-operation forms (quot,
//     sqrt64 in fv_exact64.cuh), a divisor prepared once for its quotients;
//   - HLLC's max(cL, cR) as sqrt(max(cL^2, cR^2)) (sqrt is monotone and
//     correctly rounded);
//   - products with 0.5 by exponent arithmetic (half64, exact);
//   - wave-speed min / max and region tests on bit patterns (fmin_bits,
//     gt0_bits, ...: integer pipe, same results; an FP64 comparison takes 19
//     cycles of the FP64 pipe).
#pragma once

#include "fv_device.cuh"
#include "fv_plane2d.cuh"

namespace fv {

// (u^2 + t1^2) + t2^2 with the exact zero slot dropped.
template <int ZS>
__device__ __forceinline__ X64 ke_sum3(X64 un, X64 t1, X64 t2) {
  if (ZS == 1) return un * un + t2 * t2;
  if (ZS == 2) return un * un + t1 * t1;
  return (un * un + t1 * t1) + t2 * t2;
}

// computeFlux (States.h:114-127) given e = p/(gamma-1).
template <int ZS>
__device__ __forceinline__ void euler_flux64(const Slots<X64>& q, X64 e, X64 F[5]) {
  const X64 Ek = half_of(q.r) * ke_sum3<ZS>(q.un, q.t1, q.t2);
  const X64 E = e + Ek;
  F[0] = q.r * q.un;
  F[1] = F[0] * q.un + q.p;
  F[2] = ZS == 1 ? 0.0 : F[0] * q.t1;
  F[3] = ZS == 2 ? 0.0 : F[0] * q.t2;
  F[4] = (q.p + E) * q.un;
}

// primToCons (States.h:20-31) without the internal energy: u[4] = the sum of
// the squared momenta / 2, still to be divided by the density.
template <int ZS>
__device__ __forceinline__ void prim_to_cons64(const Slots<X64>& q, X64 u[5]) {
  u[0] = q.r;
  u[1] = q.r * q.un;
  u[2] = ZS == 1 ? X64(0.0) : q.r * q.t1;
  u[3] = ZS == 2 ? X64(0.0) : q.r * q.t2;
  u[4] = half_of(ke_sum3<ZS>(u[1], u[2], u[3]));
}

// HLL with Davis wave speeds, RiemannSolvers.h:6-36.
// pout, when given, receives the interface pressure of RiemannSolvers.h:24-33
// (used only by the z-boundary flux overrides of Update.h:131-143).
template <int ZS>
__device__ __forceinline__ void hll64(const Slots<X64>& L, const Slots<X64>& R, const Consts64& K,
                                      X64 flux[5], X64* pout = nullptr) {
  // each density, prepared once, divides twice (the sound speed's p*gamma and,
  // in the star region, the kinetic energy)
  const Div64 rhoL = prepare_div(L.r), rhoR = prepare_div(R.r);
  X64 aL = L.p * K.gamma, aR = R.p * K.gamma;
  quot_pair(aL, rhoL, aR, rhoR);
  sqrt_pair(aL, aR);
  const X64 SL = fmin_bits(L.un - aL, R.un - aR);
  const X64 SR = fmax_bits(L.un + aL, R.un + aR);
  X64 e[2] = {L.p, R.p};
  quots(e, s_cell64.gm1);
  const X64 eL = e[0], eR = e[1];
  X64 FL[5], FR[5];
  euler_flux64<ZS>(L, eL, FL);
  euler_flux64<ZS>(R, eR, FR);
  if (ge0_bits(SL)) {
#pragma unroll
    for (int v = 0; v < 5; ++v) flux[v] = FL[v];
    if (pout) *pout = L.p;
  } else if (le0_bits(SR)) {
#pragma unroll
    for (int v = 0; v < 5; ++v) flux[v] = FR[v];
    if (pout) *pout = R.p;
  } else {
    if (pout) *pout = half_of(L.p + R.p);
    X64 uL[5], uR[5];
    prim_to_cons64<ZS>(L, uL);
    prim_to_cons64<ZS>(R, uR);
    quot_pair(uL[4], rhoL, uR[4], rhoR);
    uL[4] = uL[4] + eL;
    uR[4] = uR[4] + eR;
    const X64 slsr = SL * SR;
    const Div64 den = prepare_div(SR - SL);
    constexpr int N = ZS ? 4 : 5;
    X64 f[N];
    int n = 0;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      if ((ZS == 1 && v == 2) || (ZS == 2 && v == 3)) continue;
      f[n++] = (FL[v] * SR - FR[v] * SL) + (uR[v] - uL[v]) * slsr;
    }
    quots(f, den);
    n = 0;
#pragma unroll
    for (int v = 0; v < 5; ++v) flux[v] = (ZS == 1 && v == 2) || (ZS == 2 && v == 3) ? X64(0.0) : f[n++];
  }
}

// HLLC, RiemannSolvers.h:39-112; the kinetic energy uses un and t1 only, as
// the reference does.
// pout as for hll64 (RiemannSolvers.h:81-104: pL, p*, p*, pR by region).
// KE3 (corrected physics): the kinetic energy of all three velocities.
template <int ZS, bool KE3 = false>
__device__ __forceinline__ void hllc64(const Slots<X64>& L, const Slots<X64>& R, const Consts64& K,
                                       X64 flux[5], X64* pout = nullptr) {
  const X64 rL = L.r, uL = L.un, pL = L.p;
  const X64 rR = R.r, uR = R.un, pR = R.p;
  const X64 kL = KE3 ? ke_sum3<ZS>(uL, L.t1, L.t2) : (ZS == 1 ? uL * uL : uL * uL + L.t1 * L.t1);
  const X64 kR = KE3 ? ke_sum3<ZS>(uR, R.t1, R.t2) : (ZS == 1 ? uR * uR : uR * uR + R.t1 * R.t1);
  const X64 EL = half_of(rL) * kL + pL * K.inv_gm1;
  const X64 ER = half_of(rR) * kR + pR * K.inv_gm1;
  X64 c2L = pL * K.gamma, c2R = pR * K.gamma;
  quot_pair(c2L, prepare_div(rL), c2R, prepare_div(rR));
  const X64 cmax = sqrt64(fmax_bits(c2L, c2R));
  const X64 SL = fmin_bits(uL, uR) - cmax;
  const X64 SR = fmax_bits(uL, uR) + cmax;
  const X64 rcL = rL * (uL - SL);
  const X64 rcR = rR * (SR - uR);
  const Div64 D = prepare_div(rcR + rcL);
  X64 s[2] = {rcR * uR + rcL * uL + (pL - pR), rcR * pL + rcL * pR + rcL * rcR * (uL - uR)};
  quots(s, D);
  const X64 uS = s[0], pS = s[1];
  X64 sr, su, st1, st2, sp, E;
  if (gt0_bits(SL)) {
    sr = rL; su = uL; st1 = L.t1; st2 = L.t2; sp = pL; E = EL;
  } else if (gt0_bits(uS) || gt0_bits(SR)) {
    // star regions, tested in the reference's order: uS > 0 -> left star,
    // otherwise SR > 0 -> right star
    const bool left = gt0_bits(uS);
    const X64 rK = left ? rL : rR, uK = left ? uL : uR, pK = left ? pL : pR, EK = left ? EL : ER;
    const X64 SK = left ? SL : SR;
    const Div64 den = prepare_div(SK - uS);
    X64 k[2] = {rK * (SK - uK), (SK - uK) * EK - pK * uK + pS * uS};
    quots(k, den);
    sr = k[0];
    E = k[1];
    su = uS;
    sp = pS;
    st1 = left ? L.t1 : R.t1;
    st2 = left ? L.t2 : R.t2;
  } else {
    sr = rR; su = uR; st1 = R.t1; st2 = R.t2; sp = pR; E = ER;
  }
  if (pout) *pout = sp;
  flux[0] = sr * su;
  flux[1] = flux[0] * su + sp;
  flux[2] = ZS == 1 ? 0.0 : flux[0] * st1;
  flux[3] = ZS == 2 ? 0.0 : flux[0] * st2;
  flux[4] = (E + sp) * su;
}

}  // namespace fv
