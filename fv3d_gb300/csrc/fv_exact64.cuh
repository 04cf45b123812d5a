// fv_exact64.cuh -- FP64 building blocks that round exactly like the plain
// IEEE operations they replace, with fewer FP64-pipe instructions.
//
// On GB300 the FP64 pipe executes about 1/64 of the FP32 rate, so the plain
// FP64 path is bound by its count of FP64 instructions.  Every helper here
// returns bit-for-bit the value of the reference expression it stands for
// (for finite operands away from the subnormal range), so the FP64 stage
// kernel stays bit-identical to the reference's CPU arithmetic.
//
// Division by a value whose correctly rounded reciprocal is known uses
// Markstein's correction (P. Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990; see
// also Muller et al., Handbook of Floating-Point Arithmetic, the theorem on
// correcting a quotient with a fused multiply-add): with y = RN(1/b) and
// q0 = RN(a*y), which lies within one ulp of a/b, the residual
// r = a - b*q0 is exactly representable (one fma) and RN(q0 + r*y) = RN(a/b).
#pragma once

#include <cuda_runtime.h>

namespace fv {

// ---- FP64 sums and products as three-register fused operations ------------
// On GB300 a DFMA whose operands are all registers occupies the FP64 pipe for
// 16 cycles per warp and SM; DADD, DMUL and a DFMA with a constant or
// immediate operand take 19 (clock64 around 8,000 of each, 8 warps per SM).
// So a + b is issued as fma(a, 1, b) and a * b as fma(a, b, -0): one rounding
// of the same exact value, and the same zero: x * 1 is x, and adding -0
// changes no product, not even a zero one.  The 1 and the -0 must sit in
// registers the compiler cannot see through: they are read from shared memory
// (opaque64_init puts them there at the start of a kernel).
struct Opaque64 {
  double one, nzero, half, two_thirds, four_thirds;
};
static __shared__ Opaque64 s_op64;

// Every thread of a kernel that uses X64 calls it first; a __syncthreads must
// follow before the first operation.
__device__ __forceinline__ void opaque64_init() {
  if (threadIdx.x == 0) {
    Opaque64 o;  // through asm, so that no stored value is a known constant
    asm volatile("mov.f64 %0, 0d3FF0000000000000;" : "=d"(o.one));
    asm volatile("mov.f64 %0, 0d8000000000000000;" : "=d"(o.nzero));
    asm volatile("mov.f64 %0, 0d3FE0000000000000;" : "=d"(o.half));
    o.two_thirds = 2.0 / 3.0 * o.one;
    o.four_thirds = 4.0 / 3.0 * o.one;
    s_op64 = o;
  }
}

// Copies a launch parameter to shared memory (every thread calls it; a
// __syncthreads must follow): its FP64 fields then reach the arithmetic as
// registers, where a constant-bank operand would cost three more cycles.
template <class P>
__device__ __forceinline__ void param_to_shared(const P& src, P& dst) {
  static_assert(sizeof(P) % 4 == 0, "copied as 4-byte words");
  const unsigned* s = reinterpret_cast<const unsigned*>(&src);
  unsigned* d = reinterpret_cast<unsigned*>(&dst);
  for (unsigned w = threadIdx.x; w < sizeof(P) / 4; w += blockDim.x) d[w] = s[w];
}

// A double whose operators are the forms above.
struct X64 {
  double v;
  __device__ __forceinline__ X64() {}
  __device__ __forceinline__ X64(double x) : v(x) {}
};
__device__ __forceinline__ X64 operator+(X64 a, X64 b) { return fma(a.v, s_op64.one, b.v); }
__device__ __forceinline__ X64 operator-(X64 a, X64 b) { return fma(-b.v, s_op64.one, a.v); }
__device__ __forceinline__ X64 operator*(X64 a, X64 b) { return fma(a.v, b.v, s_op64.nzero); }
__device__ __forceinline__ X64 operator-(X64 a) { return -a.v; }
__device__ __forceinline__ X64& operator+=(X64& a, X64 b) { return a = a + b; }

// 2/3 and 4/3 (Viscosity.h:45-46) as operands of either precision.
template <class T>
__device__ __forceinline__ T two_thirds_of();
template <class T>
__device__ __forceinline__ T four_thirds_of();
template <>
__device__ __forceinline__ float two_thirds_of<float>() { return 2.0f / 3.0f; }
template <>
__device__ __forceinline__ float four_thirds_of<float>() { return 4.0f / 3.0f; }
template <>
__device__ __forceinline__ X64 two_thirds_of<X64>() { return s_op64.two_thirds; }
template <>
__device__ __forceinline__ X64 four_thirds_of<X64>() { return s_op64.four_thirds; }

// RN(a / b) given y = RN(1 / b): three fused operations instead of a full
// IEEE division.
__device__ __forceinline__ X64 div_by_rcp(X64 a, X64 b, X64 y) {
  const X64 q0 = a * y;
  const double r = fma(-b.v, q0.v, a.v);
  return fma(r, y.v, q0.v);
}

// Correctly rounded reciprocal, quotient and square root.
__device__ __forceinline__ X64 rcp64(X64 x) { return 1.0 / x.v; }
__device__ __forceinline__ X64 div64(X64 a, X64 b) { return a.v / b.v; }
__device__ __forceinline__ X64 sqrt64(X64 x) { return sqrt(x.v); }

// (x) / d for a cell size d: an exact multiplication by 1/d when d is a power
// of two (then 1/d is exact and scaling by it rounds nowhere), else the
// corrected quotient above (exact for any d).  P2 is a compile-time choice:
// the kernels branch once, uniformly, on "every cell size is a power of two",
// because a per-call select would issue both forms.
template <bool P2>
__device__ __forceinline__ X64 div_cell(X64 x, X64 d, X64 inv_d) {
  return P2 ? x * inv_d : div_by_rcp(x, d, inv_d);
}

// The reference formula of minmod, out of line: the rare operands that reach
// it (NaN, infinities, a product that may underflow) take a real branch, so
// its FP64 instructions are not issued on the common path.
static __device__ __noinline__ double minmod_rare(double dL, double dR) {
  if (__dmul_rn(dL, dR) < 0.0) return 0.0;
  return fabs(dL) < fabs(dR) ? dL : dR;
}

// minmod of Update.h:73-80 -- 0 if dL*dR < 0, else the argument of smaller
// magnitude, ties to dR -- decided on the bit patterns without FP64
// instructions.  The sign test equals `dL*dR < 0` whenever the product cannot
// underflow to zero (exponent sum check) and neither operand is NaN; the
// magnitude test equals `fabs(dL) < fabs(dR)` because IEEE magnitudes order
// like their bit patterns.  The remaining cases take the reference formula.
__device__ __forceinline__ X64 minmod_exact(X64 xL, X64 xR) {
  const double dL = xL.v, dR = xR.v;
  const unsigned long long a = (unsigned long long)__double_as_longlong(dL);
  const unsigned long long b = (unsigned long long)__double_as_longlong(dR);
  const unsigned long long ma = a & 0x7fffffffffffffffull, mb = b & 0x7fffffffffffffffull;
  const unsigned long long kInf = 0x7ff0000000000000ull;
  if (ma <= kInf && mb <= kInf) {
    if (ma == 0ull || mb == 0ull || ((a ^ b) >> 63) == 0ull) return ma < mb ? dL : dR;
    const unsigned ea = (unsigned)(ma >> 52), eb = (unsigned)(mb >> 52);
    if (ea != 0u && eb != 0u && ea + eb >= 972u) return 0.0;  // |dL*dR| >= 2^-1074
  }
  return minmod_rare(dL, dR);
}

// Comparisons and C99 fmin / fmax on bit patterns (integer pipe; the FP64
// pipe's DSETP / DMNMX issue at the FP64 rate).  For non-NaN operands each
// returns what the FP64 instruction returns -- min / max give one operand
// exactly; where the two operands are +0 and -0 the sign of the zero chosen
// may differ, which none of the callers can observe (their results do not
// depend on the sign of a zero speed or of a zero compared with zero).  A
// NaN operand is handled as fmin / fmax and the IEEE comparisons do.
__device__ __forceinline__ bool is_nan_bits(long long b) { return (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL; }

// Signed-integer key that orders like the double (negative values reversed).
__device__ __forceinline__ long long order_key(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffLL); }

__device__ __forceinline__ X64 fmin_bits(X64 a, X64 b) {
  const long long x = __double_as_longlong(a.v), y = __double_as_longlong(b.v);
  if (is_nan_bits(x)) return b;
  if (is_nan_bits(y)) return a;
  return order_key(y) < order_key(x) ? b : a;
}

__device__ __forceinline__ X64 fmax_bits(X64 a, X64 b) {
  const long long x = __double_as_longlong(a.v), y = __double_as_longlong(b.v);
  if (is_nan_bits(x)) return b;
  if (is_nan_bits(y)) return a;
  return order_key(y) > order_key(x) ? b : a;
}

// x >= 0.0, x > 0.0 and x <= 0.0 as IEEE comparisons (false for NaN).
__device__ __forceinline__ bool ge0_bits(X64 v) {
  const long long b = __double_as_longlong(v.v);
  return (b >= 0 && b <= 0x7ff0000000000000LL) || b == (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool gt0_bits(X64 v) {
  const long long b = __double_as_longlong(v.v);
  return b > 0 && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool le0_bits(X64 v) {
  const long long b = __double_as_longlong(v.v);
  return b == 0 || (b < 0 && !is_nan_bits(b));
}

// !(v <= limit) for a limit > 0 and a v that is >= 0 or NaN (a CFL sum).
__device__ __forceinline__ bool above_bits(double v, double limit) {
  const long long b = __double_as_longlong(v);
  return !(b >= 0 && b <= __double_as_longlong(limit));
}

// RN(0.5 * x) with integer instructions only.  For |x| >= 2^-1021 the
// product is exact: x with its exponent decremented (only the high word
// changes).  Below that the halved value is subnormal: the magnitude in units
// of 2^-1074 is halved with round-to-nearest-even.  Infinities and NaN are
// returned unchanged.
__device__ __forceinline__ double half64(double x) {
  const int hi = __double2hiint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  if (e - 2u < 0x7fdu) return __hiloint2double(hi - 0x100000, __double2loint(x));
  if (e == 0x7ffu) return x;
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long m = b & 0x7fffffffffffffffull;
  const unsigned long long r = (m >> 1) + (m & (m >> 1) & 1ull);
  return __longlong_as_double((long long)((b & 0x8000000000000000ull) | r));
}

// 0.5 * x for either precision (FP32 keeps its multiply: that pipe is fast).
__device__ __forceinline__ X64 half_of(X64 x) { return half64(x.v); }
__device__ __forceinline__ float half_of(float x) { return 0.5f * x; }

// Face-state reconstruction q + (slope*sign)*0.5 (Update.h:21): the product
// with +-0.5 is exact, so a single fused operation rounds identically.
__device__ __forceinline__ X64 recon_plus(X64 q, X64 slope) { return fma(slope.v, s_op64.half, q.v); }
__device__ __forceinline__ X64 recon_minus(X64 q, X64 slope) { return fma(-slope.v, s_op64.half, q.v); }

// Constants every FP64 kernel needs, computed on the host with IEEE double
// arithmetic exactly as the reference evaluates them.
struct Consts64 {
  X64 gamma;     // gamma0
  X64 gm1;       // gamma0 - 1 (exact for 1 < gamma0 < 3)
  X64 inv_gm1;   // RN(1 / (gamma0 - 1)), also HLLC's `entho`
};

}  // namespace fv
