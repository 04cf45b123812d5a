// fv_exact64.cuh -- FP64 building blocks that round exactly like the plain
// IEEE operations they replace, with fewer FP64-pipe instructions.
//
// On GB300 the FP64 pipe executes 1/59 of the FP32 rate at most (measured:
// 628 G FMA/s with three register operands against 36,750), so the plain
// FP64 path is bound by its count of FP64 instructions.  Every helper here
// returns bit-for-bit the value of the reference expression it stands for
// (for finite operands away from the subnormal range), so the FP64 stage
// kernel stays bit-identical to the reference's CPU arithmetic.
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

// ---- correctly rounded quotients and square roots, two FP64 operations each --
// CUDA's FP64 division and square root take 137 and 143 cycles of the FP64
// pipe per warp and SM, a reciprocal 86; the FP32 and integer pipes beside it
// are all but idle (32 other instructions per DFMA cost nothing: 497 G
// DFMA/s with them, 498 without).  So the result is first formed to about
// 2^-45 from FP32 operations on the significands, split into an unevaluated
// pair of floats (T. J. Dekker, "A floating-point technique for extending the
// available precision", Numer. Math. 18, 1971), and made a double Q by
// integer additions.  Then, for a quotient a / b,
//     r = fma(-b, Q, a),   result = fma(r, y, Q),   y = 1/b to 2^-24,
// (a square root: r = fma(-G, G, x), result = fma(r, h, G), h = 1/(2 sqrt x)):
// the value rounded by the last operation is within 2^-15 units in the last
// place of the exact one.  Whether that decides the rounding is tested (A.
// Ziv, "Fast evaluation of elementary mathematical functions with correctly
// rounded last bit", ACM TOMS 17(3), 1991): r y in units in the last place of
// Q, computed in FP32 (error below 2^-13), must lie at least 2^-12 away from
// every half, and is taken only up to 2^10 (beyond, neither bound holds; Q is
// within 2^9 of the result unless the pair crossed a power of two).  Where it
// does not (one result in 2,048), and for operands so
// small or large that a step could leave the normal range (divisors outside
// 2^-150 .. 2^150, numerators outside 2^-750 .. 2^800, roots outside 2^-700 ..
// 2^700), the IEEE operation itself is called.  The last place of a quotient is
// that of Q's own binade, which the seed need not share: a seed up to two FP32
// units below a power of two can belong to a quotient above it.  A Q within
// 2^10 of its last places of a power of two, where the spacing changes between
// it and the result, is taken only if r is zero (an exact quotient).
static __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_ieee(double x) { return sqrt(x); }

// The significand of x as h + l 2^-23: h in [1, 2) (23 bits after the point),
// l in [0, 1) the next 23 of the 29 bits left.
__device__ __forceinline__ void split_significand(unsigned hi, unsigned lo, unsigned expo, float& h, float& l) {
  h = __uint_as_float((expo << 23) | (__funnelshift_l(lo, hi, 3) & 0x007fffffu));
  l = __uint_as_float(0x3f800000u | ((lo >> 6) & 0x007fffffu)) - 1.0f;
}

// Whether the fraction of t >= 0 (a correction in units in the last place)
// stays 2^-12 clear of a half.
__device__ __forceinline__ bool clear_of_half(float t) {
  const float n = __fadd_rn(t, 12582912.0f) - 12582912.0f;  // nearest integer (t < 2^12)
  return fabsf(t - n) < 0.5f - 0x1p-12f;
}

// The largest correction taken, in units in the last place, and the high word
// (as a float's exponent) of the residual it belongs to: a quotient's
// correction is at most twice the residual, a root's at most half.
constexpr unsigned long long kCorrection = 1ull << 10;
constexpr int kMaxQuotRes = (127 + 9) << 20, kMaxRootRes = (127 + 11) << 20;

// A divisor prepared for several quotients.
struct Div64 {
  double b, y;  // the divisor, 1/b to 2^-24
  float h, l;   // its significand (split_significand; l scaled by 2^-23)
  float r;      // 1/(h + l) to 2^-24
  bool ok;      // 2^-150 <= |b| < 2^150
};

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ Div64 prepare_div(X64 b) {
  Div64 D;
  D.b = b.v;
  const unsigned hi = (unsigned)__double2hiint(b.v), lo = (unsigned)__double2loint(b.v);
  const unsigned e = hi & 0x7ff00000u;
  D.ok = e - (873u << 20) < (300u << 20);
  split_significand(hi, lo, 127u, D.h, D.l);
  D.l *= 0x1p-23f;
  const float r0 = rcp_approx(D.h);
  const float err = __fmaf_rn(-D.l, r0, __fmaf_rn(-D.h, r0, 1.0f));
  D.r = __fmaf_rn(r0, err, r0);
  const unsigned rb = __float_as_uint(D.r);  // 2^-1 < r <= 1
  D.y = __hiloint2double((int)(((rb >> 3) + ((896u + 1023u) << 20) - e) | (hi & 0x80000000u)), (int)(rb << 29));
  return D;
}

// RN(a / D.b) where `good`; else the caller takes the IEEE operation.
__device__ __forceinline__ double quot_core(double a, const Div64& D, bool& good) {
  const unsigned ahi = (unsigned)__double2hiint(a), alo = (unsigned)__double2loint(a);
  const unsigned bhi = (unsigned)__double2hiint(D.b);
  const unsigned ea = ahi & 0x7ff00000u, eb = bhi & 0x7ff00000u;
  float ah, al;
  split_significand(ahi, alo, 127u, ah, al);
  const float qh = __fmul_rn(ah, D.r);
  const float rem = __fmaf_rn(al, 0x1p-23f, __fmaf_rn(-qh, D.l, __fmaf_rn(-qh, D.h, ah)));
  const float ql = __fmul_rn(rem, D.r);
  const unsigned qb = __float_as_uint(qh);
  const bool big = qb >= 0x3f800000u;  // qh in [1, 2), else in [1/2, 1)
  const int n = __float2int_rn(__fmul_rn(ql, big ? 0x1p49f : 0x1p50f));  // ql in units of 8 last places
  const long long q = (((long long)((qb >> 3) + (896u << 20) + ea - eb) << 32) | (long long)(qb << 29)) +
                      ((long long)n << 3);
  const unsigned sign = (ahi ^ bhi) & 0x80000000u;
  const double Q = __longlong_as_double(q ^ ((long long)sign << 32));
  const double res = fma(-D.b, Q, a);
  const double out = fma(res, D.y, Q);
  // the rounding test, in units in the last place of Q's binade: [1, 2) times a power of two, or [1/2, 1)
  const bool upper = (int)(q >> 32) >= (int)(ea - eb + (1023u << 20));
  const unsigned rhi = (unsigned)__double2hiint(res) & 0x7fffffffu, rlo = (unsigned)__double2loint(res);
  const int x = (int)(rhi - ea + ((127u + 52u) << 20));
  float t = __fmul_rn(x > 0 ? __uint_as_float(__funnelshift_l(rlo, (unsigned)x, 3)) : 0.0f, D.r);
  t = upper ? t : t + t;
  const bool edge = (((unsigned long long)q + kCorrection) << 12) < (kCorrection << 13) && (rhi | rlo) != 0u;
  const bool zero = ((ahi << 1) | alo) == 0u;  // 0 / b
  good = D.ok && (zero || (ea - (273u << 20) < (1550u << 20) && x < kMaxQuotRes && clear_of_half(t) && !edge));
  return zero ? __hiloint2double((int)sign, 0) : out;
}

// Out of line, as the square roots: inlined into every face and cell these
// made a translation unit take minutes to compile, and a call costs only
// instruction issue, of which there is plenty.  One call takes as many
// quotients as the code has at hand: they overlap in it (a quotient alone
// takes 356 cycles from operands to result), calls do not.
template <int N>
struct Vals {
  double v[N];
};
template <int N>
static __device__ __noinline__ Vals<N> quots_call(Vals<N> a, Div64 D) {
  Vals<N> q;
  bool good[N], all = true;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    q.v[i] = quot_core(a.v[i], D, good[i]);
    all = all && good[i];
  }
  if (!all) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (!good[i]) q.v[i] = div_ieee(a.v[i], D.b);
  }
  return q;
}
static __device__ __noinline__ Vals<2> quot_pair_call(double a, Div64 A, double b, Div64 B) {
  Vals<2> q;
  bool ga, gb;
  q.v[0] = quot_core(a, A, ga);
  q.v[1] = quot_core(b, B, gb);
  if (!ga) q.v[0] = div_ieee(a, A.b);
  if (!gb) q.v[1] = div_ieee(b, B.b);
  return q;
}

// RN(a / D.b); of several numerators, in place; of two with a divisor each.
__device__ __forceinline__ X64 quot(X64 a, const Div64& D) { return quots_call<1>(Vals<1>{{a.v}}, D).v[0]; }
template <int N>
__device__ __forceinline__ void quots(X64 (&a)[N], const Div64& D) {
  Vals<N> x;
#pragma unroll
  for (int i = 0; i < N; ++i) x.v[i] = a[i].v;
  x = quots_call<N>(x, D);
#pragma unroll
  for (int i = 0; i < N; ++i) a[i] = x.v[i];
}
__device__ __forceinline__ void quot_pair(X64& a, const Div64& A, X64& b, const Div64& B) {
  const Vals<2> q = quot_pair_call(a.v, A, b.v, B);
  a = q.v[0];
  b = q.v[1];
}

// RN(a / b) for a divisor used once.
__device__ __forceinline__ X64 div64(X64 a, X64 b) { return quot(a, prepare_div(b)); }

// RN(sqrt(x)) where `good`.
__device__ __forceinline__ double sqrt_core(double x, bool& good) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)(hi >> 20) - 1023;
  const int odd = e & 1, half_e = (e - odd) >> 1;
  float mh, ml;  // x = (mh + ml) 4^half_e, mh in [1, 4)
  split_significand(hi, lo, (unsigned)(127 + odd), mh, ml);
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(mh));
  const float g0 = __fmul_rn(mh, y0);
  const float y1 = __fmaf_rn(__fmul_rn(0.5f, y0), __fmaf_rn(-g0, y0, 1.0f), y0);
  const float h = __fmul_rn(0.5f, y1);
  const float rem = __fmaf_rn(ml, odd ? 0x1p-22f : 0x1p-23f, __fmaf_rn(-g0, g0, mh));
  const float c = __fmul_rn(rem, h);
  const float gl = __fmaf_rn(__fmul_rn(c, c), h, c);  // (g0 + gl)^2 = mh + ml
  const unsigned gb = __float_as_uint(g0), hb = __float_as_uint(h);
  const int n = __float2int_rn(__fmul_rn(gl, 0x1p49f));
  const long long g = (((long long)((gb >> 3) + (896u << 20) + ((unsigned)half_e << 20)) << 32) |
                       (long long)(gb << 29)) + ((long long)n << 3);
  const double G = __longlong_as_double(g);
  const double H = __hiloint2double((int)((hb >> 3) + (896u << 20) - ((unsigned)half_e << 20)), (int)(hb << 29));
  const double res = fma(-G, G, x);
  const double out = fma(res, H, G);
  const unsigned rhi = (unsigned)__double2hiint(res) & 0x7fffffffu, rlo = (unsigned)__double2loint(res);
  const int s = (int)(rhi - ((unsigned)(2 * half_e + 1023) << 20) + ((127u + 52u) << 20));
  const float t = __fmul_rn(s > 0 ? __uint_as_float(__funnelshift_l(rlo, (unsigned)s, 3)) : 0.0f, h);
  const bool inside = gb - 0x3f800001u < 0x007ffffeu;  // 1 < g0 < 2, not beside either
  good = hi - (323u << 20) < (1400u << 20) && s < kMaxRootRes && clear_of_half(t) &&
                    (inside || (rhi | rlo) == 0u);
  return out;
}

static __device__ __noinline__ double sqrt_call(double x) {
  bool good;
  const double s = sqrt_core(x, good);
  return good ? s : sqrt_ieee(x);
}
static __device__ __noinline__ Vals<2> sqrt_pair_call(double a, double b) {
  Vals<2> s;
  bool ga, gb;
  s.v[0] = sqrt_core(a, ga);
  s.v[1] = sqrt_core(b, gb);
  if (!ga) s.v[0] = sqrt_ieee(a);
  if (!gb) s.v[1] = sqrt_ieee(b);
  return s;
}

// RN(sqrt(x)).
__device__ __forceinline__ X64 sqrt64(X64 x) { return sqrt_call(x.v); }
__device__ __forceinline__ void sqrt_pair(X64& a, X64& b) {
  const Vals<2> s = sqrt_pair_call(a.v, b.v);
  a = s.v[0];
  b = s.v[1];
}

// The reference formula of minmod, out of line: the rare operands that reach
// it (NaN, infinities, a product that may underflow) take a real branch, so
// its FP64 instructions are not issued on the common path.
static __device__ __noinline__ double minmod_rare(double dL, double dR) {
  if (__dmul_rn(dL, dR) < 0.0) return 0.0;
  return fabs(dL) < fabs(dR) ? dL : dR;
}

// Bits of x without the sign, shifted up by one: they order like |x|.  (A
// mask in place of the shift is recognised as an absolute value and issued as
// a DADD.)
__device__ __forceinline__ unsigned long long abs_key(double x) {
  return (unsigned long long)__double_as_longlong(x) << 1;
}
constexpr unsigned long long kInfKey = 0xffe0000000000000ull;

// minmod of Update.h:73-80 -- 0 if dL*dR < 0, else the argument of smaller
// magnitude, ties to dR -- decided on the bit patterns without FP64
// instructions.  The sign test equals `dL*dR < 0` whenever the product cannot
// underflow to zero (exponent sum check) and neither operand is NaN; the
// magnitude test equals `fabs(dL) < fabs(dR)` because IEEE magnitudes order
// like their bit patterns.  The remaining cases take the reference formula.
__device__ __forceinline__ X64 minmod_exact(X64 xL, X64 xR) {
  const double dL = xL.v, dR = xR.v;
  const unsigned long long ma = abs_key(dL), mb = abs_key(dR);
  if (ma <= kInfKey && mb <= kInfKey) {
    const bool opposite = (__double2hiint(dL) ^ __double2hiint(dR)) < 0;
    if (!opposite || ma == 0ull || mb == 0ull) return ma < mb ? dL : dR;
    const unsigned ea = (unsigned)(ma >> 53), eb = (unsigned)(mb >> 53);
    if (ea != 0u && eb != 0u && ea + eb >= 972u) return 0.0;  // |dL*dR| >= 2^-1074
  }
  return minmod_rare(dL, dR);
}

// x with its sign flipped when f (integer: a negation selected by a flag is
// issued as a DADD).
__device__ __forceinline__ X64 flip_sign(X64 x, bool f) {
  return __hiloint2double(__double2hiint(x.v) ^ (f ? (int)0x80000000 : 0), __double2loint(x.v));
}

// Comparisons and C99 fmin / fmax on bit patterns (integer pipe; the FP64
// pipe's DSETP / DMNMX issue at the FP64 rate).  For non-NaN operands each
// returns what the FP64 instruction returns -- min / max give one operand
// exactly; where the two operands are +0 and -0 the sign of the zero chosen
// may differ, which none of the callers can observe (their results do not
// depend on the sign of a zero speed or of a zero compared with zero).  A
// NaN operand is handled as fmin / fmax and the IEEE comparisons do.
__device__ __forceinline__ bool is_nan_bits(long long b) { return ((unsigned long long)b << 1) > kInfKey; }

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
  X64 inv_gm1;   // RN(1 / (gamma0 - 1)), also HLLC's `entho`
};

}  // namespace fv
