// fv_plane2d.cuh -- per-cell FP64 helpers shared by the 2-D kernels.
//
// A 2-D run stores its state in "storage order" (rho, m_a, m_b, m_c, E):
// m_a is the x-momentum, m_b the momentum along the second active axis (y in
// the x-y plane, z in the x-z plane) and m_c the momentum along the
// degenerate axis.  These helpers restate the reference's per-cell formulas in
// that order, rounding exactly as the reference does.
#pragma once

#include "fv_device.cuh"
#include "fv_exact64.cuh"

namespace fv {

// The constant divisors of a problem -- cell sizes and gamma - 1 -- prepared
// in shared memory once per kernel (or work item).
struct CellDiv64 {
  Div64 d[3];     // dx, dy, dz
  Div64 gm1;
  double inv[3];  // RN(1/d)
  int pow2;       // every cell size is a power of two: 1/d is exact
};
static __shared__ CellDiv64 s_cell64;

// Every thread calls it, after a __syncthreads that follows opaque64_init and
// the store of G; another must come before the first division.
__device__ __forceinline__ void cell_div_init(const Grid& G) {
  const int t = threadIdx.x;
  if (t < 3) {
    s_cell64.d[t] = prepare_div(t == 0 ? G.dx : (t == 1 ? G.dy : G.dz));
    s_cell64.inv[t] = t == 0 ? G.inv_dx : (t == 1 ? G.inv_dy : G.inv_dz);
  }
  if (t == 3) s_cell64.gm1 = prepare_div(G.gm1);
  if (t == 4) s_cell64.pow2 = G.pow2_all;
}

// x / d for the cell size of an axis: an exact multiplication by 1/d when the
// cell sizes are powers of two (then 1/d is exact and scaling by it rounds
// nowhere; a uniform branch), else a quotient.
__device__ __forceinline__ X64 div_cell(X64 x, int axis) {
  if (s_cell64.pow2) return x * s_cell64.inv[axis];
  return quot(x, s_cell64.d[axis]);
}

// x[v] / d of several values, in place.
template <int N>
__device__ __forceinline__ void div_cells(X64 (&x)[N], int axis) {
  if (s_cell64.pow2) {
#pragma unroll
    for (int v = 0; v < N; ++v) x[v] = x[v] * s_cell64.inv[axis];
  } else {
    quots(x, s_cell64.d[axis]);
  }
}

// u[v] += x[v] / d for the cell size of an axis and N values: with powers of
// two one fused operation each (the product is exact, so it rounds as the
// quotient and the sum do).
template <int N>
__device__ __forceinline__ void add_div_cell(X64 (&u)[N], X64 (&x)[N], int axis) {
  if (s_cell64.pow2) {
#pragma unroll
    for (int v = 0; v < N; ++v) u[v] = fma(x[v].v, s_cell64.inv[axis], u[v].v);
  } else {
    quots(x, s_cell64.d[axis]);
#pragma unroll
    for (int v = 0; v < N; ++v) u[v] = u[v] + x[v];
  }
}

// Storage slot (1 = a, 2 = b, 3 = c) of the reference's physical velocity
// component var (1 = x, 2 = y, 3 = z).
template <int PLANE>
__device__ __forceinline__ constexpr int phys_slot(int var) {
  return var == 1 ? 1 : (PLANE == PLANE_XY ? (var == 2 ? 2 : 3) : (var == 2 ? 3 : 2));
}

// consToPrim (States.h:34-45) of a state held in storage order; returns
// (rho, u_a, u_b, u_c, p) and, through D, the prepared density.  The kinetic energy sums
// the physical x, y, z velocities in the reference's order; with WACT false
// the degenerate velocity is exactly zero and its (exact) zero terms are
// dropped.  The divisions by rho share its preparation (quot, fv_exact64.cuh).
template <int PLANE, bool WACT>
__device__ __forceinline__ void cons_to_prim64(const X64 u[5], X64 gm1, X64 q[5], Div64& D) {
  const X64 r = u[0];
  D = prepare_div(r);
  X64 m[WACT ? 3 : 2] = {u[1], u[2]};
  if (WACT) m[2] = u[3];
  quots(m, D);
  const X64 va = m[0], vb = m[1], vc = WACT ? m[2] : X64(0.0);
  X64 ke;
  if (WACT) {
    const X64 vx = va, vy = PLANE == PLANE_XY ? vb : vc, vz = PLANE == PLANE_XY ? vc : vb;
    ke = vx * vx + vy * vy + vz * vz;
  } else {
    ke = va * va + vb * vb;
  }
  const X64 Ek = half_of(r) * ke;
  q[0] = r;
  q[1] = va;
  q[2] = vb;
  q[3] = vc;
  q[4] = (u[4] - Ek) * gm1;
}

// Hyperbolic inverse time step of one cell, ComputeDt.h:49-52:
// (cs + |u|)/dx + (cs + |v|)/dy + (cs + |w|)/dz with cs = sqrt(p*gamma/rho).
// qout, when given, receives the primitives consToPrim computes on the way.
template <int PLANE, bool WACT>
__device__ __forceinline__ X64 inv_dt_hyp64(const X64 u[5], const Grid& G, X64* qout = nullptr) {
  X64 q[5];
  Div64 D;
  cons_to_prim64<PLANE, WACT>(u, G.gm1, q, D);
  if (qout) {
#pragma unroll
    for (int v = 0; v < 5; ++v) qout[v] = q[v];
  }
  const X64 cs = sqrt64(quot(q[4] * G.gamma, D));
  const X64 vx = q[1], vy = PLANE == PLANE_XY ? q[2] : q[3], vz = PLANE == PLANE_XY ? q[3] : q[2];
  X64 tx = cs + fabs(vx.v), ty = cs + fabs(vy.v), tz = cs + fabs(vz.v);
  if (s_cell64.pow2)  // exact products: each fused operation rounds as quotient and sum do
    return fma(tz.v, s_cell64.inv[2], fma(ty.v, s_cell64.inv[1], (tx * s_cell64.inv[0]).v));
  quot_pair(tx, s_cell64.d[0], ty, s_cell64.d[1]);
  return tx + ty + quot(tz, s_cell64.d[2]);
}

// Block-wide max of non-negative doubles held as bit patterns (IEEE order of
// non-negative doubles equals unsigned order; NaN sorts above +inf) and one
// atomic max per CTA.  Every thread of the block must call it.
__device__ __forceinline__ void block_max_atomic(unsigned long long v, unsigned long long* slot,
                                                 unsigned long long* s_red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  const int nw = (blockDim.x * blockDim.y + 31) >> 5;
  if ((tid & 31) == 0) s_red[tid >> 5] = v;
  __syncthreads();
  if (tid == 0) {
    unsigned long long m = s_red[0];
    for (int w = 1; w < nw; ++w) m = s_red[w] > m ? s_red[w] : m;
    atomicMax(slot, m);
  }
}

}  // namespace fv
