// fv_march3d32.cu -- the FP32-mixed stage of 3-D problems, marched over z with
// the z stencil in registers.
//
// A CTA of 16 warps owns a block of at most 30 x 15 columns and a run of z
// layers.  A warp is a row of the block, a lane a column (lane 0 and 31 and the
// last warp only serve their neighbours).  Per layer m:
//   - the x face right of every column: slopes once per cell, the neighbour's
//     face state and the flux of the face on the left by warp shuffles;
//   - the y face below every row, its flux handed to the row below through
//     shared memory (double buffered: one barrier per layer, arrived at
//     before the z face and the update and waited for after them);
//   - the z face m - 1/2 from differences, face states and fluxes carried in
//     registers from layer to layer, and the update of layer m - 1.
// Shared memory holds a ring of four layers of primitives with a two-cell halo
// (a halo cell each for the threads of the last five warps).
// Conductive and viscous fluxes are carried beside the hydrodynamic ones and
// differenced on their own, as in the 2-D form; the z branch of the viscosity,
// whose terms belong to the cell, gives each face one flux per side.
//
// Bound by instruction issue and latency (65-69 % issue active with 16 warps),
// as the block form (fv_stage3d32.cu) it replaces where it is the faster one:
// that one forms each slope twice, reads every primitive of a face four times
// and evaluates every viscous face from both cells (52 and 56 warp instructions
// per cell against some 44 and 46 here).  192^3, RK2, a step: PLM with
// conduction and viscosity 1,000 -> 765 us, with conduction 829 -> 603, hydro
// alone 749 -> 596, PCM with both 865 -> 736; 100x80x90, PLM with both 124 ->
// 95; 24^3 55 -> 40.  Two CTAs of 8 warps (30 x 7 columns) measured 8 % slower,
// one of 12 or 14 warps (168 or 144 registers, no spills) 19-21 % on 192^3,
// prefetching the cells' own values of the update into L1 2 %, a barrier
// without the split arrival 11 %.
//
// Arithmetic and precision split as the 2-D form (fv_march32.cuh), written with
// _rn intrinsics.  The z-boundary physics (C91, well-balanced fluxes, fixed
// conduction boundaries) and the corrected physics stay with the block form.
#include "fv_march32.cuh"

namespace fv {

namespace {

constexpr int kWarps = 16, kThreads3 = 32 * kWarps;
constexpr int kBX = 30, kBY = kWarps - 1;   // most useful columns and rows of a block
constexpr int kCols = 34, kRows = kWarps + 3;  // columns x0-2 .. x0+31, rows y0-2 .. y0+16
constexpr int kHalo = 3 * kCols + 2 * kWarps;  // cells around the threads' own
constexpr int kHaloThreads = (kHalo + 31) / 32 * 32;
constexpr int kPlane = kCols * kRows;
constexpr int kSlot = 6 * kPlane;           // five primitives and the temperature
constexpr int kFb = 4 * kSlot;              // y-face fluxes [2][9][kWarps][32]: hydrodynamic 0-4, diffusive of slot v at 4 + v
constexpr int kFace = kWarps * 32;
constexpr size_t kSmemBytes = sizeof(float) * (size_t)(kFb + 2 * 9 * kFace);

// Layers [k0, k1) of the bw x bh columns from (x0, y0) on.  KIND, flip, red and
// bad as march_item32; mbar / phase: the CTA's barrier (an arrival per warp) and
// its phase; late: a wait on it ran out.
// VISC: some problem of the group is viscous.
template <int KIND, bool VISC>
__device__ __forceinline__ void march_block32(const BatchInst& I, int flip, float2 dtp, int x0, int y0, int bw, int bh,
                                              int k0, int k1, float* smem, unsigned long long* mbar, unsigned& phase,
                                              bool& late, float& red, bool& bad) {
  using namespace m32;
  constexpr bool STAR = KIND == STAGE_RK_2;
  constexpr int kSz = STAR ? 4 : 8;
  constexpr unsigned kAll = 0xffffffffu;
  const Grid& G = I.G;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rs = I.rs;
  const bool plm = G.recon == R_PLM, wb_z = G.recon == R_PCM_WB;
  const bool tc = G.tc != 0, visc = VISC && G.visc != 0, grav = G.gravity != 0;
  const float gamma = G.gamma_f, gm1 = G.gm1_f, inv_gm1 = G.inv_gm1_f;
  const float odx = G.inv_dx_f, ody = G.inv_dy_f, odz = G.inv_dz_f;
  const float dt = dtp.x;
  const float dtdx = mul_to(dtp, I.inv_d[0]), dtdy = mul_to(dtp, I.inv_d[1]), dtdz = mul_to(dtp, I.inv_d[2]);
  const size_t fs = (size_t)G.fstride * 8;
  const char* in0 = reinterpret_cast<const char*>(STAR || (KIND == STAGE_EULER && flip) ? I.B.f[0] : I.A.f[0]);
  char* un0 = reinterpret_cast<char*>(I.A.f[0]);
  char* us0 = reinterpret_cast<char*>(I.B.f[0]);
  const unsigned zstride = (unsigned)G.nb * (unsigned)G.pitch;

  // the thread's column, its offset in a layer and its place in a shared plane
  bool fa, fb;
  const int sa = bc_source(x0 - 1 + lane, G.na, G.bc_a, fa);
  const int sb = bc_source(y0 + w, G.nb, G.bc_b, fb);
  const unsigned col = (unsigned)sb * (unsigned)G.pitch + (unsigned)sa;
  const int at = (w + 2) * kCols + lane + 1;
  const bool work = w < bh;                                  // warp: this row is updated
  const bool own = work && lane >= 1 && lane <= bw;          // lane: this column too
  float* fbuf = smem + kFb + w * 32 + lane;                  // [buf][v]: + (buf * 9 + v) * kFace

  auto load_cell = [&](unsigned o, float2 c[5]) {
    const char* p = in0 + (size_t)o * kSz;
#pragma unroll
    for (int v = 0; v < 5; ++v)
      c[v] = STAR ? make_float2(*reinterpret_cast<const float*>(p + v * fs), 0.0f)
                  : *reinterpret_cast<const float2*>(p + v * fs);
  };
  // primitives (and temperature) of a loaded cell into place `p` of slot s; the
  // flags mirror its velocities
  auto put_cell = [&](const float2 c[5], bool mx, bool my, bool mz, float* p) {
    float q[5];
    const float y = STAR ? prim_of_star<true>(c, gm1, q) : prim_of_pairs<true>(c, gm1, q);
    p[0] = q[0];
    p[kPlane] = mx ? -q[1] : q[1];
    p[2 * kPlane] = my ? -q[2] : q[2];
    p[3 * kPlane] = mz ? -q[3] : q[3];
    p[4 * kPlane] = q[4];
    if (tc) p[5 * kPlane] = mul(q[4], y);
  };
  // the halo cell this thread loads of each layer, if any (the last five
  // warps): rows -2, -1 and kWarps (34 columns), the outer columns of the rows between
  const int hi = (int)threadIdx.x - (kThreads3 - kHaloThreads);
  const bool halo = hi >= 0 && hi < kHalo;
  unsigned hcol = 0;
  int hat = 0;
  bool hx = false, hy = false;
  if (halo) {
    int r, c;
    if (hi < 3 * kCols) {
      const int t = hi / kCols;
      c = hi - t * kCols;
      r = t < 2 ? t : kRows - 1;
    } else {
      const int t = hi - 3 * kCols;
      c = t & 1 ? kCols - 1 : 0;
      r = 2 + (t >> 1);
    }
    const int xa = bc_source(x0 + c - 2, G.na, G.bc_a, hx);
    const int yb = bc_source(y0 + r - 2, G.nb, G.bc_b, hy);
    hcol = (unsigned)yb * (unsigned)G.pitch + (unsigned)xa;
    hat = r * kCols + c;
  }

  for (int kg = k0 - 2; kg <= k0; ++kg) {
    bool mz;
    const int sz = bc_source(kg, G.nc, G.bc_c, mz);
    float* slot = smem + ((kg + 4) & 3) * kSlot;
    float2 c[5];
    load_cell((unsigned)sz * zstride + col, c);
    put_cell(c, fa, fb, mz, slot + at);
    if (halo) {
      load_cell((unsigned)sz * zstride + hcol, c);
      put_cell(c, hx, hy, mz, slot + hat);
    }
  }
  __syncthreads();

  float q0[5], q1[5], T0, T1;  // own column: layers j, j + 1
  {
    const float* a = smem + ((k0 + 2) & 3) * kSlot + at;
    const float* b = smem + ((k0 + 3) & 3) * kSlot + at;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      q0[v] = a[v * kPlane];
      q1[v] = b[v * kPlane];
    }
    T0 = tc ? a[5 * kPlane] : 0.0f;
    T1 = tc ? b[5 * kPlane] : 0.0f;
  }
  // of the 2-D form: Fb, the hydrodynamic flux of face j - 1/2; duA, everything else of layer j but its upper face
  float d[5], Ls[5], Fb[5], duA[5], Fx[6];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    d[v] = sub(q1[v], q0[v]);
    Ls[v] = Fb[v] = duA[v] = 0.0f;
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) Fx[k] = 0.0f;

  const float vx1 = visc ? mul_to(dtp, I.mu_d[0]) : 0.0f, vy1 = visc ? mul_to(dtp, I.mu_d[1]) : 0.0f,
              vz1 = visc ? mul_to(dtp, I.mu_d[2]) : 0.0f;
  const float cx = mul(0.25f, vx1), cy = mul(0.25f, vy1), cz = mul(0.25f, vz1);
  constexpr float k23 = 2.0f / 3.0f, k43 = 4.0f / 3.0f;
  const float ktx = tc ? mul_to(dtp, I.kappa_d2[0]) : 0.0f, kty = tc ? mul_to(dtp, I.kappa_d2[1]) : 0.0f,
              ktz = tc ? mul_to(dtp, I.kappa_d2[2]) : 0.0f;

#pragma unroll 1
  for (int j = k0 - 2; j < k1; ++j) {
    const int m = j + 1;
    // layer j + 3 on its way
    const bool more = j + 3 <= k1 + 1;
    bool mz = false;
    float2 raw[5];
    unsigned zoff = 0;
    if (more) {
      zoff = (unsigned)bc_source(j + 3, G.nc, G.bc_c, mz) * zstride;
      load_cell(zoff + col, raw);
      if (halo) {  // asked into L1, loaded when it is converted
        const char* p = in0 + (size_t)(zoff + hcol) * kSz;
#pragma unroll
        for (int v = 0; v < 5; ++v) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + v * fs));
      }
    }
    // layer j: the cell's own values, used at the end of the layer (viscous
    // problems have no registers to hold them and load them there)
    const size_t o = (size_t)((unsigned)j * zstride + col);
    float2 un[5];
    float us[5];
    if (!VISC && own && j >= k0) {
      const char* p = (KIND == STAGE_RK_2 ? un0 : in0) + o * 8;
      const char* r = us0 + o * 4;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        un[v] = *reinterpret_cast<const float2*>(p + v * fs);
        if (STAR) us[v] = *reinterpret_cast<const float*>(r + v * fs);
      }
    }
    const float* P = smem + ((m + 4) & 3) * kSlot + at;   // layer m
    const float* U = smem + ((m + 5) & 3) * kSlot + at;   // layer m + 1
    const float* D = smem + ((m + 3) & 3) * kSlot + at;   // layer m - 1
    float qn[5], dn[5], mm[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      qn[v] = U[v * kPlane];
      dn[v] = sub(qn[v], q1[v]);
      mm[v] = plm ? minmod(d[v], dn[v]) : 0.0f;
    }
    const float Tn = tc ? U[5 * kPlane] : 0.0f;
    float duN[5], FbN[5], VbN[5], Vup[5], Fy[5], FxN[6];
    float* fy = fbuf + (m & 1) * 9 * kFace;
#pragma unroll
    for (int v = 0; v < 5; ++v) duN[v] = FbN[v] = VbN[v] = Vup[v] = Fy[v] = 0.0f;
#pragma unroll
    for (int k = 0; k < 6; ++k) FxN[k] = 0.0f;
    const bool faces = m >= k0 && m < k1;  // layer k1 is another item's
    if (w <= bh && (visc || faces)) {
      // ---- layer m: differences to the neighbours along x (dl, dR) and y (below: by, above: ay)
      float dl[5], dR[5], by[5], ay[5];
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        dl[v] = sub(q1[v], P[v * kPlane - 1]);
        dR[v] = sub(P[v * kPlane + 1], q1[v]);
        by[v] = sub(q1[v], P[v * kPlane - kCols]);
        ay[v] = sub(P[v * kPlane + kCols], q1[v]);
      }
      if (visc) {
        // for the z branch: right u, v; (w above - v below), (v above - w below);
        // left u and w summed over this row and the one above (the cell's upper face)
        const float ul = sub(q1[1], dl[1]), wl = sub(q1[3], dl[3]);
        FxN[0] = add(q1[1], dR[1]);
        FxN[1] = add(q1[2], dR[2]);
        FxN[2] = sub(add(q1[3], ay[3]), sub(q1[2], by[2]));
        FxN[3] = sub(add(q1[2], ay[2]), sub(q1[3], by[3]));
        FxN[4] = add(ul, P[kPlane + kCols - 1]);
        FxN[5] = add(wl, P[3 * kPlane + kCols - 1]);
      }
      if (faces) {
        const float ez[3] = {sub(qn[1], q0[1]), sub(qn[2], q0[2]), sub(qn[3], q0[3])};
        // ---- y face below row w
        {
          float L[5], R[5];
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            const float b = P[v * kPlane - kCols];
            const float sB = plm ? minmod(sub(b, P[v * kPlane - 2 * kCols]), by[v]) : 0.0f;
            const float sC = plm ? minmod(by[v], ay[v]) : 0.0f;
            L[v] = fma_(0.5f, sB, b);
            R[v] = fma_(-0.5f, sC, q1[v]);
          }
          if (rs == 0) hll<2, 1, 3, true>(L, R, gamma, inv_gm1, Fy);
          else hllc<2, 1, 3, true>(L, R, gamma, inv_gm1, Fy);
#pragma unroll
          for (int v = 0; v < 5; ++v) fy[v * kFace] = Fy[v];
          float ve = tc ? mul(kty, sub(T1, P[5 * kPlane - kCols])) : 0.0f;
          if (visc) {  // IY (Viscosity.h:188-213)
            const float su = add(add(dl[1], dR[1]), sub(P[kPlane - kCols + 1], P[kPlane - kCols - 1]));
            const float sv = add(add(dl[2], dR[2]), sub(P[2 * kPlane - kCols + 1], P[2 * kPlane - kCols - 1]));
            const float zv = add(ez[1], sub(U[2 * kPlane - kCols], D[2 * kPlane - kCols]));
            const float zw = add(ez[2], sub(U[3 * kPlane - kCols], D[3 * kPlane - kCols]));
            const float txy = fma_(vy1, by[1], mul(cx, sv));
            const float tyy = fma_(mul(k43, vy1), by[2], -mul(k23, fma_(cx, su, mul(cz, zw))));
            const float tyz = fma_(vy1, by[3], mul(cz, zv));
            const float ma = fma_(-0.5f, by[1], q1[1]), mb = fma_(-0.5f, by[2], q1[2]), mc = fma_(-0.5f, by[3], q1[3]);
            fy[5 * kFace] = txy;
            fy[6 * kFace] = tyy;
            fy[7 * kFace] = tyz;
            ve = fma_(txy, ma, fma_(tyy, mb, fma_(tyz, mc, ve)));
          }
          if (tc || visc) fy[8 * kFace] = ve;
        }
        if (work) {
          // ---- x face right of the column
          float L[5], R[5], Fa[5];
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            const float s = plm ? minmod(dl[v], dR[v]) : 0.0f;
            L[v] = fma_(0.5f, s, q1[v]);
            R[v] = __shfl_down_sync(kAll, fma_(-0.5f, s, q1[v]), 1);
          }
          if (rs == 0) hll<1, 2, 3, true>(L, R, gamma, inv_gm1, Fa);
          else hllc<1, 2, 3, true>(L, R, gamma, inv_gm1, Fa);
#pragma unroll
          for (int v = 0; v < 5; ++v) duN[v] = mul(dtdx, sub(__shfl_up_sync(kAll, Fa[v], 1), Fa[v]));
          float ve = tc ? mul(ktx, sub(P[5 * kPlane + 1], T1)) : 0.0f;
          if (visc) {  // IX (Viscosity.h:163-186)
            const float yu = add(by[1], ay[1]), yv = add(by[2], ay[2]);
            const float su = add(yu, __shfl_down_sync(kAll, yu, 1)), sv = add(yv, __shfl_down_sync(kAll, yv, 1));
            const float zu = add(ez[0], __shfl_down_sync(kAll, ez[0], 1));
            const float zw = add(ez[2], __shfl_down_sync(kAll, ez[2], 1));
            const float txx = fma_(mul(k43, vx1), dR[1], -mul(k23, fma_(cy, sv, mul(cz, zw))));
            const float txy = fma_(vx1, dR[2], mul(cy, su));
            const float txz = fma_(vx1, dR[3], mul(cz, zu));
            const float ma = fma_(0.5f, dR[1], q1[1]), mb = fma_(0.5f, dR[2], q1[2]), mc = fma_(0.5f, dR[3], q1[3]);
            duN[1] = add(duN[1], sub(txx, __shfl_up_sync(kAll, txx, 1)));
            duN[2] = add(duN[2], sub(txy, __shfl_up_sync(kAll, txy, 1)));
            duN[3] = add(duN[3], sub(txz, __shfl_up_sync(kAll, txz, 1)));
            ve = fma_(txx, ma, fma_(txy, mb, fma_(txz, mc, ve)));
          }
          if (tc || visc) duN[4] = add(duN[4], sub(ve, __shfl_up_sync(kAll, ve, 1)));
          if (grav) duN[3] = fma_(mul(dt, G.g_f), q1[0], duN[3]);
        }
      }
    }
    if (more) {
      float* slot = smem + ((j + 7) & 3) * kSlot;
      put_cell(raw, fa, fb, mz, slot + at);
      if (halo) {
        load_cell(zoff + hcol, raw);
        put_cell(raw, hx, hy, mz, slot + hat);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(mbar);
    if (work && m >= k0) {
      // ---- z face between layers j and m
      {
        float R[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) R[v] = fma_(-0.5f, mm[v], q1[v]);
        if (wb_z) {  // PCM_WB hydrostatic pressure (Update.h:27)
          Ls[4] = fma_(mul(Ls[0], G.g_dz_f), 0.5f, Ls[4]);
          R[4] = fma_(mul(R[0], G.g_dz_f), -0.5f, R[4]);
        }
        if (rs == 0) hll<3, 2, 1, true>(Ls, R, gamma, inv_gm1, FbN);
        else hllc<3, 2, 1, true>(Ls, R, gamma, inv_gm1, FbN);
      }
      if (tc) VbN[4] = Vup[4] = mul(ktz, sub(T1, T0));
      if (visc) {  // IZ with the reference's mix-ups (Viscosity.h:214-239): each cell of the face reads its own row
        const float ma = fma_(0.5f, d[1], q0[1]), mb = fma_(0.5f, d[2], q0[2]), mc = fma_(0.5f, d[3], q0[3]);
        const float ur = add(Fx[0], FxN[0]), vr = add(Fx[1], FxN[1]);
        const float tzz = fma_(mul(k43, vz1), d[3], -mul(k23, fma_(cx, ur, mul(cz, add(Fx[2], FxN[2])))));
        const float txz = fma_(vz1, d[1], mul(cx, vr));
        const float tyz = fma_(vz1, d[2], mul(cz, add(Fx[3], FxN[3])));
        // left u, w of cell m summed over its row and the one below (its lower face)
        const float ulm = add(P[kPlane - 1], P[kPlane - kCols - 1]);
        const float wlm = add(P[3 * kPlane - 1], P[3 * kPlane - kCols - 1]);
#pragma unroll
        for (int s = 0; s < 2; ++s) {  // cell j (its upper face), cell m (its lower face)
          float* V = s == 0 ? Vup : VbN;
          const float zz = fma_(mul(k23, cx), s == 0 ? Fx[4] : ulm, tzz);
          const float xz = fma_(-cx, s == 0 ? Fx[5] : wlm, txz);
          V[1] = xz;
          V[2] = tyz;
          V[3] = zz;
          V[4] = fma_(xz, ma, fma_(tyz, mb, fma_(zz, mc, V[4])));
        }
#pragma unroll
        for (int v = 1; v < 4; ++v) duN[v] = sub(duN[v], VbN[v]);
      }
      if (tc || visc) duN[4] = sub(duN[4], VbN[4]);
      // ---- layer j: increments, accumulation on the pairs, CFL term
      if (own && j >= k0) {
        if (VISC) {
          const char* p = (KIND == STAGE_RK_2 ? un0 : in0) + o * 8;
          const char* r = us0 + o * 4;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            un[v] = *reinterpret_cast<const float2*>(p + v * fs);
            if (STAR) us[v] = *reinterpret_cast<const float*>(r + v * fs);
          }
        }
        float du[5];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          du[v] = fma_(dtdz, sub(Fb[v], FbN[v]), duA[v]);
          if (v == 4 ? tc || visc : v > 0 && visc) du[v] = add(du[v], Vup[v]);
        }
        if (grav)  // half the mass fluxes of both faces (Update.h:150)
          du[4] = fma_(mul(mul(0.5f, dt), G.g_f), add(Fb[0], FbN[0]), du[4]);
        // density floor on the hydro update (Update.h:160)
        const bool low = (STAR ? add(us[0], du[0]) : add(add(un[0].x, du[0]), un[0].y)) < 1.0e-6f;
        if (low) {
          if (!STAR) un[0] = make_float2(1.0e-6f, 0.0f);
          du[0] = 0.0f;
        }
        if (KIND == STAGE_RK_1) {
          float o5[5];
#pragma unroll
          for (int v = 0; v < 4; ++v) o5[v] = add(un[v].x, add(un[v].y, du[v]));
          // U* keeps its internal energy (fv_tile32.cuh)
          o5[4] = internal_energy(pair_add(un[4], du[4]), kinetic_star<true>(o5));
          char* r = us0 + o * 4;
#pragma unroll
          for (int v = 0; v < 5; ++v) *reinterpret_cast<float*>(r + v * fs) = o5[v];
        } else {
          float2 fin[5];
          if (KIND == STAGE_RK_2) {  // 0.5 (U^n + U* + dU)
            const float2 k = kinetic_star<true>(us);
            const float2 e = two_sum(k.x, us[4]);
            if (low) us[0] = 1.0e-6f;
#pragma unroll
            for (int v = 0; v < 5; ++v) {
              const float2 a = two_sum(un[v].x, v == 4 ? e.x : us[v]);
              const float2 b = two_sum(a.x, du[v]);
              const float lo = add(add(a.y, b.y), v == 4 ? add(un[v].y, add(e.y, k.y)) : un[v].y);
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
          const float y = prim_of_pairs<true>(fin, gm1, q);
          const float cs = sqrt_(mul(mul(q[4], gamma), y));
          const float inv =
              fma_(add(cs, fabsf(q[1])), odx, fma_(add(cs, fabsf(q[2])), ody, mul(add(cs, fabsf(q[3])), odz)));
          bad |= !(inv <= 3.0e38f);
          red = fmaxf(red, inv);
        }
      }
    }
    // every row has handed on its flux and its cells of layer j + 3
    if (!late && !mbar_wait(mbar, phase)) late = true;
    phase ^= 1u;
    if (work && faces) {  // the y face above: the one below the next row
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        duN[v] = fma_(dtdy, sub(Fy[v], fy[v * kFace + 32]), duN[v]);
        if (v == 4 ? tc || visc : v > 0 && visc)
          duN[v] = add(duN[v], sub(fy[(4 + v) * kFace + 32], fy[(4 + v) * kFace]));
      }
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      Ls[v] = fma_(0.5f, mm[v], q1[v]);
      Fb[v] = FbN[v];
      duA[v] = duN[v];
      q0[v] = q1[v];
      q1[v] = qn[v];
      d[v] = dn[v];
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) Fx[k] = FxN[k];
    T0 = T1;
    T1 = Tn;
  }
}

// ONE: a group of one problem, its descriptor in the launch parameters.
template <int KIND, bool VISC, bool ONE>
__global__ void __launch_bounds__(kThreads3, 1)
march_stage3d32(const BatchInst* __restrict__ insts, int ninst, int ntiles, unsigned* queue, int flip,
                const __grid_constant__ BatchInst one) {
  extern __shared__ float smem_f[];
  __shared__ BatchInst s_inst;
  __shared__ int s_tile;
  __shared__ __align__(8) unsigned long long s_mbar;
  const BatchInst& I = ONE ? one : s_inst;
  unsigned phase = 0;
  bool late = false;
  if (threadIdx.x == 0) mbar_init(&s_mbar, kWarps);  // visible after the __syncthreads below
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
    if (!ONE) {
      int lo = 0, hi = ninst - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (insts[mid].tile0 <= t) lo = mid;
        else hi = mid - 1;
      }
      const unsigned long long* s = reinterpret_cast<const unsigned long long*>(insts + lo);
      unsigned long long* d = reinterpret_cast<unsigned long long*>(&s_inst);
      for (int i = threadIdx.x; i < (int)(sizeof(BatchInst) / 8); i += blockDim.x) d[i] = s[i];
      __syncthreads();
    }
    StepCtrl* ctrl = I.ctrl;
    const int lt = t - I.tile0;
    const int per_layer = I.tiles_x * I.tiles_y;
    const int bz = lt / per_layer, rem = lt - bz * per_layer;
    const int by = rem / I.tiles_x, bx = rem - by * I.tiles_x;
    // blocks of equal size; none is empty: bw <= kBX and na > (tiles_x - 1) kBX, likewise the rows
    const int bw = (I.G.na + I.tiles_x - 1) / I.tiles_x, bh = (I.G.nb + I.tiles_y - 1) / I.tiles_y;
    const int x0 = bx * bw, y0 = by * bh, k0 = bz * I.tz, k1 = min(k0 + I.tz, I.G.nc);
    const int nx = min(bw, I.G.na - x0), ny = min(bh, I.G.nb - y0);
    if (!ctrl->active) {
      if (KIND == STAGE_EULER) {  // an inactive Euler step hands its state on
        for (int i = threadIdx.x; i < nx * ny * (k1 - k0); i += kThreads3) {
          const int k = i / (nx * ny), r = i - k * nx * ny;
          const size_t o = ((size_t)(k0 + k) * I.G.nb + y0 + r / nx) * I.G.pitch + x0 + r % nx;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            float2* a = reinterpret_cast<float2*>(I.A.f[v]);
            float2* b = reinterpret_cast<float2*>(I.B.f[v]);
            if (flip) a[o] = b[o];
            else b[o] = a[o];
          }
        }
      }
      continue;
    }
    float red = 0.0f;
    bool bad = false;
    march_block32<KIND, VISC>(I, flip, ctrl->dt_pair, x0, y0, nx, ny, k0, k1, smem_f, &s_mbar, phase, late, red, bad);
    report_late(late, &ctrl->err);
    if (KIND != STAGE_RK_1) {
      const unsigned mx = __reduce_max_sync(0xffffffffu, __float_as_uint(red));  // non-negative floats order like their bits
      const bool any_bad = __any_sync(0xffffffffu, bad);
      if ((threadIdx.x & 31) == 0) {
        if (any_bad) atomicOr(&ctrl->err, 1);
        if (mx) atomicMax(&ctrl->slot[ctrl->parity ^ 1], (unsigned long long)__double_as_longlong((double)__uint_as_float(mx)));
      }
    }
  }
}

template <bool VISC, bool ONE>
MarchKernel kernel3_of(int kind) {
  switch (kind) {
    case STAGE_RK_1: return march_stage3d32<STAGE_RK_1, VISC, ONE>;
    case STAGE_RK_2: return march_stage3d32<STAGE_RK_2, VISC, ONE>;
    default: return march_stage3d32<STAGE_EULER, VISC, ONE>;
  }
}

MarchKernel kernel3(int kind, bool visc, bool one) {
  if (visc) return one ? kernel3_of<true, true>(kind) : kernel3_of<true, false>(kind);
  return one ? kernel3_of<false, true>(kind) : kernel3_of<false, false>(kind);
}

bool prepare3() {
  static bool done = false;
  if (done) return true;
  for (int kind : {STAGE_EULER, STAGE_RK_1, STAGE_RK_2})
    for (int k = 0; k < 4; ++k)
      if (cudaFuncSetAttribute(kernel3(kind, k & 1, k & 2), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kSmemBytes) != cudaSuccess)
        return false;
  done = true;
  return true;
}

}  // namespace

int march3d_block(int* cols, int* rows) {
  *cols = kBX;
  *rows = kBY;
  return kThreads3;
}

int march3d_occupancy(int kind, bool visc, bool one) {
  if (!prepare3()) return 0;
  int nb = 0;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel3(kind, visc, one), kThreads3, kSmemBytes) == cudaSuccess
             ? nb
             : 0;
}

cudaError_t launch_march3d32(const BatchInst* insts, int ninst, int ntiles, unsigned* queue, int kind, int flip, bool visc,
                             int grid, cudaStream_t st, const BatchInst* one) {
  if (!prepare3()) return cudaErrorInvalidConfiguration;
  static const BatchInst empty{};
  const cudaError_t e = launch_pdl(kernel3(kind, visc, one != nullptr), dim3(grid), dim3(kThreads3), kSmemBytes, st, insts,
                                   ninst, ntiles, queue, flip, one ? *one : empty);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace fv
