// Line-marching convective kernels of the explicit RK stage.
//
// Every face of a line (fixed transverse cell, family d) needs the limited
// MUSCL states of its two cells; the limiter of cell c depends only on its
// two slopes dq(c) = q(c) - q(c-1) and dq(c+1), and gives both the state of
// c on its lower face (for face c) and on its upper face (for face c+1) from
// one sensor (limit_i/j/k, src/flux.f90:3472-3888, where the two sensors of a
// cell are the same expression).  So a thread that walks a line evaluates each
// cell's sensor once instead of twice and loads each cell once instead of four
// times:
//
//   d = 2, 3   lanes along i (coalesced), each thread marches along j or k
//              over a segment of faces, carrying a cell, a slope and the
//              pending left state;
//   d = 1      lanes along i as well: lane l owns cell c = i0 - 1 + l, gets
//              the neighbouring cells through L1, and passes its upper state
//              to lane l + 1 with a warp shuffle; lanes 1..31 compute faces
//              i0 .. i0 + 30.
//
// One warp is one CTA, so that everything a task holds (block, bases, strides,
// loop bounds) is uniform over the CTA and the strong-boundary cases are
// uniform branches off the loop instead of selects in it.
//
// Two schedules use these loops (picked by size, launch_split_tail):
//   store   one launch over all faces, fluxes to memory, then k_cells: the
//           most parallel form, for grids that leave the chip idle;
//   chain   i, then j, then k launches, each adding its family's flux
//           difference to the running sum D of the cell (the reference's
//           bresid order), the last one finishing the stage: D is 40 bytes a
//           cell where the three families' fluxes are 120 written and read.
// The face and cell arithmetic is shared, so both give the same bits.
//
// The stage input's halo cells are primitive (k_halo); its interior is
// conservative and converted on load (CONV, c2p5_nr with the positivity test
// of bprtest), or primitive: in the viscous path's copy, and between the
// stages of an iteration (launch_iteration).
//
// What bounds them: issue and FP64 latency.  A face takes about 230 FP64
// operations (limiter and states 17 a variable, Roe flux 129); the three
// families of the 30.7 M-cell duct take 3.9 ms a stage, 2.5 ms of it at the
// FP64 pipe's rate, and move 464 B/cell (2.2 ms at 6.65 TB/s).  Before: 755 to
// 840 warp instructions a face with selects for the strong boundaries,
// 64-bit addresses per access and register-staged prefetch, fluxes through
// memory (530 B/cell with the cell pass): 5.3 ms.
//
// MIXED: slopes are FP64 differences rounded to FP32, the limiter
// and the whole Roe flux run in FP32, and the flux enters FP64 as
//     F = ds * ( g(q_L cell) + [ (Dg_L + Dg_R)/2 - |A| dq / 2 ] )
// with g(q) = f(q).n the unit-normal flux of the left cell's FP64 state and
// Dg_X = g(q_X) - g(q_L cell) the exact change of g to the FP32 face state
// X, expanded so that every FP32 term is proportional to the differences:
// the FP32 rounding error scales with the local jumps, not with the state.
#pragma once
#include "fused.cuh"

// one warp's share of a face family: d = 1: rows j = ta .. ta + nf - 1 at
// k = tb, lanes cells i0 - 1 + lane; d = 2: lanes i = i0 + lane, k = tb, faces
// j = f0 .. f0 + nf - 1; d = 3: lanes i = i0 + lane, j = tb, faces k = f0 ..
// f0 + nf - 1
struct __align__(16) FaceTask {
  int blk, d, n, i0, ta, tb, f0, nf;
};

// FP32 limiter of one cell (the mixed path's counterpart of limit_cell64):
// from the slopes a = dq(c), b = dq(c+1), dqp(c) and dqm(c+1), limit_face's
// algebra with fast division; ilim 1, 2 and 4 share their sensor
__device__ __forceinline__ void limit_cell32(int ilim, float eps, float rkap, float a, float b, float &dqp,
                                             float &dqm) {
  if (ilim == 1) {
    const float s = __fdividef(2.0f * b * a + eps, b * b + a * a + eps);
    const float rkp = 1.0f + rkap * s, rkm = 1.0f - rkap * s;
    dqp = -s * (rkp * a + rkm * b) * 0.25f;
    dqm = s * (rkm * a + rkp * b) * 0.25f;
  } else if (ilim == 0) {
    const float rkp = 1.0f + rkap, rkm = 1.0f - rkap;
    dqp = -(rkp * a + rkm * b) * 0.25f;
    dqm = (rkm * a + rkp * b) * 0.25f;
  } else if (ilim == 2) {
    const float rkp = 1.0f + rkap, rkm = 1.0f - rkap;
    const float bb = (3.0f - rkap) / (1.0f - rkap);
    const float sg = (copysignf(1.0f, a) + copysignf(1.0f, b)) * 0.5f;
    const float dqmx = sg * fminf(fabsf(a), fabsf(b) * bb);
    const float dqpx = sg * fminf(fabsf(b), fabsf(a) * bb);
    dqp = -(rkp * dqmx + rkm * dqpx) * 0.25f;
    dqm = (rkm * dqmx + rkp * dqpx) * 0.25f;
  } else if (ilim == 3) {
    const float epsq = eps * eps;
    dqp = -0.5f * __fdividef(a * (b * b + 2.0f * epsq) + b * (2.0f * (a * a) + epsq),
                             2.0f * (a * a) - a * b + 2.0f * (b * b) + 3.0f * epsq);
    dqm = 0.5f * __fdividef(b * (a * a + 2.0f * epsq) + a * (2.0f * (b * b) + epsq),
                            2.0f * (b * b) - b * a + 2.0f * (a * a) + 3.0f * epsq);
  } else {  // ilim == 4
    const float epsq = eps * eps;
    const float x = __fdividef(b * (a * a + epsq) + a * (b * b + epsq), b * b + a * a + 2.0f * epsq);
    dqp = -0.5f * x;
    dqm = 0.5f * x;
  }
}

// g(q) . n of a primitive state (rho, u, v, w, p) in FP64: the unit-normal
// Euler flux roflux_b builds from each face state (src/flux.f90:119-136)
// (MV: relative to a face moving with normal speed ubn, src/flux.f90:122-148)
template <bool MV>
__device__ __forceinline__ void unit_flux64(double g_gm1, double kx, double ky, double kz, const double *q, double *g,
                                            double ubn) {
  const double un = MV ? q[1] * kx + q[2] * ky + q[3] * kz - ubn : q[1] * kx + q[2] * ky + q[3] * kz;
  const double ru = q[0] * un;
  const double e = g_gm1 * q[4] + q[0] * (q[1] * q[1] + q[2] * q[2] + q[3] * q[3]) / 2;
  g[0] = ru;
  g[1] = ru * q[1] + q[4] * kx;
  g[2] = ru * q[2] + q[4] * ky;
  g[3] = ru * q[3] + q[4] * kz;
  g[4] = MV ? e * un + q[4] * ubn : e * un;
}

// base quantities of the FP32 expansions for the left cell: the state, its
// q^2 and E = G p + rho q^2 / 2 (rho h0)
struct Base32 {
  float r, u, v, w, p, q2, e;
};
__device__ __forceinline__ Base32 make_base32(float g_gm1, const float *b) {
  Base32 o;
  o.r = b[0]; o.u = b[1]; o.v = b[2]; o.w = b[3]; o.p = b[4];
  o.q2 = o.u * o.u + o.v * o.v + o.w * o.w;
  o.e = g_gm1 * o.p + 0.5f * o.r * o.q2;
  return o;
}

// Dg = g(base + d) - g(base) for the unit normal (kx, ky, kz), exactly
// rearranged so every term carries a factor of the difference d:
//   D(rho U)     = drho U + rho' dU
//   D(rho u U)   = D(rho U) u' + rho U du          (+ dp kx)
//   D(E)         = G dp + (drho q'^2 + rho (q'^2 - q^2)) / 2
//   D(E U)       = D(E) U' + E dU
// with primes for base + d and U = u.n
// (U is the normal velocity relative to the face; MV adds the change of the
// energy flux's p ubn term)
template <bool MV>
__device__ __forceinline__ void delta_flux32(float g_gm1, const Base32 &B, float U, float rU, float kx, float ky,
                                             float kz, const float *d, float *dg, float ubn) {
  const float dU = d[1] * kx + d[2] * ky + d[3] * kz;
  const float r1 = B.r + d[0], U1 = U + dU;
  const float u1 = B.u + d[1], v1 = B.v + d[2], w1 = B.w + d[3];
  const float drU = d[0] * U + r1 * dU;
  dg[0] = drU;
  dg[1] = drU * u1 + rU * d[1] + d[4] * kx;
  dg[2] = drU * v1 + rU * d[2] + d[4] * ky;
  dg[3] = drU * w1 + rU * d[3] + d[4] * kz;
  const float dq2 = d[1] * (B.u + u1) + d[2] * (B.v + v1) + d[3] * (B.w + w1);
  const float de = g_gm1 * d[4] + 0.5f * (d[0] * (B.q2 + dq2) + B.r * dq2);
  dg[4] = MV ? de * U1 + B.e * dU + d[4] * ubn : de * U1 + B.e * dU;
}

// Roe dissipation |A| (qR - qL) of roflux_b (src/flux.f90:137-230) in FP32
// from the FP32 face states and their jump dq (computed from differences)
template <bool MV>
__device__ __forceinline__ void roe_diss32(const PhysPar &P, float g, float g_gm1, float kx, float ky, float kz,
                                           const float *qr, const float *ql, const float *dq, float *df, float ubn) {
  const float rsr = rsqrtf(qr[0]), rsl = rsqrtf(ql[0]);
  const float h0r = g_gm1 * qr[4] * (rsr * rsr) + 0.5f * (qr[1] * qr[1] + qr[2] * qr[2] + qr[3] * qr[3]);
  const float h0l = g_gm1 * ql[4] * (rsl * rsl) + 0.5f * (ql[1] * ql[1] + ql[2] * ql[2] + ql[3] * ql[3]);
  const float rhols = ql[0] * rsl, rhors = qr[0] * rsr;
  const float rho = rhols * rhors;
  const float rden = __fdividef(1.0f, rhols + rhors);
  const float u = (rhols * ql[1] + rhors * qr[1]) * rden;
  const float v = (rhols * ql[2] + rhors * qr[2]) * rden;
  const float w = (rhols * ql[3] + rhors * qr[3]) * rden;
  const float un = u * kx + v * ky + w * kz;
  const float h0 = (rhols * h0l + rhors * h0r) * rden;
  const float q2 = u * u + v * v + w * w;
  const float a2 = (g - 1.0f) * (h0 - 0.5f * q2);
  const float ria = rsqrtf(a2);
  const float a = a2 * ria;
  const float drho = dq[0], du = dq[1], dv = dq[2], dw = dq[3], dp = dq[4];
  const float dun = du * kx + dv * ky + dw * kz;
  const float unr = MV ? un - ubn : un;  // normal velocity relative to the face
  float rm123 = fabsf(unr), rm4 = fabsf(unr + a), rm5 = fabsf(unr - a);
  if (P.efx_setup_f) {
    float rdelta = (float)P.cntrpy_f * ((float)P.w1 * (float)P.entfxctf_f + (float)P.w2 * (sqrtf(q2) + a) +
                                        (float)P.w3 * 0.2f * (fabsf(un) + a + (MV ? fabsf(ubn) : 0.0f)));
    rdelta = fmaxf(rdelta, 1.0e-12f);
    if (rm123 <= rdelta && P.efx_all_f) rm123 = 0.5f * (rm123 * rm123 + rdelta * rdelta) / rdelta;
    if (rm4 <= rdelta) rm4 = 0.5f * (rm4 * rm4 + rdelta * rdelta) / rdelta;
    if (rm5 <= rdelta) rm5 = 0.5f * (rm5 * rm5 + rdelta * rdelta) / rdelta;
  }
  if (P.eig_limit_f) {
    const float c = (float)P.eig_cutoff_f;
    if (rm123 <= c) rm123 = c;
    if (P.eig_lim_all_f && rm4 <= c) rm4 = c;
    if (P.eig_lim_all_f && rm5 <= c) rm5 = c;
  }
  const float dpa2 = dp * (ria * ria), rdua = rho * dun * ria;
  const float al1 = rm123 * (drho - dpa2);
  const float al2 = rm123 * rho;
  const float al3 = rm4 * (dpa2 + rdua) * 0.5f;
  const float al4 = rm5 * (dpa2 - rdua) * 0.5f;
  df[0] = al1 + al3 + al4;
  df[1] = al1 * u + al2 * (du - dun * kx) + al3 * (u + a * kx) + al4 * (u - a * kx);
  df[2] = al1 * v + al2 * (dv - dun * ky) + al3 * (v + a * ky) + al4 * (v - a * ky);
  df[3] = al1 * w + al2 * (dw - dun * kz) + al3 * (w + a * kz) + al4 * (w - a * kz);
  df[4] = al1 * (q2 * 0.5f) + al2 * (u * du + v * dv + w * dw - un * dun) + al3 * (h0 + a * un) +
          al4 * (h0 - a * un);
}

// mixed-precision face flux between cells L (FP64 state qL64, FP32 copy bL)
// and R (FP32 copy bR): dqL / dqR the FP32 offsets of the face states from
// their cells, dLR = (float)(qR64 - qL64)
template <bool MV>
__device__ __forceinline__ void face_flux_mixed(const PhysPar &P, float g, float g_gm1, const double *met,
                                                const double *qL64, const float *bL, const float *bR,
                                                const float *dLR, const float *dqL, const float *dqR,
                                                double *F, double ubn = 0.0) {
  const double kx = met[0], ky = met[1], kz = met[2], ds = met[3];
  const float fkx = (float)kx, fky = (float)ky, fkz = (float)kz, fub = (float)ubn;
  double g64[5];
  unit_flux64<MV>(P.g_gm1, kx, ky, kz, qL64, g64, ubn);
  const Base32 B = make_base32(g_gm1, bL);
  const float U = MV ? B.u * fkx + B.v * fky + B.w * fkz - fub : B.u * fkx + B.v * fky + B.w * fkz;
  const float rU = B.r * U;
  float dLs[5], dRs[5], ql[5], qr[5], jump[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    dLs[m] = dqL[m];              // face state L - cell L
    dRs[m] = dLR[m] + dqR[m];     // face state R - cell L
    ql[m] = bL[m] + dqL[m];
    qr[m] = bR[m] + dqR[m];
    jump[m] = dRs[m] - dLs[m];    // face state R - face state L
  }
  float dgl[5], dgr[5], df[5];
  delta_flux32<MV>(g_gm1, B, U, rU, fkx, fky, fkz, dLs, dgl, fub);
  delta_flux32<MV>(g_gm1, B, U, rU, fkx, fky, fkz, dRs, dgr, fub);
  roe_diss32<MV>(P, g, g_gm1, fkx, fky, fkz, qr, ql, jump, df, fub);
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const float t = 0.5f * (dgl[m] + dgr[m] - df[m]);
    F[m] = (g64[m] + (double)t) * ds;
  }
}

// scheme constants of the line kernels, passed by value: kernel parameters sit
// in the constant bank, where FP64 instructions read them as operands instead
// of holding them in registers across the marching loop
struct LinePar {
  PhysPar ph;
  double gamma, qmin_rho, qmin_p;
  int S, S2, hbmove;
};
inline LinePar make_line_par(const cosa_params &P) {
  LinePar o;
  o.ph = make_phys(P);
  o.gamma = P.gamma; o.qmin_rho = P.qmin[0]; o.qmin_p = P.qmin[4];
  o.S = 2 * P.nharms + 1; o.S2 = 2 * P.nharms * P.hbmove + 1; o.hbmove = P.hbmove;
  return o;
}
// arrays of a line launch
struct LineArgs {
  const DevBlock *blocks;
  const FaceTask *tasks;
  const double *q;               // stage input or its primitive copy
  const double *s[3];            // face metrics of the three families
  const uint8_t *strong;
  const StrongMap *smap;
  int first_order;
  int64_t n0;
  double *cf;                    // store: fluxes of the three families; chain: D (F0 layout)
  const double *vf;              // viscous fluxes of the three families (F0 planes of nv cells), added to the faces', or null
  int64_t nv;
  int *status;
  FaceVel fv;
};

// interior cells of a conservative stage input: to primitive variables, with
// bprtest's positivity test
__device__ __forceinline__ void to_prim(double gamma, double qmin_rho, double qmin_p, int &st, double *v) {
  c2p5_nr(gamma, v);
  if (v[4] <= qmin_p) st |= COSA_ERR_NEG_P;
  else if (v[0] <= qmin_rho) st |= COSA_ERR_NEG_RHO;
}
// asynchronous copies global -> shared memory, 8 and 16 bytes a lane
__device__ __forceinline__ void cp8(double *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp16(double2 *dst, const double *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// staging of one step: what it needs comes one step ahead without holding
// registers.  I: cells (with the two beyond the warp's) and metrics; M: the
// next cell, the face's metrics and, in the chain, the running balance D, the
// base state and the time step of the cell that the face closes
template <bool VIS>
struct StageI {
  double q[2][5][34];
  double2 met[2][2][32];
  double vis[2][VIS ? 5 : 1][32];
};
template <int OUT, bool VIS>
struct StageM {
  double q[2][5][32];
  double2 met[2][2][32];
  double D[2][OUT >= 1 ? 5 : 1][32];
  double base[2][OUT == 2 ? 6 : 1][32];
  double vis[2][VIS ? 5 : 1][32];
};
// normal speed of a face from its velocity: sijk(5)*kx + sijk(6)*ky +
// sijk(7)*kz, roflux_b's order (src/flux.f90:110-113)
__device__ __forceinline__ double face_ubn(const double *__restrict__ v, double kx, double ky, double kz) {
  return __fma_rn(__ldg(v + 2), kz, __fma_rn(__ldg(v + 1), ky, __dmul_rn(__ldg(v), kx)));
}

// what a cell's flux balance r goes through after the three families:
// harmonic-balance source, norms, forcing, update (k_cells and the
// last launch of the chain).  co: the cell in the state arrays (variable 1 of
// snapshot n), P3 their variable stride; q0: the cell's base state (read when
// A.update)
template <bool RMS>
__device__ __forceinline__ void finish_cell(const StageArgs &A, const cosa_params &P, int S, int n, int64_t co,
                                            int64_t P3, double vol_omega, double dt, double *r, const double *q0,
                                            double gamma, double qmin_rho, double qmin_p, double *acc, int &st) {
  double qw[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    const int64_t o = co + m * P3;
    if (A.vol) {
      // src_bhb (src/src.f90:556-613)
      double qhb = 0.0;
      for (int nj2 = 0; nj2 < S; ++nj2)
        qhb = __fma_rn(__dmul_rn(vol_omega, P.dhb[n * S + nj2]), A.qin[o + (nj2 - n) * 5 * P3], qhb);
      r[m] = r[m] + qhb;
    }
    if (RMS) acc[m] += r[m] * r[m];
    if (A.rhs_mode) {
      double *rh = A.rhs + o;
      if (A.rhs_mode == 2) {
        const double rn = *rh + r[m];
        *rh = rn;
        r[m] = r[m] - rn;
      } else {
        r[m] = r[m] - *rh;
      }
    }
    if (A.res_out) A.res_out[o] = r[m];
    if (A.update) {
      if (A.qold_copy) A.qold_copy[o] = q0[m];
      qw[m] = __fma_rn(-__dmul_rn(A.ar, r[m]), dt, q0[m]);
    }
  }
  if (A.update) {
    // the next stage reads primitive variables: one conversion here for the
    // three families' loads (and bprtest's test of that stage's input)
    if (A.prim_out) to_prim(gamma, qmin_rho, qmin_p, st, qw);
#pragma unroll
    for (int m = 0; m < 5; ++m) A.qout[co + m * P3] = qw[m];
  }
}

// i-face rows of one task.  OUT 0: fluxes stored; 1: D = F(c+1) - F(c) of the
// 30 cells between the task's 31 faces
template <bool MIXED, bool CONV, bool MV, bool LIM1, int OUT, bool VIS>
__device__ __forceinline__ void line_i(const FaceTask &T, const LinePar &LP, const LineArgs &L, StageI<VIS> &B, int lane) {
  const DevBlock &b = L.blocks[T.blk];
  const PhysPar &ph = LP.ph;
  const int n = T.n, nh = n * LP.hbmove, k = T.tb, mx = b.im;
  const bool fo = L.first_order != 0;
  const StrongMap &sm = L.smap[T.blk];
  const bool strong = sm.off[0][0] >= 0 || sm.off[0][1] >= 0;
  int st = 0;
  // lane l: cell c, column l + 1; lanes 0 and 31 also bring columns 0 and 33.
  // Cells past the line's last halo cell repeat it, faces past the line repeat
  // the last metrics; nothing of them is stored.
  const int c = T.i0 - 1 + lane;
  const bool face = lane >= 1 && c >= 1 && c <= mx, edge = lane == 0 || lane == 31;
  const int ecol = lane == 0 ? 0 : 33, ce = lane == 0 ? c - 1 : c + 1;
  const bool in_0 = c >= 1 && c <= mx - 1, in_e = ce >= 1 && ce <= mx - 1;
  const unsigned P3 = (unsigned)b.P3, qrow = (unsigned)b.I3;
  const double *qb = L.q + p3_var(b, 5, LP.S, 1, n) + p3_cell(b, 0, T.ta, k);
  const unsigned o0 = (unsigned)min(c, mx + 1), oe = (unsigned)min(ce, mx + 1);
  const int64_t e0 = p2_idx(b, LP.S2, 1, min(c, mx), T.ta, k, nh);
  const double *sp = L.s[0] + e0, *vp = MV ? L.fv.f[0] + e0 / 4 * 3 : nullptr;
  const unsigned fv = (unsigned)b.im * (unsigned)b.jm * (unsigned)b.km;  // variable stride of an F0 array
  double *Fp = L.cf + f0_idx(b, 5, LP.S, min(max(c, 1), mx), T.ta, k, 1, n);
  const int64_t mrow = (int64_t)(b.im + 2) * 4;
  const int frow = b.im;
  const double *Vp = VIS ? L.vf + f0_idx(b, 5, LP.S, min(max(c, 1), mx), T.ta, k, 1, n) : nullptr;
  auto issue = [&](int slot) {
#pragma unroll
    for (int m = 0; m < 5; ++m) cp8(&B.q[slot][m][lane + 1], qb + (int)o0 + (int64_t)m * P3);
    if (edge) {
#pragma unroll
      for (int m = 0; m < 5; ++m) cp8(&B.q[slot][m][ecol], qb + (int)oe + (int64_t)m * P3);
    }
    cp16(&B.met[slot][0][lane], sp);
    cp16(&B.met[slot][1][lane], sp + 2);
    if (VIS) {
#pragma unroll
      for (int m = 0; m < 5; ++m) cp8(&B.vis[slot][VIS ? m : 0][lane], Vp + (int64_t)m * fv);
    }
    cp_commit();
  };
  issue(0);
  for (int row = 0; row < T.nf; ++row) {
    const int slot = row & 1;
    __syncwarp();  // every lane is done with the slot that is filled next
    if (row + 1 < T.nf) {
      qb += qrow;
      sp += mrow;
      if (VIS) Vp += frow;
      issue(slot ^ 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    double qm[5], q0[5], qp[5], F[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) q0[m] = B.q[slot][m][lane + 1];
    if (CONV) {
      if (in_0) {
        to_prim(LP.gamma, LP.qmin_rho, LP.qmin_p, st, q0);
#pragma unroll
        for (int m = 1; m < 5; ++m) B.q[slot][m][lane + 1] = q0[m];
      }
      if (edge && in_e) {
        double v[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) v[m] = B.q[slot][m][ecol];
        to_prim(LP.gamma, LP.qmin_rho, LP.qmin_p, st, v);
#pragma unroll
        for (int m = 1; m < 5; ++m) B.q[slot][m][ecol] = v[m];
      }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 5; ++m) { qm[m] = B.q[slot][m][lane]; qp[m] = B.q[slot][m][lane + 2]; }
    const double2 ma = B.met[slot][0][lane], mb = B.met[slot][1][lane];
    const double met[4] = {ma.x, ma.y, mb.x, mb.y};
    bool slo = false, shi = false;
    if (strong) {
      slo = strong_at(L.strong, sm, 0, 0, T.ta + row, k);
      shi = strong_at(L.strong, sm, 0, 1, T.ta + row, k);
    }
    if (!MIXED) {
      double qr[5], ql[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        double a = q0[m] - qm[m], bb = qp[m] - q0[m];
        if (strong) {
          // per-slope doubling on strong-boundary faces (muscl_b*, src/flux.f90:1318-1406)
          if ((c == 1 && slo) || (c == mx && shi)) a = a * 2;
          if ((c == 0 && slo) || (c == mx - 1 && shi)) bb = bb * 2;
        }
        double up;
        if (fo) { qr[m] = q0[m]; up = q0[m]; }
        else cell_states64<LIM1>(ph.ilimf, ph.epslimf, ph.rkap, q0[m], a, bb, qr[m], up);
        ql[m] = __shfl_up_sync(0xffffffffu, up, 1);
      }
      if (strong) {
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          if (c == 1 && slo) { qr[m] = qm[m]; ql[m] = qm[m]; }
          if (c == mx && shi) { qr[m] = q0[m]; ql[m] = q0[m]; }
        }
      }
      const double ubn = MV ? face_ubn(vp, met[0], met[1], met[2]) : 0.0;
      roe_flux_euler<MV>(ph, met[0], met[1], met[2], met[3], qr, ql, F, ubn);
    } else {
      const float eps32 = (float)ph.epslimf, rk32 = (float)ph.rkap;
      float dqL[5], dqR[5], b0[5], bm1[5], dlr[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        float a = (float)(q0[m] - qm[m]), bb = (float)(qp[m] - q0[m]);
        dlr[m] = a;
        b0[m] = (float)q0[m];
        bm1[m] = (float)qm[m];
        if (strong) {
          if ((c == 1 && slo) || (c == mx && shi)) a = a * 2.0f;
          if ((c == 0 && slo) || (c == mx - 1 && shi)) bb = bb * 2.0f;
        }
        float dm = 0.0f;
        dqR[m] = 0.0f;
        if (!fo) limit_cell32(LIM1 ? 1 : ph.ilimf, eps32, rk32, a, bb, dqR[m], dm);
        dqL[m] = __shfl_up_sync(0xffffffffu, dm, 1);
      }
      if (strong) {
#pragma unroll
        for (int m = 0; m < 5; ++m) {
          if (c == 1 && slo) { dqL[m] = 0.0f; dqR[m] = -dlr[m]; }  // both states = cell L
          if (c == mx && shi) { dqL[m] = dlr[m]; dqR[m] = 0.0f; }  // both states = cell R
        }
      }
      const double ubn = MV ? face_ubn(vp, met[0], met[1], met[2]) : 0.0;
      face_flux_mixed<MV>(ph, (float)ph.g, (float)ph.g_gm1, met, qm, bm1, b0, dlr, dqL, dqR, F, ubn);
    }
    if (VIS) {
#pragma unroll
      for (int m = 0; m < 5; ++m) F[m] = F[m] + B.vis[slot][VIS ? m : 0][lane];
    }
    if (OUT == 0) {
      if (face) {
#pragma unroll
        for (int m = 0; m < 5; ++m) Fp[(int64_t)m * fv] = F[m];
      }
    } else {
#pragma unroll
      for (int m = 0; m < 5; ++m) F[m] = __shfl_down_sync(0xffffffffu, F[m], 1) - F[m];
      if (lane >= 1 && lane <= 30 && c <= mx - 1) {
#pragma unroll
        for (int m = 0; m < 5; ++m) Fp[(int64_t)m * fv] = F[m];
      }
    }
    Fp += frow;
    if (MV) vp += mrow / 4 * 3;
  }
  if (CONV && st && L.status) atomicOr(L.status, st);
}

// a segment of j or k faces, lanes along i.  OUT 0: fluxes stored; 1: the
// flux differences of the segment's nf - 1 cells added to D; 2: D with them
// added goes through finish_cell
template <bool MIXED, bool CONV, bool MV, bool LIM1, int OUT, bool RMS, bool VIS>
__device__ __forceinline__ void line_m(const FaceTask &T, const LinePar &LP, const LineArgs &L, const StageArgs &A,
                                       const cosa_params *Pp, int part_row, StageM<OUT, VIS> &B, int lane) {
  const DevBlock &b = L.blocks[T.blk];
  const PhysPar &ph = LP.ph;
  const int d = T.d, n = T.n, nh = n * LP.hbmove, tb = T.tb, f0 = T.f0, f1 = T.f0 + T.nf;
  const bool fo = L.first_order != 0;
  const int mx = d == 2 ? b.jm : b.km;
  int st = 0;
  const bool act = T.i0 + lane <= b.im - 1;
  const int i = min(T.i0 + lane, b.im - 1);
  bool slo, shi;
  {
    const StrongMap &sm = L.smap[T.blk];
    slo = d == 2 ? strong_at(L.strong, sm, 1, 0, i, tb) : strong_at(L.strong, sm, 2, 0, i, tb);
    shi = d == 2 ? strong_at(L.strong, sm, 1, 1, i, tb) : strong_at(L.strong, sm, 2, 1, i, tb);
  }
  const unsigned P3 = (unsigned)b.P3;
  const unsigned step = d == 2 ? (unsigned)b.I3 : (unsigned)b.I3 * (unsigned)b.J3;
  const int64_t mstep = d == 2 ? (int64_t)(b.im + 2) * 4 : (int64_t)(b.im + 2) * (b.jm + 2) * 4;
  const unsigned fstep = d == 2 ? (unsigned)b.im : (unsigned)b.im * (unsigned)b.jm;
  const unsigned fv = (unsigned)b.im * (unsigned)b.jm * (unsigned)b.km;
  const int64_t cell0 = p3_var(b, 5, LP.S, 1, n) + (d == 2 ? p3_cell(b, i, f0, tb) : p3_cell(b, i, tb, f0));
  const double *pq = L.q + cell0;  // cell f0
  const int64_t e0 = d == 2 ? p2_idx(b, LP.S2, 1, i, f0, tb, nh) : p2_idx(b, LP.S2, 1, i, tb, f0, nh);
  const double *sp = (d == 2 ? L.s[1] : L.s[2]) + e0;
  const double *vp = MV ? (d == 2 ? L.fv.f[1] : L.fv.f[2]) + e0 / 4 * 3 : nullptr;
  double *Fp = L.cf + (OUT == 0 ? (int64_t)(d - 1) * L.n0 * 5 * LP.S : 0) +
               (d == 2 ? f0_idx(b, 5, LP.S, i, f0, tb, 1, n) : f0_idx(b, 5, LP.S, i, tb, f0, 1, n));
  const double *Vp = VIS ? L.vf + (int64_t)(d - 1) * L.nv * 5 * LP.S +
                               (d == 2 ? f0_idx(b, 5, LP.S, i, f0, tb, 1, n) : f0_idx(b, 5, LP.S, i, tb, f0, 1, n))
                         : nullptr;
  double qc[5];
  double acc[5] = {0, 0, 0, 0, 0};
  // the running left state: cell f - 1 on face f; FP64: ql the state, a the
  // slope of cell f (doubled at a strong boundary); mixed: dm the FP32 offset
  // from cell f - 1 (qb, fb), sB the undoubled slope
  double a[5], ql[5], qb[5];
  float dm[5], sB[5], fb[5], fc[5];
  const float eps32 = (float)ph.epslimf, rk32 = (float)ph.rkap;
  // step f's data: cell f + 1, the metrics of face f; the chain: D, base state
  // and time step of cell f - 1.  All addresses advance by constant strides
  // (computed afresh, 420 instructions a cell in the last launch, a cycle of the
  // 30.7 M-cell duct took 17.0 ms, now 16.0)
  const double *nq = pq + step, *ns = sp, *nD = Fp, *nb = nullptr, *nt = nullptr;
  int64_t co = cell0;
  if (OUT == 2) {
    nb = A.qold + cell0;
    nt = A.dtvol + (d == 2 ? p1_idx(b, LP.S, i, f0, tb, n) : p1_idx(b, LP.S, i, tb, f0, n));
  }
  const int64_t tstep = d == 2 ? (int64_t)(b.im + 1) : (int64_t)(b.im + 1) * (b.jm + 1);
  auto issue = [&](bool first, int slot) {
#pragma unroll
    for (int m = 0; m < 5; ++m) cp8(&B.q[slot][m][lane], nq + (int64_t)m * P3);
    nq += step;
    cp16(&B.met[slot][0][lane], ns);
    cp16(&B.met[slot][1][lane], ns + 2);
    ns += mstep;
    if (VIS) {
#pragma unroll
      for (int m = 0; m < 5; ++m) cp8(&B.vis[slot][VIS ? m : 0][lane], Vp + (int64_t)m * fv);
      Vp += fstep;
    }
    if (OUT >= 1 && !first) {
#pragma unroll
      for (int m = 0; m < 5; ++m) cp8(&B.D[slot][m][lane], nD + (int64_t)m * fv);
      nD += fstep;
      if (OUT == 2 && A.update) {
#pragma unroll
        for (int m = 0; m < 5; ++m) cp8(&B.base[slot][m][lane], nb + (int64_t)m * P3);
        nb += step;
        cp8(&B.base[slot][OUT == 2 ? 5 : 0][lane], nt);
        nt += tstep;
      }
    }
    cp_commit();
  };
  issue(true, f0 & 1);
  {
    double qa[5], q1[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double *p = pq + (int64_t)m * P3;
      qa[m] = __ldg(p - 2 * (int64_t)step);
      q1[m] = __ldg(p - (int64_t)step);
      qc[m] = __ldg(p);
    }
    if (CONV) {
      // interior: cells 1 .. mx - 1, tested where they are marched over
      int skip = 0;
      if (f0 - 2 >= 1) to_prim(LP.gamma, LP.qmin_rho, LP.qmin_p, skip, qa);
      if (f0 - 1 >= 1) to_prim(LP.gamma, LP.qmin_rho, LP.qmin_p, skip, q1);
      if (f0 <= mx - 1) to_prim(LP.gamma, LP.qmin_rho, LP.qmin_p, st, qc);
    }
    const bool dlo = f0 == 2 && slo, dmi = (f0 == 1 && slo) || (f0 == mx && shi);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      if (!MIXED) {
        double a0 = q1[m] - qa[m];
        a[m] = qc[m] - q1[m];
        if (dlo) a0 = a0 * 2;
        if (dmi) a[m] = a[m] * 2;
        double lo_;
        if (fo) ql[m] = q1[m];
        else cell_states64<LIM1>(ph.ilimf, ph.epslimf, ph.rkap, q1[m], a0, a[m], lo_, ql[m]);
        if (f0 == 1 && slo) ql[m] = q1[m];  // strong lower boundary: both states of face 1 are cell 0
      } else {
        const float a0 = (float)(q1[m] - qa[m]);
        sB[m] = (float)(qc[m] - q1[m]);
        qb[m] = q1[m];
        fb[m] = (float)q1[m];
        fc[m] = (float)qc[m];
        float lo_;
        dm[m] = 0.0f;
        if (!fo) limit_cell32(LIM1 ? 1 : ph.ilimf, eps32, rk32, dlo ? a0 * 2.0f : a0, dmi ? sB[m] * 2.0f : sB[m], lo_, dm[m]);
        if (f0 == 1 && slo) dm[m] = 0.0f;
      }
    }
  }
  double Fprev[5];
  for (int f = f0; f < f1; ++f) {
    const int slot = f & 1;
    if (f + 1 < f1) {
      issue(false, slot ^ 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    double qn[5], F[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) qn[m] = B.q[slot][m][lane];
    if (CONV && f + 1 <= mx - 1) to_prim(LP.gamma, LP.qmin_rho, LP.qmin_p, st, qn);
    if (!MIXED) {
      double qr[5], up[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        double bb = qn[m] - qc[m];
        if (f + 1 == mx && shi) bb = bb * 2;
        if (fo) { qr[m] = qc[m]; up[m] = qc[m]; }
        else cell_states64<LIM1>(ph.ilimf, ph.epslimf, ph.rkap, qc[m], a[m], bb, qr[m], up[m]);
        a[m] = bb;
      }
      if (f == 1 && slo) {
#pragma unroll
        for (int m = 0; m < 5; ++m) qr[m] = ql[m];
      }
      if (f == mx && shi) {
#pragma unroll
        for (int m = 0; m < 5; ++m) { qr[m] = qc[m]; ql[m] = qc[m]; }
      }
#pragma unroll
      for (int m = 0; m < 5; ++m) qc[m] = qn[m];
      const double2 ma = B.met[slot][0][lane], mb = B.met[slot][1][lane];
      const double ubn = MV ? face_ubn(vp, ma.x, ma.y, mb.x) : 0.0;
      roe_flux_euler<MV>(ph, ma.x, ma.y, mb.x, mb.y, qr, ql, F, ubn);
#pragma unroll
      for (int m = 0; m < 5; ++m) ql[m] = up[m];
    } else {
      float dqL[5], dqR[5], bbv[5], up[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        bbv[m] = (float)(qn[m] - qc[m]);
        const float al = (f == 1 && slo) || (f == mx && shi) ? sB[m] * 2.0f : sB[m];
        dqL[m] = dm[m];
        dqR[m] = 0.0f;
        up[m] = 0.0f;
        if (!fo) limit_cell32(LIM1 ? 1 : ph.ilimf, eps32, rk32, al, f + 1 == mx && shi ? bbv[m] * 2.0f : bbv[m], dqR[m], up[m]);
        if (f == 1 && slo) dqR[m] = -sB[m];
        if (f == mx && shi) { dqL[m] = sB[m]; dqR[m] = 0.0f; }
      }
      const double2 ma = B.met[slot][0][lane], mb = B.met[slot][1][lane];
      const double met[4] = {ma.x, ma.y, mb.x, mb.y};
      const double ubn = MV ? face_ubn(vp, met[0], met[1], met[2]) : 0.0;
      face_flux_mixed<MV>(ph, (float)ph.g, (float)ph.g_gm1, met, qb, fb, fc, sB, dqL, dqR, F, ubn);
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        qb[m] = qc[m];
        qc[m] = qn[m];
        fb[m] = fc[m];
        fc[m] = (float)qn[m];
        sB[m] = bbv[m];
        dm[m] = up[m];
      }
    }
    if (VIS) {
#pragma unroll
      for (int m = 0; m < 5; ++m) F[m] = F[m] + B.vis[slot][VIS ? m : 0][lane];
    }
    if (OUT == 0) {
      if (act) {
#pragma unroll
        for (int m = 0; m < 5; ++m) Fp[(int64_t)m * fv] = F[m];
      }
      Fp += fstep;
    } else {
      if (f > f0 && act) {
        // bresid order: i, then j, then k (src/cosa.f90:1800-1876)
        double D[5];
#pragma unroll
        for (int m = 0; m < 5; ++m) D[m] = B.D[slot][m][lane] + F[m] - Fprev[m];
        if (OUT == 1) {
#pragma unroll
          for (int m = 0; m < 5; ++m) Fp[(int64_t)m * fv] = D[m];
        } else {
          double q0[5];
#pragma unroll
          for (int m = 0; m < 5; ++m) q0[m] = B.base[slot][OUT == 2 ? m : 0][lane];
          const double ov = A.vol ? Pp->omega * A.vol[p1_idx(b, 1, i, tb, f - 1, 0)] : 0.0;
          finish_cell<RMS>(A, *Pp, LP.S, n, co, (int64_t)P3, ov, B.base[slot][OUT == 2 ? 5 : 0][lane], D, q0,
                           LP.gamma, LP.qmin_rho, LP.qmin_p, acc, st);
        }
      }
      if (f > f0) { Fp += fstep; co += step; }
#pragma unroll
      for (int m = 0; m < 5; ++m) Fprev[m] = F[m];
    }
    if (MV) vp += mstep / 4 * 3;
  }
  if (OUT == 2 && RMS) {
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      double x = acc[m];
      for (int w = 16; w > 0; w >>= 1) x += __shfl_down_sync(0xffffffffu, x, w);
      if (lane == 0) A.part[(int64_t)part_row * 8 + m] = x;
    }
  }
  if (st && L.status) atomicOr(L.status, st);
}

// Resident warps per SM that the line kernels are compiled for.  FP64 i lines
// and the store kernel at 16 (128 registers, a few words spilled), the marching
// chain kernels at 12 (168 registers).  Measured, one cycle of the 30.7 M-cell
// duct: i lines at 12 / 16 / 18 warps 16.95 / 16.84 / - ms; marching at 11 /
// 12 / 14 warps 17.3 / 16.8 / 18.9 ms (spills).  Five cycles of the pitching
// aerofoil (store) at 10 / 14 / 16 warps 1.59 / 1.55 / 1.49 ms.  Mixed
// precision fits 16 everywhere (18: 6.2 against 5.2 ms on the 4.2 M-cell duct).
constexpr int kWarpsStore = 16, kWarpsI = 16, kWarpsM = 12, kWarpsMixed = 16;

// store schedule: all faces, the task's family picks the loop.  VIS: viscous
// flows, whose stage input is the primitive copy and whose faces add their
// viscous flux (a flux balance of its own moved 200 B a cell more: one cycle of
// the 4.2 M-cell laminar duct 7.27 ms with it, 6.17 ms without)
template <bool MIXED, bool CONV, bool MV, bool LIM1, bool VIS>
__global__ void __launch_bounds__(32, MIXED ? kWarpsMixed : kWarpsStore)
k_line_store(const LinePar LP, const LineArgs L) {
  __shared__ union {
    StageI<VIS> i;
    StageM<0, VIS> m;
  } B;
  const FaceTask T = L.tasks[blockIdx.x];
  if (T.d == 1) line_i<MIXED, CONV, MV, LIM1, 0, VIS>(T, LP, L, B.i, threadIdx.x);
  else line_m<MIXED, CONV, MV, LIM1, 0, false, VIS>(T, LP, L, StageArgs{}, nullptr, 0, B.m, threadIdx.x);
}
// chain schedule: family FAM; FAM 3 finishes the stage
template <int FAM, bool MIXED, bool CONV, bool LIM1, bool RMS, bool VIS>
__global__ void __launch_bounds__(32, MIXED ? kWarpsMixed : FAM == 1 ? kWarpsI : kWarpsM)
k_line_chain(const LinePar LP, const LineArgs L, const StageArgs A, const cosa_params *__restrict__ Pp) {
  const FaceTask T = L.tasks[blockIdx.x];
  if constexpr (FAM == 1) {
    __shared__ StageI<VIS> B;
    line_i<MIXED, CONV, false, LIM1, 1, VIS>(T, LP, L, B, threadIdx.x);
  } else {
    __shared__ StageM<FAM - 1, VIS> B;
    line_m<MIXED, CONV, false, LIM1, FAM - 1, RMS, VIS>(T, LP, L, A, Pp, blockIdx.x, B, threadIdx.x);
  }
}
