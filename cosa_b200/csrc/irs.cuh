// Implicit residual smoothing (cirs_b / ccirs_b, src/cosa.f90:2035-2443,
// 5206-5650): the tridiagonal solves of one direction, gw lines per warp (32;
// 16 or 8 where longer lines would not fit shared memory).
//
// Row m of a line's system is -e_m x_{m-1} + (1 + 2 e_m) x_m - e_m x_{m+1} =
// r_m (first and last rows without the outer term).  A lane sweeps one line of
// one variable (tridi, src/cosa.f90:2418-2443) with the right-hand sides
// staged in shared memory, so the global accesses are coalesced in every
// direction (i lines are transposed on the way in and out) and the sweep's
// chain is two operations a row forward and one back.  With a constant
// coefficient (irsop 1) the pivots are the same on every line and come from a
// table made once (irs_pivots); else each lane makes its line's pivots on the
// way, one reciprocal a row.
//
// The first direction can take the scaling by dt/V (scalef) with its loads
// and the last one its inverse (scaleb) with its stores.
//
// Bound by the sweep's chain and the latency of its loads at a few hundred
// lines, by memory (read and write of R per direction) on large grids; groups
// are narrower while the launch would leave the chip idle.  Before: cyclic
// reduction, one warp per line and variable, the matrix eliminated anew for
// each variable with two divisions a row and step, and two scaling passes.
// Five cycles on the 512 x 128 x 2 aerofoil grid: laminar 4.10 -> 3.69 ms,
// k-omega 7.5 -> 7.1 ms; k-omega SST on 128 x 32 x 2 2.37 -> 2.09 ms.  Sweeps
// with plain staged loads were slower than the reduction (5.7 ms laminar).
#pragma once
#include "faces.cuh"

// doubles of shared memory of one warp: the lines, their pivots when the
// coefficient varies, and the factors of a scaled first direction
__host__ __device__ __forceinline__ int irs_warp_doubles(int nmax, int gw, bool const_eps, bool scaled) {
  return (1 + (const_eps ? 0 : 1) + (scaled ? 1 : 0)) * gw * (nmax | 1);
}

template <int D, bool CONST_EPS>
__global__ void k_irs_tri(BlockList bs_, int npde, int S, double *__restrict__ res, const double *__restrict__ ores,
                          const double *__restrict__ beta, const double2 *__restrict__ piv, double eps, int vs, int ve,
                          int with_halo, int nmax, int gw, const double *__restrict__ fin, const double *__restrict__ fint,
                          const double *__restrict__ fout, const double *__restrict__ foutt) {
  extern __shared__ double irs_sm[];
  const DevBlock b = bs_.get();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int im = b.im - 1, jm = b.jm - 1, km = b.km - 1;
  const int len = D == 1 ? im : (D == 2 ? jm : km);
  // D = 1: a group is gw consecutive (j, k) lines; else gw consecutive i at one transverse index
  const int nlines = jm * km, nig = (im + gw - 1) / gw, nt = D == 2 ? km : jm;
  const int ngrp = D == 1 ? (nlines + gw - 1) / gw : nig * nt;
  const int64_t nwork = (int64_t)ngrp * S * (ve - vs + 1);
  const int row = nmax | 1;
  double *x = irs_sm + (size_t)warp * irs_warp_doubles(nmax, gw, CONST_EPS, fin != nullptr);
  double *rr = x + gw * row;                     // coefficients, then ratios r_m (varying coefficient)
  double *ff = x + (CONST_EPS ? 1 : 2) * gw * row;  // factors of the first direction
  auto at = [&](int m) { return D == 1 ? lane * row + m : m * gw + lane; };
  for (int64_t w = blockIdx.x * (int64_t)nw + warp; w < nwork; w += (int64_t)gridDim.x * nw) {
    int64_t q_ = w;
    const int g = (int)(q_ % ngrp); q_ /= ngrp;
    const int s = (int)(q_ % S), v = vs + (int)(q_ / S);
    const int64_t base = p3_var(b, npde, S, v, s);
    const double *src = (ores ? ores : res) + base;
    double *dst = res + base;
    const double *fi = v >= 6 ? fint : fin, *fo = v >= 6 ? foutt : fout;
    // this lane's line
    const int line = g * gw + lane;
    const int i = D == 1 ? 1 : (g % nig) * gw + lane + 1;
    const int t3 = D == 1 ? line / jm + 1 : g / nig + 1, t2 = D == 1 ? line % jm + 1 : i;
    const bool act = lane < gw && (D == 1 ? line < nlines : i <= im);
    const int nl = D == 1 ? min(gw, nlines - g * gw) : 0;
    // first cell of the line in the state and in the coefficient arrays, and
    // the strides along it
    const int64_t c0 = act ? (D == 1 ? p3_cell(b, 1, t2, t3) : D == 2 ? p3_cell(b, i, 1, t3) : p3_cell(b, i, t3, 1)) : 0;
    const int64_t e0 = act ? (D == 1 ? p1_idx(b, S, 1, t2, t3, s) : D == 2 ? p1_idx(b, S, i, 1, t3, s)
                                                                           : p1_idx(b, S, i, t3, 1, s)) : 0;
    const int64_t cs = D == 1 ? 1 : D == 2 ? (int64_t)b.I3 : (int64_t)b.I3 * b.J3;
    const int64_t es = D == 1 ? 1 : D == 2 ? (int64_t)b.im + 1 : (int64_t)(b.im + 1) * (b.jm + 1);
    __syncwarp();
    // all of the lines' right-hand sides (and factors, coefficients) are
    // requested at once: asynchronous copies, i lines row by row (coalesced)
    if (D == 1) {
      for (int r = 0; r < nl; ++r) {
        const int64_t cr = __shfl_sync(0xffffffffu, c0, r), er = __shfl_sync(0xffffffffu, e0, r);
        for (int m = lane; m < len; m += 32) {
          cp8(&x[r * row + m], src + cr + m);
          if (!CONST_EPS) cp8(&rr[r * row + m], beta + er + m);
          if (fi) cp8(&ff[r * row + m], fi + er + m);
        }
      }
    } else if (act) {
      for (int m = 0; m < len; ++m) {
        cp8(&x[m * gw + lane], src + c0 + m * cs);
        if (!CONST_EPS) cp8(&rr[m * gw + lane], beta + e0 + m * es);
        if (fi) cp8(&ff[m * gw + lane], fi + e0 + m * es);
      }
    }
    cp_commit();
    cp_wait<0>();
    __syncwarp();
    if (act) {
      double h1 = 0.0, h2 = 0.0;
      if (with_halo) {
        // the last row's halo wins on a single-cell line, as in ccirs_b
        if (len > 1) h1 = (CONST_EPS ? eps : rr[at(0)]) * dst[c0 - cs];
        h2 = (CONST_EPS ? eps : rr[at(len - 1)]) * dst[c0 + len * cs];
      }
      // rows in batches of 8, a batch's shared-memory and table reads before
      // its chain (a store between two reads would order them)
      constexpr int NB = 8;
      double t = 0.0, r = 0.0;
      for (int m0 = 0; m0 < len; m0 += NB) {
        double y[NB], c[NB], f[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const int m = min(m0 + u, len - 1);
          y[u] = x[at(m)];
          c[u] = CONST_EPS ? __ldg(&piv[m].y) : rr[at(m)];
          f[u] = fi ? ff[at(m)] : 1.0;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const int m = m0 + u;
          if (m >= len) break;
          double v_ = fi ? y[u] * f[u] : y[u];
          if (with_halo) v_ += (m == 0 ? h1 : 0.0) + (m == len - 1 ? h2 : 0.0);
          if (CONST_EPS) {
            t = fma(eps, t, v_) * c[u];
          } else {
            const double e = c[u], inv = rcp_nr(fma(r, e, 1 + 2 * e));
            r = -e * inv;
            c[u] = r;
            t = fma(e, t, v_) * inv;
          }
          y[u] = t;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          if (m0 + u >= len) break;
          x[at(m0 + u)] = y[u];
          if (!CONST_EPS) rr[at(m0 + u)] = c[u];
        }
      }
      double *dl = dst + c0 + (len - 1) * cs;
      const double *fl = fo ? fo + e0 + (len - 1) * es : nullptr;
      if (D != 1) *dl = fo ? t * rcp_nr(*fl) : t;
      for (int m0 = len - 2; m0 >= 0; m0 -= NB) {
        double y[NB], c[NB], f[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          const int m = max(m0 - u, 0);
          y[u] = x[at(m)];
          c[u] = CONST_EPS ? __ldg(&piv[m].x) : rr[at(m)];
          f[u] = D != 1 && fo ? __ldg(fl - (int64_t)min(u + 1, m0 + 1) * es) : 1.0;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          if (m0 - u < 0) break;
          t = fma(-c[u], t, y[u]);
          if (D == 1) x[at(m0 - u)] = t;
          else dl[-(int64_t)(u + 1) * cs] = fo ? t * rcp_nr(f[u]) : t;
        }
        dl -= NB * cs;
        if (fo) fl -= NB * es;
      }
    }
    if (D == 1) {
      __syncwarp();
      for (int r = 0; r < nl; ++r) {
        const int64_t cr = __shfl_sync(0xffffffffu, c0, r), er = __shfl_sync(0xffffffffu, e0, r);
#pragma unroll 4
        for (int m = lane; m < len; m += 32) {
          const double y = x[r * row + m];
          dst[cr + m] = fo ? y * rcp_nr(fo[er + m]) : y;
        }
      }
    }
  }
}

// ratios r_m and reciprocal pivots of the constant-coefficient system (rows 1
// .. n; the last row of a shorter line has the same pivot, and its ratio is
// not used)
__global__ void k_irs_pivots(int n, double eps, double2 *__restrict__ piv) {
  if (blockIdx.x || threadIdx.x) return;
  double r = 0.0;
  for (int m = 0; m < n; ++m) {
    const double inv = 1.0 / fma(r, eps, 1 + 2 * eps);
    r = -eps * inv;
    piv[m] = make_double2(r, inv);
  }
}
