// Fused RK stage for sm_100a: halo fill, stage arguments, norm reduction.
//
// One RK stage of smooth() (src/cosa.f90:1719-2016) for the explicit Euler
// path is cons2prim -> bc -> cutman_q -> prtest -> [lambda, deltat] ->
// muscl/roflux/resid x3 -> prim2cons -> [resg_rms] -> update: about 25
// full-array sweeps.  Here it is k_halo, then the line kernels of faces.cuh:
//
//  k_halo        two threads per boundary/cut face cell and snapshot: read
//                the interior next to the face, convert it to primitive form
//                (first stage; later stages hold primitive values), apply the
//                BC (or the cut copy) and write the primitive halo values
//                into the halo slots of the same state array.  Halo cells
//                written twice in the reference keep the reference's last
//                writer (mask computed on the host).
#pragma once
#include "physics.cuh"
#include "kernels_ref.cuh"

// one boundary or cut face cell: 48 bytes, read as three 16-byte words.
// Cell indices inside a block fit 32 bits (2^31 cells are 17 GB a variable).
struct __align__(16) HaloItem {
  int h1, h2;       // halo cells (p3 cell index in dblk)
  int c1, c2;       // interior cells (p3 cell index in sblk)
  int dblk, sblk;   // destination / source block (0-based)
  unsigned mface;   // metric cell index (i + I2*(j + J2*k)) of the face in dblk
  int ps;           // slot of the flow conditions (BC values) in the params array
  int type;         // BC type, -1 = cut copy
  signed char idir; // direction of the face (1..3)
  signed char mask; // bit0: write first halo layer, bit1: second
  signed char sgn;  // sign applied to the face normal
  signed char nl;   // multigrid level of the item's block (the low-speed cut-off epsp(nl))
  int pad[2];
};

// strong-boundary flags of one block: for each direction d and side s
// (0 = min, 1 = max) a byte per tangential cell (t2,t3), t2 fastest, with
// (t2,t3) = (j,k) for d=1, (i,k) for d=2, (i,j) for d=3 (1-based cells).
struct StrongMap {
  int64_t off[3][2];
  int n2[3];
};

__device__ __forceinline__ bool strong_at(const uint8_t *flags, const StrongMap &m, int d, int side, int t2, int t3) {
  const int64_t o = m.off[d][side];
  if (o < 0) return false;
  return flags[o + (t2 - 1) + (int64_t)m.n2[d] * (t3 - 1)] != 0;
}

// ---- k_halo ------------------------------------------------------------------------
// face velocities of a moving grid, the reference's sijk(5:7) of the three
// families: (3, 0:imax+1, 0:jmax+1, 0:kmax+1, 0:S2-1) per block at op2*3*S2
struct FaceVel {
  const double *f[3];
};

// the boundary values of every flow-condition slot and level (make_bcpar:
// sines, cosines and a power), once per upload of the parameters instead of
// once per halo cell: k_halo on the 24-block duct of 4.2 M cells (463 k items)
// took 92 us with them inside, on the 128 x 64 x 2 channel 19.7 us
__global__ void k_bcpar(const cosa_params *__restrict__ Pp, int nslots, BcPar *__restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nslots * COSA_MAX_LEVELS) out[t] = make_bcpar(Pp[t / COSA_MAX_LEVELS], t % COSA_MAX_LEVELS + 1);
}

// scalars of k_halo, passed by value
struct HaloPar {
  int S, S2, hbmove, test;  // test: bprtest of the i halos (fused stages)
  double gamma, qmin_rho, qmin_p;
};
inline HaloPar make_halo_par(const cosa_params &P, int test) {
  HaloPar h;
  h.test = test;
  h.S = 2 * P.nharms + 1; h.S2 = 2 * P.nharms * P.hbmove + 1; h.hbmove = P.hbmove;
  h.gamma = P.gamma; h.qmin_rho = P.qmin[0]; h.qmin_p = P.qmin[4];
  return h;
}

// Bound by the latency of one item's chain on small grids, by the strided
// cells of the i faces on large ones.  SPLIT: two threads per item, one per
// halo layer (neighbouring lanes share the item), for launches that leave the
// chip idle anyway: the subsonic inlet's two Newton iterations, the longest
// chain here (powers), run side by side (kHaloSplit in cosa_gpu.cu).
// Snapshot n = blockIdx.y.
template <bool CONS, int NV, bool SPLIT>
__global__ void __launch_bounds__(128)
k_halo(const DevBlock *__restrict__ blocks, const HaloItem *__restrict__ items, int nitems,
       const HaloPar H, const cosa_params *__restrict__ Pp, const BcPar *__restrict__ bcp,
       double *__restrict__ q, const double *__restrict__ si, const double *__restrict__ sj,
       const double *__restrict__ sk, int *status, const double *__restrict__ dist = nullptr,
       FaceVel fvel = FaceVel{{nullptr, nullptr, nullptr}}) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t item = SPLIT ? t >> 1 : t;
  if (item >= nitems) return;
  const int n = blockIdx.y;
  const HaloItem it = items[item];
  // the layers of this thread; a layer that a later item overwrites is not
  // written, but an inlet's Newton iteration is checked wherever it stands
  const int mine = SPLIT ? 1 << (int)(t & 1) : 3;
  int write = it.mask & mine;
  if (!write && it.type != 21) return;
  int st = 0;
  const DevBlock &db = blocks[it.dblk], &sb = blocks[it.sblk];
  const double *qs = q + p3_var(sb, NV, H.S, 1, n);
  const int64_t sP3 = sb.P3, dP3 = db.P3;
  double h1[NV], h2[NV];
  if (it.type < 0) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if (mine & 1) h1[v] = qs[v * sP3 + it.c1];
      if (mine & 2) h2[v] = qs[v * sP3 + it.c2];
    }
    if (CONS) {
      if (mine & 1) { if (NV > 5) c2p7(H.gamma, h1); else c2p5(H.gamma, h1); }
      if (mine & 2) { if (NV > 5) c2p7(H.gamma, h2); else c2p5(H.gamma, h2); }
    }
  } else {
    double c1[NV], c2[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      c1[v] = qs[v * sP3 + it.c1];
      c2[v] = qs[v * sP3 + it.c2];
    }
    double nx = 0, ny = 0, nz = 0;
    if (it.type == 14 || it.type == 21 || it.type == 30 || it.type == 31 || (NV > 5 && it.type / 100 == 15)) {
      const double *s = it.idir == 1 ? si : (it.idir == 2 ? sj : sk);
      const int64_t I2 = db.im + 2, J2 = db.jm + 2, K2 = db.km + 2;
      const int64_t e = ((db.op2 * H.S2) + (int64_t)(n * H.hbmove) * I2 * J2 * K2 + it.mface) * 4;
      const double2 a = __ldg(reinterpret_cast<const double2 *>(s + e));
      nx = a.x * it.sgn; ny = a.y * it.sgn; nz = __ldg(s + e + 2) * it.sgn;
    }
    if (CONS) {
      if (NV > 5) { c2p7(H.gamma, c1); c2p7(H.gamma, c2); }
      else { c2p5(H.gamma, c1); c2p5(H.gamma, c2); }
    }
    const BcPar &B = bcp[it.ps * COSA_MAX_LEVELS + it.nl - 1];
    int err = 0;
    // moving walls: the velocity of the wall face (snapshot nh)
    double wv[3];
    const double *wvp = nullptr;
    const double *f = it.idir == 1 ? fvel.f[0] : (it.idir == 2 ? fvel.f[1] : fvel.f[2]);
    if ((it.type == 14 || it.type / 100 == 15) && f) {
      const int64_t I2 = db.im + 2, J2 = db.jm + 2, K2 = db.km + 2;
      const int64_t e = ((db.op2 * H.S2) + (int64_t)(n * H.hbmove) * I2 * J2 * K2 + it.mface) * 3;
      wv[0] = f[e]; wv[1] = f[e + 1]; wv[2] = f[e + 2];
      wvp = wv;
    }
    int mask = 0;
    switch (it.type) {
      case 80: mask = bc_sym(it.idir, NV, c1, c2, h1, h2); break;
      case 4: mask = bc_extrapol(NV, c1, h1, h2); break;
      case 14: mask = bc_walinv(NV, nx, ny, nz, c1, c2, h1, h2, wvp); break;
      case 21:
        if (SPLIT) {
          bc_insub_layer<NV>(B, nx, ny, nz, c1, c2, (int)(t & 1), h1, &err);
#pragma unroll
          for (int v = 0; v < NV; ++v) h2[v] = h1[v];
        } else {
          bc_insub_layer<NV>(B, nx, ny, nz, c1, c2, 0, h1, &err);
          bc_insub_layer<NV>(B, nx, ny, nz, c1, c2, 1, h2, &err);
        }
        mask = 3;
        break;
      case 91: mask = bc_outsub<NV>(B, c1, c2, h1, h2); break;
      case 30: mask = bc_far0<NV>(B, nx, ny, nz, c1, h1, h2); break;
      case 31: mask = bc_far1<NV>(B, nx, ny, nz, c1, h1, h2); break;
      default:
        if (it.type / 100 == 15) {
          mask = bc_walvis(H.gamma, c1, c2, h1, h2, wvp);
          if (NV > 5) {
            // k-omega wall values from the wall distance of the first cell
            if (!dist) { st |= COSA_ERR_ARG; break; }
            const int I3 = db.I3, J3 = db.J3;
            const int ci = it.c1 % I3 - 1, cj = (it.c1 / I3) % J3 - 1, ck = it.c1 / (I3 * J3) - 1;
            bc_walvis_kom(*Pp, nx, ny, nz, dist[p1_idx(db, 1, ci, cj, ck, 0)], c1, h1, h2, wvp);
          }
        } else {
          st |= COSA_ERR_UNSUPPORTED;
        }
        break;
    }
    if (err) st |= COSA_ERR_INFLOW;
    write &= mask;
  }
  double *qd = q + p3_var(db, NV, H.S, 1, n);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    if (write & 1) qd[v * dP3 + it.h1] = h1[v];
    if (write & 2) qd[v * dP3 + it.h2] = h2[v];
  }
  if (H.test && it.idir == 1) {  // bprtest also checks the i halos of the state (src/cosa.f90:1000)
    if (write & 1) { if (h1[4] <= H.qmin_p) st |= COSA_ERR_NEG_P; else if (h1[0] <= H.qmin_rho) st |= COSA_ERR_NEG_RHO; }
    if (write & 2) { if (h2[4] <= H.qmin_p) st |= COSA_ERR_NEG_P; else if (h2[0] <= H.qmin_rho) st |= COSA_ERR_NEG_RHO; }
  }
  if (st) atomicOr(status, st);
}

// ---- stage arguments ------------------------------------------------------------------
struct StageArgs {
  const double *qin;     // stage input
  double *qout;          // stage output (interior written)
  const double *qold;    // RK base state q^n
  double *qold_copy;     // if set, q^n interior is copied here (stage 1)
  double *dtvol;         // Delta t / V
  const double *si, *sj, *sk;
  double *part;          // residual sums of squares (8 doubles per row) or null
  double *rhs;           // multigrid forcing term of a coarse level, or null
  int rhs_mode;          // 1: r -= rhs; 2: rhs += r first (forcing), then r -= rhs
  double *res_out;       // if set, the residual is stored here (P3 layout)
  double *bx, *by, *bz;  // IRS coefficients written with the time step (irsop >= 2)
  const double *vol;     // cell volumes when the harmonic-balance source is on
  const uint8_t *strong; // strong-boundary flags
  const StrongMap *smap; // per block
  int *status;
  double ar;
  int compute_dt;
  int first_order;
  int update;            // 0: residual only (restriction pass)
  int prim_out;          // 1: the output's interior is stored primitive (the next stage reads it so)
  const double *cfl_blk; // per-block CFL number (serving: each solve's own), or null for P.cfl
};

// ---- deterministic reduction of partial rows -> resrms ------------------
// many rows (the chain's last launch has one per warp) are first summed to
// gridDim.x rows, row p of `part` into row p % gridDim.x
__global__ void k_rms_mid(const double *__restrict__ part, int nparts, int npde, double *__restrict__ out) {
  __shared__ double red[8][8];
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int64_t p = blockIdx.x + (int64_t)gridDim.x * threadIdx.x; p < nparts; p += (int64_t)gridDim.x * blockDim.x)
    for (int v = 0; v < npde; ++v) acc[v] += part[p * 8 + v];
  for (int v = 0; v < npde; ++v) {
    double x = acc[v];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[v][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < npde) {
    double x = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) x += red[threadIdx.x][w];
    out[(int64_t)blockIdx.x * 8 + threadIdx.x] = x;
  }
}

// resg_rms (src/cosa.f90:4458-4501): sqrt(sum/ncell), total sqrt(sum/ncell/npde)
__global__ void k_rms_final(const double *__restrict__ part, int nparts, int npde, double ncell,
                            double *__restrict__ out, int *row_counter, int nrows_max) {
  __shared__ double red[8][32];
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int p = threadIdx.x; p < nparts; p += blockDim.x)
    for (int v = 0; v < npde; ++v) acc[v] += part[(int64_t)p * 8 + v];
  for (int v = 0; v < npde; ++v) {
    double x = acc[v];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[v][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    double tot[8], all = 0;
    for (int v = 0; v < npde; ++v) {
      double x = 0;
      for (int w = 0; w < nw; ++w) x += red[v][w];
      tot[v] = x;
      all = all + x;
    }
    int row = 0;
    if (row_counter) { row = *row_counter; if (row < nrows_max) *row_counter = row + 1; else row = nrows_max - 1; }
    double *o = out + (int64_t)row * (npde + 1);
    for (int v = 0; v < npde; ++v) o[v] = sqrt(tot[v] / ncell);
    o[npde] = sqrt(all / ncell / npde);
  }
}

// per-segment version of k_rms_final: CTA s reduces rows [seg[2s], +seg[2s+1])
// in the same fixed order into out[s * (npde + 1) ...]
__global__ void k_rms_seg(const double *__restrict__ part, const int *__restrict__ seg,
                          const double *__restrict__ seg_ncell, int npde, double *__restrict__ out) {
  __shared__ double red[8][32];
  const int s = blockIdx.x;
  const double *pp = part + (int64_t)seg[2 * s] * 8;
  const int nparts = seg[2 * s + 1];
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int p = threadIdx.x; p < nparts; p += blockDim.x)
    for (int v = 0; v < npde; ++v) acc[v] += pp[(int64_t)p * 8 + v];
  for (int v = 0; v < npde; ++v) {
    double x = acc[v];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[v][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    const double ncell = seg_ncell[s];
    double tot[8], all = 0;
    for (int v = 0; v < npde; ++v) {
      double x = 0;
      for (int w = 0; w < nw; ++w) x += red[v][w];
      tot[v] = x;
      all = all + x;
    }
    double *o = out + (int64_t)s * (npde + 1);
    for (int v = 0; v < npde; ++v) o[v] = sqrt(tot[v] / ncell);
    o[npde] = sqrt(all / ncell / npde);
  }
}

// ---- interior copy (odd stage counts end in the second buffer) --------------------------
template <class BS>
__global__ void k_copy_interior(BS bs_, int nvar_snap, const double *__restrict__ src, double *__restrict__ dst) {
  const DevBlock b = bs_.get();
  const int ni = b.im - 1, nj = b.jm - 1, nk = b.km - 1;
  const int64_t n = (int64_t)ni * nj * nk * nvar_snap;
  const int64_t base = b.op3 * nvar_snap;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = t;
    const int i = (int)(r % ni) + 1; r /= ni;
    const int j = (int)(r % nj) + 1; r /= nj;
    const int k = (int)(r % nk) + 1; r /= nk;
    const int64_t o = base + r * b.P3 + p3_cell(b, i, j, k);
    dst[o] = src[o];
  }
}

// ---- stage finalisation: face halos of q in conservative form ----------------------------
// After smooth(), the reference's q holds prim2cons of the last stage's
// halo values (src/cosa.f90:1908).  src holds those values in primitive form.
template <int NV>
__global__ void k_halo_p2c(const DevBlock *__restrict__ blocks, const HaloItem *__restrict__ items, int nitems,
                           int S, double gamma, const double *__restrict__ src, double *__restrict__ dst) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nitems) return;
  const HaloItem it = items[t];
  const DevBlock &db = blocks[it.dblk];
  const int64_t P3 = db.P3, o = p3_var(db, NV, S, 1, blockIdx.y);
  double v[2][NV];
#pragma unroll
  for (int m = 0; m < NV; ++m) {
    v[0][m] = src[o + m * P3 + it.h1];
    v[1][m] = src[o + m * P3 + it.h2];
  }
  p2c(gamma, v[0], NV);
  p2c(gamma, v[1], NV);
#pragma unroll
  for (int m = 0; m < NV; ++m) {
    if (it.mask & 1) dst[o + m * P3 + it.h1] = v[0][m];
    if (it.mask & 2) dst[o + m * P3 + it.h2] = v[1][m];
  }
}
