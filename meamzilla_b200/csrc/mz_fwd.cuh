// Forward kernels of the objective (see mz_device.cu for the call sequence).
#pragma once

#include "mz_spline.cuh"

namespace mzb {

// ------------------------------------------------------------------ k_prep

// Coefficient vectors -> per-candidate knot tables, one CTA per candidate.
// cmap has the table's layout: cmap[toff+k] (knot k) and cmap[toff+2n+e]
// (end e) hold the coefficient index, or -1 where the value is fixed and
// comes from base.  The work is a few hundred numbers, so only latency
// counts: the table is gathered by all threads into shared memory, y'' is
// the refresh matrix M times (y, end slopes), a lane per row, and all threads
// write the results.  One thread per spline walking global memory through
// the tridiagonal solve (a serial chain of divisions) took 20 us of a 70 us
// call (one candidate, 3 splines of 8 to 10 knots); the solve, still a thread
// per spline but in shared memory, serves callers without M.
// SM: the table and the solve's scratch fit shared memory (prep_smem);
// otherwise they stay in global memory (tabs and ptabs hold them).
__host__ __device__ inline size_t prep_smem(int stride) { return sizeof(double) * 2 * (size_t)stride; }

template <bool SM>
__global__ void __launch_bounds__(256)
    k_prep(int P, const double *__restrict__ params, const double *__restrict__ base, const int *__restrict__ cmap,
           const SplineGeom *__restrict__ geom, const int *__restrict__ nat, int nsplines, int stride,
           double *__restrict__ tabs, int pstride, double *__restrict__ ptabs, float *__restrict__ ptabf,
           float *__restrict__ wtab, int s_g, int ng, int nbp, const double *__restrict__ M) {
  extern __shared__ double psm[];
  const int c = blockIdx.x, tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const double *pc = params + (size_t)c * P;
  double *gtab = tabs + (size_t)c * stride, *gp = ptabs + (size_t)c * pstride;
  double *tab = SM ? psm : gtab;
  for (int e = tid; e < stride; e += T) tab[e] = cmap[e] >= 0 ? pc[cmap[e]] : base[e];
  __syncthreads();
  for (int s = tid; s < nsplines && !M; s += T) {
    const SplineGeom g = geom[s];
    if (g.q5) continue;
    // Spline3Eq::refresh_basis (spline3eq.cpp:192-225)
    const int n = g.n;
    double *y = tab + g.toff, *ypp = y + n;
    double *u = SM ? psm + stride + g.toff : gp + g.poff;  // n values; the pieces below overwrite them
    const double inv = g.invstep;
    const double gl = y[2 * n], gr = y[2 * n + 1];
    if (nat[2 * s]) {
      ypp[0] = 0;
      u[0] = 0;
    } else {
      ypp[0] = -0.5;
      u[0] = (3.0 * inv) * ((y[1] - y[0]) * inv - gl);
    }
    for (int i = 1; i < n - 1; ++i) {
      double p = 0.5 * ypp[i - 1] + 2.0;
      ypp[i] = (-0.5) / p;
      double ui = (y[i + 1] - y[i]) * inv - (y[i] - y[i - 1]) * inv;
      u[i] = (6.0 * ui * 0.5 * inv - 0.5 * u[i - 1]) / p;
    }
    double qn, un;
    if (nat[2 * s + 1]) {
      qn = un = 0.0;
    } else {
      qn = 0.5;
      un = (3.0 * inv) * (gr - (y[n - 1] - y[n - 2]) * inv);
    }
    ypp[n - 1] = (un - qn * u[n - 2]) / (qn * ypp[n - 2] + 1.0);
    for (int k = n - 2; k >= 0; --k) ypp[k] = ypp[k] * ypp[k + 1] + u[k];
  }
  // With M, ypp = M (y, grad) (spline5eq: (ypp, yp4) = M (y, grad, grad2)): the
  // refreshes (Spline3Eq::refresh_basis, Spline5Eq::refresh_basis,
  // spline5eq.cpp:209-293) are linear, and M is solved once on the host.  A
  // warp per spline, a lane per row.  A cubic's row r takes y - y_r, which its
  // y'' depend on alone (the solve forms the same differences): the products
  // of y itself would cancel, and their rounding grow with a constant in y.
  for (int s = warp; s < nsplines && M; s += T / 32) {
    const SplineGeom g = geom[s];
    const int n = g.n, nc = g.q5 ? n + 4 : n + 2;
    double *t = tab + g.toff;
    const double *g2 = t + 3 * n + 2;
    for (int r = lane; r < (g.q5 ? 2 * n : n); r += 32) {
      const double *row = M + g.moff + (size_t)r * nc, y0 = g.q5 ? 0.0 : t[r];
      double acc = 0.0;
#pragma unroll 4
      for (int q = 0; q < n; ++q) acc += row[q] * (t[q] - y0);
      acc += row[n] * t[2 * n] + row[n + 1] * t[2 * n + 1];
      if (g.q5) acc += row[n + 2] * g2[0] + row[n + 3] * g2[1];
      if (r < n) t[n + r] = acc;
      else t[2 * n + 2 + r - n] = acc;
    }
  }
  __syncthreads();
  if (SM)
    for (int e = tid; e < stride; e += T) gtab[e] = tab[e];
  // evaluation tables: the polynomial of every interval in its shift, and
  // their FP32 copy (mixed precision).  A warp per spline, a lane per interval.
  for (int s = warp; s < nsplines; s += T / 32) {
    const SplineGeom g = geom[s];
    const int n = g.n;
    const double *y = tab + g.toff, *ypp = y + n;
    if (g.q5) {
      const double *yp4 = y + 2 * n + 2;
      const double H2 = g.step * g.step / 6.0, H4 = g.step * g.step * g.step * g.step / 360.0;
      for (int k = lane; k < n - 1; k += 32) {
        const double p1 = y[k], p2 = y[k + 1], d21 = ypp[k], d22 = ypp[k + 1], d41 = yp4[k], d42 = yp4[k + 1];
        double q[6];
        q[0] = p1;
        q[1] = p2 - p1 + H2 * (-2.0 * d21 - d22) + H4 * (8.0 * d41 + 7.0 * d42);
        q[2] = 3.0 * H2 * d21;
        q[3] = H2 * (d22 - d21) + H4 * (-20.0 * d41 - 10.0 * d42);
        q[4] = 15.0 * H4 * d41;
        q[5] = H4 * (3.0 * d42 - 3.0 * d41);
        for (int j = 0; j < 6; ++j) {
          gp[g.poff + 6 * k + j] = q[j];
          if (ptabf) ptabf[(size_t)c * pstride + g.poff + 6 * k + j] = (float)q[j];
        }
      }
      continue;
    }
    const double H = g.step * g.step / 6.0;
    for (int k = lane; k < n - 1; k += 32) {
      double q[4];
      q[0] = y[k];
      q[1] = y[k + 1] - y[k] - (2.0 * ypp[k] + ypp[k + 1]) * H;
      q[2] = 3.0 * ypp[k] * H;
      q[3] = (ypp[k + 1] - ypp[k]) * H;
      for (int j = 0; j < 4; ++j) {
        gp[g.poff + 4 * k + j] = q[j];
        if (ptabf) ptabf[(size_t)c * pstride + g.poff + 4 * k + j] = (float)q[j];
      }
    }
    if (wtab && lane == 0 && s >= s_g && s < s_g + ng) {
      // Cubic B-spline coefficients of g on its uniform grid (basis function m
      // centred on knot m-1): S(x_i) = (w_i + 4 w_i+1 + w_i+2)/6 and
      // S''(x_i) = (w_i - 2 w_i+1 + w_i+2)/h^2 give w_i+1 = y_i - h^2/6 y''_i,
      // and the two outer coefficients follow from S'' at the end knots.
      // Their differences are the coefficients of g' (times h) in the
      // quadratic B-spline basis; both are stored: [w_0 .. w_nbp-1, dw_0 .. dw_nbp-2].
      float *w = wtab + ((size_t)c * ng + (s - s_g)) * (2 * nbp - 1);
      const double h2 = g.step * g.step;
      double wm[66];
      for (int i = 0; i < n; ++i) wm[i + 1] = y[i] - h2 / 6.0 * ypp[i];
      wm[0] = h2 * ypp[0] + 2.0 * wm[1] - wm[2];
      wm[n + 1] = h2 * ypp[n - 1] + 2.0 * wm[n] - wm[n - 1];
      for (int i = 0; i < nbp; ++i) w[i] = i < n + 2 ? (float)wm[i] : 0.f;
      for (int i = 0; i + 1 < nbp; ++i) w[nbp + i] = i + 1 < n + 2 ? (float)(wm[i + 1] - wm[i]) : 0.f;
    }
  }
}

inline void prep_launch(int ncand, int P, const double *params, const double *base, const int *cmap,
                        const SplineGeom *geom, const int *nat, int nsplines, int stride, double *tabs, int pstride,
                        double *ptabs, float *ptabf, float *wtab, int s_g, int ng, int nbp, const double *M,
                        cudaStream_t st) {
  const size_t sm = prep_smem(stride);
  if (sm <= 48 * 1024)
    k_prep<true><<<ncand, 256, sm, st>>>(P, params, base, cmap, geom, nat, nsplines, stride, tabs, pstride, ptabs,
                                         ptabf, wtab, s_g, ng, nbp, M);
  else
    k_prep<false><<<ncand, 256, 0, st>>>(P, params, base, cmap, geom, nat, nsplines, stride, tabs, pstride, ptabs,
                                         ptabf, wtab, s_g, ng, nbp, M);
}

// ----------------------------------------------------------- atom blocks

// Shared state of one atom block, common to the forward and adjoint kernels.
struct BlockRows {
  int atom_lo, na, slot_lo, nslot;
};

__device__ __forceinline__ BlockRows block_rows(const DevDb &db, int blk) {
  BlockRows b;
  b.atom_lo = db.blk_atom0[blk];
  b.na = db.blk_atom0[blk + 1] - b.atom_lo;
  b.slot_lo = db.pair_off[b.atom_lo];
  b.nslot = db.pair_off[b.atom_lo + b.na] - b.slot_lo;
  return b;
}

// Owner atom of slot t: the last a with a_lo[a] <= t.
__device__ __forceinline__ int slot_owner(const int *a_lo, int na, int t) {
  int lo = 0, hi = na;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (a_lo[mid] <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Pair functions of one slot: phi, rho, f with slopes (pot_meam_spline.cpp:152-191).
template <bool MEAM, typename R>
struct PairEval {
  R ux, uy, uz, r, invr;
  R phi, dphi, rho, drho, f, df;
  int kphi, krho, kf, tj, pij;
  R bphi, brho, bf;
  R p[2], dp[2], bp[2];  // JMEAM p (p2) (pot_jmeam_spline.cpp:196-202)
  int kp[2];
};

template <bool MEAM, typename R, bool Q5 = false>
__device__ __forceinline__ PairEval<MEAM, R> eval_pair(const DevDb &db, const DevPot &pot, const SplineGeom *sg,
                                                      const R *ptab, int64_t gs, int ti) {
  PairEval<MEAM, R> p;
  const int64_t Np = db.npairs;
  if (sizeof(R) == 8) {
    p.ux = (R)db.pair_ux[gs]; p.uy = (R)db.pair_uy[gs]; p.uz = (R)db.pair_uz[gs]; p.r = (R)db.pair_r[gs];
  } else {
    p.ux = (R)db.pair_uxf[gs]; p.uy = (R)db.pair_uyf[gs]; p.uz = (R)db.pair_uzf[gs]; p.r = (R)db.pair_rf[gs];
  }
  p.invr = R(1) / p.r;
  const int kn = db.pair_knot[gs];
  p.kphi = (kn & 0xff) - 1;
  p.krho = ((kn >> 8) & 0xff) - 1;
  p.kf = ((kn >> 16) & 0xff) - 1;
  p.tj = db.atom_type[db.pair_nbr[gs]];
  p.pij = pair_ij_index(ti, p.tj, pot.ntypes);
  p.phi = p.dphi = p.rho = p.drho = p.f = p.df = R(0);
  p.bphi = p.brho = p.bf = R(0);
  if (p.kphi >= 0) {
    const SplineGeom &g = sg[pot.s_phi + p.pij];
    p.bphi = sizeof(R) == 8 ? (R)db.pair_shift[gs] : (R)db.pair_shiftf[gs];
    p.phi = piece_val_grad<Q5, R>(ptab + g.poff, p.kphi, p.bphi, (R)g.invstep, p.dphi, g.q5);
  }
  if (p.krho >= 0) {
    const SplineGeom &g = sg[pot.s_rho + p.tj];
    p.brho = sizeof(R) == 8 ? (R)db.pair_shift[Np + gs] : (R)db.pair_shiftf[Np + gs];
    p.rho = piece_val_grad<Q5, R>(ptab + g.poff, p.krho, p.brho, (R)g.invstep, p.drho, g.q5);
  }
  if (MEAM && p.kf >= 0) {
    const SplineGeom &g = sg[pot.s_f + p.pij];
    p.bf = sizeof(R) == 8 ? (R)db.pair_shift[2 * Np + gs] : (R)db.pair_shiftf[2 * Np + gs];
    p.f = piece_val_grad<Q5, R>(ptab + g.poff, p.kf, p.bf, (R)g.invstep, p.df, g.q5);
  }
  return p;
}

// The JMEAM radial functions p (p2) of one slot.
template <bool MEAM, typename R, bool Q5 = false>
__device__ __forceinline__ void eval_pair_p(const DevDb &db, const DevPot &pot, const SplineGeom *sg, const R *ptab,
                                            int64_t gs, PairEval<MEAM, R> &p) {
  const int64_t Np = db.npairs;
  const int kn = db.pair_knot[gs];
  p.kp[0] = ((kn >> 24) & 0xff) - 1;
  p.kp[1] = pot.nj > 1 ? (int)db.pair_knot_p2[gs] : -1;
  for (int m = 0; m < 2; ++m) {
    p.p[m] = p.dp[m] = p.bp[m] = R(0);
    if (m < pot.nj && p.kp[m] >= 0) {
      const SplineGeom &g = sg[pot.s_p[m] + p.pij];
      p.bp[m] = sizeof(R) == 8 ? (R)db.pair_shift[(3 + m) * Np + gs] : (R)db.pair_shiftf[(3 + m) * Np + gs];
      p.p[m] = piece_val_grad<Q5, R>(ptab + g.poff, p.kp[m], p.bp[m], (R)g.invstep, p.dp[m], g.q5);
    }
  }
}

// ------------------------------------------------------------------ k_atoms

// Shared-memory layout of k_atoms (dynamic), see atoms_smem_bytes():
//   double red[10][BLOCK_SLOTS]       per-slot partials for the per-atom sums
//   double a_dF[BLOCK_ATOMS], a_U[BLOCK_ATOMS]
//   SplineGeom sg[nsplines]
//   int a_lo[BLOCK_ATOMS+2]
//   R ptab[pstride]                    this candidate's evaluation table
//   R4 srow[BLOCK_SLOTS]               (u_x, u_y, u_z, f) of every slot of the block
//   int stype[BLOCK_SLOTS+8]           neighbour type of every slot (GMEAM)
//   R spv[nj][BLOCK_SLOTS+8]           JMEAM p (p2) of every slot
template <typename R>
struct Vec4;
template <>
struct Vec4<float> {
  using T = float4;
};
template <>
struct Vec4<double> {
  using T = double4;
};

template <typename R>
__host__ __device__ inline size_t atoms_smem_bytes(int nsplines, int pstride, int nj = 0) {
  size_t b = sizeof(double) * (10 * BLOCK_SLOTS + 2 * BLOCK_ATOMS);
  b += sizeof(SplineGeom) * nsplines;
  b += sizeof(int) * (BLOCK_ATOMS + 2);
  b = (b + 31) & ~size_t(31);
  b += sizeof(R) * (pstride + 4);
  b = (b + 31) & ~size_t(31);
  b += 4 * sizeof(R) * (BLOCK_SLOTS + 8);
  b += sizeof(int) * (BLOCK_SLOTS + 8);  // neighbour type of every slot (GMEAM's g index)
  b += sizeof(R) * (size_t)nj * (BLOCK_SLOTS + 8);
  return b;
}

// g spline of the triplet (i; j, k) in GMEAM: Triplet_i_jk
// (PotFns::get_3body_alloy_idx, pot_fns.cpp:166-168).
__device__ __forceinline__ int gmeam_g_index(const DevPot &pot, int ti, int tj, int tk) {
  return pot.s_g + ti * pot.npair + pair_ij_index(tj, tk, pot.ntypes);
}

// Dot product of unit vectors: exact (no fused multiply-add, as the
// reference computes Triplet::cos) in FP64, fused in FP32.
__device__ __forceinline__ double cos_dot(double ax, double ay, double az, double bx, double by, double bz) {
  return cos_exact(ax, ay, az, bx, by, bz);
}
__device__ __forceinline__ float cos_dot(float ax, float ay, float az, float bx, float by, float bz) {
  return fmaf(ax, bx, fmaf(ay, by, az * bz));
}

// Row sums of one angular channel for slot `tid`: with w_k the partner's
// radial weight (f_k for g, p_k for a JMEAM q) and s the channel's spline,
//   S = sum_k s(cos) w_k,  T = sum_k s'(cos) w_k cos,  v = sum_k s'(cos) w_k u_k
// over the row's other slots whose cosine has a knot of s.  FP32 chunks of 8
// terms are added to FP64 totals (as the g loop of k_atoms).
template <bool Q5, typename R, typename R4, class W>
__device__ __forceinline__ void channel_row_sums(const R4 *srow, W weight, int row_lo, int row_hi, int tid, R ux,
                                                 R uy, R uz, const SplineGeom &gs, const R *spc, double &S, double &T,
                                                 double &vx, double &vy, double &vz) {
  const R x0 = (R)gs.x0, inv = (R)gs.invstep, cut = g_cut<R>(gs);
  S = T = vx = vy = vz = 0.0;
  for (int kb = row_lo; kb < row_hi; kb += 8) {
    R s8 = 0, t8 = 0, x8 = 0, y8 = 0, z8 = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = kb + u;
      const R4 o = srow[k];
      const R cs = cos_dot(ux, uy, uz, o.x, o.y, o.z);
      const bool ok = (k < row_hi) && (k != tid) && (cs < cut);
      const R wk = ok ? weight(k) : R(0);
      R b;
      const int kk = g_knot<R>(cs, x0, inv, gs.n, b);
      R ds;
      const R sv = piece_val_grad<Q5, R>(spc, kk, b, inv, ds, gs.q5);
      const R dsw = ds * wk;
      s8 += sv * wk;
      t8 += dsw * cs;
      x8 += dsw * o.x;
      y8 += dsw * o.y;
      z8 += dsw * o.z;
    }
    S += (double)s8;
    T += (double)t8;
    vx += (double)x8;
    vy += (double)y8;
    vz += (double)z8;
  }
}


// Warp-cooperative sum over the slots [lo, hi) of `n` per-slot arrays
// red[q * BLOCK_SLOTS + s]; the result is valid on lane 0.  Fixed order.
template <int NQ>
__device__ __forceinline__ void warp_slot_sums(const double *red, int lo, int hi, int lane, double *out) {
#pragma unroll
  for (int q = 0; q < NQ; ++q) out[q] = 0.0;
  for (int s = lo + lane; s < hi; s += 32) {
#pragma unroll
    for (int q = 0; q < NQ; ++q) out[q] += red[q * BLOCK_SLOTS + s];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    for (int o = 16; o > 0; o >>= 1) out[q] += __shfl_down_sync(0xffffffffu, out[q], o);
}

// One CTA per (atom block, candidate), one thread per pair slot.  A single
// pass over each slot's row gives G_p, H_p and vk_p; the density
// rho_i = sum_p rho_p + 1/2 sum_p f_p G_p (each j<k triplet seen from both
// ends) and every force term follow from them (pot_meam_spline.cpp:143-269):
//   V_p = u_p (phi'_p/2 + rho'_p U') + U' [u_p (f'_p G_p - f_p H_p / r_p)
//                                          + f_p vk_p / r_p]
// is the force atom i's terms add to atom i along slot p; the neighbour
// receives -V_p (k_force).  In FP32 the row sums are taken in chunks of 8
// terms, each chunk added to an FP64 total.
template <bool MEAM, typename R, bool AUX, bool GM = false, bool JM = false, bool Q5 = false>
__global__ void __launch_bounds__(BLOCK_SLOTS, JM ? 2 : sizeof(R) == 4 ? 4 : 3)
    k_atoms(DevDb db, DevPot pot, const SplineGeom *__restrict__ geom, const double *__restrict__ tabs,
            const double *__restrict__ ptabs, double *__restrict__ Vout, double *__restrict__ aout,
            double *__restrict__ aux) {
  using R4 = typename Vec4<R>::T;
  extern __shared__ __align__(32) unsigned char smem_raw[];
  const int cand = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  const int N = db.natoms;
  const int64_t Np = db.npairs;

  double *red = reinterpret_cast<double *>(smem_raw);
  double *a_dF = red + 10 * BLOCK_SLOTS;
  double *a_U = a_dF + BLOCK_ATOMS;
  SplineGeom *sg = reinterpret_cast<SplineGeom *>(a_U + BLOCK_ATOMS);
  int *a_lo = reinterpret_cast<int *>(sg + pot.nsplines);
  size_t off = sizeof(double) * (10 * BLOCK_SLOTS + 2 * BLOCK_ATOMS) + sizeof(SplineGeom) * pot.nsplines +
               sizeof(int) * (BLOCK_ATOMS + 2);
  off = (off + 31) & ~size_t(31);
  R *ptab = reinterpret_cast<R *>(smem_raw + off);
  off += sizeof(R) * (pot.pow_stride + 4);
  off = (off + 31) & ~size_t(31);
  R4 *srow = reinterpret_cast<R4 *>(smem_raw + off);
  int *stype = reinterpret_cast<int *>(srow + BLOCK_SLOTS + 8);
  R *spv = reinterpret_cast<R *>(stype + BLOCK_SLOTS + 8);

  const BlockRows br = block_rows(db, blockIdx.x);
  const double *tc = tabs + (size_t)cand * pot.tab_stride;
  const double *pc = ptabs + (size_t)cand * pot.pow_stride;
  for (int i = tid; i < pot.pow_stride; i += blockDim.x) ptab[i] = (R)pc[i];
  for (int i = tid; i < pot.nsplines; i += blockDim.x) sg[i] = geom[i];
  for (int a = tid; a <= br.na; a += blockDim.x) a_lo[a] = db.pair_off[br.atom_lo + a] - br.slot_lo;
  __syncthreads();

  const bool have = tid < br.nslot;
  const int me = have ? slot_owner(a_lo, br.na, tid) : 0;
  const int ti = db.atom_type[br.atom_lo + me];
  const int64_t gs = (int64_t)br.slot_lo + tid;

  PairEval<MEAM, R> pe;
  {
    R4 v;
    v.x = v.y = v.z = v.w = R(0);
    if (have) {
      pe = eval_pair<MEAM, R, Q5>(db, pot, sg, ptab, gs, ti);
      v.x = pe.ux; v.y = pe.uy; v.z = pe.uz; v.w = pe.f;
    }
    srow[tid] = v;
    if (tid < 8) srow[BLOCK_SLOTS + tid] = R4{};
    if (GM) {
      stype[tid] = have ? pe.tj : 0;
      if (tid < 8) stype[BLOCK_SLOTS + tid] = 0;
    }
    if (JM) {
      if (have) eval_pair_p<MEAM, R, Q5>(db, pot, sg, ptab, gs, pe);
      for (int m = 0; m < pot.nj; ++m) {
        spv[m * (BLOCK_SLOTS + 8) + tid] = have ? pe.p[m] : R(0);
        if (tid < 8) spv[m * (BLOCK_SLOTS + 8) + BLOCK_SLOTS + tid] = R(0);
      }
    }
  }
  __syncthreads();

  // ---- the one pass over the row: G_p, H_p, vk_p
  double G = 0, H = 0, vkx = 0, vky = 0, vkz = 0;
  if (GM && have && (AUX || pe.f != R(0) || pe.df != R(0))) {
    // GMEAM: the g spline depends on the partner's neighbour type as well
    const int row_lo = a_lo[me], row_hi = a_lo[me + 1];
    for (int kb = row_lo; kb < row_hi; kb += 8) {
      R g8 = 0, h8 = 0, x8 = 0, y8 = 0, z8 = 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = kb + u;
        const R4 o = srow[k];
        const SplineGeom &g2 = sg[gmeam_g_index(pot, ti, pe.tj, stype[k])];
        const R ginv = (R)g2.invstep;
        const R cs = cos_dot(pe.ux, pe.uy, pe.uz, o.x, o.y, o.z);
        const bool ok = (k < row_hi) && (k != tid) && (cs < g_cut<R>(g2));  // triplet_meam_spline.cpp:66-70
        const R fk = ok ? o.w : R(0);
        R b;
        const int kk = g_knot<R>(cs, (R)g2.x0, ginv, g2.n, b);
        R dg;
        const R gv = piece_val_grad<Q5, R>(ptab + g2.poff, kk, b, ginv, dg, g2.q5);
        const R dgfk = dg * fk;
        g8 += gv * fk;
        h8 += dgfk * cs;
        x8 += dgfk * o.x;
        y8 += dgfk * o.y;
        z8 += dgfk * o.z;
      }
      G += (double)g8;
      H += (double)h8;
      vkx += (double)x8;
      vky += (double)y8;
      vkz += (double)z8;
    }
    if (AUX) {
      double *ax = aux + (size_t)cand * (JM ? pot.aux_rows : (int)AUX_COUNT) * Np;
      ax[AUX_G * Np + gs] = G;
      ax[AUX_H * Np + gs] = H;
      ax[AUX_VX * Np + gs] = vkx;
      ax[AUX_VY * Np + gs] = vky;
      ax[AUX_VZ * Np + gs] = vkz;
    }
  } else if (!GM && MEAM && have && (AUX || pe.f != R(0) || pe.df != R(0))) {
    const SplineGeom gg = sg[pot.s_g + ti];
    const R *gpc = ptab + gg.poff;
    const R gx0 = (R)gg.x0, ginv = (R)gg.invstep;
    const R gcut = g_cut<R>(gg);
    const int row_lo = a_lo[me], row_hi = a_lo[me + 1];
    for (int kb = row_lo; kb < row_hi; kb += 8) {
      R g8 = 0, h8 = 0, x8 = 0, y8 = 0, z8 = 0;
      // Branch-free chunk of 8 partners: a partner that is this slot, past
      // the row, or not a triplet contributes with weight zero.  srow is
      // padded with zero rows past the block's last slot.
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = kb + u;
        const R4 o = srow[k];
        const R cs = cos_dot(pe.ux, pe.uy, pe.uz, o.x, o.y, o.z);
        const bool ok = (k < row_hi) && (k != tid) && (cs < gcut);  // triplet_meam_spline.cpp:66-70
        const R fk = ok ? o.w : R(0);
        R b;
        const int kk = g_knot<R>(cs, gx0, ginv, gg.n, b);
        R dg;
        const R gv = piece_val_grad<Q5, R>(gpc, kk, b, ginv, dg, gg.q5);
        const R dgfk = dg * fk;
        g8 += gv * fk;
        h8 += dgfk * cs;
        x8 += dgfk * o.x;
        y8 += dgfk * o.y;
        z8 += dgfk * o.z;
      }
      G += (double)g8;
      H += (double)h8;
      vkx += (double)x8;
      vky += (double)y8;
      vkz += (double)z8;
    }
    if (AUX) {
      double *ax = aux + (size_t)cand * (JM ? pot.aux_rows : (int)AUX_COUNT) * Np;
      ax[AUX_G * Np + gs] = G;
      ax[AUX_H * Np + gs] = H;
      ax[AUX_VX * Np + gs] = vkx;
      ax[AUX_VY * Np + gs] = vky;
      ax[AUX_VZ * Np + gs] = vkz;
    }
  }
  // ---- JMEAM: the same row sums for each (p, q) term (pot_jmeam_spline.cpp:208-219)
  double G2[2] = {0, 0}, H2[2] = {0, 0}, v2x[2] = {0, 0}, v2y[2] = {0, 0}, v2z[2] = {0, 0};
  if (JM && have) {
    for (int m = 0; m < pot.nj; ++m) {
      if (!AUX && pe.p[m] == R(0) && pe.dp[m] == R(0)) continue;
      const SplineGeom qg = sg[pot.s_q[m] + ti];
      const R *wm = spv + m * (BLOCK_SLOTS + 8);
      channel_row_sums<Q5, R>(srow, [&](int k) { return wm[k]; }, a_lo[me], a_lo[me + 1], tid, pe.ux, pe.uy, pe.uz,
                          qg, ptab + qg.poff, G2[m], H2[m], v2x[m], v2y[m], v2z[m]);
      if (AUX) {
        double *ax = aux + ((size_t)cand * pot.aux_rows + AUX_COUNT * (1 + m)) * Np;
        ax[AUX_G * Np + gs] = G2[m];
        ax[AUX_H * Np + gs] = H2[m];
        ax[AUX_VX * Np + gs] = v2x[m];
        ax[AUX_VY * Np + gs] = v2y[m];
        ax[AUX_VZ * Np + gs] = v2z[m];
      }
    }
  }
  if (have) red[tid] = (double)pe.rho + (MEAM ? 0.5 * (double)pe.f * G : 0.0);
  __syncthreads();

  // ---- embedding (pot_meam_spline.cpp:208-223): one warp per atom
  for (int a = warp; a < br.na; a += nwarp) {
    double rho;
    warp_slot_sums<1>(red, a_lo[a], a_lo[a + 1], lane, &rho);
    if (lane == 0 && pot.pair) {
      double *ao = aout + (size_t)cand * AO_COUNT * N;
      a_dF[a] = a_U[a] = 0.0;
      ao[AO_PEN * N + br.atom_lo + a] = 0.0;
      ao[AO_RHO * N + br.atom_lo + a] = 0.0;
    } else if (lane == 0) {
      const int ia = br.atom_lo + a;
      const SplineGeom &gU = sg[pot.s_U + db.atom_type[ia]];
      const double w = db.cell_w[db.atom_cell[ia]];
      double pen = 0.0;
      const double lo = gU.x0, hi = gU.xN;
      const double rho_raw = rho;
      if (rho < lo) {
        pen = w * 100.0 * 10. * (lo - rho) * (lo - rho);
        if (!pot.embed_extrap) rho = lo;
      } else if (rho > hi) {
        pen = w * 100.0 * 10. * (rho - hi) * (rho - hi);
        if (!pot.embed_extrap) rho = hi;
      }
      const PointEval U = spl_point_t<Q5>(tc, gU, rho);  // FP64 table of this candidate
      a_dF[a] = U.grad;
      a_U[a] = U.val;
      double *ao = aout + (size_t)cand * AO_COUNT * N;
      ao[AO_PEN * N + ia] = pen;
      ao[AO_RHO * N + ia] = rho_raw;
    }
  }
  __syncthreads();

  // ---- V_p and the slot's stress (stress.h:134-137; pot_meam_spline.cpp:171-173, 234-236, 265-268)
  if (have) {
    const double dF = a_dF[me];
    const double ux = (double)pe.ux, uy = (double)pe.uy, uz = (double)pe.uz;
    const double sp = MEAM ? 0.5 : phi_share(pot, db.pair_nbr[gs] == br.atom_lo + me);
    double cu = sp * (double)pe.dphi + (double)pe.drho * dF;
    double Vx = 0, Vy = 0, Vz = 0;
    double e3 = 0.0;  // JMEAM: 1/2 sum_m p_m G2_m, this slot's share of the p p q energy
    if (MEAM) {
      const double ip = (double)pe.invr, fp = (double)pe.f;
      cu += dF * ((double)pe.df * G - fp * ip * H);
      const double ck = dF * fp * ip;
      Vx = ck * vkx;
      Vy = ck * vky;
      Vz = ck * vkz;
      if (JM)
        for (int m = 0; m < pot.nj; ++m) {
          // the q terms' dfj without U' (pot_jmeam_spline.cpp:263-273)
          const double pm = (double)pe.p[m];
          cu += (double)pe.dp[m] * G2[m] - pm * ip * H2[m];
          Vx += pm * ip * v2x[m];
          Vy += pm * ip * v2y[m];
          Vz += pm * ip * v2z[m];
          e3 += 0.5 * pm * G2[m];
        }
    }
    Vx += ux * cu;
    Vy += uy * cu;
    Vz += uz * cu;
    double *Vc = Vout + ((size_t)cand * Np + gs) * db.vs;  // (x, y, z) per slot
    store_vec(Vc, db.vs, Vx, Vy, Vz);
    const double rr = db.pair_r[gs];
    const double dx = db.pair_ux[gs], dy = db.pair_uy[gs], dz = db.pair_uz[gs];
    red[0 * BLOCK_SLOTS + tid] = Vx;
    red[1 * BLOCK_SLOTS + tid] = Vy;
    red[2 * BLOCK_SLOTS + tid] = Vz;
    red[3 * BLOCK_SLOTS + tid] = sp * (double)pe.phi + e3;
    red[4 * BLOCK_SLOTS + tid] = -(dx * (Vx * rr));
    red[5 * BLOCK_SLOTS + tid] = -(dy * (Vy * rr));
    red[6 * BLOCK_SLOTS + tid] = -(dz * (Vz * rr));
    red[7 * BLOCK_SLOTS + tid] = -(dx * (Vy * rr));
    red[8 * BLOCK_SLOTS + tid] = -(dy * (Vz * rr));
    red[9 * BLOCK_SLOTS + tid] = -(dz * (Vx * rr));
  }
  __syncthreads();
  for (int a = warp; a < br.na; a += nwarp) {
    double acc[10];
    warp_slot_sums<10>(red, a_lo[a], a_lo[a + 1], lane, acc);
    if (lane == 0) {
      const int ia = br.atom_lo + a;
      double *ao = aout + (size_t)cand * AO_COUNT * N;
      ao[AO_AX * N + ia] = acc[0];
      ao[AO_AY * N + ia] = acc[1];
      ao[AO_AZ * N + ia] = acc[2];
      ao[AO_E * N + ia] = acc[3] + a_U[a];
#pragma unroll
      for (int q = 0; q < 6; ++q) ao[(AO_S0 + q) * N + ia] = acc[4 + q];
    }
  }
}

// ------------------------------------------------------------------ k_force

// F_i = sum of V over the atom's own slots - sum of V over the slots whose
// neighbour is i; then the force residual w (F - F0) (potential.cpp:468-478)
// and, for the adjoint, lambda_i = dF/dF_i = 2 w e_i.  Eight lanes per atom:
// a lane per atom walked its 16 to 60 incoming slots one dependent read after
// another (16 us for 21 k atoms of 16 slots, one candidate; this takes 6).
// The reads are scattered, and three 8-byte loads a slot kept the L1 busy 97 %
// of the time: V is stored as records of 32 bytes that one load fetches (18 k
// atoms of 42 slots, 128 candidates: 592 -> 558 us, 5.2 TB/s; k_rows, which
// writes them without staging, 1408 -> 1200 us there and 1171 -> 1145 us for
// 21 k atoms of 16 slots, 56 candidates).  Two candidates a thread gave 530 us
// there, but 48 for 35 us with one candidate.  V is packed to 24 bytes where
// the row kernels do not serve (spline5eq, rows of more than 128 slots), where
// records would make a launch hold fewer candidates than were asked for, and
// in the run without allocations, whose workspace the caller sized.
constexpr int FORCE_LANES = 8;

template <int VS>
__global__ void __launch_bounds__(256)
    k_force(DevDb db, const double *__restrict__ V, double *__restrict__ aout, double *__restrict__ forces,
            double *__restrict__ errvec, int esize, double *__restrict__ lam) {
  const int c = blockIdx.y, N = db.natoms, l = threadIdx.x % FORCE_LANES;
  const int i0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) / FORCE_LANES), i = min(i0, N - 1);
  double *ao = aout + (size_t)c * AO_COUNT * N;
  const double *Vc = V + (size_t)c * VS * db.npairs;
  const int q1 = db.in_off[i + 1], cell = db.atom_cell[i], comp = min(l, 2);
  const double own = ao[(AO_AX + comp) * N + i], f0 = db.force0[3 * i + comp];
  double f[3] = {0.0, 0.0, 0.0};
#pragma unroll 4
  for (int q = db.in_off[i] + l; q < q1; q += FORCE_LANES) {
    const double *v = Vc + VS * (int64_t)db.in_slot[q];
    double x, y, z;
    if (VS == 4) {
      load_vec4(v, x, y, z);
    } else {
      x = v[0];
      y = v[1];
      z = v[2];
    }
    f[0] += x;
    f[1] += y;
    f[2] += z;
  }
#pragma unroll
  for (int o = FORCE_LANES / 2; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 3; ++q) f[q] += __shfl_xor_sync(0xffffffffu, f[q], o);
  // lane l < 3 of the atom: component l
  const double w = db.cell_w[cell], F = own - (l == 0 ? f[0] : l == 1 ? f[1] : f[2]), r = w * (F - f0);
  double sq = r * r;
  sq += __shfl_xor_sync(0xffffffffu, sq, 1);      // lanes 0 and 1: x + y
  sq += __shfl_down_sync(0xffffffffu, r * r, 2);  // lane 0: + z
  if (i0 >= N) return;
  if (l == 0) ao[AO_FSQ * N + i] = sq;
  if (l < 3) {
    if (forces) forces[(size_t)c * 3 * N + 3 * i + l] = F;
    if (errvec) errvec[(size_t)c * esize + 7 * (cell + 1) + 3 * i + l] = r;
    if (lam) lam[((size_t)c * 3 + l) * N + i] = 2.0 * w * r;
  }
}

// ------------------------------------------------------------------ k_cells

// largest |y| of a spline's knots, by the lanes of a warp
__device__ __forceinline__ double warp_max_abs_y(const SplineGeom &g, const double *tab, int lane) {
  double m = 0.0;
  for (int k = lane; k < g.n; k += 32) m = fmax(m, fabs(tab[g.toff + k]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// Sum of the style's punishment entries squared; writes them to ev (may be
// null).  All lanes of one warp.
__device__ __forceinline__ double warp_punishments(const DevPot &pot, const SplineGeom *__restrict__ geom,
                                                   const double *__restrict__ tab, double *ev, int lane) {
  double total = 0.0;
  if (pot.pair) return 0.0;  // PotPairSpline::fast_compute, pot_pair_spline.cpp:133
  const bool meam = pot.style == MZ_STYLE_MEAM_SPLINE || pot.nj > 0;
  const int npen = pot.gmeam ? pot.npair : meam ? 1 + pot.nj : pot.ntypes;
  for (int q = 0; q < npen; ++q) {
    double e = 0.0;
    if (pot.omit_pen) {
    } else if (pot.gmeam || meam) {
      // f-potential magnitude punishment (pot_meam_spline.cpp:274-278), JMEAM's
      // p (p2) magnitudes (pot_jmeam_spline.cpp:286-299); GMEAM: one per f
      // spline (pot_gmeam_spline.cpp:173-178)
      const int s0 = pot.gmeam ? pot.s_f + q : q == 0 ? pot.s_f : pot.s_p[q - 1];
      const int ns = pot.gmeam ? 1 : pot.npair;
      double m = 0.0;
      for (int f = 0; f < ns; ++f) m = fmax(m, warp_max_abs_y(geom[s0 + f], tab, lane));
      e = 100. * 25. * (1.0 - m) * (1.0 - m);
    } else {
      // U'(mid-range) punishment per type (pot_eam_spline.cpp:211-218)
      const SplineGeom &g = geom[pot.s_U + q];
      e = 100. * spl_point_any(tab, g, 0.5 * (g.x0 + g.xN)).grad;
    }
    total += e * e;
    if (ev && lane == 0) ev[q] = e;
  }
  return total;
}

// One CTA per cell and candidate: energy per atom, stress / volume, constraint
// and the residual entries (potential.cpp:450-485), with `seeds` also the
// adjoint seeds dF/dE_atom, dF/dS_cell and dF/dpen of the cell.  The CTA that
// counts itself last of a candidate adds the cells' sums of squares in a
// fixed order, and the style's punishments, into the objective (the work of a
// launch of its own before: 9 us with one candidate).  count [ncand] is zero
// at every launch and left zero.  Every sum is in an order that depends on
// the database alone.  A warp per cell took 27 us on cells of up to 1024
// atoms (one candidate); a CTA per cell 10.
constexpr int CELL_T = 128;

__global__ void __launch_bounds__(CELL_T)
    k_cells(DevDb db, DevPot pot, const SplineGeom *__restrict__ geom, const double *__restrict__ tabs,
            const double *__restrict__ aout, double *cellobj, double *__restrict__ obj, double *__restrict__ errvec,
            int esize, double *__restrict__ energy, double *__restrict__ stress, double *__restrict__ seeds,
            int *count) {
  __shared__ double part[CELL_T / 32][9];
  __shared__ double tree[CELL_T];
  __shared__ int slast;
  const int cell = blockIdx.x, c = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = db.natoms, NC = db.ncells;
  const double *ao = aout + (size_t)c * AO_COUNT * N;
  const int a0 = db.cell_atom0[cell], a1 = db.cell_atom0[cell + 1];
  double v[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) v[q] = 0.0;
#pragma unroll 2
  for (int a = a0 + tid; a < a1; a += CELL_T) {
    v[0] += ao[AO_E * N + a];
#pragma unroll
    for (int q = 0; q < 6; ++q) v[1 + q] += ao[(AO_S0 + q) * N + a];
    v[7] += ao[AO_PEN * N + a];
    v[8] += ao[AO_FSQ * N + a];
  }
  if (a1 - a0 > 32 * warp) {  // warps past a small cell's atoms have nothing to sum
#pragma unroll
    for (int q = 0; q < 9; ++q)
      for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  }
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < 9; ++q) part[warp][q] = v[q];
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < 9; ++q)
      for (int w = 1; w < CELL_T / 32; ++w) v[q] += part[w][q];
    const int na = a1 - a0;
    const double w = db.cell_w[cell];
    const double E = v[0] / na;
    const double ew = w * db.cell_ew[cell] * pot.energy_weight;
    const double eE = ew * na * (E - db.cell_e0[cell]);
    double sum = eE * eE;
    double eS[6], sig[6];
    const double sw = w * db.cell_sw[cell] * pot.stress_weight;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      sig[q] = v[1 + q] / db.cell_vol[cell];
      eS[q] = sw * (sig[q] - db.cell_s0[6 * cell + q]);
      sum += eS[q] * eS[q];
    }
    sum += v[8];
    const double cons = v[7];
    sum += cons * cons;
    cellobj[(size_t)c * NC + cell] = sum;
    __threadfence();
    slast = atomicAdd(count + c, 1) == NC - 1;
    if (slast) {
      __threadfence();
      count[c] = 0;
    }
    if (errvec) {
      double *e = errvec + (size_t)c * esize + 7 * cell + 3 * a0;
      e[0] = eE;
      for (int q = 0; q < 6; ++q) e[1 + q] = eS[q];
      if (!pot.pair) errvec[(size_t)c * esize + 7 * NC + 3 * N + cell] = cons;
    }
    if (energy) energy[(size_t)c * NC + cell] = E;
    if (stress)
      for (int q = 0; q < 6; ++q) stress[((size_t)c * NC + cell) * 6 + q] = sig[q];
    if (seeds) {
      double *sd = seeds + (size_t)c * CS_COUNT * NC;
      sd[CS_EPS * NC + cell] = 2.0 * eE * ew;
      for (int q = 0; q < 6; ++q) sd[(CS_MU0 + q) * NC + cell] = 2.0 * eS[q] * sw / db.cell_vol[cell];
      sd[CS_KAPPA * NC + cell] = 2.0 * cons;
    }
  }
  __syncthreads();
  if (!slast) return;
  // ---- the last cell of the candidate: the objective
  double s = 0.0;
  for (int i = tid; i < NC; i += CELL_T) s += __ldcg(cellobj + (size_t)c * NC + i);
  tree[tid] = s;
  __syncthreads();
  for (int o = CELL_T / 2; o > 0; o >>= 1) {
    if (tid < o) tree[tid] += tree[tid + o];
    __syncthreads();
  }
  if (warp == 0) {
    double *ev = errvec ? errvec + (size_t)c * esize + 8 * NC + 3 * N : nullptr;
    const double pen = warp_punishments(pot, geom, tabs + (size_t)c * pot.tab_stride, ev, lane);
    if (lane == 0) obj[c] = tree[0] + pen;
  }
}

// ------------------------------------------------------------------ k_final

// Signed largest-|y| knot of one spline (Spline::get_max_y_mag, spline.cpp:58-67).
__device__ __forceinline__ double spline_max_y(const SplineGeom &g, const double *tab, int *which) {
  double sm = 0.0;
  int sat = -1;
  for (int k = 0; k < g.n; ++k) {
    const double y = tab[g.toff + k];
    if (fabs(sm) < fabs(y)) {
      sm = y;
      sat = g.toff + k;
    }
  }
  if (which) *which = sat;
  return sm;
}
// Signed largest-|y| knot over a Pair_ij group (PotFns::get_max_y_mag,
// pot_fns.cpp:100-111) whose first spline is s0: f, or JMEAM's p (p2).
__device__ __forceinline__ double group_max_y(const DevPot &pot, int s0, const SplineGeom *geom, const double *tab,
                                              int *which) {
  double my = 0.0;
  int at = -1;
  const int nf = pot.ntypes * (pot.ntypes + 1) / 2;
  for (int f = 0; f < nf; ++f) {
    int sat;
    const double sm = spline_max_y(geom[s0 + f], tab, &sat);
    if (fabs(my) < fabs(sm)) {
      my = sm;
      at = sat;
    }
  }
  if (which) *which = at;
  return my;
}

// The moment path's end (k_fm_cells has the cells' sums): sum of squares over
// cells + the style's punishment entries.
__global__ void k_final(DevDb db, DevPot pot, const SplineGeom *__restrict__ geom,
                        const double *__restrict__ tabs, const double *__restrict__ cellobj,
                        double *__restrict__ obj, double *__restrict__ errvec, int esize) {
  __shared__ double part[256];
  const int c = blockIdx.x;
  const int t = threadIdx.x;
  double s = 0.0;
  for (int i = t; i < db.ncells; i += blockDim.x) s += cellobj[(size_t)c * db.ncells + i];
  part[t] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (t < o) part[t] += part[t + o];
    __syncthreads();
  }
  if (t < 32) {
    double *ev = errvec ? errvec + (size_t)c * esize + 8 * db.ncells + 3 * db.natoms : nullptr;
    const double pen = warp_punishments(pot, geom, tabs + (size_t)c * pot.tab_stride, ev, t);
    if (t == 0) obj[c] = part[0] + pen;
  }
}

}  // namespace mzb
