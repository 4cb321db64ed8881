// FP64 adjoint over neighbour rows, a warp for a few atoms (the layout of
// mz_rows.cuh), for spline3eq eam, meam, gmeam and pair potentials; the
// formulas are k_adj's (mz_adj.cuh).
//
// k_adj<double> kept its sums in a fixed order by handing every slot's 12
// table contributions round its warp by shuffles, one slot after another:
// 8000 cycles per warp of slots, some 500 of them in the triplet loop.  Here
// - k_rows_adj only forms, per slot, the weights of its three radial functions
//   (a_p and the weight of f's value; with the atom's chi, U' and eps the rest
//   follows), and sums the angular functions' gradient in a table of each
//   lane's own (shared memory, power basis about the interval's middle);
// - k_rows_radial sums the radial gradients: which interval of which spline a
//   slot falls into does not depend on the candidate, so the slots of every
//   segment (256 to 2048) are sorted by it once (k_rows_sort), and a warp adds
//   up one bucket in registers;
// - both leave partials in an order fixed by the database, summed in order by
//   k_grad_sum: the gradient is bit-identical from call to call.
//
// In the triplet loop the table takes the ordered pair's term seen from the
// partner: sum over (j, k) of f_j (chi f_k / 2 + U' a_k f'_k) and, for the
// slope, f_j U' T_k with T_k = (f_k / r_k) (Lambda_k . u_j - a_k cos), which
// are the weights of dK/df_j that the loop forms anyway; with Lambda's part
// along u_k taken off, T_k = (f_k / r_k) (Lambda_k - a_k u_k) . u_j.
//
// Bounds: 28 FP64 instructions and 26 shared-memory wavefronts per partner
// and warp (8 of them pieces, 16 the table's read and write); 12 warps an SM
// (18 KB of rows and tables each), so also the latency of each group's loads.
// Measured (k_adj -> k_rows_adj + k_rows_radial, one candidate): MEAM, 21 k
// atoms of 16 slots 302 -> 64 + 17 us; two-species gmeam, 6 k atoms of 25
// slots 264 -> 84 + 15 us.
#pragma once

#include "mz_rows.cuh"
#include "mz_rows.hpp"

namespace mzb {

constexpr int RADJ_MAXW = 12;      // most warps per CTA (170 registers a thread on a full SM)
constexpr int RADIAL_T = 256;

struct RadjLayout {
  RowsLayout rows;   // the tables (one candidate); its rows are replaced by:
  int np;            // pieces of one angular spline's table (the largest n + 1)
  int ntab;          // angular tables per lane: 1, GMEAM npair
  int part;          // doubles of a warp's partial: 4 per angular piece, the U tables
  int warps;         // per CTA
  size_t o_w, row_bytes, tab_bytes, warp_bytes, bytes;
};

__host__ __device__ inline RadjLayout radj_layout(const DevPot &pot, int lpa, bool meam, int warps) {
  RadjLayout L;
  L.rows = rows_layout(pot, lpa, 4, meam, 1);
  L.np = pot.g_nmax + 1;
  L.ntab = pot.gmeam ? pot.npair : 1;
  L.part = 4 * L.rows.nang + L.rows.u_len;
  L.o_w = L.rows.o_rows;
  const int aw = 32 / lpa;
  L.row_bytes = meam ? (size_t)aw * L.rows.rs * (4 * sizeof(double2) + (pot.gmeam ? sizeof(int) : 0)) : 0;
  L.row_bytes = (L.row_bytes + 15) & ~size_t(15);
  L.tab_bytes = meam ? (size_t)L.ntab * L.np * 2 * 32 * sizeof(double2) : 0;
  L.warp_bytes = L.row_bytes + L.tab_bytes + ((sizeof(double) * (size_t)L.part + 15) & ~size_t(15));
  L.warps = warps;
  L.bytes = L.o_w + warps * L.warp_bytes;
  return L;
}

// A staged row as the loop reads it.
struct RadjRow {
  // (u_x, u_y), (u_z, W), (Q_x, Q_y), (Q_z, U' a f') with Q = U'/h f/r (Lambda - a u)
  const double2 *uxy, *uzw, *qxy, *qzx;
  const int *type;
};

// One pass over the row for a lane's NS slots: dk = U' dK/df's loop part, and
// the angular gradient of the slots as f_j times the partner's weights.
template <bool CL, int NS, int LPA, bool GM>
__device__ __forceinline__ void radj_pass(const RadjRow &R, int nk, int l, const double (&u)[4][3],
                                          const double (&f)[4], const double2 *alo, const double2 *ahi,
                                          const RowSpl *ang, const DevPot &pot, const int (&tj)[4], double2 *tab,
                                          int np, double (&dk)[4]) {
  RowSpl a0;
  if (!GM) a0 = ang[0];
#pragma unroll
  for (int s = 0; s < NS; ++s) dk[s] = 0.0;
  auto step = [&](const double (&x)[NS], const double (&y)[NS], const double (&z)[NS], const double (&W)[NS],
                  const double (&Qx)[NS], const double (&Qy)[NS], const double (&Qz)[NS], const double (&qx)[NS],
                  const bool (&out)[NS], const int (&tk)[NS]) {
    double b[NS], c[NS], T[NS], q[NS], t[NS], m[NS], w[NS], p[NS];
    double2 lo[NS], hi[NS];
    RowSpl g[NS];
    int k[NS], at[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s)
      c[s] = CL ? cos_exact(u[s][0], u[s][1], u[s][2], x[s], y[s], z[s])
                : fma(u[s][0], x[s], fma(u[s][1], y[s], u[s][2] * z[s]));
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      g[s] = a0;
      at[s] = 0;
      if (GM) {
        const int pj = pair_ij_index(tj[s], tk[s], pot.ntypes);
        g[s] = ang[pj];
        at[s] = pj * np;
      }
      k[s] = rows_knot<CL>(c[s], g[s], b[s]);
      at[s] = (at[s] + k[s] + 1) * 64;
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      lo[s] = alo[g[s].p0 + k[s]];
      hi[s] = ahi[g[s].p0 + k[s]];
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) T[s] = fma(Qx[s], u[s][0], fma(Qy[s], u[s][1], Qz[s] * u[s][2]));
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const bool no = out[s] || (CL && !(c[s] < g[s].cut));
      if (GM) T[s] *= g[s].inv;
      if (no) T[s] = 0.0;
      w[s] = f[s] * (no ? 0.0 : W[s]);
      p[s] = no ? 0.0 : qx[s];
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) q[s] = b[s] * hi[s].y;
#pragma unroll
    for (int s = 0; s < NS; ++s) t[s] = hi[s].x + q[s];
#pragma unroll
    for (int s = 0; s < NS; ++s) m[s] = fma(b[s], t[s], lo[s].y);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      dk[s] = fma(fma(b[s], m[s], lo[s].x), p[s], dk[s]);
      dk[s] = fma(fma(b[s], t[s] + q[s], m[s]), T[s], dk[s]);
    }
    // value weight w, slope weight v = f T: w b^j + j v b^(j-1), j = 0..3
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      q[s] = f[s] * T[s];
      t[s] = fma(w[s], b[s], q[s]);
      m[s] = t[s] + q[s];
      q[s] = m[s] + q[s];
      p[s] = b[s] * b[s];
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      double2 A = tab[at[s]], B = tab[at[s] + 32];
      A.x += w[s];
      A.y += t[s];
      B.x = fma(b[s], m[s], B.x);
      B.y = fma(p[s], q[s], B.y);
      tab[at[s]] = A;
      tab[at[s] + 32] = B;
    }
  };
  double x[NS], y[NS], z[NS], W[NS], Qx[NS], Qy[NS], Qz[NS], qx[NS];
  bool out[NS];
  int tk[NS];
#pragma unroll
  for (int s0 = 0; s0 < NS; ++s0) {  // runs of LPA partners: the slot itself is none (see rows_pass)
    const int len = min(nk - s0 * LPA, LPA);
#pragma unroll 1
    for (int i = 0; i < len; ++i) {
      const int k = s0 * LPA + i;
      const double2 a = R.uxy[k], c = R.uzw[k], d = R.qxy[k], e = R.qzx[k];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        x[s] = a.x;
        y[s] = a.y;
        z[s] = c.x;
        W[s] = c.y;
        Qx[s] = d.x;
        Qy[s] = d.y;
        Qz[s] = e.x;
        qx[s] = e.y;
        out[s] = s == s0 && i == l;
        tk[s] = GM ? R.type[k] : 0;
      }
      step(x, y, z, W, Qx, Qy, Qz, qx, out, tk);
    }
  }
}

// Groups of up to 32 / LPA atoms of one type, a contiguous run per warp;
// desc [ngroups][32 / LPA] (atom or -1, first slot, slots | type << 16, cell).
// aout: reads rho, leaves chi, U' and eps of the atom in its force rows;
// W1 [ncand][3][Np]: a_p and f's value weight; part [ncand][gridDim.x][L.part].
template <bool MEAM, bool GM, int LPA>
__global__ void __launch_bounds__(32 * RADJ_MAXW, 1)
    k_rows_adj(DevDb db, DevPot pot, RadjLayout L, const int4 *__restrict__ desc, int ngroups,
               const SplineGeom *__restrict__ geom, const double *__restrict__ tabs, const double *__restrict__ ptabs,
               double *aout, const double *__restrict__ aux, const double *__restrict__ lam,
               const double *__restrict__ seeds, double *__restrict__ W1, double *__restrict__ part) {
  extern __shared__ __align__(16) unsigned char rsm[];
  constexpr int AW = 32 / LPA, SPL = 4;
  const int cand = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l = lane % LPA, sub = lane / LPA;
  const int N = db.natoms, NC = db.ncells;
  const int64_t Np = db.npairs;
  rows_stage(rsm, L.rows, pot, geom, tabs, ptabs, cand, cand + 1);
  const SplineGeom *sg = reinterpret_cast<const SplineGeom *>(rsm + L.rows.o_geo);
  const RowSpl *spl = reinterpret_cast<const RowSpl *>(rsm + L.rows.o_spl);
  const double2 *plo = reinterpret_cast<const double2 *>(rsm), *phi = plo + L.rows.npiece, *alo = phi + L.rows.npiece,
                *ahi = alo + L.rows.nang;
  const double *tU = reinterpret_cast<const double *>(rsm + L.rows.o_u) - L.rows.u_off;
  unsigned char *wm = rsm + L.o_w + warp * L.warp_bytes;
  const int rs = L.rows.rs;
  double2 *ruxy = reinterpret_cast<double2 *>(wm) + sub * rs, *ruzw = ruxy + AW * rs, *rqxy = ruzw + AW * rs,
          *rqzx = rqxy + AW * rs;
  int *rt = reinterpret_cast<int *>(wm + 4 * sizeof(double2) * AW * rs) + sub * rs;
  double2 *tab = reinterpret_cast<double2 *>(wm + L.row_bytes) + lane;
  double *out = reinterpret_cast<double *>(wm + L.row_bytes + L.tab_bytes);  // [part] sums of the warp
  double *ut = out + 4 * L.rows.nang;                                        // its U-table gradients
  const RadjRow row{ruxy, ruzw, rqxy, rqzx, rt};

  const int nwarps = gridDim.x * L.warps, wid = blockIdx.x * L.warps + warp;
  for (int i = lane; i < L.part; i += 32) out[i] = 0.0;
  if (MEAM)
    for (int i = 0; i < L.ntab * L.np * 2; ++i) tab[32 * i] = make_double2(0.0, 0.0);
  __syncwarp();
  // the lanes' angular tables of centre type t into the warp's partial
  auto flush = [&](int t) {
    for (int v = 0; v < L.ntab; ++v) {
      const int s = pot.s_g + t * L.ntab + v;
      for (int k = -1; k < sg[s].n; ++k) {
        const int at = (v * L.np + k + 1) * 64;
        const double2 A = tab[at], B = tab[at + 32];
        tab[at] = tab[at + 32] = make_double2(0.0, 0.0);
        // two halving exchanges (lane bit 0 takes q >= 2, bit 1 the odd q), then the rest of the lanes
        const bool h0 = lane & 1, h1 = lane & 2;
        const double x = (h0 ? B.x : A.x) + __shfl_xor_sync(0xffffffffu, h0 ? A.x : B.x, 1);
        const double y = (h0 ? B.y : A.y) + __shfl_xor_sync(0xffffffffu, h0 ? A.y : B.y, 1);
        double d = (h1 ? y : x) + __shfl_xor_sync(0xffffffffu, h1 ? x : y, 2);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane < 4) out[4 * (spl[s].p0 + k) + (lane & 1) * 2 + (lane >> 1)] = d;
      }
    }
  };
  const double2 *uxy = db.pair2, *uzr = uxy + Np, *irf = uzr + Np;
  double *ao = aout + (size_t)cand * AO_COUNT * N;
  const double *ax = aux + (size_t)cand * AUX_COUNT * Np;
  const double *Lm = lam + (size_t)cand * 3 * N;
  const double *sd = seeds + (size_t)cand * CS_COUNT * NC;
  double *wa = W1 + (size_t)cand * 3 * Np, *wf = wa + Np;

  int tcur = -1;
  const int g0 = (int)((int64_t)ngroups * wid / nwarps), g1 = (int)((int64_t)ngroups * (wid + 1) / nwarps);
  int4 next = g0 < g1 ? desc[(int64_t)g0 * AW + sub] : make_int4(-1, 0, 0, 0);
  for (int grp = g0; grp < g1; ++grp) {
    const int4 dsc = next;
    if (grp + 1 < g1) next = desc[(int64_t)(grp + 1) * AW + sub];
    const bool live = dsc.x >= 0;
    const int i = max(dsc.x, 0), lo = dsc.y, n = dsc.z & 0xffff, ti = dsc.z >> 16;  // one type per group
    if (MEAM && tcur >= 0 && ti != tcur) flush(tcur);
    tcur = ti;
    const int nw = __reduce_max_sync(0xffffffffu, n);
    const int cell = dsc.w;
    const double lix = Lm[i], liy = Lm[N + i], liz = Lm[2 * N + i];
    const double mxx = sd[(CS_MU0 + 0) * NC + cell], myy = sd[(CS_MU0 + 1) * NC + cell],
                 mzz = sd[(CS_MU0 + 2) * NC + cell], mxy = sd[(CS_MU0 + 3) * NC + cell],
                 myz = sd[(CS_MU0 + 4) * NC + cell], mzx = sd[(CS_MU0 + 5) * NC + cell];
    const double eps = sd[CS_EPS * NC + cell], kap = sd[CS_KAPPA * NC + cell];
    // ---- U', U'' at the atom's density (every lane)
    double dF = 0.0, d2F = 0.0, rt_ = 0.0, dpen = 0.0, drt = 1.0;
    PointEval U{};
    if (!pot.pair) {
      const double rho = ao[AO_RHO * N + i], w = db.cell_w[cell];
      const SplineGeom &gU = sg[pot.s_U + ti];
      const double x0 = gU.x0, xN = gU.xN;
      rt_ = rho;
      if (rho < x0) {
        dpen = -w * 100.0 * 10. * 2.0 * (x0 - rho);
        if (!pot.embed_extrap) { rt_ = x0; drt = 0.0; }
      } else if (rho > xN) {
        dpen = w * 100.0 * 10. * 2.0 * (rho - xN);
        if (!pot.embed_extrap) { rt_ = xN; drt = 0.0; }
      }
      U = spl_point(tU, gU, rt_);
      dF = U.grad;
      d2F = U.grad2;
    }
    // ---- per slot: Lambda, a_p and its share k_p of K
    const double ginv = MEAM && !GM ? spl[pot.s_g + ti].inv : 1.0, sc = dF * ginv;
    double u[SPL][3], f[SPL], base[SPL], G[SPL], K = 0.0;
    int tj[SPL] = {};
#pragma unroll
    for (int s = 0; s < SPL; ++s) {
      if (s * LPA >= nw) break;
      const int p = l + s * LPA, gs = lo + p;
      u[s][0] = u[s][1] = u[s][2] = f[s] = base[s] = G[s] = 0.0;
      double q[3] = {0.0, 0.0, 0.0}, qx = 0.0;
      if (p < n) {
        const double2 xy = uxy[gs], zr = uzr[gs], rf = irf[gs];
        const int2 m = db.pair_meta[gs];
        const int j = db.pair_nbr[gs];
        const double r = zr.y;
        u[s][0] = xy.x;
        u[s][1] = xy.y;
        u[s][2] = zr.x;
        tj[s] = m.y;
        const double Lx = lix - Lm[j] - r * (mxx * xy.x + mzx * zr.x);
        const double Ly = liy - Lm[N + j] - r * (myy * xy.y + mxy * xy.x);
        const double Lz = liz - Lm[2 * N + j] - r * (mzz * zr.x + myz * xy.y);
        const double ap = Lx * xy.x + Ly * xy.y + Lz * zr.x;
        wa[gs] = ap;
        const int krho = ((m.x >> 8) & 0xff) - 1;
        double d;
        if (krho >= 0) {
          const RowSpl &g = spl[pot.s_rho + m.y];
          rows_piece(plo, phi, g.p0 + krho, db.pair_shift[Np + gs], d);
          K += ap * d * g.inv;
        }
        if (MEAM) {
          const int kf = ((m.x >> 16) & 0xff) - 1;
          const double Gp = ax[AUX_G * Np + gs], H = ax[AUX_H * Np + gs];
          const double J = Lx * ax[AUX_VX * Np + gs] + Ly * ax[AUX_VY * Np + gs] + Lz * ax[AUX_VZ * Np + gs];
          double df = 0.0;
          if (kf >= 0) {
            const RowSpl &g = spl[pot.s_f + pair_ij_index(ti, m.y, pot.ntypes)];
            f[s] = rows_piece(plo, phi, g.p0 + kf, rf.y, d);
            df = d * g.inv;
          }
          const double JH = rf.x * (J - ap * H);
          K += ap * df * Gp + f[s] * JH;
          G[s] = Gp;
          base[s] = dF * JH;
          qx = dF * ap * df;
          const double fi = sc * f[s] * rf.x;
          q[0] = fi * (Lx - ap * xy.x);
          q[1] = fi * (Ly - ap * xy.y);
          q[2] = fi * (Lz - ap * zr.x);
        }
      }
      if (MEAM) {
        ruxy[p] = make_double2(u[s][0], u[s][1]);
        ruzw[p] = make_double2(u[s][2], qx);  // W once chi is known
        rqxy[p] = make_double2(q[0], q[1]);
        rqzx[p] = make_double2(q[2], qx);
        if (GM) rt[p] = tj[s];
      }
    }
#pragma unroll
    for (int o = 1; o < LPA; o <<= 1) K += __shfl_xor_sync(0xffffffffu, K, o);
    const double chi = (eps * dF + d2F * K) * drt + kap * dpen;
    if (live && l == 0) {
      ao[AO_AX * N + i] = chi;
      ao[AO_AY * N + i] = dF;
      ao[AO_AZ * N + i] = eps;
    }
    // the U table's gradient, the atoms of the warp one after another
    if (!pot.pair)
      for (int a = 0; a < AW; ++a) {
        if (lane == a * LPA && live) {
          const SplineGeom &gU = sg[pot.s_U + ti];
          double *at = ut + gU.toff - L.rows.u_off;
          spl_point_adjoint(gU, U, rt_, eps, K, [&](int ix, double x) { at[ix] += x; });
        }
        __syncwarp();
      }
    if (MEAM) {
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        if (s * LPA >= nw) break;
        ruzw[l + s * LPA].y += 0.5 * chi * f[s];
      }
      __syncwarp();
      double dk[SPL] = {};
      const RowSpl *a = spl + pot.s_g + ti * L.ntab;
      auto go = [&](auto cl) {
        constexpr bool CL = decltype(cl)::value;
        if (nw > 3 * LPA) radj_pass<CL, 4, LPA, GM>(row, nw, l, u, f, alo, ahi, a, pot, tj, tab, L.np, dk);
        else if (nw > 2 * LPA) radj_pass<CL, 3, LPA, GM>(row, nw, l, u, f, alo, ahi, a, pot, tj, tab, L.np, dk);
        else if (nw > LPA) radj_pass<CL, 2, LPA, GM>(row, nw, l, u, f, alo, ahi, a, pot, tj, tab, L.np, dk);
        else radj_pass<CL, 1, LPA, GM>(row, nw, l, u, f, alo, ahi, a, pot, tj, tab, L.np, dk);
      };
      if (nw == 0) {  // no row is staged: the shared rows hold anything
      } else if (pot.ang_cover) {
        go(std::integral_constant<bool, false>{});
      } else {
        go(std::integral_constant<bool, true>{});
      }
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        const int p = l + s * LPA;
        if (p < n) wf[lo + p] = chi * G[s] + dk[s] + base[s];
      }
      __syncwarp();  // the next group reuses the rows
    }
  }
  if (MEAM && tcur >= 0) flush(tcur);
  __syncthreads();
  // the CTA's warps in order
  for (int e = threadIdx.x; e < L.part; e += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < L.warps; ++w)
      s += reinterpret_cast<const double *>(rsm + L.o_w + w * L.warp_bytes + L.row_bytes + L.tab_bytes)[e];
    part[((size_t)cand * gridDim.x + blockIdx.x) * L.part + e] = s;
  }
}

// ------------------------------------------------------------ radial sums

__device__ __forceinline__ int radial_bucket(const DevPot &pot, const RadialPlan &R, int F, int kn, int ti, int tj) {
  const int k = ((kn >> (8 * F)) & 0xff) - 1;
  if (k < 0) return -1;
  const int s = F == 1 ? tj : pair_ij_index(ti, tj, pot.ntypes);
  return s * R.nint[F] + k;
}

// One CTA per segment: its slots by bucket, in slot order within a bucket.
__global__ void __launch_bounds__(RADIAL_T) k_rows_sort(DevDb db, DevPot pot, RadialPlan R) {
  __shared__ short bk[RADIAL_SEG];
  __shared__ unsigned short cnt[RADIAL_MAXB];
  const int64_t s0 = (int64_t)blockIdx.x * R.seg, Np = db.npairs;
  const int len = (int)min((int64_t)R.seg, Np - s0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the owner of each slot: the last atom whose row starts at or before it
  for (int s = tid; s < len; s += RADIAL_T) {
    int lo = 0, hi = db.natoms;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (db.pair_off[mid] <= s0 + s) lo = mid;
      else hi = mid;
    }
    R.slot_atom[s0 + s] = lo;
  }
  int items = 0;  // thread 0's
  for (int F = 0; F < R.nfun; ++F) {
    const int nb = R.b0[F + 1] - R.b0[F];
    for (int s = tid; s < len; s += RADIAL_T) {
      const int2 m = db.pair_meta[s0 + s];
      bk[s] = (short)radial_bucket(pot, R, F, m.x, db.atom_type[R.slot_atom[s0 + s]], m.y);
    }
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
      for (int b = warp; b < nb; b += RADIAL_T / 32) {
        int at = pass ? cnt[b] : 0;
        for (int c = 0; c < len; c += 32) {
          const bool hit = c + lane < len && bk[c + lane] == b;
          const unsigned mask = __ballot_sync(0xffffffffu, hit);
          if (pass && hit) R.order[F * Np + s0 + at + __popc(mask & ((1u << lane) - 1))] = (unsigned short)(c + lane);
          at += __popc(mask);
        }
        if (!pass && lane == 0) cnt[b] = (unsigned short)at;
      }
      __syncthreads();
      if (!pass && tid == 0) {  // starts
        int a = 0;
        for (int b = 0; b < nb; ++b) {
          const int c = cnt[b];
          cnt[b] = (unsigned short)a;
          R.off[(size_t)blockIdx.x * (R.nb + R.nfun) + R.b0[F] + F + b] = (unsigned short)a;
          R.item[(size_t)blockIdx.x * (R.nb + 1) + R.b0[F] + b] = (unsigned short)items;
          a += c;
          items += (c + RADIAL_ITEM - 1) / RADIAL_ITEM;
        }
        if (F == R.nfun - 1) R.item[(size_t)blockIdx.x * (R.nb + 1) + R.nb] = (unsigned short)items;
        R.off[(size_t)blockIdx.x * (R.nb + R.nfun) + R.b0[F] + F + nb] = (unsigned short)a;
      }
      __syncthreads();
    }
  }
}

// The radial functions' gradient sums in the power basis of the shift.
// Buckets are uneven (the shells of a crystal fill two or three intervals),
// so the unit of work is an item, RADIAL_ITEM slots of one bucket at most:
// eight lanes sum it, and its bucket's items are added in order.  The CTA's
// segments in order; part [ncand][gridDim.x][4 nb].  Bound by the latency of
// its gathers (order -> atom -> chi).
__host__ __device__ inline size_t radial_smem(const RadialPlan &R) {
  return sizeof(double) * (9 * (size_t)R.nb + 4 * (size_t)R.nfun * R.seg / RADIAL_ITEM) +
         ((sizeof(unsigned short) * (2 * (size_t)R.nb + R.nfun + 1) + 15) & ~size_t(15));
}

__global__ void __launch_bounds__(RADIAL_T)
    k_rows_radial(DevDb db, DevPot pot, RadialPlan R, const SplineGeom *__restrict__ geom,
                  const double *__restrict__ aout, const double *__restrict__ aux, const double *__restrict__ W1,
                  double *__restrict__ part) {
  extern __shared__ double acc[];  // [nb][4] buckets; [nb] 1 / h; items [][4]; their and the slots' starts
  const int cand = blockIdx.y, tid = threadIdx.x, l = tid & 7, N = db.natoms, nb = R.nb;
  const int64_t Np = db.npairs;
  const double *ao = aout + (size_t)cand * AO_COUNT * N;
  const double *chi = ao + AO_AX * N, *dF = ao + AO_AY * N, *eps = ao + AO_AZ * N;
  const double *wa = W1 + (size_t)cand * 3 * Np, *wf = wa + Np;
  const double *G = aux + ((size_t)cand * AUX_COUNT + AUX_G) * Np;
  double *binv = acc + 4 * nb, *isum = binv + nb;
  unsigned short *it0 = reinterpret_cast<unsigned short *>(isum + 4 * (nb + R.nfun * R.seg / RADIAL_ITEM)),
                 *off = it0 + nb + 1;
  const int f1 = R.b0[1], f2 = R.nfun > 1 ? R.b0[2] : nb;  // first buckets of rho and f
  for (int b = tid; b < nb; b += RADIAL_T) {
    const int F = b < f1 ? 0 : b < f2 ? 1 : 2;
    const int s0 = F == 0 ? pot.s_phi : F == 1 ? pot.s_rho : pot.s_f;
    const int b0 = F == 0 ? 0 : F == 1 ? f1 : f2, ni = F == 0 ? R.nint[0] : F == 1 ? R.nint[1] : R.nint[2];
    binv[b] = geom[s0 + (b - b0) / ni].invstep;
    for (int q = 0; q < 4; ++q) acc[4 * b + q] = 0.0;
  }
  const int per = (R.nseg + gridDim.x - 1) / gridDim.x, seg1 = min(R.nseg, (int)(blockIdx.x + 1) * per);
  for (int seg = blockIdx.x * per; seg < seg1; ++seg) {
    const int64_t s0 = (int64_t)seg * R.seg;
    for (int b = tid; b <= nb; b += RADIAL_T) it0[b] = R.item[(size_t)seg * (nb + 1) + b];
    for (int b = tid; b < nb + R.nfun; b += RADIAL_T) off[b] = R.off[(size_t)seg * (nb + R.nfun) + b];
    __syncthreads();
    const int items = it0[nb];
    for (int ii = 0; ii < items; ii += RADIAL_T / 8) {
      const int it = ii + tid / 8;
      double d[4] = {0.0, 0.0, 0.0, 0.0};
      if (it < items) {
        int b = 0, hb = nb;  // the bucket of the item: the last that starts at or before it
        while (hb - b > 1) {
          const int mid = (b + hb) >> 1;
          if (it0[mid] <= it) b = mid;
          else hb = mid;
        }
        const int F = b < f1 ? 0 : b < f2 ? 1 : 2;
        const int lo = off[b + F] + (it - it0[b]) * RADIAL_ITEM, hi = min((int)off[b + F + 1], lo + RADIAL_ITEM);
        const double inv = binv[b];
#pragma unroll
        for (int q = 0; q < RADIAL_ITEM / 8; ++q) {
          const int e = lo + l + 8 * q;
          if (e >= hi) continue;
          const int64_t gs = s0 + R.order[F * Np + s0 + e];
          const int i = R.slot_atom[gs];
          const double x = db.pair_shift[F * Np + gs], ap = wa[gs];
          double cv, cd;
          if (F == 0) {
            const double sh = phi_share(pot, pot.pair && db.pair_nbr[gs] == i);
            cv = sh * eps[i];
            cd = sh * ap;
          } else if (F == 1) {
            cv = chi[i];
            cd = dF[i] * ap;
          } else {
            cv = wf[gs];
            cd = dF[i] * ap * G[gs];
          }
          cd *= inv;
          const double c1 = fma(cv, x, cd);
          d[0] += cv;
          d[1] += c1;
          d[2] = fma(x, c1 + cd, d[2]);
          d[3] = fma(x * x, c1 + (cd + cd), d[3]);
        }
      }
      const bool h0 = l & 1, h1 = l & 2;
      const double x = (h0 ? d[2] : d[0]) + __shfl_xor_sync(0xffffffffu, h0 ? d[0] : d[2], 1);
      const double y = (h0 ? d[3] : d[1]) + __shfl_xor_sync(0xffffffffu, h0 ? d[1] : d[3], 1);
      double t = (h1 ? y : x) + __shfl_xor_sync(0xffffffffu, h1 ? x : y, 2);
      t += __shfl_xor_sync(0xffffffffu, t, 4);
      if (it < items && l < 4) isum[4 * it + (l & 1) * 2 + (l >> 1)] = t;
    }
    __syncthreads();
    for (int e = tid; e < 4 * nb; e += RADIAL_T)
      for (int it = it0[e / 4]; it < it0[e / 4 + 1]; ++it) acc[e] += isum[4 * it + (e & 3)];
    __syncthreads();
  }
  __syncthreads();  // a CTA without a segment has only zeroed its sums
  double *out = part + ((size_t)cand * gridDim.x + blockIdx.x) * 4 * nb;
  for (int i = tid; i < 4 * nb; i += RADIAL_T) out[i] = acc[i];
}

}  // namespace mzb
