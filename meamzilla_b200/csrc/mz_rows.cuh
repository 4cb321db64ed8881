// FP64 row kernels: the forward pass over neighbour rows for spline3eq
// potentials, a warp on its own (no block barriers after the tables are
// staged).
//
// LPA lanes take one atom, each holding up to 4 slots of its row (slot p on
// lane p % LPA) in registers, so a warp works on 32 / LPA atoms at once and a
// partner read from shared memory serves all slots of a lane.  LPA follows
// the database's longest row (rows_lpa): the fewest lanes whose 4 slots hold
// it, so that few lanes idle in short rows.
//
// What bounds it, and why this form: k_atoms (a CTA of 256 slots, an atom per
// warp in its per-atom steps) spends some 900 cycles per warp of slots outside
// the triplet loop -- barriers, a table staged per 256 slots, ten doubles per
// slot written to shared memory and summed with 100 shuffles per atom -- and
// its loads of double4 pieces at a 32-byte stride collide in pairs: shared
// memory 83 % busy, FP64 pipe 49 %.  Here the tables are staged once per CTA
// for many atoms and up to four candidates, pieces lie as two 16-byte halves
// (no collisions), the slots' sums stay in registers until one halving
// exchange over the LPA lanes, H = u . vk follows from vk instead of being
// summed, and a lane's slots advance side by side (the FP64 pipe takes 1.8
// instructions a clock from warps with four independent chains, 1.25 from
// any number of warps with one).  Measured (k_atoms -> k_rows): 84 k atoms of
// 41 slots, 1 candidate 581 -> 378 us (L1 and shared memory 70 %, FP64 52 %); 21 k
// atoms of 16 slots, 56 candidates 2397 -> 1145 us; EAM, 18 k atoms of 42
// slots, 128 candidates 4811 -> 1200 us.
#pragma once

#include <type_traits>

#include "mz_spline.cuh"

namespace mzb {

constexpr int ROWS_W = 4;       // warps per CTA
constexpr int ROWS_MAXROW = 128;  // longest row (LPA = 32, SPL = 4)

// A spline as the row kernels read it.  Radial: p0 is its first piece in the
// table of the shift b, piece k: c0 + b (c1 + b (c2 + b c3)).  Angular: p0 is
// the piece of interval 0 in a second table whose polynomials are in b - 1/2
// and which has one piece more on either side (the end polynomials
// continued), so that no interval needs clamping while the knots reach to
// within 0.9 of an interval of [-1, 1] (DevPot::ang_cover).
struct RowSpl {
  double inv, c0, cut;  // 1 / h, -x0 / h - 1/2, upper cut
  int p0, nmax;         // first piece, last interval
};

struct RowsLayout {
  int npiece, nang, ang0;  // pieces of a candidate's evaluation table; of the angular table; its first source piece
  int u_off, u_len;        // the U splines' part of the knot table
  int ncb;                 // candidates per CTA
  int rs;                  // slots of a staged row (RL + 2: the rows of a warp start on other banks)
  size_t o_u, o_geo, o_spl, o_rows, tab_bytes, row_bytes, bytes;
};

// per candidate: both piece tables as halves (c0, c1) and (c2, c3), the U
// splines' knot table; then the geometry; then the warps' rows: (u_x, u_y),
// (u_z, f) and per JMEAM term p; the neighbour types (GMEAM)
__host__ __device__ inline RowsLayout rows_layout(const DevPot &pot, int lpa, int spl, bool rows, int ncb) {
  RowsLayout L;
  L.npiece = pot.pow_stride / 4;
  L.ang0 = rows ? pot.ang_p0 : L.npiece;
  L.nang = rows ? L.npiece - L.ang0 + 2 * (pot.nsplines - pot.s_g) : 0;
  L.u_off = pot.u_off;
  L.u_len = pot.u_len;
  L.ncb = ncb;
  L.rs = lpa * spl + 2;
  const int aw = 32 / lpa;
  size_t b = 2 * sizeof(double2) * (size_t)(L.npiece + L.nang);
  L.o_u = b;
  b += sizeof(double) * (size_t)L.u_len;
  L.tab_bytes = b = (b + 15) & ~size_t(15);
  b *= ncb;
  L.o_geo = b;
  b += sizeof(SplineGeom) * (size_t)pot.nsplines;
  b = (b + 15) & ~size_t(15);
  L.o_spl = b;
  b += sizeof(RowSpl) * (size_t)pot.nsplines;
  b = (b + 15) & ~size_t(15);
  L.o_rows = b;
  L.row_bytes = rows ? (size_t)aw * L.rs * (2 * sizeof(double2) + sizeof(double) * pot.nj + (pot.gmeam ? sizeof(int) : 0))
                     : 0;
  L.row_bytes = (L.row_bytes + 15) & ~size_t(15);
  L.bytes = b + ROWS_W * L.row_bytes;
  return L;
}

// The tables of candidates cand0 .. cand0 + ncb - 1 and the splines' geometry
// into shared memory (every thread of the CTA; a barrier at the end).
__device__ __forceinline__ void rows_stage(unsigned char *sm, const RowsLayout &L, const DevPot &pot,
                                           const SplineGeom *__restrict__ geom, const double *__restrict__ tabs,
                                           const double *__restrict__ ptabs, int cand0, int ncand) {
  const int tid = threadIdx.x, T = blockDim.x;
  SplineGeom *sg = reinterpret_cast<SplineGeom *>(sm + L.o_geo);
  RowSpl *spl = reinterpret_cast<RowSpl *>(sm + L.o_spl);
  for (int i = tid; i < pot.nsplines; i += T) {
    const SplineGeom g = geom[i];
    sg[i] = g;
    const bool a = L.nang > 0 && i >= pot.s_g;
    spl[i] = RowSpl{g.invstep, -g.x0 * g.invstep - 0.5, g.cut,
                    a ? g.poff / 4 - L.ang0 + 2 * (i - pot.s_g) + 1 : g.poff / 4, g.n - 2};
  }
  __syncthreads();
  for (int cc = 0; cc < L.ncb && cand0 + cc < ncand; ++cc) {
    unsigned char *t = sm + cc * L.tab_bytes;
    double2 *lo = reinterpret_cast<double2 *>(t), *hi = lo + L.npiece, *alo = hi + L.npiece, *ahi = alo + L.nang;
    double *sU = reinterpret_cast<double *>(t + L.o_u);
    const double2 *pc = reinterpret_cast<const double2 *>(ptabs + (size_t)(cand0 + cc) * pot.pow_stride);
    for (int i = tid; i < L.npiece; i += T) {
      lo[i] = pc[2 * i];
      hi[i] = pc[2 * i + 1];
    }
    for (int i = tid; i < L.u_len; i += T) sU[i] = tabs[(size_t)(cand0 + cc) * pot.tab_stride + L.u_off + i];
    if (L.nang > 0)
      for (int s = pot.s_g + tid / 32; s < pot.nsplines; s += T / 32)
        for (int k = tid % 32 - 1; k < sg[s].n; k += 32) {
          // interval k's polynomial around its middle; -1 and n - 1 continue the end pieces
          const int kk = min(max(k, 0), sg[s].n - 2);
          const double2 a = pc[2 * (sg[s].poff / 4 + kk)], c = pc[2 * (sg[s].poff / 4 + kk) + 1];
          const double x = 0.5 + (double)(k - kk);
          alo[spl[s].p0 + k] = make_double2(a.x + x * (a.y + x * (c.x + x * c.y)), a.y + x * (2.0 * c.x + 3.0 * x * c.y));
          ahi[spl[s].p0 + k] = make_double2(c.x + 3.0 * x * c.y, c.y);
        }
  }
  __syncthreads();
}

// value and slope times h of piece `at`
__device__ __forceinline__ double rows_piece(const double2 *lo, const double2 *hi, int at, double b, double &der) {
  const double2 a = lo[at], c = hi[at];
  const double q = b * c.y, t = c.x + q, m = fma(b, t, a.y);
  der = fma(b, t + q, m);
  return fma(b, m, a.x);
}

// The interval of a cosine c and its distance from the interval's middle:
// (c - x0) / h - 1/2 rounded to an integer by adding 1.5 2^52 (a tie, c on a
// knot, may give the interval below, which evaluates to the same value and
// slope to rounding).
template <bool CL>
__device__ __forceinline__ int rows_knot(double c, const RowSpl &g, double &b) {
  constexpr double MAGIC = 6755399441055744.0;
  const double h = fma(c, g.inv, g.c0), m = h + MAGIC;
  int k = __double2loint(m);
  if (CL) {
    k = k < 0 ? 0 : (k > g.nmax ? g.nmax : k);
    b = h - (__hiloint2double(0x43380000, k) - MAGIC);
  } else {
    b = h - (m - MAGIC);
  }
  return k;
}

// The sums over the row's other slots for a lane's NS slots, with partner
// weights weight(k, f_k): S = sum s(cos) w, v = h sum s'(cos) w u_k (GMEAM,
// whose spline depends on the partner: h not taken out).
// The slot itself is no partner: its weight is zero, so that nothing of the
// spline at cos = 1, which no pair of neighbours may reach, enters the sums.
// RUNS: the row is walked in runs of LPA partners; in run s0 only a lane's slot
// s0 can meet itself, so one comparison and select per partner does it (MEAM,
// 21 k atoms of 16 slots, 56 candidates: 1381 us a call).  Without, every slot
// compares, in one loop: for JMEAM, whose passes would otherwise be four loops
// each (10 k atoms, 16 candidates: 573 us a call, in runs 603).
// CL: knots that do not cover the cosines -- the interval is clamped, and a
// partner beyond the upper cut is no triplet.
template <bool CL, int NS, int SPL, int LPA, bool GM, bool RUNS, class W>
__device__ __forceinline__ void rows_pass(const double2 *rxy, const double2 *rzf, const int *rt, W weight, int nk,
                                          int l, const double (&u)[SPL][3], const double2 *alo, const double2 *ahi,
                                          const RowSpl *ang, const DevPot &pot, const int (&tj)[SPL],
                                          double (&S)[SPL], double (&v)[SPL][3]) {
  RowSpl a0;
  if (!GM) a0 = ang[0];
#pragma unroll
  for (int s = 0; s < NS; ++s) S[s] = v[s][0] = v[s][1] = v[s][2] = 0.0;
  // One step for the NS slots side by side: the FP64 pipe takes 1.8
  // instructions a clock from warps with four independent chains each, but 1.25
  // from any number of warps with one.
  auto step = [&](const double (&x)[NS], const double (&y)[NS], const double (&z)[NS], const double (&wk)[NS],
                  const int (&tk)[NS]) {
    double b[NS], t[NS], m[NS], q[NS], w[NS];
    double2 lo[NS], hi[NS];
    RowSpl g[NS];
    int k[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s)  // whether beyond the cut decides whether a triplet exists: then as the reference rounds it
      t[s] = CL ? cos_exact(u[s][0], u[s][1], u[s][2], x[s], y[s], z[s])
                : fma(u[s][0], x[s], fma(u[s][1], y[s], u[s][2] * z[s]));
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      g[s] = a0;
      if (GM) g[s] = ang[pair_ij_index(tj[s], tk[s], pot.ntypes)];
      w[s] = CL && !(t[s] < g[s].cut) ? 0.0 : wk[s];  // triplet_meam_spline.cpp:66-70
      k[s] = g[s].p0 + rows_knot<CL>(t[s], g[s], b[s]);
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      lo[s] = alo[k[s]];
      hi[s] = ahi[k[s]];
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) q[s] = b[s] * hi[s].y;
#pragma unroll
    for (int s = 0; s < NS; ++s) t[s] = hi[s].x + q[s];
#pragma unroll
    for (int s = 0; s < NS; ++s) m[s] = fma(b[s], t[s], lo[s].y);
#pragma unroll
    for (int s = 0; s < NS; ++s) t[s] = fma(b[s], t[s] + q[s], m[s]) * w[s];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      S[s] = fma(fma(b[s], m[s], lo[s].x), w[s], S[s]);
      if (GM) t[s] *= g[s].inv;
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      v[s][0] = fma(t[s], x[s], v[s][0]);
      v[s][1] = fma(t[s], y[s], v[s][1]);
      v[s][2] = fma(t[s], z[s], v[s][2]);
    }
  };
  double x[NS], y[NS], z[NS], wk[NS];
  int tk[NS];
  auto partner = [&](int k, auto own) {
    const double2 a = rxy[k], c = rzf[k];
    const double f = weight(k, c.y);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      x[s] = a.x;
      y[s] = a.y;
      z[s] = c.x;
      wk[s] = own(s) ? 0.0 : f;
      tk[s] = GM ? rt[k] : 0;
    }
    step(x, y, z, wk, tk);
  };
  if (RUNS) {
#pragma unroll
    for (int s0 = 0; s0 < NS; ++s0) {
      const int m = min(nk - s0 * LPA, LPA);
#pragma unroll 1
      for (int q = 0; q < m; ++q) partner(s0 * LPA + q, [&](int s) { return s == s0 && q == l; });
    }
  } else {
#pragma unroll 1
    for (int k = 0; k < nk; ++k) partner(k, [&](int s) { return k == l + s * LPA; });
  }
}

// Ten sums over the LPA lanes of an atom: eight by halving (each exchange
// keeps half of the sums), two by a full exchange.  On return lane l of the
// atom holds sum l & 7 in q[0] (bit-reversed, see rows_sum_index) and every lane holds
// the sums 8 and 9 in e0, e1.
template <int LPA>
__device__ __forceinline__ void rows_sums10(double (&q)[8], double &e0, double &e1, int l) {
#pragma unroll
  for (int h = 4, bit = 1; h > 0; h >>= 1, bit <<= 1) {
    const bool up = l & bit;
#pragma unroll
    for (int j = 0; j < h; ++j) {
      const double give = up ? q[j] : q[j + h], keep = up ? q[j + h] : q[j];
      q[j] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
  }
#pragma unroll
  for (int bit = 8; bit < LPA; bit <<= 1) q[0] += __shfl_xor_sync(0xffffffffu, q[0], bit);
#pragma unroll
  for (int bit = 1; bit < LPA; bit <<= 1) {
    e0 += __shfl_xor_sync(0xffffffffu, e0, bit);
    e1 += __shfl_xor_sync(0xffffffffu, e1, bit);
  }
}
__device__ __forceinline__ int rows_sum_index(int l) { return (l & 1) * 4 + (l & 2) + ((l >> 2) & 1); }

// The objective's forward pass (see k_atoms for the formulas): per-atom
// sums, reaction vectors V, and with AUX the per-slot triplet sums for the
// adjoint, for L.ncb candidates a CTA.  VS: db.vs where it is known at compile
// time (without angular terms the test would spill: 1846 -> 1873 us for 18 k
// atoms of 42 slots, 128 candidates), else 0.
template <bool MEAM, bool AUX, bool GM, bool JM, int LPA, int SPL, int VS>
__global__ void __launch_bounds__(32 * ROWS_W, JM ? 3 : 4)
    k_rows(DevDb db, DevPot pot, RowsLayout L, int ncand, const SplineGeom *__restrict__ geom,
           const double *__restrict__ tabs, const double *__restrict__ ptabs, double *__restrict__ Vout,
           double *__restrict__ aout, double *__restrict__ aux) {
  extern __shared__ __align__(16) unsigned char rsm[];
  constexpr int AW = 32 / LPA;
  const int vs = VS ? VS : db.vs;
  const int cand0 = blockIdx.y * L.ncb, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l = lane % LPA, sub = lane / LPA;
  const int N = db.natoms;
  const int64_t Np = db.npairs;
  rows_stage(rsm, L, pot, geom, tabs, ptabs, cand0, ncand);
  const SplineGeom *sg = reinterpret_cast<const SplineGeom *>(rsm + L.o_geo);
  const RowSpl *spl = reinterpret_cast<const RowSpl *>(rsm + L.o_spl);
  unsigned char *wrow = rsm + L.o_rows + warp * L.row_bytes;
  // this lane's atom's rows
  double2 *rxy = reinterpret_cast<double2 *>(wrow) + sub * L.rs;
  double2 *rzf = reinterpret_cast<double2 *>(wrow) + (AW + sub) * L.rs;
  double *rp = reinterpret_cast<double *>(wrow + 2 * sizeof(double2) * AW * L.rs) + sub * L.rs;  // + m AW rs
  int *rt = reinterpret_cast<int *>(wrow + 2 * sizeof(double2) * AW * L.rs) + sub * L.rs;
  const double2 *uxy = db.pair2, *uzr = uxy + Np, *irf = uzr + Np, *pr = irf + Np;

  const int ngroups = (N + AW - 1) / AW;
  for (int grp = blockIdx.x * ROWS_W + warp; grp < ngroups; grp += gridDim.x * ROWS_W) {
    const int i = grp * AW + sub;
    const bool live = i < N;
    const int lo = live ? db.pair_off[i] : 0, n = live ? db.pair_off[i + 1] - lo : 0;
    const int ti = live ? db.atom_type[i] : 0;
    const int nw = __reduce_max_sync(0xffffffffu, n);
    // kept over the candidates: the unit vectors, and without a row loop, which
    // needs the registers, everything else of the slots
    constexpr bool KEEP = !MEAM;
    double u[SPL][3], rk[SPL];
    int2 mk[SPL];
    double2 sk[SPL];
#pragma unroll
    for (int s = 0; s < SPL; ++s) {
      const int p = l + s * LPA, gs = lo + p;
      u[s][0] = u[s][1] = u[s][2] = rk[s] = 0.0;
      mk[s] = make_int2(0, 0);
      sk[s] = make_double2(0.0, 0.0);
      if (p < n) {
        const double2 a = uxy[gs], b = uzr[gs];
        u[s][0] = a.x;
        u[s][1] = a.y;
        u[s][2] = b.x;
        if (KEEP) {
          rk[s] = b.y;
          mk[s] = db.pair_meta[gs];
          sk[s] = pr[gs];
        }
      }
    }
    const double w = live ? db.cell_w[db.atom_cell[i]] : 0.0;
#pragma unroll 1
    for (int cc = 0; cc < L.ncb && cand0 + cc < ncand; ++cc) {
      const int cand = cand0 + cc;
      unsigned char *t = rsm + cc * L.tab_bytes;
      const double2 *plo = reinterpret_cast<const double2 *>(t), *phi = plo + L.npiece, *alo = phi + L.npiece,
                    *ahi = alo + L.nang;
      const double *tU = reinterpret_cast<const double *>(t + L.o_u) - L.u_off;
      double S[SPL], v[SPL][3];
      int tj[SPL] = {};  // GMEAM: the slots' types
      double Vd[SPL][3], cd[SPL], e3 = 0.0;  // JMEAM: the direct terms' part of V (vector, along u) and energy
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        S[s] = v[s][0] = v[s][1] = v[s][2] = 0.0;
        if (JM) Vd[s][0] = Vd[s][1] = Vd[s][2] = cd[s] = 0.0;
      }
      if (MEAM) {
#pragma unroll
        for (int s = 0; s < SPL; ++s) {
          if (s * LPA >= nw) break;
          const int p = l + s * LPA, gs = lo + p;
          double f = 0.0, pm[2] = {0.0, 0.0};
          int2 m2 = make_int2(0, 0);
          if (p < n) {
            m2 = db.pair_meta[gs];
            const int kf = ((m2.x >> 16) & 0xff) - 1, pij = pair_ij_index(ti, m2.y, pot.ntypes);
            double d;
            if (kf >= 0) f = rows_piece(plo, phi, spl[pot.s_f + pij].p0 + kf, irf[gs].y, d);
            if (JM)
              for (int m = 0; m < pot.nj; ++m) {
                const int kp = m ? (int)db.pair_knot_p2[gs] : ((m2.x >> 24) & 0xff) - 1;
                if (kp >= 0)
                  pm[m] = rows_piece(plo, phi, sg[pot.s_p[m] + pij].poff / 4 + kp, db.pair_shift[(3 + m) * Np + gs], d);
              }
          }
          rxy[p] = make_double2(u[s][0], u[s][1]);
          rzf[p] = make_double2(u[s][2], f);
          if (JM)
            for (int m = 0; m < pot.nj; ++m) rp[m * AW * L.rs + p] = pm[m];
          if (GM) rt[p] = tj[s] = m2.y;
        }
        __syncwarp();
        auto pass = [&](const RowSpl *a, auto weight) {
          if (nw == 0) return;  // no row is staged: the shared rows hold anything
          // as many slots a lane as the warp's longest row needs
          auto go = [&](auto cl) {
            constexpr bool CL = decltype(cl)::value;
            if (nw > 3 * LPA)
              rows_pass<CL, 4, SPL, LPA, GM, !JM>(rxy, rzf, rt, weight, nw, l, u, alo, ahi, a, pot, tj, S, v);
            else if (nw > 2 * LPA)
              rows_pass<CL, 3, SPL, LPA, GM, !JM>(rxy, rzf, rt, weight, nw, l, u, alo, ahi, a, pot, tj, S, v);
            else if (nw > LPA)
              rows_pass<CL, 2, SPL, LPA, GM, !JM>(rxy, rzf, rt, weight, nw, l, u, alo, ahi, a, pot, tj, S, v);
            else
              rows_pass<CL, 1, SPL, LPA, GM, !JM>(rxy, rzf, rt, weight, nw, l, u, alo, ahi, a, pot, tj, S, v);
          };
          if (pot.ang_cover) go(std::integral_constant<bool, false>{});
          else go(std::integral_constant<bool, true>{});
        };
        if (JM) {
          // the q terms' dfj without U' (pot_jmeam_spline.cpp:208-219, 263-273)
          for (int m = 0; m < pot.nj; ++m) {
            const RowSpl *a = spl + pot.s_q[m] + ti;
            const double *wp = rp + m * AW * L.rs;
            pass(a, [&](int k, double) { return wp[k]; });
#pragma unroll
            for (int s = 0; s < SPL; ++s) {
              const int p = l + s * LPA, gs = lo + p;
              if (p >= n) continue;
              const double vx = v[s][0] * a->inv, vy = v[s][1] * a->inv, vz = v[s][2] * a->inv;
              const double H = fma(u[s][0], vx, fma(u[s][1], vy, u[s][2] * vz));
              const int2 m2 = db.pair_meta[gs];
              const int kp = m ? (int)db.pair_knot_p2[gs] : ((m2.x >> 24) & 0xff) - 1;
              if (kp >= 0) {
                const SplineGeom &rg = sg[pot.s_p[m] + pair_ij_index(ti, m2.y, pot.ntypes)];
                double d;
                const double pv = rows_piece(plo, phi, rg.poff / 4 + kp, db.pair_shift[(3 + m) * Np + gs], d);
                const double pi = pv * irf[gs].x;
                cd[s] += fma(d * rg.invstep, S[s], -(pi * H));
                Vd[s][0] += pi * vx;
                Vd[s][1] += pi * vy;
                Vd[s][2] += pi * vz;
                e3 += 0.5 * pv * S[s];
              }
              if (AUX) {
                double *ax = aux + ((size_t)cand * pot.aux_rows + AUX_COUNT * (1 + m)) * Np + gs;
                ax[AUX_G * Np] = S[s];
                ax[AUX_H * Np] = H;
                ax[AUX_VX * Np] = vx;
                ax[AUX_VY * Np] = vy;
                ax[AUX_VZ * Np] = vz;
              }
            }
          }
        }
        pass(spl + (GM ? pot.s_g + ti * pot.npair : pot.s_g + ti), [](int, double f) { return f; });
      }
      // ---- per slot: V = u (A + U' B) + U' C, with C left in v.  Sums of products are written as fma, so that every
      // instance of the kernel (with and without AUX) rounds alike.
      const double ginv = MEAM && !GM ? spl[pot.s_g + ti].inv : 1.0;
      double A[SPL], B[SPL], rho = 0.0, ep = e3;
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        A[s] = B[s] = 0.0;
        const int p = l + s * LPA, gs = lo + p;
        if (p >= n) continue;
        const int2 m2 = KEEP ? mk[s] : db.pair_meta[gs];
        const double2 b = KEEP ? sk[s] : pr[gs];  // shifts of phi, rho
        const int kphi = (m2.x & 0xff) - 1, krho = ((m2.x >> 8) & 0xff) - 1;
        const int pij = pair_ij_index(ti, m2.y, pot.ntypes);
        const double share = MEAM ? 0.5 : phi_share(pot, pot.pair && db.pair_nbr[gs] == i);
        double d;
        if (kphi >= 0) {
          const RowSpl &g = spl[pot.s_phi + pij];
          ep += share * rows_piece(plo, phi, g.p0 + kphi, b.x, d);
          A[s] = share * d * g.inv;
        }
        if (krho >= 0) {
          const RowSpl &g = spl[pot.s_rho + m2.y];
          rho += rows_piece(plo, phi, g.p0 + krho, b.y, d);
          B[s] = d * g.inv;
        }
        if (MEAM) {
          const double vx = v[s][0] * ginv, vy = v[s][1] * ginv, vz = v[s][2] * ginv;
          const double H = fma(u[s][0], vx, fma(u[s][1], vy, u[s][2] * vz));
          const int kf = ((m2.x >> 16) & 0xff) - 1;
          const double2 c = irf[gs];  // 1 / r, shift of f
          double fi = 0.0;
          if (kf >= 0) {
            const RowSpl &g = spl[pot.s_f + pij];
            const double f = rows_piece(plo, phi, g.p0 + kf, c.y, d);
            rho += 0.5 * f * S[s];
            fi = f * c.x;
            B[s] += fma(d * g.inv, S[s], -(fi * H));
          }
          if (AUX) {
            double *ax = aux + (size_t)cand * pot.aux_rows * Np + gs;
            ax[AUX_G * Np] = S[s];
            ax[AUX_H * Np] = H;
            ax[AUX_VX * Np] = vx;
            ax[AUX_VY * Np] = vy;
            ax[AUX_VZ * Np] = vz;
          }
          v[s][0] = fi * vx;
          v[s][1] = fi * vy;
          v[s][2] = fi * vz;
        }
      }
#pragma unroll
      for (int o = 1; o < LPA; o <<= 1) rho += __shfl_xor_sync(0xffffffffu, rho, o);
      // ---- embedding (pot_meam_spline.cpp:208-223), every lane of the atom
      double dF = 0.0, Uv = 0.0, pen = 0.0;
      const double rho_raw = pot.pair ? 0.0 : rho;
      if (!pot.pair && live) {
        const SplineGeom &gU = sg[pot.s_U + ti];
        const double x0 = gU.x0, xN = gU.xN;
        if (rho < x0) {
          pen = w * 100.0 * 10. * (x0 - rho) * (x0 - rho);
          if (!pot.embed_extrap) rho = x0;
        } else if (rho > xN) {
          pen = w * 100.0 * 10. * (rho - xN) * (rho - xN);
          if (!pot.embed_extrap) rho = xN;
        }
        const PointEval U = spl_point(tU, gU, rho);
        dF = U.grad;
        Uv = U.val;
      }
      // ---- V and the slot's stress (stress.h:134-137; pot_meam_spline.cpp:171-173, 234-236, 265-268)
      double q[8], s8 = 0.0, s9 = 0.0;  // force 3, energy, stress xx yy zz xy | yz, zx
#pragma unroll
      for (int j = 0; j < 8; ++j) q[j] = 0.0;
      q[3] = ep;
      double *Vc = Vout + ((size_t)cand * Np + lo) * vs;
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        const int p = l + s * LPA;
        if (p >= n) continue;
        double cu = fma(dF, B[s], A[s]), V[3];
        if (JM) cu += cd[s];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          V[k] = u[s][k] * cu;
          if (MEAM) V[k] = fma(dF, v[s][k], V[k]);
          if (JM) V[k] += Vd[s][k];
          q[k] += V[k];
        }
        if (vs == 4) {
          store_vec4(Vc + 4 * (int64_t)p, V[0], V[1], V[2]);
        } else {
#pragma unroll
          for (int k = 0; k < 3; ++k) Vc[3 * (int64_t)p + k] = V[k];
        }
        const double r = KEEP ? rk[s] : uzr[lo + p].y, x = V[0] * r, y = V[1] * r, z = V[2] * r;
        q[4] -= u[s][0] * x;
        q[5] -= u[s][1] * y;
        q[6] -= u[s][2] * z;
        q[7] -= u[s][0] * y;
        s8 -= u[s][1] * z;
        s9 -= u[s][2] * x;
      }
      rows_sums10<LPA>(q, s8, s9, l);
      if (live) {
        double *ao = aout + (size_t)cand * AO_COUNT * N + i;
        const int qi = rows_sum_index(l);
        if (l < 8) ao[(qi < 3 ? AO_AX + qi : qi == 3 ? (int)AO_E : AO_S0 + qi - 4) * N] = qi == 3 ? q[0] + Uv : q[0];
        if (l == 0) {
          ao[(AO_S0 + 4) * N] = s8;
          ao[(AO_S0 + 5) * N] = s9;
          ao[AO_PEN * N] = pen;
          ao[AO_RHO * N] = rho_raw;
        }
      }
      if (MEAM) __syncwarp();  // the next candidate or group reuses the rows
    }
  }
}

// (LPA, SPL) for rows of up to max_row slots: 4 slots a lane, and as few
// lanes as hold the row (idle lanes in short rows cost as much as busy ones);
// 0 when the row is too long for the warp kernels.
inline int rows_lpa(int max_row) { return max_row <= 32 ? 8 : max_row <= 64 ? 16 : max_row <= ROWS_MAXROW ? 32 : 0; }

}  // namespace mzb
