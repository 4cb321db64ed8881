// The FP64 row kernels as the evaluator calls them (mz_rows.cu).
#pragma once

#include <cuda_runtime.h>

#include "mz_device.cuh"

namespace mzb {

struct RowsForward {
  DevDb db;
  DevPot pot;
  bool meam;          // a style with angular terms
  int max_row;        // longest neighbour row
  int ncand, nsm;
  int smem_block;     // most shared memory a block may opt into
  const SplineGeom *geom;
  const double *tabs, *ptabs;  // knot tables, evaluation tables of the candidates
  double *V, *aout;            // reaction vectors, per-atom sums
  double *aux;                 // per-slot triplet sums for the adjoint, or null
  cudaStream_t stream;
};
cudaError_t rows_forward(const RowsForward &a);
size_t rows_forward_bytes(const DevPot &pot, int lpa);  // shared memory of a CTA

// ------------------------------------------------------------- adjoint

constexpr int RADIAL_SEG = 2048;   // most slots per segment of the radial sums
constexpr int RADIAL_MAXB = 512;   // most buckets of the radial sums (44 KB a CTA)
constexpr int RADIAL_ITEM = 32;    // most slots per item of the radial sums

// Which bucket (radial function, spline, interval) every slot falls into:
// function F's bucket is b0[F] + (spline within the group) nint[F] + interval.
struct RadialPlan {
  int nfun, b0[4], nint[3], nb;  // functions (phi, rho, f), first buckets, intervals per spline, buckets
  int seg, nseg;           // slots per segment, segments
  unsigned short *order;   // [nfun][Np] slots of a segment by bucket
  unsigned short *off;     // [nseg][nb + 1] starts within (segment, function); see k_rows_sort
  unsigned short *item;    // [nseg][nb + 1] first item of each bucket
  int *slot_atom;          // [Np]
};

struct RowsAdjoint {
  DevDb db;
  DevPot pot;
  bool meam;
  int max_row, ncand, smem_block;
  RadialPlan radial;
  const int4 *desc;    // groups of atoms, see k_rows_adj
  int ngroups;
  int warps;           // per CTA of k_rows_adj
  int ctas, rctas;     // of k_rows_adj and k_rows_radial, per candidate
  const SplineGeom *geom;
  const double *tabs, *ptabs;
  double *aout;
  const double *aux, *lam, *seeds;
  double *W1;                  // [ncand][3][Np] scratch (the reaction vectors' place)
  double *part, *rpart;        // [ncand][ctas][part], [ncand][rctas][4 nb]
  cudaStream_t stream;
};
int rows_adj_lpa(int max_row);
struct RowsAdjShape {
  int warps, per_sm;  // warps per CTA (0: does not fit), CTAs per SM
  int part, nang;     // doubles of a warp's partial, angular pieces
};
RowsAdjShape rows_adj_shape(const DevPot &pot, int max_row, bool meam, size_t smem_block, size_t smem_sm);
cudaError_t rows_sort(const DevDb &db, const DevPot &pot, const RadialPlan &R, cudaStream_t st);
cudaError_t rows_adjoint(const RowsAdjoint &a);
cudaError_t rows_radial(const RowsAdjoint &a);

// The summed pieces of one candidate (ang [4 per angular piece, U tables],
// rad [4 nb]) added into the table gradient ext [stride] (zeroed): entry by
// entry, so in a fixed order.  All threads of a CTA.
__device__ __forceinline__ void rows_pieces_to_table(const DevPot &pot, const SplineGeom *__restrict__ geom,
                                                     const RadialPlan &R, int nang, int ang0,
                                                     const double *__restrict__ ang, const double *__restrict__ rad,
                                                     double *ext) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int s = warp; s < pot.nsplines; s += blockDim.x / 32) {
    const SplineGeom g = geom[s];
    const int n = g.n;
    if (!pot.pair && s >= pot.s_U && s < pot.s_U + pot.ntypes) {
      for (int e = lane; e < 2 * n + 2; e += 32) ext[g.toff + e] = ang[4 * nang + g.toff - pot.u_off + e];
      continue;
    }
    const bool angular = nang > 0 && s >= pot.s_g;
    // dF/dc of interval m's polynomial in the shift
    auto piece = [&](int m, double (&d)[4]) {
      d[0] = d[1] = d[2] = d[3] = 0.0;
      if (m < 0 || m > n - 2) return;
      if (angular) {
        const int p0 = g.poff / 4 - ang0 + 2 * (s - pot.s_g) + 1;
        for (int k = m == 0 ? -1 : m; k <= (m == n - 2 ? n - 1 : m); ++k) {
          const double *e = ang + 4 * (p0 + k);
          const double x = 0.5 + (double)(k - m);
          d[0] += e[0];
          d[1] += x * e[0] + e[1];
          d[2] += x * (x * e[0] + 2.0 * e[1]) + e[2];
          d[3] += x * (x * (x * e[0] + 3.0 * e[1]) + 3.0 * e[2]) + e[3];
        }
      } else {
        const int F = !pot.pair && s >= pot.s_rho && s < pot.s_rho + pot.ntypes ? 1 : s < pot.s_phi + pot.npair ? 0 : 2;
        const int s0 = F == 0 ? pot.s_phi : F == 1 ? pot.s_rho : pot.s_f;
        const double *e = rad + 4 * (R.b0[F] + (s - s0) * R.nint[F] + m);
        for (int q = 0; q < 4; ++q) d[q] = e[q];
      }
    };
    // y_m: c0, c1 of piece m and c1 of piece m - 1; y''_m likewise (see power_to_table)
    const double H = g.step * g.step / 6.0;
    for (int m = lane; m < n; m += 32) {
      double a[4], b[4];
      piece(m, a);
      piece(m - 1, b);
      ext[g.toff + m] = (a[0] - a[1]) + b[1];
      ext[g.toff + n + m] = (-2.0 * H * a[1] + 3.0 * H * a[2] - H * a[3]) + (-H * b[1] + H * b[3]);
    }
    if (lane < 2) ext[g.toff + 2 * n + lane] = 0.0;
  }
}

}  // namespace mzb
