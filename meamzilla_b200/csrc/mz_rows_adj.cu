// Launches of the FP64 row adjoint (mz_rows_adj.cuh).
#include <cuda_runtime.h>

#include <algorithm>

#include "mz_b200.h"
#include "mz_device.cuh"
#include "mz_rows_adj.cuh"

namespace mzb {

namespace {

using AdjKernel = void (*)(DevDb, DevPot, RadjLayout, const int4 *, int, const SplineGeom *, const double *,
                           const double *, double *, const double *, const double *, const double *, double *,
                           double *);

template <int LPA>
AdjKernel pick(const DevPot &pot, bool meam) {
  if (!meam) return k_rows_adj<false, false, LPA>;
  return pot.gmeam ? k_rows_adj<true, true, LPA> : k_rows_adj<true, false, LPA>;
}

AdjKernel kernel(const RowsAdjoint &a) {
  const int lpa = rows_lpa(a.max_row);
  return lpa == 8 ? pick<8>(a.pot, a.meam) : lpa == 16 ? pick<16>(a.pot, a.meam) : pick<32>(a.pot, a.meam);
}

}  // namespace

int rows_adj_lpa(int max_row) { return rows_lpa(max_row); }

// Warps per CTA: as many as give an SM the most, by shared memory (a warp's
// rows and its lanes' angular tables are 18 KB for 8 angular knots) and by
// the kernel's 12 warps of registers.
RowsAdjShape rows_adj_shape(const DevPot &pot, int max_row, bool meam, size_t smem_block, size_t smem_sm) {
  RowsAdjShape best{};
  int most = 0;
  for (int w = 1; w <= RADJ_MAXW; ++w) {
    const RadjLayout L = radj_layout(pot, rows_lpa(max_row), meam, w);
    if (L.bytes > smem_block) break;
    const int per = std::min((int)(smem_sm / (L.bytes + 1024)), RADJ_MAXW / w);
    if (per * w > most) {
      most = per * w;
      best = RowsAdjShape{w, per, L.part, L.rows.nang};
    }
  }
  return best;
}

cudaError_t rows_sort(const DevDb &db, const DevPot &pot, const RadialPlan &R, cudaStream_t st) {
  if (R.nseg > 0) k_rows_sort<<<R.nseg, RADIAL_T, 0, st>>>(db, pot, R);
  return cudaGetLastError();
}

cudaError_t rows_adjoint(const RowsAdjoint &a) {
  const RadjLayout L = radj_layout(a.pot, rows_lpa(a.max_row), a.meam, a.warps);
  AdjKernel k = kernel(a);
  // the limit is the kernel's, shared by all contexts: always the largest
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, a.smem_block);
  if (e != cudaSuccess) return e;
  k<<<dim3(a.ctas, a.ncand), 32 * L.warps, L.bytes, a.stream>>>(a.db, a.pot, L, a.desc, a.ngroups, a.geom, a.tabs,
                                                               a.ptabs, a.aout, a.aux, a.lam, a.seeds, a.W1, a.part);
  return cudaGetLastError();
}

cudaError_t rows_radial(const RowsAdjoint &a) {
  k_rows_radial<<<dim3(a.rctas, a.ncand), RADIAL_T, radial_smem(a.radial), a.stream>>>(
      a.db, a.pot, a.radial, a.geom, a.aout, a.aux, a.W1, a.rpart);
  return cudaGetLastError();
}

}  // namespace mzb
