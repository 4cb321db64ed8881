// Launches of the FP64 row kernels (mz_rows.cuh).
#include <cuda_runtime.h>

#include <algorithm>

#include "mz_b200.h"
#include "mz_device.cuh"
#include "mz_rows.cuh"
#include "mz_rows.hpp"

namespace mzb {

namespace {

RowsLayout rows_forward_layout(const DevPot &pot, int lpa, int ncb) {
  return rows_layout(pot, lpa, 4, pot.s_g > 0, ncb);
}

template <bool MEAM, bool AUX, bool GM, bool JM, int LPA, int VS = 0>
cudaError_t forward(const RowsForward &a) {
  auto k = k_rows<MEAM, AUX, GM, JM, LPA, 4, VS>;
  // One group of atoms a warp and one candidate a CTA while that is less than
  // eight waves of CTAs (4 resident per SM); then up to four candidates, which
  // share the slots' loads, and up to eight groups, which share the tables.
  // Without angular terms, where the loads are a larger part, up to eight
  // candidates (18 k atoms of 42 slots, 128 candidates: 1408 -> 1329 us, 1383
  // with sixteen; with angular terms 1171 -> 1221 us for 21 k atoms, 56).
  const int64_t groups = ((int64_t)a.db.natoms * LPA + 31) / 32;
  const int64_t ctas = (groups + ROWS_W - 1) / ROWS_W, wave = 4 * (int64_t)a.nsm;
  int ncb = (int)std::min<int64_t>(std::min(a.ncand, a.meam ? 4 : 8), std::max<int64_t>(1, ctas * a.ncand / (8 * wave)));
  RowsLayout L = rows_forward_layout(a.pot, LPA, ncb);
  while (ncb > 1 && L.bytes > 48 * 1024) L = rows_forward_layout(a.pot, LPA, --ncb);  // four CTAs on an SM
  const int64_t ny = (a.ncand + ncb - 1) / ncb;
  const int64_t it = std::min<int64_t>(8, std::max<int64_t>(1, ctas * ny / (8 * wave)));
  if (L.bytes > 48 * 1024) {  // the limit is the kernel's, shared by all contexts: always the largest
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, a.smem_block);
    if (e != cudaSuccess) return e;
  }
  k<<<dim3((unsigned)((ctas + it - 1) / it), (unsigned)ny), 32 * ROWS_W, L.bytes, a.stream>>>(
      a.db, a.pot, L, a.ncand, a.geom, a.tabs, a.ptabs, a.V, a.aout, a.aux);
  return cudaGetLastError();
}

template <int LPA>
cudaError_t forward_lpa(const RowsForward &a) {
  if (!a.meam)
    return a.db.vs == 4 ? forward<false, false, false, false, LPA, 4>(a) : forward<false, false, false, false, LPA, 3>(a);
  if (a.pot.nj > 0)
    return a.aux ? forward<true, true, false, true, LPA>(a) : forward<true, false, false, true, LPA>(a);
  if (a.pot.gmeam)
    return a.aux ? forward<true, true, true, false, LPA>(a) : forward<true, false, true, false, LPA>(a);
  return a.aux ? forward<true, true, false, false, LPA>(a) : forward<true, false, false, false, LPA>(a);
}

}  // namespace

size_t rows_forward_bytes(const DevPot &pot, int lpa) { return rows_forward_layout(pot, lpa, 1).bytes; }

cudaError_t rows_forward(const RowsForward &a) {
  switch (rows_lpa(a.max_row)) {
    case 8: return forward_lpa<8>(a);
    case 16: return forward_lpa<16>(a);
    default: return forward_lpa<32>(a);
  }
}

}  // namespace mzb
