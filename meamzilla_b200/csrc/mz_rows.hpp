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
  const SplineGeom *geom;
  const double *tabs, *ptabs;  // knot tables, evaluation tables of the candidates
  double *V, *aout;            // reaction vectors, per-atom sums
  double *aux;                 // per-slot triplet sums for the adjoint, or null
  cudaStream_t stream;
};
cudaError_t rows_forward(const RowsForward &a);
size_t rows_forward_bytes(const DevPot &pot, int lpa);  // shared memory of a CTA

}  // namespace mzb
