// Stage products as convolutions over the beam grid (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "beam_grid.h"
#include "common.cuh"
#include "kernels.h"

namespace trhepd {

// max over columns and twins of |conj(u[e1]) - w[e2]| > 1e-14 |u[0]| sets *bad
void launch_conv_check(const TableEntry* table, int ncol, int nv, const int* twins, int ntwins,
                       int* bad, cudaStream_t st);

size_t conv_spectrum_elems(int m);  // complex values per stage column
// Spectra of `ncol` consecutive columns per problem (tables: device array of nprob
// table pointers, or nullptr for the single `table`).
void launch_conv_spectra(const TableEntry* table, const TableEntry* const* tables, int nprob,
                         size_t col0, int ncol, int nv, const int* entry, int m, int sx, int sy,
                         cd* spec, size_t spec_stride, cudaStream_t st);

// `nstage` stages of P += cb (Q V + Q o D), Q += ca P on every row, V of stage i at
// spec + i * conv_spectrum_elems(m) (+ problem * spec_stride).  Stage i has the
// coefficients of k = i mod s; stage 0 takes cb0 instead.
struct ConvStages {
  cd* Q;
  cd* P;
  const cd* spec;
  size_t spec_stride;
  const int* cell;
  const unsigned* mask;
  const double* D;  // nang x sy x m (real: D = -gamma^2), 0 in cells without a beam
  int n, ld, rows, rows_b, m, sx, sy, nstage, s;
  double cb0, cb[11], ca[11];
};
void launch_conv_stages(const ConvStages& a, int max_ctas, cudaStream_t st);

}  // namespace trhepd
