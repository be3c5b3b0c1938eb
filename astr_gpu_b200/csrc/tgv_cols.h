// The column passes of the RK3 step: along y and z (tgv_cols.cu) and along x (tgv_rows.cu).
#pragma once
#include "tgv.cuh"

namespace astr {

// Derivative and filter of one direction in common chunks of rows.
struct ColDir {
  DevColOp d, f;
};
// The x passes' operators: rows per chunk (S of c and f.S, 0: the box is too wide) and lines per CTA.
struct RowShape {
  int S, NL;
};
struct RowOps {
  DevColOp d, f;
  RowShape c{0, 0};
};
RowShape row_c_shape(int nsys);
int row_f_rows(int nsys);
int row_c_tiles(const BoxGeo& g, const RowOps& r);   // CTAs of pass C, one partial sum each
cudaError_t launch_row_c(const PassArgs& p, const RowOps& r, cudaStream_t st);
cudaError_t launch_row_filter(const PassArgs& p, const RowOps& r, cudaStream_t st);

// Directions 1 and 2 of cols[3] and the x operators, from the operators of the three directions: all but
// the device copy of their table (load_colops).
cudaError_t fill_coldirs(const HostOp* hd, const HostOp* hf, ColDir* cols, RowOps& rows, std::vector<ColSpec>& specs,
                         std::vector<double>& tab);
int col_lines(const ColDir& d);   // lines per CTA
// pass: ColPass of tgv_cols.cuh (0 filter in place, 1 gradients, 2 R += D(G), 3 update and filter);
// G: the fields that passes 1 to 3 differentiate.
cudaError_t launch_col_pass(int pass, const PassArgs& p, const double* G, const ColDir& d, cudaStream_t st);
// u, v, w, T of p.q into four fields.
cudaError_t launch_prims(const PassArgs& p, double* U, cudaStream_t st);

}  // namespace astr
