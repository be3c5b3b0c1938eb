// The column passes of the RK3 step along y and z (tgv_cols.cu).
#pragma once
#include "tgv.cuh"

namespace astr {

// Derivative and filter of one direction in common chunks of rows.
struct ColDir {
  DevColOp d, f;
};
// Directions 1 and 2 of out[3], from the operators of the three directions.
cudaError_t make_coldirs(const HostOp* hd, const HostOp* hf, ColDir* out);
void free_coldirs(ColDir* dirs);
int col_lines(const ColDir& d);   // lines per CTA
// pass: ColPass of tgv_cols.cuh (0 filter in place, 1 gradients, 2 R += D(G), 3 update and filter);
// G: the fields that passes 1 to 3 differentiate.
cudaError_t launch_col_pass(int pass, const PassArgs& p, const double* G, const ColDir& d, cudaStream_t st);
// u, v, w, T of p.q into four fields.
cudaError_t launch_prims(const PassArgs& p, double* U, cudaStream_t st);

}  // namespace astr
