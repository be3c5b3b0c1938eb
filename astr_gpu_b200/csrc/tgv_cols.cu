// Launches of the column passes (tgv_cols.cuh).
#include "tgv_cols.h"

#include "tgv_cols.cuh"

namespace astr {

namespace {

// Lines per CTA: 32 while two CTAs of 128 registers per thread fit on an SM (up to 8 chunks).
int lines_per_cta(int nch) { return nch <= 8 ? 32 : 16; }

template <int PASS, int S, int LW, int DIR>
cudaError_t launch(const ColArgs& a, const ColDir& d, int ntiles, size_t smem, cudaStream_t st) {
  auto kern = col_detail::k_col<PASS, S, LW, DIR>;
  const int threads = (d.d.op.nch * LW + 31) / 32 * 32;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kern<<<(unsigned)(ntiles * col_fields(PASS)), threads, smem, st>>>(a, d.d.consts<S>(), d.f.consts<S>());
  return cudaGetLastError();
}

template <int S, int LW, int DIR>
cudaError_t launch_pass(int pass, const ColArgs& a, const ColDir& d, int ntiles, size_t smem, cudaStream_t st) {
  switch (pass) {
    case COL_FILTER: return launch<COL_FILTER, S, LW, DIR>(a, d, ntiles, smem, st);
    case COL_GRAD: return launch<COL_GRAD, S, LW, DIR>(a, d, ntiles, smem, st);
    case COL_DIV: return launch<COL_DIV, S, LW, DIR>(a, d, ntiles, smem, st);
    default: return launch<COL_UPDATE, S, LW, DIR>(a, d, ntiles, smem, st);
  }
}

template <int DIR>
cudaError_t launch_dir(int pass, const ColArgs& a, const ColDir& d, int LW, int ntiles, size_t smem, cudaStream_t st) {
  switch (d.d.S) {
    case 9: return launch_pass<9, 32, DIR>(pass, a, d, ntiles, smem, st);
    case 17: return launch_pass<17, 32, DIR>(pass, a, d, ntiles, smem, st);
    case 33:
      return LW == 32 ? launch_pass<33, 32, DIR>(pass, a, d, ntiles, smem, st)
                      : launch_pass<33, 16, DIR>(pass, a, d, ntiles, smem, st);
    case 37: return launch_pass<37, 16, DIR>(pass, a, d, ntiles, smem, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

int col_lines(const ColDir& d) { return lines_per_cta(d.d.op.nch); }

cudaError_t fill_coldirs(const HostOp* hd, const HostOp* hf, ColDir* out, RowOps& rows, std::vector<ColSpec>& specs,
                         std::vector<double>& tab) {
  for (int d = 1; d < 3; ++d) {
    const int S = col_rows_per_chunk(hf[d].nsys(), d);
    specs.push_back({&hd[d], S, (hf[d].nsys() - hd[d].nsys()) / 2, &out[d].d});
    specs.push_back({&hf[d], S, 0, &out[d].f});
  }
  rows.c = row_c_shape(hd[0].nsys());
  if (rows.c.S) specs.push_back({&hd[0], rows.c.S, 0, &rows.d});
  if (const int S = row_f_rows(hf[0].nsys())) specs.push_back({&hf[0], S, 0, &rows.f});
  return fill_colops(specs.data(), (int)specs.size(), tab);
}

cudaError_t launch_col_pass(int pass, const PassArgs& p, const double* G, const ColDir& d, cudaStream_t st) {
  ColArgs a{};
  a.g = p.g;
  a.th = p.th;
  a.od = d.d.op;
  a.of = d.f.op;
  a.wd = col_weights(d.d, p.g.rd[p.dir]);
  a.wf = col_weights(d.f, 1.0);
  for (int r = 0; r < 3; ++r)
    for (int j = 0; j < 11; ++j) a.ch[r][j] = d.f.line.ch[r][j];
  const int o2 = p.dir == 2 ? 1 : 2;
  const int LW = lines_per_cta(a.od.nch);
  const int64_t nx = p.g.N[0] + 1, n2 = p.g.N[o2] + 1;
  a.ntx = (int)((nx + LW - 1) / LW);
  a.flat = 10 * (int64_t)a.ntx * LW > 11 * nx;   // more than a tenth of the lanes past the edge
  const int ntiles = (int)(a.flat ? (nx * n2 + LW - 1) / LW : a.ntx * n2);
  a.q = p.q; a.qout = p.qout; a.R = p.R; a.D = p.D; a.qsave = p.qsave; a.G = G;
  a.do_filter = p.do_filter;
  a.c1 = p.c1; a.c2 = p.c2; a.c3 = p.c3; a.dt = p.dt; a.pdt = p.pdt;
  size_t smem = (size_t)2 * a.od.nch * LW * sizeof(double);
  if (pass == COL_UPDATE && p.do_filter) smem += (size_t)(p.g.N[p.dir] + 1 + 2 * COL_IMG) * LW * sizeof(double);
  return p.dir == 1 ? launch_dir<1>(pass, a, d, LW, ntiles, smem, st) : launch_dir<2>(pass, a, d, LW, ntiles, smem, st);
}

cudaError_t launch_prims(const PassArgs& p, double* U, cudaStream_t st) {
  const int64_t n2 = p.g.fs / 2;   // rows are padded to a multiple of 16 nodes
  col_detail::k_prims<<<(unsigned)((n2 + 255) / 256), 256, 0, st>>>(p.q, U, n2, p.g.fs, p.th);
  return cudaGetLastError();
}

}  // namespace astr
