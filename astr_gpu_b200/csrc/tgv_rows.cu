// Launches of the x passes (tgv_rows.cuh).
#include <algorithm>

#include "tgv_cols.h"
#include "tgv_rows.cuh"

namespace astr {

namespace {

// Smallest pitch of at least `need` doubles that is `res` mod 16.
int pitch(int need, int res) { return need + ((res - need) % 16 + 16) % 16; }

template <class K, class C>
cudaError_t launch(K kern, dim3 grid, int threads, size_t smem, cudaStream_t st, const RowArgs& a, const C& c) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, smem, st>>>(a, c);
  return cudaGetLastError();
}

template <int S, int NL>
cudaError_t launch_c(RowArgs& a, const RowOps& r, cudaStream_t st) {
  a.LT = (a.g.N[0] + 2) & ~1;
  a.LG = pitch(a.g.N[0] + 1 + 2 * ROW_HX, NL == 2 ? 2 : 1);
  const size_t smem = ((size_t)5 * NL * (a.LT + a.LG) + S + 8 + 2 * (size_t)a.op.nch * 5 * NL) * sizeof(double);
  const dim3 grid((unsigned)((a.g.N[1] + NL) / NL), (unsigned)(a.g.N[2] + 1));
  const ColConst<S> k = r.d.consts<S>();
  return a.partials ? launch(row_detail::k_row_c<S, NL, true>, grid, 256, smem, st, a, k)
                    : launch(row_detail::k_row_c<S, NL, false>, grid, 256, smem, st, a, k);
}

template <int S>
cudaError_t launch_f(RowArgs& a, const RowOps& r, cudaStream_t st) {
  a.LG = pitch(a.g.N[0] + 1 + 2 * ROW_HF, 2);
  const size_t smem = ((size_t)8 * a.LG + S + 8 + 2 * (size_t)a.op.nch * 8) * sizeof(double);
  const unsigned ctas = 5u * (unsigned)((a.g.N[1] + 8) / 8) * (unsigned)(a.g.N[2] + 1);
  return launch(row_detail::k_row_filter<S>, dim3(ctas), (a.op.nch * 8 + 31) / 32 * 32, smem, st, a, r.f.consts<S>());
}

RowArgs row_args(const PassArgs& p, const DevColOp& op, double scale) {
  RowArgs a{};
  a.g = p.g;
  a.th = p.th;
  a.op = op.op;
  a.w = col_weights(op, scale);
  for (int r = 0; r < 3; ++r)
    for (int j = 0; j < 11; ++j) a.ch[r][j] = op.line.ch[r][j];
  a.q = p.q; a.DA = p.DA; a.DB = p.DB; a.VF = p.VF; a.R = p.R; a.DC = p.DC;
  a.partials = p.partials; a.err = p.err;
  return a;
}

}  // namespace

// Lines per CTA and rows per chunk of pass C: five fields x NL lines x chunks in 256 threads, two CTAs
// per SM of tiles. Measured, ms per launch: 512^3 25 rows 2 lines 7.6, 33 rows 2 lines 8.2, 17 rows 2
// lines in 320 threads of 96 registers 8.5, 25 rows 1 line in 128 threads 7.7; 256^3 25 rows 4 lines
// 0.98, 2 lines 1.30. Boxes wider than 822 nodes keep the lane-scan kernel (one CTA per SM either way).
RowShape row_c_shape(int nsys) {
  if (nsys <= 45) return {9, 8};
  if (nsys <= 102) return {17, 8};
  if (nsys <= 204) return {17, 4};
  if (nsys <= 300) return {25, 4};
  if (nsys <= 625) return {25, 2};
  if (nsys <= 825) return {33, 2};
  return {0, 0};
}
// Rows per chunk of the filter along x: at most 32 chunks.
int row_f_rows(int nsys) {
  if (nsys <= 45) return 9;
  if (nsys <= 176) return 17;
  if (nsys <= 1056) return 33;
  return 0;
}

int row_c_tiles(const BoxGeo& g, const RowOps& r) { return (g.N[1] + r.c.NL) / r.c.NL * (g.N[2] + 1); }

cudaError_t launch_row_c(const PassArgs& p, const RowOps& r, cudaStream_t st) {
  RowArgs a = row_args(p, r.d, p.g.rd[0]);
  switch (r.c.S * 10 + r.c.NL) {
    case 98: return launch_c<9, 8>(a, r, st);
    case 178: return launch_c<17, 8>(a, r, st);
    case 174: return launch_c<17, 4>(a, r, st);
    case 254: return launch_c<25, 4>(a, r, st);
    case 252: return launch_c<25, 2>(a, r, st);
    case 332: return launch_c<33, 2>(a, r, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_row_filter(const PassArgs& p, const RowOps& r, cudaStream_t st) {
  RowArgs a = row_args(p, r.f, 1.0);
  if (r.f.S == 9) return launch_f<9>(a, r, st);
  if (r.f.S == 17) return launch_f<17>(a, r, st);
  if (r.f.S == 33) return launch_f<33>(a, r, st);
  return cudaErrorInvalidValue;
}

}  // namespace astr
