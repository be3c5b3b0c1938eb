// The y and z passes of the RK3 step as column solves (colsolve.cuh): one field of LW adjacent lines
// per CTA, read from HBM straight into registers.
//
// 512^3 on a B200, ms per launch (GB/s of the fields read and written): filter 2.8 (3820), derivative
// of u, v, w, T 1.82 (5350), R += D(G) 3.17 (5110), flux + update + filter 5.86 (4300 on the mean of the
// stages); the lane-scan forms of tgv_kernels.cuh took 3.0, 3.97, 4.22 and 9.03. Registers hold the
// tile, so 16 warps per SM are resident: load latency and the solve's two barriers bound it, not the
// FP64 pipe (12-24 % busy).
//
// Derivative and filter use the same chunks of rows: the derivative's system (nodes -1..N+1) is
// embedded in the filter's (nodes -3..N+3) with identity rows, so the solution of the flux derivative
// is in the registers of the thread that updates and filters those nodes.
#pragma once
#include "tgv.cuh"

namespace astr {

struct ColArgs {
  BoxGeo g;
  Thermo th;
  ColOp od, of;             // derivative (embedded) and filter
  ColWeights wd, wf;        // right-hand side weights (the derivative's with 1/dx)
  double ch[3][11];         // the filter's halo closure rows
  int ntx, flat;            // tiles along x (flat: tiles of the flattened plane)
  double* q;
  double* qout;
  double* R;
  double* D;
  const double* qsave;
  const double* G;          // fields to differentiate: 5 fluxes, or u, v, w, T
  int do_filter;
  double c1, c2, c3, dt;
  const double* pdt;        // dt on the device when not null
};

enum ColPass { COL_FILTER = 0, COL_GRAD = 1, COL_DIV = 2, COL_UPDATE = 3 };
__host__ __device__ constexpr int col_fields(int pass) { return pass == COL_GRAD ? 4 : 5; }
constexpr int COL_IMG = 8;  // rows of the update pass's tile before node 0 and after node N (5 periodic images)

namespace col_detail {

// This thread's line: element offset of its node 0; false when it is past the last line (the offset
// is then some valid line's).
template <int DIR, int LW>
__device__ __forceinline__ bool col_line(const ColArgs& a, int tile, int l, int64_t& base) {
  constexpr int o2 = DIR == 2 ? 1 : 2;
  const int nx = a.g.N[0] + 1, n2 = a.g.N[o2] + 1;
  int x, y;
  bool valid;
  if (a.flat) {
    const unsigned id = (unsigned)tile * LW + l;
    y = (int)(id / (unsigned)nx);
    x = (int)id - y * nx;
    valid = y < n2;
    if (!valid) x = y = 0;
  } else {
    y = tile / a.ntx;
    x = (tile - y * a.ntx) * LW + l;
    valid = x < nx;
    if (!valid) x = nx - 1;
  }
  base = x + (int64_t)y * a.g.st[o2];
  return valid;
}

// Window of the line's nodes b..b+W-1, periodic. RO: the field is not written by this kernel.
template <int W, bool RO>
__device__ __forceinline__ void line_window(double* w, const double* f, int b, int dim, int64_t sd) {
  if (b >= 0 && b + W - 1 <= dim) {
    const double* p = f + (int64_t)b * sd;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      w[i] = RO ? __ldg(p) : *p;
      p += sd;
    }
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const double* p = f + (int64_t)wrap_node(b + i, dim) * sd;
      w[i] = RO ? __ldg(p) : *p;
    }
  }
}

// Whether slot t of chunk c is a node of the box: not left over, not one of the three rows before node
// 0 or past node N. Two of the three conditions hold for most t at compile time.
template <int S>
__device__ __forceinline__ bool is_node(int t, int c, int nch, int nv) {
  return t < nv && (t >= 3 || c != 0) && (t < S - 3 || c != nch - 1);
}
template <int S>
__device__ __forceinline__ void store_rows(double* dst, const double (&v)[S], int c, int nch, int nv, int64_t sd) {
#pragma unroll
  for (int t = 0; t < S; ++t) {
    if (is_node<S>(t, c, nch, nv)) *dst = v[t];
    dst += sd;
  }
}

// ------------------------------------------------------------------ filter, in place (filterq)
template <int S, int LW, int DIR>
__device__ __forceinline__ void col_filter_body(const ColArgs& a, const ColConst<S>& kf, int blk, double* sm) {
  const int m = blk % 5, tile = blk / 5;
  const int l = threadIdx.x % LW, c = col_chunk(a.of, threadIdx.x / LW), dim = a.g.N[DIR], nch = a.of.nch;
  const bool act = c < nch;
  int64_t base;
  const bool valid = col_line<DIR, LW>(a, tile, l, base);
  double* f = a.q + m * a.g.fs + base;
  const int64_t sd = a.g.st[DIR];
  const int n0 = col_node<S>(a.of, c);
  double v[S];
  if (act) {
    double w[S + 10];
    line_window<S + 10, false>(w, f, n0 - 5, dim, sd);
    col_rhs_filter<S, false>(v, w, a.wf, a, c, nch);
    col_zero_ragged<S>(v, a.of, c);
  }
  col_solve<S, LW>(v, a.of, kf, c, l, act, sm, sm + nch * LW);
  if (act && valid) store_rows<S>(f + (int64_t)n0 * sd, v, c, nch, col_rows<S>(a.of, c), sd);
}

// The derivative of the chunk's rows of a field.
template <int S, int LW, int DIR>
__device__ __forceinline__ void deriv_rows(double (&v)[S], const ColArgs& a, const ColConst<S>& kd, const double* f, int c,
                                          int l, bool act, double* sm) {
  if (act) {
    double w[S + 6];
    w[0] = w[S + 5] = 0.0;
    line_window<S + 4, true>(w + 1, f, col_node<S>(a.od, c) - 2, a.g.N[DIR], a.g.st[DIR]);
    col_rhs_deriv<S, 2>(v, w, a.wd, c, a.od.nch, false, false);
    col_zero_ragged<S>(v, a.od, c);
  }
  col_solve<S, LW>(v, a.od, kd, c, l, act, sm, sm + a.od.nch * LW);
}

// ------------------------------------------------------------------ gradients (gradcal)
// D_k = d(u, v, w, T)_k / dx_DIR of the primitive fields that k_prims has stored.
template <int S, int LW, int DIR>
__device__ __forceinline__ void col_grad_body(const ColArgs& a, const ColConst<S>& kd, int blk, double* sm) {
  const int m = blk & 3, tile = blk >> 2;
  const int l = threadIdx.x % LW, c = col_chunk(a.od, threadIdx.x / LW);
  const bool act = c < a.od.nch;
  int64_t base;
  const bool valid = col_line<DIR, LW>(a, tile, l, base);
  double v[S];
  deriv_rows<S, LW, DIR>(v, a, kd, a.G + m * a.g.fs + base, c, l, act, sm);
  if (act && valid)
    store_rows<S>(a.D + m * a.g.fs + base + col_node<S>(a.od, c) * a.g.st[DIR], v, c, a.od.nch, col_rows<S>(a.od, c),
                  a.g.st[DIR]);
}

// ------------------------------------------------------------------ R += D(G)
template <int S, int LW, int DIR>
__device__ __forceinline__ void col_div_body(const ColArgs& a, const ColConst<S>& kd, int blk, double* sm) {
  const int m = blk % 5, tile = blk / 5;
  const int l = threadIdx.x % LW, c = col_chunk(a.od, threadIdx.x / LW), nch = a.od.nch;
  const bool act = c < nch;
  int64_t base;
  const bool valid = col_line<DIR, LW>(a, tile, l, base);
  double v[S];
  deriv_rows<S, LW, DIR>(v, a, kd, a.G + m * a.g.fs + base, c, l, act, sm);
  if (!act || !valid) return;
  const int n0 = col_node<S>(a.od, c), nv = col_rows<S>(a.od, c);
  const int64_t sd = a.g.st[DIR];
  double* R = a.R + m * a.g.fs + base + (int64_t)n0 * sd;
  constexpr int NB = 17;   // rows whose loads are in flight together
#pragma unroll
  for (int t0 = 0; t0 < S; t0 += NB) {
    double r[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (t0 + j < S) {
        const int t = t0 + j;
        r[j] = is_node<S>(t, c, nch, nv) ? R[(int64_t)t * sd] : 0.0;
      }
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (t0 + j < S) {
        const int t = t0 + j;
        if (is_node<S>(t, c, nch, nv)) R[(int64_t)t * sd] = r[j] + v[t];
      }
  }
}

// ------------------------------------------------------------------ flux, update, filter
// q_out = F(c1 qsave + c2 q + c3 dt (R + D(G))): the updated nodes pass through a shared-memory tile
// (with their periodic images) to reach the windows of the neighbouring chunks.
template <int S, int LW, int DIR>
__device__ __forceinline__ void col_update_body(const ColArgs& a, const ColConst<S>& kd, const ColConst<S>& kf, int blk,
                                                double* sm) {
  const int m = blk % 5, tile = blk / 5;
  const int l = threadIdx.x % LW, c = col_chunk(a.of, threadIdx.x / LW), dim = a.g.N[DIR], nch = a.od.nch;
  const bool act = c < nch;
  int64_t base;
  const bool valid = col_line<DIR, LW>(a, tile, l, base);
  const int64_t fo = m * a.g.fs + base, sd = a.g.st[DIR];
  double v[S];
  deriv_rows<S, LW, DIR>(v, a, kd, a.G + fo, c, l, act, sm);
  const int n0 = col_node<S>(a.od, c), nv = col_rows<S>(a.od, c);
  double* line = sm + 2 * nch * LW + COL_IMG * LW + l;   // node n at line[n * LW]
  if (act) {
    const double c1 = a.c1, c2 = a.c2, c3 = a.c3, dt = a.pdt ? __ldg(a.pdt) : a.dt;
    // one predicated form for all chunks: a second one for whole chunks takes the kernel's code past the
    // instruction cache (512^3: 7.5 -> 9.9 ms; with range tests per row instead of is_node 5.9 -> 7.5)
    const int64_t o0 = fo + (int64_t)n0 * sd;
    const double *R = a.R + o0, *qs = a.qsave + o0, *qq = a.q + o0;
    constexpr int NB = 7;   // rows whose loads are in flight together
#pragma unroll
    for (int t0 = 0; t0 < S; t0 += NB) {
      double r[NB], s[NB], x[NB];
#pragma unroll
      for (int j = 0; j < NB; ++j)
        if (t0 + j < S) {
          const int t = t0 + j;
          const bool in = is_node<S>(t, c, nch, nv);
          const int64_t off = (int64_t)t * sd;
          r[j] = in ? R[off] : 0.0;
          s[j] = in ? qs[off] : 0.0;
          x[j] = (in && c2 != 0.0) ? qq[off] : 0.0;
        }
#pragma unroll
      for (int j = 0; j < NB; ++j)
        if (t0 + j < S) {
          const int t = t0 + j;
          const double rhs = r[j] + v[t];
          // (c1 qsave + c2 q) + (c3 qrhs) dt in the reference's order (rk3, tgvsolver.F90:1055-1057),
          // rounded at every step so that the result does not depend on how it is contracted
          const double qc = (c2 != 0.0) ? __dmul_rn(c2, x[j]) : 0.0;
          const double qn = __dadd_rn(__dadd_rn(__dmul_rn(c1, s[j]), qc), __dmul_rn(__dmul_rn(c3, rhs), dt));
          v[t] = qn;
          if (a.do_filter && is_node<S>(t, c, nch, nv)) line[(n0 + t) * LW] = qn;
        }
    }
    if (a.do_filter) {   // periodic images of nodes 1..5 and N-5..N-1, at fixed slots of the end chunks
#pragma unroll
      for (int k = 1; k <= 5; ++k) {
        if (c == 0) line[(dim + k) * LW] = v[3 + k];
        if (c == nch - 1) line[-k * LW] = v[S - 4 - k];
      }
    }
  }
  if (a.do_filter) {
    __syncthreads();
    if (act) {
      double w[S + 10];
      const double* wl = line + (n0 - 5) * LW;   // nodes -8..N+8; the outer three on each side are not used
#pragma unroll
      for (int i = 0; i < S + 10; ++i) w[i] = wl[i * LW];
      col_rhs_filter<S, false>(v, w, a.wf, a, c, nch);
      col_zero_ragged<S>(v, a.of, c);
    }
    col_solve<S, LW>(v, a.of, kf, c, l, act, sm, sm + nch * LW);
  }
  if (act && valid) store_rows<S>(a.qout + fo + (int64_t)n0 * sd, v, c, nch, nv, sd);
}

template <int PASS, int S, int LW, int DIR>
__device__ __forceinline__ void col_body(const ColArgs& a, const ColConst<S>& kd, const ColConst<S>& kf, int blk, double* sm) {
  if constexpr (PASS == COL_FILTER) col_filter_body<S, LW, DIR>(a, kf, blk, sm);
  else if constexpr (PASS == COL_GRAD) col_grad_body<S, LW, DIR>(a, kd, blk, sm);
  else if constexpr (PASS == COL_DIV) col_div_body<S, LW, DIR>(a, kd, blk, sm);
  else col_update_body<S, LW, DIR>(a, kd, kf, blk, sm);
}

template <int PASS, int S, int LW, int DIR>
__global__ void __launch_bounds__(512) k_col(const __grid_constant__ ColArgs a, const __grid_constant__ ColConst<S> kd,
                                             const __grid_constant__ ColConst<S> kf) {
  extern __shared__ double sm[];
  col_body<PASS, S, LW, DIR>(a, kd, kf, blockIdx.x, sm);
}

// u, v, w, T of every node (q2fvar, tgvsolver.F90:92-121) into four fields, one division per node:
// once for the gradients along y and z, which then are plain derivatives of one field each.
__global__ void __launch_bounds__(256) k_prims(const double* __restrict__ q, double* __restrict__ U, int64_t n2, int64_t fs,
                                               Thermo th) {
  const int64_t p = blockIdx.x * (int64_t)256 + threadIdx.x;   // node pairs: rows are padded to whole lines
  if (p >= n2) return;
  double2 x[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) x[m] = __ldg(reinterpret_cast<const double2*>(q + m * fs) + p);
  auto prim = [&](double r, double qu, double qv, double qw, double e, double& u, double& v, double& w, double& t) {
    const double ri = 1.0 / r;
    u = qu * ri;
    v = qv * ri;
    w = qw * ri;
    t = (e - 0.5 * r * (u * u + v * v + w * w)) * th.gm1 * ri * th.const2;
  };
  double2 u, v, w, t;
  prim(x[0].x, x[1].x, x[2].x, x[3].x, x[4].x, u.x, v.x, w.x, t.x);
  prim(x[0].y, x[1].y, x[2].y, x[3].y, x[4].y, u.y, v.y, w.y, t.y);
  reinterpret_cast<double2*>(U)[p] = u;
  reinterpret_cast<double2*>(U + fs)[p] = v;
  reinterpret_cast<double2*>(U + 2 * fs)[p] = w;
  reinterpret_cast<double2*>(U + 3 * fs)[p] = t;
}

}  // namespace col_detail
}  // namespace astr
