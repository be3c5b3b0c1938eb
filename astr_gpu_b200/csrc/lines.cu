// Line-level operators over arbitrary Fortran-ordered arrays: the drop-in for
//   df = fds%central(asolver, f, dim)      src/derivative.F90:22-41, 171-198
//   ff = compact_filter(afilter, f, dim)   src/filter.F90:112-144
//   fh = flux_compact(asolver, f, dim)     src/flux.F90:125-150 (interfaces -1..dim)
// applied to every line of a 3-D array along one direction; the interface flux can also leave
// its differences fh(i) - fh(i-1) at the nodes (the flux-form derivative of convrsdcmp,
// src/solver.F90:1509-1513, and of the reference's flux test, src/test.F90:755-765).
//
// One CTA takes LW lines of one field, one thread per line and chunk of S rows (colsolve.cuh).
// y and z lines: the LW lines are adjacent in x, so each row is one piece of LW * 8 bytes that goes
// from HBM into the registers of LW threads; nothing is staged. x lines: the lines are copied to a
// shared-memory tile with asynchronous copies (node-fastest), each thread reads its chunk's window
// from its line, and results go back through the tile for coalesced stores. 16 lines with an odd
// pitch, or from 33 rows per chunk on 8 lines with a pitch of 2 mod 16: either way a half warp hits
// 16 different bank pairs.
#include "internal.h"

namespace astr {

namespace {

__device__ __forceinline__ void cp8(double* sdst, const double* gsrc) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp16(double* sdst, const double* gsrc) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

constexpr int HL = 5;   // halo nodes of a line that an operator reads

// The chunk's window of W nodes from node b, zeros outside nodes lo..hi.
template <int W>
__device__ __forceinline__ void window(double (&w)[W], const double* src, int64_t sd, int b, int lo, int hi) {
  const double* p = src + (int64_t)b * sd;
  if (b >= lo && b + W - 1 <= hi) {
#pragma unroll
    for (int i = 0; i < W; ++i) { w[i] = *p; p += sd; }
  } else {
#pragma unroll
    for (int i = 0; i < W; ++i) {
      w[i] = (b + i >= lo && b + i <= hi) ? *p : 0.0;
      p += sd;
    }
  }
}

template <int S, int KIND>
__device__ __forceinline__ void line_rhs(double (&v)[S], const double (&w)[S + Win<KIND>::EXTRA], const ColWeights& k,
                                         const LineOp& op, const ColOp& co, int c) {
  if constexpr (KIND == OP_DERIV) col_rhs_deriv<S>(v, w, k, c, co.nch, op.left_phys, op.right_phys);
  else if constexpr (KIND == OP_EXPLICIT) col_explicit<S>(v, w, c, co.nch, op.left_phys, op.right_phys);
  else if constexpr (KIND == OP_FILTER) col_rhs_filter<S>(v, w, k, op, c, co.nch);
  else col_rhs_flux<S>(v, w, k, op, c, co.nch);
  col_zero_ragged<S>(v, co, c);
}

struct LineArgs {
  const double* f;
  double* out;
  ArrDesc fa, oa;
  int dir, flags;
  double scale;
  ColWeights k;
};

}  // namespace

// y and z lines. Registers bound it: the window of S + 10 doubles (filter) is the largest live set.
template <int S, int KIND, int LW>
__global__ void __launch_bounds__(S >= 17 ? 512 : 256, S >= 17 ? 1 : 2)
    k_line_col(LineOp op, ColOp co, ColConst<S> k, LineArgs a) {
  extern __shared__ double sm[];
  double* exf = sm;
  double* exb = sm + co.nch * LW;
  const int dir = a.dir, o2 = dir == 2 ? 1 : 2;
  const int l = threadIdx.x % LW, c = col_chunk(co, threadIdx.x / LW);
  // the line: tiles of LW lines along x per index of the third axis, or (blockIdx.y unused) of LW
  // consecutive lines of the flattened (x, third axis) plane
  int64_t x1 = (int64_t)blockIdx.x * LW + l, x2 = blockIdx.y;
  bool valid;
  if (gridDim.y == 1) {
    const unsigned nx = (unsigned)a.oa.n[0], q = (unsigned)x1 / nx;
    valid = q < (dir == 2 ? a.oa.n[1] : a.oa.n[2]);
    x1 -= (int64_t)q * nx;
    x2 = q;
    if (!valid) x1 = x2 = 0;
  } else {
    valid = x1 < a.oa.n[0];
    if (!valid) x1 = a.oa.n[0] - 1;   // lines past the edge repeat the last one (never stored)
  }
  const int64_t i1 = a.oa.lb[0] + x1, i2 = a.oa.lb[o2] + x2;
  const bool act = c < co.nch;
  const int dim = op.dim;
  constexpr int W = S + Win<KIND>::EXTRA;
  const int n0 = col_node<S>(co, c), nv = col_rows<S>(co, c);
  double v[S], keep = 0.0;
  if (act) {
    const int64_t fd = dir == 1 ? a.fa.s[1] : a.fa.s[2], fo = dir == 1 ? a.fa.s[2] : a.fa.s[1];
    const int64_t fl = dir == 1 ? a.fa.lb[1] : a.fa.lb[2], fn = dir == 1 ? a.fa.n[1] : a.fa.n[2];
    const int64_t flo = dir == 1 ? a.fa.lb[2] : a.fa.lb[1];
    const double* src = a.f + (int64_t)blockIdx.z * a.fa.fs + (i2 - flo) * fo + (i1 - a.fa.lb[0]) - fl * fd;
    const int lo = (int)max((int64_t)-HL, fl), hi = (int)min((int64_t)(dim + HL), fl + fn - 1);
    double w[W];
    window<W>(w, src, fd, n0 - Win<KIND>::LO, lo, hi);
    // physical-boundary reset ff(0)=f(0), ff(dim)=f(dim) of compact_filter (filter.F90:141-142)
    if (KIND == OP_FILTER) keep = c == 0 ? w[5] : w[S + 4];
    line_rhs<S, KIND>(v, w, a.k, op, co, c);
  }
  if (KIND == OP_EXPLICIT) __syncthreads();   // every window is read before the first store
  else col_solve<S, LW>(v, co, k, c, l, act, exf, exb);
  // outputs: nodes 0..dim, or the interfaces -1..dim of the flux (their differences with LINE_DIFF)
  const bool diff = KIND == OP_FLUX && (a.flags & LINE_DIFF);
  const int out_lo = (KIND == OP_FLUX && !diff) ? -1 : 0;
  if (diff) {
    // the interface before the chunk's first row: the last row of the chunk before (exf is free:
    // every thread read it before the solve's second barrier)
    if (act) {
      double last = v[0];
#pragma unroll
      for (int t = 1; t < S; ++t) last = t < nv ? v[t] : last;
      exf[c * LW + l] = last;
    }
    __syncthreads();
    if (act) {
      double prev = 0.0;
      if (c > 0) prev = (c == 2 && co.nv == 0) ? exf[l] : exf[(c - 1) * LW + l];
#pragma unroll
      for (int t = 0; t < S; ++t) {
        const double x = v[t];
        v[t] = x - prev;
        prev = x;
      }
    }
  }
  if (!act || !valid) return;
  const int64_t od = dir == 1 ? a.oa.s[1] : a.oa.s[2], oo = dir == 1 ? a.oa.s[2] : a.oa.s[1];
  const int64_t ol = dir == 1 ? a.oa.lb[1] : a.oa.lb[2];
  double* dst = a.out + (int64_t)blockIdx.z * a.oa.fs + (i2 - a.oa.lb[o2]) * oo + (i1 - a.oa.lb[0]) + (n0 - ol) * od;
  auto res = [&](double x) { return KIND == OP_FILTER ? x : a.scale * x; };
  if (KIND == OP_FILTER) {
    if (c == 0 && op.left_phys) v[0] = keep;
    if (c == co.nch - 1 && op.right_phys) v[S - 1] = keep;
  }
  if (a.flags & LINE_ADD) {
#pragma unroll
    for (int t0 = 0; t0 < S; t0 += 11) {   // loads of 11 rows in flight
      double old[11];
#pragma unroll
      for (int j = 0; j < 11; ++j)
        if (t0 + j < S) {
          const int n = n0 + t0 + j;
          old[j] = (t0 + j < nv && n >= out_lo && n <= dim) ? dst[(int64_t)(t0 + j) * od] : 0.0;
        }
#pragma unroll
      for (int j = 0; j < 11; ++j)
        if (t0 + j < S) {
          const int n = n0 + t0 + j;
          if (t0 + j < nv && n >= out_lo && n <= dim) dst[(int64_t)(t0 + j) * od] = old[j] + res(v[t0 + j]);
        }
    }
  } else if (nv == S && n0 >= out_lo && n0 + S - 1 <= dim) {
#pragma unroll
    for (int t = 0; t < S; ++t) { *dst = res(v[t]); dst += od; }
  } else {
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const int n = n0 + t;
      if (t < nv && n >= out_lo && n <= dim) *dst = res(v[t]);
      dst += od;
    }
  }
}

// x lines, through a tile of LW lines with nodes -HL..dim+HL (pitch LP).
template <int S, int KIND, int LW>
__global__ void __launch_bounds__(S >= 17 ? 512 : 320, S >= 17 ? 1 : 2)
    k_line_row(LineOp op, ColOp co, ColConst<S> k, LineArgs a, int LP) {
  extern __shared__ double sm[];
  double* exf = sm;
  double* exb = exf + co.nch * LW;
  double* tile = exb + co.nch * LW;
  const int dim = op.dim;
  const int64_t i2 = a.oa.lb[2] + blockIdx.y;
  const int64_t i1_0 = a.oa.lb[1] + (int64_t)blockIdx.x * LW;
  const int nl = (int)min((int64_t)LW, a.oa.lb[1] + a.oa.n[1] - i1_0);
  const int lo = (int)max((int64_t)-HL, a.fa.lb[0]), hi = (int)min((int64_t)(dim + HL), a.fa.lb[0] + a.fa.n[0] - 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const double* src0 = a.f + (int64_t)blockIdx.z * a.fa.fs + (i2 - a.fa.lb[2]) * a.fa.s[2] + (i1_0 - a.fa.lb[1]) * a.fa.s[1] - a.fa.lb[0];
  for (int r = warp; r < LW; r += nwarp) {
    double* row = tile + r * LP + HL;
    if (r >= nl) {
      for (int n = -HL + lane; n <= dim + HL; n += 32) row[n] = 0.0;
      continue;
    }
    const double* src = src0 + r * a.fa.s[1];
    for (int n = -HL + lane; n < lo; n += 32) row[n] = 0.0;
    for (int n = hi + 1 + lane; n <= dim + HL; n += 32) row[n] = 0.0;
    int first = lo;
    if ((((uintptr_t)(src + lo) ^ (uintptr_t)(row + lo)) & 15u) == 0) {   // node pairs share the phase
      if (((uintptr_t)(row + lo) & 15u) != 0) {
        if (lane == 0) cp8(row + lo, src + lo);
        ++first;
      }
      const int np = (hi - first + 1) >> 1;
      for (int p = lane; p < np; p += 32) cp16(row + first + 2 * p, src + first + 2 * p);
      first += 2 * np;
    }
    for (int n = first + lane; n <= hi; n += 32) cp8(row + n, src + n);
  }
  cp_wait_all();
  __syncthreads();
  const int l = threadIdx.x % LW, c = col_chunk(co, threadIdx.x / LW);
  const bool act = c < co.nch;
  constexpr int W = S + Win<KIND>::EXTRA;
  const int n0 = col_node<S>(co, c);
  double* line = tile + l * LP + HL;
  double v[S], keep = 0.0;
  if (act) {
    double w[W];
    window<W>(w, line, 1, n0 - Win<KIND>::LO, -HL, dim + HL);
    if (KIND == OP_FILTER) keep = c == 0 ? w[5] : w[S + 4];
    line_rhs<S, KIND>(v, w, a.k, op, co, c);
  }
  if (KIND == OP_EXPLICIT) __syncthreads();   // every window is read before the first store
  else col_solve<S, LW>(v, co, k, c, l, act, exf, exb);
  // the barriers of the solve lie between every thread's window reads and these writes
  const bool diff = KIND == OP_FLUX && (a.flags & LINE_DIFF);
  const int out_lo = KIND == OP_FLUX ? -1 : 0;
  const int nv = col_rows<S>(co, c);
  if (act) {
    if (KIND == OP_FILTER) {
      if (c == 0 && op.left_phys) v[0] = keep;
      if (c == co.nch - 1 && op.right_phys) v[S - 1] = keep;
    }
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const int n = n0 + t;
      if (t < nv && n >= out_lo && n <= dim) line[n] = v[t];
    }
  }
  __syncthreads();
  const double sc = KIND == OP_FILTER ? 1.0 : a.scale;
  const bool add = a.flags & LINE_ADD;
  double* dst0 = a.out + (int64_t)blockIdx.z * a.oa.fs + (i2 - a.oa.lb[2]) * a.oa.s[2] + (i1_0 - a.oa.lb[1]) * a.oa.s[1] - a.oa.lb[0];
  for (int r = warp; r < nl; r += nwarp) {
    const double* row = tile + r * LP + HL;
    double* dst = dst0 + r * a.oa.s[1];
    if (diff) {
#pragma unroll 4
      for (int n = lane; n <= dim; n += 32) {
        const double d = sc * (row[n] - row[n - 1]);
        dst[n] = add ? dst[n] + d : d;
      }
    } else if (add) {
#pragma unroll 4
      for (int n = out_lo + lane; n <= dim; n += 32) dst[n] += sc * row[n];
    } else {
#pragma unroll 4
      for (int n = out_lo + lane; n <= dim; n += 32) dst[n] = sc * row[n];
    }
  }
}

template <int S, int KIND, int LW>
static cudaError_t launch_col(const DevColOp& op, const LineArgs& a, int nfields, cudaStream_t st) {
  const int threads = (op.op.nch * LW + 31) / 32 * 32;
  const size_t smem = (size_t)2 * op.op.nch * LW * sizeof(double);
  const int64_t n1 = a.oa.n[0], n2 = a.oa.n[a.dir == 2 ? 1 : 2];
  // tiles along x waste the lanes past the edge of every row; flattened tiles (rows that wrap to the
  // next index of the third axis, unaligned pieces) take over where that is more than a tenth
  const int64_t nx = (n1 + LW - 1) / LW;
  const bool flat = 10 * nx * LW > 11 * n1 && n1 * n2 < (int64_t(1) << 31);
  const dim3 grid((unsigned)(flat ? (n1 * n2 + LW - 1) / LW : nx), (unsigned)(flat ? 1 : n2), (unsigned)nfields);
  k_line_col<S, KIND, LW><<<grid, threads, smem, st>>>(op.line, op.op, op.consts<S>(), a);
  return cudaGetLastError();
}

template <int S, int KIND>
static cudaError_t launch_sk(const DevColOp& op, const LineArgs& a, int nfields, cudaStream_t st) {
  if (a.dir != 0) {
    // 32 lines per CTA up to eight chunks, 16 beyond: two CTAs of 128 registers fit on an SM
    if constexpr (S < 37) {   // 37 rows: 29 chunks or more
      if (op.op.nch <= 8) return launch_col<S, KIND, 32>(op, a, nfields, st);
    }
    if constexpr (S >= 33) return launch_col<S, KIND, 16>(op, a, nfields, st);
    return cudaErrorInvalidValue;
  }
  // long chunks: 8 lines with a pitch of 2 mod 16 (a half warp is 8 lines on the even bank pairs and the
  // next chunk, an odd number of rows away, on the odd ones), several small CTAs per SM; else 16 lines
  // with an odd pitch. GB/s with 16 / 8 lines: derivative 512 nodes 3715 / 3919, filter 512 nodes 3362 /
  // 3514, 1050 nodes 2314 / 2726, 256 nodes 3339 / 3395
  constexpr int LW = S >= 33 ? 8 : 16;
  const int threads = (op.op.nch * LW + 31) / 32 * 32;
  const dim3 grid((unsigned)((a.oa.n[1] + LW - 1) / LW), (unsigned)a.oa.n[2], (unsigned)nfields);
  const int need = op.line.dim + 1 + 2 * HL;
  const int LP = LW == 8 ? need + (18 - need % 16) % 16 : need | 1;
  const size_t smem = ((size_t)2 * op.op.nch * LW + (size_t)LW * LP) * sizeof(double);
  auto kern = k_line_row<S, KIND, LW>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, smem, st>>>(op.line, op.op, op.consts<S>(), a, LP);
  return cudaGetLastError();
}

template <int S>
static cudaError_t launch_s(const DevColOp& op, const LineArgs& a, int nfields, cudaStream_t st) {
  if (op.line.kind == OP_DERIV) return launch_sk<S, OP_DERIV>(op, a, nfields, st);
  if (op.line.kind == OP_EXPLICIT) return launch_sk<S, OP_EXPLICIT>(op, a, nfields, st);
  if (op.line.kind == OP_FLUX) return launch_sk<S, OP_FLUX>(op, a, nfields, st);
  if constexpr (S >= 5) return launch_sk<S, OP_FILTER>(op, a, nfields, st);   // five closure rows at a wall
  return cudaErrorInvalidValue;
}

cudaError_t launch_line_api(const DevColOp& op, int dir, const double* f, const ArrDesc& fa, double* out,
                            const ArrDesc& oa, int nfields, double scale, cudaStream_t st, int flags) {
  const LineArgs a{f, out, fa, oa, dir, flags, scale, col_weights(op, 1.0)};
  switch (op.S) {
    case 3: return launch_s<3>(op, a, nfields, st);
    case 5: return launch_s<5>(op, a, nfields, st);
    case 9: return launch_s<9>(op, a, nfields, st);
    case 17: return launch_s<17>(op, a, nfields, st);
    case 33: return launch_s<33>(op, a, nfields, st);
    case 37: return launch_s<37>(op, a, nfields, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace astr
