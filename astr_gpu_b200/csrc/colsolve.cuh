// The column solve: a line's tridiagonal system cut into chunks of S consecutive rows, one thread
// per (line, chunk), LW adjacent lines per CTA (thread = chunk * LW + line). A warp holds the same
// rows of 32 neighbouring lines (or two chunks of 16), so
//  * y and z lines go from HBM straight into registers, 256 (128) contiguous bytes per row, and
//    back, with no staging in shared memory;
//  * the row coefficients are the same for all lines of a chunk. The factors of the tridiagonal
//    system converge after a few rows, so all chunks but the first few and the last share one
//    set of coefficients, which are kernel parameters (operands from the constant bank, no loads);
//  * the recurrences of a chunk are serial in a thread and need no shuffles: the carries between
//    chunks are one value per line and chunk in shared memory, which each thread combines itself
//    (Horner over the chunks before it). Two CTA barriers per solve.
// The lane-scan solve of ops.cuh spends a shuffle scan, a table load per row and two shared-memory
// passes per row on the same system (1 row/clock/SM measured, whatever the layout).
//
// Rows: the system's nsys rows fill nch chunks of S slots. The slots left over are the last ones of
// chunk 1 (it holds nv rows), so the first row is slot 0 of chunk 0, the last row slot S-1 of the
// last chunk, and closure rows sit at fixed slots (register indices known at compile time). A
// left-over slot passes both recurrences' carries on unchanged (ac2 = 0, ac3 = -1, ac1 = -1, its
// forward value replaced by zero before the backward sweep).
//
// The chunks whose coefficients differ from the converged set (the first c_lo and the last one) read
// them from a table. They come first in the thread order (col_chunk), an even number of them where
// there are others, so that with 16 lines per CTA no warp holds one chunk of each kind and runs both
// forms of the sweeps.
#pragma once
#include "ops.cuh"

namespace astr {

// Converged coefficients: forward y = d - y*k3 (the right-hand side carries the factor ac2, see
// ColWeights), backward x = y - k1*x, and the products that carry a chunk's incoming values to its
// rows, pf[t] = (-k3)^(t+1), qb[t] = (-k1)^(S-t).
template <int S>
struct ColConst {
  double k3, k1;
  double pf[S], qb[S];
};

// Right-hand side weights times ks = (converged ac2) * (output scale); closure rows are multiplied by
// ks. w: derivative 7/9, 1/36; filter 2 c0, c1..c5; interface flux its four weights.
struct ColWeights {
  double ks;
  double w[6];
};

// tab: (chunk*S + t)*6 + {ac2 / converged ac2, ac3, pf, ac1, qb, 0}, then the chunk products mf[nch]
// (of -ac3) and mb[nch] (of -ac1). Chunks c_lo..nch-2 have the coefficients of ColConst.
struct ColOp {
  const double* tab;
  int nch, nv, n_first, c_lo;
};

// Chunk of the p-th group of LW threads.
__device__ __forceinline__ int col_chunk(const ColOp& op, int p) {
  return p < op.c_lo || p >= op.nch ? p : (p == op.c_lo ? op.nch - 1 : p - 1);
}
// Node of slot 0 of chunk c.
template <int S>
__device__ __forceinline__ int col_node(const ColOp& op, int c) {
  return op.n_first + c * S - (c > 1 ? S - op.nv : 0);
}
// Number of rows in chunk c (the remaining slots are left over).
template <int S>
__device__ __forceinline__ int col_rows(const ColOp& op, int c) {
  return c == 1 ? op.nv : S;
}

// Solve the chunk's rows: v holds the weighted right-hand sides on entry (zero in left-over slots) and
// the solution on exit. exf, exb: nch * LW doubles of shared memory each, not touched by anything
// else between the call's barriers. Every thread of the CTA calls it; `act` is false for threads
// past the last chunk.
template <int S, int LW>
__device__ __forceinline__ void col_solve(double (&v)[S], const ColOp& op, const ColConst<S>& k, int c, int l, bool act,
                                          double* exf, double* exb) {
  const bool cst = c >= op.c_lo && c < op.nch - 1;
  const double2* tb = reinterpret_cast<const double2*>(op.tab) + (size_t)c * S * 3;
  const double* mf = op.tab + (size_t)op.nch * S * 6;
  const double* mb = mf + op.nch;
  double g = 0.0;
  if (cst) {
#pragma unroll
    for (int t = 0; t < S; ++t) {
      g = fma(-k.k3, g, v[t]);
      v[t] = g;
    }
  } else if (act) {
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const double2 a = __ldg(tb + 3 * t);
      g = fma(-a.y, g, v[t] * a.x);
      v[t] = g;
    }
  }
  if (act) exf[c * LW + l] = g;
  __syncthreads();
  double cin = 0.0;
  if (act) {
    const int ct = min(c, op.c_lo);
    for (int j = 0; j < ct; ++j) cin = fma(__ldg(mf + j), cin, exf[j * LW + l]);
#pragma unroll 4
    for (int j = ct; j < c; ++j) cin = fma(k.pf[S - 1], cin, exf[j * LW + l]);
  }
  g = 0.0;
  if (cst) {
#pragma unroll
    for (int t = S - 1; t >= 0; --t) {
      g = fma(-k.k1, g, fma(k.pf[t], cin, v[t]));
      v[t] = g;
    }
  } else if (act) {
    const int nv = col_rows<S>(op, c);
#pragma unroll
    for (int t = S - 1; t >= 0; --t) {
      const double2 a = __ldg(tb + 3 * t + 1);
      const double y = t < nv ? fma(a.x, cin, v[t]) : 0.0;
      g = fma(-a.y, g, y);
      v[t] = g;
    }
  }
  if (act) exb[c * LW + l] = g;
  __syncthreads();
  if (act && c < op.nch - 1) {
    double cb = exb[(op.nch - 1) * LW + l];
    int j = op.nch - 2;
#pragma unroll 4
    for (; j > c && j >= op.c_lo; --j) cb = fma(k.qb[0], cb, exb[j * LW + l]);
    for (; j > c; --j) cb = fma(__ldg(mb + j), cb, exb[j * LW + l]);
    if (cst) {
#pragma unroll
      for (int t = 0; t < S; ++t) v[t] = fma(k.qb[t], cb, v[t]);
    } else {
#pragma unroll
      for (int t = 0; t < S; ++t) v[t] = fma(__ldg(op.tab + ((size_t)c * S + t) * 6 + 4), cb, v[t]);
    }
  }
}

// ---------------------------------------------------------------- right-hand sides
// Windows: w[i] = f(n0 - B + i) with n0 the node of slot 0 and B = WIN_LO of the operator kind.
// Interior rows first, then the closure rows of the first and the last chunk, whose slots and
// window positions are fixed (OFS: left-over rows before the first and after the last row, for an
// operator embedded in a longer system).
template <int KIND>
struct Win {};
template <>
struct Win<OP_DERIV> { static constexpr int LO = 3, EXTRA = 6; };    // the closure rows reach 3 nodes
template <>
struct Win<OP_EXPLICIT> { static constexpr int LO = 3, EXTRA = 6; };
template <>
struct Win<OP_FILTER> { static constexpr int LO = 5, EXTRA = 10; };
template <>
struct Win<OP_FLUX> { static constexpr int LO = 2, EXTRA = 5; };     // interface rows: f(j-2)..f(j+3)

template <int S, int OFS = 0>
__device__ __forceinline__ void col_rhs_deriv(double (&v)[S], const double (&w)[S + 6], const ColWeights& k, int c, int nch,
                                              bool left_phys, bool right_phys) {
#pragma unroll
  for (int t = 0; t < S; ++t) v[t] = k.w[0] * (w[t + 4] - w[t + 2]) + k.w[1] * (w[t + 5] - w[t + 1]);
  auto six = [&](int i) { return k.ks * (0.75 * (w[i + 1] - w[i - 1]) - 0.15 * (w[i + 2] - w[i - 2]) + (1.0 / 60.0) * (w[i + 3] - w[i - 3])); };
  if (c == 0) {
#pragma unroll
    for (int t = 0; t < OFS; ++t) v[t] = 0.0;
    constexpr int i = 3 + OFS;   // window position of the first row's node
    if (left_phys) {
      v[OFS] = k.ks * (-2.5 * w[i] + 2.0 * w[i + 1] + 0.5 * w[i + 2]);
      v[OFS + 1] = k.ks * (0.75 * (w[i + 2] - w[i]));
    } else {
      v[OFS] = six(i);
    }
  }
  if (c == nch - 1) {
#pragma unroll
    for (int t = 0; t < OFS; ++t) v[S - 1 - t] = 0.0;
    constexpr int i = S + 2 - OFS;
    if (right_phys) {
      v[S - 1 - OFS] = k.ks * (2.5 * w[i] - 2.0 * w[i - 1] - 0.5 * w[i - 2]);
      v[S - 2 - OFS] = k.ks * (0.75 * (w[i] - w[i - 2]));
    } else {
      v[S - 1 - OFS] = six(i);
    }
  }
}

// The explicit 6th-order derivative with its closures (diff6ec, derivative.F90:350-413): rows are
// nodes 0..dim, already the result.
template <int S>
__device__ __forceinline__ void col_explicit(double (&v)[S], const double (&w)[S + 6], int c, int nch, bool left_phys,
                                             bool right_phys) {
#pragma unroll
  for (int t = 0; t < S; ++t)
    v[t] = 0.75 * (w[t + 4] - w[t + 2]) - 0.15 * (w[t + 5] - w[t + 1]) + (1.0 / 60.0) * (w[t + 6] - w[t]);
  if (c == 0 && left_phys) {
    v[0] = -0.5 * w[5] + 2.0 * w[4] - 1.5 * w[3];
    v[1] = 0.5 * (w[5] - w[3]);
    v[2] = (2.0 / 3.0) * (w[6] - w[4]) - (1.0 / 12.0) * (w[7] - w[3]);
  }
  if (c == nch - 1 && right_phys) {
    v[S - 3] = (2.0 / 3.0) * (w[S + 1] - w[S - 1]) - (1.0 / 12.0) * (w[S + 2] - w[S - 2]);
    v[S - 2] = 0.5 * (w[S + 2] - w[S]);
    v[S - 1] = 0.5 * w[S] - 2.0 * w[S + 1] + 1.5 * w[S + 2];
  }
}

// WALLS = false: a periodic line (of op only ch is read).
template <int S, bool WALLS = true, class Op = LineOp>
__device__ __forceinline__ void col_rhs_filter(double (&v)[S], const double (&w)[S + 10], const ColWeights& k, const Op& op,
                                               int c, int nch) {
#pragma unroll
  for (int t = 0; t < S; ++t)
    v[t] = k.w[0] * w[t + 5] + k.w[1] * (w[t + 6] + w[t + 4]) + k.w[2] * (w[t + 7] + w[t + 3]) +
           k.w[3] * (w[t + 8] + w[t + 2]) + k.w[4] * (w[t + 9] + w[t + 1]) + k.w[5] * (w[t + 10] + w[t]);
  auto halo_lo = [&]() {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < 11; ++j) s += op.ch[r][j] * w[3 + j];
      v[r] = k.ks * s;
    }
  };
  auto halo_hi = [&]() {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < 11; ++j) s += op.ch[r][j] * w[S + 6 - j];
      v[S - 1 - r] = k.ks * s;
    }
  };
  if constexpr (!WALLS) {
    if (c == 0) halo_lo();
    if (c == nch - 1) halo_hi();
  } else {
    if (c == 0) {
      if (op.left_phys) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          double s = 0.0;
#pragma unroll
          for (int j = 0; j < 7; ++j) s += op.cb[r][j] * w[5 + j];
          v[r] = k.ks * s;
        }
        v[3] = k.ks * (op.c6[0] * (w[8] + w[8]) + op.c6[1] * (w[9] + w[7]) + op.c6[2] * (w[10] + w[6]) + op.c6[3] * (w[11] + w[5]));
        v[4] = k.ks * (op.c8[0] * (w[9] + w[9]) + op.c8[1] * (w[10] + w[8]) + op.c8[2] * (w[11] + w[7]) +
               op.c8[3] * (w[12] + w[6]) + op.c8[4] * (w[13] + w[5]));
      } else {
        halo_lo();
      }
      if (op.no_filter_note) v[0] = k.ks * w[5];
    }
    if (c == nch - 1) {
      if (op.right_phys) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          double s = 0.0;
#pragma unroll
          for (int j = 0; j < 7; ++j) s += op.cb[r][j] * w[S + 4 - j];
          v[S - 1 - r] = k.ks * s;
        }
        v[S - 4] = k.ks * (op.c6[0] * (w[S + 1] + w[S + 1]) + op.c6[1] * (w[S + 2] + w[S]) + op.c6[2] * (w[S + 3] + w[S - 1]) +
                   op.c6[3] * (w[S + 4] + w[S - 2]));
        v[S - 5] = k.ks * (op.c8[0] * (w[S] + w[S]) + op.c8[1] * (w[S + 1] + w[S - 1]) + op.c8[2] * (w[S + 2] + w[S - 2]) +
                   op.c8[3] * (w[S + 3] + w[S - 3]) + op.c8[4] * (w[S + 4] + w[S - 4]));
      } else {
        halo_hi();
      }
      if (op.no_filter_note) v[S - 1] = k.ks * w[S + 4];
    }
  }
}

// Interface flux rows (row j between nodes j and j + 1): w[i] = f(n0 - 2 + i).
template <int S>
__device__ __forceinline__ void col_rhs_flux(double (&v)[S], const double (&w)[S + 5], const ColWeights& k, const LineOp& op,
                                             int c, int nch) {
  if (op.wind > 0) {
#pragma unroll
    for (int t = 0; t < S; ++t) v[t] = k.w[0] * w[t + 1] + k.w[1] * w[t + 2] + k.w[2] * w[t + 3] + k.w[3] * w[t + 4];
  } else {
#pragma unroll
    for (int t = 0; t < S; ++t) v[t] = k.w[0] * w[t + 4] + k.w[1] * w[t + 3] + k.w[2] * w[t + 2] + k.w[3] * w[t + 1];
  }
  auto central = [&](int i) { return k.ks * ((37.0 / 60.0) * (w[i] + w[i + 1]) - (2.0 / 15.0) * (w[i - 1] + w[i + 2]) + (1.0 / 60.0) * (w[i - 2] + w[i + 3])); };
  if (c == 0) {
    if (op.left_phys) {
      v[0] = k.ks * (2.5 * w[3] + 0.5 * w[4]);
      v[1] = k.ks * (0.75 * w[3] + 0.75 * w[4]);
    } else {
      v[0] = central(2);
    }
  }
  if (c == nch - 1) {
    if (op.right_phys) {
      v[S - 1] = k.ks * (2.5 * w[S + 1] + 0.5 * w[S]);
      v[S - 2] = k.ks * (0.75 * w[S + 1] + 0.75 * w[S]);
    } else {
      v[S - 1] = central(S + 1);
    }
  }
}

// Zero the left-over slots of chunk 1.
template <int S>
__device__ __forceinline__ void col_zero_ragged(double (&v)[S], const ColOp& op, int c) {
  if (c == 1 && op.nv < S) {
#pragma unroll
    for (int t = 0; t < S; ++t)
      if (t >= op.nv) v[t] = 0.0;
  }
}

}  // namespace astr
