// The x passes of the RK3 step as column solves on shared-memory tiles (colsolve.cuh): the flux pass C
// and the filter along x.
//
// x lines are contiguous, so a CTA takes whole lines by bulk copies and any few lines make full-width
// accesses. Pass C keeps five primitive tiles and five gradient/flux tiles of NL lines; all gradient
// (then all flux) systems of the tile are solved at once, one thread per field, line and chunk of rows:
// two barriers for the four gradients and two for the five fluxes, where the lane-scan form took the
// systems of a line one or four at a time with a shuffle scan each. Two CTAs per SM overlap each
// other's copies, flux loop and solves.
//
// 512^3 on a B200, ms per launch (GB/s of the fields read and written): pass C 9.74 -> 7.6 (4000), the
// filter 2.98 -> 2.10 (5130). C is bound by latency: 16 warps per SM (128 registers, 85 KB of tiles)
// wait for the flux loop's loads (25 % of their cycles) and at the solves' barriers (23 %); the FP64 pipe
// is 20 % busy (256^3).
//
// Bank conflicts: a warp's lanes run over the lines, then the fields, then the chunks. With NL = 2 (and
// 8 lines in the filter) the pitch is 2 mod 16 doubles, so eight systems hit the even bank pairs and
// the next chunk, an odd number of rows away, the odd ones; with NL = 4 and 8 it is 1 mod 16.
#pragma once
#include "bulkcopy.cuh"
#include "tgv.cuh"

namespace astr {

constexpr int ROW_HX = 4;    // periodic images on each side of a gradient/flux line
constexpr int ROW_HF = 8;    // rows before node 0 in the filter's tile (5 periodic images)

struct RowArgs {
  BoxGeo g;
  Thermo th;
  ColOp op;
  ColWeights w;
  double ch[3][11];          // the filter's halo closure rows
  double* q;
  const double* DA;
  const double* DB;
  double* VF;
  double* R;
  double* DC;
  double* partials;
  int* err;
  int LT, LG;                // tile pitches: primitives; gradients and fluxes (filter: LG only)
};

namespace row_detail {

__device__ __forceinline__ double viscosity(const Thermo& th, double t) { return t * sqrt(t) * th.tc1 / (t + th.tc); }

// Values of NF fields (tiles gs apart) at node n of a line, with their periodic images.
template <int NF>
__device__ __forceinline__ void put(double* line, int gs, int n, int dim, const double (&v)[NF]) {
#pragma unroll
  for (int f = 0; f < NF; ++f) line[f * gs + n] = v[f];
  if (n <= ROW_HX || n >= dim - ROW_HX) {
    if (n >= 1 && n <= ROW_HX) {
#pragma unroll
      for (int f = 0; f < NF; ++f) line[f * gs + dim + n] = v[f];
    }
    if (n >= dim - ROW_HX && n < dim) {
#pragma unroll
      for (int f = 0; f < NF; ++f) line[f * gs + n - dim] = v[f];
    }
  }
}

// The derivatives of NF fields of the NL lines, in place in the tiles G.
template <int S, int NL, int NF>
__device__ __forceinline__ void solve_tiles(const RowArgs& a, const ColConst<S>& k, double* G, double* ex) {
  constexpr int LW = NL * NF;
  const int sys = threadIdx.x % LW, p = threadIdx.x / LW;
  const int c = col_chunk(a.op, p), nch = a.op.nch;
  const bool act = p < nch;
  double* line = G + sys * a.LG + ROW_HX;
  const int n0 = col_node<S>(a.op, c);
  double v[S];
  if (act) {
    double w[S + 6];
#pragma unroll
    for (int i = 0; i < S + 6; ++i) w[i] = line[n0 - 3 + i];
    col_rhs_deriv<S>(v, w, a.w, c, nch, false, false);
    col_zero_ragged<S>(v, a.op, c);
  }
  col_solve<S, LW>(v, a.op, k, c, sys, act, ex, ex + nch * LW);
  if (act) {
    const int nv = col_rows<S>(a.op, c);
#pragma unroll
    for (int t = 0; t < S; ++t)
      if (t < nv && (t >= 1 || c != 0) && (t < S - 1 || c != nch - 1)) line[n0 + t] = v[t];
  }
}

// The Euler flux along direction d (0, 1, 2) from the primitives (convection, tgvsolver.F90:559-564, q
// rebuilt by fvar2q); E is the total energy.
template <int D>
__device__ __forceinline__ void euler(double rho, double u, double v, double w, double p, double E, double (&F)[5]) {
  const double m = rho * (D == 0 ? u : (D == 1 ? v : w)), ud = D == 0 ? u : (D == 1 ? v : w);
  F[0] = m;
  F[1] = m * u;
  F[2] = m * v;
  F[3] = m * w;
  F[1 + D] += p;
  F[4] = (E + p) * ud;
}

// Pass C: gradients along x of (u, v, w, T); viscous stress and heat flux at every node (diffusion,
// tgvsolver.F90:635-694) with the gradients along y and z; the combined fluxes G = VF - F along y and
// z stored for the other passes; R = D_x(G_x). DIAG: with the diagnostics' partial sums (stacal,
// tgvsolver.F90:913-931; diss_rate_cal, statistic.F90:1009-1034).
template <int S, int NL, bool DIAG>
__global__ void __launch_bounds__(256, 2) k_row_c(const __grid_constant__ RowArgs a, const __grid_constant__ ColConst<S> k) {
  extern __shared__ __align__(16) double sm[];
  __shared__ uint64_t bar;
  __shared__ double red[3 * 8];
  constexpr int NT = 256, TPL = NT / NL;
  const int dim = a.g.N[0], LT = a.LT, LG = a.LG;
  double* T = sm;                       // primitive m of line l at (m * NL + l) * LT
  double* G = T + 5 * NL * LT;          // gradient / flux f of line l at (f * NL + l) * LG + ROW_HX
  double* ex = G + 5 * NL * LG + S + 8; // past the window overhang of the last line
  const int y0 = blockIdx.x * NL, z = blockIdx.y;
  const int nl = min(NL, a.g.N[1] + 1 - y0);
  const int64_t fs = a.g.fs, row0 = (int64_t)y0 * a.g.st[1] + (int64_t)z * a.g.st[2];
  const unsigned bytes = (unsigned)(((dim + 1) * 8 + 15) & ~15);   // within the padded row
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, bytes * 5u * (unsigned)nl);
  if (threadIdx.x < 32) {
    __syncwarp();
    for (int r = threadIdx.x; r < 5 * nl; r += 32) {
      const int m = r / nl, l = r - m * nl;
      bulk_g2s(T + (m * NL + l) * LT, a.q + m * fs + row0 + l * a.g.st[1], bytes, &bar);
    }
  } else if (threadIdx.x < 32 + 8 * NL) {   // the gradients along y and z start moving into L2
    const int r = threadIdx.x - 32, m = r / NL, l = r - m * NL;
    if (l < nl) {
      const double* src = (m < 4 ? a.DA + m * fs : a.DB + (m - 4) * fs) + row0 + l * a.g.st[1];
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
    }
  }
  if (nl < NL)   // lines past the box: finite filler for the solves, never stored
    for (int r = threadIdx.x; r < 5 * NL * LG; r += NT)
      if ((r / LG) % NL >= nl) G[r] = 0.0;
  mbar_wait_or_flag(&bar, a.err);
  const int l = threadIdx.x / TPL, j0 = threadIdx.x % TPL;
  const bool on = l < nl;
  double* Tl = T + l * LT;
  double* Gl = G + l * LG + ROW_HX;
  const int ts = NL * LT, gs = NL * LG;
  if (on) {
    // q -> (rho, u, v, w, p) (q2fvar, tgvsolver.F90:92-121), one division per node
#pragma unroll 2
    for (int n = j0; n <= dim; n += TPL) {
      const double r = Tl[n], ri = 1.0 / r;
      const double u = Tl[ts + n] * ri, v = Tl[2 * ts + n] * ri, w = Tl[3 * ts + n] * ri;
      const double p = (Tl[4 * ts + n] - 0.5 * r * (u * u + v * v + w * w)) * a.th.gm1;
      Tl[ts + n] = u;
      Tl[2 * ts + n] = v;
      Tl[3 * ts + n] = w;
      Tl[4 * ts + n] = p;
      const double x[4] = {u, v, w, p * ri * a.th.const2};
      put<4>(Gl, gs, n, dim, x);
    }
  }
  __syncthreads();
  solve_tiles<S, NL, 4>(a, k, G, ex);
  __syncthreads();
  const int64_t row = row0 + l * a.g.st[1];
  if (a.DC && on) {   // kept for the discrete adjoint
    for (int f = 0; f < 4; ++f)
      for (int n = j0; n <= dim; n += TPL) a.DC[f * fs + row + n] = Gl[f * gs + n];
  }
  double ke = 0.0, en = 0.0, di = 0.0;
  int bad = 0;
  if (on) {
    const double* DA = a.DA + row;
    const double* DB = a.DB + row;
    double* VF = a.VF + row;
    const bool counted = y0 + l >= 1 && z >= 1;
    constexpr int NB = 2;   // nodes whose 8 gradient loads are in flight together
    for (int nb = j0; nb <= dim; nb += NB * TPL) {
      double gy[NB][4], gz[NB][4];
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = min(nb + b * TPL, dim);
#pragma unroll
        for (int f = 0; f < 4; ++f) { gy[b][f] = __ldg(DA + f * fs + n); gz[b][f] = __ldg(DB + f * fs + n); }
      }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = nb + b * TPL;
        if (n > dim) break;
        const double q0 = Tl[n], u = Tl[ts + n], v = Tl[2 * ts + n], w = Tl[3 * ts + n], p = Tl[4 * ts + n];
        const double ux = Gl[n], vx = Gl[gs + n], wx = Gl[2 * gs + n], tx = Gl[3 * gs + n];
        if (!(q0 > 0.0) || !isfinite(p)) bad = 1;
        const double tmp = p * (1.0 / q0) * a.th.const2;
        const double s12 = 0.5 * (gy[b][0] + vx), s13 = 0.5 * (gz[b][0] + wx), s23 = 0.5 * (gz[b][1] + gy[b][2]);
        const double div = ux + gy[b][1] + gz[b][2], skk = (1.0 / 3.0) * div;
        const double miu = viscosity(a.th, tmp) * a.th.inv_re, miu2 = 2.0 * miu, hcc = miu * a.th.inv_prc5;
        const double t11 = miu2 * (ux - skk), t12 = miu2 * s12, t13 = miu2 * s13;
        const double t22 = miu2 * (gy[b][1] - skk), t23 = miu2 * s23, t33 = miu2 * (gz[b][2] - skk);
        const double E = p * a.th.const6 + q0 * (0.5 * (u * u + v * v + w * w));
        double F[5];
        euler<1>(q0, u, v, w, p, E, F);
        VF[n] = -F[0];
        VF[fs + n] = t12 - F[1];
        VF[2 * fs + n] = t22 - F[2];
        VF[3 * fs + n] = t23 - F[3];
        VF[4 * fs + n] = (hcc * gy[b][3] + t12 * u + t22 * v + t23 * w) - F[4];
        euler<2>(q0, u, v, w, p, E, F);
        VF[5 * fs + n] = -F[0];
        VF[6 * fs + n] = t13 - F[1];
        VF[7 * fs + n] = t23 - F[2];
        VF[8 * fs + n] = t33 - F[3];
        VF[9 * fs + n] = (hcc * gz[b][3] + t13 * u + t23 * v + t33 * w) - F[4];
        euler<0>(q0, u, v, w, p, E, F);
        if (DIAG && n >= 1 && counted) {
          ke += q0 * (u * u + v * v + w * w);
          const double o1 = gy[b][2] - gz[b][1], o2 = gz[b][0] - wx, o3 = vx - gy[b][0];
          en += q0 * (o1 * o1 + o2 * o2 + o3 * o3);
          di += miu2 * (ux * ux + gy[b][1] * gy[b][1] + gz[b][2] * gz[b][2] + 2.0 * (s12 * s12 + s13 * s13 + s23 * s23) -
                        (1.0 / 3.0) * (div * div));
        }
        // node n's gradients are read: its fluxes take their place
        const double x[5] = {-F[0], t11 - F[1], t12 - F[2], t13 - F[3],
                             (hcc * tx + t11 * u + t12 * v + t13 * w) - F[4]};
        put<5>(Gl, gs, n, dim, x);
      }
    }
  }
  if (bad) atomicOr(a.err, 1);
  if (DIAG) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      ke += __shfl_down_sync(FULL, ke, off);
      en += __shfl_down_sync(FULL, en, off);
      di += __shfl_down_sync(FULL, di, off);
    }
    if ((threadIdx.x & 31) == 0) {
      red[3 * (threadIdx.x >> 5)] = ke;
      red[3 * (threadIdx.x >> 5) + 1] = en;
      red[3 * (threadIdx.x >> 5) + 2] = di;
    }
  }
  __syncthreads();
  if (DIAG && threadIdx.x < 3) {
    double s = 0.0;
    for (int w = 0; w < NT / 32; ++w) s += red[3 * w + threadIdx.x];
    a.partials[3 * ((int64_t)z * gridDim.x + blockIdx.x) + threadIdx.x] = s;
  }
  solve_tiles<S, NL, 5>(a, k, G, ex);
  __syncthreads();
  if (on) {
    double* R = a.R + row;
#pragma unroll
    for (int f = 0; f < 5; ++f)
      for (int n = j0; n <= dim; n += TPL) R[f * fs + n] = Gl[f * gs + n];
  }
}

// The filter along x, in place, 8 lines of one field per CTA; rows move by bulk copies both ways.
template <int S>
__global__ void __launch_bounds__(256, 2) k_row_filter(const __grid_constant__ RowArgs a, const __grid_constant__ ColConst<S> k) {
  constexpr int LW = 8;
  extern __shared__ __align__(16) double sm[];
  __shared__ uint64_t bar;
  const int dim = a.g.N[0], LG = a.LG, nch = a.op.nch;
  double* G = sm;                              // node n of line l at l * LG + ROW_HF + n
  double* ex = G + LW * LG + S + 8;
  const int ntx = (a.g.N[1] + LW) / LW;        // tiles along y of one plane
  const int m = blockIdx.x % 5, tile = blockIdx.x / 5, z = tile / ntx, y0 = (tile - z * ntx) * LW;
  const int nl = min(LW, a.g.N[1] + 1 - y0);
  double* f = a.q + m * a.g.fs + (int64_t)y0 * a.g.st[1] + (int64_t)z * a.g.st[2];
  const unsigned bytes = (unsigned)(((dim + 1) * 8 + 15) & ~15);
  if (threadIdx.x == 0) mbar_init(&bar, 1);
  __syncthreads();
  if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, bytes * (unsigned)nl);
  if (threadIdx.x < 32) {
    __syncwarp();
    if (threadIdx.x < nl) bulk_g2s(G + threadIdx.x * LG + ROW_HF, f + threadIdx.x * a.g.st[1], bytes, &bar);
  }
  const int l = threadIdx.x % LW, p = threadIdx.x / LW, c = col_chunk(a.op, p);
  const bool act = p < nch;
  double* line = G + l * LG + ROW_HF;
  mbar_wait_or_flag(&bar, a.err);
  const int n0 = col_node<S>(a.op, c);
  double v[S];
  if (act) {
    double w[S + 10];
    if (c == 0 || c == nch - 1 || n0 + S + 4 > dim) {
#pragma unroll
      for (int i = 0; i < S + 10; ++i) w[i] = line[wrap_node(n0 - 5 + i, dim)];
    } else {
#pragma unroll
      for (int i = 0; i < S + 10; ++i) w[i] = line[n0 - 5 + i];
    }
    col_rhs_filter<S, false>(v, w, a.w, a, c, nch);
    col_zero_ragged<S>(v, a.op, c);
  }
  col_solve<S, LW>(v, a.op, k, c, l, act, ex, ex + nch * LW);
  if (act) {
    const int nv = col_rows<S>(a.op, c);
#pragma unroll
    for (int t = 0; t < S; ++t)
      if (t < nv && (t >= 3 || c != 0) && (t < S - 3 || c != nch - 1)) line[n0 + t] = v[t];
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tile's writes before the bulk stores
  __syncthreads();
  if (threadIdx.x < nl) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(f + threadIdx.x * a.g.st[1]),
                 "r"(smem_u32(G + threadIdx.x * LG + ROW_HF)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
}

}  // namespace row_detail
}  // namespace astr
