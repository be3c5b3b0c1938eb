// Host construction of the line operators: the reference's scheme set-up restated in C++, and
// the lane tables the segmented solve reads.
//   fd_scheme_initiate          src/derivative.F90:63-158
//   compact_filter_initiate     src/filter.F90:31-100
//   filter_coefficient_cal      src/filter.F90:299-432
//   compact_flux_initiate       src/flux.F90:32-112
//   tridiagonal_thomas_proprocess src/commfunc.F90:752-774
#include <algorithm>
#include <cmath>
#include <cstring>

#include "internal.h"

namespace astr {

static void thomas_factor(HostOp& op) {
  const int n = op.nsys();
  op.ac1.assign(n, 0.0); op.ac2.assign(n, 0.0); op.ac3.assign(n, 0.0);
  op.ac1[0] = op.c[0];
  for (int i = 1; i < n; ++i) {
    const double piv = 1.0 - op.a[i] * op.ac1[i - 1];
    op.ac1[i] = op.c[i] / piv;
    op.ac2[i] = 1.0 / piv;
    op.ac3[i] = op.a[i] / piv;
  }
}

static void set_range(HostOp& op, int ntype, int dim, int ext) {
  op.ntype = ntype;
  op.dim = dim;
  op.left_phys = (ntype == 1 || ntype == 4);
  op.right_phys = (ntype == 2 || ntype == 4);
  op.first_node = op.left_phys ? 0 : -ext;
  op.last_node = op.right_phys ? dim : dim + ext;
}

bool build_fd_op(HostOp& op, const char* scheme, int ntype, int dim) {
  if (ntype < 1 || ntype > 4 || dim < 8) return false;
  const int nscheme = (scheme[0] - '0') * 100 + (scheme[1] - '0') * 10 + (scheme[2] - '0');
  if (scheme[3] == 'e' && nscheme / 100 == 6) {
    // explicit central scheme: diff6ec has no system; rows are nodes 0..dim
    op.kind = OP_EXPLICIT;
    op.ntype = ntype; op.dim = dim;
    op.left_phys = (ntype == 1 || ntype == 4);
    op.right_phys = (ntype == 2 || ntype == 4);
    op.first_node = 0; op.last_node = dim;
    const int n = op.nsys();
    op.a.assign(n, 0.0); op.c.assign(n, 0.0);
    thomas_factor(op);
    return true;
  }
  if (scheme[3] != 'c' || nscheme != 643) return false;
  op.kind = OP_DERIV;
  set_range(op, ntype, dim, 1);
  const int n = op.nsys();
  op.a.assign(n, 1.0 / 3.0);
  op.c.assign(n, 1.0 / 3.0);
  // explicit 6th-order rows at interfaces
  op.a[0] = op.c[0] = 0.0;
  op.a[n - 1] = op.c[n - 1] = 0.0;
  if (op.left_phys) {
    op.a[0] = op.c[0] = 2.0;      // 3rd-order biased compact closure
    op.a[1] = op.c[1] = 0.25;     // 4th-order compact
  }
  if (op.right_phys) {
    op.a[n - 1] = op.c[n - 1] = 2.0;
    op.a[n - 2] = op.c[n - 2] = 0.25;
  }
  thomas_factor(op);
  return true;
}

void build_filter_op(HostOp& op, int ntype, int dim, double alfa, double bh, double bb, bool note) {
  op.kind = OP_FILTER;
  set_range(op, ntype, dim, 3);
  op.no_note = note;
  const int n = op.nsys();
  // end-row LHS coefficients are fixed by ntype (filter.F90:44-68)
  const double b0 = op.left_phys ? 0.98 : 1.11;
  const double bm = op.right_phys ? 0.98 : 1.11;
  op.a.assign(n, alfa);
  op.c.assign(n, alfa);
  if (note) {
    op.a[0] = op.c[0] = 0.0;
    op.a[n - 1] = op.c[n - 1] = 0.0;
  } else {
    op.a[0] = op.c[0] = b0;
    op.a[n - 1] = op.c[n - 1] = bm;
  }
  thomas_factor(op);
  // RHS coefficients
  op.c6[0] = (11.0 + 10.0 * alfa) / 32.0;
  op.c6[1] = (15.0 + 34.0 * alfa) / 64.0;
  op.c6[2] = (-3.0 + 6.0 * alfa) / 32.0;
  op.c6[3] = (1.0 - 2.0 * alfa) / 64.0;
  op.c8[0] = (93.0 + 70.0 * alfa) / 256.0;
  op.c8[1] = (7.0 + 18.0 * alfa) / 32.0;
  op.c8[2] = (-7.0 + 14.0 * alfa) / 64.0;
  op.c8[3] = (1.0 - 2.0 * alfa) / 32.0;
  op.c8[4] = (-1.0 + 2.0 * alfa) / 256.0;
  op.c10[0] = (193.0 + 126.0 * alfa) / 512.0;
  op.c10[1] = (105.0 + 302.0 * alfa) / 512.0;
  op.c10[2] = (-15.0 + 30.0 * alfa) / 128.0;
  op.c10[3] = (45.0 - 90.0 * alfa) / 1024.0;
  op.c10[4] = (-5.0 + 10.0 * alfa) / 512.0;
  op.c10[5] = (1.0 - 2.0 * alfa) / 1024.0;
  // one-sided rows 0..2 (row 0 carries beta_bound)
  const double b[3][7] = {
      {(63.0 + 1.0 * bb) / 64.0, (3.0 + 29.0 * bb) / 32.0, (-15.0 + 15.0 * bb) / 64.0, (5.0 - 5.0 * bb) / 16.0,
       (-15.0 + 15.0 * bb) / 64.0, (3.0 - 3.0 * bb) / 32.0, (-1.0 + 1.0 * bb) / 64.0},
      {(1.0 + 62.0 * alfa) / 64.0, (29.0 + 6.0 * alfa) / 32.0, (15.0 + 34.0 * alfa) / 64.0, (-5.0 + 10.0 * alfa) / 16.0,
       (15.0 - 30.0 * alfa) / 64.0, (-3.0 + 6.0 * alfa) / 32.0, (1.0 - 2.0 * alfa) / 64.0},
      {(-1.0 + 2.0 * alfa) / 64.0, (3.0 + 26.0 * alfa) / 32.0, (49.0 + 30.0 * alfa) / 64.0, (5.0 + 6.0 * alfa) / 16.0,
       (-15.0 + 30.0 * alfa) / 64.0, (3.0 - 6.0 * alfa) / 32.0, (-1.0 + 2.0 * alfa) / 64.0}};
  std::memcpy(op.cb, b, sizeof(b));
  // halo-closure rows 0..2 (row 0 carries beta_halo)
  const double h[3][11] = {
      {(-1.0 + 1.0 * bh) / 1024.0, (5.0 - 5.0 * bh) / 512.0, (979.0 + 45.0 * bh) / 1024.0, (15.0 + 113.0 * bh) / 128.0,
       (-105.0 + 105.0 * bh) / 512.0, (63.0 - 63.0 * bh) / 256.0, (-105.0 + 105.0 * bh) / 512.0,
       (15.0 - 15.0 * bh) / 128.0, (-45.0 + 45.0 * bh) / 1024.0, (5.0 - 5.0 * bh) / 512.0, (-1.0 + 1.0 * bh) / 1024.0},
      {(1.0 - 2.0 * alfa) / 1024.0, (-5.0 + 10.0 * alfa) / 512.0, (45.0 + 934.0 * alfa) / 1024.0,
       (113.0 + 30.0 * alfa) / 128.0, (105.0 + 302.0 * alfa) / 512.0, (-63.0 + 126.0 * alfa) / 256.0,
       (105.0 - 210.0 * alfa) / 512.0, (-15.0 + 30.0 * alfa) / 128.0, (45.0 - 90.0 * alfa) / 1024.0,
       (-5.0 + 10.0 * alfa) / 512.0, (1.0 - 2.0 * alfa) / 1024.0},
      {(-1.0 + 2.0 * alfa) / 1024.0, (5.0 - 10.0 * alfa) / 512.0, (-45.0 + 90.0 * alfa) / 1024.0,
       (15.0 + 98.0 * alfa) / 128.0, (407.0 + 210.0 * alfa) / 512.0, (63.0 + 130.0 * alfa) / 256.0,
       (-105.0 + 210.0 * alfa) / 512.0, (15.0 - 30.0 * alfa) / 128.0, (-45.0 + 90.0 * alfa) / 1024.0,
       (5.0 - 10.0 * alfa) / 512.0, (-1.0 + 2.0 * alfa) / 1024.0}};
  std::memcpy(op.ch, h, sizeof(h));
}

// The '543' compact interface-flux scheme: interfaces i_0..i_m with i_0 = -1 at a physical left
// end (ntype 1, 4) else -2, i_m = dim at a physical right end (ntype 2, 4) else dim + 1. Interior
// LHS a, c biased by the wind and blended by bfac (the MP-LD b factor, bfacmpld of commvar);
// explicit central rows (a = c = 0) at interfaces; at physical ends the 3rd-order rows with
// a = c = 2 and a = c = 1/4 next to them.
bool build_flux_op(HostOp& op, int scheme, int ntype, int dim, int wind, double bfac) {
  if (ntype < 1 || ntype > 4 || dim < 8 || scheme != 543 || (wind != 1 && wind != -1)) return false;
  op.kind = OP_FLUX;
  op.ntype = ntype;
  op.dim = dim;
  op.left_phys = (ntype == 1 || ntype == 4);
  op.right_phys = (ntype == 2 || ntype == 4);
  op.first_node = op.left_phys ? -1 : -2;
  op.last_node = op.right_phys ? dim : dim + 1;
  op.wind = wind;
  op.bfac = bfac;
  const int n = op.nsys();
  const double a = (wind == 1) ? 0.5 - (1.0 / 6.0) * bfac : (1.0 / 6.0) + (1.0 / 6.0) * bfac;
  const double c = (wind == 1) ? (1.0 / 6.0) + (1.0 / 6.0) * bfac : 0.5 - (1.0 / 6.0) * bfac;
  op.a.assign(n, a);
  op.c.assign(n, c);
  op.a[0] = op.c[0] = 0.0;
  op.a[n - 1] = op.c[n - 1] = 0.0;
  if (op.left_phys) {
    op.a[0] = op.c[0] = 2.0;
    op.a[1] = op.c[1] = 0.25;
  }
  if (op.right_phys) {
    op.a[n - 1] = op.c[n - 1] = 2.0;
    op.a[n - 2] = op.c[n - 2] = 0.25;
  }
  thomas_factor(op);
  op.cfl[0] = 1.0 / 18.0 - (1.0 / 36.0) * bfac;
  op.cfl[1] = 19.0 / 18.0 - (9.0 / 36.0) * bfac;
  op.cfl[2] = 5.0 / 9.0 + (9.0 / 36.0) * bfac;
  op.cfl[3] = (1.0 / 36.0) * bfac;
  return true;
}

std::vector<double> lane_tables(const HostOp& op, int S, int nseg) {
  const int nsys = op.nsys();
  const int WPL = nseg / 32;
  const size_t base = (size_t)5 * S * nseg;
  const size_t slot_off = base + (size_t)T_NSEGTAB * nseg + 2 * (size_t)WPL;
  std::vector<double> t(slot_off + (size_t)(nseg + 1) / 2, 0.0);
  // f: 0 ac1, 1 ac2, 2 ac3, 3 pf, 4 qb (see the layout in ops.cuh)
  auto at = [&](int f, int tt, int seg) -> double& {
    const size_t rs = (size_t)tt * nseg + seg;
    switch (f) {
      case 1: return t[2 * rs];
      case 2: return t[2 * rs + 1];
      case 3: return t[(size_t)2 * S * nseg + rs];
      case 0: return t[(size_t)3 * S * nseg + 2 * rs];
      default: return t[(size_t)3 * S * nseg + 2 * rs + 1];
    }
  };
  auto sg = [&](int k, int seg) -> double& { return t[base + (size_t)k * nseg + seg]; };
  std::vector<double> mf(nseg), mb(nseg);
  for (int seg = 0; seg < nseg; ++seg) {
    double e1[64], e2[64], e3[64];
    for (int tt = 0; tt < S; ++tt) {
      const int r = seg * S + tt;
      if (r < nsys) {
        e1[tt] = (r == nsys - 1) ? 0.0 : op.ac1[r];  // back substitution starts at x_n = d_n
        e2[tt] = (r == 0) ? 1.0 : op.ac2[r];         // row 1 of the forward sweep is untouched
        e3[tt] = (r == 0) ? 0.0 : op.ac3[r];
      } else {
        e1[tt] = e2[tt] = e3[tt] = 0.0;              // padding rows solve to zero
      }
      at(0, tt, seg) = e1[tt];
      at(1, tt, seg) = e2[tt];
      at(2, tt, seg) = e3[tt];
    }
    double p = 1.0;
    for (int tt = 0; tt < S; ++tt) { p *= -e3[tt]; at(3, tt, seg) = p; }
    mf[seg] = p;
    double q = 1.0;
    for (int tt = S - 1; tt >= 0; --tt) { q *= -e1[tt]; at(4, tt, seg) = q; }
    mb[seg] = q;
  }
  // scan composites within each warp (see seg_solve)
  for (int w = 0; w < WPL; ++w) {
    const int s0 = 32 * w;
    for (int l = 0; l < 32; ++l) {
      for (int k = 0; k < 5; ++k) {
        const int off = 1 << k;
        double pf = 0.0, pb = 0.0;
        if (l >= off) { pf = 1.0; for (int j = l - off + 1; j <= l; ++j) pf *= mf[s0 + j]; }
        if (l + off <= 31) { pb = 1.0; for (int j = l; j <= l + off - 1; ++j) pb *= mb[s0 + j]; }
        sg(T_FS + k, s0 + l) = pf;
        sg(T_BS + k, s0 + l) = pb;
      }
      double fe = 1.0, be = 1.0;
      for (int j = 0; j < l; ++j) fe *= mf[s0 + j];
      for (int j = l + 1; j < 32; ++j) be *= mb[s0 + j];
      sg(T_FE, s0 + l) = fe;
      sg(T_BE, s0 + l) = be;
    }
    double mw = 1.0, mwb = 1.0;
    for (int j = 0; j < 32; ++j) { mw *= mf[s0 + j]; mwb *= mb[s0 + j]; }
    t[base + (size_t)T_NSEGTAB * nseg + w] = mw;
    t[base + (size_t)T_NSEGTAB * nseg + WPL + w] = mwb;
  }
  // Row-coefficient slot of every segment: the first segment whose (ac2, ac3, pf, ac1, qb)
  // column is bitwise the same. Interior segments (converged factors) share one slot, so the
  // lanes of a warp read the same addresses and the loads are broadcasts.
  int* slot = reinterpret_cast<int*>(t.data() + slot_off);
  for (int seg = 0; seg < nseg; ++seg) {
    slot[seg] = seg;
    for (int o = 0; o < seg; ++o) {
      bool same = true;
      for (int f = 0; f < 5 && same; ++f)
        for (int tt = 0; tt < S && same; ++tt) same = at(f, tt, o) == at(f, tt, seg);
      if (same) { slot[seg] = o; break; }
    }
  }
  return t;
}

Layout pick_layout(int nsys_max) {
  if (nsys_max <= 96) return {3, 1};
  if (nsys_max <= 160) return {5, 1};
  if (nsys_max <= 288) return {9, 1};
  if (nsys_max <= 576) return {9, 2};
  if (nsys_max <= 1152) return {9, 4};
  return {0, 0};
}

void fill_lineop(const HostOp& h, LineOp& o) {
  o.tab = nullptr;
  o.nsys = h.nsys();
  o.ext_lo = -h.first_node;
  o.dim = h.dim;
  o.kind = h.kind;
  o.left_phys = h.left_phys;
  o.right_phys = h.right_phys;
  o.no_filter_note = h.no_note;
  o.nseg = 0;
  o.S = 0;
  // closure rows with their own RHS formulas (derivative.F90:230-294, filter.F90:176-269)
  if (h.kind == OP_FILTER) {
    o.spec_lo = h.left_phys ? 5 : 3;
    o.spec_hi = h.right_phys ? 5 : 3;
  } else {   // derivative and interface flux: two closure rows at a physical end, else one
    o.spec_lo = h.left_phys ? 2 : 1;
    o.spec_hi = h.right_phys ? 2 : 1;
  }
  std::memcpy(o.c10, h.c10, sizeof(o.c10));
  std::memcpy(o.ch, h.ch, sizeof(o.ch));
  std::memcpy(o.cb, h.cb, sizeof(o.cb));
  std::memcpy(o.c6, h.c6, sizeof(o.c6));
  std::memcpy(o.c8, h.c8, sizeof(o.c8));
  o.wind = h.wind;
  std::memcpy(o.cfl, h.cfl, sizeof(o.cfl));
}

cudaError_t make_devop(const HostOp& h, Layout lay, DevOp& out) {
  out.S = lay.S;
  out.WPL = lay.WPL;
  const int nseg = 32 * lay.WPL;
  std::vector<double> tab = lane_tables(h, lay.S, nseg);
  cudaError_t e = cudaMalloc(&out.dtab, tab.size() * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMemcpy(out.dtab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return e;
  LineOp& o = out.op;
  fill_lineop(h, o);
  o.tab = out.dtab;
  o.nseg = nseg;
  o.S = lay.S;
  return cudaSuccess;
}

void free_devop(DevOp& d) {
  if (d.dtab) cudaFree(d.dtab);
  d.dtab = nullptr;
}

// Measured on a B200 (derivative / filter, GB/s of read + written nodes; lines of 32 adjacent in x
// per CTA along y): 256 nodes 33 rows 5400 / 4160, 17 rows 3570 / 3050; 128 nodes 33 rows 4135 /
// 2876, 17 rows 3465 / 2892; 64 nodes 17 rows 2055 / 1488, 33 rows 1707 / 1486. Along x (16 lines
// through shared memory) 128 nodes 33 rows 2960 / 2142, 17 rows 2739 / 2410; 256 nodes 33 rows
// 3540 / 3130, 17 rows 3094 / 2741.
int col_rows_per_chunk(int nsys, int dir) {
  if (nsys < 15) return 3;
  if (nsys < 18) return 5;
  if (nsys <= 45) return 9;
  if (nsys <= (dir == 0 ? 176 : 90)) return 17;
  if (nsys <= 1056) return 33;
  if (nsys <= 1152) return 37;
  return 0;
}

// The column solve's view of the system with `pad` identity rows before and after it (pad > 0
// embeds an operator in the chunks of one with a longer system).
// Everything but the device copy of the table `t`.
static cudaError_t fill_colop(const HostOp& h, int S, int pad, DevColOp& out, std::vector<double>& t) {
  const int n0 = h.nsys(), nsys = n0 + 2 * pad;
  if (S < 1 || S > COL_MAXS || nsys < 2 * S) return cudaErrorInvalidValue;
  fill_lineop(h, out.line);
  out.S = S;
  const int nch = std::max(3, (nsys + S - 1) / S);
  ColOp& o = out.op;
  o.nch = nch;
  o.nv = nsys - (nch - 1) * S;
  o.n_first = h.first_node - pad;
  o.c_lo = nch - 1;
  if (h.kind == OP_EXPLICIT) return cudaSuccess;   // rows but no system
  const size_t rows = (size_t)nch * S;
  t.assign(rows * 6 + 2 * (size_t)nch, 0.0);
  for (int c = 0; c < nch; ++c) {
    double p = 1.0, q = 1.0;
    double* tc = t.data() + (size_t)c * S * 6;
    for (int k = 0; k < S; ++k) {
      double e1, e2, e3;
      const int r = c * S + k - (c > 1 ? S - o.nv : 0) - pad;   // row of the operator's own system
      if (c == 1 && k >= o.nv) { e1 = -1.0; e2 = 0.0; e3 = -1.0; }   // left over: passes the carries on
      else if (r < 0 || r >= n0) { e1 = 0.0; e2 = 1.0; e3 = 0.0; }   // identity row
      else {
        e1 = (r == n0 - 1) ? 0.0 : h.ac1[r];   // back substitution starts at the last row
        e2 = (r == 0) ? 1.0 : h.ac2[r];        // the first row of the forward sweep is untouched
        e3 = (r == 0) ? 0.0 : h.ac3[r];
      }
      tc[6 * k] = e2;
      tc[6 * k + 1] = e3;
      p *= -e3;
      tc[6 * k + 2] = p;
      tc[6 * k + 3] = e1;
    }
    for (int k = S - 1; k >= 0; --k) { q *= -tc[6 * k + 3]; tc[6 * k + 4] = q; }
    t[rows * 6 + c] = p;
    t[rows * 6 + nch + c] = q;
  }
  // chunks from c_lo on have one coefficient set, bitwise that of the last chunk but one
  const double* tr = t.data() + (size_t)(nch - 2) * S * 6;
  bool flat = nch > 3;
  for (int k = 1; k < S && flat; ++k) flat = tr[6 * k] == tr[0] && tr[6 * k + 1] == tr[1] && tr[6 * k + 3] == tr[3];
  if (flat) {
    o.c_lo = nch - 2;
    while (o.c_lo > 2 && std::memcmp(t.data() + (size_t)(o.c_lo - 1) * S * 6, tr, (size_t)S * 6 * sizeof(double)) == 0) --o.c_lo;
    if (o.c_lo % 2 == 0) ++o.c_lo;   // with the last one an even number of table chunks
    o.c_lo = std::min(o.c_lo, nch - 1);
  }
  for (int k = 0; k < S; ++k) { out.pf[k] = tr[6 * k + 2]; out.qb[k] = tr[6 * k + 4]; }
  out.k3 = tr[1];
  out.k1 = tr[3];
  out.k2 = flat ? tr[0] : 1.0;
  for (size_t r = 0; r < rows; ++r) t[6 * r] /= out.k2;
  return cudaSuccess;
}

// Column operators share one device table: theirs one after the other in `tab`.
cudaError_t fill_colops(ColSpec* specs, int n, std::vector<double>& tab) {
  tab.clear();
  for (int i = 0; i < n; ++i) {
    std::vector<double> t;
    const cudaError_t e = fill_colop(*specs[i].h, specs[i].S, specs[i].pad, *specs[i].out, t);
    if (e != cudaSuccess) return e;
    specs[i].at = tab.size();
    tab.insert(tab.end(), t.begin(), t.end());
    tab.resize((tab.size() + 1) / 2 * 2);   // 16-byte rows
  }
  return cudaSuccess;
}

cudaError_t load_colops(const ColSpec* specs, int n, const std::vector<double>& tab, double* dev, cudaStream_t st) {
  // st holds nothing else: on the context's stream this would wait for all work queued there, on the
  // legacy stream for the caller's
  cudaError_t e = cudaMemcpyAsync(dev, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  for (int i = 0; i < n; ++i) specs[i].out->op.tab = dev + specs[i].at;
  return e;
}

cudaError_t make_colops(ColSpec* specs, int n, cudaStream_t st) {
  std::vector<double> tab;
  cudaError_t e = fill_colops(specs, n, tab);
  if (e != cudaSuccess || tab.empty()) return e;   // explicit operators have no table
  DevColOp& own = *specs[0].out;
  if ((e = cudaMalloc(&own.dtab, tab.size() * sizeof(double))) != cudaSuccess) return e;
  return load_colops(specs, n, tab, own.dtab, st);
}

ColWeights col_weights(const DevColOp& d, double scale) {
  ColWeights k{};
  k.ks = d.k2 * scale;
  const LineOp& o = d.line;
  if (o.kind == OP_DERIV) {
    k.w[0] = (7.0 / 9.0) * k.ks;
    k.w[1] = (1.0 / 36.0) * k.ks;
  } else if (o.kind == OP_FILTER) {
    for (int i = 0; i < 6; ++i) k.w[i] = (i == 0 ? 2.0 : 1.0) * o.c10[i] * k.ks;
  } else if (o.kind == OP_FLUX) {
    for (int i = 0; i < 4; ++i) k.w[i] = o.cfl[i] * k.ks;
  }
  return k;
}

void free_colop(DevColOp& d) {
  if (d.dtab) cudaFree(d.dtab);
  d.dtab = nullptr;
}

int tile_pitch(int dim, int TI, int S) {
  const int need = dim + 1 + 2 * HT + win_slack(S);   // halos and the window slack (ops.cuh)
  const int want = TI >= 16 ? 1 : 16 / TI;   // residue mod 16 for conflict-free line-fastest access
  int lp = need;
  while ((lp % 16) != (want % 16)) ++lp;
  return lp;
}

}  // namespace astr
