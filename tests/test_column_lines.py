"""The column solve of the line operators (csrc/colsolve.cuh): chunks of S rows per thread, the
left-over slots at the end of chunk 1, carries combined over the chunks.

On the CPU: the algorithm restated in numpy against the reference's sequential Thomas sweep
(commfunc.F90:790-813) on the oracle's factors. On the GPU: every operator at the sizes where the
rows per chunk, the lines per CTA or the tile walk change, against the oracle."""
import numpy as np
import pytest

import oracle

HM = 5


def _thomas(ac, d):
    a1, a2, a3 = ac
    y = np.empty_like(d)
    y[0] = d[0]
    for r in range(1, len(d)):
        y[r] = d[r] * a2[r] - y[r - 1] * a3[r]
    for r in range(len(d) - 2, -1, -1):
        y[r] = y[r] - a1[r] * y[r + 1]
    return y


def _tables(ac, S, pad):
    """fill_colop's chunk tables (schemes.cu): the system with `pad` identity rows before and after it,
    the slots left over as the last ones of chunk 1, the chunks c_lo..nch-2 with one coefficient set,
    and the converged ac2 (k2) taken out of every row's."""
    n0 = len(ac[0])
    n = n0 + 2 * pad
    nch = max(3, -(-n // S))
    nv = n - (nch - 1) * S
    e1, e2, e3 = -np.ones((nch, S)), np.zeros((nch, S)), -np.ones((nch, S))
    for c in range(nch):
        for k in range(S):
            r = c * S + k - (S - nv if c > 1 else 0) - pad
            if c == 1 and k >= nv:
                continue
            if r < 0 or r >= n0:
                e1[c, k], e2[c, k], e3[c, k] = 0.0, 1.0, 0.0
            else:
                e1[c, k] = 0.0 if r == n0 - 1 else ac[0][r]
                e2[c, k], e3[c, k] = (1.0, 0.0) if r == 0 else (ac[1][r], ac[2][r])
    tabs = np.stack([e1, e2, e3], axis=-1)
    c_lo, k2 = nch - 1, 1.0
    if nch > 3 and np.all(tabs[nch - 2] == tabs[nch - 2, 0]):
        c_lo, k2 = nch - 2, e2[nch - 2, 0]
        while c_lo > 2 and np.array_equal(tabs[c_lo - 1], tabs[nch - 2]):
            c_lo -= 1
        c_lo = min(c_lo + (c_lo % 2 == 0), nch - 1)
    return e1, e2 / k2, e3, nch, nv, c_lo, k2


def _columns(ac, d, S, pad=0):
    """col_solve's sweeps (colsolve.cuh): converged chunks take no factor per row (the right-hand side
    carries k2), table chunks the rest of ac2."""
    e1, e2, e3, nch, nv, c_lo, k2 = _tables(ac, S, pad)
    rows = np.concatenate([np.zeros(pad), d, np.zeros(pad)]) * k2
    v = np.zeros((nch, S))
    for c in range(nch):
        m = nv if c == 1 else S
        r = c * S - (S - nv if c > 1 else 0)
        v[c, :m] = rows[r:r + m]
    const = [c_lo <= c < nch - 1 for c in range(nch)]
    last = nch - 2
    pf, qb = np.cumprod(-e3, axis=1), np.cumprod((-e1)[:, ::-1], axis=1)[:, ::-1]
    k1, k3 = e1[last, 0], e3[last, 0]
    G, B = np.zeros(nch), np.zeros(nch)
    for c in range(nch):
        g = 0.0
        for t in range(S):
            g = v[c, t] - k3 * g if const[c] else v[c, t] * e2[c, t] - e3[c, t] * g
            v[c, t] = g
        G[c] = g
    for c in range(nch):
        cin = 0.0
        for j in range(c):
            cin = (pf[j, -1] if j < c_lo else pf[last, -1]) * cin + G[j]
        y = (pf[last] if const[c] else pf[c]) * cin + v[c]
        if c == 1:
            y[nv:] = 0.0
        g = 0.0
        for t in range(S - 1, -1, -1):
            g = y[t] - (k1 if const[c] else e1[c, t]) * g
            v[c, t] = g
        B[c] = g
    for c in range(nch - 1):
        cb = B[nch - 1]
        for j in range(nch - 2, c, -1):
            cb = (qb[last, 0] if j >= c_lo else qb[j, 0]) * cb + B[j]
        v[c] += (qb[last] if const[c] else qb[c]) * cb
    x = np.concatenate([v[c, :nv if c == 1 else S] for c in range(nch)])
    return x[pad:len(x) - pad]


# S as col_rows_per_chunk picks it, and 25 as pass C has it; 263 and 1049 leave no slot over
@pytest.mark.parametrize("dim,S", [(16, 5), (20, 9), (32, 9), (38, 9), (39, 17), (85, 17), (131, 33), (257, 33), (258, 33),
                                   (263, 33), (600, 25), (1040, 33), (1049, 33), (1060, 37)])
@pytest.mark.parametrize("kind", ["deriv", "filter", "slow filter", "flux"])
@pytest.mark.parametrize("ntype", [1, 2, 3, 4])
@pytest.mark.parametrize("pad", [0, 2])
def test_chunks_equal_thomas(kind, ntype, dim, S, pad):
    sch = {"deriv": lambda: oracle.fd_scheme_initiate("643c", ntype, dim),
           "filter": lambda: oracle.compact_filter_initiate(ntype, dim, 0.49, 1.11, 0.98),
           # factors that go on changing along the line: no converged chunks
           "slow filter": lambda: oracle.compact_filter_initiate(ntype, dim, 0.5, 1.11, 0.98),
           "flux": lambda: oracle.compact_flux_initiate(ntype, dim, "-", 0.3)}[kind]()
    ac = sch.ac()[2:]
    if len(ac[0]) + 2 * pad < 2 * S:
        pytest.skip("fewer than two chunks of rows")
    d = np.random.default_rng(dim).standard_normal(len(ac[0]))
    ref, got = _thomas(ac, d), _columns(ac, d, S, pad)
    # both orders round each row a few times; errors decay along the line with the factors, or at
    # alpha = 0.5 add up over it
    eps = 40 * (dim if kind == "slow filter" else 1) * np.finfo(float).eps
    assert np.abs(got - ref).max() <= eps * np.abs(ref).max()
    if dim >= 600:   # the sizes that exercise converged chunks do have them
        nch, _, c_lo = _tables(ac, S, pad)[3:6]
        assert (c_lo < nch - 1) == (kind != "slow filter")


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def _apply(ag, ctx, kind, ntype, dim, f, d, lb, wind="+", alfa=0.49, **kw):
    if kind == "deriv":
        return ag.central(ctx, ag.fd_scheme_initiate(ctx, "643c", ntype, dim), f, d, lbound=lb, **kw)
    if kind == "explicit":
        return ag.central(ctx, ag.fd_scheme_initiate(ctx, "643e", ntype, dim), f, d, lbound=lb, **kw)
    if kind == "filter":
        return ag.compact_filter(ctx, ag.compact_filter_initiate(ctx, ntype, dim, alfa, 1.11, 0.98), f, d, lbound=lb, **kw)
    sch = ag.compact_flux_initiate(ctx, ntype, dim, wind, 0.3)
    return (ag.flux_compact if kind == "flux" else ag.flux_difference)(ctx, sch, f, d, lbound=lb, **kw)


def _oracle(kind, ntype, dim, f, d, lb, wind="+", alfa=0.49):
    if kind in ("deriv", "explicit"):
        return oracle.fd_scheme_initiate("643c" if kind == "deriv" else "643e", ntype, dim).apply3d(f, d, lbound=lb)
    if kind == "filter":
        return oracle.compact_filter_initiate(ntype, dim, alfa, 1.11, 0.98).apply3d(f, d, lbound=lb)
    fh = oracle.compact_flux_initiate(ntype, dim, wind, 0.3).apply3d(f, d, lbound=lb)
    if kind == "flux":
        return fh
    n = fh.shape[d]
    return np.asfortranarray(fh.take(range(1, n), axis=d) - fh.take(range(n - 1), axis=d))


@pytest.fixture(scope="module")
def ctx():
    import astr_gpu_b200 as ag
    return ag.Context(0)


def _lines(dim, d, rng):
    shape, lb = [35, 34, 3], [0, 0, 0]   # other extents past one tile of 32 lines
    if d == 2:
        shape = [35, 3, 3]
    shape[d], lb[d] = dim + 1 + 2 * HM, -HM
    return np.asfortranarray(rng.standard_normal(shape)), lb


# around every change of the rows per chunk (systems of 15, 18, 46, 91, 177, 1057 rows), of the lines
# per CTA (8 chunks of 33 rows: 264) and the longest system; 16 and 34 rows leave whole or no
# left-over slots
@pytest.mark.gpu
@pytest.mark.parametrize("dim", [8, 9, 11, 13, 16, 17, 38, 39, 40, 44, 84, 85, 90, 169, 170, 176, 257, 258, 263, 1049, 1050,
                                 1056, 1145])
@pytest.mark.parametrize("kind", ["deriv", "explicit", "filter", "flux", "fluxdiff"])
@pytest.mark.parametrize("ntype", [3, 4])
def test_sizes(ctx, kind, ntype, dim):
    import astr_gpu_b200 as ag
    if kind == "filter" and dim < 16:
        pytest.skip("the filter needs 16 nodes")
    rng = np.random.default_rng(dim)
    for d in range(3):
        f, lb = _lines(dim, d, rng)
        assert _rel(_apply(ag, ctx, kind, ntype, dim, f, d, lb), _oracle(kind, ntype, dim, f, d, lb)) <= 1e-12


# one physical end, and the downwind flux, at the same edges
@pytest.mark.gpu
@pytest.mark.parametrize("dim", [16, 17, 39, 90, 176, 263, 1050])
@pytest.mark.parametrize("kind,wind", [("deriv", "+"), ("explicit", "+"), ("filter", "+"), ("flux", "-"), ("fluxdiff", "-")])
@pytest.mark.parametrize("ntype", [1, 2, 3])
def test_one_physical_end(ctx, kind, wind, ntype, dim):
    import astr_gpu_b200 as ag
    for d in range(3):
        f, lb = _lines(dim, d, np.random.default_rng(dim))
        ref = _oracle(kind, ntype, dim, f, d, lb, wind)
        assert _rel(_apply(ag, ctx, kind, ntype, dim, f, d, lb, wind), ref) <= 1e-12


# alpha = 0.5: factors that never converge, every chunk reads its own. The system's condition grows with
# the square of its length, and with it what rounding the right-hand side and each sweep may change
@pytest.mark.gpu
@pytest.mark.parametrize("dim", [17, 39, 90, 176, 263, 1050])
@pytest.mark.parametrize("ntype", [3, 4])
def test_filter_without_converged_factors(ctx, ntype, dim):
    import astr_gpu_b200 as ag
    a1, a2, a3 = oracle.compact_filter_initiate(ntype, dim, 0.5, 1.11, 0.98).ac()[2:]
    lower, upper = a3[1:] / a2[1:], a1[:-1] / np.concatenate([[1.0], a2[1:-1]])
    A = np.eye(len(a1)) + np.diag(lower, -1) + np.diag(upper, 1)
    tol = 16 * np.finfo(float).eps * np.linalg.cond(A, np.inf)
    assert tol <= 1e-7
    for d in range(3):
        f, lb = _lines(dim, d, np.random.default_rng(dim))
        assert _rel(_apply(ag, ctx, "filter", ntype, dim, f, d, lb, alfa=0.5),
                    _oracle("filter", ntype, dim, f, d, lb, alfa=0.5)) <= max(tol, 1e-12)


# a line that holds a NaN or an infinity leaves the lines beside it as they are, bit for bit
@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("dim", [39, 176, 300])
@pytest.mark.parametrize("kind", ["deriv", "filter", "flux"])
def test_bad_line_stays_alone(ctx, kind, dim, bad):
    import astr_gpu_b200 as ag
    for d in range(3):
        f, lb = _lines(dim, d, np.random.default_rng(dim))
        ref = _apply(ag, ctx, kind, 3, dim, f, d, lb)
        at = [2, 2, 2]
        at[d] = HM + dim // 2
        f[tuple(at)] = bad
        got = _apply(ag, ctx, kind, 3, dim, f, d, lb)
        at[d] = slice(None)
        assert not np.isfinite(got[tuple(at)]).all()
        got[tuple(at)] = ref[tuple(at)] = 0.0
        np.testing.assert_array_equal(got, ref)


# x extents at the edges of flattened and per-row tiles (16 and 32 lines)
@pytest.mark.gpu
@pytest.mark.parametrize("nx", [1, 15, 16, 17, 31, 32, 33, 64, 97, 600])
@pytest.mark.parametrize("dim", [40, 100, 300])
def test_tile_edges(ctx, nx, dim):
    import astr_gpu_b200 as ag
    rng = np.random.default_rng(nx)
    for d in (1, 2):
        shape, lb = [nx, 5, 5], [0, 0, 0]
        shape[d], lb[d] = dim + 1 + 2 * HM, -HM
        f = np.asfortranarray(rng.standard_normal(shape + [2]))
        for kind in ("deriv", "filter"):
            assert _rel(_apply(ag, ctx, kind, 3, dim, f, d, lb), _oracle(kind, 3, dim, f, d, lb)) <= 1e-12


# the result over the input: every line is read before it is written
@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["deriv", "explicit", "filter"])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_in_place(ctx, kind, d):
    import ctypes
    import torch
    import astr_gpu_b200 as ag
    dim = 70
    shape, lb = [40, 37, 6], [0, 0, 0]
    shape[d], lb[d] = dim + 1 + 2 * HM, -HM
    f = np.asfortranarray(np.random.default_rng(d).standard_normal(shape))
    ref = _oracle(kind, 3, dim, f, d, lb)
    t = torch.from_numpy(np.ascontiguousarray(f.T)).cuda()
    torch.cuda.synchronize()
    i64 = lambda v: (ctypes.c_int64 * 3)(*v)  # noqa: E731
    p = ctypes.c_void_p(t.data_ptr())
    if kind == "filter":
        s = ag.compact_filter_initiate(ctx, 3, dim, 0.49, 1.11, 0.98)
        ctx.check(ctx.L.astr_filter_lines(ctx._h, s._h, d, p, i64(shape), i64(lb), p, i64(shape), i64(lb), 1, ag.ASTR_DEVICE))
    else:
        s = ag.fd_scheme_initiate(ctx, "643c" if kind == "deriv" else "643e", 3, dim)
        ctx.check(ctx.L.astr_deriv_lines(ctx._h, s._h, d, p, i64(shape), i64(lb), p, i64(shape), i64(lb), 1, 1.0, ag.ASTR_DEVICE))
    ctx.synchronize()
    got = t.cpu().numpy().T
    inner = [slice(None)] * 3
    inner[d] = slice(HM, HM + dim + 1)
    assert _rel(got[tuple(inner)], ref) <= 1e-12
    halo = [slice(None)] * 3
    halo[d] = slice(0, HM)
    assert np.array_equal(got[tuple(halo)], f[tuple(halo)])
