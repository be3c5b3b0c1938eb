"""The column solve of the line operators (csrc/colsolve.cuh): chunks of S rows per thread, the
left-over slots in the middle chunk, carries combined over the chunks.

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


def _columns(ac, d, S):
    a1, a2, a3 = (x.copy() for x in ac)
    n = len(d)
    a1[-1], a2[0], a3[0] = 0.0, 1.0, 0.0
    nch = max(3, -(-n // S))
    rag, nv = nch // 2, n - (nch - 1) * S
    e1, e2, e3, v = -np.ones((nch, S)), np.zeros((nch, S)), -np.ones((nch, S)), np.zeros((nch, S))
    for c in range(nch):
        m = nv if c == rag else S
        r = c * S - (S - nv if c > rag else 0)
        e1[c, :m], e2[c, :m], e3[c, :m], v[c, :m] = a1[r:r + m], a2[r:r + m], a3[r:r + m], d[r:r + m]
    G, B = np.zeros(nch), np.zeros(nch)
    for c in range(nch):
        g = 0.0
        for t in range(S):
            g = v[c, t] * e2[c, t] - g * e3[c, t]
            v[c, t] = g
        G[c] = g
    for c in range(nch):
        cin = 0.0
        for j in range(c):
            cin = np.prod(-e3[j]) * cin + G[j]
        y = np.cumprod(-e3[c]) * cin + v[c]
        if c == rag:
            y[nv:] = 0.0
        g = 0.0
        for t in range(S - 1, -1, -1):
            g = y[t] - e1[c, t] * g
            v[c, t] = g
        B[c] = g
    for c in range(nch):
        cb = 0.0
        for j in range(nch - 1, c, -1):
            cb = np.prod(-e1[j]) * cb + B[j]
        v[c] += np.cumprod((-e1[c])[::-1])[::-1] * cb
    return np.concatenate([v[c, :nv if c == rag else S] for c in range(nch)])


@pytest.mark.parametrize("dim,S", [(16, 5), (20, 9), (32, 9), (38, 9), (39, 17), (85, 17), (131, 33), (257, 33), (258, 33),
                                   (1040, 33), (1060, 37)])
@pytest.mark.parametrize("kind", ["deriv", "filter"])
@pytest.mark.parametrize("ntype", [1, 2, 3, 4])
def test_chunks_equal_thomas(kind, ntype, dim, S):
    sch = {"deriv": lambda: oracle.fd_scheme_initiate("643c", ntype, dim),
           "filter": lambda: oracle.compact_filter_initiate(ntype, dim, 0.49, 1.11, 0.98)}[kind]()
    ac = sch.ac()[2:]
    d = np.random.default_rng(dim).standard_normal(len(ac[0]))
    ref, got = _thomas(ac, d), _columns(ac, d, S)
    # both orders round each row a few times; errors decay along the line with the factors
    assert np.abs(got - ref).max() <= 40 * np.finfo(float).eps * np.abs(ref).max()


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def _apply(ag, ctx, kind, ntype, dim, f, d, lb, **kw):
    if kind == "deriv":
        return ag.central(ctx, ag.fd_scheme_initiate(ctx, "643c", ntype, dim), f, d, lbound=lb, **kw)
    if kind == "explicit":
        return ag.central(ctx, ag.fd_scheme_initiate(ctx, "643e", ntype, dim), f, d, lbound=lb, **kw)
    if kind == "filter":
        return ag.compact_filter(ctx, ag.compact_filter_initiate(ctx, ntype, dim, 0.49, 1.11, 0.98), f, d, lbound=lb, **kw)
    sch = ag.compact_flux_initiate(ctx, ntype, dim, "+", 0.3)
    return (ag.flux_compact if kind == "flux" else ag.flux_difference)(ctx, sch, f, d, lbound=lb, **kw)


def _oracle(kind, ntype, dim, f, d, lb):
    if kind in ("deriv", "explicit"):
        return oracle.fd_scheme_initiate("643c" if kind == "deriv" else "643e", ntype, dim).apply3d(f, d, lbound=lb)
    if kind == "filter":
        return oracle.compact_filter_initiate(ntype, dim, 0.49, 1.11, 0.98).apply3d(f, d, lbound=lb)
    fh = oracle.compact_flux_initiate(ntype, dim, "+", 0.3).apply3d(f, d, lbound=lb)
    if kind == "flux":
        return fh
    n = fh.shape[d]
    return np.asfortranarray(fh.take(range(1, n), axis=d) - fh.take(range(n - 1), axis=d))


@pytest.fixture(scope="module")
def ctx():
    import astr_gpu_b200 as ag
    return ag.Context(0)


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
        shape, lb = [35, 34, 3], [0, 0, 0]   # other extents past one tile of 32 lines
        if d == 2:
            shape = [35, 3, 3]
        shape[d], lb[d] = dim + 1 + 2 * HM, -HM
        f = np.asfortranarray(rng.standard_normal(shape))
        assert _rel(_apply(ag, ctx, kind, ntype, dim, f, d, lb), _oracle(kind, ntype, dim, f, d, lb)) <= 1e-12


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
