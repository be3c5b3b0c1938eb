"""The passes of the RK3 step as column solves (csrc/tgv_cols.cuh, tgv_rows.cuh) against the oracle, on
boxes whose systems (N + 7 rows; N + 3 in pass C) sit at the edges where the rows per chunk, the lines
per CTA and the tile walk (x extent against 16 and 32 lines, y extent against 2, 4 and 8) change;
with and without the filter, and with one pass at a time on its lane-scan kernel."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# fields after a few steps: last-bit differences of the solves, scaled by each field's largest value
TOL = 1e-12


@pytest.fixture(scope="module")
def ctx():
    import astr_gpu_b200 as ag
    return ag.Context(0)


def _start(dims, seed):
    """A smooth field with content along every axis, mach 0.3."""
    rng = np.random.default_rng(seed)
    x = [2 * np.pi * np.remainder(np.arange(n + 1), n) / n for n in dims]
    X, Y, Z = np.meshgrid(*x, indexing="ij")
    u = [np.sin(X) * np.cos(Y) * np.cos(Z), -np.cos(X) * np.sin(Y) * np.cos(Z), np.zeros_like(X)]
    for _ in range(3):
        k = rng.integers(1, 4, 3)
        for c in range(3):
            u[c] = u[c] + 0.1 * rng.standard_normal() * np.cos(k[0] * X + k[1] * Y + k[2] * Z + rng.uniform(0, 6))
    p = 1.0 / (1.4 * 0.09) + 0.05 * np.cos(2 * X) * np.cos(Z)
    rho = p * 1.4 * 0.09
    q = np.stack([rho, rho * u[0], rho * u[1], rho * u[2], p / 0.4 + 0.5 * rho * (u[0]**2 + u[1]**2 + u[2]**2)], axis=-1)
    return np.asfortranarray(q)


def _oracle(dims, q0, dt, steps, filt):
    o = oracle.TGVOracle(*dims, params=oracle.FlowParams(mach=0.3, reynolds=400.0, filter_on=filt))
    o.set_q(q0)
    o.set_dt(dt)
    o.steps(steps)
    return o.get_q()


def _run(ctx, dims, q0, dt, steps, filt, pin=None):
    import astr_gpu_b200 as ag
    s = ag.TGVSolver(ctx, *dims, params=ag.FlowParams(mach=0.3, reynolds=400.0, filter_on=filt))
    s.autotune(False)
    if pin:
        s.set_launch_shape(*pin)
    s.set_q(q0)
    s.rk3(dt, steps)
    q = s.get_q()
    s.close()
    return q


def _err(a, b):
    return max(np.abs(a[..., m] - b[..., m]).max() / np.abs(b[..., m]).max() for m in range(5))


@pytest.mark.parametrize("dims", [(16, 16, 16), (17, 20, 38), (31, 39, 19), (32, 83, 44), (33, 84, 16), (47, 16, 84),
                                  (16, 257, 39), (20, 258, 38), (15 + 16, 60, 258), (16, 20, 300), (16, 1050, 16),
                                  (600, 17, 18),
                                  # the x passes: rows per chunk, lines per CTA, the widest boxes
                                  (38, 16, 17), (39, 17, 16), (42, 23, 17), (43, 24, 16), (99, 17, 16), (100, 18, 16),
                                  (169, 16, 16), (170, 25, 16), (201, 16, 17), (202, 17, 16), (297, 19, 16), (298, 16, 16),
                                  (622, 17, 16), (623, 16, 17), (822, 16, 16), (823, 17, 16), (1049, 16, 16),
                                  (1050, 16, 17)])
@pytest.mark.parametrize("filt", [True, False])
def test_boxes(ctx, dims, filt):
    q0 = _start(dims, sum(dims))
    dt = 0.3 / ((1.5 + 1 / 0.3) * sum(n / (2 * np.pi) for n in dims))
    assert _err(_run(ctx, dims, q0, dt, 2, filt), _oracle(dims, q0, dt, 2, filt)) <= TOL


@pytest.mark.parametrize("name", ["A", "B", "C", "A'", "B'", "F_C", "F_A"])
def test_one_pass_on_its_lane_scan_kernel(ctx, name):
    """The two forms of a pass can be mixed: the primitives are stored by whichever gradient pass runs
    as a column solve first."""
    dims = (40, 56, 48)
    q0 = _start(dims, 1)
    pin = (name, 3, 1, 4)
    assert _err(_run(ctx, dims, q0, 2e-3, 2, True, pin), _run(ctx, dims, q0, 2e-3, 2, True)) <= TOL


def test_reported_shapes(ctx):
    import astr_gpu_b200 as ag
    s = ag.TGVSolver(ctx, 32, 128, 300)
    sh = s.launch_shapes()
    assert sh["A"] == (33, 0, 32, 0, 1, 1) and sh["B"] == (33, 0, 16, 0, 1, 1) and sh["C"] == (9, 0, 8, 0, 1, 5) and sh["F_C"] == (9, 0, 8, 0, 1, 1)
    s.set_launch_shape("B", 9, 2, 8)
    assert s.launch_shapes()["B"][:3] == (9, 2, 8)
    s.close()


def test_tuning_leaves_the_filter_where_the_caller_put_it(ctx):
    """split_filter(False), then autotune(True): the tuned step still applies the filter along y in
    pass A (the timings then hold no launch of it as a pass of its own)."""
    import ctypes
    import astr_gpu_b200 as ag
    s = ag.TGVSolver(ctx, 40, 64, 32)   # 71 rows along y: the smallest layout is a candidate
    s.split_filter(False)
    s.autotune(True)
    s.init_tgv()
    s.rk3(1e-3, 2)
    ms = (ctypes.c_double * 8)()
    ctx.check(ctx.L.astr_pass_timings(s._h, 1e-3, 1, ms))
    assert ms[0] > 0.0 and ms[7] == 0.0
    s.close()
