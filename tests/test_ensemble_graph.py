"""The ensemble step as one graph of parallel branches: more boxes than branches, a box on lane-scan
kernels (whose update takes the time step by value), and changes of the time steps between calls all
give the states of the same boxes stepped alone, bit for bit (the same kernels run)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _boxes(ctx, sizes, pin=None):
    import astr_gpu_b200 as ag
    out = []
    for i, n in enumerate(sizes):
        s = ag.TGVSolver(ctx, n, params=ag.FlowParams(mach=0.2, reynolds=300.0 + 10 * i))
        if i == pin:
            s.set_launch_shape("B'", 3, 1, 4)
        s.init_tgv()
        out.append(s)
    return out


@pytest.mark.parametrize("sizes,pin", [([16 + k % 9 for k in range(37)], None), ([40, 16, 33, 24], 2), ([20], None)])
def test_graph_equals_boxes_alone(sizes, pin):
    import astr_gpu_b200 as ag
    ctx = ag.Context(0)
    alone, together = _boxes(ctx, sizes, pin), _boxes(ctx, sizes, pin)
    dt = np.array([0.05 / n for n in sizes])
    ens = ag.Ensemble(ctx, together)
    for steps, f in ((2, 1.0), (1, 0.5), (2, 0.5), (1, 1.0)):
        ens.step(dt * f, steps)
        for s, d in zip(alone, dt * f):
            s.rk3(d, steps)
    _equal(alone, together)
    ens.close()


def _equal(alone, together):
    for a, b in zip(alone, together):
        np.testing.assert_array_equal(a.get_q(), b.get_q())
        np.testing.assert_array_equal(a.history(), b.history())


def test_time_steps_changed_by_a_call_of_no_steps():
    """The new time steps reach every box also when the call that brings them makes no step."""
    import astr_gpu_b200 as ag
    ctx = ag.Context(0)
    sizes = [24, 16, 40]
    alone, together = _boxes(ctx, sizes, 0), _boxes(ctx, sizes, 0)
    dt = np.array([0.05 / n for n in sizes])
    ens = ag.Ensemble(ctx, together)
    for steps, f in ((2, 1.0), (0, 0.5), (1, 0.5), (0, 2.0), (0, 0.25), (2, 0.25)):
        ens.step(dt * f, steps)
        for s, d in zip(alone, dt * f):
            s.rk3(d, steps)
    _equal(alone, together)
    ens.close()


@pytest.mark.parametrize("change", [lambda s: s.set_launch_shape("A'", 3, 1, 4), lambda s: s.split_filter(False)])
def test_shapes_changed_after_the_first_step(change):
    """A box's passes run in the form it is set to, also when the ensemble has stepped it before."""
    import astr_gpu_b200 as ag
    ctx = ag.Context(0)
    sizes = [24, 33]
    alone, together = _boxes(ctx, sizes), _boxes(ctx, sizes)
    dt = np.array([0.05 / n for n in sizes])
    ens = ag.Ensemble(ctx, together)
    for _ in range(2):
        ens.step(dt, 3)
        for s, d in zip(alone, dt):
            s.rk3(d, 3)
        change(alone[1])
        change(together[1])
    _equal(alone, together)
    ens.close()


@pytest.mark.parametrize("own", [True, False])
def test_creation_waits_for_no_queued_work(own):
    """Boxes and schemes are made while the context's stream (own) or the legacy stream is busy."""
    import torch
    import astr_gpu_b200 as ag
    side = torch.cuda.Stream()
    ctx = ag.Context(0, stream=side)
    make = lambda: (ag.TGVSolver(ctx, 24), ag.fd_scheme_initiate(ctx, "643c", 3, 48))  # noqa: E731
    keep = [make()]
    torch.cuda.synchronize()
    with torch.cuda.stream(side if own else torch.cuda.default_stream()):
        torch.cuda._sleep(1_000_000_000)   # about half a second
        busy = torch.cuda.Event()
        busy.record()
    keep.append(make())
    assert not busy.query()
    torch.cuda.synchronize()


def test_lane_scan_box_on_a_blocking_stream():
    """A stream that synchronises with the legacy stream: the tables of a box's lane-scan kernels are
    made before the step is captured."""
    import ctypes
    import torch
    import astr_gpu_b200 as ag
    torch.zeros(1, device="cuda")
    raw = ctypes.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(raw))) == 0
    ctx = ag.Context(0, stream=raw.value)
    sizes = [24, 16]
    alone, together = _boxes(ctx, sizes, 1), _boxes(ctx, sizes, 1)
    dt = np.array([0.05 / n for n in sizes])
    ens = ag.Ensemble(ctx, together)
    ens.step(dt, 2)
    for s, d in zip(alone, dt):
        s.rk3(d, 2)
    _equal(alone, together)
    ens.close()
    for s in alone + together:
        s.close()
    ctx.synchronize()
    ctx.close()
    torch.cuda.cudart().cudaStreamDestroy(raw.value)
