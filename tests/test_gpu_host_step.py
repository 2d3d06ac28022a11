"""cumc_rungekutta's step as a graph: what another call, a caller's capture or
per-kernel timing between the steps must not change."""
import ctypes

import numpy as np
import pytest

from cumpic_b200 import _native as N
from cumpic_b200 import problems as P
from compare import diffs

pytestmark = pytest.mark.gpu


def _same(g, o):
    d = diffs(g.download(), o.download())
    bad = {k: v for k, v in d.items() if v != 0.0}
    assert not bad, bad


def _pair(p):
    from cumpic_b200.solver import CUMC3D
    from _oracle import Oracle
    g, o = CUMC3D(p), Oracle(p, threads=8)
    for s in (g, o):
        s.upload()
        s.initial_update()
    return g, o


def _steps(g, o, n):
    for _ in range(n):
        dg, do = g.finddt(), o.finddt()
        assert dg == do
        g.rungekutta(dg)
        o.rungekutta(do)


def _captured(g, work):
    """work() under a capture of the context's stream; returns the graph"""
    import torch
    s = ctypes.c_void_p()
    assert g._lib.cumc_get_stream(g._h, ctypes.byref(s)) == N.CUMC_OK
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(s.value), capture_error_mode="thread_local"):
        work()
    return graph


def test_replays_between_other_calls():
    g, o = _pair(P.orszag_tang(14, ny=12, nz=11))
    _steps(g, o, 4)
    g.advance(3)
    for _ in range(3):
        o.rungekutta(o.finddt())
    _same(g, o)
    _steps(g, o, 2)
    N_ = g._lib
    assert N_.cumc_profile(g._h, 1) == N.CUMC_OK
    _steps(g, o, 2)
    assert N_.cumc_profile(g._h, 0) == N.CUMC_OK
    _steps(g, o, 2)
    _same(g, o)
    for s in (g, o):  # a new state in the same context
        s.upload()
        s.initial_update()
    _steps(g, o, 3)
    _same(g, o)
    g.upload()
    g.adjoint(2, 1)
    o.upload()
    o.initial_update()
    for _ in range(2):
        o.rungekutta(o.finddt())
    _steps(g, o, 3)
    _same(g, o)


def test_step_under_a_callers_capture():
    import torch
    g, o = _pair(P.orszag_tang(12, ny=9, nz=10))
    _steps(g, o, 3)
    dt = g.finddt()
    assert dt == o.finddt()
    graph = _captured(g, lambda: g.rungekutta(dt))
    torch.cuda.synchronize()
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    o.rungekutta(dt)
    o.rungekutta(dt)
    _same(g, o)
    _steps(g, o, 2)
    _same(g, o)


def test_dt_after_a_capture_that_never_ran():
    """a captured step leaves no CFL step behind until its graph runs"""
    g, o = _pair(P.orszag_tang(12, ny=9, nz=10))
    _captured(g, lambda: g.rungekutta(1e-4))
    assert g.finddt() == o.finddt()


def test_l_rk_is_stale_after_a_step():
    """cumc_download_lrk refuses an l_rk that a step has outdated, also where
    the step's launches come from a graph"""
    from cumpic_b200.solver import CUMC3D
    g = CUMC3D(P.orszag_tang(10, ny=9, nz=8))
    g.upload()
    g.initial_update()
    out = np.empty(g.shape + (8,))
    ptr = out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    for move in (lambda: g.rungekutta(g.finddt()), lambda: g.advance(1)):
        for _ in range(10):
            move()
            assert g._lib.cumc_download_lrk(g._h, ptr) == N.CUMC_ERR_STATE
            g.spatial()
            assert g._lib.cumc_download_lrk(g._h, ptr) == N.CUMC_OK


@pytest.mark.parametrize("coordinate", [N.CYLINDRICAL, N.SPHERICAL], ids=["cylindrical", "spherical"])
@pytest.mark.parametrize("scale,amp", [(1e-61, 1.0), (1e-60, 1.0), (1e60, 1.0), (1e61, 1.0), (1.0, 1e-155),
                                       (1.0, 1e-290), (1.0, 1e-318)])
def test_range_edges_on_curvilinear_grids(coordinate, scale, amp):
    """the quotient groups of the combine and the CT curl where their operands
    leave the range (faint velocities, extreme densities and pressures)"""
    p = P.shell(coordinate, 13, 12, 9)
    p.prim[..., [P.IRHO, P.ITAU]] *= scale
    p.prim[..., P.IBX:P.IBZ + 1] *= np.sqrt(scale) if amp == 1.0 else 0.0
    p.prim[..., P.IVX:P.IVZ + 1] *= amp
    g, o = _pair(p)
    _steps(g, o, 3)
    _same(g, o)


def test_negative_radii():
    """radii below zero in the inner cells: negative divisors"""
    p = P.shell(N.CYLINDRICAL, 12, 9, 8)
    p.xf = P.uniform_faces(-0.3, 1.2, 12)
    g, o = _pair(p)
    for _ in range(3):
        g.rungekutta(1e-4)
        o.rungekutta(1e-4)
    _same(g, o)


def test_steps_beside_another_streams_capture():
    """a capture that the caller has open on a stream of its own (global mode)
    survives the step whose graph is made"""
    import torch
    g, o = _pair(P.orszag_tang(12, ny=9, nz=10))
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x += 1.0
        for _ in range(9):
            g.rungekutta(1e-3)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 1.0
    for _ in range(9):
        o.rungekutta(1e-3)
    _same(g, o)
