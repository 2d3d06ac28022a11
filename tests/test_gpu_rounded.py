"""The sweeps, the stage combine and the CT update where their rounded-quotient
forms switch to the plain operators, and at the edges of the x sweep's tiles:
bit for bit against the FP64 oracle.

* numerators that fade through the denormals (a faint velocity in a field at rest);
* densities and pressures outside [2^-200, 2^200);
* boxes longer than 65,535 planes or tiles of a grid dimension;
* row lengths around multiples of the x sweep's 58 faces, odd and even, down
  to the smallest box.
"""
import numpy as np
import pytest

from cumpic_b200 import _native as N
from cumpic_b200 import problems as P
from compare import diffs

pytestmark = pytest.mark.gpu

STEPS = 4


def _check(p, steps=STEPS):
    from cumpic_b200.solver import CUMC3D
    from _oracle import Oracle
    g, o = CUMC3D(p), Oracle(p, threads=8)
    for s in (g, o):
        s.upload()
        s.initial_update()
    for n in range(steps):
        dg, do = g.finddt(), o.finddt()
        assert dg == do, (n, dg, do)
        g.rungekutta(dg)
        o.rungekutta(do)
    d = diffs(g.download(), o.download())
    bad = {k: v for k, v in d.items() if v != 0.0}
    assert not bad, bad


@pytest.mark.parametrize("recon", [N.PPMC, N.TVDMM], ids=["ppm", "tvd"])
@pytest.mark.parametrize("amp", [1e-140, 1e-155, 1e-290, 1e-307, 1e-318])
def test_faint_velocities(amp, recon):
    p = P.orszag_tang(13, ny=12, nz=9, recon=recon)
    p.prim[..., P.IVX:P.IVZ + 1] *= amp
    p.prim[..., P.IBX:P.IBZ + 1] = 0.0
    p.prim[..., P.IBZ] = 1e-3 * p.prim[..., P.IRHO]
    _check(p)


@pytest.mark.parametrize("scale", [1e-80, 1e-61, 1e-60, 1e60, 1e61, 1e80])
def test_densities_outside_the_range(scale):
    p = P.orszag_tang(12, ny=9, nz=10)
    p.prim[..., [P.IRHO, P.ITAU]] *= scale
    p.prim[..., P.IBX:P.IBZ + 1] *= np.sqrt(scale)
    _check(p)


@pytest.mark.parametrize("nx", [3, 4, 22, 23, 51, 52, 53, 58, 109, 110, 111, 168])
def test_row_lengths(nx):
    _check(P.orszag_tang(nx, ny=5, nz=4))


@pytest.mark.parametrize("axis,n", [(2, 65_600), (1, 262_200), (0, 70_000)], ids=["z", "y", "x"])
def test_long_thin_boxes(axis, n):
    shape = [3, 3, 3]
    shape[axis] = n
    _check(P.brio_wu(*shape, axis=axis), steps=1)
