"""The FP32 flux forms its face terms in FP32 and sums them per cell in FP64.  Lengths multiply
every term and leave the states alone, so a box scaled by a power of two has the terms of the unit
box, scaled without rounding, and meshes near the ends of FP32's range show what the sums hold."""
import numpy as np
import pytest

from fosolvers_gb300 import mesh as M
from fosolvers_gb300.euler import FLUX_FP32
from helpers import Case, perturbed, rel_err

pytestmark = pytest.mark.gpu


def box(cells, dims, length, jitter):
    m = M.box_mesh(*dims, extent=(length,) * 3, jitter=jitter, seed=1, cells=cells)
    st = M.freestream_state(dims[0] * dims[1] * dims[2] * (6 if cells == "tet" else 1), 1.0, 0.0, 1.0)
    return Case(M.Workload("box", m, st, np.zeros(0, np.int32), np.zeros(0, np.int32),
                           np.zeros((0, 5)), order=1, dt=1e-3, nsteps=1), flags=FLUX_FP32)


@pytest.mark.parametrize("cells,dims", [("tet", (4, 3, 5)), ("hex", (7, 5, 6))])
def test_rounding_errors_of_small_terms_are_kept(cuda, cells, dims):
    """At a length of 2^-48 the terms are near 2^-102: normal FP32 numbers (only one in a hundred
    million is too small to be one), whose sums in FP32 have rounding errors below the smallest
    normal number, 2^-126.  The residual is 2^48 times that of the unit box to 1e-10 of its
    largest; sums that lose those errors are about 2^-25 off."""
    f = []
    for e in (0, -48):
        c = box(cells, dims, 2.0 ** e, 0.0)
        y = perturbed(c.y0, c.nC, 3, amp=0.3)
        out = np.zeros_like(y)
        assert c.gpu.rhs(0.0, y, out) == 0
        f.append(np.ldexp(out, e).reshape(5, -1))
    for q in range(5):
        assert np.abs(f[0][q] - f[1][q]).max() <= 1e-10 * np.abs(f[0][q]).max()


@pytest.mark.parametrize("cells", ["tet", "hex"])
def test_sums_beyond_the_range_of_the_terms(cuda, cells):
    """A cell at twice its neighbours' pressure in a box so long that each of its faces' energy
    terms is an FP32 number and their sum, 2^128.8, is not: within 2e-5 of the FP64 oracle."""
    def case(length):
        c = box(cells, (3, 3, 3), length, 0.0)
        inner = np.flatnonzero(((c.grid.neib > 0) & (c.grid.neib <= c.nC)).sum(1) == (4 if cells == "tet" else 6))
        x = c.grid.p[inner] / length - 0.5
        y = c.y0.copy().reshape(5, -1)
        y[4, inner[np.argmin((x * x).sum(1))]] *= 2.0
        return c, y.reshape(-1)
    c, y = case(1.0)
    s = np.abs(c.oracle_rhs(y).reshape(5, -1) * c.grid.v[:c.nC]).max()
    c, y = case(float(np.sqrt(2.0 ** 128.8 / s)))
    ref = c.oracle_rhs(y)
    assert np.abs(ref.reshape(5, -1) * c.grid.v[:c.nC]).max() > 2.0 ** 128.5
    out = np.zeros_like(y)
    assert c.gpu.rhs(0.0, y, out) == 0
    assert rel_err(out, ref) <= 2e-5
