"""rcp64 and rsqrt64 (fos_device.cuh), which take the place of the division and square
root operators, against those operators (numpy's: correctly rounded).

Bounds.  rcp64 rounds once after a step that leaves 2^-60, so it is the correctly rounded value or
its neighbour; rsqrt64's product a y is rounded before, which adds half a unit in the last place to
both of its results: neighbours too for the root (1 unit at most), and 1/sqrt is compared with
1 / sqrt(x), itself rounded twice (2 units).  rcp64 is the division for zeros, infinities and NaN."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from fosolvers_gb300 import mesh as M
from fosolvers_gb300.euler import ILU_COLOR, ILU_FP32
from helpers import Case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def recips(cuda, tmp_path_factory):
    import torch
    from fosolvers_gb300 import build as b
    so = tmp_path_factory.mktemp("recips") / "recips.so"
    src = b.HERE.parent / "tests" / "reciprocals.cu"
    r = subprocess.run([b._nvcc(), "-std=c++17", "-O3", *b.ARCH, "-I", str(b.CSRC), "-I",
                        str(b.HERE.parent / "include"), "-shared", "-Xcompiler", "-fPIC", str(src),
                        "-o", str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(so))
    lib.recips.argtypes = [C.c_long, C.c_void_p, C.c_void_p]

    def run(x):
        xd = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        out = torch.empty(4 * len(x), dtype=torch.float64, device="cuda")
        assert lib.recips(len(x), xd.data_ptr(), out.data_ptr()) == 0
        return out.cpu().numpy().reshape(4, -1)
    return run


def ulps(a, b):  # numbers of one sign: the distance of their bit patterns
    assert np.array_equal(np.signbit(a), np.signbit(b))
    return np.abs(a.view(np.int64) - b.view(np.int64)).max()


def numbers(lo, hi, each, seed):
    """Exponent fields lo .. hi, each with random significands, the power of two, its neighbours
    above and the significands of (all but) ones, of both signs."""
    rng = np.random.default_rng(seed)
    e = np.arange(lo, hi + 1, dtype=np.uint64)
    m = rng.integers(0, 1 << 52, (len(e), each), dtype=np.uint64)
    edge = np.array([0, 1, 2, (1 << 52) - 1, (1 << 52) - 2, 1 << 51], np.uint64)
    m = np.concatenate([m, np.broadcast_to(edge, (len(e), 6))], axis=1)
    x = ((e[:, None] << np.uint64(52)) | m).reshape(-1).view(np.float64)
    return np.concatenate([x, -x])


def test_normal_numbers(recips):
    x = numbers(1, 2044, 500, 1)
    out = recips(x)
    assert ulps(out[0], 1.0 / x) <= 1
    assert np.array_equal(out[0], out[3])
    p = x > 0
    assert ulps(out[2][p], np.sqrt(x[p])) <= 1
    assert ulps(out[1][p], 1.0 / np.sqrt(x[p])) <= 2
    assert np.isnan(out[1][~p]).all() and np.isnan(out[2][~p]).all()


def test_near_one(recips):
    """The significands next to a power of two, where one unit in the last place doubles."""
    x = (np.float64(1.0).view(np.int64) + np.arange(-200000, 200000)).view(np.float64)
    out = recips(x)
    assert ulps(out[0], 1.0 / x) <= 1
    assert ulps(out[2], np.sqrt(x)) <= 1


def test_arguments_that_are_not_normal(recips):
    """Zeros, infinities and NaN as the division has them; rcp64 takes subnormal arguments for
    zeros, and a reciprocal that is subnormal is zero or right to one unit (that of a number next
    to 2^1022 is: the seed does not see its last bits)."""
    rng = np.random.default_rng(4)
    sub = rng.integers(1, 1 << 52, 5000, dtype=np.uint64).view(np.float64)
    huge = numbers(2045, 2046, 500, 5)
    x = np.concatenate([[0.0, -0.0, np.inf, -np.inf, np.nan], sub, -sub])
    out = recips(x)
    with np.errstate(all="ignore"):
        ref = 1.0 / np.where(np.abs(x) < 2.0 ** -1022, np.copysign(0.0, x), x)
    assert np.array_equal(out[0], ref, equal_nan=True)
    out = recips(huge)
    assert np.array_equal(np.signbit(out[0]), np.signbit(huge))
    some = out[0] != 0.0
    assert ulps(out[0][some], 1.0 / huge[some]) <= 1


@pytest.mark.parametrize("flags", [0, ILU_COLOR, ILU_COLOR | ILU_FP32])
def test_an_infinite_pivot_spoils_no_other_row(cuda, flags):
    """P = I but for one infinite diagonal entry: its row of the inverse is zero, and the others
    are those of I."""
    c = Case(M.make_workload("sod16", scale=4), flags=flags)
    g, gamma = c.gpu, 1e-3
    assert g.pset(0.0, c.y0, None, 0, gamma) == (0, 1)
    rowptr, col, val = g.jacobian()
    pos2old = np.argsort(g.ilu_order())
    p, a = c.nC // 2, 2
    val[:] = 0.0
    val[rowptr[p] + list(col[rowptr[p]:rowptr[p + 1]]).index(p), a, a] = -np.inf
    g.set_jacobian(val)
    assert g.pset(0.0, c.y0, None, 1, gamma) == (0, 0)
    r = np.random.default_rng(0).normal(size=c.N).astype(np.float32).astype(np.float64)
    z, ref = np.zeros_like(r), r.copy()
    assert g.psol(0.0, c.y0, None, r, z, gamma) == 0
    ref[a * c.nC + pos2old[p]] = 0.0
    assert np.array_equal(z, ref)
