"""ILUT at the edges of its arguments: what ilut and lusol do there, the GPU class does too
(factors bit for bit the oracle's, solves within 1e-12, as in the tests of ordinary arguments)."""
import numpy as np
import pytest

from fosolvers_gb300 import mesh as M
from fosolvers_gb300.euler import PREC_ILUT
from helpers import Case, perturbed
from oracle import pyoracle as O
from test_gpu_ilut import assert_same_factors, gpu_ilu, oracle_ilut
from test_oracle_kat import _random_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("droptol", [-0.0, -1e-6, -np.inf])
@pytest.mark.parametrize("n,density,lfil", [(40, 0.15, 39), (200, 0.05, 10), (203, 0.3, 60)])
def test_drop_tolerance_below_zero_keeps_every_entry(cuda, n, density, lfil, droptol):
    """ilut drops |w| <= droptol |row| only, so nothing at a negative tolerance (zeros stored in
    the matrix neither), and -0.0 is 0."""
    _, a, ja, ia = _random_csr(n, density, n)
    a[::7] = np.where(np.abs(a[::7]) < 2.0, 0.0, a[::7])  # stored zeros off the diagonal
    ref = oracle_ilut(n, a, ja, ia, lfil, droptol)
    assert len(ref[0]) > 3 * n  # (an empty U would leave about 2 n)
    p = gpu_ilu(n, a, ja, ia, lfil, droptol)
    assert_same_factors(p, ref)
    if np.isfinite(droptol):
        y = np.random.default_rng(n).normal(size=n)
        xr = O.lusol(n, y, *ref)
        assert np.abs(p.solve(y) - xr).max() <= 1e-12 * np.abs(xr).max()


def test_context_drop_tolerance_of_minus_zero(cuda):
    """A context accepts -0.0 (it is not below 0) and preconditions as with 0."""
    m = M.box_mesh(4, 3, 5, jitter=0.1, seed=1, cells="tet")
    wl = M.Workload("box", m, M.sine_state(m.centroids(), 1), np.zeros(0, np.int32),
                    np.zeros(0, np.int32), np.zeros((0, 5)), order=2, dt=5e-4, nsteps=1)
    c = Case(wl, flags=PREC_ILUT)
    y = perturbed(c.y0, c.nC, 2)
    r = np.random.default_rng(2).normal(size=c.N)
    z = []
    for droptol in (0.0, -0.0):
        c.gpu.set_ilut(30, droptol)
        assert c.gpu.pset(0.0, y, None, 0, 5e-3)[0] == 0
        z.append(np.zeros_like(r))
        assert c.gpu.psol(0.0, y, None, r, z[-1], 5e-3) == 0
    assert np.array_equal(z[0], z[1])


@pytest.mark.parametrize("upper", [False, True], ids=["L", "U"])
@pytest.mark.parametrize("entry,y11", [(0.0, np.inf), (0.0, np.nan), (np.inf, 12.0)])
def test_factors_and_unknowns_that_are_not_finite(cuda, entry, y11, upper):
    """A negative tolerance keeps zeros in the factors, and 0 x inf is a NaN in the rows that have
    them, in lusol as here; an infinite entry makes its row infinite, not a NaN.  Rows depend on
    the rows three away (mostly of their group of five) and seven away."""
    n = 23
    ia, ja, a = [1], [], []
    for i in range(n):
        cols = {i: 2.0}
        for d in (3, 7):
            j = i + d if upper else i - d
            if 0 <= j < n:
                cols[j] = entry if entry == 0.0 or j == 11 else 0.25
        ja += [j + 1 for j in sorted(cols)]
        a += [cols[j] for j in sorted(cols)]
        ia.append(len(ja) + 1)
    a, ja, ia = np.array(a), np.array(ja, np.int32), np.array(ia, np.int32)
    ref = oracle_ilut(n, a, ja, ia, 5, -1.0)
    p = gpu_ilu(n, a, ja, ia, 5, -1.0)
    assert_same_factors(p, ref)
    y = np.arange(1.0, n + 1)
    y[11] = y11
    xr = O.lusol(n, y, *ref)
    assert (~np.isfinite(xr)).sum() > 3 and np.isfinite(xr).sum() > 3
    np.testing.assert_allclose(p.solve(y), xr, rtol=1e-12)


@pytest.mark.parametrize("first", [False, True], ids=["refactor", "first"])
def test_solves_are_refused_after_the_ordering_ran_out(cuda, first):
    """Upper triangular: no row waits in the factor, but the claim order of the backward sweep
    waits for the level of a row that is withheld.  The factor call reports it and a solve has no
    order to go by; published again, the same object factors and solves."""
    n = 1000
    ia = np.concatenate([[1], np.cumsum(np.minimum(n - np.arange(n), 7)) + 1]).astype(np.int32)
    ja = np.concatenate([np.arange(i, min(n, i + 7)) + 1 for i in range(n)]).astype(np.int32)
    a = np.random.default_rng(1).normal(size=len(ja))
    a[ia[:-1] - 1] = 9.0
    ref = oracle_ilut(n, a, ja, ia, 9, 0.0)
    y = np.random.default_rng(2).normal(size=n)
    xr = O.lusol(n, y, *ref)
    import torch
    from fosolvers_gb300.ilut import ILU
    dev = lambda x, t: torch.from_numpy(np.ascontiguousarray(x, t)).cuda()
    csr = (dev(ia - 1, np.int32), dev(ja - 1, np.int32), dev(a, np.float64))
    p = ILU(n, 9)
    if not first:
        p.factor_csr(*csr, 0.0)
        assert np.abs(p.solve(y) - xr).max() <= 1e-12 * np.abs(xr).max()
    p.set_wait_limit(polls=4096, withhold_row=700)
    with pytest.raises(RuntimeError, match="dependency wait ran out"):
        p.factor_csr(*csr, 0.0)
    with pytest.raises(RuntimeError, match="no factorisation"):
        p.solve(y)
    p.set_wait_limit(0, -1)
    p.factor_csr(*csr, 0.0)
    assert_same_factors(p, ref)
    assert np.abs(p.solve(y) - xr).max() <= 1e-12 * np.abs(xr).max()


@pytest.mark.parametrize("n,density", [(5, 0.3), (203, 0.02), (701, 0.01)])
def test_levels_are_read_while_a_stream_is_captured(cuda, n, density):
    """fos_ilut_info reads what the factor call left: the levels of the graphs of rows, equal to
    those counted from the factors, also while a stream that waits for the default one is being
    captured (when work on the default stream is an error and ends the capture)."""
    import ctypes as C
    from fosolvers_gb300 import _lib
    rt = C.CDLL("libcudart.so.13")  # (the one that torch has loaded)
    _, a, ja, ia = _random_csr(n, density, 3)
    p = gpu_ilu(n, a, ja, ia, n, 0.0)
    info = (C.c_long * 6)()
    stream, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 0) == 0
    rc = _lib.lib().fos_ilut_info(p.handle, info)
    ended = rt.cudaStreamEndCapture(stream, C.byref(graph))
    rt.cudaGetLastError()
    if ended == 0:
        rt.cudaGraphDestroy(graph)
    rt.cudaStreamDestroy(stream)
    assert (rc, ended) == (0, 0)
    _, jlu, ju = p.msr()
    lo, up = np.zeros(n, int), np.zeros(n, int)
    for i in range(n):
        lo[i] = 1 + max([lo[c - 1] for c in jlu[jlu[i] - 1:ju[i] - 1]], default=0)
    for i in reversed(range(n)):
        up[i] = 1 + max([up[c - 1] for c in jlu[ju[i] - 1:jlu[i + 1] - 1]], default=0)
    assert (info[4], info[5]) == (lo.max(), up.max())


def test_two_threads_with_rows_of_different_lengths(cuda):
    """Factorisations of short and of long rows (working capacities of 256 and 1024 entries, so
    launches with different amounts of shared memory) by two threads at a time, each on a stream
    of its own: every one succeeds, with the oracle's factors."""
    import threading
    import torch
    from fosolvers_gb300.ilut import ILU
    errors = []

    def work(n, dense, rounds):
        try:
            A = np.diag(4.0 + np.arange(n) % 3).astype(float)
            A[:dense] += 0.01 * (1.0 + np.arange(n) % 7)
            a, ja = A[A != 0], np.nonzero(A)[1].astype(np.int32)
            ia = np.concatenate([[0], np.cumsum((A != 0).sum(1))]).astype(np.int32)
            ref = oracle_ilut(n, a, ja + 1, ia + 1, n, 0.0)
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                csr = tuple(torch.from_numpy(x).cuda() for x in (ia, ja, a))
                stream.synchronize()
                for _ in range(rounds):
                    p = ILU(n, n)
                    p.factor_csr(*csr, 0.0, stream=stream)
                assert_same_factors(p, ref)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in ((40, 2, 400), (700, 2, 60))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("below,above", [(0, 7), (7, 0), (1, 1), (3, 4)])
@pytest.mark.parametrize("n,lfil", [(40003, 8), (40003, 40)])
def test_orders_of_chains(cuda, n, lfil, below, above):
    """Bands: every row depends on the one next to it, so the graphs are chains, whose levels the
    host counts where that is faster (the narrow storage) and the device elsewhere."""
    import ctypes as C
    from fosolvers_gb300 import _lib
    d = np.arange(-below, above + 1)
    ja = np.arange(n)[:, None] + d
    inside = (ja >= 0) & (ja < n)
    a = np.where(d == 0, 9.0, np.random.default_rng(n).uniform(-1.0, 1.0, ja.shape))[inside]
    ia = np.concatenate([[1], 1 + np.cumsum(inside.sum(1))]).astype(np.int32)
    ja = ja[inside].astype(np.int32) + 1
    ref = oracle_ilut(n, a, ja, ia, lfil, 1e-3)
    p = gpu_ilu(n, a, ja, ia, lfil, 1e-3)
    assert_same_factors(p, ref)
    _, jlu, ju = (x.tolist() for x in ref)
    lo, up = [0] * (n + 1), [0] * (n + 1)
    for i in range(n):
        lo[i + 1] = 1 + max([lo[c] for c in jlu[jlu[i] - 1:ju[i] - 1]], default=0)
    for i in reversed(range(n)):
        up[i + 1] = 1 + max([up[c] for c in jlu[ju[i] - 1:jlu[i + 1] - 1]], default=0)
    info = (C.c_long * 6)()
    assert _lib.lib().fos_ilut_info(p.handle, info) == 0
    assert (info[4], info[5]) == (max(lo), max(up))
    y = np.random.default_rng(1).normal(size=n)
    xr = O.lusol(n, y, *ref)
    assert np.abs(p.solve(y) - xr).max() <= 1e-12 * np.abs(xr).max()


def _stencil(nx, ny, nz):
    """7-point stencil in natural order: 0-based CSR."""
    n = nx * ny * nz
    i = np.arange(n)
    x, y, z = i % nx, i // nx % ny, i // (nx * ny)
    ja = np.stack([i - nx * ny, i - nx, i - 1, i, i + 1, i + nx, i + nx * ny], 1)
    inside = np.stack([z > 0, y > 0, x > 0, x >= 0, x < nx - 1, y < ny - 1, z < nz - 1], 1)
    a = np.where(np.arange(7) == 3, 6.1, -1.0) * np.ones((n, 1))
    return (np.concatenate([[0], np.cumsum(inside.sum(1))]).astype(np.int32),
            ja[inside].astype(np.int32), a[inside])


def _random_triangle(n, per_row, upper):
    rng = np.random.default_rng(n)
    ia, ja, a = [0], [], []
    for i in range(n):
        lo, hi = (i + 1, n) if upper else (0, i)
        cols = np.unique(np.concatenate([[i], rng.integers(lo, hi, min(per_row, hi - lo)) if hi > lo else []]))
        ja += cols.astype(int).tolist()
        a += [12.0 if c == i else rng.uniform(-1.0, 1.0) for c in cols]
        ia.append(len(ja))
    return np.array(ia, np.int32), np.array(ja, np.int32), np.array(a)


# the sweeps take rows one at a time, or groups of five where these make few enough levels: both, one
# of each, and a diagonal on either side of the size where that is decided
SWEEPS = {
    "stencil": (lambda: _stencil(13, 14, 15), 8, 1e-4),
    "stencil, groups forward": (lambda: _stencil(41, 5, 3), 60, 0.0),
    "lower": (lambda: _random_triangle(5003, 4, False), 9, 1e-3),
    "upper": (lambda: _random_triangle(5003, 4, True), 9, 1e-3),
    "wide rows": (lambda: _random_triangle(701, 90, False), 120, 0.0),
    "diagonal 1": (lambda: _random_triangle(1, 0, False), 3, 0.0),
    "diagonal 3000": (lambda: _random_triangle(3000, 0, False), 3, 0.0),
    "diagonal 3200": (lambda: _random_triangle(3200, 0, False), 3, 0.0),
}


@pytest.mark.parametrize("name", SWEEPS)
def test_sweeps_by_rows_and_by_groups(cuda, name):
    make, lfil, droptol = SWEEPS[name]
    ia, ja, a = make()
    n = len(ia) - 1
    lfil = max(1, min(lfil, n - 1))
    ref = oracle_ilut(n, a, ja + 1, ia + 1, lfil, droptol) if n > 1 else None
    p = gpu_ilu(n, a, ja + 1, ia + 1, lfil, droptol)
    y = np.random.default_rng(1).normal(size=n)
    xr = O.lusol(n, y, *ref) if n > 1 else y / a
    if n > 1:
        assert_same_factors(p, ref)
    for _ in range(3):
        assert np.abs(p.solve(y) - xr).max() <= 1e-12 * np.abs(xr).max()


def test_solves_take_the_time_of_the_levels_of_rows(cuda):
    """A stencil whose rows five in a row do not belong together: 500 levels of rows, and 6,300 of
    groups of five.  A level takes 2-3 us, so a solve stays below 8 us a level of rows."""
    import torch
    from fosolvers_gb300.ilut import ILU
    ia, ja, a = _stencil(27, 28, 29)
    n = len(ia) - 1
    p = ILU(n, 5)
    p.factor_csr(*(torch.from_numpy(v).cuda() for v in (ia, ja, a)), 1e-3)
    _, jlu, ju = (v.tolist() for v in p.msr())
    lo, up = [1] * n, [1] * n
    for i in range(n):
        lo[i] = 1 + max([lo[c - 1] for c in jlu[jlu[i] - 1:ju[i] - 1]], default=0)
    for i in reversed(range(n)):
        up[i] = 1 + max([up[c - 1] for c in jlu[ju[i] - 1:jlu[i + 1] - 1]], default=0)
    y = torch.ones(n, dtype=torch.float64, device="cuda")
    x = torch.empty_like(y)
    times = []
    for _ in range(8):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        p.solve_dev(y, x)
        e[1].record()
        torch.cuda.synchronize()
        times.append(e[0].elapsed_time(e[1]) * 1e3)
    assert min(times) <= 8.0 * (max(lo) + max(up))


@pytest.mark.parametrize("upper", [False, True], ids=["L", "U"])
@pytest.mark.parametrize("entry,y11", [(0.0, np.inf), (0.0, np.nan), (np.inf, 12.0)])
def test_unknowns_that_are_not_finite_in_groups(cuda, entry, y11, upper):
    """Zeros that a negative tolerance keeps, and an infinite entry, where every row reads the one
    next to it (a chain, which is swept in groups) and the one seven away."""
    n = 23
    ia, ja, a = [0], [], []
    for i in range(n):
        cols = {i: 2.0}
        for d in (1, 7):
            j = i + d if upper else i - d
            if 0 <= j < n:
                cols[j] = entry if j == 11 and d == 1 or (entry == 0.0 and d == 7) else 0.25
        ja += sorted(cols)
        a += [cols[j] for j in sorted(cols)]
        ia.append(len(ja))
    a, ja, ia = np.array(a), np.array(ja, np.int32) + 1, np.array(ia, np.int32) + 1
    ref = oracle_ilut(n, a, ja, ia, 5, -1.0)
    p = gpu_ilu(n, a, ja, ia, 5, -1.0)
    assert_same_factors(p, ref)
    y = np.arange(1.0, n + 1)
    y[11] = y11
    xr = O.lusol(n, y, *ref)
    assert (~np.isfinite(xr)).sum() > 3 and np.isfinite(xr).sum() > 3
    np.testing.assert_allclose(p.solve(y), xr, rtol=1e-12)
