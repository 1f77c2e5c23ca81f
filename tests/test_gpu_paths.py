"""Edges of the kernels' tiles and both sides of the rules that choose between them, against the
oracle (or the other path of the library) with the tolerances of the tests of the same entry
points: 1e-11 / 2e-5 for an FP64 / FP32-flux residual, equality for the two FP32 set-ups, 1e-5
for FP32 factors, equality and 1e-12 for ILUT factors and solves, 1e-10 for a BDF step."""
import numpy as np
import pytest

from fosolvers_gb300 import mesh as M
from fosolvers_gb300.euler import FLUX_FP32, ILU_COLOR, ILU_FP32
from helpers import Case, perturbed, rel_err, with_all_conditions
from oracle import pyoracle as O
from test_gpu_bdf import gpu_run, oracle_run
from test_gpu_ilut import assert_same_factors, gpu_ilu, oracle_ilut

pytestmark = pytest.mark.gpu


def box(cells, dims, seed=1, nsteps=1):
    m = M.box_mesh(*dims, jitter=0.1, seed=seed, cells=cells)
    return M.Workload("box", m, M.sine_state(m.centroids(), seed), np.zeros(0, np.int32),
                      np.zeros(0, np.int32), np.zeros((0, 5)), order=2, dt=5e-4, nsteps=nsteps)


@pytest.mark.parametrize("flags,tol", [(0, 1e-11), (FLUX_FP32, 2e-5)])
@pytest.mark.parametrize("cells,dims", [("hex", (1, 1, 1)), ("hex", (2, 1, 1)), ("tet", (1, 1, 1)),
                                        ("hex", (5, 4, 7)), ("tet", (3, 5, 4))])
def test_boundary_faces_by_condition(cuda, cells, dims, flags, tol):
    """Boundary faces taken through the list sorted by condition, every condition present: a cell
    without interior faces, cells with several conditions, blocks that are not full."""
    c = Case(with_all_conditions(box(cells, dims)), flags=flags)
    y = perturbed(c.y0, c.nC, 4, amp=0.1)
    out = np.zeros_like(y)
    assert c.gpu.rhs(0.0, y, out) == 0
    assert rel_err(out, c.oracle_rhs(y)) <= tol


def _bar():
    from test_grid import bar_tet_mesh
    from fosolvers_gb300.euler import PolyFvGrid
    m = bar_tet_mesh()
    return M.Workload("bar", m, M.sod_state(PolyFvGrid.from_mesh(m).p), np.zeros(0, np.int32),
                      np.zeros(0, np.int32), np.zeros((0, 5)), 1, 1e-3, 1)


@pytest.mark.parametrize("cells,dims", [("hex", (3, 3, 3)), ("hex", (4, 4, 4)), ("hex", (13, 5, 1)),
                                        ("tet", (3, 3, 3)), ("tet", (8, 4, 2)), ("bar", None)])
def test_fp32_colours_at_tile_edges(cuda, cells, dims):
    """Colours of fewer than 32 rows, of a multiple of 32 and of a remainder: the one-kernel
    set-up's factors equal the two-kernel path's bit for bit, and the sweeps by colour agree
    with the oracle's factors in the same order."""
    c = Case(_bar() if cells == "bar" else box(cells, dims), flags=ILU_FP32 | ILU_COLOR)
    y = perturbed(c.y0, c.nC, 7)
    g = 4e-3
    c.match_ilu_order()
    assert c.gpu.pset(0.0, y, None, 0, g) == (0, 1)
    r = np.random.default_rng(3).normal(size=c.N)
    z_fused, z_two, z_ref = (np.zeros_like(r) for _ in range(3))
    assert c.gpu.psol(0.0, y, None, r, z_fused, g) == 0
    c.oracle.pset(0.0, y, None, 0, g)
    c.oracle.psol(0.0, None, None, r, z_ref, g)
    assert rel_err(z_fused, z_ref) <= 1e-5
    c.gpu.set_jacobian(c.gpu.jacobian()[2])
    assert c.gpu.pset(0.0, y, None, 1, g) == (0, 0)
    assert c.gpu.psol(0.0, y, None, r, z_two, g) == 0
    assert np.array_equal(z_fused, z_two)


@pytest.mark.parametrize("n,row,lfil,droptol,ties", [
    (6, 3, 2, 0.0, False), (33, 20, 7, 0.0, True),
    (203, 80, 20, 0.0, False), (204, 80, 33, 0.0, True), (331, 150, 3, 1e-8, False),
    (331, 150, 100, 1e-8, True)])
def test_ilut_split_and_sweep_edges(cuda, n, row, lfil, droptol, ties):
    """Rows of up to several hundred entries split down to a few and to many (with equal
    magnitudes too, where the split's order shows), and sizes that leave a block of five rows
    with one to four."""
    rng = np.random.default_rng(n + lfil)
    A = np.zeros((n, n))
    for i in range(n):
        j = rng.choice(n, min(row, n), replace=False)
        A[i, j] = rng.choice([-0.5, 0.25, 0.5], len(j)) if ties else rng.normal(size=len(j))
        A[i, i] = 2.0 * row + rng.integers(4)
    a, ja = A[A != 0], np.nonzero(A)[1].astype(np.int32) + 1
    ia = np.concatenate([[0], np.cumsum((A != 0).sum(1))]).astype(np.int32) + 1
    ref = oracle_ilut(n, a, ja, ia, lfil, droptol)
    p = gpu_ilu(n, a, ja, ia, lfil, droptol)
    assert_same_factors(p, ref)
    y = rng.normal(size=n)
    xr = O.lusol(n, y, *ref)
    assert np.abs(p.solve(y) - xr).max() <= 1e-12 * np.abs(xr).max()


@pytest.mark.parametrize("cells,dims,precond", [("hex", (3, 3, 3), 0), ("hex", (5, 5, 5), 1),
                                                ("tet", (7, 5, 3), 0), ("hex", (39, 39, 40), 1),
                                                ("hex", (40, 40, 40), 1)])
def test_krylov_sums_both_shapes(cuda, cells, dims, precond):
    """Sums of an odd number of unknowns, of less than a block of them, and of 304,200 and
    320,000: either side of 152 x 256 x 8, where the launch shape changes."""
    c = Case(box(cells, dims))
    kw = dict(newton_rtol=1e-11)
    y_ref, _ = oracle_run(c, use_prec=precond, **kw)
    y, st = gpu_run(c, precond=precond, **kw)
    assert st["n_lin_iters"] > st["n_newton"]
    assert rel_err(y, y_ref) <= 1e-10


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 3, 3), (4, 4, 4), (7, 6, 5)])
def test_gnn_edges_from_slots_equal_edges_from_faces(cuda, dims):
    """Tiles of 64 cells (partial, full, several) and chunks of 256: a context with the per-cell
    copies of the face data gives the bits of one without, which is within 2e-2 of the
    reference (BF16 roundings)."""
    import torch
    from fosolvers_gb300.learned import GNN
    from oracle import gnn_ref as R
    g = GNN(seed=2)
    w = g.params()
    w[R.OFF_D:R.OFF_DB] = 0.05 * np.random.default_rng(5).standard_normal(R.OFF_DB - R.OFF_D)
    g.set_params(w)
    z = []
    for flags in (0, FLUX_FP32):
        c = Case(with_all_conditions(box("tet", dims)), flags=flags)
        y = perturbed(c.y0, c.nC, 6)
        v = np.random.default_rng(6).standard_normal(c.N)
        yi, vi, zi, zr = (torch.empty(c.N, dtype=torch.float64, device="cuda") for _ in range(4))
        c.gpu.to_internal(torch.from_numpy(y).cuda(), yi)
        c.gpu.to_internal(torch.from_numpy(v).cuda(), vi)
        g.apply_dev(c.gpu, yi, vi, zi, 2e-3)
        c.gpu.to_reference(zi, zr)
        z.append(zr.cpu().numpy())
    assert np.array_equal(z[0], z[1])
    ref = R.forward(R.split(w), R.Graph(c.grid), y, v, 2e-3)
    assert np.linalg.norm(z[0] - ref) <= 2e-2 * np.linalg.norm(ref - v)
