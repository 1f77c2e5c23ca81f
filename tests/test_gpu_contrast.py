"""The FP64 residual and Jacobian on states of neighbouring cells that differ by orders of magnitude
(random densities, pressures and velocities), against the scheme in numpy's longdouble: their errors
stay those of a few roundings of the largest terms.  An average formed as u_L + w (u_R - u_L) does
not pass: where u_L is large and its weight small, it loses as many digits as they differ by."""
import numpy as np
import pytest

from fosolvers_gb300 import mesh as M
from helpers import Case

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(np.finfo(np.longdouble).eps > 2.0 ** -60, reason="no longer double")]

LD = np.longdouble
U = 2.0 ** -53
GAMMA, G1 = LD(1.4), LD(1.4) - 1


def case(cells, dims):
    m = M.box_mesh(*dims, jitter=0.1, seed=1, cells=cells)
    return Case(M.Workload("box", m, M.sine_state(m.centroids(), 1), np.zeros(0, np.int32),
                           np.zeros(0, np.int32), np.zeros((0, 5)), order=1, dt=1e-3, nsteps=1))


def states(nC, ratio):
    for seed in range(8):
        rng = np.random.default_rng(seed)
        rho, p = np.exp(np.log(ratio) * rng.uniform(-0.5, 0.5, (2, nC)))
        u = rng.normal(size=(3, nC)) * np.sqrt(p / rho)
        yield np.concatenate([[rho], rho * u, [p / 0.4 + 0.5 * rho * (u * u).sum(0)]]).reshape(-1)


class Faces:
    """Both sides' primitives and the Roe averages of every face, walls as mirrored states."""

    def __init__(self, g, y):
        y = y.astype(LD).reshape(5, -1)
        self.i = g.iEP.astype(int) - 1
        self.n, self.a, nPi = g.normP.astype(LD).T, g.aP.astype(LD), g.nPi
        left = y[:, self.i[:, 0]]
        right = left.copy()
        right[:, :nPi] = y[:, self.i[:nPi, 1]]
        nb = self.n[:, nPi:]
        right[1:4, nPi:] -= 2 * (right[1:4, nPi:] * nb).sum(0) * nb
        self.L, self.R = (self.prim(s) for s in (left, right))
        (rl, ul, pl, hl), (rr, ur, pr, hr) = self.L, self.R
        sl, sr = np.sqrt(rl), np.sqrt(rr)
        self.rho = sl * sr
        self.u, self.H = (sl * ul + sr * ur) / (sl + sr), (sl * hl + sr * hr) / (sl + sr)
        self.q = (self.u ** 2).sum(0) / 2
        self.c = np.sqrt(G1 * (self.H - self.q))
        self.vn = (self.u * self.n).sum(0)

    @staticmethod
    def prim(s):
        u = s[1:4] / s[0]
        p = G1 * (s[4] - (s[1:4] ** 2).sum(0) / s[0] / 2)
        return s[0], u, p, (s[4] + p) / s[0]

    def flows(self):
        (rl, ul, pl, hl), (rr, ur, pr, hr) = self.L, self.R
        uJ, pJ = ur - ul, pr - pl
        nJ = (uJ * self.n).sum(0)
        e = abs(self.vn) * (rr - rl - pJ / self.c ** 2)
        s = abs(self.vn) * self.rho
        d = np.concatenate([[e], e * self.u + s * (uJ - self.n * nJ),
                            [e * self.q + s * ((self.u * uJ).sum(0) - self.vn * nJ)]])
        for w in (-1, 1):
            k = abs(self.vn + w * self.c) * (pJ + w * self.rho * self.c * nJ) / (2 * self.c ** 2)
            d += k * np.concatenate([[1 + 0 * k], self.u + w * self.c * self.n,
                                     [self.H + w * self.c * self.vn]])
        ml, mr = rl * (ul * self.n).sum(0), rr * (ur * self.n).sum(0)
        f = np.concatenate([[ml + mr], ml * ul + mr * ur + (pl + pr) * self.n, [ml * hl + mr * hr]])
        return self.a / 2 * (f - d)

    def blocks(self, nPi):
        """Off-diagonal blocks (L, R) and (R, L) of the interior faces."""
        n, u, c, vn, av = (x[..., :nPi] for x in (self.n, self.u, self.c, self.vn, abs(self.vn)))
        A = np.zeros((nPi, 5, 5), LD)
        A[:, range(5), range(5)] = av[:, None]
        A[:, 1:4, 0] -= (av * u).T
        for w in (-1, 1):
            k = (abs(vn + w * c) - av) / (2 * c ** 2)
            row = np.concatenate([[G1 * self.q[:nPi] - w * c * vn], w * c * n - G1 * u, [G1 + 0 * c]])
            col = np.concatenate([[1 + 0 * c], u + w * c * n, [self.H[:nPi] + w * c * vn]])
            A += np.einsum("f,af,bf->fab", k, col, row)
        F = []
        for _, u, _, H in (self.L, self.R):
            u, H = u[:, :nPi], H[:nPi]
            vn, k = (u * n).sum(0), G1 * (u * u).sum(0) / 2
            B = np.zeros((nPi, 5, 5), LD)
            B[:, 0, 1:4] = n.T
            B[:, 1:4, 0] = (n * k - u * vn).T
            B[:, 1:4, 1:4] = (np.einsum("if,jf->fij", u, n) - G1 * np.einsum("if,jf->fij", n, u)
                              + vn[:, None, None] * np.eye(3))
            B[:, 1:4, 4] = G1 * n.T
            B[:, 4, 0], B[:, 4, 4] = (k - H) * vn, GAMMA * vn
            B[:, 4, 1:4] = (H * n - G1 * vn * u).T
            F.append(B)
        h = self.a[:nPi, None, None] / 2
        return h * (A - F[1]), h * (A + F[0])


@pytest.mark.parametrize("cells,dims", [("tet", (4, 3, 4)), ("hex", (6, 5, 4))])
@pytest.mark.parametrize("ratio", [10.0, 1e3, 1e6])
def test_residual(cuda, cells, dims, ratio):
    """Relative l2 error 4 units roundoff, largest error 10 units of its field's largest value."""
    c = case(cells, dims)
    l2, most = [], []
    for y in states(c.nC, ratio):
        f = Faces(c.grid, y)
        ref = np.zeros((5, c.nC), LD)
        for q, flow in enumerate(f.flows()):
            np.subtract.at(ref[q], f.i[:, 0], flow)
            np.add.at(ref[q], f.i[:c.grid.nPi, 1], flow[:c.grid.nPi])
        ref /= c.grid.v[:c.nC].astype(LD)
        out = np.zeros_like(y)
        assert c.gpu.rhs(0.0, y, out) == 0
        d = abs(out.reshape(5, -1) - ref)
        l2.append(np.sqrt((d ** 2).sum() / (ref ** 2).sum()))
        most.append((d / abs(ref).max(1, keepdims=True)).max())
    assert np.mean(l2) <= 4 * U
    assert np.mean(most) <= 10 * U


@pytest.mark.parametrize("cells,dims", [("tet", (4, 3, 4)), ("hex", (6, 5, 4))])
@pytest.mark.parametrize("ratio", [10.0, 1e3, 1e6])
def test_jacobian(cuda, cells, dims, ratio):
    """Relative error of a block (Frobenius norm) 5 units roundoff in the mean."""
    c = case(cells, dims)
    nPi, err = c.grid.nPi, []
    for y in states(c.nC, ratio):
        assert c.gpu.pset(0.0, y, None, 0, 1e-9)[0] == 0
        rowptr, col, val = c.gpu.jacobian()
        f = Faces(c.grid, y)
        at = c.gpu.ilu_order()[f.i[:nPi]]
        for (p, q), ref in zip((at.T, at.T[::-1]), f.blocks(nPi)):
            slot = [rowptr[a] + np.searchsorted(col[rowptr[a]:rowptr[a + 1]], b) for a, b in zip(p, q)]
            d = np.sqrt(((val[slot] - ref) ** 2).sum((1, 2)) / (ref ** 2).sum((1, 2)))
            err.append(d.mean())
    assert np.mean(err) <= 5 * U
