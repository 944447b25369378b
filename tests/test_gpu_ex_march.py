"""The direct-march operator kernels against plain numpy stencils at the sizes
where tiles and chunks end: extents below, at and beyond one tile (32 along k,
8 along j), odd remainders, chunks of one plane, all stencil widths, walls.

Tolerance: every output is a sum of at most 72 products; with unit roundoff
u = 1.1e-16 and terms bounded by the sum of absolute terms S, |error| <= 72 u S
per side.  S is at most 40 times the largest output on these white-noise fields
(weights sum to < 6/delta per direction, three directions), so 1e-12 of the
largest output bounds both sides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COEF = {2: (1.0,), 4: (4 / 3, -1 / 3), 6: (1.5, -0.6, 0.1), 8: (1.6, -0.8, 24 / 105, -8 / 280)}
TOL = 1e-12


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


class Ref:
    """central differences; y walls mirror with the sign of each component (Neumann 0: +, Dirichlet 0: -)"""

    def __init__(self, N, L, m, walls):
        c = COEF[m]
        self.walls, d = walls, [L[a] / N[a] for a in range(3)]
        self.a = [[c[i] / 2 / (i + 1) / d[x] for i in range(len(c))] for x in range(3)]
        self.b = [[c[i] / ((i + 1) * d[x]) ** 2 for i in range(len(c))] for x in range(3)]

    def sh(self, f, x, s, par):
        if x != 1 or not self.walls:
            return np.roll(f, -s, x)
        n = f.shape[1]
        j = np.arange(n) + s
        m = np.where(j < 0, -j, np.where(j >= n, 2 * (n - 1) - j, j))
        sign = np.where((j < 0) | (j >= n), par, 1.0)
        return f[:, m] * sign[None, :, None]

    def D(self, f, x, par=1):
        return sum(w * (self.sh(f, x, i + 1, par) - self.sh(f, x, -i - 1, par)) for i, w in enumerate(self.a[x]))

    def Q(self, f, x, par=1):
        return sum(2 * w * (self.sh(f, x, i, par) - self.sh(f, x, -i - 1, par)) for i, w in enumerate(self.a[x]))

    def lap(self, f, par=1):
        return sum(w * (self.sh(f, x, i + 1, par) + self.sh(f, x, -i - 1, par) - 2 * f)
                   for x in range(3) for i, w in enumerate(self.b[x]))

    def lap_f(self, nu, f, par=1):
        return sum(w * (self.sh(nu, x, i, 1) * (self.sh(f, x, i + 1, par) - f)
                        + self.sh(nu, x, -i - 1, 1) * (self.sh(f, x, -i - 1, par) - f))
                   for x in range(3) for i, w in enumerate(self.b[x]))

    def skew(self, V, f, pv, pf):
        r = f * sum(self.D(V[x], x, pv[x]) for x in range(3))
        for x in range(3):
            r = r + self.D(V[x] * f, x, pv[x] * pf) + V[x] * self.D(f, x, pf)
        return 0.5 * r


def close(got, want):
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("N,m,walls", [
    ((9, 8, 32), 6, 0), ((7, 9, 33), 6, 0), ((1, 5, 3), 6, 0), ((33, 47, 29), 6, 0), ((70, 17, 64), 2, 0),
    ((20, 24, 40), 4, 0), ((12, 31, 65), 8, 0), ((150, 7, 9), 6, 0), ((14, 16, 34), 6, 1), ((9, 9, 31), 8, 1)])
def test_operators(nova, N, m, walls):
    L = (2.0, 3.0, 2.5)
    M = nova.Mesh(N, L=L, m=m, walls=(0, walls, 0))
    R, rng = Ref(N, L, m, walls), np.random.default_rng(17)
    par = (1, -1, 1) if walls else (1, 1, 1)

    def field(nc):
        x = rng.standard_normal((nc,) + M.shape)
        return x, nova.Field(M, nc).upload_soa(x)
    U, fU = field(3)
    s, fs = field(1)
    T, fT = field(9)
    S, fS = field(6)
    if walls:
        bc = [0] * 18
        for c in range(3):
            bc[6 * c] = bc[1 + 6 * c] = 2 if c == 1 else 1
        fU.set_bc(bc)
    ex = nova.ex
    close(ex.grad(fs).download_soa(), np.stack([R.D(s[0], x) for x in range(3)]))
    close(ex.grad(fU).download_soa(), np.stack([R.Q(U[c], x, par[c]) for c in range(3) for x in range(3)]))
    close(ex.div(fU).download_soa()[0], sum(R.D(U[x], x, par[x]) for x in range(3)))
    g = {(c, x): R.Q(U[c], x, par[c]) for c in range(3) for x in range(3)}
    close(ex.curl(fU).download_soa(), np.stack([g[2, 1] - g[1, 2], g[0, 2] - g[2, 0], g[1, 0] - g[0, 1]]))
    close(ex.laplacian(0.3, fU).download_soa(), np.stack([0.3 * R.lap(U[c], par[c]) for c in range(3)]))
    close(ex.laplacian(fs, fU).download_soa(), np.stack([R.lap_f(s[0], U[c], par[c]) for c in range(3)]))
    close(ex.div(fU, fU).download_soa(), np.stack([R.skew(U, U[c], par, par[c]) for c in range(3)]))
    close(ex.div(fU, fs).download_soa()[0], R.skew(U, s[0], par, 1))
    close(ex.div(fT).download_soa(), np.stack([sum(R.D(T[3 * c + x], x) for x in range(3)) for c in range(3)]))
    q = ((0, 1, 2), (1, 3, 4), (2, 4, 5))
    close(ex.div(fS).download_soa(), np.stack([sum(R.D(S[q[c][x]], x) for x in range(3)) for c in range(3)]))
    close(ex.div(fs, fT).download_soa(), np.stack([sum(R.D(s[0] * T[3 * c + x], x) for x in range(3))
                                                   for c in range(3)]))
