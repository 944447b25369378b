"""The sums of a history row are a tree's: the kinetic energy against the same state's in
extended precision.

Each addition errs by at most u = 1.1e-16 of its result (rms u/sqrt(3), or less).  In a
tree the last addition errs so, the two before it by half as much in the mean square
of the total, and so on: sqrt(2) u/sqrt(3) = 9e-17 rms at most, and the two products
with 1/2 and 1/(N0 N1 N2) are exact for powers of two.  Adding 64 rows in order gives
sqrt(64/3) u/sqrt(3) = 3e-16 at most.  Over 24 states the rms of the former stays below
1.6e-16 (three standard deviations, 15% each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


def energy(U):
    x = U.reshape(-1).astype(np.longdouble)
    return 0.5 * (x * x).sum() / (x.size // 3)


@pytest.mark.parametrize("steps", [1, 2])  # the row of the last step (diagnostics kernel), and the stage kernel's
def test_energy_is_a_trees(nova, steps):
    err = []
    for n in (64, 128):
        x = np.arange(n) * 2 * np.pi / n
        X, Y, Z = np.meshgrid(x, x, x, indexing="ij")
        M = nova.Mesh((n, n, n))
        U, p = nova.Field(M, 3), nova.Field(M, 1)
        rd = nova.run_desc(dt=1e-4, nu=1e-3)
        for seed in range(12):
            g = np.random.default_rng(seed)
            a, b, c = 6.0 * g.random(3)
            U0 = np.stack([np.sin(X + a) * np.cos(Y + b) * np.cos(Z + c),
                           -np.cos(X + a) * np.sin(Y + b) * np.cos(Z + c), 0 * X])
            U0 += 1e-3 * g.standard_normal(U0.shape)
            U.upload_soa(U0)
            nova.advance(M, rd, U, p, nsteps=1, history=False)
            want = energy(U.download_soa())  # after step 1
            U.upload_soa(U0)
            h = nova.advance(M, rd, U, p, nsteps=steps)
            err.append(float((np.longdouble(h[0, 2]) - want) / want))
    assert np.sqrt(np.mean(np.square(err))) < 1.6e-16
