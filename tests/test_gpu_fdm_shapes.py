"""The implicit solve's residual and line sweeps at the shapes where their
blocks change: rows of 32..256 and more nodes per thread group, remainders of
the row groups, and line counts on both sides of one wave of blocks (444 and
592 of 32 lines).  Reference: numpy's residual of the downloaded matrix (sums of
at most 2^21 positive terms: relative 1e-12), and the exact FFT solution of the
constant-coefficient system after convergence (1e-11, as the existing solve
test)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


@pytest.mark.parametrize("N", [(3, 5, 7), (9, 10, 33), (7, 6, 65), (5, 4, 130), (4, 5, 257), (111, 128, 16),
                               (148, 20, 128), (149, 24, 100)])
def test_residual_and_solution(nova, N):
    L, mu, c = (2.0, 1.5, 3.0), 1e-3, 2.0
    rng = np.random.default_rng(sum(N))
    x0, f = rng.standard_normal((1,) + N), rng.standard_normal((1,) + N)
    M = nova.Mesh(N, L=L)
    x = nova.Field(M, 1).upload_soa(x0)
    A = nova.im.laplacian(mu, x)
    A.add_diagonal(-c).eq(nova.Field(M, 1).upload_soa(f))
    al, ap, b = A.download()
    sh = [(1, -1), (1, 1), (0, -1), (0, 1), (2, -1), (2, 1)]
    r = b - ap * x0[0] - sum(al[q] * np.roll(x0[0], s, a) for q, (a, s) in enumerate(sh))
    w = [np.where(np.arange(n) == 0, 2.0, 1.0) for n in N]
    want = np.sqrt((r * r * w[0][:, None, None] * w[1][None, :, None] * w[2]).sum() / np.prod([n + 1 for n in N]))
    assert A.residual() == pytest.approx(want, rel=1e-12)
    its, res = A.solve(1e-13, 300)
    assert res <= 1e-13
    sym = ap.flat[0]
    for a, q in ((0, 2), (1, 0), (2, 4)):
        sym = sym + (al[q].flat[0] * 2 * np.cos(2 * np.pi * np.arange(N[a]) / N[a])).reshape(
            [-1 if y == a else 1 for y in range(3)])
    exact = np.fft.ifftn(np.fft.fftn(b) / sym).real
    got = x.download_soa()[0]
    assert np.linalg.norm(got - exact) <= 1e-11 * np.linalg.norm(exact)
