"""The spectral solve's line transforms: every supported length along i, j and
k (nova_spec.cuh), remainders of rows and columns per block, and a mix with
lengths that fall back to cuFFT, against numpy.

Tolerance: both FFTs are accurate to about 6 u log2(N) <= 1e-14 of the norm
(u = 1.1e-16, N <= 2^17); the solve weighs modes by 1/k'^2, largest for the
lowest modes, which carry at least 1/sqrt(N) of a white right-hand side's norm
of up to 100 -- so 1e-12 of the solution's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = (16, 20, 24, 25, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 90, 96, 100, 108, 120, 128, 144, 150,
           160, 180, 192, 240, 256)


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


def k2(n, L, fold):
    c, d = (1.5, -0.6, 0.1), L / n
    i = np.arange(n)
    kk = np.where(2 * i < n, i, n - i) * (2 * np.pi / L) if fold else i[: n // 2 + 1] * (2 * np.pi / L)
    kp = sum(c[q] / (q + 1) * np.sin((q + 1) * kk * d) / d for q in range(3))
    return kp * kp


def reference(f, L):
    N = f.shape
    q = (k2(N[0], L[0], True)[:, None, None] + k2(N[1], L[1], True)[None, :, None] + k2(N[2], L[2], False)[None, None])
    h = np.fft.rfftn(f)
    h = np.where(q < 1e-16, 0.0, -h / np.where(q < 1e-16, 1.0, q))
    return np.fft.irfftn(h, s=N, axes=(0, 1, 2))


def check(nova, N):
    L = (2.0, 3.0, 2.5)
    f = np.random.default_rng(sum(N)).standard_normal(N)
    M = nova.Mesh(N, L=L)
    p = nova.Field(M, 1)
    s = nova.poisson(p)
    s.rhs(nova.Field(M, 1).upload_soa(f[None]))
    s.solve()
    want = reference(f, L)
    assert np.linalg.norm(p.download_soa()[0] - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("n", LENGTHS)
def test_length_along_each_axis(nova, n):
    for N in ((n, 16, 32), (16, n, 40), (20, 25, 2 * n)):
        check(nova, N)


@pytest.mark.parametrize("N", [(16, 16, 32), (25, 75, 90), (64, 45, 180), (17, 32, 64), (32, 33, 64), (32, 64, 65),
                               (128, 64, 62), (2, 2, 2), (1, 16, 32)])
def test_remainders_and_fallbacks(nova, N):
    check(nova, N)


@pytest.mark.parametrize("N", [(48, 40, 60), (32, 256, 64), (25, 256, 50), (30, 31, 64)])
def test_wall_solves_match_the_cufft_plans(nova, monkeypatch, N):
    """One step of a wall mesh in both Poisson modes with the line transforms and with NOVA_FFT=cufft.  The projection
    moves U by dt grad p: a relative 1e-12 of p is well under 1e-12 of U here."""
    rng = np.random.default_rng(3)
    U0 = rng.standard_normal((3, N[0], N[1] + 1, N[2]))
    bc = [0] * 18
    for c in range(3):
        bc[6 * c] = bc[1 + 6 * c] = 2 if c == 1 else 1
    for mode in ("fft", "dct"):
        out = []
        for env in ("own", "cufft"):
            monkeypatch.setenv("NOVA_FFT", env)
            M = nova.Mesh(N, walls=(0, 1, 0))
            U, p = nova.Field(M, 3).set_bc(bc).upload_soa(U0), nova.Field(M, 1).set_bc([1, 1] + [0] * 16)
            nova.advance(M, nova.run_desc(dt=1e-3, nu=1e-2, poisson=mode), U, p, nsteps=1, history=False)
            out.append((U.download_soa(), p.download_soa()))
        for a, b in zip(*out):
            assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
