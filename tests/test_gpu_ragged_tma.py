"""The TMA-fed kernels on meshes whose last tile along k or j is ragged, down to
the three nodes a neighbour's halo needs, and on meshes they must leave to the
march (one or two nodes left over, odd rows).  The Navier-Stokes kernels do
the march's arithmetic in its order, so whole runs agree bit for bit; the MHD
and adjoint kernels contract other products (tests/test_gpu_stage_tma.py,
test_gpu_adjoint.py use 1e-13 of the norm for the same pair of kernels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (N1, N2): FP64 tiles 32 x 16 (stage, projection) and 32 x 8 (MHD, adjoint), FP32 32 x 8 and 32 x 16
RAGGED = [(35, 36), (47, 62), (32, 100), (39, 44), (40, 96), (45, 35), (34, 64), (33, 66), (51, 40)]


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


def mesh(nova, monkeypatch, impl, N, **kw):
    monkeypatch.setenv("NOVA_STAGE_IMPL", impl)
    return nova.Mesh(N, **kw)


@pytest.mark.parametrize("prec", ["F64", "F32SPLIT"])
@pytest.mark.parametrize("n1,n2", RAGGED)
def test_ns(nova, monkeypatch, n1, n2, prec):
    N, p = (11, n1, n2), getattr(nova, prec)
    U0 = 0.3 * np.random.default_rng(n1 * n2).standard_normal((3,) + N)

    def run(impl, rk):
        M = mesh(nova, monkeypatch, impl, N)
        U, q = nova.Field(M, 3, p).upload_soa(U0), nova.Field(M, 1)
        h = nova.advance(M, nova.run_desc(rk_mode=rk, precision=p, dt=2e-3, nu=1e-2), U, q, nsteps=2)
        return U.download_soa(), q.download_soa(), np.delete(h, 4, axis=1)  # without max|div U|, rounding noise
    for rk in ("classical", "literal"):
        a, b = run("auto", rk), run("march", rk)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        np.testing.assert_allclose(a[2], b[2], rtol=1e-13)


@pytest.mark.parametrize("prec", ["F64", "F32SPLIT"])
@pytest.mark.parametrize("n1,n2", [(32, 32), (33, 36), (39, 64), (46, 44), (64, 96), (47, 62)])
def test_walls(nova, monkeypatch, n1, n2, prec):
    """n1 + 1 stored rows; non-zero wall values exercise both ghost formulas."""
    N, p = (9, n1, n2), getattr(nova, prec)
    U0 = 0.3 * np.random.default_rng(n1 + n2).standard_normal((3, N[0], N[1] + 1, N[2]))
    types, vals = [0] * 18, [0.0] * 18
    for c in range(3):
        types[6 * c] = types[6 * c + 1] = 2 if c == 1 else 1
        vals[6 * c], vals[6 * c + 1] = 0.1 * (c + 1), -0.05 * (c + 1)

    def run(impl, rk):
        M = mesh(nova, monkeypatch, impl, N, walls=(0, 1, 0))
        U, q = nova.Field(M, 3, p).set_bc(types, vals).upload_soa(U0), nova.Field(M, 1).set_bc([1, 1] + [0] * 16)
        nova.advance(M, nova.run_desc(rk_mode=rk, precision=p, dt=2e-3, nu=1e-2, poisson="dct"), U, q, nsteps=2,
                     history=False)
        return U.download_soa(), q.download_soa()
    for rk in ("classical", "shear", "literal"):
        a, b = run("auto", rk), run("march", rk)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("prec", ["F64", "F32SPLIT"])
@pytest.mark.parametrize("n1,n2", RAGGED)
def test_mhd_and_adjoint(nova, monkeypatch, n1, n2, prec):
    N, p = (10, n1, n2), getattr(nova, prec)
    rng = np.random.default_rng(n1 * n2)
    U0, B0 = 0.3 * rng.standard_normal((3,) + N), 0.3 * rng.standard_normal((3,) + N)
    tol = 1e-13 if prec == "F64" else 1e-6  # split: a few FP32 roundings of the increments

    def close(a, b, tol):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)

    def run(impl):
        M = mesh(nova, monkeypatch, impl, N)
        rd = nova.run_desc(model="mhd", precision=p, dt=2e-3, nu=1e-2, eta=1e-2)
        U, B = nova.Field(M, 3, p).upload_soa(U0), nova.Field(M, 3, p).upload_soa(B0)
        J, g, gB = nova.adjoint_grad(M, rd, U, 3, 2, B0=B, total_energy=True)
        nova.advance(M, rd, U, nova.Field(M, 1), B, nova.Field(M, 1), nsteps=2, history=False)
        return J, g.download_soa(), gB.download_soa(), U.download_soa(), B.download_soa()
    a, b = run("auto"), run("march")
    assert a[0] == pytest.approx(b[0], rel=max(tol, 1e-13))
    for x, y in zip(a[1:], b[1:]):
        close(x, y, tol)
