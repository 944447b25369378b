"""Marches cut along i into chunks: meshes with fewer planes than the stencil
reaches, one plane more or less than a chunk, and remainders.  The TMA kernels
and the tile march do the same arithmetic in the same order, so whole runs
agree bit for bit; the history row's sums run over other blocks (relative
1e-13: sums of at most 2^18 positive terms in two orders, pairwise by blocks)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


@pytest.mark.parametrize("prec", ["F64", "F32SPLIT"])
@pytest.mark.parametrize("n0", [1, 2, 5, 6, 7, 13, 37, 101])
def test_ns_run_matches_the_march(nova, monkeypatch, n0, prec):
    N, p = (n0, 32, 64), getattr(nova, prec)
    U0 = np.random.default_rng(n0).standard_normal((3,) + N)

    def run(impl):
        monkeypatch.setitem(os.environ, "NOVA_STAGE_IMPL", impl)
        M = nova.Mesh(N)
        U, q = nova.Field(M, 3, p).upload_soa(U0), nova.Field(M, 1)
        h = nova.advance(M, nova.run_desc(precision=p, dt=1e-3, nu=1e-2), U, q, nsteps=2)
        return U.download_soa(), q.download_soa(), h
    a, b = run("tma"), run("march")
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    keep = [c for c in range(nova.HIST_COLS) if c != 4]  # max|div U| is rounding noise after the projection
    np.testing.assert_allclose(a[2][:, keep], b[2][:, keep], rtol=1e-13)
