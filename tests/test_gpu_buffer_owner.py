"""A field that another context works on: its buffer goes to the owner's next
field only when that work is done, and the owner sees the work's result.
Every comparison is exact (no arithmetic, or the same arithmetic twice)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (128, 128, 128)  # a sweep takes tens of microseconds: it outlasts the calls that follow it


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


def matrix(nova, B, x):
    """im::laplacian of A's field x, made by context B"""
    h = C.c_void_p()
    B.check(B.lib.nova_im_laplacian(B.h, 0.1, x.h, C.byref(h)))
    Q = nova.FdMatrix(B, x, h)
    Q.add_diagonal(-1.0)
    return Q


def test_next_field_after_another_contexts_solve_is_zero(nova):
    A, B = nova.Mesh(N), nova.Mesh(N)
    v = 1.0 + np.random.default_rng(5).random((1,) + N)
    for _ in range(5):
        x = nova.Field(A, 1).upload_soa(v)
        Q = matrix(nova, B, x)
        assert Q.solve(0.0, 2)[0] == 2  # an even number of iterations: the last sweep writes x, nothing is copied
        x.close()
        y = nova.Field(A, 1)
        assert not y.download_soa().any()
        Q.close()
        y.close()


def test_owner_sees_another_contexts_solve(nova):
    A, B = nova.Mesh(N), nova.Mesh(N)
    v = 1.0 + np.random.default_rng(6).random((1,) + N)
    x, own = nova.Field(A, 1).upload_soa(v), nova.Field(B, 1).upload_soa(v)
    Q, P = matrix(nova, B, x), matrix(nova, B, own)
    for its in (2, 1, 2):
        Q.solve(0.0, its)
        got = x.download_soa()  # on A's stream
        P.solve(0.0, its)
        assert np.array_equal(got, own.download_soa())
