"""Idle buffers of one context go back to the device when another context's
allocation, or an FFT plan's own work area, does not fit beside them."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


@contextlib.contextmanager
def only(leave):
    """device memory taken up but for about `leave` bytes"""
    import torch
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info(0)[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def idle_gib(nova):
    """a context that keeps 0.75 GiB of a dropped field"""
    A = nova.Mesh((256, 256, 256))
    nova.Field(A, 6).close()
    return A


def test_field_of_another_context(nova):
    A, B = idle_gib(nova), nova.Mesh((256, 256, 256))
    with only(GIB // 4):
        f = nova.Field(B, 3)  # 3/8 GiB
    assert not f.download_soa().any()
    A.close()


def test_plan_work_area(nova):
    N = (250, 250, 250)  # no length of the line transforms: 3-D plans, a work area of 126 MB each
    x = np.random.default_rng(8).standard_normal((1,) + N)
    x -= x.mean()

    def solver():
        M = nova.Mesh(N)
        r, p = nova.Field(M, 1).upload_soa(x), nova.Field(M, 1)
        e = nova.poisson(p)
        e.rhs(r)
        return M, p, e
    M, p, e = solver()
    e.solve()  # the kernels are loaded
    want = p.download_soa()
    p.close()
    M.close()
    B, q, e = solver()
    A = idle_gib(nova)
    with only(GIB // 16):
        e.solve()
    assert np.array_equal(q.download_soa(), want)
    A.close()
