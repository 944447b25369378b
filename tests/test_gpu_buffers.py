"""Buffers of dropped fields and matrices are reused by their context: a new
field still starts at zero, whatever the buffer held, fields of two contexts
stay apart, and a matrix or a field outlives its context's handle.  Every
comparison is exact (no arithmetic is involved)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


def test_reused_buffer_starts_at_zero(nova):
    M = nova.Mesh((12, 10, 8))
    for prec in (nova.F64, nova.F32SPLIT, nova.F64):
        for _ in range(3):
            f = nova.Field(M, 3, prec)
            assert not f.download_soa().any()
            f.upload_soa(np.full((3, 12, 10, 8), 7.5))
            f.close()


def test_two_contexts_do_not_share_buffers_in_use(nova):
    import torch
    A, B = nova.Mesh((16, 16, 16)), nova.Mesh((16, 16, 16))
    x = np.random.default_rng(1).standard_normal((1, 16, 16, 16))
    f = nova.Field(A, 1).upload_soa(x)
    out = torch.empty(x.shape, dtype=torch.float64, device="cuda")
    B.check(B.lib.nova_field_copy_to_device(B.h, f.h, out.data_ptr()))  # A's field through B's stream
    f.close()
    nova.Field(A, 1).upload_soa(-x)
    nova.Field(B, 1).upload_soa(2 * x)
    assert np.array_equal(out.cpu().numpy(), x)


def test_matrix_and_field_outlive_their_mesh_handle(nova):
    M = nova.Mesh((8, 9, 10))
    x = nova.Field(M, 1).upload_soa(np.random.default_rng(2).standard_normal((1, 8, 9, 10)))
    Q = nova.im.laplacian(0.1, x)
    Q.add_diagonal(-1.0)
    Q.solve(0.0, 2)
    h = x.h
    M.close()
    Q.close()
    x.h = None
    assert nova.load_library().nova_field_destroy(None, h) == nova.OK


def test_fields_dropped_from_several_threads(nova):
    M = nova.Mesh((8, 8, 8))
    fields = [nova.Field(M, 1 + q % 3) for q in range(24)]

    def drop(part):
        for f in part:
            f.close()
    t = [threading.Thread(target=drop, args=(fields[q::4],)) for q in range(4)]
    for w in t:
        w.start()
    for w in t:
        w.join()
    assert not nova.Field(M, 2).download_soa().any()
