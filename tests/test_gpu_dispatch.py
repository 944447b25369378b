"""Which kernels a mesh takes.  The TMA-fed kernels and the march give the same
values (tests/test_gpu_ragged_tma.py), so a fit rule that had become narrower
would show in no result: forcing the TMA stage kernel is accepted exactly on the
meshes of the rule, and by default the kernels that run are its (their names, from
the profiler)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the ragged meshes of tests/test_gpu_ragged_tma.py, and whole tiles
MESHES = [(35, 36), (47, 62), (32, 100), (39, 44), (40, 96), (45, 35), (34, 64), (33, 66), (51, 40), (64, 64)]


def fits(n1, n2, align, rows, walls=False):
    """rows of whole 16 bytes, one tile along k and two along j, and no last tile
    of one or two nodes (along j: periodic meshes)"""
    return (n2 >= 32 and n2 % align == 0 and n2 % 32 not in (1, 2) and n1 >= 2 * rows and
            (walls or n1 % rows not in (1, 2)))


@pytest.fixture(scope="module")
def nova():
    from novaclone_b200 import nova
    return nova


def kernels(run):
    """names of the kernels that run() launches"""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    names = {e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA}
    if not any("nova::" in n for n in names):
        pytest.skip("the profiler records no kernels here")
    return " ".join(names)


def noise(N, seed):
    return 0.3 * np.random.default_rng(seed).standard_normal((3,) + N)


@pytest.mark.parametrize("prec,align,rows", [("F64", 2, 16), ("F32SPLIT", 4, 8)])
@pytest.mark.parametrize("n1,n2", MESHES)
def test_forced_stage_kernel(nova, monkeypatch, n1, n2, prec, align, rows):
    monkeypatch.setenv("NOVA_STAGE_IMPL", "tma")
    N, p = (9, n1, n2), getattr(nova, prec)
    M = nova.Mesh(N)
    U, q = nova.Field(M, 3, p).upload_soa(noise(N, 1)), nova.Field(M, 1)

    def run():
        nova.advance(M, nova.run_desc(precision=p, dt=2e-3, nu=1e-2), U, q, history=False)
    if fits(n1, n2, align, rows):
        run()
    else:
        with pytest.raises(nova.NovaError) as e:
            run()
        assert e.value.status == nova.E_UNSUPPORTED


@pytest.mark.parametrize("prec,align,stage,mhd", [("F64", 2, 16, 8), ("F32SPLIT", 4, 8, 16)])
@pytest.mark.parametrize("n1,n2", MESHES)
def test_kernels_by_default(nova, n1, n2, prec, align, stage, mhd):
    N, p = (9, n1, n2), getattr(nova, prec)
    M = nova.Mesh(N)
    t = "double" if prec == "F64" else "float"
    U, B, q, qB = (nova.Field(M, 3, p).upload_soa(noise(N, 1)), nova.Field(M, 3, p).upload_soa(noise(N, 2)),
                   nova.Field(M, 1), nova.Field(M, 1))
    ns = kernels(lambda: nova.advance(M, nova.run_desc(precision=p, dt=2e-3, nu=1e-2), U, q, history=False))
    assert ("k_stage_tma<" + t in ns) == fits(n1, n2, align, stage)
    assert ("k_stage<" + t in ns) != fits(n1, n2, align, stage)
    assert ("k_proj_tma<" in ns) == fits(n1, n2, 2, 16)  # an FP64 U* either way
    rd = nova.run_desc(model="mhd", precision=p, dt=2e-3, nu=1e-2, eta=1e-2)
    assert ("k_mhd_tma<" + t in kernels(lambda: nova.advance(M, rd, U, q, B, qB, history=False))) == fits(
        n1, n2, align, mhd)
    if prec == "F64":
        rd = nova.run_desc(dt=2e-3, nu=1e-2)
        assert ("k_adj_tma<" in kernels(lambda: nova.adjoint_grad(M, rd, U, 2, 2))) == fits(n1, n2, 2, 8)


@pytest.mark.parametrize("prec,align,rows", [("F64", 2, 16), ("F32SPLIT", 4, 8)])
@pytest.mark.parametrize("n1,n2", [(32, 32), (33, 36), (39, 64), (46, 44), (64, 96), (47, 62), (33, 35)])
def test_kernels_between_walls(nova, n1, n2, prec, align, rows):
    N, p = (9, n1, n2), getattr(nova, prec)
    M = nova.Mesh(N, walls=(0, 1, 0))
    U = nova.Field(M, 3, p).upload_soa(noise((9, n1 + 1, n2), 3))
    q = nova.Field(M, 1).set_bc([1, 1] + [0] * 16)
    rd = nova.run_desc(precision=p, dt=2e-3, nu=1e-2, poisson="dct")
    ks = kernels(lambda: nova.advance(M, rd, U, q, history=False))
    t = "double" if prec == "F64" else "float"
    assert ("k_stage_tma<" + t in ks) == fits(n1 + 1, n2, align, rows, walls=True)
    assert ("k_proj_tma<" in ks) == fits(n1 + 1, n2, 2, 16, walls=True)
