"""The chunked ring kernels (k_scalar_f64_chunk, k_block_f64_chunk) where their
rings, back-sweep stages and passes over the SMs begin and end: level counts
around the stage sizes, column counts that leave a ragged last tile, and, with
a small scratch budget, several tiles per warp.  Bit for bit with the oracle on
every tile's first and last columns."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def default_budgets(pkg):
    yield
    pkg.set_scalar_scratch_budget(0)
    pkg.set_block_scratch_budget(0)


def sample(ncol):
    edge = np.arange(0, ncol, 32)
    return np.unique(np.concatenate([edge, edge - 1, [0, ncol - 1]]).clip(0, ncol - 1))[:: max(1, ncol // 4000)]


@pytest.mark.parametrize("nk", [1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16, 17, 25, 57])
@pytest.mark.parametrize("B", [1, 2, 3])
def test_stage_edges(pkg, orc, B, nk):
    import torch
    ncol = 67
    ld = pkg.batch.pad_ld(ncol)
    st = torch.cuda.current_stream()
    if B == 1:
        a, b, c, f = pkg.synth.scalar_system(nk, ncol, 0.25, 3 + nk)
        d = [pkg.batch.level_scalar(v, ld, "cuda") for v in (a, b, c, f)]
        x = torch.zeros_like(d[3])
        pkg.trsolv_dev(*d, x, nk, nk, ncol, layout=pkg.TG_LAYOUT_LEVEL, ld=ld, stream=st)
        assert np.array_equal(pkg.batch.from_level_scalar(x, ncol), orc.trsolv_ng(a, b, c, f, nk))
        return
    P, Q, R, f = pkg.synth.block_system(B, nk, ncol, 0.25, 5 + nk)
    d = [pkg.batch.level_matrix(v, ld, "cuda") for v in (P, Q, R)] + [pkg.batch.level_vector(f, ld, "cuda")]
    u = torch.zeros_like(d[3])
    pkg.blksolve_dev(B, *d, u, nk, nk, ncol, layout=pkg.TG_LAYOUT_LEVEL, ld=ld, stream=st)
    assert np.array_equal(pkg.batch.from_level_vector(u, ncol), orc.blksolve(P, Q, R, f, nk))


@pytest.mark.parametrize("B,nk", [(1, 57), (1, 29), (2, 57), (3, 30)])
def test_several_tiles_per_warp(pkg, orc, B, nk):
    """The smallest budget leaves three warps per SM: every warp takes three or four tiles."""
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    ncol = 32 * (nsm * 3 * 3 + 70) + 5
    ld = pkg.batch.pad_ld(ncol)
    g = torch.Generator(device="cuda").manual_seed(9)
    law = dict(d0_range=(1e-4, 1e-1), loss=("lognormal", -6.0, 2.0), d_span=None, device="cuda")
    cols = sample(ncol)
    pkg.set_scalar_scratch_budget(1e-3)
    pkg.set_block_scratch_budget(1e-3)
    pick = torch.from_numpy(cols).cuda()
    if B == 1:
        d = pkg.batch.gen_scalar_device(nk, ncol, ld, 0.25, g, **law)
        x = torch.zeros_like(d[3])
        pkg.trsolv_dev(*d, x, nk, nk, ncol, layout=pkg.TG_LAYOUT_LEVEL, ld=ld)
        h = [np.asfortranarray(v[:, pick].cpu().numpy()) for v in d]
        assert np.array_equal(x[:, pick].cpu().numpy(), orc.trsolv_ng(*h, nk))
        return
    d = pkg.batch.gen_block_device(B, nk, ncol, ld, 0.25, g, **law)
    u = torch.zeros_like(d[3])
    pkg.blksolve_dev(B, *d, u, nk, nk, ncol, layout=pkg.TG_LAYOUT_LEVEL, ld=ld)
    h = [np.asfortranarray(np.transpose(v[..., pick].cpu().numpy(), (2, 1, 0, 3))) for v in d[:3]]
    f = np.asfortranarray(np.transpose(d[3][..., pick].cpu().numpy(), (1, 0, 2)))
    got = np.transpose(u[..., pick].cpu().numpy(), (1, 0, 2))
    assert np.array_equal(got, orc.blksolve(*h, f, nk))
