"""Launches whose warps discard the scratch of finished tiles: on both sides of
the rule that chooses, several tiles per warp, the call repeated with the L2
cache turned over in between.  Bit for bit with the oracle on every tile's
edges, and the same bits every time."""
import numpy as np
import pytest

from test_gpu_chunk import sample

pytestmark = pytest.mark.gpu

LAW = dict(d0_range=(1e-4, 1e-1), loss=("lognormal", -6.0, 2.0), d_span=None, device="cuda")


@pytest.mark.parametrize("B,nk,tiles_per_sm", [(1, 6, 8), (1, 57, 9), (2, 6, 4), (2, 29, 5), (3, 48, 8), (3, 47, 8)])
@pytest.mark.parametrize("less", [0, 33])
def test_repeated_solves(pkg, orc, B, nk, tiles_per_sm, less):
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    ncol = 32 * nsm * tiles_per_sm - less
    ld = pkg.batch.pad_ld(ncol)
    g = torch.Generator(device="cuda").manual_seed(B + nk)
    cols = sample(ncol)
    pick = torch.from_numpy(cols).cuda()
    turn = torch.empty(1 << 25, dtype=torch.float64, device="cuda")
    if B == 1:
        d = pkg.batch.gen_scalar_device(nk, ncol, ld, 0.25, g, **LAW)
    else:
        d = pkg.batch.gen_block_device(B, nk, ncol, ld, 0.25, g, **LAW)
    first = None
    for rep in range(3):
        x = torch.full_like(d[3], float("nan"))
        if B == 1:
            pkg.trsolv_dev(*d, x, nk, nk, ncol, layout=pkg.TG_LAYOUT_LEVEL, ld=ld)
        else:
            pkg.blksolve_dev(B, *d, x, nk, nk, ncol, layout=pkg.TG_LAYOUT_LEVEL, ld=ld)
        turn.fill_(float(rep))
        x = x[..., :ncol].clone()
        assert first is None or torch.equal(x.view(torch.int64), first.view(torch.int64))
        first = x
    if B == 1:
        h = [np.asfortranarray(v[:, pick].cpu().numpy()) for v in d]
        assert np.array_equal(first[:, pick].cpu().numpy(), orc.trsolv_ng(*h, nk))
        return
    h = [np.asfortranarray(np.transpose(v[..., pick].cpu().numpy(), (2, 1, 0, 3))) for v in d[:3]]
    f = np.asfortranarray(np.transpose(d[3][..., pick].cpu().numpy(), (1, 0, 2)))
    assert np.array_equal(np.transpose(first[..., pick].cpu().numpy(), (1, 0, 2)), orc.blksolve(*h, f, nk))


@pytest.mark.parametrize("refine", [False, True])
def test_plan_discards_for_every_kind(pkg, orc, refine):
    """A large scalar kind makes the small block kinds discard too; the plan
    run three times over, the graph twice more."""
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(3)
    segs = []
    for kind, nk, ncol in ((0, 29, 32 * nsm * 8 + 40), (2, 29, 333), (3, 29, 65)):
        ld = pkg.batch.pad_ld(ncol)
        gen = pkg.batch.gen_scalar_device if kind == 0 else lambda *a, k=kind, **kw: pkg.batch.gen_block_device(k, *a, **kw)
        a, b, c, f = gen(nk, ncol, ld, 0.25, g, **LAW)
        segs.append(dict(kind=kind or pkg.TG_KIND_SCALAR, nk=nk, k2=nk, ncol=ncol, ld=ld, a=a, b=b, c=c, f=f,
                         x=torch.full_like(f, float("nan"))))
    plan = pkg.Plan(segs, pkg.TG_PREC_F32_REFINE if refine else pkg.TG_PREC_F64)
    turn = torch.empty(1 << 25, dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    first = None
    with torch.cuda.stream(st):
        for rep in range(5):
            for s in segs:
                s["x"].fill_(float("nan"))
            if rep == 3:
                plan.capture_graph(st)
            plan.execute(st)
            turn.fill_(float(rep))
            got = [s["x"][..., :s["ncol"]].clone() for s in segs]
            assert first is None or all(torch.equal(p.view(torch.int64), q.view(torch.int64)) for p, q in zip(got, first))
            first = got
    assert plan.status()[0] in ((pkg.TG_OK, pkg.TG_ENOCONV) if refine else (pkg.TG_OK,))
    plan.close()
    cols = sample(segs[0]["ncol"])
    pick = torch.from_numpy(cols).cuda()
    h = [np.asfortranarray(segs[0][k][:, pick].cpu().numpy()) for k in "abcf"]
    want = orc.trsolv_ng(*h, 29)
    x = first[0][:, pick].cpu().numpy()
    if refine:   # the refinement's own tolerance, as in the other plans
        assert np.max(np.abs(x - want)) <= 1e-10 * np.max(np.abs(want))
    else:
        assert np.array_equal(x, want)
