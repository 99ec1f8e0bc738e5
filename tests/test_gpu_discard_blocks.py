"""The block kinds of a plan whose large scalar kind makes the FP64 kinds discard
their finished scratch (the refinement kernels of blocks keep theirs): against
the oracle, the plan run twice with the L2 cache turned over in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAW = dict(d0_range=(1e-4, 1e-1), loss=("lognormal", -6.0, 2.0), d_span=None, device="cuda")


@pytest.mark.parametrize("refine", [False, True])
def test_small_block_kinds(pkg, orc, refine):
    import torch
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(13)
    segs, nk = [], 29
    for kind, ncol in ((0, 32 * nsm * 8 + 40), (2, 333), (3, 65)):
        ld = pkg.batch.pad_ld(ncol)
        gen = pkg.batch.gen_scalar_device if kind == 0 else lambda *a, k=kind, **kw: pkg.batch.gen_block_device(k, *a, **kw)
        a, b, c, f = gen(nk, ncol, ld, 0.25, g, **LAW)
        segs.append(dict(kind=kind or pkg.TG_KIND_SCALAR, nk=nk, k2=nk, ncol=ncol, ld=ld, a=a, b=b, c=c, f=f,
                         x=torch.full_like(f, float("nan"))))
    plan = pkg.Plan(segs, pkg.TG_PREC_F32_REFINE if refine else pkg.TG_PREC_F64)
    turn = torch.empty(1 << 25, dtype=torch.float64, device="cuda")
    for rep in range(2):
        for s in segs:
            s["x"].fill_(float("nan"))
        plan.execute(torch.cuda.current_stream())
        turn.fill_(float(rep))
        torch.cuda.synchronize()
        for s in segs[1:]:
            B, n = s["kind"], s["ncol"]
            P, Q, R = (np.asfortranarray(np.transpose(s[k][..., :n].cpu().numpy(), (2, 1, 0, 3))) for k in "abc")
            f, x = (np.transpose(s[k][..., :n].cpu().numpy(), (1, 0, 2)) for k in "fx")
            want = orc.blksolve(P, Q, R, np.asfortranarray(f), nk)
            assert np.all(np.isfinite(x)) and np.all(np.isfinite(want)), B
            if refine:   # the refinement's own tolerance, as in the other plans
                assert np.max(np.abs(x - want)) <= 1e-10 * np.max(np.abs(want)), B
            else:
                assert np.array_equal(x, want), B
    plan.close()
