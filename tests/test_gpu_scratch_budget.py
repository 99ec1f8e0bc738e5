"""The scratch budgets cap what is in flight, as include/tg_colsolve.h states."""
import re

import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def in_flight(pkg, kind, nk, ncol, refine=False):
    """Bytes of sweep scratch (refining: and the iterate) that the resident warps of a solve hold, and its solution."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(nk + ncol)
    ld = pkg.batch.pad_ld(ncol)
    law = dict(d0_range=(1e-4, 1e-1), loss=("uniform", 0.0, 1e-3), d_span=None)
    a, b, c, f = (pkg.batch.gen_scalar_device(nk, ncol, ld, 14.0 / nk, g, device="cuda", **law) if not kind else
                  pkg.batch.gen_block_device(kind, nk, ncol, ld, 14.0 / nk, g, device="cuda", **law))
    x = torch.zeros_like(f)
    plan = pkg.Plan([dict(kind=kind or pkg.TG_KIND_SCALAR, nk=nk, k2=nk, ncol=ncol, ld=ld, a=a, b=b, c=c, f=f, x=x)],
                    pkg.TG_PREC_F32_REFINE if refine else pkg.TG_PREC_F64)
    text = plan.describe()
    plan.execute(torch.cuda.current_stream())
    torch.cuda.synchronize()
    plan.close()
    assert "chunk" in text or "refine_ring" in text, text
    threads, blocks = (int(re.search(k + r"=(\d+)", text).group(1)) for k in ("threads", "blocks"))
    per = (20 if refine else 16) if not kind else 8 * (kind * kind + kind) if not refine else 56
    return threads * blocks * per * nk, x[..., :ncol]


@pytest.mark.parametrize("kind,refine", [(0, False), (0, True), (2, False), (3, False)])
@pytest.mark.parametrize("nk,ncol,mb", [(57, 41472, 4.0), (57, 41472, 0.5), (113, 12000, 16.0), (57, 33000, 30.0)])
def test_a_set_budget_is_a_cap(pkg, kind, refine, nk, ncol, mb):
    import torch
    _, want = in_flight(pkg, kind, nk, ncol, refine)
    set_budget = pkg.set_block_scratch_budget if kind else pkg.set_scalar_scratch_budget
    try:
        set_budget(mb)
        held, x = in_flight(pkg, kind, nk, ncol, refine)
    finally:
        set_budget(0)
    assert held <= mb * MB
    assert torch.equal(x, want)


def test_block_refinement_takes_no_budget(pkg):
    want = in_flight(pkg, 2, 57, 41472, True)[0]
    try:
        pkg.set_block_scratch_budget(4.0)
        assert in_flight(pkg, 2, 57, 41472, True)[0] == want
    finally:
        pkg.set_block_scratch_budget(0)


@pytest.mark.parametrize("kind,nk,ncol", [(0, 4000, 14400), (3, 700, 14400)])
def test_tall_columns_keep_the_default_scratch_bounded(pkg, kind, nk, ncol):
    assert in_flight(pkg, kind, nk, ncol)[0] <= 512 * MB
