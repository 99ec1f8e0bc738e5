"""tg_oplus_ng_subcycle_dev refuses buffers that it would overwrite before their
last read, and takes the filter's in-place forms (host side only: the pointers
are never followed)."""
import ctypes

import pytest

OP, OPTM1, SMOOTH, OP_A, TM_A, OP_B, TM_B, BND, FACTOR, EXPL = (0x1000000 * i for i in range(1, 11))


def call(pkg, nsub=3, **kw):
    import torch
    if torch.cuda.is_available():
        pytest.skip("the pointers are not device memory")
    cs = pkg.colsolve
    a = dict(op=OP, expl=EXPL, optm1=OPTM1, smooth=SMOOTH, op_a=OP_A, tm_a=TM_A, op_b=OP_B, tm_b=TM_B, bnd=BND, factor=FACTOR,
             smooth2=0x20000000)
    a.update(kw)
    F = cs.OplusFields(*[{"op": a["op"], "explicit_h": a["expl"], "optm1_smooth2": a["smooth2"]}.get(n, 0x30000000 + 0x100000 * i)
                         for i, n in enumerate(cs.OPLUS_FIELDS)])
    C = cs.OplusConsts()
    C.nstep_sub = nsub
    mask = None if a["bnd"] is None else 0x50000000
    return cs.lib().tg_oplus_ng_subcycle_dev(ctypes.byref(F), ctypes.byref(C), 0x60000000, 0x61000000, a["factor"], a["optm1"],
                                             a["smooth"], 0.003, a["op_a"], a["tm_a"], a["op_b"], a["tm_b"], 57, 8, 4, 96, mask,
                                             a["bnd"], 0.95, 0.025, None, None)


@pytest.mark.parametrize("kw", [
    dict(op_a=OP), dict(op_a=OPTM1), dict(op_a=TM_A), dict(op_a=BND), dict(op_b=OP_A), dict(op_b=TM_A), dict(op_b=TM_B),
    dict(op_b=BND), dict(op_a=TM_B), dict(op_a=EXPL), dict(tm_a=EXPL), dict(tm_a=BND), dict(smooth=OP), dict(smooth=OPTM1),
    dict(smooth=TM_A), dict(smooth=OP_A), dict(smooth=BND), dict(smooth=EXPL), dict(factor=OP_B), dict(factor=OPTM1),
    dict(factor=EXPL), dict(nsub=1, op_a=OP), dict(nsub=2, op_b=OP_A)])
def test_overwritten_reads_are_refused(pkg, kw):
    assert call(pkg, **kw) == pkg.TG_EINVAL


@pytest.mark.parametrize("kw", [
    dict(), dict(bnd=None), dict(tm_a=OPTM1), dict(tm_a=OP), dict(tm_b=TM_A), dict(tm_b=OPTM1), dict(tm_a=OPTM1, tm_b=OPTM1),
    dict(smooth2=SMOOTH), dict(nsub=1, op_b=OP_A, tm_b=TM_A), dict(nsub=1, op_a=EXPL), dict(op_b=OP)])
def test_in_place_filters_are_taken(pkg, kw):
    """The arguments pass; the call stops at the missing device."""
    assert call(pkg, **kw) == pkg.TG_ENODEV
