"""oplus_ng's row kernels (rows between the boundaries have a form of their own;
launches of few blocks form level quantities and rows in one kernel) against
the column walk, bit for bit, from the smallest column on and on both sides of
the rule that chooses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,ncol,pad,cap", [(3, 1, 0, 0.), (4, 127, 1, 1e5), (5, 128, 0, 0.), (6, 129, 0, 1e7),
                                             (11, 31, 0, 0.), (12, 33, 1, 0.), (29, 257, 3, 0.), (57, 300, 0, 0.),
                                             (113, 64, 0, 1e6), (12, 21300, 2, 0.), (12, 21400, 0, 0.),
                                             (3, 42700, 1, 1e5), (22, 21400, 0, 0.)])
@pytest.mark.parametrize("bz", [1., 1e-140])
def test_rows_are_the_walks(pkg, nk, ncol, pad, cap, bz):
    import torch
    F, C = pkg.synth.oplus_inputs(nk, ncol, 0.25, 17 + nk, opdiffcap=cap)
    F["bz"] = F["bz"] * bz      # 1e-140: dj*bz**2 leaves the normal quotients' range
    ld = ncol + pad
    dev = {}
    for k, v in F.items():
        v = np.asarray(v)
        if k == "zpint":
            dev[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
            continue
        dev[k] = torch.full((*v.shape[:-1], ld), float("nan"), dtype=torch.float64, device="cuda")
        dev[k][..., :ncol] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    got = {}
    try:
        for mode in (0, 1, 2):
            pkg.set_assembly_mode(mode)
            outs = [torch.zeros((nk, ld), dtype=torch.float64, device="cuda") for _ in range(5)]
            rows = torch.zeros((4, nk, ld), dtype=torch.float64, device="cuda")
            stat = torch.zeros(1, dtype=torch.int32, device="cuda")
            pkg.oplus_ng_dev(dev, C, outs[0], outs[1], outs[2], nk, ncol, ld, Fe=outs[3], Fn=outs[4], system_out=rows,
                             status=stat)
            torch.cuda.synchronize()
            got[mode] = [x[..., :ncol].clone() for x in (*outs, rows[:, :nk - 1])] + [int(stat.item())]
    finally:
        pkg.set_assembly_mode(-1)
    for mode in (1, 2):
        assert got[mode][6] == got[0][6]
        for a, b in zip(got[mode][:6], got[0][:6]):
            assert torch.equal(a.view(torch.int64), b.view(torch.int64))
