"""comp_ng's fused solve (k_comp_solve) against the column walk that forms its
own rows, bit for bit: at the edges of its chunks and back-sweep stages, on
ragged tiles, with either number of producer warps and with a level spacing
that is a power of two and one that is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,ncol,pad,dz", [(3, 33, 0, 0.25), (4, 1, 2, 0.25), (5, 65, 0, 0.2), (6, 31, 1, 0.5), (7, 64, 0, 0.125),
                                            (8, 40, 3, 0.3), (9, 96, 0, 0.25), (29, 300, 0, 0.5), (57, 1001, 7, 0.25),
                                            (113, 257, 0, 0.1), (12, 14300, 4, 0.25), (13, 14300, 0, 0.3)])
@pytest.mark.parametrize("calc_helium", [1, 0])
def test_solve_is_the_walk(pkg, nk, ncol, pad, dz, calc_helium):
    import torch
    F, C = pkg.synth.comp_inputs(nk, ncol, dz, 7 + nk, calc_helium=calc_helium)
    ld = ncol + pad
    dev = {}
    for k, v in F.items():
        v = np.asarray(v)
        v = np.moveaxis(v, 1, 2) if k == "fs" else v
        if k in ("expz", "difk"):
            dev[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
            continue
        dev[k] = torch.full((*v.shape[:-1], ld), float("nan"), dtype=torch.float64, device="cuda")
        dev[k][..., :ncol] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    got = {}
    try:
        for mode in (2, 1):
            pkg.set_assembly_mode(mode)
            out = torch.zeros((3, nk, ld), dtype=torch.float64, device="cuda")
            rows = torch.zeros((36, nk, ld), dtype=torch.float64, device="cuda")
            stat = torch.zeros(1, dtype=torch.int32, device="cuda")
            pkg.comp_ng_dev(dev, C, out, nk, ncol, ld, system_out=rows, status=stat)
            torch.cuda.synchronize()
            got[mode] = (out[..., :ncol].clone(), rows[:30, :, :ncol].clone(), int(stat.item()))
    finally:
        pkg.set_assembly_mode(-1)
    assert torch.equal(got[2][0].view(torch.int64), got[1][0].view(torch.int64))
    assert torch.equal(got[2][1].view(torch.int64), got[1][1].view(torch.int64))
    assert got[2][2] == got[1][2] == pkg.TG_OK
