"""minor_ng's three-pass form at the edges of its blocks of 8 levels x 32
columns, against the column walks bit for bit, with a level spacing that is a
power of two and one that is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,ncol,pad", [(3, 1, 0), (7, 31, 1), (8, 32, 0), (9, 33, 0), (16, 64, 2), (17, 95, 0),
                                         (57, 300, 4), (113, 65, 1)])
@pytest.mark.parametrize("dz", [0.25, 0.3])
def test_system_is_the_walk(pkg, nk, ncol, pad, dz):
    import torch
    F, C = pkg.synth.minor_inputs(nk, ncol, dz, 13 + nk)
    ld = ncol + pad
    dev = {}
    for k, v in F.items():
        v = np.asarray(v)
        if k in ("expz", "difk"):
            dev[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
            continue
        dev[k] = torch.full((*v.shape[:-1], ld), float("nan"), dtype=torch.float64, device="cuda")
        dev[k][..., :ncol] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    got = {}
    try:
        for mode in (0, 1, 2):
            pkg.set_assembly_mode(mode)
            out = torch.zeros((nk, ld), dtype=torch.float64, device="cuda")
            rows = torch.zeros((4, nk, ld), dtype=torch.float64, device="cuda")
            stat = torch.zeros(1, dtype=torch.int32, device="cuda")
            pkg.minor_ng_dev(dev, C, out, nk, ncol, ld, system_out=rows, status=stat)
            torch.cuda.synchronize()
            got[mode] = (out[..., :ncol].clone(), rows[..., :ncol].clone(), int(stat.item()))
    finally:
        pkg.set_assembly_mode(-1)
    for mode in (1, 2):
        for a, b in zip(got[mode][:2], got[0][:2]):
            assert torch.equal(a.view(torch.int64), b.view(torch.int64))
        assert got[mode][2] == got[0][2] == pkg.TG_OK
