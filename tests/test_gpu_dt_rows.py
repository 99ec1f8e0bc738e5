"""dt_ng's row kernel against the column walk that forms its own rows, bit for
bit: level spacings that are and are not powers of two, ragged tiles, a mean
mass beyond the exact divisions' range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,ncol,pad,dz,mass", [(3, 1, 0, 0.25, 1.), (4, 127, 1, 0.3, 1.), (5, 129, 0, 0.125, 1e160),
                                                 (29, 300, 4, 0.5, 1.), (57, 257, 0, 0.1, 1.), (9, 64, 0, 0.2, 1e-160)])
def test_rows_are_the_walks(pkg, nk, ncol, pad, dz, mass):
    import torch
    F, C = pkg.synth.dt_inputs(nk, ncol, dz, 11 + nk)
    F["mbar"] = F["mbar"] * mass
    ld = ncol + pad
    dev = {}
    for k, v in F.items():
        v = np.asarray(v)
        if v.shape[-1] != ncol or k in ("expz", "dift"):
            dev[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
            continue
        dev[k] = torch.full((*v.shape[:-1], ld), float("nan"), dtype=torch.float64, device="cuda")
        dev[k][..., :ncol] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    got = {}
    try:
        for mode in (0, 2):
            pkg.set_assembly_mode(mode)
            out = torch.zeros((nk, ld), dtype=torch.float64, device="cuda")
            rows = torch.zeros((4, nk, ld), dtype=torch.float64, device="cuda")
            stat = torch.zeros(1, dtype=torch.int32, device="cuda")
            pkg.dt_ng_dev(dev, C, out, nk, ncol, ld, system_out=rows, status=stat)
            torch.cuda.synchronize()
            got[mode] = (out[..., :ncol].clone(), rows[:, :nk - 1, :ncol].clone(), int(stat.item()))
    finally:
        pkg.set_assembly_mode(-1)
    for a, b in zip(got[2][:2], got[0][:2]):
        assert torch.equal(a.view(torch.int64), b.view(torch.int64))
    assert got[2][2] == got[0][2]
