"""settei_ng's three-pass form at the edges of its blocks of 4 levels x 32
columns, against the single column walk bit for bit, and both against the
oracle where the level losses take their other branches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(pkg, F, C, qt, mode, pad):
    import torch
    nk, ncol = F["tn"].shape
    ld = ncol + pad
    dev = {}
    for k, v in F.items():
        v = np.asarray(v)
        dev[k] = torch.full((*v.shape[:-1], ld), float("nan"), dtype=torch.float64, device="cuda")
        dev[k][..., :ncol] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    te, ti, q2 = (torch.zeros((nk, ld), dtype=torch.float64, device="cuda") for _ in range(3))
    q2[:, :ncol] = torch.from_numpy(qt).cuda()
    rows = torch.zeros((4, nk, ld), dtype=torch.float64, device="cuda")
    stat = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        pkg.set_assembly_mode(mode)
        pkg.settei_ng_dev(dev, C, te, ti, q2, nk, ncol, ld, system_out=rows, status=stat)
        torch.cuda.synchronize()
    finally:
        pkg.set_assembly_mode(-1)
    return [x[..., :ncol].cpu().numpy() for x in (te, ti, q2, rows[:, :nk - 1])] + [int(stat.item())]


@pytest.mark.parametrize("nk,ncol,pad,et,eh", [(3, 1, 0, 1, 0), (4, 31, 1, 0, 6), (5, 32, 0, 1, 6), (6, 33, 0, 0, 0),
                                               (8, 64, 2, 1, 0), (9, 95, 0, 1, 6), (57, 300, 4, 1, 6), (113, 65, 1, 0, 6)])
def test_system_is_the_walk(pkg, nk, ncol, pad, et, eh):
    F, C, qt = pkg.synth.settei_inputs(nk, ncol, 0.25, 3 + nk, et=et, electron_heating=eh)
    want = run(pkg, F, C, qt, 0, pad)
    assert want[4] == pkg.TG_OK
    for mode in (1, 2):
        got = run(pkg, F, C, qt, mode, pad)
        assert got[4] == want[4]
        for a, b in zip(got[:4], want[:4]):
            assert np.array_equal(a.view(np.int64), b.view(np.int64))


@pytest.mark.parametrize("case", ["te over the rate's three ranges", "te equal to tn", "n2 where its weight turns",
                                  "te beyond the roots' range"])
def test_losses_match_the_oracle(pkg, orc, case):
    # of each plane's largest value: the functions differ by a few ulp (1e-15), which 1 - exp(-y)
    # amplifies by 1/y, y >= 1e-3 here
    F, C, qt = pkg.synth.settei_inputs(9, 67, 0.25, 21, et=1, electron_heating=6)
    rng = np.random.default_rng(5)
    if case.startswith("te over"):
        F["te"] = rng.choice([300., 999.9, 1000., 1500., 2000., 2000.1, 2600.], F["te"].shape)
    elif case.startswith("te equal"):
        F["te"] = F["tn"] + rng.choice([0., 5e-7, 0.5], F["te"].shape)
    elif case.startswith("n2"):
        # ad + sd*n2n falls through the guard and below alam
        F["n2"] = -rng.uniform(0.2, 1.2, F["n2"].shape) * 1e8 / (F["xnmbar"] * C["rmassinv_n2"])
    else:
        F["te"] = F["te"] * 1e62
        F["tn"] = F["tn"] * 1e62
    got = run(pkg, F, C, qt, 2, 3)
    (_, _, q2), sys_ref = orc.settei_ng(F, C, qt, with_system=True)
    for a, b in zip([*got[3], got[2]], [*(x[:8] for x in sys_ref), q2]):
        # an extrapolated top temperature below zero has no root, here or there
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.nanmax(np.abs(a - b)) <= 1e-11 * np.nanmax(np.abs(b))
