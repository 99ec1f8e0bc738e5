"""The O+ sub-cycle in one call (tg_oplus_ng_subcycle_dev) against its parts
(factor, then smoothing and solve per sub-step): the same bits, at the edges of
its column tiles, of the levels a thread holds and of the fused kernel's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nlon,nlat,ldpad,nsub", [
    (57, 52, 33, 0, 10), (29, 11, 9, 0, 3), (57, 1, 1, 0, 2), (3, 9, 2, 0, 2), (4, 40, 3, 1, 2), (64, 12, 5, 0, 1),
    (65, 12, 5, 3, 2), (113, 13, 6, 0, 3), (128, 12, 4, 0, 2), (129, 12, 4, 0, 2), (57, 160, 100, 0, 2)])
@pytest.mark.parametrize("bnd", [True, False])
def test_subcycle_is_its_parts(pkg, nk, nlon, nlat, ldpad, nsub, bnd):
    import torch
    cs, dyn = pkg.colsolve, pkg.dynamics
    grid = dyn.Grid(nk, nlon, nlat, 14.0 / (nk - 1), lat0_deg=20.0, dlat_deg=0.3)
    if ldpad:
        grid.ld = grid.ncol + ldpad
    ld, st = grid.ld, torch.cuda.current_stream()
    Fh, C = pkg.synth.oplus_inputs(nk, grid.ncol, grid.dz, 3 + nk, nstep_sub=nsub)
    F = dyn._dev_fields(Fh, grid, ("zpint",), "cuda")
    rng = np.random.default_rng(nk)
    optm1 = pkg.batch.level_scalar(np.asfortranarray(Fh["op"] * rng.uniform(0.98, 1.02, Fh["op"].shape)), ld, "cuda")
    vals = pkg.batch.level_scalar(np.asfortranarray(Fh["op"] * 1.03), ld, "cuda")
    mask = torch.from_numpy(np.pad(grid.boundary_mask(), (0, ld - grid.ncol))).cuda()
    z = lambda: torch.zeros((nk, ld), dtype=torch.float64, device="cuda")  # noqa: E731
    fac = lambda: torch.zeros(cs.oplus_ng_factor_doubles(nk, ld), dtype=torch.float64, device="cuda")  # noqa: E731
    x2p, x2d, sm, f1, stat = z(), z(), z(), fac(), torch.zeros(1, dtype=torch.int32, device="cuda")
    op, tm = [z(), z()], [z(), z()]
    cs.oplus_ng_subcycle_dev(F, C, x2p, x2d, f1, optm1, sm, 0.003, op, tm, nk, nlon, nlat, ld, 0.95, 0.025,
                             bnd_mask=mask if bnd else None, bnd=vals if bnd else None, status=stat, stream=st)
    y2p, y2d, f2 = z(), z(), fac()
    cs.oplus_ng_factor_dev(F, C, y2p, y2d, f2, nk, grid.ncol, ld, stream=st)
    o, t, want = F["op"], optm1, None
    for _ in range(nsub):
        so, sx, sn = z(), z(), z()
        cs.smooth_ng_dev(t, 0.003, so, nk, nlon, nlat, ld, stream=st)
        post = dict(cur=o, prev=t, nm_upd=sn, bnd_mask=mask if bnd else None, bnd=vals if bnd else None, dtsmooth=0.95,
                    dtsmooth_div2=0.025)
        cs.oplus_ng_solve_dev(dict(F, optm1_smooth2=so), C, f2, sx, nk, grid.ncol, ld, post, stream=st)
        o, t = sx, sn
        want = (sx, sn)
    torch.cuda.synchronize()
    n = grid.ncol
    last = (nsub - 1) % 2
    for got, ref in ((op[last], want[0]), (tm[last], want[1]), (x2p, y2p), (x2d, y2d)):
        assert torch.equal(got[:, :n].view(torch.int64), ref[:, :n].view(torch.int64))
    assert int(stat.item()) == pkg.TG_OK


@pytest.mark.parametrize("nk,nlon,nlat", [(29, 60, 30), (30, 120, 90), (31, 40, 40), (57, 90, 60), (57, 120, 75), (57, 140, 74),
                                          (57, 150, 84), (57, 156, 96), (61, 30, 20), (61, 60, 50)])
def test_every_register_variant(pkg, nk, nlon, nlat):
    """On each side of the rules that choose the sub-step's registers."""
    test_subcycle_is_its_parts(pkg, nk, nlon, nlat, 0, 2, True)
