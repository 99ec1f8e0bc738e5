"""What tg_oplus_ng_subcycle_dev and its factor pass read and where they may
write, as include/tg_colsolve.h states it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

S_EX = 9   # the factor buffer's right-hand-side plane, which only full rows fill


def setup(pkg, nk, nlon, nlat, nsub):
    import torch
    grid = pkg.dynamics.Grid(nk, nlon, nlat, 14.0 / (nk - 1), lat0_deg=20.0, dlat_deg=0.3)
    Fh, C = pkg.synth.oplus_inputs(nk, grid.ncol, grid.dz, 7 + nk, nstep_sub=nsub)
    F = pkg.dynamics._dev_fields(Fh, grid, ("zpint",), "cuda")
    rng = np.random.default_rng(nk)
    optm1 = pkg.batch.level_scalar(np.asfortranarray(Fh["op"] * rng.uniform(0.98, 1.02, Fh["op"].shape)), grid.ld, "cuda")
    bnd = pkg.batch.level_scalar(np.asfortranarray(Fh["op"] * 1.03), grid.ld, "cuda")
    mask = torch.from_numpy(np.pad(grid.boundary_mask(), (0, grid.ld - grid.ncol))).cuda()
    return grid, F, C, optm1, bnd, mask


def same(a, b, ncol):
    import torch
    return torch.equal(a[..., :ncol].contiguous().view(torch.int64), b[..., :ncol].contiguous().view(torch.int64))


# both sides of the rule that forms level quantities and rows in one kernel
@pytest.mark.parametrize("nk,nlon,nlat", [(3, 9, 2), (4, 40, 3), (29, 11, 9), (57, 52, 33), (57, 140, 74), (113, 60, 50)])
def test_factor_forms_no_right_hand_side(pkg, nk, nlon, nlat):
    """Without a right-hand side to form, explicit_h and optm1_smooth2 do not
    enter the factor buffer and its right-hand-side plane is not written."""
    import torch
    cs = pkg.colsolve
    grid, F, C, optm1, bnd, mask = setup(pkg, nk, nlon, nlat, 2)
    ld, ncol, st = grid.ld, grid.ncol, torch.cuda.current_stream()
    z = lambda: torch.zeros((nk, ld), dtype=torch.float64, device="cuda")  # noqa: E731
    res = []
    for fill in (0.0, float("nan")):
        G = dict(F, explicit_h=torch.full_like(F["tn"], fill), optm1_smooth2=torch.full_like(F["tn"], fill))
        fac = torch.full((cs.oplus_ng_factor_doubles(nk, ld),), -7.0, dtype=torch.float64, device="cuda")
        p, d = z(), z()
        cs.oplus_ng_factor_dev(G, C, p, d, fac, nk, ncol, ld, stream=st)
        torch.cuda.synchronize()
        planes = fac[:nk * ld * (fac.numel() // (nk * ld))].view(-1, nk, ld)
        assert bool((planes[S_EX] == -7.0).all())
        res.append((planes, p, d))
    for a, b in zip(*res):
        assert same(a, b, ncol)


@pytest.mark.parametrize("nk,nlon,nlat", [(57, 52, 33), (57, 140, 74), (57, 160, 100), (131, 12, 4)])
def test_subcycle_does_not_read_optm1_smooth2(pkg, nk, nlon, nlat):
    import torch
    cs = pkg.colsolve
    grid, F, C, optm1, bnd, mask = setup(pkg, nk, nlon, nlat, 2)
    ld, ncol, st = grid.ld, grid.ncol, torch.cuda.current_stream()
    z = lambda: torch.zeros((nk, ld), dtype=torch.float64, device="cuda")  # noqa: E731
    res = []
    for fill in (0.0, float("nan")):
        G = dict(F, optm1_smooth2=torch.full_like(F["tn"], fill))
        fac = torch.zeros(cs.oplus_ng_factor_doubles(nk, ld), dtype=torch.float64, device="cuda")
        op, tm = [z(), z()], [z(), z()]
        cs.oplus_ng_subcycle_dev(G, C, z(), z(), fac, optm1, z(), 0.003, op, tm, nk, nlon, nlat, ld, 0.95, 0.025,
                                 bnd_mask=mask, bnd=bnd, stream=st)
        torch.cuda.synchronize()
        res.append((*op, *tm))
    for a, b in zip(*res):
        assert same(a, b, ncol) and bool(torch.isfinite(b[:, :ncol]).all())


# (optm1_a, optm1_b) in place of a buffer that the sub-step filters
@pytest.mark.parametrize("where", [("optm1", None), (None, "optm1_a"), ("optm1", "optm1_a"), ("op", None), ("op", "optm1_a"),
                                   (None, "optm1")])
@pytest.mark.parametrize("nk,nlon,nlat", [(29, 11, 9), (57, 52, 33), (57, 160, 100), (131, 12, 4)])
def test_subcycle_filters_in_place(pkg, nk, nlon, nlat, where):
    """optm1_a and optm1_b where the filter's nm_upd may lie: the bits of
    separate buffers, on both sides of the fused sub-step's range."""
    import torch
    cs = pkg.colsolve
    grid, F, C, optm1, bnd, mask = setup(pkg, nk, nlon, nlat, 3)
    ld, ncol, st = grid.ld, grid.ncol, torch.cuda.current_stream()
    z = lambda: torch.zeros((nk, ld), dtype=torch.float64, device="cuda")  # noqa: E731

    def call(a, b):
        G, prev = dict(F, op=F["op"].clone()), optm1.clone()
        place = {"optm1": prev, "op": G["op"]}
        tm_a = place[a] if a else z()
        tm_b = tm_a if b == "optm1_a" else place[b] if b else z()
        fac, op = torch.zeros(cs.oplus_ng_factor_doubles(nk, ld), dtype=torch.float64, device="cuda"), [z(), z()]
        cs.oplus_ng_subcycle_dev(G, C, z(), z(), fac, prev, z(), 0.003, op, [tm_a, tm_b], nk, nlon, nlat, ld, 0.95, 0.025,
                                 bnd_mask=mask, bnd=bnd, stream=st)
        torch.cuda.synchronize()
        return op[0], tm_a     # sub-step 2's, the last

    for got, want in zip(call(*where), call(None, None)):
        assert same(got, want, ncol)
