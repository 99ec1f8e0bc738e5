"""tg_horiz_ng_dev (several fields in one launch) against its parts, bit for
bit: more fields than one launch takes, one kind alone, tiny and ragged grids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,nlon,nlat,n_adv,n_smo", [(5, 40, 21, 3, 3), (3, 1, 1, 1, 2), (2, 28, 4, 9, 1), (2, 29, 5, 0, 10),
                                                      (57, 52, 33, 2, 0)])
def test_batch_is_its_parts(pkg, nk, nlon, nlat, n_adv, n_smo):
    import torch
    cs = pkg.colsolve
    grid = pkg.dynamics.Grid(nk, nlon, nlat, 0.25, lat0_deg=20.0, dlat_deg=0.3)
    ld, st = grid.ld, torch.cuda.current_stream()
    g = torch.Generator(device="cuda").manual_seed(nlon)
    r = lambda s: (torch.rand((nk, ld), dtype=torch.float64, device="cuda", generator=g) - 0.4) * s  # noqa: E731
    un, vn, racs = r(1e4), r(1e4), torch.from_numpy(np.ascontiguousarray(grid.racs)).cuda()
    f, fin = [r(800.0) for _ in range(n_adv)], [r(1e-3) for _ in range(n_smo)]
    if n_adv:
        f[0][:, ::5] = f[0][:, :1]           # equal neighbours: zero differences
    had, fo = [torch.zeros_like(un) for _ in f], [torch.zeros_like(un) for _ in fin]
    cs.horiz_ng_dev(f, had, fin, fo, un, vn, racs, grid.dlamda, grid.dphi, grid.re_inv, 0.03, nk, nlon, nlat, ld, stream=st)
    want = torch.zeros_like(un)
    for a, b in zip(f, had):
        cs.advec_ng_dev(a, un, vn, racs, grid.dlamda, grid.dphi, grid.re_inv, want, nk, nlon, nlat, ld, stream=st)
        assert torch.equal(b.view(torch.int64), want.view(torch.int64))
    for a, b in zip(fin, fo):
        want.zero_()
        cs.smooth_ng_dev(a, 0.03, want, nk, nlon, nlat, ld, stream=st)
        assert torch.equal(b.view(torch.int64), want.view(torch.int64))
    with pytest.raises(pkg.TgError):
        cs.horiz_ng_dev([un], [un], [], [], un, vn, racs, 1.0, 1.0, 1.0, 0.03, nk, nlon, nlat, ld, stream=st)
