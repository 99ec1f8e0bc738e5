"""The three-pass walks (tg_walk.cu) where their tiles, stages and copies begin
and end: level counts around the ring's stages, ragged last tiles, 16-byte and
8-byte row copies, and the post-solve steps on the ring-streamed walk."""
import numpy as np
import pytest

from test_gpu_post import _level, _post_inputs, _separate
from test_gpu_walks import _planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk", [1, 2, 3, 4, 5, 8, 9, 13, 29, 113])
@pytest.mark.parametrize("ncol,pad", [(33, 31), (33, 0), (47, 1), (16600, 24), (16599, 1), (16599, 0)])
@pytest.mark.parametrize("top", [0, 1])
def test_walk_edges(cuda, pkg, orc, nk, ncol, pad, top):
    torch = cuda
    K = nk - 1 if top == 1 else nk
    if top == 1 and K < 2:
        pytest.skip("the extrapolated top row needs two solved rows")
    small = 65
    a, b, c, f = (np.array(v) for v in pkg.synth.scalar_system(nk, small, 0.25, 31 + nk))
    reps = -(-ncol // small)
    wide = [np.asfortranarray(np.tile(v, (1, reps))[:, :ncol]) for v in (a, b, c, f)]
    buf = _planes(torch, wide + [np.full((nk, ncol), -7.0, order="F")], nk, ncol + pad)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    pkg.selftest_walk(0, buf, nk, K, top, ncol, ncol + pad, st)
    torch.cuda.synchronize()
    got = buf[4, :, :ncol].cpu().numpy()
    want = np.tile(orc.trsolv_ng(*(np.asfortranarray(v) for v in (a, b, c, f)), K), (1, reps))[:, :ncol]
    assert np.array_equal(got[:K], want[:K])
    if top == 1:
        assert np.array_equal(got[K], want[K - 1] * want[K - 1] / want[K - 2])
    else:
        assert np.all(got[K:] == -7.0)


@pytest.mark.parametrize("nk,ncol,pad", [(57, 16600, 8), (113, 7200, 2), (57, 17001, 31)])
@pytest.mark.parametrize("alias", [False, True])
def test_ring_walk_post_steps(cuda, pkg, nk, ncol, pad, alias):
    torch = cuda
    F, C = pkg.synth.dt_inputs(nk, ncol, 0.25, 5)
    dev, ld = _level(pkg, torch, F, nk, ncol, ("expz", "dift"), ld=ncol + pad)
    cur = dev["tn"]
    prev, bnd, mask, nm = _post_inputs(torch, cur, nk, ncol, ld, 1, 50.0, 1500.0, alias)
    prev0 = prev.clone()
    x = torch.zeros((nk, ld), dtype=torch.float64, device="cuda")
    pkg.dt_ng_dev(dev, C, x, nk, ncol, ld)
    want_x, want_nm = _separate(pkg, torch, pkg.TG_FILTER_DT, x, cur, prev0, bnd, mask, 0.95, 0.025, nk, ncol, ld)
    y = torch.zeros((nk, ld), dtype=torch.float64, device="cuda")
    pkg.dt_ng_post_dev(dev, C, y, nk, ncol, ld, dict(cur=cur, prev=nm if alias else prev, nm_upd=nm, bnd_mask=mask,
                                                     bnd=bnd, dtsmooth=0.95, dtsmooth_div2=0.025))
    torch.cuda.synchronize()
    assert torch.equal(y[:, :ncol], want_x[:, :ncol])
    assert torch.equal(nm[:, :ncol], want_nm[:, :ncol])
