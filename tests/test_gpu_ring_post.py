"""The ring filter where chunks are one or a few longitudes wide or leave a
remainder, and comp_ng's post-solve steps at the edges of their blocks."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlon,chunks", [(36, (3, 36, 18, 12)), (35, (35, 17, 34, 3, 4)), (130, (129, 65, 64, 43)),
                                         (5, (3, 5, 4))])
@pytest.mark.parametrize("order,poly", [(1, 0), (2, 1)])
def test_ring_chunk_widths(cuda, pkg, orc, nlon, chunks, order, poly):
    nlat, nk = 2 * len(chunks) + 1, 3
    f = pkg.synth.ring_field(nk, nlon, nlat, 5 + nlon)
    dl = 2.0 * math.pi / nlon
    got = f.copy(order="F")
    pkg.ringfilter(got, order, poly, chunks, dl)
    assert np.array_equal(got, orc.ringfilter(f, order, poly, chunks, dl))


def test_three_fields_as_one(cuda, pkg):
    """A contiguous group of fields filtered as 3*nk levels: the same bits."""
    torch = cuda
    nlon, nlat, nk = 72, 36, 7
    ch, dl, ld = pkg.synth.RING_CHUNKS[(nlon, nlat)], 2.0 * math.pi / nlon, (nlon + 4) * nlat + 6
    a = torch.rand((3, nk, ld), dtype=torch.float64, device="cuda")
    b = a.clone()
    for i in range(3):
        pkg.ringfilter_dev(a[i], nk, nlon, nlat, 1, 0, ch, dl, ld)
    pkg.ringfilter_dev(b, 3 * nk, nlon, nlat, 1, 0, ch, dl, ld)
    torch.cuda.synchronize()
    assert torch.equal(a, b)


@pytest.mark.parametrize("nk,ncol,pad", [(3, 1, 0), (31, 15, 1), (32, 16, 0), (33, 17, 0), (64, 33, 3), (65, 47, 0),
                                         (129, 100, 4)])
def test_post_blocks(cuda, pkg, orc, nk, ncol, pad):
    # log and exp within a few ulp of the host library's, as for the other post-solve checks
    torch = cuda
    F, C = pkg.synth.comp_post_inputs(nk, ncol, 0.25, 3 + nk)
    ld = ncol + pad
    up = lambda v: pkg.batch.level_scalar(v, ld, "cuda")  # noqa: E731
    dev = {k: up(F[k]) for k in pkg.colsolve.POST_INPUTS}
    mask = np.zeros(ncol, dtype=np.uint8)
    mask[::3] = 1
    bnd = [F[k].copy(order="F")[:, ::-1].copy(order="F") for k in ("o2", "o1", "he")]
    upd = [up(F[k]) for k in ("o2_upd", "o1_upd", "he_upd")]
    nm = [torch.zeros((nk, ld), dtype=torch.float64, device="cuda") for _ in range(3)]
    zp = torch.from_numpy(np.ascontiguousarray(F["zpmid"], dtype=np.float64)).cuda()
    pkg.comp_post_ng_dev(dev, zp, C, upd, nm, nk, ncol, ld, bnd_mask=torch.from_numpy(np.pad(mask, (0, pad))).cuda(),
                         bnd=[up(b) for b in bnd])
    torch.cuda.synchronize()
    G = dict(F)
    for k, b in zip(("o2_upd", "o1_upd", "he_upd"), bnd):
        G[k] = F[k].copy(order="F")
        G[k][:, mask.astype(bool)] = b[:, mask.astype(bool)]
    for got, want in zip(upd + nm, orc.comp_post_ng(G, C)):
        got = pkg.batch.from_level_scalar(got, ncol)
        assert np.max(np.abs(got - want)) <= 1e-15 * np.max(np.abs(want))
