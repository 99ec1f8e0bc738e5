"""tg_selftest_walk leaves the rows that it solves as they were, on both sides
of the rule that chooses the walk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,ncol", [(29, 40), (57, 2072), (57, 20000), (113, 9000)])
@pytest.mark.parametrize("top", [0, 1])
def test_rows_are_kept(pkg, nk, ncol, top):
    import torch
    ld = pkg.batch.pad_ld(ncol)
    rng = np.random.default_rng(nk + ncol + top)
    rows = torch.zeros((5, nk, ld), dtype=torch.float64, device="cuda")
    rows[:4, :, :ncol] = torch.from_numpy(rng.uniform(0.1, 1.0, (4, nk, ncol))).cuda()
    rows[1] += 3.0
    want, st = rows[:4].clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
    K = nk - top
    pkg.selftest_walk(0, rows, nk, K, top, ncol, ld, st)
    torch.cuda.synchronize()
    assert int(st.item()) == pkg.TG_OK and torch.equal(rows[:4], want)
    x = rows[4, :K, :ncol]
    res = want[1, :K, :ncol] * x - want[3, :K, :ncol]
    res[1:] += want[0, 1:K, :ncol] * x[:-1]
    res[:-1] += want[2, :K - 1, :ncol] * x[1:]
    assert float(res.abs().max()) <= 1e-13     # rows of at most 6, |x| below 1: some tens of roundings of 1.1e-16
