"""The diagnostics' level quantities for level spacings that are no power of two,
whose divisions are not the exact products of the model's 1/2, 1/4 and 1/8: the
tolerances of the model's spacings (tests/test_gpu_diag.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(got, want):
    return float(np.max(np.abs(got - want) / np.maximum(np.max(np.abs(want), axis=0), 1e-300)))


@pytest.mark.parametrize("nk,dz,ncol", [(57, 0.25, 200), (47, 0.3, 200), (15, 1.0 / 3.0, 33), (4, 0.7, 5)])
def test_minor_diag(pkg, orc, nk, dz, ncol):
    F, C = pkg.synth.minor_inputs(nk, ncol, dz, 21)
    x = orc.minor_ng(F, C)
    got, want = pkg.minor_diag_ng(F, C, x), orc.minor_diag_ng(F, C, x)
    for name in pkg.colsolve.MINOR_DIAG_NAMES:
        if name in ("MOLDIF", "EDDYDIF"):
            assert rel(got[name], want[name]) <= 1e-12, name
        else:
            assert np.array_equal(got[name], want[name]), name


@pytest.mark.parametrize("nk,dz,ncol", [(57, 0.25, 200), (47, 0.3, 200), (15, 1.0 / 3.0, 33), (4, 0.7, 5)])
def test_comp_diag(pkg, orc, nk, dz, ncol):
    F, C = pkg.synth.comp_inputs(nk, ncol, dz, 22)
    upd = orc.comp_ng(F, C)
    got, want = pkg.comp_diag_ng(F, C, *[np.asfortranarray(u) for u in upd]), orc.comp_diag_ng(F, C, upd)
    for name in pkg.colsolve.COMP_DIAG_NAMES:
        if name.endswith("_MOLDIF") or name.endswith("_EDDYDIF"):
            assert rel(got[name], want[name]) <= 1e-11, name
        else:
            assert np.array_equal(got[name], want[name]), name
