"""comp_ng's post steps on both sides of the rules that choose a block's columns
and threads (148 SMs: 4,736, 9,472 and 18,944 columns, 85 levels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nk,dz,ncol", [(29, 0.5, 4736), (29, 0.5, 4737), (33, 0.5, 9472), (33, 0.5, 9473), (9, 0.5, 18944),
                                        (85, 0.125, 18945), (86, 0.125, 18945), (3, 0.5, 31)])
def test_every_block_shape(pkg, orc, nk, dz, ncol):
    F, C = pkg.synth.comp_post_inputs(nk, ncol, dz, 11)
    upd = [F[k].copy(order="F") for k in ("o2_upd", "o1_upd", "he_upd")]
    nm = [np.zeros((nk, ncol), order="F") for _ in range(3)]
    assert pkg.comp_post_ng(F, C, upd, nm) == pkg.TG_OK
    for got, want in zip(upd + nm, orc.comp_post_ng(F, C)):
        # the device log and exp in the extrapolated levels: the tolerance of the other sizes
        assert float(np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-300))) <= 1e-15
