"""The marching kernel of the dynamic procedure at the edges of its tiles
(14 rows x 28 columns of output cells, march segments cut to fill the SMs):
bit-identical to the oracle in both setups."""
import numpy as np
import pytest

from tests.helpers import random_state, spatial_params, temporal_params

pytestmark = pytest.mark.gpu


# one cell short of, at, and one over a tile in y and z; the smallest grid; a
# march of one, two and many planes per segment
@pytest.mark.parametrize("L,H,D", [(2, 2, 2), (3, 13, 27), (5, 14, 28), (4, 15, 29), (33, 29, 57), (150, 5, 3)])
@pytest.mark.parametrize("setup", ["temporal", "spatial"])
def test_march_equals_oracle(L, H, D, setup):
    import freeshearlayer_b200 as fsl
    from oracle import oracle as orc
    orc.build()
    p = temporal_params(L, H, D) if setup == "temporal" else spatial_params(L, H, D, BL_HIG=min(2, H - H // 2))
    s = random_state(p, seed=7)
    o = orc.Oracle(p)
    o.set_state(s)
    o.ghost()
    o.dynsmag()
    d = fsl.Domain(p)
    d.upload_state(s)
    d.ghost_bc()
    d.dynamic_smagorinsky()
    assert np.array_equal(d.cells(3), o.cells(3))
    if L * H * D > 1000:
        assert np.any(d.cells(3) > 0)
