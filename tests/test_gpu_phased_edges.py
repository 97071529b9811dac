"""The per-phase kernels on planes of one cell below, at and above a block of
threads in each face direction: bit for bit against the oracle."""
import numpy as np
import pytest

from tests.helpers import random_state, spatial_params, temporal_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,H,D", [(2, 2, 2), (3, 3, 43), (2, 8, 16), (3, 127, 2), (2, 2, 127), (4, 5, 129)])
@pytest.mark.parametrize("setup", ["temporal", "spatial"])
@pytest.mark.parametrize("recon", ["reference", "ppm"])
def test_phased_step_equals_oracle(L, H, D, setup, recon):
    import freeshearlayer_b200 as fsl
    from oracle import oracle as orc
    orc.build()
    p = temporal_params(L, H, D, deltaT=1e-6) if setup == "temporal" else spatial_params(L, H, D, BL_HIG=min(2, H - H // 2))
    if recon == "ppm":
        p["recon"] = fsl.RECON_PPM
    s = random_state(p, seed=7)
    o = orc.Oracle(p)
    o.set_state(s)
    o.step(2)
    d = fsl.Domain(p)
    d.upload_state(s)
    d.step_phased(2)
    assert np.array_equal(d.download_state(), o.state())
