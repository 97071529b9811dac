"""The FP64 kernels' branch-free quotients and the divisions they fall back on:
bit for bit against the oracle on states inside the checked range, outside it
(units that scale every conserved variable), with significands that end in ones,
and with positive and negative zero momenta."""
import numpy as np
import pytest

from tests.helpers import random_state, spatial_params, temporal_params

pytestmark = pytest.mark.gpu


def _states(p):
    s = random_state(p, seed=3)
    L, H, D = p["LEN"], p["HIG"], p["DEP"]
    yield "ordinary", s
    yield "below the range", s * 1e-30
    yield "above the range", s * 1e30
    mixed = s.copy().reshape(L, H, 5, D)
    mixed[::2] *= 1e-25  # neighbouring cells on either side of the limit
    yield "mixed", mixed.ravel()
    ones = s.copy().reshape(L, H, 5, D)
    r = ones[:, :, 0].copy().view(np.int64)
    ones[:, :, 0] = (r | 0xFFFFFFFF).view(np.float64)
    yield "ones", ones.ravel()
    zero = s.copy().reshape(L, H, 5, D)
    zero[:, :, 2] = 0.0
    zero[:, :, 3] = -0.0
    zero[:, :, 4] = 2.5e5 + 0.5 * zero[:, :, 1] ** 2 / zero[:, :, 0]
    yield "zeros", zero.ravel()


@pytest.mark.parametrize("path", ["chosen", "ring", "ppm", "phased"])
@pytest.mark.parametrize("setup", ["temporal", "spatial"])
def test_quotients_equal_divisions(path, setup):
    import freeshearlayer_b200 as fsl
    from oracle import oracle as orc
    orc.build()
    p = temporal_params(9, 6, 7, deltaT=1e-6) if setup == "temporal" else spatial_params(9, 6, 7)
    if path == "ppm":
        p["recon"] = fsl.RECON_PPM
    for name, s in _states(p):
        o = orc.Oracle(p)
        o.set_state(s)
        o.step(1)
        d = fsl.Domain(p)
        if path == "ring":
            d.tune(d.TUNE_STAGE_ROWS, 16)
        d.upload_state(s)
        d.step_phased(1) if path == "phased" else d.step(1)
        a, b = d.download_state(), o.state()
        assert np.array_equal(np.isnan(a), np.isnan(b)), name
        assert np.array_equal(a[~np.isnan(a)], b[~np.isnan(b)]), name
