"""The FP64 stage kernels the grid chooses between (rows 0): the direction-split
kernel (tiles of 4 x 32 cells) and the ring tile with its planes per block
chosen by the grid, bit for bit against the 16-row ring tile and the oracle."""
import numpy as np
import pytest

from tests.helpers import random_state, spatial_params, temporal_params

pytestmark = pytest.mark.gpu

# the smallest grid; one cell short of, at and over a tile in y and z; marches of
# one plane, a few planes and several waves; a grid that keeps the ring
SIZES = [(2, 2, 2), (3, 3, 31), (2, 4, 32), (4, 5, 33), (7, 8, 64), (37, 9, 30), (65, 12, 2), (40, 30, 30)]


@pytest.mark.parametrize("L,H,D", SIZES)
@pytest.mark.parametrize("setup", ["temporal", "spatial"])
@pytest.mark.parametrize("sgs", [0, 2])
def test_chosen_kernel_equals_ring_and_oracle(L, H, D, setup, sgs):
    import freeshearlayer_b200 as fsl
    from oracle import oracle as orc
    orc.build()
    p = temporal_params(L, H, D, deltaT=1e-6) if setup == "temporal" else spatial_params(L, H, D, BL_HIG=min(2, H - H // 2))
    p["sgs"] = sgs
    s = random_state(p, seed=11)
    o = orc.Oracle(p)
    o.set_state(s)
    o.step(2)
    out = []
    for rows in (0, 16):
        d = fsl.Domain(p)
        d.tune(d.TUNE_STAGE_ROWS, rows)
        d.upload_state(s)
        d.step(2)
        out.append((d.download_state(), [d.cells(0, v) for v in range(5)], d.info().maxCo))
    assert np.array_equal(out[0][0], o.state())
    assert np.array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):  # ghost layer included
        assert np.array_equal(a, b)
    assert out[0][2] == out[1][2]


@pytest.mark.parametrize("L,H,D", [(2, 2, 2), (30, 11, 31), (90, 20, 40)])
def test_ppm_with_chosen_segments_equals_ring(L, H, D):
    import freeshearlayer_b200 as fsl
    p = temporal_params(L, H, D, recon=fsl.RECON_PPM, deltaT=1e-6)
    s = random_state(p, seed=5)
    out = []
    for rows in (0, 12):
        d = fsl.Domain(p)
        d.tune(d.TUNE_STAGE_ROWS, rows)
        d.upload_state(s)
        d.step(2)
        out.append(d.download_state())
    assert np.array_equal(*out)
