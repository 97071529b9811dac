"""FP32 marches cut into parts for the SMs a small grid leaves idle: the cut shows in
no bit, ghost cells, Courant number and velocities for the closure included."""
import numpy as np
import pytest

from tests.helpers import random_state, spatial_params, temporal_params

pytestmark = pytest.mark.gpu

# the smallest grid, marches shorter than and just past the planes a part computes
# ahead, several tiles, several marches per tile (the last one short)
SIZES = [(2, 2, 2), (3, 16, 32), (5, 40, 3), (17, 16, 33), (64, 32, 32), (97, 15, 31), (203, 33, 31)]


def _run(d, s, how):
    d.upload_state(s)
    how(d)
    return d.download_state(), [d.cells(0, v) for v in range(5)], d.info().maxCo


def _same(a, b):
    assert np.all(np.isfinite(a[0]))
    assert np.array_equal(a[0], b[0]) and a[2] == b[2]
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("L,H,D", SIZES)
@pytest.mark.parametrize("sgs", [0, 2])
def test_split_march_equals_whole(L, H, D, sgs):
    import freeshearlayer_b200 as fsl
    p = temporal_params(L, H, D, deltaT=1e-6, precision=1, sgs=sgs)
    s = random_state(p, seed=3)

    def together(d):  # the multi-domain launch keeps whole marches
        e = fsl.Ensemble([d])
        e.set_chunk(3)
        e.step(3)
        e.sync()
        assert e.persistent() == 1
        e.close()
    _same(_run(fsl.Domain(p), s, lambda d: d.step(3)), _run(fsl.Domain(p), s, together))


@pytest.mark.parametrize("L,H,D", SIZES)
@pytest.mark.parametrize("setup", ["temporal", "spatial"])
@pytest.mark.parametrize("sgs", [0, 2])
def test_split_ppm_march_equals_whole(L, H, D, setup, sgs):
    import freeshearlayer_b200 as fsl
    kw = dict(precision=1, sgs=sgs, recon=fsl.RECON_PPM)
    p = (temporal_params(L, H, D, deltaT=1e-6, **kw) if setup == "temporal"
         else spatial_params(L, H, D, BL_HIG=min(2, H - H // 2), **kw))
    s = random_state(p, seed=5)
    d = fsl.Domain(p)
    d.tune(d.TUNE_STAGE_ROWS, 12)  # a tile height whose marches are never cut
    _same(_run(fsl.Domain(p), s, lambda d: d.step(3)), _run(d, s, lambda d: d.step(3)))
