"""State planes between the padded fields and the caller's layout (rows of single
values or of pairs; device buffers in place, host buffers staged), and the row
sums over segments of planes."""
import numpy as np
import pytest

from tests.helpers import random_state, temporal_params

pytestmark = pytest.mark.gpu


# odd and even rows; shorter than, at and past the 128 values a warp keeps in flight
@pytest.mark.parametrize("L,H,D", [(2, 2, 2), (3, 2, 3), (5, 3, 64), (4, 3, 65), (3, 2, 130), (2, 3, 257), (3, 2, 520)])
@pytest.mark.parametrize("offset", [0, 1])  # a device buffer on 16 bytes, on 8 only
def test_planes_round_trip(L, H, D, offset):
    import freeshearlayer_b200 as fsl
    import torch
    p = temporal_params(L, H, D)
    s = random_state(p, seed=3)
    d = fsl.Domain(p)
    ps = d.plane_size()
    for where in ("device", "host"):
        for i0, n in ((1, L), (2, L - 1), (L, 1)):
            d.upload_state(s)
            buf = torch.zeros(n * ps + 2, dtype=torch.float64, device="cuda" if where == "device" else "cpu")
            view = buf[offset:offset + n * ps]
            arg = view if where == "device" else view.numpy()
            d.get_planes(i0, n, arg)
            want = s.reshape(-1)[(i0 - 1) * ps:(i0 - 1 + n) * ps]
            assert np.array_equal(view.cpu().numpy(), want)
            assert float(buf[:offset].abs().sum()) == 0. and float(buf[offset + n * ps:].abs().sum()) == 0.
            view.mul_(2.)
            torch.cuda.synchronize()
            d.set_planes(i0, n, arg)
            ref = s.reshape(-1).copy()
            ref[(i0 - 1) * ps:(i0 - 1 + n) * ps] *= 2.
            assert np.array_equal(d.download_state().reshape(-1), ref)


# one segment, a ragged last one, many
@pytest.mark.parametrize("L,H,D", [(2, 2, 2), (3, 5, 7), (61, 3, 33), (40, 90, 16)])
def test_row_sums(L, H, D):
    import freeshearlayer_b200 as fsl
    p = temporal_params(L, H, D)
    s = random_state(p, seed=4)
    d = fsl.Domain(p)
    d.upload_state(s)
    q = s.reshape(L, H, 5, D)
    r, u, v, w = q[:, :, 0], q[:, :, 1] / q[:, :, 0], q[:, :, 2] / q[:, :, 0], q[:, :, 3] / q[:, :, 0]
    terms = [r, r * u, r * v, r * w, r * u * u, r * v * v, r * w * w, r * u * v]
    got = d.plane_sums()
    # sums of N terms, each side within N + 4 roundings of the magnitudes' sum
    n = L * D
    for c, t in enumerate(terms):
        bound = 2 * (n + 4) * 2. ** -53 * np.abs(t).sum(axis=(0, 2))
        assert (np.abs(got[:, c] - t.sum(axis=(0, 2))) <= bound).all()
