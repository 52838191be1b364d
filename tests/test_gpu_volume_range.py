"""Volume rotation for float32 results at the top of the float32 range: the spline
coefficients reach 27 times the largest voxel and the recursions 403 times, so
float pairs need their scale; sums beyond the range are infinite, as float64
arithmetic rounded to float32 gives them, and never NaN."""

import numpy as np
import pytest
from scipy.ndimage import affine_transform

from py4dstem_gb300.tomography import VolumeOps, rotation_transform

pytestmark = pytest.mark.gpu

TOP = np.finfo(np.float32).max


def _volume(kind, shape):
    rng = np.random.default_rng(5)
    if kind == "alternating":  # the pattern with the largest coefficients
        i = np.indices(shape).sum(0)
        return np.where(i % 2 == 0, TOP, -TOP).astype(np.float32)
    if kind == "constant":
        return np.full(shape, TOP, np.float32)
    return (rng.uniform(-1.0, 1.0, size=shape) * float(TOP)).astype(np.float32)


@pytest.mark.parametrize("kind", ["alternating", "constant", "random"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("mode", [0, 2])
def test_rotation_at_the_top_of_the_range(cuda, kind, dtype, mode):
    import torch

    shape = (12, 33, 20)
    vol = _volume(kind, shape)
    c, s = np.cos(np.deg2rad(10.0)), np.sin(np.deg2rad(10.0))
    rot = np.array([[1, 0, 0], [0, c, -s], [0, s, c]])
    tf, off = rotation_transform(shape, rot)
    want = affine_transform(vol.astype(np.float64), tf, offset=off, order=3, mode="constant")
    out = torch.zeros(shape, dtype=torch.float32, device="cuda")
    if mode == 2:
        start = np.where(np.random.default_rng(6).random(shape) < 0.5, -0.75, 0.5) * float(TOP)
        out.copy_(torch.from_numpy(start.astype(np.float32)))
        want = want + start.astype(np.float32).astype(np.float64)
    VolumeOps(shape, 1, torch.device("cuda")).rotate(
        torch.from_numpy(vol.astype(dtype)).cuda(), out, rot, mode)
    got = out.cpu().numpy().astype(np.float64)
    limit = float(TOP)
    # half an ulp and a pair error of 1e-12 of the largest coefficient
    tol = 6.1e-8 * np.abs(want) + 27e-12 * limit
    inside = np.abs(want) < limit * (1 - 1e-7)
    over = np.abs(want) > limit * (1 + 1e-7)
    assert not np.isnan(got).any()
    assert np.all(np.abs(got - want)[inside] <= tol[inside])
    assert np.all(got[over] == np.sign(want[over]) * np.inf)
