"""Volume rotation for float32 results in float pairs (csrc/ptycho_volume.cu) at
the edges of its index work: every choice of the stored innermost axis, extents
below and above a warp and of 1 and 2, coordinates on faces, float64 input, the
adding form, and the scale of the values."""

import numpy as np
import pytest
from scipy.ndimage import affine_transform

from py4dstem_gb300.tomography import VolumeOps, rotation_transform

pytestmark = pytest.mark.gpu


def rotation(axis, deg):
    t = np.deg2rad(deg)
    c, s = np.cos(t), np.sin(t)
    i, j = [k for k in range(3) if k != axis]
    m = np.eye(3)
    m[i, i] = m[j, j] = c
    m[i, j], m[j, i] = -s, s
    return m


@pytest.mark.parametrize("shape", [(33, 40, 65), (5, 34, 3), (1, 32, 2), (2, 1, 31), (40, 2, 34)])
@pytest.mark.parametrize("axis,deg", [(0, 17.0), (1, -50.0), (2, 90.0), (0, 0.0)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_rotation_matches_scipy(cuda, shape, axis, deg, dtype):
    """Results are SciPy's float64 values rounded to float32: half an ulp, plus a
    pair error of 1e-12 of the largest value."""
    import torch

    rng = np.random.default_rng(axis + int(abs(deg)) + shape[0])
    vol = rng.normal(size=shape).astype(dtype)
    add = rng.normal(size=shape).astype(np.float32)
    rot = rotation(axis, deg)
    ops = VolumeOps(shape, 1, torch.device("cuda"))
    tf, off = rotation_transform(shape, rot)
    want = affine_transform(vol.astype(np.float64), tf, offset=off, order=3, mode="constant")
    src = torch.from_numpy(vol).cuda()
    out = torch.empty(shape, dtype=torch.float32, device="cuda")
    ops.rotate(src, out, rot, 0)
    tol = np.spacing(np.abs(want).astype(np.float32)) * 0.5001 + 1e-12 * np.abs(want).max()
    assert np.all(np.abs(out.cpu().numpy().astype(np.float64) - want) <= tol)
    out.copy_(torch.from_numpy(add))
    ops.rotate(src, out, rot, 2)
    total = want + add
    tol = np.spacing(np.abs(total).astype(np.float32)) * 0.5001 + 1e-12 * np.abs(want).max()
    assert np.all(np.abs(out.cpu().numpy().astype(np.float64) - total) <= tol)


@pytest.mark.parametrize("scale", [1e-20, 1e37])
def test_values_far_from_one(cuda, scale):
    import torch

    shape = (12, 33, 20)
    vol = (np.random.default_rng(1).uniform(0.1, 1.0, size=shape) * scale).astype(np.float32)
    rot = rotation(0, 10.0)
    tf, off = rotation_transform(shape, rot)
    want = affine_transform(vol.astype(np.float64), tf, offset=off, order=3, mode="constant")
    ops = VolumeOps(shape, 1, torch.device("cuda"))
    out = torch.empty(shape, dtype=torch.float32, device="cuda")
    ops.rotate(torch.from_numpy(vol).cuda(), out, rot, 0)
    got = out.cpu().numpy().astype(np.float64)
    assert np.all(np.abs(got - want) <= 6.1e-8 * np.abs(want) + 1e-12 * np.abs(want).max())
