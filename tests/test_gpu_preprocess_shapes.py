"""Centre of mass and normalisation at the shapes the perfect-tree kernels branch on:
one leaf with a tail, few leaves, rows shorter than a chain's step and than the
padded pitch, rows that end within a leaf, non-finite samples. Bits of the host path,
as in test_gpu_preprocess.py."""

import numpy as np
import pytest

from test_gpu_preprocess import _host

pytestmark = pytest.mark.gpu

SHAPES = [(3, 4), (2, 8), (64, 4), (512, 4), (1024, 16), (16, 1024), (64, 24), (32, 48),
          (128, 128), (2048, 1)]


@pytest.mark.parametrize("shape", SHAPES)
def test_com_shapes(cuda, shape):
    from py4dstem_gb300 import device_preprocess

    rng = np.random.default_rng(shape[0] * 7 + shape[1])
    data = rng.random((2, 3) + shape, dtype=np.float32) + 0.1
    kya, kxa = np.meshgrid(np.arange(shape[1], dtype=np.float32),
                           np.arange(shape[0], dtype=np.float32))
    flat = data.reshape(2, 3, -1)
    isum = np.sum(flat, axis=-1)
    ref_x = np.sum(flat * kxa.reshape(1, 1, -1), axis=-1) / isum
    ref_y = np.sum(flat * kya.reshape(1, 1, -1), axis=-1) / isum
    cx, cy = device_preprocess.pattern_com(device_preprocess.upload_intensities(data), None)
    np.testing.assert_array_equal(cx.reshape(2, 3), ref_x)
    np.testing.assert_array_equal(cy.reshape(2, 3), ref_y)


@pytest.mark.parametrize("shape,crop", [(s, False) for s in SHAPES if min(s) > 1] +
                         [((32, 48), True), ((128, 128), True)])
def test_normalize_shapes(cuda, shape, crop):
    from py4dstem_gb300 import device_preprocess

    rng = np.random.default_rng(shape[0] * 5 + shape[1])
    rs = (3, 2)
    data = (rng.random(rs + shape, dtype=np.float32) - 0.1).astype(np.float32)
    data[1, 1, shape[0] // 2, shape[1] // 2] = np.nan
    data[2, 0, 0, 0] = np.inf
    cfx = (shape[0] / 2 + rng.normal(size=rs)).astype(np.float32)
    cfy = (shape[1] / 2 + rng.normal(size=rs)).astype(np.float32)
    with np.errstate(invalid="ignore"):
        ref = _host()._normalize_intensities(data, cfx, cfy, None, crop, False)[0]
    gpu = _host()
    gpu._device = "gpu"
    amps = gpu._normalize_intensities_device(device_preprocess.upload_intensities(data), cfx, cfy,
                                             None, crop)[0]
    np.testing.assert_array_equal(amps.cpu().numpy(), ref)
