"""Objects with more rows or columns than 16 bits count: the object reduction's
tile origins and the packed kernels' copies of the object, against the oracle
(float32 rounding, 2e-5 as in test_gpu_wave.py)."""

import numpy as np
import pytest

from gpu_helpers import gpu_reconstruct, make_state, rel
from oracle.ptycho_np import Oracle

pytestmark = pytest.mark.gpu
OFF = dict(fix_probe_com=False, fix_potential_baseline=False, orthogonalize_probe=False)


def _check(S, shape, positions):
    st = make_state(S=S, J=len(positions), seed=11, obj_px=S + 40)
    rng = np.random.default_rng(shape[0])
    st.object = np.exp(0.3j * rng.standard_normal(shape)).astype(np.complex64)
    st.fov_mask_inverse = np.zeros(shape, bool)
    st.positions_px = np.array(positions, np.float32)
    o = Oracle(st)
    kw = dict(num_iter=1, max_batch_size=len(positions), seed_random=1, **OFF)
    o.reconstruct(**kw)
    obj, probe, err = gpu_reconstruct(st, **kw)
    assert rel(obj, o.object) < 2e-5
    assert rel(probe, o.probe) < 2e-5
    assert abs(err[0] - o.error_iterations[0]) < 2e-5 * o.error_iterations[0]


LONG = [17.2, 100.3, 107.9, 20000.4, 32760.1, 33000.0, 39990.2]


@pytest.mark.parametrize("length", [40000, 70000])
@pytest.mark.parametrize("axis", [0, 1])
def test_tiles_of_long_objects(cuda, length, axis):
    """Patches that start inside a tile, near the start, in the middle and across
    the end of objects of more than 2^15 and 2^16 pixels on one axis."""
    pos = [(40.0 + 3 * i, x + (length - 40000 if i > 3 else 0)) for i, x in enumerate(LONG)]
    shape = (80, length) if axis else (length, 80)
    _check(48, shape, pos if axis else [p[::-1] for p in pos])


def test_copies_of_long_objects(cuda):
    """More rows than a grid's second axis holds (65535), on a packed kernel."""
    _check(96, (70000, 128), [(x + (30000 if i > 3 else 0), 60.0 + 3 * i)
                              for i, x in enumerate(LONG)])
