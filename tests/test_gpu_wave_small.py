"""The packed kernels of the smaller regions (csrc/ptycho_wave.cuh) where they run:
plain gradient descent at 48 x 48 and 64 x 64 from 257 positions a batch (up to 256
the general kernel does), 32 x 32 with two slices or modes. Against the oracle, with
the tolerances of test_gpu_wave.py."""

import numpy as np
import pytest

from gpu_helpers import gpu_reconstruct, make_state, rel
from oracle.ptycho_np import Oracle

pytestmark = pytest.mark.gpu
OFF = dict(fix_probe_com=False, fix_potential_baseline=False, orthogonalize_probe=False)


def _check(st, J, **kw):
    kw = dict(num_iter=1, max_batch_size=J, seed_random=1, **OFF, **kw)
    o = Oracle(st)
    o.reconstruct(**kw)
    obj, probe, err = gpu_reconstruct(st, **kw)
    assert rel(obj, o.object) < 2e-5
    assert np.allclose(probe, o.probe, rtol=2e-5, atol=2e-5 * np.abs(o.probe).max())
    assert abs(err[0] - o.error_iterations[0]) < 2e-5 * o.error_iterations[0]


@pytest.mark.parametrize("S,J,model", [(48, 257, {}), (64, 257, {}), (48, 300, dict(potential=True)),
                                       (32, 16, dict(slices=2)), (32, 16, dict(modes=2))])
@pytest.mark.parametrize("width", [0, 1])
def test_wrapped_patches(cuda, S, J, model, width):
    """Patches that wrap around every edge of objects of even and odd width."""
    st = make_state(S=S, J=J, seed=S + width, obj_px=S + 20 + width, **model)
    st.positions_px = np.random.default_rng(S).uniform(
        -3.0, S + 23.0, size=(J, 2)).astype(np.float32)
    _check(st, J)


@pytest.mark.parametrize("S", [48, 64])
@pytest.mark.parametrize("factor", [0.0, 1e-18])
def test_exact_zeros_and_small_squares(cuda, S, factor):
    """A zero probe (phase 0 everywhere) and one whose far field squares below the
    projection's fast range."""
    J = 257
    st = make_state(S=S, J=J, seed=5)
    st.probe = (st.probe * np.float32(factor)).astype(np.complex64)
    _check(st, J)


@pytest.mark.parametrize("S", [48, 64])
def test_batches_around_the_limit(cuda, S):
    """256 positions in the general kernel, 257 in the packed one."""
    for J in (256, 257):
        _check(make_state(S=S, J=J, seed=S), J)
