"""The packed wave kernels (csrc/ptycho_wave.cuh) where their work split has
edges: batches below, at and above one position per resident block, patches that
wrap around objects of odd width, exact zeros of the far field, and the batches
that the general kernels take instead."""

import ctypes

import numpy as np
import pytest

from gpu_helpers import gpu_reconstruct, make_state, rel
from oracle.ptycho_np import Oracle
from py4dstem_gb300 import _native, engine

pytestmark = pytest.mark.gpu
OFF = dict(fix_probe_com=False, fix_potential_baseline=False, orthogonalize_probe=False)


def both_schedules(state, **kw):
    lib = _native.lib()
    try:
        lib.ptycho_set_kernel_schedule(128, 3)
        g = gpu_reconstruct(state, **kw)
        lib.ptycho_set_kernel_schedule(128, 1)
        return g, gpu_reconstruct(state, **kw)
    finally:
        lib.ptycho_set_kernel_schedule(128, 0)


@pytest.mark.parametrize("J,batch", [(1, 1), (152, 152), (153, 153), (400, 331)])
@pytest.mark.parametrize("potential", [False, True])
def test_resident_blocks_walk_the_batch(cuda, J, batch, potential):
    """Per-position results of a block's first and later positions, and the probe
    terms it sums: float32 rounding (about 1e-7 a term, 1e-6 after the update)
    away from the general kernel."""
    st = make_state(S=128, J=J, potential=potential, seed=J, obj_px=2 * 128 + 31)
    g, b = both_schedules(st, num_iter=1, max_batch_size=batch, seed_random=3, **OFF)
    assert rel(g[0], b[0]) < 2e-6
    assert rel(g[1], b[1]) < 2e-6
    assert abs(g[2][0] - b[2][0]) < 2e-6 * b[2][0]


@pytest.mark.parametrize("S", [32, 48, 64, 96, 128])
@pytest.mark.parametrize("width", [0, 1])
def test_wrapped_patches(cuda, S, width):
    """Patches that wrap around every edge of objects of even and odd width, at
    even and odd corners."""
    st = make_state(S=S, J=16, seed=S + width, obj_px=S + 20 + width)
    rng = np.random.default_rng(S)
    st.positions_px = rng.uniform(-3.0, S + 23.0, size=(16, 2)).astype(np.float32)
    o = Oracle(st)
    o.reconstruct(num_iter=1, max_batch_size=16, seed_random=1, **OFF)
    obj, probe, err = gpu_reconstruct(st, num_iter=1, max_batch_size=16, seed_random=1, **OFF)
    assert rel(obj, o.object) < 2e-5
    assert rel(probe, o.probe) < 2e-5
    assert abs(err[0] - o.error_iterations[0]) < 2e-5 * o.error_iterations[0]


@pytest.mark.parametrize("S", [64, 128])
def test_exact_zeros_and_extreme_values(cuda, S):
    """A zero probe has phase 0 everywhere (the object term is 0 and the probe
    takes the amplitudes' transform); a probe of 1e-18 squares below the fast
    range of the projection; an infinite amplitude makes the error non-finite."""
    st = make_state(S=S, J=6, seed=5)
    for factor in (0.0, 1e-18):
        st.probe = (make_state(S=S, J=6, seed=5).probe * np.float32(factor)).astype(np.complex64)
        o = Oracle(st)
        o.reconstruct(num_iter=1, max_batch_size=6, seed_random=1, **OFF)
        obj, probe, err = gpu_reconstruct(st, num_iter=1, max_batch_size=6, seed_random=1, **OFF)
        assert np.allclose(probe, o.probe, rtol=2e-5, atol=2e-5 * np.abs(o.probe).max())
        assert abs(err[0] - o.error_iterations[0]) < 2e-5 * o.error_iterations[0]
    st = make_state(S=S, J=6, seed=5)
    st.amplitudes[3, 1, 2] = np.inf
    with pytest.raises(RuntimeError):
        gpu_reconstruct(st, num_iter=1, max_batch_size=6, seed_random=1, **OFF)


def test_general_kernels_take_what_the_wave_kernels_do_not(cuda):
    """Amplitudes 4 bytes off a 16-byte boundary run the general kernel, with the
    same results."""
    import torch

    lib = _native.lib()
    st = make_state(S=64, J=9, seed=2)

    def batch(offset):
        s = engine.create_state(
            roi_shape=(64, 64), object_array=st.object, probe_array=st.probe,
            amplitudes=st.amplitudes, positions_px=st.positions_px, num_slices=1, num_probes=1,
            potential=False, max_batch=9)
        flat = torch.zeros(s.amplitudes.numel() + 4, dtype=torch.float32, device="cuda")
        flat[offset:offset + s.amplitudes.numel()] = s.amplitudes.reshape(-1)
        amps = ctypes.c_void_p(flat.data_ptr() + 4 * offset)
        _native.check(lib.ptycho_gd_batch(
            ctypes.byref(s.geometry), engine._ptr(s.object), engine._ptr(s.probe), amps, None,
            engine._ptr(s.positions), None, 9, 0.5, 1.0, 0, None, None,
            engine._ptr(s.error_accum), engine._ws_ptr(s), s.workspace_bytes,
            engine._stream()))
        return s.object.cpu().numpy(), s.probe.cpu().numpy()

    want = batch(0)
    got = batch(1)
    assert rel(got[0], want[0]) < 2e-6 and rel(got[1], want[1]) < 2e-6
