"""Calls that have more than one kernel to go to: every route gives the results
of the others, and one call keeps to one route."""

import ctypes
import threading

import numpy as np
import pytest

from gpu_helpers import make_state, rel
from py4dstem_gb300 import _native, engine

pytestmark = pytest.mark.gpu


def _batch(lib, s, n):
    return lib.ptycho_gd_batch(
        ctypes.byref(s.geometry), engine._ptr(s.object), engine._ptr(s.probe),
        engine._ptr(s.amplitudes), None, engine._ptr(s.positions), None, n, 0.5, 1.0, 0, None,
        None, engine._ptr(s.error_accum), engine._ws_ptr(s), s.workspace_bytes, engine._stream())


def test_schedule_set_by_another_thread_during_batches(cuda):
    """A batch takes the 128^2 schedule it finds when it begins: with another
    thread changing it all the time, every batch gives the result that the
    schedules agree on (float32 rounding, 2e-6 as between schedules)."""
    lib = _native.lib()
    J = 331
    st = make_state(S=128, J=J, seed=17, obj_px=2 * 128 + 31)
    s = engine.create_state(
        roi_shape=(128, 128), object_array=st.object, probe_array=st.probe,
        amplitudes=st.amplitudes, positions_px=st.positions_px, num_slices=1, num_probes=1,
        potential=False, max_batch=J)
    obj0, probe0 = s.object.clone(), s.probe.clone()

    def once():
        s.object.copy_(obj0)
        s.probe.copy_(probe0)
        assert _batch(lib, s, J) == 0, lib.ptycho_last_error()
        return s.object.cpu().numpy(), s.probe.cpu().numpy()

    want = once()
    stop = threading.Event()

    def change():
        while not stop.is_set():
            lib.ptycho_set_kernel_schedule(128, 1)
            lib.ptycho_set_kernel_schedule(128, 3)

    t = threading.Thread(target=change)
    t.start()
    try:
        got = [once() for _ in range(400)]
    finally:
        stop.set()
        t.join()
        lib.ptycho_set_kernel_schedule(128, 0)
    assert max(rel(o, want[0]) for o, _ in got) < 2e-6
    assert max(rel(p, want[1]) for _, p in got) < 2e-6


@pytest.mark.parametrize("S,obj,J", [(32, 1024, 500), (96, 1000, 60)])
def test_noalloc_and_least_workspace(cuda, S, obj, J):
    """Batches whose scratch fits without the copies of the object, by both entry
    points, against the full workspace: the same bits where the kernel is the same
    (32), float32 rounding where the copies made the difference (96)."""
    torch = cuda
    lib = _native.lib()
    st = make_state(S=S, J=J, seed=3, obj_px=obj)
    s = engine.create_state(
        roi_shape=(S, S), object_array=st.object, probe_array=st.probe,
        amplitudes=st.amplitudes, positions_px=st.positions_px, num_slices=1, num_probes=1,
        potential=False, max_batch=J)
    assert s.workspace_bytes > 32 << 20
    obj0, probe0 = s.object.clone(), s.probe.clone()

    def run(call):
        s.object.copy_(obj0)
        s.probe.copy_(probe0)
        s.error_accum.zero_()
        assert call() == 0, lib.ptycho_last_error()
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (s.object, s.probe, s.error_accum)]

    want = run(lambda: _batch(lib, s, J))
    got = [run(lambda: lib.ptycho_gd_batch_noalloc(
        ctypes.byref(s.geometry), engine._ptr(s.object), engine._ptr(s.probe),
        engine._ptr(s.amplitudes), None, engine._ptr(s.positions), None, J, 0.5, 1.0, 0, None,
        None, engine._ptr(s.error_accum), engine._stream()))]
    s.workspace_bytes = int(lib.ptycho_workspace_bytes(ctypes.byref(s.geometry), J)) - 1
    got.append(run(lambda: _batch(lib, s, J)))
    for g in got:
        for a, b in zip(g, want):
            if S == 32:
                np.testing.assert_array_equal(a, b)
            else:
                assert rel(a, b) < 2e-6


def _iteration(torch, st, offset, projection=False, correction=False, graph=False):
    J, S = st.amplitudes.shape[0], st.amplitudes.shape[-1]
    flat = torch.zeros(J * S * S + 4, dtype=torch.float32, device="cuda")
    amps = flat[offset:offset + J * S * S].reshape(J, S, S)
    amps.copy_(torch.from_numpy(st.amplitudes))
    s = engine.create_state(
        roi_shape=(S, S), object_array=st.object, probe_array=st.probe, amplitudes=amps,
        positions_px=st.positions_px, num_slices=st.num_slices, num_probes=st.num_probes,
        potential=False, max_batch=J - 1, propagators=st.propagators, projection=projection,
        mixed_state=st.mixed, positions_initial=st.positions_px if correction else None)
    assert s.amplitudes.data_ptr() % 16 == 4 * offset
    drv = engine.IterationDriver(
        s, max_batch=J - 1, projection=projection, step_size=0.5, graph=graph,
        projection_abc=(-1.0, 1.0, 2.0) if projection else (0.0, 0.0, 0.0),
        mean_intensity=st.mean_intensity, fix_probe_com=False, orthogonalize_probe=False,
        **(dict(position_correction=dict(step_size=0.9, max_update_px=0.5, max_total_px=2.0,
                                         center_of_mass=False)) if correction else {}))
    order = np.arange(J) if projection else np.random.default_rng(1).permutation(J)
    drv.iterate(order)
    if graph:
        for _ in range(2):
            drv.iterate(order)
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (s.object, s.probe, s.error_accum, s.positions)]


@pytest.mark.parametrize("model", [dict(), dict(slices=2), dict(modes=2), dict(slices=2, modes=2)])
@pytest.mark.parametrize("kind", ["gd", "projection", "correction"])
@pytest.mark.parametrize("offset", [1, 2])
def test_amplitudes_off_a_boundary(cuda, model, kind, offset):
    """128 x 128 amplitudes that start 4 or 8 bytes off a 16-byte boundary go through
    an aligned copy to the same kernels: the same bits. (Multislice correction and
    batches that keep the far field of projection sets have one kernel anyway.)"""
    st = make_state(S=128, J=11, seed=29, **model)
    kw = dict(projection=kind == "projection", correction=kind == "correction")
    want = _iteration(cuda, st, 0, **kw)
    got = _iteration(cuda, st, offset, **kw)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


def test_amplitudes_off_a_boundary_in_a_graph(cuda):
    """The same inside a captured iteration, and a 96 x 96 batch (general kernel,
    float32 rounding)."""
    st = make_state(S=128, J=11, seed=30)
    for a, b in zip(_iteration(cuda, st, 3, graph=True), _iteration(cuda, st, 0, graph=True)):
        np.testing.assert_array_equal(a, b)
    st = make_state(S=96, J=11, seed=31)
    for a, b in zip(_iteration(cuda, st, 1), _iteration(cuda, st, 0)):
        assert rel(a, b) < 2e-6


@pytest.mark.parametrize("S", [32, 48, 64])
def test_correction_of_small_and_large_batches(cuda, S):
    """A position's correction does not depend on how many others share its batch:
    40 positions corrected alone and among 300, with nothing else updated, move by
    the same bits. (Positions near 0, where float32 shows the last bits of a move.)"""
    torch = cuda
    lib = _native.lib()
    J, few = 300, 40
    st = make_state(S=S, J=J, seed=S, obj_px=S + 24)
    pos = np.random.default_rng(S).uniform(-0.4, 0.4, size=(J, 2)).astype(np.float32)

    def moved(n):
        s = engine.create_state(
            roi_shape=(S, S), object_array=st.object, probe_array=st.probe,
            amplitudes=st.amplitudes, positions_px=pos, num_slices=1, num_probes=1,
            potential=False, max_batch=J, positions_initial=pos)
        s.geometry.flags |= _native.FLAG_KEEP_FARFIELD
        nbytes = int(lib.ptycho_workspace_bytes(ctypes.byref(s.geometry), J))
        ws = torch.empty(nbytes + 256, dtype=torch.uint8, device="cuda")
        ws_ptr = ctypes.c_void_p((ws.data_ptr() + 255) & ~255)
        assert lib.ptycho_gd_batch(
            ctypes.byref(s.geometry), engine._ptr(s.object), engine._ptr(s.probe),
            engine._ptr(s.amplitudes), None, engine._ptr(s.positions), None, n, 0.0, 1.0, 1,
            None, None, engine._ptr(s.error_accum), ws_ptr, nbytes, engine._stream()) == 0
        assert lib.ptycho_position_correction(
            ctypes.byref(s.geometry), engine._ptr(s.object), engine._ptr(s.probe), None,
            engine._ptr(s.amplitudes), None, engine._ptr(s.positions),
            engine._ptr(s.positions_initial), None, n, 0.9, 0.5, 2.0, ws_ptr, nbytes,
            engine._stream()) == 0
        torch.cuda.synchronize()
        return s.positions.cpu().numpy()

    a, b = moved(few), moved(J)
    assert np.all(a[few:] == pos[few:]) and np.all(np.any(a[:few] != pos[:few], axis=1))
    np.testing.assert_array_equal(a[:few], b[:few])
