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
