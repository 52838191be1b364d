"""Which kernels a call takes, as far as the host decides it: no GPU needed."""

import ctypes

import pytest

from py4dstem_gb300 import _native, multiscan


@pytest.fixture(scope="module")
def lib():
    return _native.lib()


def test_schedule_can_be_read_without_setting_it(lib):
    prev = lib.ptycho_set_kernel_schedule(128, 2)
    try:
        assert lib.ptycho_get_kernel_schedule(128) == 2
        assert lib.ptycho_get_kernel_schedule(64) == 0
    finally:
        lib.ptycho_set_kernel_schedule(128, prev)
    assert lib.ptycho_get_kernel_schedule(128) == prev


def test_multiscan_graph_lookup_leaves_the_schedule_alone(monkeypatch, lib):
    """Looking up a captured graph must not write the process-wide setting, not
    even to put it back: other threads' batches read it meanwhile."""
    calls = []

    class Recorder:
        def __getattr__(self, name):
            calls.append(name)
            return getattr(lib, name)

    monkeypatch.setattr(multiscan._native, "lib", lambda: Recorder())
    scans = multiscan.MultiScanReconstruction.__new__(multiscan.MultiScanReconstruction)
    scans._graphs = {(True, lib.ptycho_get_kernel_schedule(128)): "graph"}
    assert scans._graph(True) == "graph"
    assert "ptycho_set_kernel_schedule" not in calls


@pytest.mark.parametrize("roi,obj,batch", [(32, 1024, 500), (32, 1450, 64), (96, 1000, 60)])
def test_noalloc_takes_batches_that_fit_without_the_copies(lib, roi, obj, batch):
    """ptycho_workspace_bytes includes room for copies of the object that a batch can
    do without: the entry point without allocation refuses by what is needed. (The
    null object stops the call before any GPU work.)"""
    g = _native.Geometry(roi, roi, obj, obj, 1, 1, 0, 0)
    assert lib.ptycho_workspace_bytes(ctypes.byref(g), batch) > 32 << 20
    p = ctypes.c_void_p(0x1000)
    assert lib.ptycho_gd_batch_noalloc(ctypes.byref(g), None, p, p, None, p, None, batch, 0.5,
                                       1.0, 0, None, None, p, None) != 3
    assert lib.ptycho_gd_batch_noalloc(ctypes.byref(g), None, p, p, None, p, None, 4 * batch + 500,
                                       0.5, 1.0, 0, None, None, p, None) == 3


@pytest.mark.parametrize("nb,H,W", [(1, 1, 1 << 30), (1, 1 << 20, 1 << 10), (255, 2895, 2896)])
def test_wgrad_workspace_of_the_largest_images(lib, nb, H, W):
    """Near 2^31 pixels the padded line of pixels no longer fits an int: the parts
    of the gathered GEMM, at most 64, are all the workspace that is asked for."""
    parts = 4 * 9 * 16 * 32
    assert lib.ptycho_nn_conv3x3_wgrad_workspace_bytes(nb, H, W, 16, 32) == 64 * parts
