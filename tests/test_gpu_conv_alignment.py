"""The weight gradient on activations and gradients that start off a 16-byte
boundary (views into a larger buffer): the tile kernels' 16-byte copies do not
take those, so the gathered GEMM does. Tolerances as in test_gpu_conv_tiles.py."""

import ctypes

import numpy as np
import pytest

import nn_reference as ref
from py4dstem_gb300 import _native

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("x_off,dy_off", [(1, 0), (0, 1), (4, 3)])
@pytest.mark.parametrize("nb,H,W,cin,cout", [(2, 7, 40, 24, 48), (2, 130, 128, 16, 32)])
def test_weight_gradient_of_offset_arrays(cuda, nb, H, W, cin, cout, x_off, dy_off):
    torch = cuda
    lib = _native.lib()
    rng = np.random.default_rng(H + x_off + dy_off)
    x = ref.bf16_round(rng.standard_normal((nb, H, W, cin)).astype(np.float32))
    dy = ref.bf16_round(rng.standard_normal((nb, H, W, cout)).astype(np.float32))

    def at(a, offset):
        flat = torch.zeros(a.size + 8, dtype=torch.int16, device="cuda")
        view = flat[offset:offset + a.size]
        view.copy_(torch.from_numpy(ref.bf16_bits(a).view(np.int16).reshape(-1)).cuda())
        assert view.data_ptr() % 16 == 2 * offset
        return view

    tx, tdy = at(x, x_off), at(dy, dy_off)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dw = torch.empty((cout, 9, cin), dtype=torch.float32, device="cuda")
    db = torch.empty(cout, dtype=torch.float32, device="cuda")
    nbytes = int(lib.ptycho_nn_conv3x3_wgrad_workspace_bytes(nb, H, W, cin, cout))
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    assert lib.ptycho_nn_conv3x3_backward_weight(
        _p(tx), _p(tdy), nb, H, W, cin, cout, _p(dw), _p(db), _p(ws), nbytes, _p(err),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    want_dw, want_db = ref.conv3x3_backward_weight(x, dy)
    for got, want in ((dw, want_dw), (db, want_db)):
        tol = 1e-5 * np.sqrt(nb * H * W) * np.max(np.abs(want)) + 1e-6
        assert np.all(np.abs(got.cpu().numpy() - want) <= tol)
