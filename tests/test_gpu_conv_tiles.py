"""The halo-tile convolutions (csrc/nn_conv_tile.cuh) at the edges of their index
work, against the NumPy reference: images of one row, channel counts that leave
half a stage, columns and rows beyond one block, rows too wide for a tile, and the
least weight-gradient workspace. Tolerances as in test_gpu_nn.py: float32
accumulation of bf16 products, one bf16 rounding of bf16 outputs."""

import ctypes

import numpy as np
import pytest

import nn_reference as ref
from py4dstem_gb300 import _native

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _bf16(torch, a):
    return torch.from_numpy(ref.bf16_bits(a).view(np.int16)).cuda()


CASES = [(1, 1, 8, 8, 16), (3, 5, 24, 24, 48), (2, 7, 40, 136, 80), (1, 2, 3200, 8, 16),
         (5, 3, 8, 264, 272), (2, 130, 128, 16, 32)]


@pytest.mark.parametrize("nb,H,W,cin,cout", CASES)
@pytest.mark.parametrize("least", [False, True])
def test_conv_passes(cuda, nb, H, W, cin, cout, least):
    torch = cuda
    lib = _native.lib()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(nb + H + W + cin)
    x = ref.bf16_round(rng.standard_normal((nb, H, W, cin)).astype(np.float32))
    w = ref.bf16_round((rng.standard_normal((cout, 9, cin)) * 0.1).astype(np.float32))
    dy = ref.bf16_round(rng.standard_normal((nb, H, W, cout)).astype(np.float32))
    bias = rng.standard_normal(cout).astype(np.float32)
    tx, tw, tdy = _bf16(torch, x), _bf16(torch, w), _bf16(torch, dy)
    twt = _bf16(torch, np.ascontiguousarray(w.transpose(2, 1, 0)))
    tb = torch.from_numpy(bias).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    y = torch.empty((nb, H, W, cout), dtype=torch.int16, device="cuda")
    dx = torch.empty((nb, H, W, cin), dtype=torch.float32, device="cuda")
    dw = torch.empty((cout, 9, cin), dtype=torch.float32, device="cuda")
    db = torch.empty(cout, dtype=torch.float32, device="cuda")
    splits = min(64, max(1, -(-nb * H * W // 2048)))
    nbytes = (4 * splits * 9 * cin * cout if least else
              int(lib.ptycho_nn_conv3x3_wgrad_workspace_bytes(nb, H, W, cin, cout)))
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    assert lib.ptycho_nn_conv3x3_forward(_p(tx), nb, H, W, cin, _p(tw), _p(tb), cout, 1, _p(y),
                                         _p(err), stream) == 0
    assert lib.ptycho_nn_conv3x3_backward_data(_p(tdy), nb, H, W, cout, _p(twt), cin, _p(dx),
                                               _p(err), stream) == 0
    assert lib.ptycho_nn_conv3x3_backward_weight(_p(tx), _p(tdy), nb, H, W, cin, cout, _p(dw),
                                                 _p(db), _p(ws), nbytes, _p(err), stream) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0

    def close(got, want, terms, step=0.0):
        tol = step * np.abs(want) + 1e-5 * np.sqrt(terms) * np.max(np.abs(want)) + 1e-6
        assert np.all(np.abs(got - want) <= tol)

    got = ref.bf16_to_f32(y.cpu().numpy().view(np.uint16))
    close(got, ref.conv3x3(x, w, bias, relu=True), 9 * cin, 2.0 ** -8)
    close(dx.cpu().numpy(), ref.conv3x3_backward_data(dy, w), 9 * cout)
    want_dw, want_db = ref.conv3x3_backward_weight(x, dy)
    close(dw.cpu().numpy(), want_dw, nb * H * W)
    close(db.cpu().numpy(), want_db, nb * H * W)
