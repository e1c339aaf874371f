"""Convolution kernels at the edges of their tiles: sides around the 32-column,
4- and 8-row tiles of the first layer, parity classes with and without a last
odd position, row counts around 128, K around the 64-wide chunks and their
splits, every channel width, against the float64 oracle (tolerances as in
test_gpu_cnn: 1/128 of the value plus 1e-3 of the largest for bf16 outputs, 1e-3
of the largest for fp32 weight gradients)."""

import numpy as np
import pytest

from oracle import cnn
from tests.test_gpu_cnn import _close_bf16, _net_lib, _p, _packed, _stream, _t

pytestmark = pytest.mark.gpu

# (batch, side, c_in, c_out)
CASES = [(3, 2, 16, 16), (1, 5, 16, 64), (2, 9, 64, 16), (3, 11, 32, 32), (5, 4, 64, 64), (1, 17, 16, 32),
         (2, 33, 1, 32), (1, 66, 1, 16), (3, 7, 1, 64), (1, 2, 1, 16), (2, 65, 1, 16)]


@pytest.mark.parametrize("b,d,cin,cout", CASES)
def test_edges_match_oracle(b, d, cin, cout):
    import torch

    L, net = _net_lib()
    rng = np.random.default_rng(1000 * b + d + cin + cout)
    do = (d + 1) // 2
    x = cnn.bf16(np.maximum(rng.standard_normal((b, d, d, d, cin)), 0.0))
    w = cnn.bf16(rng.standard_normal((cout, cin, 27)) / np.sqrt(27 * cin))
    bias = rng.standard_normal(cout) * 0.1
    dz = cnn.bf16(rng.standard_normal((b, do, do, do, cout)))
    wk, wkt = _packed(L, net, w, cin, cout)
    tx, tdz = _t(x, torch.bfloat16), _t(dz, torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    y = torch.empty(b * do ** 3 * cout, dtype=torch.bfloat16, device="cuda")
    assert L.pmg_cnn_conv_fwd(_p(tx), _p(wk), _p(_t(bias, torch.float32)), _p(y), b, d, cin, cout, _p(err),
                              _stream()) == 0
    want = np.maximum(cnn.conv_fwd(x, w, bias), 0.0)
    _close_bf16(y.float().cpu().numpy().reshape(want.shape), want)

    dx_want, dw, db = cnn.conv_bwd(x, w, dz)
    if cin >= 16:
        dx = torch.empty(b * d ** 3 * cin, dtype=torch.bfloat16, device="cuda")
        assert L.pmg_cnn_conv_dgrad(_p(tdz), _p(wkt), _p(tx), _p(dx), b, d, cin, cout, _p(err), _stream()) == 0
        dx_want = dx_want * (x > 0)
        _close_bf16(dx.float().cpu().numpy().reshape(dx_want.shape), dx_want)

    buf = torch.empty(27 * cin * cout, dtype=torch.float32, device="cuda")
    grad = torch.empty(cout * cin * 27, dtype=torch.float32, device="cuda")
    gb = torch.empty(cout, dtype=torch.float32, device="cuda")
    assert L.pmg_cnn_conv_wgrad(_p(tx), _p(tdz), _p(buf), _p(grad), _p(gb), b, d, cin, cout, _p(err), _stream()) == 0
    assert L.pmg_cnn_check(_p(err), _stream()) == 0
    assert np.abs(grad.cpu().numpy().reshape(dw.shape) - dw).max() <= 1e-3 * np.abs(dw).max()
    assert np.abs(gb.cpu().numpy() - db).max() <= 1e-3 * max(1.0, np.abs(db).max())
