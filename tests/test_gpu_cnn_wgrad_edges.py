"""Weight gradients with a work buffer that is not 16-byte aligned, and with inputs
that are not finite at the edge of the volume."""

import numpy as np
import pytest

from oracle import cnn
from tests.test_gpu_cnn import _net_lib, _p, _stream, _t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 2, 3, 4])
@pytest.mark.parametrize("b,d,cin,cout", [(2, 9, 16, 32), (1, 12, 64, 16)])
def test_unaligned_work_buffer(b, d, cin, cout, offset):
    import torch

    L, _ = _net_lib()
    rng = np.random.default_rng(offset + cin)
    do = (d + 1) // 2
    x = cnn.bf16(rng.standard_normal((b, d, d, d, cin)))
    dz = cnn.bf16(rng.standard_normal((b, do, do, do, cout)))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    buf = torch.empty(27 * cin * cout + offset, dtype=torch.float32, device="cuda")
    grad = torch.empty(cout * cin * 27, dtype=torch.float32, device="cuda")
    gb = torch.empty(cout, dtype=torch.float32, device="cuda")
    tx, tdz = _t(x, torch.bfloat16), _t(dz, torch.bfloat16)
    assert L.pmg_cnn_conv_wgrad(_p(tx), _p(tdz), _p(buf[offset:]), _p(grad), _p(gb), b, d, cin, cout, _p(err),
                                _stream()) == 0
    assert L.pmg_cnn_check(_p(err), _stream()) == 0
    _, dw, _ = cnn.conv_bwd(x, np.zeros((cout, cin, 27)), dz)
    assert np.abs(grad.cpu().numpy().reshape(dw.shape) - dw).max() <= 1e-3 * np.abs(dw).max()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("cin", [1, 16])
def test_input_that_is_not_finite_reaches_its_own_tap_alone(cin, bad):
    """An even side: the last column is read by tap 2 of the last output, and would be
    by tap 0 of one beyond it."""
    import torch

    L, _ = _net_lib()
    rng = np.random.default_rng(9)
    d, do, cout = 6, 3, 16
    x = cnn.bf16(rng.standard_normal((1, d, d, d, cin)))
    dz = cnn.bf16(rng.standard_normal((1, do, do, do, cout)))
    _, dw, _ = cnn.conv_bwd(x, np.zeros((cout, cin, 27)), dz)
    for at, tap in (((2, 2, 5), 14), ((2, 5, 2), 16), ((5, 2, 2), 22)):
        xb = x.copy()
        xb[(0,) + at + (0,)] = bad
        tx, tdz = _t(xb, torch.bfloat16), _t(dz, torch.bfloat16)
        err = torch.zeros(1, dtype=torch.int32, device="cuda")
        buf = torch.empty(27 * cin * cout, dtype=torch.float32, device="cuda")
        grad = torch.empty(cout * cin * 27, dtype=torch.float32, device="cuda")
        gb = torch.empty(cout, dtype=torch.float32, device="cuda")
        assert L.pmg_cnn_conv_wgrad(_p(tx), _p(tdz), _p(buf), _p(grad), _p(gb), 1, d, cin, cout, _p(err), _stream()) == 0
        assert L.pmg_cnn_check(_p(err), _stream()) == 0
        got = grad.cpu().numpy().reshape(dw.shape)
        assert not np.isfinite(got[:, 0, tap]).any()
        got[:, 0, tap] = dw[:, 0, tap]
        assert np.abs(got - dw).max() <= 1e-3 * np.abs(dw).max()
