"""The convolutions' 32-byte rows and the weight gradient's several CTAs per SM.
Small whole numbers make every product and sum exact in FP32, so results are equal."""
import ctypes as C

import pytest

from parallelcmacionize_b200 import _lib
from parallelcmacionize_b200.warmstart import UNet

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _ints(shape, seed, top=2):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(-top, top + 1, shape, generator=g).to(torch.bfloat16).cuda()


def _taps(x):
    """x (B, Z, Y, X, C) at the 27 taps, zero outside."""
    B, Z, Y, X, c = x.shape
    p = torch.zeros((B, Z + 2, Y + 2, X + 2, c), dtype=torch.float64, device="cuda")
    p[:, 1:-1, 1:-1, 1:-1] = x.double()
    return [p[:, a:a + Z, b:b + Y, d:d + X] for a in range(3) for b in range(3) for d in range(3)]


@pytest.mark.parametrize("cin,cout,shape", [
    (16, 16, (1, 4, 16, 16)), (48, 16, (2, 4, 16, 24)), (32, 48, (1, 2, 8, 8)),
    (16, 16, (1, 32, 64, 64))])
def test_rows_at_any_16_byte_offset(cin, cout, shape):
    B, Z, Y, X = shape
    net = UNet()
    try:
        x = _ints(shape + (cin,), 1)
        w = _ints((cout, 27, cin), 2).float()
        packed = torch.zeros(27 * cin * cout, dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        _lib.check_unet(net._L.cmi_unet_pack_weights(
            net._h, C.c_void_p(w.data_ptr()), cout, cin, 0, C.c_void_p(packed.data_ptr())))
        n = B * Z * Y * X * cout
        outs = []
        for shift in (0, 8):  # elements: 32- and 16-byte aligned rows
            buf = torch.full((n + 32,), 7.0, dtype=torch.bfloat16, device="cuda")
            torch.cuda.synchronize()
            _lib.check_unet(net._L.cmi_unet_conv3(
                net._h, C.c_void_p(x.data_ptr()), cin, C.c_void_p(packed.data_ptr()), None,
                C.c_void_p(buf.data_ptr() + 2 * shift), cout, 0, B, (C.c_int32 * 3)(X, Y, Z)))
            torch.cuda.synchronize()
            assert (buf[:shift] == 7.0).all() and (buf[shift + n:] == 7.0).all()
            outs.append(buf[shift:shift + n].clone())
        ref = sum(t @ w[:, k].double().T for k, t in enumerate(_taps(x)))
        assert torch.equal(outs[0], ref.reshape(-1).to(torch.bfloat16))
        assert torch.equal(outs[0], outs[1])
    finally:
        net.close()


@pytest.mark.parametrize("cin,cout,shape", [
    (16, 16, (1, 1, 16, 8)),      # one tile
    (16, 16, (1, 32, 64, 64)),    # three units: two CTAs per SM, several tiles each
    (16, 16, (2, 10, 8, 72)),     # 8 x 8 x 2 tiles
    (48, 16, (1, 5, 64, 64)), (32, 48, (1, 3, 32, 40))])
def test_weight_gradient_is_exact(cin, cout, shape):
    B, Z, Y, X = shape
    net = UNet()
    try:
        x, dy = _ints(shape + (cin,), 3, 1), _ints(shape + (cout,), 4, 1)
        dw = torch.empty((cout, 27, cin), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        _lib.check_unet(net._L.cmi_unet_conv3_wgrad(
            net._h, C.c_void_p(x.data_ptr()), cin, C.c_void_p(dy.data_ptr()), cout, B,
            (C.c_int32 * 3)(X, Y, Z), C.c_void_p(dw.data_ptr())))
        d = dy.double().reshape(-1, cout)
        ref = torch.stack([d.T @ t.reshape(-1, cin) for t in _taps(x)], dim=1)
        assert torch.equal(dw.double(), ref)
    finally:
        net.close()
