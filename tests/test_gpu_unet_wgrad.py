"""Weight-gradient kernels (and the bias sums they take along) at the edges of their tiles: single rows and odd
heights against stages of two rows, one and several 64-pixel segments, output
channels that fill a part of a 128-channel tile, one row per CTA at the image's
edges, unaligned gradients, against a 64-bit sum.

Products of bf16 values are exact in f32, so only the K additions of a sum round,
each by at most 2^-23 of a partial sum (truncation), which the sum of the
magnitudes bounds: |error| <= K 2^-23 sum |dy| |x|."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu


def _taps(dy, x):
    n, h, w, co = dy.shape
    X = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    D = dy.reshape(-1, co)
    t = [D.T @ X[:, a:a + h, b:b + w].reshape(-1, x.shape[3]) for a in range(3) for b in range(3)]
    return torch.stack(t, dim=1)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,h,w", [(1, 1, 64), (2, 2, 64), (3, 3, 192), (1, 17, 128), (20, 16, 64)])
@pytest.mark.parametrize("cin,cout", [(32, 32), (96, 32), (64, 32), (32, 64), (64, 64), (192, 64), (128, 64), (64, 96), (32, 128),
                                      (96, 160), (256, 256)])
def test_wgrad_edges(n, h, w, cin, cout, offset):
    L = lr.lib()
    L.rfk_unet_wgrad3x3_bias.restype = C.c_int
    L.rfk_unet_wgrad3x3_bias.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 7 + [C.c_void_p] * 4
    g = torch.Generator(device="cuda").manual_seed(cin + 3 * cout + h)
    dy = torch.randn(n, h, w, cout, device="cuda", generator=g).bfloat16()
    wide = torch.randn(n, h, w, cin + 64, device="cuda", generator=g).bfloat16()
    buf = torch.zeros(cout * 9 * cin + 8, device="cuda")
    dw = buf[offset:offset + cout * 9 * cin].view(cout, 9, cin)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    db = torch.zeros(cout + 8, device="cuda")
    assert L.rfk_unet_wgrad3x3_bias(dy.data_ptr(), wide.data_ptr(), cin + 64, 32, n, h, w, cout, cin, dw.data_ptr(),
                                    db.data_ptr(), err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    d, x = dy.double(), wide[..., 32:32 + cin].double()
    bound = n * h * w * 2.0 ** -23 * _taps(d.abs(), x.abs())
    assert bool(((dw.double() - _taps(d, x)).abs() <= bound).all())
    assert bool(((db[:cout].double() - d.sum((0, 1, 2))).abs() <= n * h * w * 2.0 ** -23 * d.abs().sum((0, 1, 2))).all())
    assert float(db[cout:].abs().sum()) == 0.0
    assert float(buf[:offset].abs().sum()) == 0.0 and float(buf[offset + cout * 9 * cin:].abs().sum()) == 0.0
