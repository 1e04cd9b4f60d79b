"""Weight and bias gradients of whole numbers, whose f32 sums are exact in any order,
equal bit for bit to 64-bit ones: at sizes where every CTA goes round its ring of
shared-memory stages several times (152 SMs; in brackets stages a CTA takes, and its
ring's), with odd heights and runs that end inside an image column."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu


def _taps(dy, x):
    n, h, w, co = dy.shape
    X = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    D = dy.reshape(-1, co)
    return torch.stack([D.T @ X[:, a:a + h, b:b + w].reshape(-1, x.shape[3]) for a in range(3) for b in range(3)], dim=1)


@pytest.mark.parametrize("n,h,w,cin,cout", [
    (16, 255, 128, 32, 32),   # wgrad3x3_rows<32, 32>: [9 of 2]
    (16, 229, 192, 64, 32),   # <32, 64>: [10 of 3]
    (8, 255, 192, 96, 32),    # <32, 32>, three input tiles: [21 of 2]
    (12, 255, 128, 32, 64),   # <64, 32>: [21 of 5]
    (12, 133, 192, 64, 64),   # <64, 64>: [16 of 4]
    (5, 131, 192, 192, 64),   # three input tiles: [20 of 4]
    (9, 135, 128, 64, 96),    # wgrad3x3_cols, a part of its 128 output channels: [17 of 10]
    (10, 231, 128, 128, 128),  # [62 of 10]
    (3, 517, 64, 256, 256),   # [33 of 10], runs across images
])
def test_whole_numbers_are_exact_round_the_ring(n, h, w, cin, cout):
    L = lr.lib()
    L.rfk_unet_wgrad3x3_bias.restype = C.c_int
    L.rfk_unet_wgrad3x3_bias.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 7 + [C.c_void_p] * 4
    g = torch.Generator(device="cuda").manual_seed(cin + 3 * cout + h)
    dy = torch.randint(-1, 2, (n, h, w, cout), device="cuda", generator=g).bfloat16()
    x = torch.randint(-1, 2, (n, h, w, cin), device="cuda", generator=g).bfloat16()
    assert n * h * w < 2 ** 24
    dw, db = torch.zeros(cout, 9, cin, device="cuda"), torch.zeros(cout, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert L.rfk_unet_wgrad3x3_bias(dy.data_ptr(), x.data_ptr(), cin, 0, n, h, w, cout, cin, dw.data_ptr(), db.data_ptr(),
                                    err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(dw.double(), _taps(dy.double(), x.double()))
    assert torch.equal(db.double(), dy.double().sum((0, 1, 2)))


@pytest.mark.parametrize("n,h,w,cout", [(4, 256, 256, 32), (2, 511, 256, 64), (3, 345, 256, 128), (3, 345, 256, 96)])
def test_bias_sums_past_24_bits_are_exact(n, h, w, cout):
    """Sums of about 3.4e7 whole numbers in steps of 1: exact in 64 bits, not in f32."""
    L = lr.lib()
    L.rfk_unet_wgrad3x3_bias64.restype = C.c_int
    L.rfk_unet_wgrad3x3_bias64.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 7 + [C.c_void_p] * 4
    g = torch.Generator(device="cuda").manual_seed(cout + h)
    dy = torch.randint(0, 256, (n, h, w, cout), device="cuda", generator=g).bfloat16()
    x = torch.zeros((n, h, w, 32), device="cuda", dtype=torch.bfloat16)
    dw, db = torch.zeros(cout, 9, 32, device="cuda"), torch.full((cout + 2,), 0.5, device="cuda", dtype=torch.float64)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert L.rfk_unet_wgrad3x3_bias64(dy.data_ptr(), x.data_ptr(), 32, 0, n, h, w, cout, 32, dw.data_ptr(), db.data_ptr(),
                                      err.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and not dw.any()
    want = dy.double().sum((0, 1, 2))
    assert float(want.min()) > 2 ** 24
    assert torch.equal(db[:cout], want + 0.5) and bool((db[cout:] == 0.5).all())
