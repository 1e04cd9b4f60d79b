"""Convolutions of 32 dense input channels in the fixed order of sums take pixel
pairs; the same input as a slice of a wider tensor takes single pixels. Both add an
output's products in one order, so they agree bit for bit: at widths that end inside
a tile of 256 pixels, one to many bands and accumulator rings, several tasks per
strip, with and without a mask, into dense tensors, slices and four-channel images."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out", ["dense", "slice", "mask", "rgb"])
@pytest.mark.parametrize("cout", [32, 96])
@pytest.mark.parametrize("n,h,w", [(1, 2, 2), (1, 3, 8), (2, 67, 300), (1, 41, 258), (3, 5, 72), (5, 248, 512), (12, 300, 514),
                                   (40, 130, 256)])
def test_pairs_are_single_pixels_bit_for_bit(n, h, w, cout, out):
    L = _lib.lib()
    L.rfk_unet_conv3x3.restype = C.c_int
    L.rfk_unet_conv3x3.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_int,
                                   C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_int,
                                   C.c_int, C.c_void_p, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(n + 7 * h + w + cout)
    x = torch.randn(n, h, w, 32, device="cuda", generator=g).to(torch.bfloat16)
    wide = torch.randn(n, h, w, 96, device="cuda", generator=g).to(torch.bfloat16)
    wide[..., 32:64] = x
    wt = (torch.randn(cout, 9, 32, device="cuda", generator=g) / np.sqrt(288)).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda", generator=g)
    mask = torch.randn(n, h, w, cout, device="cuda", generator=g).to(torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    cs = {"dense": cout, "mask": cout, "slice": cout + 64, "rgb": 4}[out]
    off = 32 if out == "slice" else 0
    guard = 3 * w * cs
    results = []
    for src, cstride, coff in ((x, 32, 0), (wide, 96, 32)):
        y = torch.full((n * h * w * cs + guard,), 7.0, device="cuda", dtype=torch.float32 if out == "rgb" else torch.bfloat16)
        rc = L.rfk_unet_conv3x3(src.data_ptr(), n, h, w, cstride, coff, 32, wt.data_ptr(), cout,
                                None if out == "mask" else b.data_ptr(), {"rgb": 16, "mask": 0}.get(out, 1), y.data_ptr(), cs, off,
                                mask.data_ptr() if out == "mask" else None, cout if out == "mask" else 0, 0, 0, err.data_ptr(), None)
        torch.cuda.synchronize()
        assert rc == 0 and int(err.item()) == 0
        results.append(y)
    # bit patterns: the same in the output, and untouched around a slice and behind it
    bits = [r.view(torch.int32 if out == "rgb" else torch.int16) for r in results]
    assert torch.equal(bits[0], bits[1])
    assert bool((results[0][n * h * w * cs:] == 7.0).all())
    if out == "slice":
        rows = results[0][:n * h * w * cs].view(-1, cs)
        assert bool((rows[:, :32] == 7.0).all()) and bool((rows[:, 32 + cout:] == 7.0).all())


@pytest.mark.parametrize("n,h,w", [(1, 2, 2), (1, 8, 8), (2, 68, 300), (5, 248, 512), (12, 300, 514)])
def test_pool_in_the_epilogue_is_the_pool_of_the_output(n, h, w):
    L = _lib.lib()
    L.rfk_unet_conv3x3_pool.restype = L.rfk_unet_avgpool.restype = C.c_int
    L.rfk_unet_conv3x3_pool.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_int,
                                        C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_int,
                                        C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    L.rfk_unet_avgpool.argtypes = [C.c_void_p] + [C.c_int] * 6 + [C.c_void_p] * 2
    g = torch.Generator(device="cuda").manual_seed(n + 7 * h + w)
    x = torch.randn(n, h, w, 32, device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn(32, 9, 32, device="cuda", generator=g) / np.sqrt(288)).to(torch.bfloat16)
    b = torch.randn(32, device="cuda", generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    y = torch.zeros(n, h, w, 96, device="cuda", dtype=torch.bfloat16)
    px = n * h * w // 4 * 32
    pools = [torch.full((px + 256,), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    assert L.rfk_unet_conv3x3_pool(x.data_ptr(), n, h, w, 32, 0, 32, wt.data_ptr(), 32, b.data_ptr(), 1, y.data_ptr(), 96, 64,
                                   None, 0, 0, 0, pools[0].data_ptr(), err.data_ptr(), None) == 0
    assert L.rfk_unet_avgpool(y.data_ptr(), n, h, w, 96, 64, 32, pools[1].data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(pools[0].view(torch.int16), pools[1].view(torch.int16))
    # refused: odd heights, other layouts
    assert L.rfk_unet_conv3x3_pool(y.data_ptr(), n, h, w, 96, 0, 32, wt.data_ptr(), 32, b.data_ptr(), 1, x.data_ptr(), 32, 0, None, 0,
                                   0, 0, pools[0].data_ptr(), err.data_ptr(), None) != 0
