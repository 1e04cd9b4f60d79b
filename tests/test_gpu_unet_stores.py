"""The convolution's output path at the edges of its tiles: widths that end inside
a 128-pixel store, odd row counts, two-row 128-channel tiles and (any summation
order) bands of the row-streaming kernel, several per CTA and with a short last
one, into a channel slice of a wider tensor with guard rows behind it."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
F = torch.nn.functional

from refraktor_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("up", [False, True])
@pytest.mark.parametrize("any_order", [False, True])
@pytest.mark.parametrize("n,h,w,cin,cout", [(2, 5, 200, 32, 96), (1, 1, 8, 64, 96), (1, 3, 130, 128, 128), (2, 7, 127, 64, 128),
                                            (1, 9, 129, 32, 32), (1, 5, 72, 64, 64), (2, 1, 257, 128, 256),
                                            (1, 2, 136, 32, 32), (3, 67, 300, 96, 32), (1, 41, 640, 192, 64),
                                            (2, 33, 129, 384, 128)])
def test_conv_stores_only_its_slice(n, h, w, cin, cout, any_order, up):
    L = _lib.lib()
    L.rfk_unet_conv3x3.restype = C.c_int
    L.rfk_unet_conv3x3.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_int,
                                   C.c_void_p, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_int,
                                   C.c_int, C.c_void_p, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(n + 10 * h + w + cin + cout)
    x = torch.randn(n, h, w, cin, device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn(cout, 9, cin, device="cuda", generator=g) / np.sqrt(9 * cin)).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda", generator=g)
    s = 2 if up else 1
    wide, off, guard = cout + 64, 32, 3 * s * w
    px = n * s * h * s * w
    buf = torch.randn(px + guard, wide, device="cuda", generator=g).to(torch.bfloat16)
    before = buf.clone()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = L.rfk_unet_conv3x3(x.data_ptr(), n, h, w, cin, 0, cin, wt.data_ptr(), cout, b.data_ptr(), (5 if up else 1) | (8 if any_order else 0), buf.data_ptr(),
                            wide, off, None, 0, 0, 0, err.data_ptr(), None)
    torch.cuda.synchronize()
    assert rc == 0 and int(err.item()) == 0
    ref = F.conv2d(x.float().permute(0, 3, 1, 2), wt.float().reshape(cout, 3, 3, cin).permute(0, 3, 1, 2), b, padding=1)
    ref = torch.relu(ref).permute(0, 2, 3, 1)
    if up:
        ref = ref.repeat_interleave(2, dim=1).repeat_interleave(2, dim=2)
    got = buf[:px].view(n, s * h, s * w, wide)
    # one bf16 rounding (half an ulp, 2^-8 relative at most) and the summation order of 9 cin f32 products
    bound = ref.abs() * 2.0 ** -8 * 1.01 + 1e-5 * float(ref.abs().max())
    assert bool(((got[..., off:off + cout].float() - ref).abs() <= bound).all())
    assert torch.equal(buf[:px, :off], before[:px, :off]) and torch.equal(buf[:px, off + cout:], before[:px, off + cout:])
    assert torch.equal(buf[px:], before[px:])


@pytest.mark.parametrize("any_order", [False, True])
@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 8, 32, 32), (2, 5, 200, 32, 32), (1, 41, 129, 96, 32), (1, 3, 130, 64, 64)])
def test_conv_rgb_output_is_the_f32_output(n, h, w, cin, cout, any_order):
    """The first four channels, one float4 per pixel and nothing past them, bit for bit as the full f32 output has them."""
    L = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(w + cin)
    x = torch.randn(n, h, w, cin, device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn(cout, 9, cin, device="cuda", generator=g) / np.sqrt(9 * cin)).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda", generator=g)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = []
    for flag, cs in ((2, cout), (16, 4)):
        buf = torch.full((n * h * w * cs + 64,), 7.0, device="cuda")
        rc = L.rfk_unet_conv3x3(x.data_ptr(), n, h, w, cin, 0, cin, wt.data_ptr(), cout, b.data_ptr(), flag | (8 if any_order else 0),
                                buf.data_ptr(), cs, 0, None, 0, 0, 0, err.data_ptr(), None)
        torch.cuda.synchronize()
        assert rc == 0 and int(err.item()) == 0 and bool((buf[n * h * w * cs:] == 7.0).all())
        outs.append(buf[:n * h * w * cs].view(n, h, w, cs))
    assert torch.equal(outs[0][..., :4], outs[1])
