"""Conversion to floats at the line where small float3 images stop taking one pixel a
thread: every value, flipped and swapped, and nothing written past the image."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("src,cin", [(lr.HALF3, 3), (lr.HALF4, 4)])
@pytest.mark.parametrize("dst,cout", [(lr.FLOAT3, 3), (lr.FLOAT4, 4)])
@pytest.mark.parametrize("w,h,flip", [(1024, 511, True), (1024, 512, True), (1024, 512, False), (1021, 521, False)])
def test_float_conversion_on_both_sides_of_the_size_rule(src, cin, dst, cout, w, h, flip):
    g = torch.Generator(device="cuda").manual_seed(w + h)
    img = (torch.rand((h, w, cin), device="cuda", generator=g) * 3 - 1).half()
    out = torch.full((w * h * cout + 16,), 7.0, device="cuda")
    lr.converter().run(img, out, (w, h), src, dst, flip_y=flip, swap_channels=True)
    v = torch.cat([img.float(), torch.ones((h, w, 1), device="cuda")], -1)[..., [2, 1, 0, 3]]
    want = (v.flip(0) if flip else v)[..., :cout]
    assert torch.equal(out[:w * h * cout].view(h, w, cout), want)
    assert bool((out[w * h * cout:] == 7.0).all())
