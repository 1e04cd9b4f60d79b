"""Denoising and the loss run one network: against the image that `denoise` returns
the loss is 0, bit for bit (base + output - (base + output); the inputs keep the image
inside the clamp), at sizes whose convolutions take one and many tiles, bands and
128-pixel columns."""
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import denoise as dn
from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu

WEIGHTS = Path(lr.__file__).resolve().parent / "workloads" / "denoiser_weights.npz"


@pytest.mark.parametrize("w,h", [(16, 16), (136, 72), (264, 200), (1368, 768)])
def test_loss_against_the_denoised_image_is_zero(w, h):
    g = torch.Generator(device="cuda").manual_seed(w)
    d = torch.poisson(40.0 * torch.rand((h, w, 1), device="cuda", generator=g), generator=g)
    bins = torch.cat([torch.rand((h, w, 3), device="cuda", generator=g) * d, d], -1).contiguous()
    base = 0.4 + 0.2 * torch.rand((h, w, 4), device="cuda", generator=g)
    net = dn.denoiser(params=dn.read_params(WEIGHTS))
    out = torch.empty_like(bins)
    net.denoise(bins, base, out, 32.0, fmt=lr.FLOAT4)
    rgb = out[..., :3]
    assert bool(((rgb > 0) & (rgb < 1)).all()) and not torch.equal(rgb, base[..., :3])
    assert net.loss(bins[None], base[None], 32.0, out[None]) == 0.0
    # and it depends on the image
    assert net.loss(bins[None], base[None], 32.0, (out + 0.125)[None]) > 0.0
