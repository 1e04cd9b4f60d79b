"""Negative channels under a highlight power: their power is NaN, which stores 0, at
vibrancy 1 as just below it; at gamma 1 they are numbers like others."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [1.0, 2.2])
@pytest.mark.parametrize("fmt", [lr.FLOAT3, lr.FLOAT4])
def test_negative_channels_under_a_highlight(gamma, fmt):
    bins = np.zeros((6, 64, 4), np.float32)
    bins[..., :3] = 9e4  # far above 1: the highlight takes the others towards white
    bins[..., 3] = 1e5
    bins[1, :, 0], bins[2, :, 1], bins[3, :, 2], bins[4, :, :2] = -2e4, -1.0, -np.inf, -3e4
    out = {}
    for vib in (1.0, np.nextafter(np.float32(1.0), np.float32(0.0))):
        o = torch.empty((6, 64, 3 if fmt == lr.FLOAT3 else 4), device="cuda")
        lr.tonemapper().run(torch.from_numpy(bins).cuda(), o, (64, 6), 1.0, gamma, 40.0, float(vib), highlight_power=1.0, fmt=fmt)
        out[vib] = o.cpu().numpy()[..., :3]
    a, b = out.values()
    # one ulp of vibrancy moves c^(1/gamma) (up to 9e4) by its 2^-24th part into the sum
    assert np.abs(a - b).max() <= 9e4 * 2.0 ** -23
    lit = a[0].copy()
    assert (lit > 0.5).all()
    if gamma != 1.0:
        assert not a[1, :, 0].any() and not a[2, :, 1].any() and not a[4, :, :2].any()
    assert not a[3, :, 2].any()
