"""The tonemap's branches against the FP64 formula: vibrancy 1 with gamma on
both sides of 1, every density magnitude the fast variant's pair arithmetic and
its FP64 fallback take, and non-finite channels; and the vector and scalar paths of
the converter on pixel counts and buffers that are and are not aligned."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu


def _expected(bins, q, gamma, bright, vib):
    b = bins.astype(np.float64)
    d = b[..., 3]
    with np.errstate(all="ignore"):
        f = 0.5 * bright * np.log1p(d * 10.0 ** (-np.log10(q) - 0.5)) / np.log(10.0) / d
        v, w = b[..., :3] * f[..., None], (d * f)[..., None]
        rgb = (1.0 - vib) * v ** (1.0 / gamma) + vib * v * w ** (1.0 / gamma) / w
        a = np.log(d) * (4.0 / np.log(2.0)) / 96.0
    out = np.concatenate([np.clip(rgb, 0, 1), np.clip(a, 0, 1)[..., None]], -1)
    out[d == 0] = 0.0
    return out


@pytest.mark.parametrize("precise", [True, False])
@pytest.mark.parametrize("gamma", [0.8, 1.0, 2.2, 4.0])
@pytest.mark.parametrize("vib", [1.0, 0.4])
def test_tonemap_over_all_magnitudes(precise, gamma, vib):
    rng = np.random.default_rng(3)
    d = np.exp2(rng.uniform(-40.0, 40.0, size=(61, 67))).astype(np.float32)
    d[0, :7] = [0.0, 1.0, 2.0, 4.0, 1e-30, 3e7, 1e-38]
    bins = np.concatenate([(rng.uniform(0, 1, size=d.shape + (3,)) * d[..., None]), d[..., None]], -1).astype(np.float32)
    out = torch.empty((61, 67, 4), device="cuda")
    lr.tonemapper().run(torch.from_numpy(bins).cuda(), out, (67, 61), 64.0, gamma, 4.0, vib, fmt=lr.FLOAT4, precise=precise)
    got, want = out.cpu().numpy().astype(np.float64), _expected(bins, 64.0, gamma, 4.0, vib)
    # precise: the reference bound of 1e-5 relative (log1p, a division and powf of a few ulp each, the exponent's
    # rounding scaled by |log2 w| <= 40); fast: ln(1 + x) loses x below 2^-24 to the sum and lg2.approx has an
    # absolute error of 2^-22, so only densities with x = d k2 above 2^-6 are held, to 1e-4
    if precise:
        assert np.all(np.abs(got - want) <= 1e-5 * want + 1e-7)
    else:
        held = (bins[..., 3] * 10.0 ** (-np.log10(64.0) - 0.5) > 2.0 ** -6)[..., None] & np.ones(4, bool)
        assert np.all((np.abs(got - want) <= 1e-4 * want + 1e-6)[held])


@pytest.mark.parametrize("vib", [1.0, 0.4])
def test_infinite_and_nan_channels_tonemap_to_zero(vib):
    bins = np.full((4, 64, 4), 3.0, np.float32)
    bins[0, :, 0] = np.inf
    bins[1, :, 1] = np.nan
    bins[2, :, 2] = -1.0
    out = torch.empty((4, 64, 4), device="cuda")
    lr.tonemapper().run(torch.from_numpy(bins).cuda(), out, (64, 4), 4.0, 2.2, 4.0, vib, fmt=lr.FLOAT4)
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    assert not got[0, :, 0].any() and not got[1, :, 1].any() and not got[2, :, 2].any()
    assert (got[3, :, :3] > 0).all() and np.array_equal(got[0, :, 1], got[3, :, 1])


@pytest.mark.parametrize("src,cin", [(lr.HALF3, 3), (lr.HALF4, 4)])
@pytest.mark.parametrize("dst,cout,dt", [(lr.UCHAR3, 3, np.uint8), (lr.UCHAR4, 4, np.uint8), (lr.FLOAT3, 3, np.float32),
                                         (lr.FLOAT4, 4, np.float32)])
@pytest.mark.parametrize("w,h,flip,shift", [(1, 1, False, 0), (5, 3, False, 0), (8, 5, True, 0), (7, 4, True, 0), (64, 9, True, 1),
                                            (1027, 3, False, 0)])
def test_convert_vector_and_scalar_paths(src, cin, dst, cout, dt, w, h, flip, shift):
    rng = np.random.default_rng(w + h)
    img = rng.uniform(-0.2, 1.3, size=(h, w, cin)).astype(np.float16)
    img.reshape(-1)[0] = np.nan
    img.reshape(-1)[-1] = np.inf
    v = img.astype(np.float64)
    if cin == 3:
        v = np.concatenate([v, np.ones((h, w, 1))], -1)
    v = v[::-1] if flip else v
    want = v[..., :cout].astype(np.float32)
    if dt == np.uint8:
        want = np.where(np.isnan(v), 255.0, np.clip(v * 255.0, 0.0, 255.0)).astype(np.uint8)[..., :cout]
    # a buffer that starts `shift` elements past an aligned address
    buf = torch.empty(img.size + shift, dtype=torch.float16, device="cuda")
    buf[shift:] = torch.from_numpy(img.reshape(-1)).cuda()
    out = torch.zeros(w * h * cout + 16, dtype=torch.uint8 if dt == np.uint8 else torch.float32, device="cuda")
    lr.converter().run(buf[shift:], out[shift:], (w, h), src, dst, flip_y=flip)
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[shift:shift + w * h * cout].reshape(h, w, cout), want)
    assert not got[:shift].any() and not got[shift + w * h * cout:].any()
