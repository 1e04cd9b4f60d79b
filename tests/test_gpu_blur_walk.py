"""The blur kernel's walk at the sizes where it changes: widths around its
32-column strips, heights around its 8-row steps and the rows of a block, and
the three ways a source row is taken (gathered small reach, wide sources one
by one, wide sources gathered), against the FP64 oracle's scatter form."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as orc
from refraktor_gb300 import librefrakt as lr

pytestmark = pytest.mark.gpu


def _bins(w, h, kind):
    rng = np.random.default_rng(w * 1000 + h)
    if kind == "faint":  # every pixel reaches 9 px: rows with more wide sources than taps
        d = np.ones((h, w))
    elif kind == "mixed":  # small reaches with a few wide sources in between
        d = np.where(rng.uniform(size=(h, w)) < 0.1, rng.uniform(0.5, 8.0, size=(h, w)), rng.uniform(20.0, 4000.0, size=(h, w)))
    else:  # isolated sources of every reach
        d = np.where(rng.uniform(size=(h, w)) < 0.05, np.exp(rng.uniform(0.0, 9.0, size=(h, w))), 0.0)
    col = rng.uniform(0, 1, size=(h, w, 3))
    return np.ascontiguousarray(np.concatenate([col * d[..., None], d[..., None]], axis=-1), dtype=np.float32)


def _blur(bins):
    d = torch.from_numpy(bins).cuda()
    out = torch.empty_like(d)
    lr.density_blur(d, out, (bins.shape[1], bins.shape[0]), 9.0, 0.0, 0.5)
    return out.cpu().numpy()


@pytest.mark.parametrize("kind", ["faint", "mixed", "isolated"])
@pytest.mark.parametrize("w,h", [(31, 6), (33, 7), (32, 14), (64, 15), (73, 45), (96, 47), (500, 79)])
def test_blur_matches_oracle_at_strip_and_step_edges(w, h, kind):
    bins = _bins(w, h, kind)
    got = _blur(bins).astype(np.float64)
    ref = orc.density_blur(bins, 9.0, 0.0, 0.5)
    # sums of at most 19 terms per source row and 19 rows of positive values, each
    # term with 4 roundings: (19 + 19 + 4) 2^-24 = 2.5e-6 relative; the 1e-6 of the
    # maximum covers sources whose quantised radius differs by FP32 rounding
    err = np.abs(got - ref)
    assert np.all(err <= 1e-5 * np.abs(ref) + 1e-6 * np.abs(ref).max()), float(err.max())


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_source_stays_in_its_support(bad):
    bins = _bins(90, 60, "mixed")
    bins[30, 40] = (bins[30, 40, 0], 1.0, 2.0, 100.0)  # radius 1: reaches the 3 x 3 pixels around it at most
    clean = _blur(bins)
    bins[30, 40, 0] = bad
    got = _blur(bins)
    near = np.zeros((60, 90), bool)
    near[29:32, 39:42] = True
    np.testing.assert_array_equal(got[..., 1:], clean[..., 1:])
    np.testing.assert_array_equal(got[~near], clean[~near])
    assert not np.isfinite(got[30, 40, 0])
