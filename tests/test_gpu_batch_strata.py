"""The xform picks of batched renders: every chain picks independently with the
weights' chances, whatever the launch shape (stratified assignment of a
power-of-two number of chains, pick and sort of others).

Three maps x / 8 + t (t = -0.25, 0, 0.25) put a chain into a strip of the image
that names its last two xforms. The counts are held against the products of the
chances within 6 standard deviations: at most D p (1 - p) of variance for one
pick of independent draws, 3 D p for two neighbouring picks (a draw shares a pick
with the draws before and after it)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

W, H, SPP = 2048, 64, 128.0


def _strips(density):
    """Sums of the runs of columns that are parted by 8 empty columns or more."""
    col = density.sum(axis=0)
    at = np.flatnonzero(col)
    runs = np.split(at, np.flatnonzero(np.diff(at) > 8) + 1)
    return [col[r[0]:r[-1] + 1].sum() for r in runs]


@pytest.mark.parametrize("block,cpt,sort", [(256, 8, 2), (256, 1, 2), (128, 4, 2), (32, 1, 2), (96, 8, 2), (256, 8, 1), (256, 1, -1)])
@pytest.mark.parametrize("weights", [(0.5, 0.3, 0.2), (0.9, 0.0, 0.1), (0.0, 0.35, 0.65), (0.7, 0.3, 0.0), (0.004, 0.496, 0.5),
                                     (0.0, 0.0, 0.0)])
def test_batch_picks_follow_the_weights(db, weights, block, cpt, sort):
    g = syn.plain_flame(0)
    g["xforms"] = [{"weight": wt, "color": 0.5, "color_speed": 0.5, "opacity": 1.0,
                    "vchain": [{"transform": [0.125, 0, 0, 0.125, tx, 0], "mod_x": 0, "mod_y": 0, "mod_scale": 1,
                                "mod_rotate": 0, "variations": {"linear": 1.0}}]}
                   for wt, tx in zip(weights, (-0.25, 0.0, 0.25))]
    g.pop("final_xform", None)
    g.update(center_x=0.0, center_y=0.0, rotate=0.0, scale=16.0)  # about 1000 pixels a unit
    f = lr.flame.from_json(db, g)
    k = lr.flame_compiler().get_flame_kernel(db, f, block=block, chains_per_thread=cpt, sort=sort, flush=4)
    b = lr.batch(k, [lr.batch_unit(W, H, SPP, segment=0, t=0.0)], 4, out_format=-1, seed=7)
    b.set_samples(f.pack_samples(4, W, H))
    b.run()
    _, per = b.wait()
    got = _strips(b.bins(0).cpu().numpy().astype(np.float64)[..., 3])
    D = float(per[0].draw_count)
    assert sum(got) == D
    p = np.array(weights) if sum(weights) > 0 else np.array([1.0, 0.0, 0.0])
    p = p / p.sum()
    p = p[p > 0]
    n = len(p)
    assert len(got) == n * n  # an xform of weight 0 is never picked
    got = np.array(got).reshape(n, n)
    fits = []
    for c, q in ((got, p), (got, p[::-1])):  # strips by x, which may run either way
        one, two = c.sum(axis=1), np.outer(q, q)
        fits.append(np.all(np.abs(one - D * q) <= 6 * np.sqrt(D * q * (1 - q)))
                    and np.all(np.abs(c - D * two) <= 6 * np.sqrt(3 * D * two)))
    assert any(fits), (got / D, p)
