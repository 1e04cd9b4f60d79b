"""Every variation of the database, alone in an xform of a shared function (the others'
weights are 0), against the function of an xform that has only that variation."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import build
from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn
from tests.twin import variation_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("part", [0, 1])
def test_shared_variations_apply_as_their_own(db, part):
    names = db.variations()[part::2]
    params = variation_params((build.PKG / "config" / "variations_new.yml").read_text())
    rng = np.random.default_rng(part)
    values = {v: {p: float((d if d is not None else rng.uniform(0.3, 1.0)) * rng.uniform(0.6, 1.4)) for p, d in params.get(v, [])}
              for v in names}
    affine = syn._affine(rng)

    def flame(sets):
        g = syn.plain_flame(2)
        g["xforms"] = []
        for s in sets:
            x = syn._xform(np.random.default_rng(3), 0.25, [])
            x["vchain"][0]["transform"] = affine
            x["vchain"][0]["variations"] = {v: ({"weight": w, "parameters": values[v]} if values[v] else w) for v, w in s.items()}
            g["xforms"].append(x)
        return lr.flame.from_json(db, g)

    comp = lr.flame_compiler()
    own = flame([{v: 0.7} for v in names])  # 24 bodies: a function per xform
    ko = comp.get_flame_kernel(db, own, precise_math=1)
    po = ko.prepare_samples(own.pack_samples(4, 256, 256), [0], [0.0])[0]
    pts = np.concatenate([rng.uniform(-1.5, 1.5, (2048, 2)), rng.uniform(0, 1, (2048, 1))], 1).astype(np.float32)
    ks = None
    for i, v in enumerate(names):
        # the variation is live in one xform, and nothing is in the others
        f = flame([{u: 0.7 if u == v and x == i % 4 else 0.0 for u in names} for x in range(4)])
        assert "#define RFK_SHARED 1" in lr.generate_source(db, f)
        ks = ks or comp.get_flame_kernel(db, f, precise_math=1)
        ps = ks.prepare_samples(f.pack_samples(4, 256, 256), [0], [0.0])[0]
        got, want = ks.apply_xform(ps, i % 4, pts, seed=9), ko.apply_xform(po, i, pts, seed=9)
        np.testing.assert_allclose(got[:, 2:], want[:, 2:], rtol=1e-6)
        finite = np.isfinite(want[:, :2]).all(1)
        # the same operations and random draws; a multiply-add contracted differently moves a
        # point by an ulp of its terms, which a formula's conditioning magnifies at few points
        near = np.abs(got[:, :2] - want[:, :2]) <= 1e-5 * np.abs(want[:, :2]).max(1, keepdims=True) + 1e-6
        assert finite.mean() > 0.9 and near[finite].mean() > 0.99, (v, float(near[finite].mean()))
        assert np.array_equal(np.isfinite(got[:, :2]).all(1), finite), v
        assert not ks.apply_xform(ps, (i + 1) % 4, pts, seed=9)[:, :2].any(), v
