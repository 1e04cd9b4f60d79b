"""A union kernel's shared xform function applies every xform of an aligned flame
as the flame's own kernel (one function per xform) applies the original's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("final", [False, True])
def test_shared_function_applies_as_the_flames_own(final):
    db = lr.flamedb()
    comp = lr.flame_compiler()
    genomes = [syn.hd_flame(s, n_xforms=4 + s % 5, final=final) for s in range(12)]
    flames = [lr.flame.from_json(db, g) for g in genomes]
    aligned = lr.align_flames(db, flames)
    ku = comp.get_flame_kernel(db, aligned[0], precise_math=1)
    rng = np.random.default_rng(1)
    pts = np.concatenate([rng.uniform(-2, 2, size=(4096, 2)), rng.uniform(0, 1, size=(4096, 1))], 1).astype(np.float32)
    for i in (0, 3, 7):
        k = comp.get_flame_kernel(db, flames[i], precise_math=1)
        pu = ku.prepare_samples(aligned[i].pack_samples(4, 640, 360), [0], [0.0])[0]
        po = k.prepare_samples(flames[i].pack_samples(4, 640, 360), [0], [0.0])[0]
        for x in list(range(len(genomes[i]["xforms"]))) + ([-1] if final else []):
            got, want = ku.apply_xform(pu, x, pts, seed=5), k.apply_xform(po, x, pts, seed=5)
            np.testing.assert_allclose(got[:, 2:], want[:, 2:], rtol=1e-6)  # colour and opacity: one lerp
            # the same IEEE operations on the same parameters; the compiler may contract a
            # multiply-add differently, which moves a point by an ulp of its terms
            ok = np.abs(got[:, :2] - want[:, :2]) <= 1e-5 * np.abs(want[:, :2]) + 1e-6
            assert ok.mean() > 0.999, (i, x, float(ok.mean()))
