"""The line between a function per xform and a shared one, and every variation of the
database in the shared form."""
import numpy as np
import pytest

from refraktor_gb300 import build
from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn
from tests.twin import variation_params

PARAMS = variation_params((build.PKG / "config" / "variations_new.yml").read_text())


def make(names_of, n):
    rng = np.random.default_rng(n)
    g = syn.plain_flame(1)
    g["xforms"] = [syn._xform(rng, 1.0 / n, names_of(i)) for i in range(n)]
    for x in g["xforms"]:
        vs = x["vchain"][0]["variations"]
        for v in vs:
            if PARAMS.get(v):
                vs[v] = {"weight": vs[v], "parameters": {p: 0.5 for p, _ in PARAMS[v]}}
    return g


@pytest.mark.parametrize("xforms,each,union,shared", [(24, 1, 1, 0), (12, 2, 12, 0), (4, 6, 6, 0), (3, 8, 8, 0), (4, 14, 14, 0),
                                                      (10, 7, 14, 0), (71, 1, 14, 0), (12, 6, 6, 1), (12, 6, 12, 1), (6, 12, 12, 1),
                                                      (12, 14, 14, 1)])
def test_72_bodies_share_one_function(db, xforms, each, union, shared):
    f = lr.flame.from_json(db, make(lambda i: [syn.HD_SET[(i * each + j) % union] for j in range(each)], xforms))
    assert f"#define RFK_SHARED {shared}" in lr.generate_source(db, f)


def test_unions_past_the_mask_are_not_shared(db):
    names = db.variations()
    for n, shared in ((32, 1), (33, 0)):
        f = lr.flame.from_json(db, make(lambda i: names[:n], 3))
        assert f"#define RFK_SHARED {shared}" in lr.generate_source(db, f), n


@pytest.mark.parametrize("part", [0, 1])
def test_every_variation_compiles_in_the_shared_form(db, part):
    names = db.variations()[part::2]
    f = lr.flame.from_json(db, make(lambda i: names, 4))
    assert "#define RFK_SHARED 1" in lr.generate_source(db, f)
    lr.compile_check(db, f, "sm_103a")
