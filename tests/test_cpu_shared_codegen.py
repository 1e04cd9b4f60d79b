"""Which flames share one xform function (union-of-variations kernels), and that
the shared form compiles, with and without a final xform."""
import pytest

from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn


def _union(db, n, final):
    flames = [lr.flame.from_json(db, syn.hd_flame(s, n_xforms=4 + s % 5, final=final)) for s in range(n)]
    return lr.align_flames(db, flames)[0]


@pytest.mark.parametrize("final", [False, True])
def test_union_kernels_share_one_function(final):
    db = lr.flamedb()
    f = _union(db, 12, final)
    src = lr.generate_source(db, f)
    assert "#define RFK_SHARED 1" in src and "rfk_xf_shared" in src
    lr.compile_check(db, f, "sm_103a")
    lr.compile_check(db, f, "sm_103a", flush=4, chains_per_thread=8, blocks_per_sm=4)


@pytest.mark.parametrize("make", [syn.plain_flame, syn.hd_flame])
def test_single_flames_keep_a_function_per_xform(make):
    db = lr.flamedb()
    src = lr.generate_source(db, lr.flame.from_json(db, make(0)))
    assert "#define RFK_SHARED 0" in src and "RFK_FN R rfk_xf_shared(" not in src
