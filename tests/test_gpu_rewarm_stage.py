"""Repeated warm-ups of one state with other numbers of packed samples (the
memory they go through grows and is used again), against new states, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tmul", [1, 3])
@pytest.mark.parametrize("make", [syn.plain_flame, syn.hd_flame])
def test_rewarm_with_other_sample_counts(db, make, tmul):
    w, h = 96, 64
    flames = [lr.flame.from_json(db, make(1)) for _ in range(9)]
    k = lr.flame_compiler().get_flame_kernel(db, flames[0])

    def packed(n, scale):
        one = flames[0].pack_sample(w, h)
        return np.stack([one * (1.0 + 1e-3 * scale * i) for i in range(n)])

    st = k.warmup(packed(4, 1), (w, h), seed=5, count=8, temporal_multiplier=tmul)
    for n, scale, seed in ((9, 2, 6), (4, 3, 7), (5, 1, 8), (9, 1, 8)):
        st.rewarm(packed(n, scale), seed=seed, count=8)
        new = k.warmup(packed(n, scale), (w, h), seed=seed, count=8, temporal_multiplier=tmul)
        assert np.array_equal(np.asarray(st.chains()), np.asarray(new.chains()), equal_nan=True), (n, scale)
    r = k.bin(st, lr.bailout_args(iters=4, millis=0, quality=0))
    assert r.total_passes > 0
