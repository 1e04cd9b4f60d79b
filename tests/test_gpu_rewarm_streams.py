"""Re-warming a state with more and more samples, whose memory grows on the way, does
not wait for work on other streams."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def test_growing_rewarms_leave_other_streams_alone(db):
    w, h = 96, 64
    f = lr.flame.from_json(db, syn.plain_flame(1))
    k = lr.flame_compiler().get_flame_kernel(db, f)
    one = f.pack_sample(w, h)
    packed = [np.stack([one * (1.0 + 1e-3 * i) for i in range(n)]) for n in (4, 5, 6, 12, 7, 40, 41)]
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    st = k.warmup(packed[0], (w, h), seed=5, count=4, stream=mine)
    k.warmup(packed[0], (w, h), seed=5, count=4, stream=mine)  # another state, destroyed again
    torch.cuda.synchronize()
    waited = []
    for p in packed:
        with torch.cuda.stream(other):
            torch.cuda._sleep(400_000_000)  # about 0.2 s on one SM
            busy = torch.cuda.Event()
            busy.record()
        st.rewarm(p, seed=6, count=4, stream=mine)
        waited.append(busy.query())
        busy.synchronize()
    assert not any(waited), waited
    new = k.warmup(packed[-1], (w, h), seed=6, count=4)
    assert np.array_equal(np.asarray(st.chains()), np.asarray(new.chains()), equal_nan=True)
