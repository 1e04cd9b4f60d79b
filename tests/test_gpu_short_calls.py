"""Calls of fewer than 16 passes, checked after each one: the stop flag and the time
budget end them at the next check, as they end long calls."""
import pytest

torch = pytest.importorskip("torch")

from refraktor_gb300 import librefrakt as lr
from refraktor_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def _spp(k, w, h, passes):
    """Quality that takes about `passes` passes of all chains; checks come after each pass below 16."""
    return passes * k.info["grid"] * k.info["block"] * k.info["chains_per_thread"] / (w * h)


@pytest.mark.parametrize("tmul", [1, 3])
def test_abort_stops_a_short_call_at_its_first_check(db, tmul):
    w = h = 256
    f = lr.flame.from_json(db, syn.plain_flame(2))
    k = lr.flame_compiler().get_flame_kernel(db, f)
    s = torch.cuda.Stream()
    busy = k.warmup(f.pack_samples(4, w, h), (w, h), seed=5, count=10, stream=s)
    st = k.warmup(f.pack_samples(4, w, h), (w, h), seed=6, count=10, temporal_multiplier=tmul, stream=s)
    spp = _spp(k, w, h, 12 * tmul)
    full = k.bin(st, lr.bailout_args(iters=0, millis=0, quality=spp), stream=s)
    per_pass = k.info["grid"] * k.info["block"] * k.info["chains_per_thread"]
    assert full.status & 1 and full.total_passes < 16 * tmul * per_pass
    # the abort comes while an earlier call holds the stream
    k.bin_async(busy, lr.bailout_args(iters=0, millis=200, quality=0), stream=s)
    k.bin_async(st, lr.bailout_args(iters=0, millis=0, quality=spp), stream=s)
    st.abort_binning()
    busy.wait()
    r = st.wait()
    assert r.status & 4, r
    assert r.total_passes <= 2 * per_pass, r  # of 12 tmul: the first check, and a block that starts late


def test_abort_of_a_call_with_a_pass_cap(db):
    w = h = 128
    f = lr.flame.from_json(db, syn.plain_flame(2))
    k = lr.flame_compiler().get_flame_kernel(db, f)
    s = torch.cuda.Stream()
    busy = k.warmup(f.pack_samples(4, w, h), (w, h), seed=5, count=10, stream=s)
    st = k.warmup(f.pack_samples(4, w, h), (w, h), seed=6, count=10, stream=s)
    k.bin_async(busy, lr.bailout_args(iters=0, millis=200, quality=0), stream=s)
    k.bin_async(st, lr.bailout_args(iters=8, millis=0, quality=0), stream=s)
    st.abort_binning()
    busy.wait()
    r = st.wait()
    assert r.status & 8 and r.status & 4, r


def test_time_budget_ends_a_call_of_few_slow_passes(db):
    # every chain draws one pixel, whose adds are serial in L2: milliseconds a pass
    g = syn.plain_flame(1)
    for x in g["xforms"]:
        x["vchain"][0]["transform"] = [1e-5, 0.0, 0.0, 1e-5, 0.1, 0.1]
        x["vchain"][0]["variations"] = {"linear": 1.0}
    f = lr.flame.from_json(db, g)
    k = lr.flame_compiler().get_flame_kernel(db, f, block=256, chains_per_thread=8, flush=0)
    w, h = 256, 256
    st = k.warmup(f.pack_samples(4, w, h), (w, h), seed=6, count=2)
    slow = k.bin(st, lr.bailout_args(iters=14, millis=0, quality=0))
    assert slow.elapsed_ms > 2.5, slow  # or no budget fits between
    r = k.bin(st, lr.bailout_args(iters=14, millis=1, quality=_spp(k, w, h, 15)))
    assert r.status & 2, r
    assert r.total_passes < slow.total_passes, r
