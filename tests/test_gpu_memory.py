"""Fits under a device memory cap (sdb_set_debug_limits): what an engine does
where a buffer does not fit, and what it does after."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, d, seed):
    rng = np.random.default_rng(seed)
    c = rng.standard_normal((6, d))
    return (c[rng.integers(0, 6, n)] + 0.4 * rng.standard_normal((n, d))).astype(np.float32)


def _smallest_cap(fit, lo=1 << 14, hi=1 << 28, step=1 << 12):
    """The smallest cap (to `step` bytes) under which fit(cap) succeeds."""
    from sdbscan_gb300 import capi
    while hi - lo > step:
        mid = (lo + hi) // 2
        try:
            fit(mid)
            hi = mid
        except capi.SdbError as err:
            assert err.status == 6
            lo = mid
    return hi


CALLS = {
    "fit": lambda e, X: e.fit_sdbscan(X, 0.2, 6),
    "sng shared": lambda e, X: e.fit_sngdbscan(X, 0.2, 6),
    "sng blocks": lambda e, X: e.fit_sngdbscan(X, 0.2, 6),
}


def _engine(call, n, d, variant=0):
    from sdbscan_gb300 import capi
    e = capi.Engine(n, d)
    if call.startswith("sng"):
        e.set_sng_params(samplingProb=0.25, random_seed=5)
        e.set_sng_sampling(1 if call == "sng shared" else 2)
    else:
        e.set_params(n_proj=64, topK=3, topM=50, random_seed=5)
        e.set_tile_variant(variant)
    return e


@pytest.mark.parametrize("call", list(CALLS))
def test_a_shortage_turns_the_packed_tile_off_for_that_fit_only(call):
    """A fit under the smallest cap that it runs with drops the packed tile's
    copy; the engine's next fit, without the cap, uses it again."""
    n, d = 2000, 48
    X = _data(n, d, 3)

    def fit(cap):
        e = _engine(call, n, d)
        e.set_debug_limits(device_bytes_cap=cap)
        try:
            CALLS[call](e, X)
            return e.counters()["launches"]
        finally:
            e.close()

    packed = fit(0)
    cap = _smallest_cap(fit)
    e = _engine(call, n, d)
    e.set_debug_limits(device_bytes_cap=cap)
    CALLS[call](e, X)
    want = e.core()
    assert e.counters()["launches"] == packed - 1  # the copy's kernel
    e.set_debug_limits()
    CALLS[call](e, X)
    assert e.counters()["launches"] == packed
    for a, b in zip(e.core(), want):
        np.testing.assert_array_equal(a, b)
    e.close()
