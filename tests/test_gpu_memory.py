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


def _optics(call, X, eps, cap):
    from sdbscan_gb300 import capi
    n, d = X.shape
    e = capi.Engine(n, d)
    e.set_debug_limits(device_bytes_cap=cap)
    try:
        if call == "soptics":
            e.set_params(n_proj=64, topK=3, topM=50, random_seed=4)
            e.fit_soptics(X, eps, 3)
        else:
            e.set_sng_params(samplingProb=0.2, random_seed=4)
            e.set_sng_sampling(1 if call == "sngoptics shared" else 2)
            e.fit_sngoptics(X, eps, 3)
        return e.optics() + (e.core()[1],)
    finally:
        e.close()


def _table_bytes(X, eps, prob, seed):
    """sngOptics' tables for per-block samples: 8 bytes a slot, a power of two of
    at least twice a point's passes with repeats (k_sng_blocks.cu's draws)."""
    def mix(z):
        with np.errstate(over="ignore"):
            z = z + np.uint64(0x9E3779B97F4A7C15)
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            return z ^ (z >> np.uint64(31))
    n = len(X)
    S = int(np.ceil(np.float32(prob) * np.float32(n)))
    Y = X.astype(np.float64)
    Y /= np.linalg.norm(Y, axis=1, keepdims=True)
    key = mix(np.array([seed], np.uint64))[0]
    degree = np.zeros(n, np.int64)
    for b in range((n + 31) // 32):
        with np.errstate(over="ignore"):
            z = mix(key + np.arange(b * S, (b + 1) * S, dtype=np.uint64))
        q = (((z >> np.uint64(32)) * np.uint64(n)) >> np.uint64(32)).astype(np.int64)
        p = np.arange(32 * b, min(n, 32 * b + 32))
        ok = (1.0 - Y[q] @ Y[p].T <= eps) & (q[:, None] != p[None, :])
        np.add.at(degree, q, ok.sum(1))
        degree[p] += ok.sum(0)
    return 8 * sum(max(2, 1 << int(2 * c - 1).bit_length()) for c in degree if c)


@pytest.mark.parametrize("call", ["soptics", "sngoptics blocks"])
def test_ordering_needs_no_memory_beyond_the_lists(call):
    """The regrouped lists (8 bytes an entry) take the place of what the stages
    before need, or come over in pieces: beyond a fit without entries, a fit
    needs the lists (8 bytes an entry) and sngOptics its tables."""
    n = 700
    X = _data(n, 10, 7)
    eps = 1.5
    order, reach, degree = _optics(call, X, eps, 0)
    entries = int(degree.sum())
    tables = _table_bytes(X, eps, 0.2, 4) if call == "sngoptics blocks" else 0
    if call == "soptics":  # the regrouped lists would not fit where the distances were
        assert 8 * entries > 4 * n * 6 * 50 + (1 << 18)
    assert 8 * entries > 1 << 20
    cap = _smallest_cap(lambda c: _optics(call, X, eps, c))
    base = _smallest_cap(lambda c: _optics(call, X, 1e-12, c))
    assert cap - base < 8 * entries + tables + (1 << 17), (cap, base, entries, tables)
    got = _optics(call, X, eps, cap)
    for a, b in zip(got, (order, reach, degree)):
        np.testing.assert_array_equal(a, b)
