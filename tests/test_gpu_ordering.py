"""The sOPTICS ordering as independent floods (csrc/k_order.cu, optics.cu)
against the oracle's one sequential flood: non-core points between two
clusters, non-core points whose turn comes before their cluster's smallest
core point, one flood, none, and enough list entries for several threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clusters(n, d, c, spread, seed, order):
    """c clusters whose edges overlap; order "edges_first" gives the points far
    from their centre the small ids, "edges_last" the large ones."""
    rng = np.random.default_rng(seed)
    centre = rng.standard_normal((c, d))
    y = rng.integers(0, c, n)
    r = rng.random(n) ** 0.5
    z = rng.standard_normal((n, d))
    X = centre[y] + spread * r[:, None] * z
    if order != "mixed":
        i = np.argsort(-r if order == "edges_first" else r, kind="stable")
        X = X[i]
    return np.ascontiguousarray(X.astype(np.float32))


@pytest.mark.parametrize("n,d,c,spread,eps,minPts,order", [
    (3000, 8, 6, 0.6, 0.05, 8, "edges_first"),
    (3000, 8, 6, 0.6, 0.05, 8, "edges_last"),
    (20000, 16, 12, 0.35, 0.06, 10, "mixed"),   # millions of list entries, several threads
    (4000, 6, 1, 0.3, 0.3, 5, "mixed"),         # one flood
    (1500, 12, 5, 0.5, 0.001, 5, "mixed"),      # no core point
    (40, 5, 3, 0.4, 0.1, 3, "edges_first"),
])
def test_ordering_matches_oracle(n, d, c, spread, eps, minPts, order):
    from oracle.oracle import Port, build_port
    from sdbscan_gb300 import capi
    build_port()
    X = _clusters(n, d, c, spread, n + c, order)
    e = capi.Engine(n, d)
    e.set_params(n_proj=256, topK=8, topM=min(60, n), random_seed=4)
    e.fit_soptics(X, eps, minPts)
    ordering, reach = e.optics()
    core, _ = e.core()
    cd = e.core_dist()
    o_order, o_reach, o_core, o_cd, _ = Port().fit_soptics(X, eps, minPts, n_proj=256, topK=8, topM=min(60, n), seed=4,
                                                           threads=4, tie_mode=1)
    np.testing.assert_array_equal(core, o_core)
    np.testing.assert_array_equal(cd, o_cd)
    np.testing.assert_array_equal(ordering, o_order)
    np.testing.assert_array_equal(reach, o_reach)
    e.fit_soptics(X, eps, minPts)  # again on the same engine
    np.testing.assert_array_equal(e.optics()[0], o_order)
    np.testing.assert_array_equal(e.optics()[1], o_reach)
    e.close()


def test_ordering_takes_the_distances_memory_when_there_is_no_other():
    """The floods' copy of the lists fits where the pair distances were: the
    fit needs the two list arrays (8 bytes an entry) beyond a fit without
    entries, and less than that plus the copy (16 bytes an entry)."""
    from sdbscan_gb300 import capi
    n, d = 600, 12
    X = _clusters(n, d, 12, 0.25, 5, "mixed")

    def fit(eps, cap=0):
        e = capi.Engine(n, d)
        e.set_params(n_proj=256, topK=3, topM=50, random_seed=4)
        e.set_debug_limits(device_bytes_cap=cap)
        try:
            e.fit_soptics(X, eps, 2)
            return e.optics() + (int(e.core()[1].sum()),)
        finally:
            e.close()

    def smallest_cap(eps):
        lo, hi = 1 << 16, 1 << 28
        while hi - lo > 1 << 12:
            mid = (lo + hi) // 2
            try:
                fit(eps, mid)
                hi = mid
            except capi.SdbError as err:
                assert err.status == 6
                lo = mid
        return hi

    eps = 0.05
    order, reach, entries = fit(eps)
    assert 5000 < entries and 8 * entries < 4 * n * 6 * 50  # the copy is smaller than the distances
    cap = smallest_cap(eps)
    assert cap - smallest_cap(1e-9) < 12 * entries
    got = fit(eps, cap)
    np.testing.assert_array_equal(got[0], order)
    np.testing.assert_array_equal(got[1], reach)


@pytest.mark.parametrize("fit", ["soptics", "sngoptics"])
def test_n_threads_bounds_the_orderings_host_threads(fit):
    """n_threads = 1 runs the floods on the calling thread alone; the result is
    the same with any number."""
    import os
    import threading

    from sdbscan_gb300 import capi
    n, d = 20000, 16
    X = _clusters(n, d, 12, 0.35, 3, "mixed")

    def run(n_threads):
        e = capi.Engine(n, d)
        e.set_params(n_proj=256, topK=8, topM=60, random_seed=4, n_threads=n_threads)
        if fit == "sngoptics":
            e.set_sng_params(samplingProb=0.03, random_seed=4, n_threads=n_threads)
        call = e.fit_soptics if fit == "soptics" else e.fit_sngoptics
        call(X, 0.06, 10)  # whatever the CUDA runtime starts is there now
        stop = threading.Event()
        seen = []

        def watch():
            while not stop.is_set():
                seen.append(len(os.listdir("/proc/self/task")))

        w = threading.Thread(target=watch)
        w.start()
        while not seen:
            pass
        before = seen[0]
        for _ in range(5):
            call(X, 0.06, 10)
        stop.set()
        w.join()
        out = e.optics()
        entries = int(e.core()[1].sum())
        e.close()
        return out, max(seen) - before, entries

    one, extra, entries = run(1)
    assert entries > 400000  # enough for helpers
    assert extra == 0
    for threads in (3, -1):
        got, _, _ = run(threads)
        np.testing.assert_array_equal(got[0], one[0])
        np.testing.assert_array_equal(got[1], one[1])
