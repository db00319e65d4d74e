"""The packed FP32 distance tile (csrc/pair_tile.cuh, k_dist_pair.cu) against
the scalar tile (sdb_set_tile_variant 1): same sums in the same order, so
every output is equal, at the edges of its shapes -- columns per tile 32, 40,
50 and 64 and m across them, lists of a few members and of several row tiles,
dimensions that end mid-stage and mid-chunk, Chi2 entries in and out of the
packed quotient's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(dist, n, d, seed):
    rng = np.random.default_rng(seed)
    c = rng.standard_normal((6, d))
    X = (c[rng.integers(0, 6, n)] + 0.4 * rng.standard_normal((n, d))).astype(np.float32)
    return np.abs(X) if dist == "Chi2" else X


def _eps(dist, d):
    return {"Cosine": 0.2, "L1": 0.5 * d, "L2": 0.7 * d ** 0.5, "Chi2": 0.1}[dist]


def _outputs(X, dist, variant, optics, limits=None, **kw):
    from sdbscan_gb300 import capi
    e = capi.Engine(*X.shape)
    if dist != "Cosine":
        kw = dict(kw, ker_n_features=max(64, X.shape[1] + X.shape[1] % 2), ker_sigma=float(X.shape[1]))
    e.set_params(distance=dist, random_seed=5, **kw)
    e.set_tile_variant(variant)
    if limits:
        e.set_debug_limits(**limits)
    eps = _eps(dist, X.shape[1])
    if optics:
        e.fit_soptics(X, eps, 6)
        out = list(e.core()) + list(e.optics()) + [e.core_dist()]
    else:
        e.fit_sdbscan(X, eps, 6)
        out = list(e.core()) + [e.labels()[0]]
    pairs = e.counters()["pairs"]
    lab, ncl = e.fit_sdbscan_sweep(X, [0.5 * eps, eps, 0.75 * eps], 6)
    e.close()
    return out + [lab, ncl, np.array(pairs)]


@pytest.mark.parametrize("dist", ["Cosine", "L1", "L2", "Chi2"])
@pytest.mark.parametrize("m,n,d,optics", [
    (1, 300, 17, False), (31, 900, 64, False), (32, 5000, 33, True), (33, 2000, 4, False), (40, 9000, 100, False),
    (41, 700, 129, True), (50, 6000, 95, False), (51, 1500, 32, False), (64, 4000, 66, True), (65, 1000, 31, False),
    (100, 3000, 160, False), (130, 2500, 20, True)])
def test_packed_tile_equals_scalar_tile(dist, m, n, d, optics):
    X = _data(dist, n, d, 1000 * m + n)
    kw = dict(n_proj=64, topK=3, topM=m)
    want = _outputs(X, dist, 1, optics, **kw)
    got = _outputs(X, dist, 3, optics, **kw)
    assert want[0].any() and want[-1] > 0
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,d,zeroed", [(3000, 40, 1.0), (3000, 40, 0.5), (2000, 130, 0.0)])
def test_packed_chi2_tile_with_tiny_entries(n, d, zeroed):
    """Histograms with entries down to 1e-38, whose products leave the packed
    quotient's range: their tiles take the general term; rows whose tiny
    entries are zero take the packed one (a share `zeroed` of them)."""
    rng = np.random.default_rng(int(10 * zeroed) + d)
    protos = rng.dirichlet(np.full(d, 0.1), 8)
    X = rng.standard_gamma(200 * protos[rng.integers(0, 8, n)] + 0.01)
    X /= X.sum(1, keepdims=True)
    mask = (rng.random(n) < zeroed)[:, None] & (X < 1e-9)
    X = np.where(mask, 0.0, X).astype(np.float32)
    X[X < 1e-38] = 0.0
    assert zeroed == 1.0 or (X[X > 0].min() < 1e-30)
    kw = dict(n_proj=64, topK=3, topM=50)
    for optics in (False, True):
        want = _outputs(X, "Chi2", 1, optics, **kw)
        assert want[0].any()
        for a, b in zip(_outputs(X, "Chi2", 3, optics, **kw), want):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("exponents", [(0, 0), (-50, 0), (-50, -50), (-3, -30)])
def test_packed_chi2_quotient_is_correctly_rounded(exponents):
    """Distances of two-bin histograms through both tiles: 5e7 quotients with
    significands over the whole range and entries from 2^-50 to 1."""
    from sdbscan_gb300 import capi
    rng = np.random.default_rng(sum(exponents) & 0xFF)
    n, d = 2000, 64
    lo, hi = min(exponents), max(exponents)
    X = np.exp2(rng.uniform(lo, hi + 1e-3, (n, d))).astype(np.float32)
    X[:, 0] += 1.0
    out = []
    for variant in (1, 3):
        e = capi.Engine(n, d)
        e.set_params(distance="Chi2", n_proj=64, topK=4, topM=50, ker_n_features=64, random_seed=3)
        e.set_tile_variant(variant)
        e.fit_soptics(X, 2.0, 3)
        out.append((e.core_dist(), *e.optics(), e.core()[1]))
        e.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_a_fit_that_cannot_hold_the_candidate_copy_runs_without_it():
    """The smallest memory cap under which the scalar tile fits also runs the
    packed one: same results, no error."""
    from sdbscan_gb300 import capi
    X = _data("Cosine", 400, 48, 3)
    kw = dict(n_proj=256, topK=3, topM=50)
    want = _outputs(X, "Cosine", 1, False, **kw)
    lo, hi = 1 << 16, 1 << 28
    while hi - lo > 1 << 14:
        mid = (lo + hi) // 2
        try:
            _outputs(X, "Cosine", 1, False, dict(device_bytes_cap=mid), **kw)
            hi = mid
        except capi.SdbError as e:
            assert e.status == 6
            lo = mid
    for a, b in zip(_outputs(X, "Cosine", 3, False, dict(device_bytes_cap=hi), **kw), want):
        np.testing.assert_array_equal(a, b)
