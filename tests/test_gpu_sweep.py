"""Eps sweeps whose clusters merge step by step: every eps of a sweep against
its own fit.  A sweep carries the union-find from one eps to the next and looks
at new edges only, so a link that a round loses shows as a split cluster at
some later eps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chains(n, d, arcs, seed):
    """Points along great-circle arcs with gaps of all sizes."""
    rng = np.random.default_rng(seed)
    q = np.linalg.qr(rng.standard_normal((arcs, d, 2)))[0]
    y = rng.integers(0, arcs, n)
    t = np.empty(n)
    for a in range(arcs):
        at = np.flatnonzero(y == a)
        t[at] = rng.permutation(np.cumsum(rng.pareto(1.1, len(at)) + 0.2))
        t[at] *= 1.5 / t[at].max()
    X = np.cos(t)[:, None] * q[y, :, 0] + np.sin(t)[:, None] * q[y, :, 1]
    return (X + 0.002 * rng.standard_normal((n, d))).astype(np.float32)


@pytest.mark.parametrize("n,d,arcs,n_eps,seed", [
    (2000, 12, 8, 16, 1), (9000, 10, 20, 16, 2), (30000, 16, 40, 16, 3), (90000, 12, 60, 16, 4),
    (30000, 16, 40, 20, 5),   # more values than rounds kept per pair
    (110000, 12, 60, 8, 6),   # paths compressed between the hooking rounds
])
def test_every_eps_of_a_sweep_equals_its_own_fit(n, d, arcs, n_eps, seed):
    from sdbscan_gb300 import capi
    X = _chains(n, d, arcs, seed)
    eps = np.geomspace(2e-5, 2e-2, n_eps).astype(np.float32)
    e = capi.Engine(n, d)
    e.set_params(n_proj=512, topK=6, topM=50, random_seed=seed)
    want, counts = [], []
    for v in eps:
        e.fit_sdbscan(X, float(v), 6)
        lab, c = e.labels()
        want.append(lab)
        counts.append(c)
    assert len(set(counts)) > n_eps // 2, counts  # clusters appear and merge all along
    for order in (np.arange(n_eps), np.random.default_rng(seed).permutation(n_eps)):
        for _ in range(3):
            labels, ncl = e.fit_sdbscan_sweep(X, eps[order], 6)
            for i, o in enumerate(order):
                assert ncl[i] == counts[o]
                np.testing.assert_array_equal(labels[i], want[o])
    e.close()
