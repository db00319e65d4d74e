"""Neighbourhood sizes, core flags and labels of a fit's own candidates against
the oracle's lean construction, where k_core_dedupe and the cluster kernels
branch: more points of two or more lists than its seen bits hold at once
(several passes), hubs of few and of many lists, one or several mask words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,nproj,k,m,eps,minPts", [
    (100000, 16, 2048, 2, 100, 0.05, 12),  # 409600 slots: over 32768 points of two lists, several passes
    (40000, 16, 1024, 3, 100, 0.05, 12),
    (90000, 8, 2048, 2, 50, 0.02, 8),
    (500, 12, 256, 4, 60, 0.3, 10),        # every point in some 60 lists
    (30000, 20, 64, 5, 7, 0.1, 4),         # few hubs
    (7, 9, 16, 1, 3, 0.5, 2),
    (3000, 10, 128, 31, 20, 0.2, 40),
])
def test_core_stage_matches_oracle(n, d, nproj, k, m, eps, minPts):
    from oracle.oracle import Port, build_port
    from sdbscan_gb300 import capi
    build_port()
    rng = np.random.default_rng(n + m)
    c = rng.standard_normal((12, d))
    X = (c[rng.integers(0, 12, n)] + 0.25 * rng.standard_normal((n, d))).astype(np.float32)
    e = capi.Engine(n, d)
    e.set_params(n_proj=nproj, topK=k, topM=m, random_seed=9)
    e.fit_sdbscan(X, eps, minPts)
    labels, ncl = e.labels()
    core, deg = e.core()
    tK, tM = e.topk(), e.topm()
    e.close()
    if n == 100000:  # the passes are taken: more than 32768 points in two lists
        held = np.bincount(tM.ravel(), minlength=n)
        assert (held >= 2).sum() > 32768
    port = Port()
    Xt, rc = port.transform(X, "Cosine")
    assert rc == 0
    ocore, odeg, olabels, oncl = port.core_cluster_lean(Xt, "Cosine", tK, tM, eps, minPts)
    np.testing.assert_array_equal(deg, odeg)
    np.testing.assert_array_equal(core, ocore)
    np.testing.assert_array_equal(labels, olabels)
    assert ncl == oncl
