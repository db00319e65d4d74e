"""The projection kernel (csrc/k_project.cu) against the oracle, bit for bit:
each vector length it has a form for (512, 1024 and 2048 in two layouts, shorter
ones by shuffles), rows that end mid-chunk, entries in and out of the range of
its row quotient (zeros of both signs, 1e-25 to 1e15), and rows whose
projections are all equal in size, where the top-k has more candidates than
lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows_as_sets(a):
    return np.sort(np.asarray(a), axis=1)


def _data(n, d, kind, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, d)).astype(np.float32)
    if kind == "range":
        X *= np.exp2(rng.uniform(-83, 50, (n, d))).astype(np.float32)  # 1e-25 .. 1e15
        X[rng.random((n, d)) < 0.2] = 0.0
        X[rng.random((n, d)) < 0.1] = -0.0
        X[:, 0] = rng.standard_normal(n)
    elif kind == "ties":  # one entry: every projection is +-c
        X[:] = 0.0
        X[np.arange(n), rng.integers(0, d, n)] = rng.standard_normal(n).astype(np.float32)
        X[: n // 2] = rng.standard_normal((n // 2, d))
    return X


@pytest.mark.parametrize("n,d,nproj,k,m,kind", [
    (700, 300, 512, 7, 20, "range"), (300, 333, 512, 31, 9, "plain"), (500, 40, 300, 10, 30, "ties"),   # 512
    (600, 784, 1024, 10, 50, "range"), (400, 31, 1024, 5, 50, "plain"), (300, 1021, 600, 20, 8, "ties"),  # 1024
    (300, 1500, 2048, 31, 12, "range"), (200, 2047, 16, 8, 4, "plain"), (200, 60, 1500, 12, 10, "ties"),  # 2048
    (500, 17, 64, 6, 15, "range"), (300, 200, 20, 10, 9, "ties"), (40, 9, 9, 9, 5, "plain"),              # short
])
def test_projections_and_selections_match_oracle(n, d, nproj, k, m, kind):
    from oracle.oracle import Port, build_port, fht_dim
    from sdbscan_gb300 import capi
    build_port()
    port = Port()
    X = _data(n, d, kind, n + d)
    e = capi.Engine(n, d)
    e.set_params(n_proj=nproj, topK=k, topM=m, random_seed=21)
    e.fit_sdbscan(X, 0.3, 5)
    got_P, got_K, got_M = e.projections(), e.topk(), e.topm()
    e.close()
    fd = fht_dim(nproj, d)
    Xt, rc = port.transform(X, "Cosine")
    assert rc == 0
    P = port.project(Xt, "Cosine", d, 0.4, None, port.hd3_bits(3 * fd, 21), fd, nproj)
    np.testing.assert_array_equal(got_P, P)
    np.testing.assert_array_equal(_rows_as_sets(got_K[:, :k]), _rows_as_sets(port.topk_canon(P, k)[:, :k]))
    np.testing.assert_array_equal(_rows_as_sets(got_K[:, k:]), _rows_as_sets(port.topk_canon(P, k)[:, k:]))
    np.testing.assert_array_equal(_rows_as_sets(got_M[:, :m]), _rows_as_sets(port.topm_canon(P, m)[:, :m]))
    np.testing.assert_array_equal(_rows_as_sets(got_M[:, m:]), _rows_as_sets(port.topm_canon(P, m)[:, m:]))
