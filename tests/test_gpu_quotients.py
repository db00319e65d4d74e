"""The quotients that replace the compiled division (csrc/quotients.cuh) equal
it bit for bit over their ranges (quotients_check.cu), and the JS fits built on
them equal the same fits with the compiled division."""
import ctypes
import heapq
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from sdbscan_gb300 import _build
    so = str(tmp_path_factory.mktemp("quotients") / "libquotients_check.so")
    subprocess.run([_build._nvcc(), *_build.ARCH, *_build.NVCC_FLAGS, f"-I{_build.CSRC}", "-shared",
                    os.path.join(HERE, "quotients_check.cu"), "-o", so, "-lcudart"], check=True)
    L = ctypes.CDLL(so)
    for f in ("check_row", "check_js", "check_log2", "check_chi2", "check_js_terms"):
        getattr(L, f).restype = ctypes.c_longlong
    return L


# divisor and numerator exponents: both ends of the fast range, its middle, just outside
@pytest.mark.parametrize("ec,ex", [(0, 0), (0, -1), (-60, -60), (-60, 59), (59, -60), (59, 59), (-61, 0), (60, 0),
                                   (0, 60), (0, -61), (7, -20)])
def test_row_quotient(lib, ec, ex):
    assert lib.check_row(64, ec, ex) == 0


@pytest.mark.parametrize("e", range(-20, 1))
def test_js_quotient(lib, e):
    assert lib.check_js(32, e) == 0


def test_js_logarithm_over_log_2(lib):
    assert lib.check_log2() == 0


@pytest.mark.parametrize("ex,ey", [(-50, -50), (-50, 0), (-50, -1), (-1, -50), (-25, -26), (-1, -1), (-1, -2), (-3, -30)])
def test_chi2_terms(lib, ex, ey):
    assert lib.check_chi2(64, ex, ey) == 0


def test_js_terms(lib):
    assert lib.check_js_terms(64) == 0  # 2.7e8 pairs


def _histograms(n, d, seed):
    rng = np.random.default_rng(seed)
    protos = rng.dirichlet(np.full(d, 0.3), 8)
    X = rng.standard_gamma(60 * protos[rng.integers(0, 8, n)] + 0.02)
    X[X < 0.01] = 0.0
    X[:, 0] += 0.05
    return X.astype(np.float32)


def _floods(core, near, weight):
    """The sOPTICS ordering: outer loop by id, seeds by (reachability, id)."""
    n = len(core)
    reach = np.full(n, np.float32(-2147483648.0))
    done = np.zeros(n, bool)
    order = []
    for p in range(n):
        if done[p]:
            continue
        heap = [(np.float32(0), p)]
        while heap:
            r, x = heapq.heappop(heap)
            if done[x] or (x != p and r != reach[x]):
                continue
            done[x] = True
            order.append(x)
            if not core[x]:
                continue
            for y, w in zip(near[x], weight[x]):
                if not done[y] and (reach[y] == np.float32(-2147483648.0) or w < reach[y]):
                    reach[y] = w
                    heapq.heappush(heap, (w, y))
    return np.array(order), reach


@pytest.mark.parametrize("n,d,m,eps,minPts", [(700, 24, 40, 0.12, 8), (900, 65, 70, 0.16, 12)])
def test_js_soptics_equals_the_compiled_division(lib, n, d, m, eps, minPts):
    """A JS fit through the index: neighbourhood sizes, core distances, ordering
    and reachability from its own candidates and distances computed with the
    compiled division.  (The tile takes whole stages of 32 dimensions, and JS's
    1e-6 gives a row's zero padding terms of its own, 1e-6 of distance each; the
    sums here take the same padding.)"""
    import torch

    from sdbscan_gb300 import capi
    X = _histograms(n, d, n)
    k, D = 4, 64
    e = capi.Engine(n, d)
    e.set_params(distance="JS", n_proj=D, topK=k, topM=m, ker_n_features=512, random_seed=3)
    e.fit_soptics(X, eps, minPts)
    tK, tM = e.topk(), e.topm().reshape(D, 2, m)
    ordering, reach = e.optics()
    core, degree = e.core()
    core_dist = e.core_dist()
    e.close()
    Xt = X / np.add.accumulate(X, axis=1, dtype=np.float32)[:, -1:]  # sequential sums, as the engine's
    dp = (d + 31) // 32 * 32
    dev = torch.from_numpy(np.pad(Xt, ((0, 0), (0, dp - d)))).cuda()
    out = torch.empty(n, n, device="cuda")
    torch.cuda.synchronize()
    assert lib.js_distances(ctypes.c_void_p(dev.data_ptr()), n, dp, ctypes.c_void_p(out.data_ptr())) == 0
    dist = out.cpu().numpy()
    pair = np.zeros((n, n), bool)
    for p in range(n):
        cand = np.concatenate([tM[tK[p], 0 if j < k else 1][j] for j in range(2 * k)])
        pair[p, cand] = dist[p, cand] <= np.float32(eps)
    np.fill_diagonal(pair, False)
    np.testing.assert_array_equal(dist, dist.T)  # (a term's two summands commute)
    pair |= pair.T
    np.testing.assert_array_equal(degree, pair.sum(1))
    is_core = pair.sum(1) >= minPts - 1
    np.testing.assert_array_equal(core.astype(bool), is_core)
    assert is_core.mean() > 0.1
    want = np.zeros(n, np.float32)
    near = [np.flatnonzero(r) for r in pair]
    for p in np.flatnonzero(is_core):
        want[p] = np.sort(dist[p, near[p]])[minPts - 2]
    np.testing.assert_array_equal(core_dist, want)
    weight = [np.maximum(want[p], dist[p, near[p]]) for p in range(n)]
    o, r = _floods(is_core, near, weight)
    np.testing.assert_array_equal(ordering, o)
    np.testing.assert_array_equal(reach, r)


@pytest.mark.parametrize("zeroed", [1.0, 0.5, 0.0])
def test_packed_sngoptics_with_tiny_chi2_entries(port, zeroed):
    """Per-block sngOptics on histograms with entries down to 1e-38 against the
    oracle: tiles with an entry below 2^-50 take the general term, the others
    (a share `zeroed` of the rows has its tiny entries at zero) the packed one."""
    from sdbscan_gb300 import capi
    rng = np.random.default_rng(int(10 * zeroed))
    n, d = 1500, 40
    protos = rng.dirichlet(np.full(d, 0.1), 8)
    X = rng.standard_gamma(200 * protos[rng.integers(0, 8, n)] + 0.01)
    X /= X.sum(1, keepdims=True)
    X = np.where((rng.random(n) < zeroed)[:, None] & (X < 1e-9), 0.0, X).astype(np.float32)
    X[X < 1e-38] = 0.0
    assert zeroed == 1.0 or X[X > 0].min() < 1e-30
    e = capi.Engine(n, d)
    e.set_sng_params(distance="Chi2", samplingProb=0.3, random_seed=7)
    e.set_sng_sampling(2)
    e.fit_sngoptics(X, 0.1, 6)
    got = (*e.optics(), e.core()[0], e.core_dist(), e.core()[1])
    e.close()
    want = port.fit_sngoptics_blocks(X, 0.1, 6, dist="Chi2", samplingProb=0.3, seed=7, threads=4)
    assert want[2].any()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
