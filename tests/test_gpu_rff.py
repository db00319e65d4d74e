"""The random-Fourier embedding on the packed tile (csrc/k_rff.cu): points
around a row tile of 128, rows of R around a column tile of 64 (fewer, odd, one
over), dimensions around a stage of 32.  The projections agree with the
oracle's to 1e-5 of the row norm: both sum each product chain in the same
order, so they differ by CUDA's cosf / sinf alone (2 ulp an embedding entry)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,ker,nproj,dist", [
    (128, 32, 128, 128, "L2"),
    (129, 33, 130, 128, "L2"),    # h = 65: one row of R in the second column tile
    (127, 3, 74, 64, "L1"),       # h = 37, one short stage
    (300, 100, 62, 64, "L1"),     # h = 31
    (1000, 261, 254, 256, "L2"),
    (50, 1, 16, 16, "L2"),
])
def test_projections_match_oracle(n, d, ker, nproj, dist):
    from oracle.oracle import Port, build_port, fht_dim
    from sdbscan_gb300 import capi
    build_port()
    port = Port()
    X = np.random.default_rng(n + d).standard_normal((n, d)).astype(np.float32)
    sigma = float(d) if dist == "L1" else float(np.sqrt(2.0 * d))
    eng = capi.Engine(n, d)
    eng.set_params(n_proj=nproj, topK=3, topM=min(20, n), distance=dist, ker_n_features=ker, ker_sigma=sigma,
                   random_seed=6)
    eng.fit_sdbscan(X, 0.5 * sigma, 5)
    P = eng.projections()
    eng.close()
    Xt, rc = port.transform(X, dist)
    assert rc == 0
    fd = fht_dim(nproj, ker)
    want = port.project(Xt, dist, ker, 0.4, port._R(dist, ker, d, sigma, 6), port.hd3_bits(3 * fd, 6), fd, nproj)
    assert np.max(np.abs(P - want) / np.linalg.norm(want, axis=1, keepdims=True)) < 1e-5
