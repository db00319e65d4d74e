"""The top-m stage on data that arrives cluster after cluster: its bounds come
from chunks of consecutive points, and where too few chunks hold a cluster's
points every list overflows and is selected from its whole column -- the same
lists, tens of times slower."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(X, reps=5):
    from sdbscan_gb300 import capi
    e = capi.Engine(*X.shape)
    e.set_params(n_proj=512, topK=5, topM=50, random_seed=3)
    ms = []
    for _ in range(reps):
        e.fit_sdbscan_device(X.data_ptr(), 0.1, 20)
        ms.append(e.stage_ms()["topm"])
    out = e.topm()
    e.close()
    return out, min(ms)


@pytest.mark.parametrize("n,clusters,runs", [(400000, 40, 1), (400000, 100, 1), (60000, 40, 1), (400000, 40, 6),
                                             (400000, 40, 2)])
def test_sorted_data_takes_no_longer_than_shuffled(n, clusters, runs):
    """`runs`: the data are that many parts, each sorted by cluster.  A stage of
    0.1 to 0.4 ms either way (1.6 to 30 ms where every list overflows)."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    d = 64
    centre = torch.randn(clusters, d, generator=g, device="cuda")
    y = torch.randint(0, clusters, (n,), generator=g, device="cuda")
    X = (centre[y] + 0.2 * torch.randn(n, d, generator=g, device="cuda")).contiguous()
    part = torch.arange(n, device="cuda") * runs // n
    order = (part * clusters + y).sort(stable=True).indices
    mixed, mixed_ms = _fit(X)
    by_cluster, sorted_ms = _fit(X[order].contiguous())
    assert sorted_ms < 3 * mixed_ms, (sorted_ms, mixed_ms)
    o = order.cpu().numpy()  # the same points in every list (a tie at its end aside)
    same = np.sort(o[by_cluster].reshape(-1, 2, 50), axis=2) == np.sort(mixed.reshape(-1, 2, 50), axis=2)
    assert same.all(axis=2).mean() > 0.999


@pytest.mark.parametrize("offset", [100.0, -3000.0])
def test_topm_noalloc_on_projections_far_from_zero(offset):
    """Values that agree in their high 16 bits: the same lists and about the
    same time as centred ones (0.3 ms; 17 times that if every list overflows)."""
    import torch

    from sdbscan_gb300 import capi
    n, nproj, m = 150000, 512, 50
    g = torch.Generator(device="cuda")
    g.manual_seed(6)
    base = torch.randn(n, nproj, generator=g, device="cuda")

    def best(P):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        stream = torch.cuda.current_stream()
        out = torch.empty(nproj, 2 * m, dtype=torch.int32, device="cuda")
        ms = []
        for _ in range(6):
            a.record()
            capi.topm_noalloc(P.data_ptr(), n, nproj, m, out.data_ptr(), stream.cuda_stream)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        return out.long(), min(ms)

    far = base + offset
    got, far_ms = best(far)
    _, centred_ms = best(base)
    assert far_ms < 3 * centred_ms, (far_ms, centred_ms)
    for side, sign in ((0, 1.0), (1, -1.0)):
        want = (sign * far).topk(m, dim=0).values.T
        mine = (sign * far).gather(0, got[:, side * m:(side + 1) * m].T).T
        assert torch.equal(mine, want)
