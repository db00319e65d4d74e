"""The calls this package is timed on: fits of the clustering engine through its public entry points.

A case is one call that a user's program makes, with its sizes and options.
`law` names the seeded synthetic data (the repository's benchmark laws):

  unit    unit-norm von-Mises-Fisher-like clusters, 5 % uniform noise (Cosine)
  pixels  nonnegative sparse images around 10 prototypes, 784 pixels at full size (Cosine)
  gauss   50 anisotropic Gaussians, scaled so that eps sits near the 30-NN distance (L1 / L2)
  hist    Dirichlet histograms around 30 prototypes (Chi2 / JS)

and `call` the entry point: fit (fit_sDbscan), optics (fit_sOptics), module
(fit_sDbscan of the drop-in Python module, host data), sweep (test_sDbscan:
eight eps values), batch (many small sets, eight eps values each, one CUDA
graph), sng (fit_sngDbscan) and sngoptics (fit_sngOptics).
"""
import math

import numpy as np
import torch

from sdbscan_gb300 import capi
from sdbscan_gb300.datasets import cfg2_mnist_like_torch, vmf_mixture_torch

SEED = 42  # of the engine's random vectors and samples
SWEEP_EPS = (0.05, 0.10, 0.15, 0.20, 0.25, 0.30, 0.35, 0.40)


def case(name, call, law, n, d, **more):
    c = dict(name=name, call=call, law=law, n=n, d=d, distance="Cosine", n_proj=1024, topK=5, topM=50, eps=0.15,
             minPts=20, bf16=False, noise=0, prob=0.01)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a few thousand low-dimensional embeddings; latency and launches
        case("unit_2k_x64", "fit", "unit", 2000, 64),
        # an ordinary fit of an embedding table (the first benchmark configuration)
        case("unit_50k_x128", "fit", "unit", 50_000, 128),
        # odd n, d, k, m and a smaller index, noise points labelled by their nearest core (sDbscan-1NN)
        case("pixels_33k_x333_noise", "fit", "pixels", 33_333, 333, n_proj=512, topK=7, topM=37, eps=0.25, minPts=30,
             noise=1),
        # MNIST's shape through the drop-in module, from the host memory that its users hold
        case("pixels_70k_x784_module", "module", "pixels", 70_000, 784, topK=10, eps=0.25, minPts=50),
        # the headline: a million images, plain FP32 and with tensor-core screening
        case("pixels_1m_x784", "fit", "pixels", 1_000_000, 784, topK=10, eps=0.25, minPts=50),
        case("pixels_1m_x784_bf16", "fit", "pixels", 1_000_000, 784, topK=10, eps=0.25, minPts=50, bf16=True),
        # Euclidean distance through random Fourier features, m = 100
        case("gauss_150k_x256_l2", "fit", "gauss", 150_000, 256, distance="L2", topK=10, topM=100, eps=0.3, minPts=30),
        # histograms under the chi-squared kernel: ordering and reachability
        case("hist_60k_x512_chi2_optics", "optics", "hist", 60_000, 512, distance="Chi2", topK=10, eps=0.17,
             minPts=50),
        # choosing eps: one index, eight clusterings, from host memory
        case("unit_40k_x256_sweep", "sweep", "unit", 40_000, 256),
        # many small sets at once, replayed as one graph
        case("unit_batch_8", "batch", "unit", 20_000, 128, sets=8),
        # the sampled baseline with a fixed seed, and its OPTICS form
        case("pixels_200k_x784_sng", "sng", "pixels", 200_000, 784, eps=0.25, minPts=50),
        case("pixels_50k_x784_sngoptics", "sngoptics", "pixels", 50_000, 784, eps=0.25, minPts=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["fit", "fit", "fit", "module", "optics", "sweep", "batch", "sng", "sngoptics"])
    index = dict(n_proj=rng.choice([256, 512, 1024, 1024]), topK=rng.choice([5, 7, 10]), topM=rng.randint(20, 100))
    if call == "fit":
        law = rng.choice(["unit", "pixels", "pixels", "gauss", "hist"])
    elif call == "optics":
        law = rng.choice(["unit", "gauss", "hist"])
    else:
        law = rng.choice(["unit", "pixels"])
    d = _log(rng, 32, 784) if law != "pixels" else rng.randint(200, 784)
    more = dict(minPts=rng.randint(10, 50), bf16=rng.random() < 0.3)
    if call in ("fit", "module"):
        more["noise"] = rng.choice([0, 0, 0, 1])
    more["distance"] = {"gauss": ["L2", "L2", "L1"], "hist": ["Chi2", "JS"]}.get(law, ["Cosine"])
    more["distance"] = rng.choice(more["distance"])
    n = _log(rng, 2000, {"gauss": 150_000, "hist": 40_000}.get(law, 500_000))
    if call in ("optics", "module", "sweep", "batch"):
        n = min(n, _log(rng, 2000, 70_000))
    if law == "gauss":
        if more["distance"] == "L1":
            n, index["topM"] = min(n, 50_000), min(index["topM"], 50)
            more["eps"] = round(0.2368 * math.sqrt(d), 4)
        else:
            more["eps"] = 0.3
    elif law == "hist":
        more["eps"] = 0.17 if more["distance"] == "Chi2" else 0.25
        if more["distance"] == "JS":
            n, index["topM"] = min(n, 20_000), min(index["topM"], 50)
    else:
        more["eps"] = 0.15 if law == "unit" else 0.25
    if call == "batch":
        more["sets"] = rng.randint(2, 8)
        more["noise"] = 0
        n = min(n, 20_000)
    if call in ("sng", "sngoptics"):
        # the work grows with n^2 prob
        n = min(n, 100_000 if call == "sng" else 50_000)
        more["prob"] = rng.choice([0.005, 0.01]) if n > 20_000 else rng.choice([0.01, 0.05])
        if call == "sngoptics":
            more["minPts"] = rng.randint(4, 10)
        if call == "sng" and n <= 20_000 and rng.random() < 0.25:
            more["prob"] = 1.0  # exact DBSCAN
    c = case("", call, law, n, d, **index, **more)
    del c["name"]
    return c


# ---- data -----------------------------------------------------------------------

def _gauss(n, d, seed, comps=50):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    centres = 5.0 * rnd(comps, d)
    q, _ = torch.linalg.qr(rnd(comps, d, d))
    ev = 0.1 + 1.9 * torch.rand(comps, 1, d, generator=g, device="cuda")
    factors = q * ev.sqrt()  # covariance Q diag(ev) Q^T
    per = torch.randint(0, comps, (n,), generator=g, device="cuda")
    z = rnd(n, d)
    X = torch.empty(n, d, device="cuda")
    for c in range(comps):
        rows = (per == c).nonzero()[:, 0]
        X[rows] = z[rows] @ factors[c].T + centres[c]
    # 0.3 / 20.23 at d = 256, the median 30-NN distance of the unscaled law
    return X * (0.0148 * 16.0 / math.sqrt(d))


def _hist(n, d, seed, comps=30, alpha=0.1, conc=200.0):
    torch.manual_seed(seed)
    protos = torch.distributions.Dirichlet(torch.full((d,), alpha, device="cuda")).sample((comps,))
    y = torch.randint(0, comps, (n,), device="cuda")
    X = torch.distributions.Gamma(conc * protos[y] + alpha / 10.0, torch.ones((), device="cuda")).sample()
    X /= X.sum(1, keepdim=True)
    X[X < 1e-9] = 0.0
    return X / X.sum(1, keepdim=True)


def _data(law, n, d, seed):
    if law == "unit":
        return vmf_mixture_torch(n, d, 20, 0.15 / math.sqrt(d), 0.05, seed)[0]
    if law == "pixels":
        return cfg2_mnist_like_torch(n, d, seed=seed)[0]
    return (_gauss if law == "gauss" else _hist)(n, d, seed).contiguous()


def _median_distance(X):
    s = X[:2000]
    dd = torch.cdist(s.double(), s.double())
    i = torch.triu_indices(len(s), len(s), 1, device=X.device)
    return round(float(dd[i[0], i[1]].median()), 3)


def _sizes(c):
    """Points and dimensions of a batch's sets: uneven, as a sweep over many small datasets has them."""
    return [(max(2000, int(c["n"] * (i + 1) / c["sets"])), (64, c["d"], 256)[i % 3]) for i in range(c["sets"])]


def prepare(case, seed):
    c = dict(case)
    params = dict(n_proj=c["n_proj"], topK=c["topK"], topM=c["topM"], distance=c["distance"],
                  clusterNoise=c["noise"], samplingProb=c["prob"], random_seed=SEED)
    s = {"case": c}
    if c["call"] == "batch":
        s["X"] = [_data(c["law"], n, d, seed * 100 + i) for i, (n, d) in enumerate(_sizes(c))]
        torch.cuda.synchronize()
        del params["samplingProb"]
        s["batch"] = capi.Batch([(X.data_ptr(), *X.shape) for X in s["X"]], SWEEP_EPS, c["minPts"],
                                precision=int(c["bf16"]), **params)
        return s
    X = _data(c["law"], c["n"], c["d"], seed)
    if c["distance"] in ("L1", "L2"):
        params["ker_sigma"] = _median_distance(X)
    if c["call"] == "module":
        from sdbscan_gb300 import sDbscan
        s["X"] = X.cpu().numpy().T  # (d, n), column-major: the module's layout
        s["dbs"] = sDbscan.sDbscan(c["n"], c["d"])
        s["dbs"].set_params(**params)
        s["dbs"].set_precision(int(c["bf16"]))
        return s
    e = s["engine"] = capi.Engine(c["n"], c["d"])
    if c["call"] in ("sng", "sngoptics"):
        e.set_sng_params(distance=c["distance"], samplingProb=c["prob"], random_seed=SEED)
        e.set_precision(int(c["bf16"]))
    else:
        e.set_params(precision=int(c["bf16"]), **params)
    s["X"] = X.cpu().numpy() if c["call"] == "sweep" else X
    torch.cuda.synchronize()  # the engine has its own stream
    return s


def run(state):
    c = state["case"]
    call = c["call"]
    if call == "batch":
        b = state["batch"]
        b.run()
        out = []
        for i in range(b.ns):
            got = [b.labels(i, j) for j in range(len(SWEEP_EPS))]
            out.append({"labels": np.stack([g[0] for g in got]), "clusters": np.array([g[1] for g in got])})
        return out
    if call == "module":
        dbs = state["dbs"]
        dbs.fit_sDbscan(state["X"], c["eps"], c["minPts"])
        return {"labels": np.asarray(dbs.labels_, dtype=np.int32), "clusters": int(dbs.n_clusters_)}
    e, X = state["engine"], state["X"]
    if call == "sweep":
        labels, clusters = e.fit_sdbscan_sweep(X, SWEEP_EPS, c["minPts"])
        return {"labels": labels, "clusters": clusters}
    fit = {"fit": e.fit_sdbscan_device, "optics": e.fit_soptics_device, "sng": e.fit_sngdbscan_device,
           "sngoptics": e.fit_sngoptics_device}[call]
    fit(X.data_ptr(), c["eps"], c["minPts"])
    core, degree = e.core()
    out = {"core": core, "degree": degree}
    if call in ("optics", "sngoptics"):
        out["ordering"], out["reach"] = e.optics()
        out["core_dist"] = e.core_dist()
    else:
        out["labels"], out["clusters"] = e.labels()
    return out


def work(case):
    c = case
    term = {"Cosine": 2, "L1": 3, "L2": 3, "Chi2": 4, "JS": 12}[c["distance"]]  # operations per dimension of a distance

    def index(n, d):
        f = 1 << math.ceil(math.log2(max(c["n_proj"], d if c["distance"] == "Cosine" else 1024)))
        flops = 3.0 * f * math.log2(f) * n + term * 2.0 * c["topK"] * c["topM"] * d * n
        return flops + (2.0 * 512 * d * n if c["distance"] in ("L1", "L2") else 0.0)

    if c["call"] == "batch":
        sizes = _sizes(c)
        return {"bytes": float(sum(4 * n * d + 4 * n * len(SWEEP_EPS) for n, d in sizes)),
                "flops": float(sum(index(n, d) for n, d in sizes))}
    n, d = c["n"], c["d"]
    out = {"sweep": 4 * len(SWEEP_EPS), "optics": 17, "sngoptics": 17, "module": 4}.get(c["call"], 9)
    if c["call"] in ("sng", "sngoptics"):
        # every point against its draws; the exact form needs each pair once
        flops = term * (0.5 if c["prob"] >= 1 else c["prob"]) * float(n) * n * d
    else:
        flops = index(n, d)
    return {"bytes": float(4 * n * d + out * n), "flops": float(flops)}


# ---- 64-bit values ----------------------------------------------------------------

def _splitmix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def exact(case, seed):
    """Core distances of a Cosine sngOptics fit: the (minPts - 1)-th smallest of a point's distinct sampled
    neighbours within eps.  Labels, flags, orderings are whole numbers; reachability follows the ordering's
    ties; the other fits' distances depend on which candidates the FP32 index finds."""
    c = case
    if c["call"] != "sngoptics" or c["distance"] != "Cosine":
        return None
    n, S = c["n"], int(math.ceil(np.float32(c["prob"]) * np.float32(c["n"])))
    X = _data(c["law"], n, c["d"], seed).double()
    X /= X.norm(dim=1, keepdim=True)
    with np.errstate(over="ignore"):
        key = _splitmix64(np.array([SEED], np.uint64))[0]
        keys, dists = [], []
        for b in range((n + 31) // 32):
            z = _splitmix64(key + np.arange(b * S, (b + 1) * S, dtype=np.uint64))
            q = torch.from_numpy((((z >> np.uint64(32)) * np.uint64(n)) >> np.uint64(32)).astype(np.int64)).cuda()
            p = torch.arange(32 * b, min(n, 32 * b + 32), device="cuda")
            dd = 1.0 - X[q] @ X[p].T
            i, j = ((dd <= c["eps"]) & (q[:, None] != p[None, :])).nonzero(as_tuple=True)
            keys += [q[i] * n + p[j], p[j] * n + q[i]]
            dists += [dd[i, j]] * 2
    key, inverse = torch.unique(torch.cat(keys), return_inverse=True)
    dist = torch.zeros(len(key), dtype=torch.float64, device="cuda")
    dist[inverse] = torch.cat(dists)
    order = dist.sort(stable=True).indices
    order = order[(key[order] // n).sort(stable=True).indices]  # by point, then by distance
    count = torch.bincount(key // n, minlength=n)
    first = count.cumsum(0) - count
    core = count >= c["minPts"] - 1
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    out[core] = dist[order[first[core] + c["minPts"] - 2]]
    return {"core": None, "degree": None, "ordering": None, "reach": None, "core_dist": out.cpu().numpy()}
