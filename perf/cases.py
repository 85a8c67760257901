"""Performance cases of the evidence accumulation clustering (EAC) path.

Each case is one call (or one short run of calls) that a user's program makes
through the package's public entry points: the prefix sum, the graph MST and
connected components, a K-Means fit, an ensemble, the co-association matrix,
the final clustering, the whole pipeline and the batched pipeline.  Sizes come
from the repository's benchmark workloads and profiling cases, or are generic
ones between them; inputs are synthetic with those workloads' distributions
and are made on the GPU from the seed alone.
"""
import math
import random
import zlib

import numpy as np
import torch

from masters_final_b200.EAC.batched import draw_instance_params, eac_batch, k_range_rule1
from masters_final_b200.EAC.eac import EAC, eac_pipeline, sp_sl_lifetime_csr
from masters_final_b200.cluster.KMeans import K_Means, kmeans_ensemble
from masters_final_b200.graph.connected_components import connected_comps_gpu
from masters_final_b200.graph.mst import boruvka_minho_gpu
from masters_final_b200.utils.scan import exprefixsumNumba


def listed():
    return [
        # row offsets of a small CSR from its degrees: the latency of a call
        dict(name="scan_20k", kind="scan", n=20_011, itype="int32", otype="int32"),
        # the 64 Mi-element stream of the scan benchmark
        dict(name="scan_64m", kind="scan", n=1 << 26, itype="int32", otype="int32"),
        # a mesh-sized graph (the reference's own graph fixture has 15,606
        # vertices), result read on the host
        dict(name="mst_20k", kind="mst", n=20_000, knn=16, wtype="uint8", device_result=False),
        # the graph benchmark: 16 nearest neighbours of a million 3-D points,
        # the forest kept on the device for the next stage
        dict(name="mst_1m", kind="mst", n=1_000_000, knn=16, wtype="uint8", device_result=True),
        # component labels of such a graph below a cut (a fifth of the edges:
        # one large component and thousands of small ones), read on the host
        dict(name="cc_1m", kind="cc", n=1_000_000, knn=16, keep=0.2, wtype="uint8",
             device_result=False),
        # one K-Means fit with the default label mode, a size of the
        # reference's published K-Means runs (3 iterations)
        dict(name="fit_1m_2d_k1024", kind="fit", n=1_000_000, d=2, k=1024, mode="cuda"),
        # ensemble generation, default label mode, a share of the 500,000-point
        # workload's partitions
        dict(name="ensemble_500k_16d_20p_fp32", kind="ensemble", n=500_000, d=16, P=20, kmin=350,
             kmax=711, comps=50, mode="cuda"),
        # ensemble generation on the tensor cores, a share of the
        # 2,000,000-point workload's partitions
        dict(name="ensemble_2m_8d_10p_bf16", kind="ensemble", n=2_000_000, d=8, P=10, kmin=700,
             kmax=1401, comps=200, mode="bf16"),
        # the co-association matrix of the 300,000-point profiling case
        dict(name="coassoc_300k_100p", kind="coassoc", n=300_000, d=16, P=100, kmin=210, kmax=427,
             comps=50),
        # the final clustering (MST, lifetime cut, labels) of such a matrix
        dict(name="final_300k_50p", kind="final", n=300_000, d=16, P=50, kmin=210, kmax=427,
             comps=50),
        # the whole pipeline on the reference's usual experiment size
        dict(name="eac_10k_2d_100p", kind="eac", n=10_000, d=2, P=100, kmin=50, kmax=101, comps=6,
             mode="cuda"),
        # an experiment's list of datasets in one call
        dict(name="batch_48", kind="batch", m=48, nmin=1000, nmax=50_000, P=50, mode="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("scan", "scan", "mst", "mst", "cc", "fit", "ensemble", "ensemble", "coassoc",
                       "final", "eac", "batch"))
    if kind == "scan":
        itype = rng.choice(("int32", "int32", "int64"))
        otype = "int64" if itype == "int64" else rng.choice(("int32", "int64"))
        return dict(kind=kind, n=_log_int(rng, 1000, 1 << (25 if otype == "int64" else 26)),
                    itype=itype, otype=otype)
    if kind in ("mst", "cc"):
        n = _log_int(rng, 5000, 1_000_000)
        # 32-bit weights go with graphs of up to 2^15 vertices
        wtype = rng.choice(("uint8", "uint8", "uint16") + (("int32", "float32") if n <= 1 << 15 else ()))
        case = dict(kind=kind, n=n, knn=rng.randint(10, 16), wtype=wtype,
                    device_result=rng.random() < 0.5)
        if kind == "cc":
            case["keep"] = round(rng.uniform(0.1, 1.0), 3)
        return case
    if kind == "fit":
        n = _log_int(rng, 20_000, 1_000_000)
        return dict(kind=kind, n=n, d=rng.randint(2, 16), k=_log_int(rng, 16, min(1024, n // 20)),
                    mode=rng.choice(("cuda", "bf16")))
    if kind == "ensemble":
        n = _log_int(rng, 5000, 1_000_000)
        d = rng.choice((2, 3, 4, 7, 8, 12, 16, 24, 32))
        kmin, kmax = (max(2, v) for v in k_range_rule1(n))
        # at most the work of the listed ensembles
        P = _log_int(rng, 4, 100)
        P = max(1, min(P, int(8e10 / (n * kmax * d)), int(2e7 / n)))
        return dict(kind=kind, n=n, d=d, P=P, kmin=kmin, kmax=kmax + 1, comps=rng.randint(5, 50),
                    mode=rng.choice(("cuda", "bf16")))
    if kind in ("coassoc", "final"):
        n = _log_int(rng, 5000, 300_000)
        kmin, kmax = k_range_rule1(n)
        P = _log_int(rng, 10, 100 if kind == "coassoc" else 50)
        # a few clusters per component, as the listed cases have
        return dict(kind=kind, n=n, d=rng.choice((2, 3, 4, 8, 16)), P=P, kmin=kmin, kmax=kmax + 1,
                    comps=int(kmax / rng.uniform(2.5, 6.5)))
    if kind == "eac":
        n = _log_int(rng, 1000, 40_000)
        kmin, kmax = k_range_rule1(n)
        return dict(kind=kind, n=n, d=rng.choice((2, 4, 8, 16)), P=_log_int(rng, 20, 100), kmin=kmin,
                    kmax=kmax + 1, comps=rng.randint(3, 12), mode=rng.choice(("cuda", "bf16")))
    return dict(kind=kind, m=rng.randint(8, 48), nmin=1000, nmax=_log_int(rng, 5000, 50_000),
                P=rng.randint(20, 50), mode=rng.choice(("cuda", "bf16")))


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _of_case(case):
    """A seed that depends on the case alone, for what fixes output shapes."""
    return zlib.crc32(repr(sorted((k, v) for k, v in case.items() if k != "name")).encode())


def _mixture(n, d, comps, g, center_range=20.0):
    """n float32 points of `comps` equally likely Gaussians with axis scales
    in [0.5, 2], centres uniform in [-center_range, center_range]^d."""
    centers = (torch.rand((comps, d), generator=g, device="cuda") * 2 - 1) * center_range
    scale = 0.5 * 4 ** torch.rand((comps, d), generator=g, device="cuda")
    c = torch.randint(0, comps, (n,), generator=g, device="cuda")
    z = torch.randn((n, d), generator=g, device="cuda")
    return (centers[c] + scale[c] * z).contiguous()


def _spread(case):
    """Centre range that keeps the components of low-dimensional data apart
    (the lifetime cut needs clusters to find)."""
    return 20.0 if case["d"] >= 8 else 10.0 * case["comps"] ** (1.0 / case["d"])


def _draws(case, seed):
    """Clusters per partition (the same for every seed: they fix the centroid
    array's shape) and the initial sample of each, drawn on the host."""
    r = random.Random(_of_case(case))
    ks = [r.randrange(case["kmin"], case["kmax"]) for _ in range(case["P"])]
    r = random.Random(seed)
    return ks, [r.sample(range(case["n"]), k) for k in ks]


def _knn_graph(n, k, g, keep=1.0):
    """Symmetric CSR graph of (up to) the k nearest neighbours of n uniform
    points in the unit cube, found among the 27 grid cells around a point,
    and of a random share `keep` of its edges: (dest, firstEdge, outDegree,
    edge index of every entry, edges)."""
    side = max(1, int(round((n / 8.0) ** (1 / 3))))
    pts = torch.rand((n, 3), generator=g, device="cuda")
    cell = (pts * side).long().clamp_(max=side - 1)
    flat = (cell[:, 0] * side + cell[:, 1]) * side + cell[:, 2]
    order = torch.argsort(flat, stable=True)
    start = torch.zeros(side ** 3 + 1, dtype=torch.long, device="cuda")
    start[1:] = torch.cumsum(torch.bincount(flat, minlength=side ** 3), 0)
    off = torch.tensor([(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)], device="cuda")
    cap = 48                                  # of three neighbouring cells of 8 points each
    slot = torch.arange(cap, device="cuda")
    keys = []
    for i0 in range(0, n, 1 << 16):
        i = torch.arange(i0, min(n, i0 + (1 << 16)), device="cuda")
        xy = cell[i, None, :2] + off                                   # m x 9 columns of cells
        inside = ((xy >= 0) & (xy < side)).all(-1)
        col = (xy[..., 0] * side + xy[..., 1]).clamp_(0, side * side - 1) * side
        lo = start[col + (cell[i, 2] - 1).clamp_(min=0)[:, None]]
        hi = start[col + (cell[i, 2] + 1).clamp_(max=side - 1)[:, None] + 1]
        at = lo[..., None] + slot
        ok = inside[..., None] & (at < hi[..., None])
        j = order[at.clamp_(max=n - 1)].view(i.numel(), -1)
        dist = (pts[j] - pts[i, None]).square_().sum(-1)
        dist[~ok.view(i.numel(), -1) | (j == i[:, None])] = math.inf
        near, pos = torch.topk(dist, k, dim=1, largest=False)
        v = j.gather(1, pos)
        u = i[:, None].expand_as(v)
        key = torch.minimum(u, v) * n + torch.maximum(u, v)
        keys.append(key[near < math.inf])
    key = torch.unique(torch.cat(keys))
    if keep < 1.0:
        key = key[torch.rand(key.numel(), generator=g, device="cuda") < keep]
    a, b = key // n, key % n
    e = key.numel()
    src, dst = torch.cat([a, b]), torch.cat([b, a])
    order = torch.argsort(src * n + dst)
    deg = torch.bincount(src, minlength=n)
    first = torch.cumsum(deg, 0) - deg
    return dst[order].int(), first.int(), deg.int(), order % e, e


def _graph(case, seed):
    g = _generator(seed)
    dest, first, deg, edge, e = _knn_graph(case["n"], case["knn"], g, case.get("keep", 1.0))
    if case["wtype"] == "float32":
        w = torch.rand(e, generator=g, device="cuda")
    else:
        hi = {"uint8": 255, "uint16": 65535, "int32": 1 << 24}[case["wtype"]]
        w = torch.randint(1, hi + 1, (e,), generator=g, device="cuda")
        w = w.to(getattr(torch, case["wtype"]))
    # uint16 tensors are indexed through a view of the same width
    w = w.view(torch.int16)[edge].view(torch.uint16) if case["wtype"] == "uint16" else w[edge]
    return dict(dest=dest, weight=w.contiguous(), first=first, deg=deg)


def _label_matrix(case, seed):
    """The label matrix of an ensemble: every point's nearest of k sampled
    points, per partition (what one K-Means label pass gives).  The seed
    draws the order of the points, of the partitions and of the cluster ids;
    the clusters themselves are the case's, so that matrices of two seeds
    have the same number of entries."""
    own = _of_case(case)
    n = case["n"]
    X = _mixture(n, case["d"], case["comps"], _generator(own), _spread(case))
    ks, inits = _draws(case, own)
    g = _generator(seed)
    order = torch.randperm(n, generator=g, device="cuda")
    rows = torch.randperm(case["P"], generator=g, device="cuda").tolist()
    L = torch.empty((case["P"], n), dtype=torch.int32, device="cuda")
    for p, idx in enumerate(inits):
        C = X[torch.tensor(idx, device="cuda")]
        ids = torch.randperm(ks[p], generator=g, device="cuda").int()
        L[rows[p]] = ids[(C.square().sum(1) - 2.0 * (X @ C.T)).argmin(1)][order]
    return L


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "scan":
        g = _generator(seed)
        s["x"] = torch.randint(0, 1001, (case["n"],), generator=g, device="cuda").to(
            getattr(torch, case["itype"]))
        s["out"] = torch.empty(case["n"], dtype=getattr(torch, case["otype"]), device="cuda")
    elif kind in ("mst", "cc"):
        s.update(_graph(case, seed))
    elif kind == "fit":
        # the reference's published K-Means runs take uniform points
        s["X"] = torch.rand((case["n"], case["d"]), generator=_generator(seed), device="cuda")
        s["seed"] = seed
    elif kind == "ensemble":
        s["X"] = _mixture(case["n"], case["d"], case["comps"], _generator(seed), _spread(case))
        s["ks"], s["inits"] = _draws(case, seed)
    elif kind == "coassoc":
        s["labels"] = _label_matrix(case, seed)
    elif kind == "final":
        e = EAC(case["n"], sparse=True, n_partitions=case["P"])
        e.buildMatrix(_label_matrix(case, seed))
        s["coassoc"] = (e.coassoc.indptr, e.coassoc.indices, e.coassoc.data)
    elif kind == "eac":
        s["X"] = _mixture(case["n"], case["d"], case["comps"], _generator(seed), _spread(case))
        s["seed"] = seed
    else:
        r = random.Random(_of_case(case))       # the instances' sizes
        g = _generator(seed)
        s["X"], s["params"] = [], []
        for i in range(case["m"]):
            n, d = _log_int(r, case["nmin"], case["nmax"]), r.choice((2, 4, 8, 16, 32))
            comps = r.randint(3, 30)
            s["X"].append(_mixture(n, d, comps, g, _spread(dict(d=d, comps=comps))))
            s["params"].append(draw_instance_params(n, k_range_rule1(n), case["P"], seed + i))
    return s


# --------------------------------------------------------------------- run --
def run(s):
    kind = s["kind"]
    if kind == "scan":
        total = exprefixsumNumba(s["x"], s["out"])
        return dict(out=s["out"], total=total)
    if kind == "mst":
        mst, n = boruvka_minho_gpu(s["dest"], s["weight"], s["first"], s["deg"],
                                   returnDevAry=s["device_result"])
        return dict(mst=mst[:n], n=n)
    if kind == "cc":
        return dict(labels=connected_comps_gpu(s["dest"], s["weight"], s["first"], s["deg"],
                                               returnDevAry=s["device_result"]))
    if kind == "fit":
        random.seed(s["seed"])
        km = K_Means(n_clusters=s["k"], max_iter=3, label_mode=s["mode"]).fit(s["X"])
        return dict(labels=km.labels_, centroids=km.cluster_centers_, iters=km.iters_,
                    inertia=km.inertia_)
    if kind == "ensemble":
        labels, cent, dists, iters, inertia = kmeans_ensemble(s["X"], s["ks"], s["inits"],
                                                              max_iter=3, label_mode=s["mode"])
        return dict(labels=labels, centroids=cent, dists=dists, iters=iters, inertia=inertia)
    if kind == "coassoc":
        e = EAC(s["n"], sparse=True, n_partitions=s["P"])
        e.buildMatrix(s["labels"])
        c = e.coassoc
        return dict(indptr=c.indptr, indices=c.indices, data=c.data, nnz=c.nnz,
                    discarded=c.nnz_discarded)
    if kind == "final":
        n_fclusts, labels = sp_sl_lifetime_csr(*s["coassoc"], s["n"], s["P"])
        return dict(n_fclusts=n_fclusts, labels=labels)
    if kind == "eac":
        np.random.seed(s["seed"] % (1 << 32))
        random.seed(s["seed"])
        n_fclusts, labels, e = eac_pipeline(s["X"], s["P"], [s["kmin"], s["kmax"]],
                                            label_mode=s["mode"])
        return dict(n_fclusts=n_fclusts, labels=labels, nnz=e.coassoc.nnz)
    # device memory for the instances in flight: a share of the card
    res = eac_batch(s["X"], n_partitions=s["P"], params=s["params"], label_mode=s["mode"],
                    arena_bytes=8 << 30)
    return dict(labels=[r.labels for r in res], n_fclusts=np.array([r.n_fclusts for r in res]),
                nnz=np.array([r.nnz for r in res]))


# -------------------------------------------------------------------- work --
def _entries(n, comps):
    """Co-association entries, about: with partitions much finer than the
    mixture, a row co-occurs with the later points of its own component."""
    return 0.5 * n * (n / comps)


def work(case):
    kind = case["kind"]
    if kind == "scan":
        size = dict(int32=4, int64=8)
        return dict(bytes=case["n"] * (size[case["itype"]] + size[case["otype"]]), flops=case["n"])
    if kind in ("mst", "cc"):
        n = case["n"]
        e = 1.12 * case["knn"] * n * case.get("keep", 1.0)   # directed entries, pairs merged
        size = dict(uint8=1, uint16=2, int32=4, float32=4)[case["wtype"]]
        return dict(bytes=e * (4 + size) + 12 * n, flops=0)
    if kind == "batch":
        # the mean of n over a log-uniform range, 10 dimensions on average
        lo, hi = case["nmin"], case["nmax"]
        n = int((hi - lo) / math.log(hi / lo))
        one = dict(kind="eac", n=n, d=12, P=case["P"], kmin=int(math.sqrt(n) / 2),
                   kmax=int(math.sqrt(n)), comps=16)
        w = work(one)
        return dict(bytes=case["m"] * w["bytes"], flops=case["m"] * w["flops"])
    n, d, P = case["n"], case["d"], case.get("P", 1)
    k = case["k"] if kind == "fit" else 0.5 * (case["kmin"] + case["kmax"])
    if kind in ("fit", "ensemble"):
        # three label passes of a difference, a square and a sum per dimension
        # as one multiply-add each; points read once, labels and distances
        # written once
        return dict(bytes=4.0 * n * d + 8.0 * P * n + 4.0 * P * k * d, flops=3 * 2.0 * P * n * k * d)
    nnz = _entries(n, case["comps"])
    if kind == "coassoc":
        return dict(bytes=4.0 * P * n + 8.0 * n + 5.0 * nnz, flops=P * nnz)
    if kind == "final":
        return dict(bytes=12.0 * n + 5.0 * nnz, flops=0)
    return dict(bytes=4.0 * n * d + 8.0 * P * n + 10.0 * nnz, flops=3 * 2.0 * P * n * k * d)


# ------------------------------------------------------------------- exact --
def _lloyd64(X, idx, iters=3):
    """Lloyd's iterations in 64 bits from the points `idx`: centroids of the
    last label pass, squared distances and their sum; None where a cluster
    runs empty (the point it then takes has no exact value)."""
    X = X.double()
    X0 = X.mean(0)
    X = X - X0
    C = X[torch.as_tensor(idx, device=X.device)]
    step = max(1, (1 << 27) // C.shape[0])
    for it in range(iters):
        lab, dist = [], []
        for i in range(0, X.shape[0], step):
            x = X[i:i + step]
            l = (C.square().sum(1) - 2.0 * (x @ C.T)).argmin(1)
            lab.append(l)
            dist.append((x - C[l]).square().sum(1))
        lab, dist = torch.cat(lab), torch.cat(dist)
        if it + 1 == iters:
            return C + X0, dist, dist.sum()
        count = torch.bincount(lab, minlength=C.shape[0])
        if int(count.min()) == 0:
            return None
        C = torch.zeros_like(C).index_add_(0, lab, X) / count[:, None]


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed) if kind in ("fit", "ensemble") else None
    if kind == "fit":
        r = random.Random(seed)                 # the sample K_Means.fit draws
        got = _lloyd64(s["X"], r.sample(range(case["n"]), case["k"]))
        if got is None:
            return None
        return dict(labels=None, centroids=got[0], iters=None, inertia=float(got[2]))
    if kind == "ensemble":
        cent = torch.zeros((case["P"], max(s["ks"]), case["d"]), dtype=torch.float64, device="cuda")
        dists = torch.empty((case["P"], case["n"]), dtype=torch.float64, device="cuda")
        for p, idx in enumerate(s["inits"]):
            got = _lloyd64(s["X"], idx)
            if got is None:
                return None
            cent[p, :len(idx)], dists[p] = got[0], got[1]
        return dict(labels=None, centroids=cent, dists=dists, iters=None, inertia=dists.sum(1))
    # everything else is whole numbers: indices, labels and counts
    return None
