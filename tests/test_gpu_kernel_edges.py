"""Kernels and dispatch branches at the sizes where they change: tile edges,
remainders, the smallest and largest of a range.  Everything compared here is
whole numbers or float32 results with a fixed order of operations, so every
comparison is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the one-block scan's step and limit, the tile of the look-back scan
SCAN_STEP, SCAN_SMALL_MAX, SCAN_TILE = 16384, 32768, 8192


@pytest.mark.parametrize("types", ["i32_i32", "i32_i64", "i64_i64"])
@pytest.mark.parametrize("n", [1, 3, 511, 513, SCAN_STEP - 1, SCAN_STEP, SCAN_STEP + 1,
                               SCAN_SMALL_MAX - 5, SCAN_SMALL_MAX, SCAN_SMALL_MAX + 1,
                               5 * SCAN_TILE, 5 * SCAN_TILE + 1, 40 * SCAN_TILE + 4099])
@pytest.mark.parametrize("offset", [0, 1])
def test_scan_edges(types, n, offset):
    """Both scans against numpy's running sum in 64 bits, aligned and one
    element off the 16-byte boundary, negative values and an initial value."""
    import torch
    from masters_final_b200.utils.scan import exprefixsumNumba, exprefixsumNumbaSingle
    ti, to = {"i32_i32": (np.int32, np.int32), "i32_i64": (np.int32, np.int64),
              "i64_i64": (np.int64, np.int64)}[types]
    rng = np.random.default_rng(n + offset)
    hi = 1 << 31 if ti == np.int32 else 1 << 40
    x = rng.integers(-hi, hi, size=n).astype(ti)
    c = np.cumsum(x.astype(np.int64)) + 7
    want = np.concatenate([[7], c[:-1]]).astype(np.int64).astype(to)
    xd = torch.empty(n + offset, dtype=getattr(torch, np.dtype(ti).name), device="cuda")[offset:]
    od = torch.empty(n + offset, dtype=getattr(torch, np.dtype(to).name), device="cuda")[offset:]
    xd.copy_(torch.from_numpy(x))
    assert exprefixsumNumba(xd, od, 7) == int(c[-1])
    assert np.array_equal(od.cpu().numpy(), want)
    assert np.array_equal(xd.cpu().numpy(), x)
    if ti == to:                                       # in place
        assert exprefixsumNumbaSingle(xd, 7) == int(c[-1])
        assert np.array_equal(xd.cpu().numpy(), want)


@pytest.mark.parametrize("fill", [0, 255])
def test_scan_empty_stream(fill):
    """No element: the total is the initial value, and the workspace's error
    word, whatever was there, reads as no error."""
    import torch
    from masters_final_b200 import _lib
    L = _lib.load()
    total = torch.empty(1, dtype=torch.int64, device="cuda")
    for f in (L.eacb_scan_excl_i32, L.eacb_scan_excl_i32_i64, L.eacb_scan_excl_i64):
        ws = torch.full((int(L.eacb_scan_workspace_size(0)),), fill, dtype=torch.uint8, device="cuda")
        _lib.check(f(None, None, 0, 42, _lib.ptr(total), _lib.ptr(ws), ws.numel(),
                     _lib.stream_handle()), "scan")
        _lib.check(L.eacb_workspace_status(_lib.ptr(ws), _lib.stream_handle()), "scan")
        assert int(total.item()) == 42


@pytest.mark.parametrize("kind", ["random", "equal", "few", "ascending", "descending"])
@pytest.mark.parametrize("n,empty", [(40, 3), (256, 1), (257, 5), (2000, 300), (16383, 2),
                                     (16384, 2), (70001, 1), (70001, 300), (300001, 7)])
def test_empty_cluster_selection(kind, n, empty):
    """The points the empty clusters take, one block and a cluster of blocks,
    against the oracle's quickselect: pivots that keep the lower part and
    (equal, descending keys) ones that settle it and go on above."""
    import torch
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_centroids
    rng = np.random.default_rng(n + empty)
    x = rng.standard_normal((n, 2)).astype(np.float32)
    full = 5
    k = full + empty
    ids = np.sort(rng.choice(k, full, replace=False)).astype(np.int32)
    labels = ids[rng.integers(0, full, n)]
    labels[:full] = ids
    dist = {"random": rng.random(n), "equal": np.ones(n), "few": rng.integers(0, 3, n),
            "ascending": np.arange(n) / n, "descending": np.arange(n, 0, -1) / n}[kind].astype(np.float32)
    got = kmeans_centroids(x, labels, dist, k).cpu().numpy()
    want = oracle.kmeans_centroids(x, labels, dist, k)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n,ones,empty", [(256, 126, 129), (256, 126, 128), (255, 125, 129),
                                          (257, 126, 130), (40, 18, 20)])
def test_empty_cluster_selection_standing_range(n, ones, empty):
    """Two distance values with the smaller one from the middle on: the
    quickselect's range stands still for steps on end, and it takes more steps
    than the range has keys."""
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_centroids
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 2)).astype(np.float32)
    full = 5
    k = full + empty
    ids = np.sort(rng.choice(k, full, replace=False)).astype(np.int32)
    labels = ids[rng.integers(0, full, n)]
    labels[:full] = ids
    dist = np.where(np.arange(n) < ones, 1.0, 0.0).astype(np.float32)
    got = kmeans_centroids(x, labels, dist, k).cpu().numpy()
    assert np.array_equal(got, oracle.kmeans_centroids(x, labels, dist, k))


@pytest.mark.parametrize("n", [1, 7, 8, 128, 129, 255, 257, 1023, 2049, 4111, 16385, 131073, 262207,
                               1000003])
def test_inertia_order(n):
    """The inertia is numpy's pairwise float32 sum of the distances, bit for
    bit, at the sizes where its split tree changes depth."""
    from masters_final_b200.cluster.KMeans import kmeans_ensemble
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((n, 3)) * 10).astype(np.float32)
    ks = [1, min(2, n)]
    inits = [[0], list(range(ks[1]))]
    _, _, dists, _, inertia = kmeans_ensemble(x, ks, inits, max_iter=1)
    d = dists.cpu().numpy()
    for p in range(2):
        assert inertia[p].item() == np.add.reduce(d[p])


@pytest.mark.parametrize("d", [1, 2, 3, 4, 6, 8, 17, 32])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("f64", [False, True])
def test_centroid_batches(d, offset, f64):
    """Centroid sums at cluster sizes around the staging batch (1 to a few
    thousand members), rows on and off the 16-byte boundary."""
    import torch
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_centroids
    rng = np.random.default_rng(d)
    b = min(256, 1024 // d)
    sizes = [1, 2, b - 1, b, b + 1, 2 * b, 2 * b + 1, 3 * b + 7, 5000]
    labels = rng.permutation(np.repeat(np.arange(len(sizes)), sizes)).astype(np.int32)
    x = (rng.standard_normal((labels.size, d)) * 100).astype(np.float32)
    buf = torch.empty(x.size + offset, device="cuda")[offset:]
    buf.copy_(torch.from_numpy(x.reshape(-1)))
    dist = np.zeros(labels.size, dtype=np.float32)
    got = kmeans_centroids(buf.view(-1, d), labels, dist, len(sizes),
                           centroid_mode="f64" if f64 else "numba")
    assert np.array_equal(got.cpu().numpy(), oracle.kmeans_centroids(x, labels, dist, len(sizes), f64=f64))


@pytest.mark.parametrize("d", [1, 2, 3, 7, 8, 11, 16, 17, 22, 31, 32])
@pytest.mark.parametrize("per", [1, 16, 47, 48, 130])
@pytest.mark.parametrize("f64", [False, True])
def test_centroid_small_clusters(d, per, f64):
    """Centroid sums around the average size where the kernel changes, with
    clusters of one to a few hundred points, and at the dimensions whose rows
    are copied one, two or more at a time."""
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_centroids
    rng = np.random.default_rng(d * 1000 + per)
    k = 90
    labels = np.minimum((rng.random(k * per) ** 2 * k).astype(np.int32), k - 1)
    labels[:k] = np.arange(k)
    x = (rng.standard_normal((labels.size, d)) * 100).astype(np.float32)
    dist = rng.random(labels.size).astype(np.float32)
    got = kmeans_centroids(x, labels, dist, k, centroid_mode="f64" if f64 else "numba")
    assert np.array_equal(got.cpu().numpy(), oracle.kmeans_centroids(x, labels, dist, k, f64=f64))


@pytest.mark.parametrize("d", [1, 2, 3, 5, 7, 9, 13, 16, 17, 25, 32])
@pytest.mark.parametrize("k", [1, 3, 5, 127, 130, 515])
def test_label_f32_shapes(d, k):
    """The float32 label pass against the reference's loop: every padded
    dimension, ragged groups of four centroids and staging buffers, both
    points-per-thread variants, a far-off mean, ties, points on centroids."""
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_label
    rng = np.random.default_rng(100 * d + k)
    for n in (700, 310_003 if k == 130 and d in (2, 8, 16) else 3001):
        x = (rng.standard_normal((n, d)) + 300.0 * rng.standard_normal(d)).astype(np.float32)
        c = x[rng.choice(n, k, replace=False)].copy()
        if k > 2:
            c[k - 1] = c[0]                       # exact tie between distant ids
        x[:40] = c[rng.integers(0, k, 40)]
        lab, dist = kmeans_label(x, c, label_mode="cuda")
        want = oracle.kmeans_label(x, c)
        assert np.array_equal(lab.cpu().numpy(), want[0])
        assert np.array_equal(dist.cpu().numpy(), want[1])


@pytest.mark.parametrize("bad", [None, 0, 1, 2, 6])
def test_label_f32_special_values(bad):
    """Infinities, NaN points, huge and tiny values, and a NaN centroid: the
    reference never takes a NaN distance except from centroid 0."""
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_label
    rng = np.random.default_rng(5)
    x = rng.standard_normal((4000, 3)).astype(np.float32)
    c = x[:7].copy()
    x[100:110] *= np.float32(1e25)
    x[110:140] *= np.float32(1e-30)
    x[200, 1] = np.inf
    x[201, 0] = -np.inf
    x[202] = np.nan
    c[4] = 0
    if bad is not None:
        c[bad, 1] = np.nan
        c[(bad + 3) % 7, 0] = np.inf
    with np.errstate(all="ignore"):
        want = oracle.kmeans_label(x, c)
    lab, dist = kmeans_label(x, c, label_mode="cuda")
    assert np.array_equal(lab.cpu().numpy(), want[0])
    assert np.array_equal(dist.cpu().numpy(), want[1], equal_nan=True)


@pytest.mark.parametrize("offset", [0, 1, 15])
@pytest.mark.parametrize("n", [1, 14, 16, 17, 31, 64, 4096 + 5, 1 << 20, (1 << 22) + 13])
def test_diassoc_edges(n, offset):
    """top - count on spans that start and end off the 16-byte boundary; the
    bytes around the span stay as they are."""
    import torch
    from masters_final_b200 import _lib
    rng = np.random.default_rng(n)
    host = rng.integers(0, 256, n + 40, dtype=np.uint8)
    d = torch.from_numpy(host.copy()).cuda()
    span = d[offset:offset + n]
    _lib.check(_lib.load().eacb_make_diassoc(_lib.ptr(span), n, 101, _lib.stream_handle()), "diassoc")
    want = host.copy()
    want[offset:offset + n] = (101 - want[offset:offset + n].astype(np.int64)).astype(np.uint8)
    assert np.array_equal(d.cpu().numpy(), want)


@pytest.mark.parametrize("k", [1, 2, 700, 8192])
@pytest.mark.parametrize("n", [1, 31, 512, 4095, 4096, 4097, 12801])
def test_member_lists(n, k):
    """The stable counting sort behind the centroid sums at tile and warp
    edges, with one, few and the most clusters: float32 sums in point order
    tell every misplaced member."""
    import oracle
    from masters_final_b200.cluster.KMeans import kmeans_centroids
    rng = np.random.default_rng(n * 7 + k)
    labels = rng.integers(0, k, n).astype(np.int32)
    labels[n // 2:] = np.sort(labels[n // 2:])
    x = (rng.standard_normal((n, 2)) * 10.0 ** rng.integers(-3, 4, (n, 1))).astype(np.float32)
    dist = rng.random(n).astype(np.float32)
    if k - np.unique(labels).size >= n:
        pytest.skip("more empty clusters than points")
    got = kmeans_centroids(x, labels, dist, k).cpu().numpy()
    assert np.array_equal(got, oracle.kmeans_centroids(x, labels, dist, k))


@pytest.mark.parametrize("n,P,K,cap", [(300, 5, 3, 110), (4000, 9, 6, 900), (42_000, 5, 12, 4100),
                                       (41_100, 255, 9, 5000)])
def test_capped_rows(n, P, K, cap):
    """Rows over their capacity against the row restatement: spans below and
    above the rank chunk, many partitions, quotas inside a rank."""
    import torch
    import oracle
    from masters_final_b200.EAC.sparse import CoassocBuilder, capacity_indptr
    rng = np.random.default_rng(n + P)
    L = rng.integers(0, K, (P, n)).astype(np.int32)
    L[rng.random((P, n)) < 0.02] = -1
    b = CoassocBuilder(L, n)
    caps = capacity_indptr(n, cap, "constant")
    ip, ind, dat, nnz, disc, mx = b.build(caps)
    ip = ip.cpu().numpy()
    assert disc > 0
    rows = np.unique(np.concatenate([[0, 1, 2, n // 2, n - 2, n - 1], rng.integers(0, n, 40),
                                     rng.integers(0, max(1, n - 40_000), 8)]))
    want = oracle.coassoc_rows(L, caps.cpu().numpy(), rows)
    for i, (cols, counts) in zip(rows, want):
        a, e = ip[i], ip[i + 1]
        assert np.array_equal(ind[a:e].cpu().numpy(), cols), i
        assert np.array_equal(dat[a:e].cpu().numpy(), counts), i


@pytest.mark.parametrize("order", ["ascending", "shuffled"])
@pytest.mark.parametrize("off_w,off_i", [(0, 0), (4, 0), (3, 1)])
def test_final_clustering_pairs(order, off_w, off_i):
    """The last phase by pairs of components: large and small components
    (around the 32 vertices that give one a bitmap), single points, columns in
    any order, arrays off their vector boundaries, entries that are not
    between two components' least; against the oracle.  A column outside
    (row, n) in that phase is refused."""
    import torch
    import oracle
    from masters_final_b200._lib import EACBError
    from masters_final_b200.EAC.eac import sp_sl_lifetime_csr
    rng = np.random.default_rng(5)
    sizes = [700, 600, 500, 400, 300, 200, 33, 32, 31, 20, 9, 4, 2, 1, 1] + [64] * 10
    n = sum(sizes)
    group = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    a, b = np.triu_indices(n, 1)
    keep = (group[a] == group[b]) | (group[a] + group[b] > 1)        # 0 and 1 share no entry
    a, b = a[keep], b[keep]
    assert a.size >= 1 << 22
    inside = group[a] == group[b]
    w = np.where(inside, rng.integers(1, 60, a.size), rng.integers(100, 220, a.size)).astype(np.uint8)
    small = np.isin(group[a], np.nonzero(np.array(sizes) < 64)[0])
    w[inside & small] = 2                                            # whole after the first phase
    indptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(a, minlength=n), out=indptr[1:])
    cols, wts = b.astype(np.int32), w.copy()
    if order == "shuffled":
        p = np.lexsort((rng.random(a.size), a))
        cols, wts = cols[p], wts[p]

    def dev(x, off):
        t = torch.empty(x.size + off, dtype=getattr(torch, x.dtype.name), device="cuda")[off:]
        t.copy_(torch.from_numpy(x))
        return t
    wd, cd = dev(wts, off_w), dev(cols, off_i)
    for P in (219, 250):
        nc, labels = sp_sl_lifetime_csr(indptr, cd, wd, n, P)
        nc2, lab2 = oracle.sp_sl_lifetime(n, a.astype(np.int64), b.astype(np.int64), w, P)
        assert nc == nc2
        if nc > 1:
            assert np.array_equal(labels, lab2)
    at = int(np.nonzero(wts >= 210)[0][1000])
    for bad in (0, n):
        cd[at] = bad
        with pytest.raises(EACBError):
            sp_sl_lifetime_csr(indptr, cd, wd, n, 219)


@pytest.mark.parametrize("n,P,K,near", [
    (129, 2, 3, True), (3000, 7, 11, True), (2600, 8, 10, False), (5000, 100, 40, True),
    (2500, 255, 60, True),
    (2600, 200, 8, False),       # too many clusters per row block for one operand
    (6000, 255, 600, True),      # more (partition, cluster) pairs than the cluster map holds
])
def test_pair_tiles(n, P, K, near):
    """Pair counts of row blocks as one-hot products and by comparison,
    against the row restatement: row blocks of one to 128 rows, one to 32
    units of eight partitions, clusters that neighbour each other or not."""
    import oracle
    from masters_final_b200.EAC.sparse import CoassocBuilder, capacity_indptr
    rng = np.random.default_rng(n + P + K)
    pos = rng.permutation(n) / n
    if near:
        L = np.stack([((pos + rng.random()) % 1.0 * max(2, K - int(rng.integers(0, 3)))).astype(np.int32)
                      for _ in range(P)])
    else:
        L = rng.integers(0, K, (P, n)).astype(np.int32)
        L[P // 2] = rng.integers(0, K + 3, n)
    L[rng.random((P, n)) < 0.02] = -1
    b = CoassocBuilder(L, n)
    caps = capacity_indptr(n, n, "constant")
    ip, ind, dat, nnz, disc, mx = b.build(caps)
    assert disc == 0
    ip, ind, dat = (x.cpu().numpy() for x in (ip, ind, dat))
    rows = np.unique(np.concatenate([[0, 1, n - 2, n - 1], rng.integers(0, n, 200)]))
    for i, (cols, counts) in zip(rows, oracle.coassoc_rows(L, caps.cpu().numpy(), rows)):
        assert np.array_equal(ind[ip[i]:ip[i + 1]], cols), i
        assert np.array_equal(dat[ip[i]:ip[i + 1]], counts), i


@pytest.mark.parametrize("n", [11_585, 11_600])
def test_final_clustering_sampled_plan(n):
    """Just below and above 2^26 entries, where the phases are planned from a
    sample of the weights: three cliques whose light edges join them, heavy
    edges between them, some weights in one entry each."""
    import torch
    from masters_final_b200.EAC.eac import sp_sl_lifetime_csr
    assert (n * (n - 1) // 2 > 1 << 26) == (n == 11_600)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    group = torch.randint(0, 3, (n,), generator=g, device="cuda")
    i, j = torch.triu_indices(n, n, 1, device="cuda")
    w = torch.randint(2, 40, (i.numel(),), generator=g, device="cuda", dtype=torch.uint8)
    w[group[i] != group[j]] = 200
    w[torch.tensor([3, 1000, i.numel() - 1], device="cuda")] += 7
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    indptr[1:] = torch.cumsum(torch.arange(n - 1, -1, -1, device="cuda"), 0)
    nc, labels = sp_sl_lifetime_csr(indptr, j.int(), w, n, 220)
    assert nc == 3
    group = group.cpu().numpy()
    first = {}
    want = np.array([first.setdefault(int(x), len(first)) for x in group])
    assert np.array_equal(labels, want)


def _block_matrix(n, blocks, kind, offset=0):
    """All pairs of n points in equal blocks: light entries inside a block,
    heavier ones between blocks ("apart"), every weight everywhere ("mixed"),
    or only the heaviest few between blocks ("late")."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n + blocks)
    a, b = torch.triu_indices(n, n, 1, device="cuda")
    inside = a * blocks // n == b * blocks // n
    lo, hi = {"apart": (20, 100), "mixed": (256, 0), "late": (250, 252)}[kind]
    w = torch.where(inside, torch.randint(0, lo, a.shape, generator=g, device="cuda"),
                    torch.randint(hi, 256, a.shape, generator=g, device="cuda"))
    ip = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ip[1:] = torch.cumsum(torch.bincount(a, minlength=n), 0)
    dat = torch.empty(w.numel() + offset, dtype=torch.uint8, device="cuda")[offset:]
    dat.copy_(w)
    return ip, b.int(), dat


@pytest.mark.parametrize("n", [2900, 5000])
@pytest.mark.parametrize("blocks", [2, 10, 100, 300, 1500])
@pytest.mark.parametrize("kind", ["apart", "mixed", "late"])
def test_final_blocks(n, blocks, kind):
    """Dense matrices of few to many components, on both sides of the estimate
    that decides between the pairs' phase and narrow ones: the clusters equal
    those of the ordinary phases (which weights one byte off take), and the
    blocks where they are apart."""
    from masters_final_b200.EAC.eac import sp_sl_lifetime_csr
    got = sp_sl_lifetime_csr(*_block_matrix(n, blocks, kind), n, 255)
    want = sp_sl_lifetime_csr(*_block_matrix(n, blocks, kind, 1), n, 255)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
    if kind == "apart":
        assert got[0] == blocks
        assert np.array_equal(got[1], np.arange(n) * blocks // n)


def test_final_time_entries_between_components():
    """Entries between hundreds of components take no longer than between a
    few (a quarter for the timing's spread): they took half as long again when
    all of them went through the pairs of components."""
    import torch
    from masters_final_b200.EAC.eac import sp_sl_lifetime_csr

    def ms(blocks):
        m = _block_matrix(11_600, blocks, "apart")
        best = float("inf")
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            sp_sl_lifetime_csr(*m, 11_600, 255)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    assert ms(300) < 1.25 * ms(10)
