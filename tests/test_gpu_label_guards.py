"""K-Means labels where a screen of rounded scores could go wrong: NaN,
infinite, huge and tiny values, ties, ragged shapes, data far from its mean.
Both labelers promise the reference's labels and distances for any input, so
every comparison is exact."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

MODES = ["cuda", "bf16"]


def _check(x, c, mode):
    from masters_final_b200.cluster.KMeans import kmeans_label
    with np.errstate(all="ignore"):
        want = oracle.kmeans_label(x, c)
    lab, dist = kmeans_label(x, c, label_mode=mode)
    assert np.array_equal(lab.cpu().numpy(), want[0])
    assert np.array_equal(dist.cpu().numpy(), want[1], equal_nan=True)


@pytest.mark.parametrize("d", [1, 2, 3, 5, 7, 9, 13, 16, 17, 25, 32])
@pytest.mark.parametrize("k", [1, 3, 5, 127, 130, 515])
def test_label_bf16_shapes(d, k):
    """The tensor-core labeler on every padded dimension, ragged chunks and
    tiles of centroids, a far-off mean, ties, points on centroids."""
    rng = np.random.default_rng(100 * d + k)
    for n in (700, 3001):
        x = (rng.standard_normal((n, d)) + 300.0 * rng.standard_normal(d)).astype(np.float32)
        c = x[rng.choice(n, k, replace=False)].copy()
        if k > 2:
            c[k - 1] = c[0]                       # exact tie between distant ids
        x[:40] = c[rng.integers(0, k, 40)]
        _check(x, c, "bf16")


@pytest.mark.parametrize("bad", [None, 0, 1, 2, 6])
def test_label_bf16_special_values(bad):
    """Infinities, NaN points, huge and tiny values, and a NaN centroid: the
    reference never takes a NaN distance except from centroid 0."""
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
    _check(x, c, "bf16")


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("bad", [0, 1, 30])
def test_label_finite_points_nan_centroid(mode, bad):
    """Finite points and one NaN centroid.  Centroid 0: the reference keeps it
    for every point.  Elsewhere it changes nothing, also for points whose
    distances to the finite centroids, all at norms near 100, differ in their
    last digits."""
    rng = np.random.default_rng(bad)
    c = rng.standard_normal((40, 3))
    c = (100.0 * c / np.linalg.norm(c, axis=1, keepdims=True)).astype(np.float32)
    c[bad] = np.nan
    x = (rng.standard_normal((20000, 3)) * 1e-3).astype(np.float32)
    _check(x, c, mode)


@pytest.mark.parametrize("mode", MODES)
def test_ensemble_nan_row_two_passes(mode):
    """A NaN row takes label 0 in the first pass and makes centroid 0 NaN in
    the update, so the second pass gives every point label 0 at a NaN distance."""
    from masters_final_b200.cluster.KMeans import kmeans_ensemble
    rng = np.random.default_rng(11)
    x = rng.standard_normal((6000, 4)).astype(np.float32)
    x[1234] = np.nan
    init = [i for i in rng.choice(6000, 30, replace=False).tolist() if i != 1234]
    with np.errstate(all="ignore"):
        l1, d1 = oracle.kmeans_label(x, x[init])
        c2 = oracle.kmeans_centroids(x, l1, d1, len(init))
        l2, d2 = oracle.kmeans_label(x, c2)
    assert np.isnan(c2[0]).all() and (l2 == 0).all()
    lab, cent, dist, _, _ = kmeans_ensemble(x, [len(init)], [init], max_iter=2, label_mode=mode)
    assert np.array_equal(cent[0].cpu().numpy(), c2, equal_nan=True)
    assert np.array_equal(lab[0].cpu().numpy(), l2)
    assert np.array_equal(dist[0].cpu().numpy(), d2, equal_nan=True)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("d", [1, 2, 5, 16])
def test_label_overflowing_distances(mode, d):
    """Finite points whose squared distances to every centroid pass the
    largest float: the reference's distances are all infinite and it keeps
    label 0; nearer points are labelled as ever."""
    rng = np.random.default_rng(d)
    x = rng.standard_normal((4000, d)).astype(np.float32)
    side = np.where(rng.random(4000) < 0.5, 1.0, -1.0)
    x[:, 0] = side * (1.1e19 + 1e17 * rng.standard_normal(4000))
    c = rng.standard_normal((6, d)).astype(np.float32)
    c[:, 0] = [1.16e19, 1.1e19, 1.12e19, 1.07e19, 1.14e19, 1.11e19]
    _check(x, c, mode)


def _check_sample(x, c, rows):
    """The whole call on the GPU, the oracle on some of its points."""
    from masters_final_b200.cluster.KMeans import kmeans_label
    with np.errstate(all="ignore"):
        want = oracle.kmeans_label(x[rows], c)
    lab, dist = kmeans_label(x, c, label_mode="cuda")
    assert np.array_equal(lab.cpu().numpy()[rows], want[0])
    assert np.array_equal(dist.cpu().numpy()[rows], want[1], equal_nan=True)


# points from which a thread takes eight or four points at once, and fewer;
# with these clusters the work is above what the direct kernel takes alone
SCREEN = [(1, 620_003, 515), (1, 620_003, 1031), (1, 310_003, 1029), (2, 620_003, 257),
          (2, 620_003, 260), (2, 310_003, 515), (3, 620_003, 261), (3, 620_003, 150),
          (4, 620_003, 259), (4, 620_003, 131), (4, 310_003, 258), (5, 620_003, 130),
          (6, 620_003, 127), (6, 310_003, 161), (7, 620_003, 129), (8, 620_003, 66),
          (8, 310_003, 133), (9, 310_003, 129), (12, 310_003, 130), (12, 120_001, 257),
          (13, 310_003, 127), (16, 310_003, 67), (16, 120_001, 150), (17, 120_001, 161),
          (24, 120_001, 130), (25, 120_001, 129), (32, 120_001, 131)]


def _screen_case(d, n, k, spread, seed):
    """Blobs `spread` standard deviations apart at most, centroids among the
    points with two equal ones, and rows to compare: points on centroids, the
    last ones, others at random."""
    rng = np.random.default_rng(seed)
    at = rng.uniform(-spread, spread, (20, d)).astype(np.float32)
    x = rng.standard_normal((n, d), dtype=np.float32) + at[rng.integers(0, 20, n)]
    c = x[rng.choice(n, k, replace=False)].copy()
    c[k - 1] = c[0]
    x[:300] = c[rng.integers(0, k, 300)]
    rows = np.unique(np.concatenate([np.arange(300), np.arange(n - 300, n), rng.choice(n, 2500)]))
    return x, c, rows


@pytest.mark.parametrize("spread", [0.0, 3000.0])
@pytest.mark.parametrize("d,n,k", SCREEN)
def test_label_f32_screen(d, n, k, spread):
    """The screening kernel in each of its shapes: every padded dimension,
    chunks of four and eight with ragged last ones, all points-per-thread
    variants; and the direct kernel after it, for blobs so far apart that the
    screen leaves most points open."""
    assert d * n * k > 1 << 28 and k > 32
    _check_sample(*_screen_case(d, n, k, spread, d + n + k))


@pytest.mark.parametrize("d,n,k", [(2, 620_003, 260), (5, 620_003, 130), (16, 310_003, 67),
                                   (32, 120_001, 131)])
@pytest.mark.parametrize("kind", ["ties", "nan0", "inf", "tiny"])
def test_label_f32_screen_open_points(kind, d, n, k):
    """Most points left to the direct kernel's last sweep: integer points with
    ties all over, a NaN centroid 0, infinite points, subnormal squares."""
    x, c, rows = _screen_case(d, n, k, 0.0, d)
    if kind == "ties":
        x, c = np.round(x), np.round(c)
    elif kind == "nan0":
        c[0, d - 1] = np.nan
    elif kind == "inf":
        x[1::3, 0] = np.inf
        x[2::9] = np.nan
        c[0, 0] = np.inf
    else:
        x *= np.float32(1e-22)
        c *= np.float32(1e-22)
    _check_sample(x, c, rows)


def _ensemble_ms(x, k, P, mode):
    """Device time of one label pass, the best of six."""
    import torch
    from masters_final_b200.cluster.KMeans import kmeans_ensemble
    rng = np.random.default_rng(1)
    inits = [rng.choice(x.shape[0], k, replace=False).tolist() for _ in range(P)]
    best = float("inf")
    for _ in range(6):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        kmeans_ensemble(x, [k] * P, inits, max_iter=1, label_mode=mode)
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def test_label_time_far_from_mean():
    """Well-separated blobs cost more than one (a second sweep), by less than
    the factor of five that makes the screen no faster than differences to
    begin with."""
    import torch
    n, d = 400_000, 16
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    z = torch.randn((n, d), generator=g, device="cuda")
    at = (torch.rand((20, d), generator=g, device="cuda") * 2 - 1) * 3000.0
    far = at[torch.randint(0, 20, (n,), generator=g, device="cuda")] + z
    assert _ensemble_ms(far, 530, 4, "cuda") < 5.0 * _ensemble_ms(z, 530, 4, "cuda")


@pytest.mark.parametrize("odd", [1e6, float("nan")])
def test_label_time_few_rows_far_out(odd):
    """Ten rows far out do not move the centre of the others' scores: the
    tensor-core pass takes less than twice its time without them."""
    import torch
    n, d = 200_000, 32
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    z = torch.randn((n, d), generator=g, device="cuda")
    x = z.clone()
    x[:10] *= odd
    assert _ensemble_ms(x, 300, 4, "bf16") < 2.0 * _ensemble_ms(z, 300, 4, "bf16")
