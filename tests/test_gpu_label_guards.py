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
