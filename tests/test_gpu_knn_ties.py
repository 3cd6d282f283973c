"""Lists of points at equal distances: (distance, the point itself, lower index)
decides, and of a run of equal candidates longer than a row keeps the lowest
indices stay. Integer coordinates, so operands, norms and scores are exact in
every arm; the squared distances are summed as the search sums them (FP32, a
fused multiply-add a coordinate), which rounds for one far point only."""
import numpy as np
import pytest

import sc_gpu

pytestmark = pytest.mark.gpu

KEPT = 32  # candidates a row keeps of either half of the columns
ARMS = [sc_gpu.KNN_FP32, sc_gpu.KNN_BF16]


def _lattice(n, d, values, seed):
    return np.random.Generator(np.random.PCG64(seed)).integers(0, values, (n, d)).astype(np.float32)


def _expected(X, k):
    n = len(X)
    index = np.empty((n, k + 1), np.int64)
    dist = np.empty((n, k + 1), np.float32)
    ids = np.arange(n)
    for q in range(n):
        d2 = np.zeros(n, np.float32)
        for c in X.T:
            d2 = (np.float64(c - c[q]) ** 2 + d2).astype(np.float32)
        index[q] = np.lexsort((ids, ids != q, d2))[:k + 1]
        dist[q] = np.sqrt(d2[index[q]])
    return index, dist


def _copies_before(X):
    """How many points of lower index equal each point."""
    _, group = np.unique(X, axis=0, return_inverse=True)
    group = group.reshape(-1)
    order = np.argsort(group, kind="stable")
    starts = np.concatenate([[0], np.flatnonzero(np.diff(group[order])) + 1])
    rank = np.arange(len(X)) - np.repeat(starts, np.diff(np.append(starts, len(X))))
    out = np.empty(len(X), np.int64)
    out[order] = rank
    return out


def _points(kind, n, copies, seed):
    if kind == "lattice":    # 27 places: every distance is shared by many
        return _lattice(n, 3, 3, seed)
    X = _lattice(n, 12, 5, seed)
    if kind == "wide":       # a range that takes BF16 operands
        X[-1] = 2.0 ** 14
    at = np.random.Generator(np.random.PCG64(seed)).permutation(n - 1)[:copies] if kind == "scattered" \
        else np.arange(copies)
    X[np.sort(at)] = 2.0
    return X


@pytest.mark.parametrize("arm", ARMS)
@pytest.mark.parametrize("k", [10, 23, 24, 31])
@pytest.mark.parametrize("kind,n,copies", [("first", 600, 33), ("first", 600, 36), ("first", 600, 37),
                                           ("first", 600, 64), ("wide", 600, 50), ("scattered", 3000, 200),
                                           ("lattice", 500, 0), ("lattice", 2000, 0)])
def test_equal_distances_keep_the_lowest_indices(kind, n, copies, k, arm):
    X = _points(kind, n, copies, n + copies)
    index, dist = _expected(X, k)
    r = sc_gpu.knn_gaussian(X, k, precision=arm)
    rows = np.ones(n, bool)
    if kind == "wide" and arm == sc_gpu.KNN_BF16:
        rows[-1] = False  # the far point's scores are finer than its FP32 distances
    assert np.array_equal(r.distances[rows], dist[rows])
    sure = rows & (_copies_before(X) < KEPT)  # itself among the lowest of its equals
    assert sure.sum() > KEPT
    assert np.array_equal(r.index[sure], index[sure])


@pytest.mark.parametrize("arm", ARMS)
def test_equal_points_of_a_pruned_size(arm):
    """70,000 points, where the 16-bit arm prunes: 200 of them are one point."""
    n, k = 70_000, 15
    X = np.random.Generator(np.random.PCG64(4)).normal(size=(n, 12)).astype(np.float32)
    at = np.sort(np.random.Generator(np.random.PCG64(5)).permutation(n)[:200])
    X[at] = X[at[0]]
    if arm == sc_gpu.KNN_FP32:
        index = np.stack([sc_gpu.knn_search(X, k, int(i), int(i) + 1, precision=arm)[0][0] for i in at[:KEPT]])
    else:
        index = sc_gpu.knn_gaussian(X, k, precision=arm).index[at[:KEPT]]
        assert sc_gpu.knn_last_stats()["clusters"] >= 16
    for i, row in zip(at, index):
        assert np.array_equal(row, np.concatenate([[i], at[at != i]])[:k + 1])


@pytest.mark.parametrize("arm", ARMS)
@pytest.mark.parametrize("k", [10, 24, 31])
@pytest.mark.parametrize("kind,n,copies", [("first", 600, 50), ("first", 600, 200), ("wide", 600, 120),
                                           ("scattered", 3000, 200), ("lattice", 2000, 0)])
def test_every_point_heads_its_own_list(kind, n, copies, k, arm):
    """Also a point with more equals of lower index than a row keeps candidates."""
    X = _points(kind, n, copies, n + copies)
    assert (_copies_before(X) >= KEPT).any()
    index, dist = _expected(X, k)
    r = sc_gpu.knn_gaussian(X, k, precision=arm)
    rows = np.ones(n, bool)
    if kind == "wide" and arm == sc_gpu.KNN_BF16:
        rows[-1] = False  # as above
    assert np.array_equal(r.index[:, 0], np.arange(n))
    assert np.array_equal(r.index[rows], index[rows]) and np.array_equal(r.distances[rows], dist[rows])


def test_every_point_heads_its_own_list_when_pruned():
    n, k = 70_000, 15
    X = np.random.Generator(np.random.PCG64(4)).normal(size=(n, 12)).astype(np.float32)
    at = np.sort(np.random.Generator(np.random.PCG64(5)).permutation(n)[:200])
    X[at] = X[at[0]]
    r = sc_gpu.knn_gaussian(X, k)
    assert sc_gpu.knn_last_stats()["clusters"] >= 16
    assert np.array_equal(r.index[:, 0], np.arange(n))
    for i in at:
        assert np.array_equal(r.index[i], np.concatenate([[i], at[at != i]])[:k + 1])
        assert not r.distances[i].any()


@pytest.mark.parametrize("arm", ARMS)
def test_a_point_that_is_not_finite_has_no_distance_to_itself(arm):
    X = np.random.Generator(np.random.PCG64(6)).normal(size=(300, 5)).astype(np.float32)
    X[7, 2], X[8, 0] = np.inf, np.nan
    r = sc_gpu.knn_gaussian(X, 4, precision=arm)
    # no distance of theirs is finite, so neither heads its list; the infinite one's
    # 16-bit scores are -inf where the products are, and such points are listed
    assert np.all(np.isinf(r.distances[7:9]))
    assert 7 not in r.index[7] and np.all(r.index[8] == 0xFFFFFFFF)
    if arm == sc_gpu.KNN_FP32:
        assert np.all(r.index[7] == 0xFFFFFFFF)
    else:
        assert np.array_equal(r.index[7], np.flatnonzero(X[:, 2] > 0)[np.flatnonzero(X[:, 2] > 0) != 7][:5])
    others = np.delete(np.arange(300), [7, 8])
    assert np.array_equal(r.index[others, 0], others)
