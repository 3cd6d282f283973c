"""The two-scan candidate search of the 16-bit tensor-core arm against the FP32
arm (exact FP32 differences of every pair): equal lists, bit for bit, at the
edges of its tiles and lists and for point sets that drive each operand format
and each bound to its limits."""
import numpy as np
import pytest

import sc_gpu
from sc_gpu import synth

pytestmark = pytest.mark.gpu


def _points(kind, n, d, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    if kind == "mixture":
        return synth.gaussian_mixture(n, d, 6, seed=seed, sigma=(0.7, 1.5))[0]
    x = rng.normal(size=(n, d))
    if kind == "tiny":       # f16 needs its scale
        x *= 1e-7
    elif kind == "huge":     # past f16's own range without it
        x *= 1e9
    elif kind == "outlier":  # wider than f16 takes: BF16 operands
        x[0] *= 1e6
    elif kind == "small_rows":  # points far below the rest, above and below the f16 rule
        x[: n // 2] *= 2.0 ** -9
        x[n // 2: n // 2 + 3] = 0.0
    elif kind == "integers":  # exactly representable: the measured rounding error is zero
        x = np.round(3 * x)
    return x.astype(np.float32)


@pytest.mark.parametrize("kind", ["mixture", "tiny", "huge", "outlier", "small_rows"])
@pytest.mark.parametrize("n,d,k", [(1, 3, 1), (17, 3, 5), (127, 30, 10), (128, 31, 15), (129, 30, 15), (257, 62, 10),
                                   (1023, 7, 23), (1500, 50, 24), (2049, 50, 31), (5003, 30, 10)])
def test_scans_give_the_exact_lists(kind, n, d, k):
    X = _points(kind, n, d, n + d + k)
    a = sc_gpu.knn_gaussian(X, k, sigma=sc_gpu.SIGMA_KTH, sym=sc_gpu.SYM_UNION, precision=sc_gpu.KNN_FP32)
    b = sc_gpu.knn_gaussian(X, k, sigma=sc_gpu.SIGMA_KTH, sym=sc_gpu.SYM_UNION, precision=sc_gpu.KNN_BF16)
    if kind == "outlier":
        # the outlier's own scores all lie within one 16-bit rounding of its norm:
        # no 16-bit operand can rank its neighbours, so its row is left out
        assert np.array_equal(a.index[1:], b.index[1:])
        assert np.array_equal(a.distances[1:].view(np.uint32), b.distances[1:].view(np.uint32))
        return
    assert np.array_equal(a.index, b.index)
    assert np.array_equal(a.distances.view(np.uint32), b.distances.view(np.uint32))
    assert np.array_equal(a.conn_ptrs, b.conn_ptrs) and np.array_equal(a.conn_nbrs, b.conn_nbrs)
    assert np.array_equal(a.conn_w.view(np.uint32), b.conn_w.view(np.uint32))


@pytest.mark.parametrize("n,d,k", [(300, 4, 10), (3000, 12, 15)])
def test_ties_and_points_at_the_origin(n, d, k):
    """Equal distances (integer coordinates, repeated points, many points at the
    origin, where every score and bound is zero): the distances of the lists are
    the exact ones; which of the tied points is listed may differ."""
    X = _points("integers", n, d, 5)
    X[: 2 * k] = 0.0
    a = sc_gpu.knn_gaussian(X, k, precision=sc_gpu.KNN_FP32)
    b = sc_gpu.knn_gaussian(X, k, precision=sc_gpu.KNN_BF16)
    assert np.array_equal(a.distances, b.distances)
    assert np.array_equal(b.index[:, 0], np.arange(n))


@pytest.mark.parametrize("n,lo,hi", [(4000, 0, 1), (4000, 255, 1030), (4000, 3999, 4000)])
def test_query_rows_of_a_shard(n, lo, hi):
    X = _points("mixture", n, 40, 9)
    full = sc_gpu.knn_gaussian(X, 12, precision=sc_gpu.KNN_FP32)
    idx, d2 = sc_gpu.knn_search(X, 12, lo, hi)
    assert np.array_equal(idx, full.index[lo:hi])
    assert np.array_equal(np.sqrt(d2), full.distances[lo:hi])


@pytest.mark.parametrize("kind", ["mixture", "outlier"])
def test_pruned_search_of_either_operand_format(kind):
    """70,000 points: the pruned search with f16 (mixture) and BF16 (an outlier
    widens the range) operands, against the FP32 arm on sampled rows."""
    n, d, k = 70_000, 20, 15
    X = _points("mixture", n, d, 3)
    if kind == "outlier":
        X[7] = 1e6
    b = sc_gpu.knn_gaussian(X, k)
    assert sc_gpu.knn_last_stats()["clusters"] >= 16
    for lo in (0, 33_000, n - 500):
        idx, d2 = sc_gpu.knn_search(X, k, lo, lo + 500, precision=sc_gpu.KNN_FP32)
        assert np.array_equal(idx, b.index[lo:lo + 500])
        assert np.array_equal(np.sqrt(d2), b.distances[lo:lo + 500])


@pytest.mark.parametrize("d", [1, 4, 5, 31, 50, 62])
@pytest.mark.parametrize("n,k", [(2, 1), (64, 10), (65, 31), (129, 15), (200, 31), (4097, 31)])
def test_fp32_halves_against_fp64(n, d, k):
    """The FP32 arm splits the points at a whole tile (n around 64 and 128: an
    empty, a ragged and a full second half) and keeps 32 per half: its squared
    distances equal the FP64 search's within FP32 rounding (62 terms, 2^-18)."""
    X = _points("mixture", n, d, n + d)
    idx, d2 = sc_gpu.knn_search(X, k, 0, n, precision=sc_gpu.KNN_FP32)
    X64 = X.astype(np.float64)
    full = np.stack([((X64 - x) ** 2).sum(1) for x in X64])
    full[np.arange(n), np.arange(n)] = -1.0
    want = np.maximum(np.sort(full, axis=1)[:, :k + 1], 0.0)
    m = min(k + 1, n)
    assert np.array_equal(idx[:, 0], np.arange(n))
    assert np.all(np.isinf(d2[:, m:])) and np.all(idx[:, m:] == 0xFFFFFFFF)
    assert np.all(np.abs(d2[:, :m] - want[:, :m]) <= 2.0 ** -18 * want[:, :m] + 1e-30)


@pytest.mark.parametrize("n,d,k", [(640, 6, 15), (2000, 12, 15), (4099, 20, 24)])
def test_rows_that_fill_up_are_cut_back(n, d, k):
    """Groups of 64 consecutive points, later ones nearer to the group's centre:
    all near points of a query stand in the same half of a tile and the nearest
    come last, so a row fills up and is cut back again and again."""
    rng = np.random.Generator(np.random.PCG64(n + k))
    group, place = np.arange(n) // 64, np.arange(n) % 64
    u = rng.normal(size=(n, d))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    centres = rng.normal(size=(group[-1] + 1, d)) * 8.0
    X = (centres[group] + u * (4.0 - 3.0 * place / 64)[:, None]).astype(np.float32)
    a = sc_gpu.knn_gaussian(X, k, precision=sc_gpu.KNN_FP32)
    b = sc_gpu.knn_gaussian(X, k, precision=sc_gpu.KNN_BF16)
    assert np.array_equal(a.index, b.index)
    assert np.array_equal(a.distances.view(np.uint32), b.distances.view(np.uint32))


@pytest.mark.parametrize("n,d,k", [(1000, 30, 10), (9000, 17, 31), (45_000, 4, 8)])
def test_fp32_items_shared_by_blocks(n, d, k):
    """The FP32 arm's work items over the blocks: every item in parts, and (the
    largest) whole items between shared ones, also for a shard of the rows."""
    X = _points("mixture", n, d, n + d)
    a = sc_gpu.knn_gaussian(X, k, precision=sc_gpu.KNN_FP32)
    b = sc_gpu.knn_gaussian(X, k, precision=sc_gpu.KNN_BF16)
    assert np.array_equal(a.index, b.index)
    assert np.array_equal(a.distances.view(np.uint32), b.distances.view(np.uint32))
    lo, hi = n // 3, n // 3 + 300
    idx, d2 = sc_gpu.knn_search(X, k, lo, hi, precision=sc_gpu.KNN_FP32)
    assert np.array_equal(idx, a.index[lo:hi])
