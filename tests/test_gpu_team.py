"""The levels that one launch runs (sc_team.cu) against the general path, which a
batched union of one instance always takes: the same labels, at the edges of the
node counts, row lengths and id ranges that pick a kernel's branches."""
import numpy as np
import pytest

import sc_gpu
from sc_gpu import synth

pytestmark = pytest.mark.gpu


def _check(graph, **fields):
    cfg = sc_gpu.LeidenConfig(**fields)
    want = sc_gpu.leiden_batch([graph], [cfg], union=True)[0]
    got = sc_gpu.leiden(graph, cfg)
    assert got.n_clusters() == want.n_clusters()
    assert np.array_equal(got.labels(), want.labels())


CONFIGS = {
    "rb": {},
    "cpm": {"objective": sc_gpu.Cpm(0.05)},
    "louvain": {"refine": False},
    "fine": {"objective": sc_gpu.Rb(3.0), "n_iterations": 3, "patience": 1},
    "one_level": {"max_levels": 1},
    "argmax": {"refine_randomness": 0.0},
}


@pytest.mark.parametrize("cfg", CONFIGS)
@pytest.mark.parametrize("n,blocks,intra,inter", [(6, 2, 1, 1), (64, 4, 4, 1), (65, 4, 4, 1), (512, 8, 6, 2),
                                                  (4095, 16, 8, 2), (8192, 40, 12, 3), (8193, 40, 12, 3)])
def test_node_count_edges(n, blocks, intra, inter, cfg):
    src, dst, w, _ = synth.planted_partition(n, blocks, intra, inter, seed=n)
    _check(sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w), seed=n, **CONFIGS[cfg])


@pytest.mark.parametrize("cfg", ["rb", "cpm", "louvain"])
@pytest.mark.parametrize("degree", [31, 32, 33, 128, 255, 256, 257, 700])
def test_row_length_edges(degree, cfg):
    """Regular rows of one length: a single chunk, a warp's table and its limit,
    a group's accumulators."""
    n = 2 * degree + 40
    node = np.arange(n)
    half = degree // 2
    src = np.concatenate([node] * half)
    dst = np.concatenate([(node + t + 1) % n for t in range(half)])
    if degree % 2 and n % 2 == 0:
        src = np.concatenate([src, node[: n // 2]])
        dst = np.concatenate([dst, node[: n // 2] + n // 2])
    rng = np.random.Generator(np.random.PCG64(degree))
    w = rng.integers(1, 64, len(src)) / 16.0 + 8.0 * (src // 40 == dst // 40)
    _check(sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w), seed=degree, **CONFIGS[cfg])


@pytest.mark.parametrize("n", [1500, 5000])  # ids within a quarter of the accumulators, and beyond
@pytest.mark.parametrize("cfg", ["rb", "cpm"])
def test_hubs_loops_and_node_weights(n, cfg):
    rng = np.random.Generator(np.random.PCG64(n))
    src = np.concatenate([np.zeros(n - 1, int), rng.integers(0, n, 5 * n), np.arange(0, n, 11)])
    dst = np.concatenate([np.arange(1, n), rng.integers(0, n, 5 * n), np.arange(0, n, 11)])
    w = rng.integers(1, 16, len(src)) * 0.25 + 2.0 * (src % 13 == dst % 13)
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w, node_weights=rng.integers(1, 8, n) * 0.5)
    _check(g, seed=4, **CONFIGS[cfg])


def test_no_edges_and_one_node():
    for n in (1, 3, 700):
        g = sc_gpu.CSRNetwork.from_edge_arrays(n, np.zeros(0), np.zeros(0), np.zeros(0))
        assert sc_gpu.leiden(g, sc_gpu.LeidenConfig()).n_clusters() == n


def test_warm_start_labels():
    n = 2000
    src, dst, w, truth = synth.planted_partition(n, 20, 8, 2, seed=3)
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)
    for start in (truth, np.zeros(n, np.uint64), np.arange(n, dtype=np.uint64)[::-1] * 7):
        cfg = sc_gpu.LeidenConfig(seed=2, n_iterations=1)
        got = sc_gpu.leiden_from(g, cfg, start)
        assert got.n_clusters() == 20 and len(np.unique(got.labels())) == 20


def test_a_long_run_ends_in_the_team():
    """Levels of 60,000 nodes down: the general path hands its last levels over."""
    X, _ = synth.gaussian_mixture(60_000, 20, 30, seed=2, sigma=(0.7, 1.5))
    g = sc_gpu.knn_gaussian(X, 12, sigma=sc_gpu.SIGMA_KTH, sym=sc_gpu.SYM_UNION, build_graph=True).graph
    for f in ("rb", "cpm", "louvain"):
        _check(g, seed=5, **CONFIGS[f])


@pytest.mark.parametrize("cfg", ["rb", "cpm", "louvain"])
@pytest.mark.parametrize("n,hub", [(9000, 0), (40_000, 1500), (40_000, 4096), (40_000, 4097), (40_000, 9000)])
def test_last_sweeps_of_larger_levels(n, hub, cfg):
    """The last sweeps run on the team: rows of a warp, a quarter of a block, a
    block (a hub of 1,500 to 4,096 entries), and a hub past what it takes. The
    same graph in a batch of two goes through the instances' form of the kernel."""
    src, dst, w, _ = synth.planted_partition(n, 60, 8, 2, seed=n + hub)
    if hub:
        src = np.concatenate([src, np.zeros(hub, np.uint64)])
        dst = np.concatenate([dst, 1 + np.arange(hub, dtype=np.uint64)])
        w = np.concatenate([w, np.full(hub, 0.5)])
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)
    c = sc_gpu.LeidenConfig(seed=hub, **CONFIGS[cfg])
    saved = sc_gpu.get_tuning()
    want = sc_gpu.leiden(g, c)
    two = sc_gpu.leiden_batch([g, g], [c, c], union=True)
    for r in two:
        assert np.array_equal(r.labels(), want.labels())
    sc_gpu.set_tuning({**saved, "small_batch": 0, "lanes32_max_degree": 16})
    try:
        assert np.array_equal(sc_gpu.leiden(g, c).labels(), want.labels())
    finally:
        sc_gpu.set_tuning(saved)
