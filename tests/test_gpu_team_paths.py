"""Small levels and last sweeps by the team's kernels (sc_team.cu) against the same
run with a launch for every step: a team of 16 blocks, of 8, and none, which is
also what a device gets that cannot place the cluster. The labels are the same."""
import ctypes as C

import numpy as np
import pytest

import sc_gpu
from sc_gpu import _lib, synth

pytestmark = pytest.mark.gpu


class team_of:
    """The largest team of the context while the block runs."""

    def __init__(self, most):
        self.most = most

    def __enter__(self):
        assert _lib.lib().sc_test_team_cluster(sc_gpu.context(0).h, C.c_uint32(self.most)) == 0

    def __exit__(self, *exc):
        assert _lib.lib().sc_test_team_cluster(sc_gpu.context(0).h, C.c_uint32(16)) == 0


CONFIGS = {
    "rb": {},
    "cpm": {"objective": sc_gpu.Cpm(0.05)},
    "louvain": {"refine": False},
    "fine": {"objective": sc_gpu.Rb(3.0), "n_iterations": 3, "patience": 1},
    "one_level": {"max_levels": 1},
    "argmax": {"refine_randomness": 0.0},
}


def _planted(n, blocks, intra, inter, seed):
    src, dst, w, _ = synth.planted_partition(n, blocks, intra, inter, seed=seed)
    return sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)


def test_a_team_has_16_or_8_blocks_or_none():
    h = sc_gpu.context(0).h
    for most in (1, 4, 12, 32):
        assert _lib.lib().sc_test_team_cluster(h, C.c_uint32(most)) == 20  # SC_E_INVALID_ARGUMENT


@pytest.mark.parametrize("n", [64, 3000, 12_000])
def test_a_device_with_smaller_clusters_or_none(n):
    g = _planted(n, max(4, n // 200), 8, 2, n)
    cfg = sc_gpu.LeidenConfig(seed=n)
    launches, labels = {}, {}
    for most in (16, 8, 0):
        with team_of(most):
            c = sc_gpu.leiden(g, cfg)
            labels[most] = c.labels()
            launches[most] = sc_gpu.last_run_stats()["kernel_launches"]
            # beside each other on worker contexts, and as one union
            batch = sc_gpu.leiden_batch([g] * 3, [cfg] * 3) + sc_gpu.leiden_batch([g] * 3, [cfg] * 3, union=True)
        for b in batch:
            assert np.array_equal(b.labels(), labels[most])
    assert np.array_equal(labels[8], labels[16]) and np.array_equal(labels[0], labels[16])
    assert launches[0] > 2 * launches[16]  # without a team every step is a launch


def _same_without_a_team(run):
    """run(): a list of clusterings, the same ones with a launch for every step, which takes more of them."""
    got = run()
    used = sc_gpu.last_run_stats()["kernel_launches"]
    with team_of(0):
        want = run()
        assert sc_gpu.last_run_stats()["kernel_launches"] > used
    for a, b in zip(got, want):
        assert a.n_clusters() == b.n_clusters() and np.array_equal(a.labels(), b.labels())


def _leiden(graph, **fields):
    return lambda: [sc_gpu.leiden(graph, sc_gpu.LeidenConfig(**fields))]


@pytest.mark.parametrize("cfg", CONFIGS)
@pytest.mark.parametrize("n,blocks,intra,inter", [(6, 2, 1, 1), (64, 4, 4, 1), (65, 4, 4, 1), (512, 8, 6, 2),
                                                  (4095, 16, 8, 2), (8192, 40, 12, 3), (8193, 40, 12, 3)])
def test_node_counts(n, blocks, intra, inter, cfg):
    _same_without_a_team(_leiden(_planted(n, blocks, intra, inter, n), seed=n, **CONFIGS[cfg]))


def _regular(degree):
    """Rows of one length, neighbours at the nearest ids around a ring."""
    n = 2 * degree + 40
    node, half = np.arange(n), degree // 2
    src = np.concatenate([node] * half)
    dst = np.concatenate([(node + t + 1) % n for t in range(half)])
    if degree % 2:
        src, dst = np.concatenate([src, node[: n // 2]]), np.concatenate([dst, node[: n // 2] + n // 2])
    rng = np.random.Generator(np.random.PCG64(degree))
    w = rng.integers(1, 64, len(src)) / 16.0 + 8.0 * (src // 40 == dst // 40)
    return sc_gpu.CSRNetwork.from_edge_arrays(n, src.astype(np.uint64), dst.astype(np.uint64), w)


@pytest.mark.parametrize("cfg", ["rb", "cpm", "louvain"])
@pytest.mark.parametrize("degree", [31, 32, 33, 128, 255, 256, 257, 700])
def test_row_lengths(degree, cfg):
    """k_team's rows: one chunk, a warp's table up to its limit, a group's accumulators.
    The same graphs in a union: the tail's tables, from the first sweep on."""
    g = _regular(degree)
    c = sc_gpu.LeidenConfig(seed=degree, **CONFIGS[cfg])
    _same_without_a_team(lambda: [sc_gpu.leiden(g, c)])
    _same_without_a_team(lambda: sc_gpu.leiden_batch([g, g], [c, c], union=True))


def _with_hub(n, degree, seed):
    """A planted partition with node 0 joined to exactly `degree` others, near and far."""
    src, dst, w, _ = synth.planted_partition(n - 1, max(2, n // 150), 8, 2, seed=seed)
    far = 1 + np.random.Generator(np.random.PCG64(seed)).permutation(n - 1)[:degree]
    src = np.concatenate([src + np.uint64(1), np.zeros(degree, np.uint64)])
    dst = np.concatenate([dst + np.uint64(1), far.astype(np.uint64)])
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, np.concatenate([w, np.full(degree, 0.5)]))
    ptr = g.to_csr_parts()[0]
    assert ptr[1] - ptr[0] == degree == np.diff(ptr.astype(np.int64)).max()
    return g


@pytest.mark.parametrize("cfg", ["rb", "cpm", "louvain"])
@pytest.mark.parametrize("degree", [256, 257, 1024, 1025, 2048, 4095, 4096, 4097])
def test_hubs_of_every_table(degree, cfg):
    """A warp's table, a quarter of a block's, the whole block's up to its limit, and a
    row past it: in the last sweeps of a large level, and in a union of smaller
    graphs, whose first sweep is the tail's already."""
    c = sc_gpu.LeidenConfig(seed=degree, **CONFIGS[cfg])
    _same_without_a_team(lambda: [sc_gpu.leiden(_HUBS(20_000, degree), c)])
    small = _HUBS(5000, degree)
    _same_without_a_team(lambda: sc_gpu.leiden_batch([small], [c], union=True))


_built = {}


def _HUBS(n, degree):
    if (n, degree) not in _built:
        _built[n, degree] = _with_hub(n, degree, n + degree)
    return _built[n, degree]


@pytest.mark.parametrize("n", [1500, 5000])
@pytest.mark.parametrize("cfg", ["rb", "cpm"])
def test_loops_and_node_weights(n, cfg):
    rng = np.random.Generator(np.random.PCG64(n))
    src = np.concatenate([np.zeros(n - 1, int), rng.integers(0, n, 5 * n), np.arange(0, n, 11)])
    dst = np.concatenate([np.arange(1, n), rng.integers(0, n, 5 * n), np.arange(0, n, 11)])
    w = rng.integers(1, 16, len(src)) * 0.25 + 2.0 * (src % 13 == dst % 13)
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src.astype(np.uint64), dst.astype(np.uint64), w,
                                           node_weights=rng.integers(1, 8, n) * 0.5)
    _same_without_a_team(_leiden(g, seed=4, **CONFIGS[cfg]))


def test_unions_of_uneven_graphs():
    """Instances of different sizes, seeds, objectives and resolutions share sweeps."""
    rng = np.random.Generator(np.random.PCG64(8))
    for sizes in ([6, 64, 700, 2500], [100, 20_000, 900, 6000, 40]):
        graphs = [_planted(n, max(2, n // 100), 5, 2, n) for n in sizes]
        cfgs = [sc_gpu.LeidenConfig(objective=sc_gpu.Rb(float(r)), seed=int(s))
                for r, s in zip(rng.uniform(0.3, 2.5, len(sizes)), rng.integers(0, 99, len(sizes)))]
        _same_without_a_team(lambda: sc_gpu.leiden_batch(graphs, cfgs, union=True))


@pytest.mark.parametrize("cfg", ["rb", "cpm", "louvain"])
def test_long_runs_and_warm_starts(cfg):
    """60,000 nodes down: launches, the tail, then the team for the last levels."""
    X, truth = synth.gaussian_mixture(60_000, 20, 30, seed=2, sigma=(0.7, 1.5))
    g = sc_gpu.knn_gaussian(X, 12, sigma=sc_gpu.SIGMA_KTH, sym=sc_gpu.SYM_UNION, build_graph=True).graph
    _same_without_a_team(_leiden(g, seed=5, **CONFIGS[cfg]))
    c = sc_gpu.LeidenConfig(seed=6, **CONFIGS[cfg])
    _same_without_a_team(lambda: [sc_gpu.leiden_from(g, c, np.asarray(truth, np.uint64))])


TUNINGS = [
    dict(lanes8_max_degree=8, lanes16_max_degree=16, lanes32_max_degree=32, small_batch=4096),
    dict(lanes8_max_degree=0, lanes16_max_degree=0, lanes32_max_degree=0, small_batch=0),
    dict(lanes8_max_degree=0, lanes16_max_degree=16, lanes32_max_degree=16, small_batch=1 << 30),
    dict(lanes8_max_degree=8, lanes16_max_degree=8, lanes32_max_degree=32, small_batch=0),
]


@pytest.mark.parametrize("cfg", ["rb", "cpm", "louvain", "capped"])
def test_decide_kernels_agree_under_every_tuning(cfg):
    """With a launch for every step the tuned kernels decide every sweep: the labels
    are those of every routing and of the run with a team. Rows of every bucket: up
    to 8, 16 and 32 lanes, a warp, a block, a hub."""
    n = 12_000
    rng = np.random.Generator(np.random.PCG64(12))
    src, dst, w, _ = synth.planted_partition(n, 60, 3, 1, seed=12)
    parts = [(src.astype(np.int64), dst.astype(np.int64), w)]
    for node, degree in [(v, int(d)) for v, d in zip(range(0, 400, 2), rng.integers(9, 300, 200))] + \
            [(1001, 900), (2001, 1024), (3001, 1500), (4001, 3000)]:
        to = rng.permutation(n)[:degree]
        parts.append((np.full(degree, node), to, rng.integers(1, 8, degree) / 4.0))
    src, dst, w = (np.concatenate(p) for p in zip(*parts))
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src.astype(np.uint64), dst.astype(np.uint64), w)
    degree = np.diff(g.to_csr_parts()[0].astype(np.int64))
    edges = [0, 8, 16, 32, 256, 1024, n]
    assert all(((degree > a) & (degree <= b)).any() for a, b in zip(edges, edges[1:]))
    fields = {"max_community_weight": 40.0} if cfg == "capped" else CONFIGS[cfg]
    c = sc_gpu.LeidenConfig(seed=7, **fields)
    want = sc_gpu.leiden(g, c).labels()
    saved = sc_gpu.get_tuning()
    try:
        with team_of(0):
            for t in TUNINGS:
                sc_gpu.set_tuning(t)
                assert np.array_equal(sc_gpu.leiden(g, c).labels(), want), t
    finally:
        sc_gpu.set_tuning(saved)
