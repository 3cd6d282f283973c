"""aggregate's row kernels at the sizes that pick them, bit for bit against the
CPU oracle: coarse rows of a warp, of a block's table, of dense accumulators
(few groups), and rows so long that several blocks share one."""
import numpy as np
import pytest

import oracle as O
import sc_gpu

pytestmark = pytest.mark.gpu


def _graph(n, m, seed, least=1):
    rng = np.random.Generator(np.random.PCG64(seed))
    src, dst = rng.integers(0, n, m).astype(np.uint64), rng.integers(0, n, m).astype(np.uint64)
    w = (rng.integers(least, 32, m) / 16.0).astype(np.float64)
    return src, dst, w


@pytest.mark.parametrize("n,m,groups,skew", [
    (3000, 20_000, 3, 0.0),          # three rows of thousands of entries
    (30_000, 300_000, 40, 0.0),      # about 15,000 entries a row: around one part
    (30_000, 300_000, 40, 0.9),      # one row of most entries, in many parts
    (40_000, 200_000, 12_288, 0.5),  # the most groups the dense accumulators take
    (40_000, 200_000, 12_289, 0.5),  # one more: tables and the sorted big row
    (40_000, 200_000, 39_999, 0.0),  # almost no merging: short rows only
    (600, 150_000, 300, 0.0),        # dense rows: every group beside every other
])
def test_rows_of_every_kind(n, m, groups, skew):
    src, dst, w = _graph(n, m, n + groups)
    rng = np.random.Generator(np.random.PCG64(groups))
    lab = rng.integers(0, groups, n)
    lab[: min(groups, n)] = np.arange(min(groups, n))  # every group occurs
    if skew:
        tail = np.arange(n) >= groups
        lab[tail & (rng.random(n) < skew)] = groups // 2
    lab = lab.astype(np.uint64)
    og = O.Graph.from_edges(n, src=src, dst=dst, w=w)
    gg = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)
    want, got = og.aggregate(lab), gg.aggregate(lab)
    a = want.arrays()
    ptr, nbr, ww = got.to_csr_parts()
    assert np.array_equal(a["ptr"], ptr) and np.array_equal(a["nbr"], nbr)
    assert np.array_equal(a["w"].view(np.uint32), ww.view(np.uint32))
    assert og.modularity(lab) == sc_gpu.modularity(gg, lab)
    assert np.array_equal(a["strength"].view(np.uint64), got.strengths().view(np.uint64))


@pytest.mark.parametrize("least", [1, 0])
@pytest.mark.parametrize("n,m,groups", [(16_000, 3_300_000, 13_000), (60_000, 3_300_000, 13_000)])
def test_many_entries_in_long_rows_are_sorted(n, m, groups, least):
    """More entries, most of them in long rows, than the tables are the faster for;
    with and without pairs of weight zero."""
    src, dst, w = _graph(n, m, n, least)
    lab = np.random.Generator(np.random.PCG64(m)).integers(0, groups, n)
    lab[:groups] = np.arange(groups)
    lab = lab.astype(np.uint64)
    og = O.Graph.from_edges(n, src=src, dst=dst, w=w)
    gg = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)
    a = og.aggregate(lab).arrays()
    ptr, nbr, ww = gg.aggregate(lab).to_csr_parts()
    assert np.array_equal(a["ptr"], ptr) and np.array_equal(a["nbr"], nbr)
    assert np.array_equal(a["w"].view(np.uint32), ww.view(np.uint32))


@pytest.mark.parametrize("communities", [1, 1023, 1024, 1025])
def test_few_and_many_communities(communities):
    """modularity and partition sums with the communities in shared memory and past them."""
    n = 5000
    src, dst, w = _graph(n, 40_000, communities)
    lab = (np.arange(n) * 7919 % communities).astype(np.uint64)
    og = O.Graph.from_edges(n, src=src, dst=dst, w=w)
    gg = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)
    assert og.modularity(lab) == sc_gpu.modularity(gg, lab)
    for obj in (sc_gpu.Rb(0.7), sc_gpu.Cpm(0.01)):
        kind = 0 if isinstance(obj, sc_gpu.Rb) else 1
        assert og.quality(lab, kind, obj.resolution) == sc_gpu.quality(gg, lab, obj)
