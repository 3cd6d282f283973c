"""Scratch of an aggregation into few groups whose rows are long: beside the coarse
entries (8 bytes an entry of the graph) and the result, the accumulators of the
rows that several blocks share take 128 MB at most, however many such rows there are."""
import numpy as np
import pytest

import sc_gpu

pytestmark = pytest.mark.gpu


def _pool():
    from cuda.bindings import runtime as rt
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert int(err) == 0
    return rt, pool


def _used_and_reset_high():
    from cuda.bindings import driver
    rt, pool = _pool()
    rt.cudaDeviceSynchronize()
    err, used = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    assert int(err) == 0
    assert int(rt.cudaMemPoolSetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh,
                                          driver.cuuint64_t(0))[0]) == 0
    return int(used)


def _high():
    rt, pool = _pool()
    rt.cudaDeviceSynchronize()
    err, high = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh)
    assert int(err) == 0
    return int(high)


def test_accumulators_of_shared_rows_are_bounded():
    groups, long_rows, n, m = 12_288, 2740, 200_000, 23_500_000
    rng = np.random.Generator(np.random.PCG64(2))
    lab = np.arange(n) % long_rows       # long rows: 73 nodes of 235 entries each
    lab[-(groups - long_rows):] = np.arange(long_rows, groups)  # and a node a group
    inner = n - (groups - long_rows)
    src, dst = rng.integers(0, inner, m).astype(np.uint64), rng.integers(0, inner, m).astype(np.uint64)
    w = (rng.integers(1, 16, m) / 16.0).astype(np.float64)
    g = sc_gpu.CSRNetwork.from_edge_arrays(n, src, dst, w)
    ptr = g.to_csr_parts()[0].astype(np.int64)
    entries = int(ptr[-1])
    per_row = np.bincount(lab, np.diff(ptr), groups)
    assert (per_row > 16_384).sum() > 2600  # accumulators of 98,304 bytes each, were all of them shared
    lab = lab.astype(np.uint64)
    before = _used_and_reset_high()
    a = g.aggregate(lab)
    peak = _high() - before
    p2, nbr2, _ = a.to_csr_parts()
    known = 8 * entries + 12 * len(nbr2)
    assert peak <= known + (128 << 20) + (40 << 20), (peak, known)
    assert np.array_equal(a.strengths(), np.bincount(lab.astype(np.int64), g.strengths(), groups))
