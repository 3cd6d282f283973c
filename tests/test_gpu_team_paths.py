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
