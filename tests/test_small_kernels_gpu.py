"""One-block kernels for small boxes (sort, scan, moments) at the sizes where
they take over from the many-block ones and at their own edges: keys and order
equal the oracle's, and the exported octree equals the one the insertion makes.
"""
import numpy as np
import pytest

from conftest import oracle

pytestmark = pytest.mark.gpu


def _box(n, seed):
    rng = np.random.default_rng(seed)
    q = rng.integers(0, 2 ** 32, (n, 3), dtype=np.uint64)
    k = n // 4  # a clump: deep levels, long runs of equal leading digits
    q[:k] = (2 ** 31 + rng.integers(0, 2 ** 20, (k, 3), dtype=np.uint64)) & np.uint64(0xFFFFFFFF)
    return np.unique(q, axis=0).astype(np.float64) * (64.0 / 2.0 ** 32)


@pytest.mark.parametrize("n", [2, 31, 33, 1024, 1025, 2049, 4097, 8192, 8200, 16390, 24000])
def test_tree_of_a_small_box_matches_the_insertion_octree(n):
    import treepm
    pos = _box(n, n)
    m = len(pos)
    mass = np.random.default_rng(n).uniform(0.5, 1.5, m)
    s = treepm.TreePmSolver(16, 64.0, 5.0)
    s.set_particles(pos, mass)
    s.compute_forces(1e-3, 1.0)
    got = s.export_tree()
    keys, order = s.hilbert_keys(m)
    counts = s.interaction_counts(m)
    s.close()
    ref_keys, ref_order = oracle().hilbert_keys(pos)
    assert np.array_equal(keys, ref_keys) and np.array_equal(order, ref_order)
    ref = oracle().octree(pos, mass)
    live = ref["mass"] > 0.0  # the insertion also creates empty children
    a = np.lexsort((got["mass"], got["com"][:, 2], got["com"][:, 1], got["com"][:, 0], got["depth"]))
    rm, rc, rd = ref["mass"][live], ref["com"][live], ref["depth"][live]
    b = np.lexsort((rm, rc[:, 2], rc[:, 1], rc[:, 0], rd))
    assert np.array_equal(got["depth"][a], rd[b])
    assert np.array_equal(got["mass"][a], rm[b])
    assert np.array_equal(got["com"][a], rc[b])
    _, ref_counts = oracle().short_range(pos, mass, 1e-3, 1.0, 5.0, 25.0, 64.0, counts=True)
    assert np.array_equal(counts, ref_counts)
