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


@pytest.mark.parametrize("accurate", [False, True])
def test_a_refused_run_of_ties_makes_no_tree(accurate):
    """More than 16,384 particles in one cell of level 21 are refused, and neither a
    tree nor a walk is made of their keys, which are in no order.  The handle goes on."""
    import treepm
    rng = np.random.default_rng(9)
    # corners first, so the root cube is known: its level-21 cells are 2048.002
    # quanta wide, with a face at its centre
    q = 2 ** 31 + 21504 + np.unique(rng.integers(-256, 256, (20000, 3)), axis=0)
    q = np.concatenate([[[0, 0, 0], [2 ** 32 - 1] * 3], q])
    n = len(q)
    assert n > 17000
    pos = q.astype(np.float64) * (64.0 / 2.0 ** 32)
    s = treepm.TreePmSolver(16, 64.0, 5.0, accurate=accurate)
    s.set_particles(pos, np.full(n, 1.0 / n))
    for _ in range(2):
        with pytest.raises(treepm.TreePmError) as e:
            s.compute_forces(1e-3, 1.0)
        assert e.value.code == 4
        with pytest.raises(treepm.TreePmError):
            s.export_tree()
    pos = _box(5000, 3)
    s.set_particles(pos, np.full(len(pos), 1.0 / len(pos)))
    s.compute_forces(1e-3, 1.0)
    assert len(s.export_tree()["mass"]) > len(pos) and np.isfinite(s.get_state(len(pos))[2]).all()
    s.close()


def test_new_particles_have_no_tree():
    """The tree of an evaluation goes with its particles: its arrays are sized for them."""
    import treepm
    s = treepm.TreePmSolver(16, 64.0, 5.0)
    for seed, n in ((1, 500), (2, 300), (3, 5000)):  # fewer, then more than the capacity
        pos = _box(n, seed)
        s.set_particles(pos, np.full(len(pos), 1.0 / len(pos)))
        with pytest.raises(treepm.TreePmError):
            s.export_tree()
        s.compute_forces(1e-3, 1.0)
        assert np.sort(s.export_tree()["particle"])[-len(pos):].tolist() == list(range(len(pos)))
    s.close()
