"""The short-range walk where its dispatch and its packed loops can go wrong:
particle counts around the group sizes, lists of odd length, groups split at
cells, periodic images inside a group's reach, a cut beyond the fitted erfc
polynomial, a root that is a monopole itself.

The interaction set must equal the oracle's particle by particle; the
short-range forces agree within 1e-5 of their rms (FP32 pair terms: 24-bit
positions relative to a group of a quarter box at most, 2.8 r_cut, and the
erfc polynomial's 7e-8, summed over hundreds of pairs).
"""
import numpy as np
import pytest

from conftest import oracle

pytestmark = pytest.mark.gpu


def _positions(kind, n, box, seed):
    """float64 positions on the device's fixed-point lattice."""
    rng = np.random.default_rng(seed)
    if kind == "uniform":
        x = rng.uniform(0.0, box, (n, 3))
    elif kind == "lattice":
        side = int(np.ceil(n ** (1.0 / 3.0)))
        g = (np.indices((side,) * 3).reshape(3, -1).T + 0.5) * (box / side)
        x = g[:n] + rng.normal(0.0, 0.3 * box / side, (n, 3))
    elif kind == "clump":  # everything inside one terminal cell, across the corner of the box
        x = rng.normal(0.0, 2e-4 * box, (n, 3))
    elif kind == "middle":  # half of the particles in a clump, the others far apart: leaves in wide cells
        x = rng.uniform(0.0, box, (n, 3))
        x[: n // 2] = 0.5 * box + rng.normal(0.0, 5e-3 * box, (n // 2, 3))
    elif kind == "corner":  # half of the particles in a clump near a corner: nodes more than half a box away
        x = rng.uniform(0.0, box, (n, 3))
        x[: n // 2] = 0.95 * box + rng.normal(0.0, 1e-2 * box, (n // 2, 3))
    else:  # two dense clumps on a sparse background
        x = rng.uniform(0.0, box, (n, 3))
        k = n // 3
        x[:k] = 0.27 * box + rng.normal(0.0, 4e-3 * box, (k, 3))
        x[k:2 * k] = 0.97 * box + rng.normal(0.0, 2e-2 * box, (k, 3))
    q = np.floor(np.mod(x / box, 1.0) * 2.0 ** 32).astype(np.uint64) & np.uint64(0xFFFFFFFF)
    return q.astype(np.float64) * (box / 2.0 ** 32)


CASES = [
    # kind, n, mesh, r_split cells, r_cut factor, periodic
    ("uniform", 2, 32, 1.25, 4.5, True),
    ("uniform", 3, 32, 2.5, 5.0, True),
    ("uniform", 33, 16, 1.25, 4.5, True),
    ("uniform", 500, 16, 2.5, 6.0, True),  # r_cut close to the box: targets alone, the A&S erfc
    ("uniform", 1000, 32, 2.5, 5.0, True),  # r_cut above a fifth of the box
    ("uniform", 3399, 32, 1.25, 4.5, True),  # one target per group
    ("uniform", 3401, 32, 1.25, 4.5, True),  # two
    ("lattice", 13599, 32, 1.25, 4.5, True),
    ("lattice", 13601, 32, 1.25, 6.0, True),  # the A&S erfc with groups
    ("lattice", 27201, 32, 1.25, 4.5, True),  # groups of a quarter box: images inside their reach
    ("lattice", 54401, 64, 2.5, 5.0, True),
    ("clumps", 30000, 64, 1.25, 4.5, True),
    ("clumps", 60000, 128, 1.25, 5.0, True),
    ("clump", 400, 16, 1.25, 4.5, True),  # the root is terminal
    ("lattice", 13824, 32, 1.25, 4.5, False),
    ("lattice", 29791, 32, 1.25, 6.0, False),
    ("lattice", 59319, 64, 2.5, 5.0, False),
    ("lattice", 131071, 64, 1.25, 4.5, True),  # the last with exact near pairs, in groups wider than L/16
    ("lattice", 131072, 64, 1.25, 4.5, True),
    ("corner", 600, 32, 1.25, 5.0, False),  # boxes that corner targets do not open at all
    ("corner", 1500, 32, 1.25, 5.0, False),
    ("corner", 8000, 32, 1.25, 4.5, False),
    ("corner", 40000, 64, 2.5, 5.0, False),
    ("clumps", 30000, 64, 1.25, 4.5, False),
]


@pytest.mark.parametrize("kind,n,mesh,cells,factor,periodic", CASES)
def test_interactions_and_forces_match_the_oracle(kind, n, mesh, cells, factor, periodic):
    import treepm
    box = 50.0
    pos = _positions(kind, n, box, n + mesh)
    mass = np.random.default_rng(n).uniform(0.5, 1.5, n) / n
    r_split = cells * box / mesh
    eps2, g = (box / max(n, 8) ** (1.0 / 3.0) / 30.0) ** 2, 1.7
    s = treepm.TreePmSolver(mesh, box, r_split, r_cut_factor=factor, periodic_walk=periodic)
    s.set_particles(pos, mass)
    s.compute_forces(eps2, g)
    _, sr = s.force_parts(n)
    counts = s.interaction_counts(n)
    stats = s.stats()
    s.close()
    ref, ref_counts = oracle().short_range(pos, mass, eps2, g, r_split, factor * r_split, box, periodic=periodic,
                                           counts=True)
    assert np.array_equal(counts, ref_counts)
    assert stats["leaf_pairs"] + stats["monopoles"] == int(ref_counts.sum())
    scale = np.sqrt(np.mean(np.sum(ref ** 2, axis=1)))
    if scale > 0.0:
        assert np.sqrt(np.mean(np.sum((sr - ref) ** 2, axis=1))) < 1e-5 * scale
    else:
        assert not sr.any()


# Pairs far beyond the range that the erfc polynomial is fitted on: leaves of the
# aperiodic walk in wide cells (cut on the gap to the cell), and a softening that
# is longer than r_cut.
FAR = [
    # kind, n, mesh, r_split cells, r_cut factor, periodic, softening / r_cut
    ("uniform", 10, 64, 2.5, 1.0, False, 0.0),
    ("uniform", 10, 64, 2.5, 2.0, False, 0.0),
    ("uniform", 10, 64, 2.5, 3.0, False, 0.0),
    ("middle", 1000, 128, 1.25, 1.0, False, 0.05),
    ("middle", 1000, 128, 1.25, 2.0, False, 0.05),
    ("middle", 1000, 128, 1.25, 3.0, False, 0.05),
    ("middle", 1000, 128, 1.25, 3.5, False, 0.05),
    ("middle", 1000, 128, 1.25, 3.6, False, 0.05),
    ("middle", 1000, 128, 1.25, 3.65, False, 0.05),
    ("middle", 1000, 128, 1.25, 5.0, False, 0.05),
    ("middle", 1000, 32, 1.25, 1.0, True, 0.05),
    ("middle", 1000, 32, 1.25, 2.0, True, 0.0),
    ("middle", 1000, 32, 1.25, 2.0, True, 1.5),
    ("middle", 1000, 32, 1.25, 3.0, True, 4.0),
    ("middle", 1000, 32, 1.25, 4.5, True, 4.0),
    ("middle", 1000, 64, 1.25, 2.0, False, 4.0),
]


@pytest.mark.parametrize("kind,n,mesh,cells,factor,periodic,soft", FAR)
def test_each_particle_matches_the_oracle_beyond_the_fitted_range(kind, n, mesh, cells, factor, periodic, soft):
    """Per particle: 1e-6 of erfc (the A&S form in FP32 is off by 4e-7, the
    polynomial by 1e-7) times the sum of m / r^2, and 1e-5 of the sum of the
    pair forces (distances are rounded relative to a group, as above)."""
    import treepm
    from scipy.special import erfc
    box, g = 50.0, 1.7
    pos = _positions(kind, n, box, n + mesh)
    mass = np.random.default_rng(n).uniform(0.5, 1.5, n) / n
    r_split = cells * box / mesh
    eps2 = (soft * factor * r_split) ** 2
    s = treepm.TreePmSolver(mesh, box, r_split, r_cut_factor=factor, periodic_walk=periodic)
    s.set_particles(pos, mass)
    s.compute_forces(eps2, g)
    _, sr = s.force_parts(n)
    counts = s.interaction_counts(n)
    s.close()
    ref, ref_counts = oracle().short_range(pos, mass, eps2, g, r_split, factor * r_split, box, periodic=periodic,
                                           counts=True)
    assert np.array_equal(counts, ref_counts)
    d = pos[None] - pos[:, None]
    if periodic:
        d -= box * np.round(d / box)
    r2 = np.sum(d * d, axis=2) + eps2
    np.fill_diagonal(r2, np.inf)
    w = erfc(np.sqrt(r2) / (np.sqrt(2.0) * r_split))
    allowed = g * np.sum(mass[None] / r2 * (1e-6 + 1e-5 * w), axis=1)
    assert np.isfinite(sr).all()
    assert (np.linalg.norm(sr - ref, axis=1) <= allowed).all()


@pytest.mark.parametrize("n,mesh,periodic,accurate", [(13600, 16, True, False), (20000, 32, True, False),
                                                      (30000, 32, True, False), (30000, 32, False, False),
                                                      (60000, 32, True, False), (20000, 32, True, True),
                                                      (60000, 32, True, True)])
def test_tight_pairs_in_wide_groups_keep_their_bits(n, mesh, periodic, accurate):
    """Pairs far closer than their group is wide, nearly unsoftened: a position
    relative to a group of up to L/4 is off by 2^-25 L/8, a pair at L/64 (a
    sixteenth of the extent) then by 5e-7 per coordinate, 3.3e-6 in its force;
    nearer ones take exact differences.  erfc as in the test above.  The parity
    walk meets a pair alone in its cell as a centre of mass: twice the mass at half
    the distance (8 times the force), rounded to quanta (2e-10 L of the 5e-5 L or
    more between it and a particle: 8e-6 in the force)."""
    import treepm
    from scipy.special import erfc
    box, g = 50.0, 1.7
    pos = _positions("lattice", n, box, n)
    rng = np.random.default_rng(n + 1)
    k = 60  # the first particle of each pair stays, the second goes beside it
    which = rng.choice(n, 2 * k, replace=False)
    step = rng.normal(0.0, 1.0, (k, 3))
    step *= (box * 10.0 ** rng.uniform(-4.0, -3.0, k) / np.linalg.norm(step, axis=1))[:, None]
    q = np.floor(np.mod((pos[which[:k]] + step) / box, 1.0) * 2.0 ** 32)
    pos[which[k:]] = q * (box / 2.0 ** 32)
    mass = np.full(n, 1.0 / n)
    r_split, factor, eps2 = 1.25 * box / mesh, 4.5, (3e-6 * box) ** 2
    s = treepm.TreePmSolver(mesh, box, r_split, r_cut_factor=factor, periodic_walk=periodic, accurate=accurate,
                            theta=0.01 if accurate else 0.5)
    s.set_particles(pos, mass)
    s.compute_forces(eps2, g)
    _, sr = s.force_parts(n)
    s.close()
    d = pos[None] - pos[which][:, None]
    if periodic:
        d -= box * np.round(d / box)
    r2 = np.sum(d * d, axis=2)
    cut = r2 > (factor * r_split) ** 2
    r2 += eps2
    r2[np.arange(2 * k), which] = np.inf
    x = np.sqrt(r2) / (np.sqrt(2.0) * r_split)
    w = erfc(x)
    if accurate:
        w += np.where(np.isinf(x), 0.0, 2.0 / np.sqrt(np.pi) * x) * np.exp(-x * x)
        f = np.where(cut, 0.0, w) * mass[None] / r2 ** 1.5
        f[np.isinf(r2)] = 0.0
        ref = g * np.einsum("ijk,ij->ik", d, f)
    else:
        ref = oracle().short_range(pos, mass, eps2, g, r_split, factor * r_split, box, periodic=periodic)[which]
    allowed = g * np.sum(mass[None] / r2 * (1e-6 + (3.3e-6 if accurate else 8 * 1.13e-5) * w), axis=1)
    assert (np.linalg.norm(sr[which] - ref, axis=1) <= allowed).all()


@pytest.mark.parametrize("n,periodic", [(31, True), (700, True), (2100, True), (700, False)])
def test_accurate_mode_sums_the_complete_kernel(n, periodic):
    """A small opening angle leaves (nearly) only particle pairs: the direct
    sum of the complete split kernel inside r_cut."""
    import treepm
    from scipy.special import erfc
    box, mesh = 50.0, 32
    pos = _positions("uniform", n, box, n)
    mass = np.full(n, 1.0 / n)
    r_split, factor, eps2 = 1.25 * box / mesh, 4.5, 1e-3
    s = treepm.TreePmSolver(mesh, box, r_split, r_cut_factor=factor, periodic_walk=periodic, accurate=True, theta=0.01)
    s.set_particles(pos, mass)
    s.compute_forces(eps2, 1.0)
    _, sr = s.force_parts(n)
    s.close()
    d = pos[None] - pos[:, None]
    if periodic:
        d -= box * np.round(d / box)
    r2 = np.sum(d * d, axis=2)
    x = np.sqrt(r2 + eps2) / (np.sqrt(2.0) * r_split)
    w = (erfc(x) + 2.0 / np.sqrt(np.pi) * x * np.exp(-x * x)) / (r2 + eps2) ** 1.5
    w[(r2 > (factor * r_split) ** 2) & np.array(periodic)] = 0.0
    np.fill_diagonal(w, 0.0)
    ref = np.einsum("ijk,ij->ik", d, w) / n
    # the aperiodic walk cuts leaves on the gap to their cell: terms between
    # r_cut and r_cut + sqrt(3) cells stay, all below w(4.5 r_s) ~ 1e-3 of a pair at r_s
    tol = 1e-5 if periodic else 2e-3
    assert np.linalg.norm(sr - ref) < tol * np.linalg.norm(ref)
