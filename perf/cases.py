"""Performance cases of the TreePM library: what its users have it do.

A case names one call (or a short loop of calls) through the public Python
API, with the sizes and options it runs at.  The kinds are

* ``trait``: ``accelerations_for_indices``, the GravitySolver call that an
  integrator makes with its host arrays (pinned) every force evaluation, on
  the periodic or the aperiodic walk, for all particles or a rank's share;
* ``pm``: the same call on the plain PM solver;
* ``accurate``: the same call on the accurate short range (opening angle or
  the relative criterion);
* ``learned``: the same call with the committed network attached;
* ``steps``: a device-resident leapfrog loop with its in-situ power spectrum
  and the state read back, as a run does between two outputs;
* ``host_steps``: one ``kdk_step_host`` on the state that the previous call
  returned, the drop-in for the reference's leapfrog step;
* ``gradient``: the network's loss and parameter gradients on one batch of
  training patches.

``exact`` evaluates the same quantities in float64 with plain torch: the
insertion octree level by level, the walk's pair list per target breadth
first, the spectral Poisson solve on the full complex mesh, the network by
shifted matrix products and torch's autograd.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "gadget-ng_b200"))

TWO32 = float(1 << 32)
CELL = 0.78125  # mean interparticle spacing of the benchmark boxes in Mpc/h (200 / 256)
OMEGA_M, COUPLING_A = 0.31, 0.1
DT = 5e-6  # a step well inside the dynamical time of the halo cores, so that a state keeps its shape over many passes


# ---- the cases ------------------------------------------------------------------

def listed():
    return [
        # the reference's own committed TreePM run: 1000 particles on a 32^3 mesh,
        # default split scale and cut; a call of a small run is latency
        dict(name="trait_eds_n1000", kind="trait", side=10, drop=0, mesh=32, spacing=0.1, rms=0.1, halos=0.0,
             r_split_cells=0.0, r_cut_factor=5.0, periodic=True, share=1),
        # plain PM gravity of a 64^3 box with the 4-point gradient
        dict(name="pm_64_four_point", kind="pm", side=64, drop=0, mesh=64, spacing=100.0 / 64, rms=0.2, halos=0.0,
             four_point=True, deconvolve=False, share=1),
        # plain PM on a mesh twice as fine as the particle lattice
        dict(name="pm_128_mesh256", kind="pm", side=128, drop=0, mesh=256, spacing=CELL, rms=1.0, halos=0.0,
             four_point=False, deconvolve=False, share=1),
        # a small device-resident run between two outputs
        dict(name="steps_32", kind="steps", side=32, drop=0, mesh=32, spacing=CELL, rms=1.0, halos=0.0,
             r_split_cells=1.25, r_cut_factor=4.5, steps=4),
        # the trait-level aperiodic solver on a ragged clustered box, for one rank's third of the particles
        dict(name="trait_aperiodic_61", kind="trait", side=61, drop=13, mesh=64, spacing=CELL, rms=1.0, halos=0.3,
             r_split_cells=1.25, r_cut_factor=4.5, periodic=False, share=3),
        # TreePM force evaluations of lattice boxes at the benchmark's density
        dict(name="trait_64", kind="trait", side=64, drop=0, mesh=64, spacing=CELL, rms=1.0, halos=0.0,
             r_split_cells=1.25, r_cut_factor=4.5, periodic=True, share=1),
        dict(name="trait_128", kind="trait", side=128, drop=0, mesh=128, spacing=CELL, rms=1.0, halos=0.0,
             r_split_cells=1.25, r_cut_factor=4.5, periodic=True, share=1),
        # the reference's default split scale (2.5 cells) and cut (5 r_s) on a clustered box of an odd size
        dict(name="trait_default_split_99", kind="trait", side=99, drop=2, mesh=128, spacing=CELL, rms=1.0, halos=0.3,
             r_split_cells=0.0, r_cut_factor=5.0, periodic=True, share=1),
        # the headline workload, driven from host buffers
        dict(name="host_steps_clustered_256", kind="host_steps", side=256, drop=0, mesh=256, spacing=CELL, rms=1.0,
             halos=0.3, r_split_cells=1.25, r_cut_factor=4.5),
        # the accurate short range, both opening criteria
        dict(name="accurate_128", kind="accurate", side=128, drop=0, mesh=128, spacing=CELL, rms=1.0, halos=0.3,
             r_split_cells=1.25, r_cut_factor=4.5, theta=0.5, relative=False, err_tol=0.005, share=1),
        # the learned short range with the committed network
        dict(name="learned_128", kind="learned", side=128, drop=0, mesh=128, spacing=CELL, rms=1.0, halos=0.3,
             r_split_cells=1.25, r_cut_factor=4.5, theta=0.5, share=1),
        # forward and backward of one training batch of the network
        dict(name="gradient_64", kind="gradient", batch=64, width=14, c_in=10, per_volume=300),
    ]


def _near_power(side, factor, lo, hi):
    m = 2 ** round(math.log2(max(side * factor, 1.0)))
    return int(min(max(m, lo), hi))


def draw(rng):
    kind = rng.choice(["trait", "trait", "trait", "aperiodic", "pm", "steps", "host_steps", "accurate", "relative",
                       "learned", "gradient"])
    if kind == "gradient":
        return dict(kind="gradient", batch=rng.randint(3, 96), width=rng.choice([10, 14, 14, 17, 20]), c_in=10,
                    per_volume=rng.randint(40, 500))
    top = {"trait": 190, "aperiodic": 130, "pm": 230, "steps": 100, "host_steps": 210, "accurate": 140,
           "relative": 100, "learned": 140}[kind]
    side = int(round(math.exp(rng.uniform(math.log(9), math.log(top)))))
    c = dict(side=side, drop=rng.randint(0, side), mesh=_near_power(side, rng.choice([0.7, 1.0, 1.0, 1.4]), 16, 256),
             spacing=CELL, rms=round(rng.uniform(0.2, 1.2), 3), halos=rng.choice([0.0, 0.0, 0.2, 0.3]))
    if kind == "pm":
        return dict(c, kind="pm", four_point=rng.random() < 0.5, deconvolve=rng.random() < 0.5,
                    share=rng.choice([1, 2, 5]))
    split = rng.choice([1.25, 1.25, 2.0])
    if kind in ("trait", "aperiodic") and side <= 100 and rng.random() < 0.3:
        split = 0.0  # the reference's default of 2.5 cells
    if split != 1.25:
        c["mesh"] = max(c["mesh"], 32)  # r_cut stays below half the box
    c.update(r_split_cells=split, r_cut_factor=rng.choice([4.5, 5.0]))
    if kind in ("trait", "aperiodic"):
        return dict(c, kind="trait", periodic=kind == "trait", share=rng.choice([1, 1, 2, 7]))
    if kind == "steps":
        return dict(c, kind="steps", steps=rng.randint(2, 6))
    if kind == "host_steps":
        return dict(c, kind="host_steps")
    c.update(r_split_cells=1.25, r_cut_factor=4.5, theta=rng.choice([0.4, 0.5, 0.55]),
             mesh=_near_power(side, 1.0, 16, 256))
    if kind == "learned":
        return dict(c, kind="learned", theta=0.5, halos=0.3, share=1)
    return dict(c, kind="accurate", relative=kind == "relative", err_tol=rng.choice([0.005, 0.02]),
                share=rng.choice([1, 3]))


# ---- inputs -----------------------------------------------------------------------

def _count(c):
    return c["side"] ** 3 - c["drop"]


def _box(c):
    return c["side"] * c["spacing"]


def _positions(c, seed):
    """Fixed-point positions (n, 3) as int64 on the GPU: a lattice displaced by
    a Gaussian field with P(k) ~ k^-2 exp(-(k / k_Ny)^2) (rms in cells), a
    fraction `halos` of the particles in Plummer spheres of log-uniform mass."""
    dev, side, box = "cuda", c["side"], _box(c)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 7919 + 17)
    n = side ** 3
    white = torch.randn((side, side, side), generator=gen, device=dev, dtype=torch.float64)
    k = torch.fft.fftfreq(side, device=dev, dtype=torch.float64) * side
    kz = torch.fft.rfftfreq(side, device=dev, dtype=torch.float64) * side
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    inv = torch.where(k2 > 0, 1.0 / k2.clamp(min=1e-30), torch.zeros_like(k2))
    dk = torch.fft.rfftn(white) * torch.sqrt(inv * torch.exp(-k2 / (side / 2.0) ** 2))
    disp = torch.stack([torch.fft.irfftn(1j * ka * inv * dk, s=(side, side, side)).reshape(-1)
                        for ka in (k[:, None, None], k[None, :, None], kz[None, None, :])], dim=1)
    disp *= c["rms"] * c["spacing"] / torch.sqrt((disp * disp).sum(1).mean())
    g = (torch.arange(side, device=dev, dtype=torch.float64) + 0.5) * c["spacing"]
    pos = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), dim=-1).reshape(-1, 3) + disp
    del white, disp, dk
    if c["halos"] > 0:
        m = int(c["halos"] * n)
        nh = max(2, int(200 * (side / 256.0) ** 3))
        raw = torch.exp(torch.rand(nh, generator=gen, device=dev, dtype=torch.float64) * math.log(100.0))
        edge = torch.cumsum(raw / raw.sum(), 0)
        u = torch.rand((m, 4), generator=gen, device=dev, dtype=torch.float64)
        h = torch.searchsorted(edge, u[:, 3].contiguous()).clamp(max=nh - 1)
        centre = torch.rand((nh, 3), generator=gen, device=dev, dtype=torch.float64) * box
        scale = 0.05 * torch.exp(torch.rand(nh, generator=gen, device=dev, dtype=torch.float64) * math.log(10.0))
        x = (u[:, 0] * (1000.0 / 101.0 ** 1.5)).clamp(min=1e-12)
        r = scale[h] / torch.sqrt(x ** (-2.0 / 3.0) - 1.0)
        cz, phi = 2.0 * u[:, 1] - 1.0, 2.0 * math.pi * u[:, 2]
        s = torch.sqrt(1.0 - cz * cz)
        halo = centre[h] + r[:, None] * torch.stack([s * torch.cos(phi), s * torch.sin(phi), cz], dim=1)
        keep = torch.randperm(n, generator=gen, device=dev)[: n - m]
        pos = torch.cat([pos[torch.sort(keep).values], halo])
    pos = pos[: _count(c)]
    return torch.floor(torch.remainder(pos / box, 1.0) * TWO32).to(torch.int64) & 0xFFFFFFFF


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _physics(c):
    """eps^2 (spacing / 30 softening) and the coupling G a^3 for total mass 1."""
    box = _box(c)
    return (c["spacing"] / 30.0) ** 2, 3.0 * OMEGA_M * box ** 3 / (8.0 * math.pi) * COUPLING_A ** 3


def _kdk_factors():
    return DT / (2.0 * COUPLING_A), DT / COUPLING_A ** 2, DT / (2.0 * COUPLING_A)


def _r_split(c):
    return c["r_split_cells"] * _box(c) / c["mesh"]


def _batch(c, seed):
    """One training batch: volumes of features, particles in the interpolation
    range of their volume, target accelerations and loss weights (host arrays)."""
    rng = np.random.default_rng(int(seed) + 5)
    b, d, n = c["batch"], c["width"], c["batch"] * c["per_volume"]
    x0 = rng.standard_normal((b, d, d, d, c["c_in"]), dtype=np.float32)
    pb = np.repeat(np.arange(b, dtype=np.int32), c["per_volume"])
    ps = rng.uniform(0.0, d - 7 - 1e-3, (n, 3)).astype(np.float32)
    target = rng.standard_normal((n, 3), dtype=np.float32)
    weight = rng.uniform(0.5, 1.5, n).astype(np.float32)
    return x0, pb, ps, target, weight


def _weights():
    return os.path.join(ROOT, "gadget-ng_b200", "treepm", "weights", "learned_sr.npz")


def _params(c):
    """He-normal weights, as the library initialises a network to be trained."""
    from treepm import learned
    return learned.init_params(c["c_in"], 11)


def prepare(case, seed):
    import treepm
    from treepm import learned
    c = case
    if c["kind"] == "gradient":
        return dict(case=c, net=learned.Network(c["c_in"], params=_params(c)), batch=_batch(c, seed))
    n, box = _count(c), _box(c)
    pos = _pinned(_positions(c, seed).to(torch.float64) * (box / TWO32))
    mass = _pinned(torch.full((n,), 1.0 / n, dtype=torch.float64))
    eps2, g = _physics(c)
    s = dict(case=c, pos=pos, mass=mass, eps2=eps2, g=g)
    kind = c["kind"]
    if kind == "pm":
        s["solver"] = treepm.PmSolver(c["mesh"], box, four_point_gradient=c["four_point"],
                                      deconvolve_cic=c["deconvolve"])
    elif kind in ("accurate", "learned"):
        s["solver"] = treepm.TreePmSolver(c["mesh"], box, _r_split(c), r_cut_factor=c["r_cut_factor"], accurate=True,
                                          theta=c["theta"], deconvolve_cic=True, learned=kind == "learned",
                                          opening_criterion=1 if c.get("relative") else 0,
                                          err_tol_force_acc=c.get("err_tol", 0.005))
        if kind == "learned":
            s["net"] = learned.Network.load(_weights())
            s["solver"].set_learned(s["net"])
    else:
        s["solver"] = treepm.TreePmSolver(c["mesh"], box, _r_split(c), r_cut_factor=c["r_cut_factor"],
                                          periodic_walk=c.get("periodic", True))
    if kind == "steps":
        s["solver"].set_particles(pos, mass)
        s["solver"].compute_forces(eps2, g)
    elif kind == "host_steps":
        s["vel"] = _pinned(torch.zeros((n, 3), dtype=torch.float64))
    else:
        s["indices"] = _pinned(torch.arange(0, n, c["share"], dtype=torch.int64)).view(np.uint64)
        s["out"] = _pinned(torch.zeros((len(s["indices"]), 3), dtype=torch.float64))
    torch.cuda.empty_cache()  # the generator's scratch: a simulation holds no such memory
    return s


def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "gradient":
        loss, grad = s["net"].loss_grad(*s["batch"])
        return dict(loss=loss, grad=grad)
    if kind == "steps":
        kh, drift, kh2 = _kdk_factors()
        for _ in range(s["case"]["steps"]):
            s["solver"].kdk_step(kh, drift, kh2, s["eps2"], s["g"])
        k, pk, modes = s["solver"].power_spectrum()
        pos, vel, acc = s["solver"].get_state(_count(s["case"]))
        return dict(k=k, pk=pk, modes=modes, pos=pos, vel=vel, acc=acc)
    if kind == "host_steps":
        kh, drift, kh2 = _kdk_factors()
        s["solver"].kdk_step_host(s["pos"], s["vel"], s["mass"], kh, drift, kh2, s["eps2"], s["g"])
        return dict(pos=s["pos"], vel=s["vel"])
    return s["solver"].accelerations_for_indices(s["pos"], s["mass"], s["eps2"], s["g"], s["indices"], s["out"])


def _interactions(c):
    """Pair terms per target: the cells of the walk's terminal depth (half side
    below 0.1 r_cut) inside the cut sphere, or its particles where fewer."""
    cells = c["r_split_cells"] or 2.5
    r_cut = c["r_cut_factor"] * cells * _box(c) / c["mesh"]
    half = 0.5 * _box(c)
    while half >= 0.1 * r_cut:
        half *= 0.5
    density = min(1.0 / c["spacing"] ** 3, 1.0 / (2.0 * half) ** 3)
    return min(4.0 / 3.0 * math.pi * r_cut ** 3 * density, float(_count(c)))


def work(case):
    c = case
    if c["kind"] == "gradient":
        d, b, n = c["width"], c["batch"], c["batch"] * c["per_volume"]
        outs = [(d - 2) ** 3 * c["c_in"], (d - 4) ** 3 * 16, (d - 6) ** 3 * 16]
        fwd = sum(2.0 * 27 * 16 * o for o in outs) * b
        back = 2.0 * fwd - 2.0 * 27 * 16 * outs[0] * b  # weights of three layers, inputs of the last two
        params = 27 * 16 * (c["c_in"] + 32) + 48 + 51
        return dict(bytes=4.0 * b * d ** 3 * c["c_in"] + 32.0 * n + 8.0 * params, flops=fwd + back)
    n, mesh = _count(c), float(c["mesh"]) ** 3
    targets = n / c.get("share", 1)
    passes = c.get("steps", 1)
    fft = 4 * 2.5 * mesh * math.log2(mesh)
    pair = 0.0 if c["kind"] == "pm" else 37.0 * _interactions(c) * (n if "share" not in c else targets)
    if c["kind"] == "learned":
        pair = 0.3 * pair + 2.0 * 27 * 16 * 42 * mesh
    flops = passes * (fft + 120.0 * n + pair)
    if c["kind"] == "steps":
        return dict(bytes=n * 72.0, flops=flops)
    if c["kind"] == "host_steps":
        return dict(bytes=n * (24 + 24 + 8 + 48.0), flops=flops)
    return dict(bytes=n * 32.0 + targets * 32.0, flops=flops)


def tolerance(case):
    kind = case["kind"]
    if kind == "gradient":
        return dict(rel=1e-2, max=0.5)  # bf16 operands and activations, fp32 sums
    if kind == "learned":
        # bf16 activations in the network part, and particles whose cells lie on its density limit
        return dict(rel=5e-3, max=0.9, differ=0.0)
    # 32-bit pair terms and mesh, sums in another order; an acceleration whose parts cancel is worst
    return dict(rel=8e-6, max=2e-3, differ=0.0)


# ---- the same quantities in float64 -----------------------------------------------------

def _cic(pos, box, nm):
    c = pos * (nm / box)
    c = torch.where(c >= nm, c - nm, c)
    i0 = torch.floor(c)
    t = c - i0
    i0 = i0.to(torch.int64)
    for corner in range(8):
        bits = [(corner >> d) & 1 for d in range(3)]
        idx = [(i0[:, d] + bits[d]) % nm for d in range(3)]
        w = torch.ones_like(t[:, 0])
        for d in range(3):
            w = w * (t[:, d] if bits[d] else 1.0 - t[:, d])
        yield (idx[2] * nm + idx[1]) * nm + idx[0], w


def _density(pos, mass, box, nm):
    rho = torch.zeros(nm ** 3, dtype=torch.float64, device=pos.device)
    for idx, w in _cic(pos, box, nm):
        rho.index_add_(0, idx, mass * w)
    return rho


def _long_range(pos, mass, box, nm, r_split, four_point, deconvolve, want_phi=False):
    """Filtered spectral Poisson solve and CIC gather, per unit G."""
    dev = pos.device
    rho = _density(pos, mass, box, nm)
    cell = box / nm
    f = torch.fft.fftfreq(nm, device=dev, dtype=torch.float64) * nm
    k = 2.0 * math.pi / box * f
    fil = torch.exp(-0.5 * k * k * r_split * r_split)
    if deconvolve:
        fil = fil / torch.sinc(f / nm) ** 4
    der = (8.0 * torch.sin(k * cell) - torch.sin(2.0 * k * cell)) / (6.0 * cell) if four_point else k.clone()
    der[nm // 2] = 0.0
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    w = torch.where(k2 > 0, -4.0 * math.pi / cell ** 3 / k2.clamp(min=1e-300), torch.zeros_like(k2))
    w = w * fil[:, None, None] * fil[None, :, None] * fil[None, None, :]
    phi = torch.fft.fftn(rho.view(nm, nm, nm)) * w
    acc = torch.zeros_like(pos)
    for a, d in enumerate((der[None, None, :], der[None, :, None], der[:, None, None])):
        mesh = torch.fft.ifftn(-1j * d * phi).real.reshape(-1)
        for idx, wt in _cic(pos, box, nm):
            acc[:, a] += mesh[idx] * wt
    return (acc, rho, torch.fft.ifftn(phi).real.reshape(-1)) if want_phi else acc


def _octree(pos, mass, thr, quad):
    """The insertion octree, breadth first: per node COM, mass, half side,
    first child, child count, particle (leaves), with terminal nodes (half side
    below thr) left unopened; quad: cell centres and |Q|_F as well."""
    dev, n = pos.device, pos.shape[0]
    lo, hi = pos.min(0).values, pos.max(0).values
    half = float(((hi - lo) * 0.5).max())
    half += max(half * 1e-6, 1e-12)
    part = torch.arange(n, device=dev)
    node = torch.zeros(n, dtype=torch.int64, device=dev)  # index within the level
    centre = (0.5 * (lo + hi))[None]
    levels, base, depth = [], 0, 0
    count, leaf_of = torch.tensor([n], device=dev), torch.full((1,), -1, device=dev)
    while True:
        m, p = mass[part], pos[part]
        nn = centre.shape[0]
        tot = torch.zeros(nn, dtype=torch.float64, device=dev).index_add_(0, node, m)
        com = torch.zeros((nn, 3), dtype=torch.float64, device=dev).index_add_(0, node, m[:, None] * p)
        com = com / tot[:, None]
        lv = dict(com=com, mass=tot, leaf=leaf_of, centre=centre,
                  half=torch.full((nn,), half, dtype=torch.float64, device=dev))
        if quad:
            s = p - com[node]
            q = m[:, None] * torch.stack([3 * s[:, i] * s[:, j] - (i == j) * (s * s).sum(1)
                                          for i in range(3) for j in range(i, 3)], dim=1)
            q = torch.zeros((nn, 6), dtype=torch.float64, device=dev).index_add_(0, node, q)
            lv["qf"] = torch.sqrt((q * q).sum(1))
        opened = (count >= 2) & (half >= thr)
        live = opened[node]
        lv["first"] = torch.zeros(nn, dtype=torch.int64, device=dev)
        lv["nchild"] = torch.zeros(nn, dtype=torch.int64, device=dev)
        levels.append(lv)
        base += nn
        if not bool(live.any()) or depth > 60:
            break
        part, node, p = part[live], node[live], p[live]
        c = centre[node]
        octant = ((p >= c) * torch.tensor([1, 2, 4], device=dev)).sum(1)
        uniq, inv, count = torch.unique(node * 8 + octant, return_inverse=True, return_counts=True)
        parent, digit = uniq // 8, uniq % 8
        lv["nchild"].index_add_(0, parent, torch.ones_like(parent))
        lv["first"] = base + torch.cumsum(lv["nchild"], 0) - lv["nchild"]
        half *= 0.5
        sign = torch.stack([((digit >> d) & 1) * 2 - 1 for d in range(3)], dim=1).to(torch.float64)
        centre = centre[parent] + sign * half
        leaf_of = torch.full_like(uniq, -1)
        alone = count[inv] == 1
        leaf_of[inv[alone]] = part[alone]
        node, depth = inv, depth + 1
    return {k: torch.cat([lv[k] for lv in levels]) for k in levels[0]}


def _erfc(x):
    """Abramowitz & Stegun 7.1.26, the erfc of the split kernel."""
    t = 1.0 / (1.0 + 0.3275911 * x)
    p = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))
    return p * torch.exp(-x * x)


def _short_range(pos, mass, targets, box, r_split, r_cut, eps2, mode, theta=0.5, err_tol=0.005):
    """Short-range accelerations of `targets`, per unit G.  mode: periodic,
    aperiodic, angle (accurate) or relative (accurate, relative criterion)."""
    dev, accurate = pos.device, mode in ("angle", "relative")
    rc2, thr = r_cut * r_cut, 0.0 if accurate else 0.1 * r_cut
    t = _octree(pos, mass, thr, mode == "relative")
    image = (lambda d: d) if mode == "aperiodic" else (lambda d: d - box * torch.round(d / box))
    out = torch.zeros((targets.numel(), 3), dtype=torch.float64, device=dev)
    # wider nodes may be seen through two images: the relative criterion opens them
    top = 0.5 * (7.0 / 16.0 * box - 1.001 * r_cut)
    chunk = 16384 if not accurate else 4096
    for c0 in range(0, targets.numel(), chunk):
        ids = targets[c0:c0 + chunk]
        x = pos[ids]
        who = torch.arange(ids.numel(), device=dev)
        node = torch.zeros_like(who)
        while who.numel():
            d = image(t["com"][node] - x[who])
            h, leaf = t["half"][node], t["leaf"][node]
            is_leaf = leaf >= 0
            wide = 2.0 * h if accurate else h
            if mode != "aperiodic":  # the periodic walks cut leaves on their bare distance
                wide = torch.where(is_leaf, torch.zeros_like(h), wide)
            e = (d.abs() - wide[:, None]).clamp(min=0.0)
            seen = ((e * e).sum(1) <= rc2) & (leaf != ids[who])
            d2 = (d * d).sum(1)
            if mode == "angle":
                accept = 4.0 * h * h < theta * theta * d2
            elif mode == "relative":
                inside = (image(t["centre"][node] - x[who]).abs() <= 1.0001 * h[:, None]).all(1)
                accept = ~inside & (d2 > 0) & (t["qf"][node] * (d2 + eps2) < err_tol * t["mass"][node] * d2 ** 2.5)
                accept &= h < top
            else:
                accept = h < thr
            take = seen & (is_leaf | accept)
            r2 = d2[take] + eps2
            r = torch.sqrt(r2)
            xx = r / (math.sqrt(2.0) * r_split)
            w = _erfc(xx)
            if accurate:
                w = w + 2.0 / math.sqrt(math.pi) * xx * torch.exp(-xx * xx)
            out[c0:c0 + chunk].index_add_(0, who[take], (t["mass"][node[take]] * w / (r2 * r))[:, None] * d[take])
            go = seen & ~is_leaf & ~accept
            who, node = who[go], node[go]
            nc = t["nchild"][node]
            off = torch.arange(int(nc.sum()), device=dev) - torch.repeat_interleave(torch.cumsum(nc, 0) - nc, nc)
            who = torch.repeat_interleave(who, nc)
            node = torch.repeat_interleave(t["first"][node], nc) + off
    return out


def _unflatten(p, c_in):
    shapes = [(27, 16, c_in), (16,), (27, 16, 16), (16,), (27, 16, 16), (16,), (3, 16), (3,)]
    parts, at = [], 0
    for s in shapes:
        k = int(np.prod(s))
        parts.append(p[at:at + k].view(s))
        at += k
    return parts


def _network(p, c_in, x):
    """x [B, Z, Y, X, c] -> head output, three valid 3^3 convolutions with GELU."""
    w1, b1, w2, b2, w3, b3, wh, bh = _unflatten(p, c_in)
    for w, b in ((w1, b1), (w2, b2), (w3, b3)):
        _, Z, Y, X, _ = x.shape
        z = b.expand(x.shape[0], Z - 2, Y - 2, X - 2, 16)
        for tap in range(27):
            i, j, k = tap % 3, (tap // 3) % 3, tap // 9
            z = z + x[:, k:k + Z - 2, j:j + Y - 2, i:i + X - 2] @ w[tap].T
        x = torch.nn.functional.gelu(z)
    return x @ wh.T + bh


def _exact_gradient(c, seed):
    x0, pb, ps, target, weight = (torch.from_numpy(a).cuda() for a in _batch(c, seed))
    p = torch.from_numpy(_params(c)).cuda().double().requires_grad_(True)
    out = _network(p, c["c_in"], x0.double())
    i0 = torch.floor(ps.double()).long()
    f = ps.double() - i0
    pred = 0.0
    for corner in range(8):
        o = [(corner >> d) & 1 for d in range(3)]
        w = 1.0
        for d in range(3):
            w = w * (f[:, d] if o[d] else 1.0 - f[:, d])
        pred = pred + w[:, None] * out[pb.long(), i0[:, 2] + o[2], i0[:, 1] + o[1], i0[:, 0] + o[0]]
    w = weight.double()
    loss = (w[:, None] * (pred - target.double()) ** 2).sum() / w.sum()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=p.grad.cpu().numpy())


def _exact_learned(c, pos, mass, box, nm, r_split, r_cut, eps2):
    z = np.load(_weights())
    c_in = int(z["c_in"])
    lr, rho, phi = _long_range(pos, mass, box, nm, r_split, False, True, want_phi=True)
    m_cell, cell = float(mass.sum()) / nm ** 3, box / nm
    # octant masses of the cell centred on each node
    u = pos * (nm / box) + 0.5
    fl = torch.floor(u)
    bits = ((u - fl >= 0.5) * torch.tensor([1, 2, 4], device=pos.device)).sum(1)
    i = fl.long() % nm
    octants = torch.zeros((nm ** 3) * 8, dtype=torch.float64, device=pos.device)
    octants.index_add_(0, (((i[:, 2] * nm + i[:, 1]) * nm + i[:, 0]) << 3) + bits, mass)
    feat = torch.cat([torch.log1p(rho / m_cell)[:, None], (phi * cell / m_cell)[:, None],
                      torch.log1p(octants.view(-1, 8) * 8.0 / m_cell)], dim=1)[:, :c_in]
    feat = (feat - torch.from_numpy(z["shift"]).cuda().double()) * torch.from_numpy(z["scale"]).cuda().double()
    wrap = (torch.arange(nm + 6, device=pos.device) - 3) % nm
    vol = feat.view(nm, nm, nm, c_in)[wrap][:, wrap][:, :, wrap][None]
    head = _network(torch.from_numpy(z["params"]).cuda().double(), c_in, vol).view(-1, 3)
    sr = torch.zeros_like(pos)
    net = torch.ones(pos.shape[0], dtype=torch.bool, device=pos.device)
    for idx, w in _cic(pos, box, nm):
        net &= rho[idx] <= (1.0 + float(z["delta_max"])) * m_cell
        sr += head[idx] * w[:, None]
    sr *= float(z["out_scale"]) * m_cell / cell ** 2
    rest = torch.nonzero(~net).reshape(-1)
    sr[rest] = _short_range(pos, mass, rest, box, r_split, r_cut, eps2, "angle", c["theta"])
    return lr + sr


def _acceleration(c, pos, mass, targets):
    """Total acceleration of `targets` (float64 positions in the box)."""
    box, nm, kind = _box(c), c["mesh"], c["kind"]
    eps2, g = _physics(c)
    if kind == "pm":
        return g * _long_range(pos, mass, box, nm, 0.0, c["four_point"], c["deconvolve"])[targets]
    r_split = (c["r_split_cells"] or 2.5) * box / nm
    r_cut = c["r_cut_factor"] * r_split
    if kind == "learned":
        return g * _exact_learned(c, pos, mass, box, nm, r_split, r_cut, eps2)[targets]
    lr = _long_range(pos, mass, box, nm, r_split, False, kind == "accurate")[targets]
    mode = "periodic" if c.get("periodic", True) else "aperiodic"
    if kind == "accurate":
        mode = "relative" if c["relative"] else "angle"
    return g * (lr + _short_range(pos, mass, targets, box, r_split, r_cut, eps2, mode, c.get("theta", 0.5),
                                  c.get("err_tol", 0.005)))


def _spectrum(pos, mass, box, nm):
    """P(k) in shells floor(|k| - 1/2) of the fundamental, |delta_k|^2 over the CIC window."""
    f = torch.fft.fftfreq(nm, device=pos.device, dtype=torch.float64) * nm
    f[nm // 2] = nm // 2
    delta = torch.fft.fftn(_density(pos, mass, box, nm).view(nm, nm, nm)) * (nm ** 3 / float(mass.sum()))
    s = torch.sinc(f / nm)
    p = (delta.abs() / (s[:, None, None] * s[None, :, None] * s[None, None, :])) ** 2 * (box ** 3 / nm ** 3) ** 2
    kk = torch.sqrt(f[:, None, None] ** 2 + f[None, :, None] ** 2 + f[None, None, :] ** 2)
    ok = (kk >= 0.5) & (kk - 0.5 < nm // 2)
    shell = (kk[ok] - 0.5).long()
    modes = torch.bincount(shell, minlength=nm // 2)
    pk = torch.zeros(nm // 2, dtype=torch.float64, device=pos.device).index_add_(0, shell, p[ok]) / modes.clamp(min=1)
    keep = modes > 0
    k = (torch.arange(nm // 2, device=pos.device, dtype=torch.float64) + 1.0) * 2.0 * math.pi / box
    return k[keep].cpu().numpy(), pk[keep].cpu().numpy(), modes[keep].cpu().numpy()


def exact(case, seed):
    c = case
    if c["kind"] == "gradient":
        return _exact_gradient(c, seed)
    n, box = _count(c), _box(c)
    per_pass = c.get("steps", 1) + (c["kind"] in ("steps", "host_steps"))
    if n * per_pass * (1 if c["kind"] == "pm" else 4 if c["kind"] in ("accurate", "learned") else 2) > 1.2e7:
        return None
    pos = _positions(c, seed).to(torch.float64) * (box / TWO32)
    mass = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    every = torch.arange(n, device="cuda")
    if c["kind"] in ("steps", "host_steps"):
        kh, drift, kh2 = _kdk_factors()
        vel, acc = torch.zeros_like(pos), _acceleration(c, pos, mass, every)
        for _ in range(c.get("steps", 1)):
            vel = vel + acc * kh
            pos = torch.remainder(pos + vel * drift, box)
            acc = _acceleration(c, pos, mass, every)
            vel = vel + acc * kh2
        out = dict(pos=pos.cpu().numpy(), vel=vel.cpu().numpy())
        if c["kind"] == "steps":
            k, pk, modes = _spectrum(pos, mass, box, c["mesh"])
            out.update(k=k, pk=pk, modes=modes, acc=acc.cpu().numpy())
        return out
    return _acceleration(c, pos, mass, torch.arange(0, n, c["share"], device="cuda")).cpu().numpy()
