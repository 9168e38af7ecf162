"""Performance cases of the engine: the work that a user's program has it do through the public
Python API, over the range of sizes, methods and precisions that it is used for.

Kinds of case:

* ``md_water``: rigid-water dynamics, `Context.step(steps)` and then `get_state` of positions,
  velocities and energy, as a trajectory reporter does.  PME, optionally at constant pressure.
* ``force_water``: the engine as a force provider of an outside program (a minimiser, a sampler,
  a rescoring loop): new positions from the host, forces and energy back.
* ``md_chain`` / ``force_chain``: the same two uses for implicit-solvent chains (GBSAOBCForce),
  one chain or a batch, without a cutoff or with one, with exact or learned Born radii.
* ``mlp``: the learned-radii network on device tensors, tail and input gradient.

Water is placed on a cubic-ice (diamond) lattice whose hydrogens obey the ice rules, at the
density of the liquid, jittered and with vacancies: a low-energy start that needs no
equilibration by the engine itself and has the neighbour counts of the liquid.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "openmm-rs_b200"))

import ommb200  # noqa: E402
from ommb200 import synth, systems  # noqa: E402

ICE_CELL = (8.0 / 33.43) ** (1.0 / 3.0)  # nm: 8 waters per cubic cell, 33.43 waters per nm^3
KE = 138.93545764438198                  # kJ/mol nm / e^2
CUTOFF, TOL = 0.9, 5e-4                  # water boxes: cutoff (nm), Ewald error tolerance
FLOPS_PAIR = 62                          # LJ + screened Coulomb, energy-free, FMA = 2
FLOPS_GB = 150                           # LJ + Coulomb + descreening, GB pair, their gradients


def listed():
    water = dict(kind="md_water", precision="mixed", barostat=False)
    force = dict(kind="force_water", precision="mixed", method="PME")
    chain = dict(kind="md_chain", chains=1, lo=0, cutoff=0.0, learned=False)
    return [
        # a small box, as in free-energy windows and tests: launch latency counts
        dict(water, name="md-water-1524", kx=4, ky=4, kz=4, vacant=4, steps=100),
        # the 24k-atom box of the benchmark, 2 fs, constant volume
        dict(water, name="md-water-23958", kx=10, ky=10, kz=10, vacant=14, steps=100),
        # a large solvated system (the list is long enough for the large-box kernels)
        dict(water, name="md-water-255477", kx=22, ky=22, kz=22, vacant=25, steps=20),
        # constant pressure: a volume move every 25 steps
        dict(water, name="npt-water-8217", kx=7, ky=7, kz=7, vacant=5, steps=50, barostat=True),
        # double precision dynamics, for validation runs, in an uneven box
        dict(water, name="md-water-double-9387", kx=8, ky=7, kz=7, vacant=7, steps=20,
             precision="double"),
        # forces and energy of a mid-size box for an outside program
        dict(force, name="force-water-52713", kx=13, ky=13, kz=13, vacant=5),
        # the smallest call: reaction field with switching, small uneven box
        dict(force, name="force-water-rf-2397", kx=5, ky=5, kz=4, vacant=1, method="RF"),
        # one small implicit-solvent chain, 1 fs: launch latency counts
        dict(chain, name="md-chain-603", atoms=603, steps=100),
        # many uneven chains in one batch, no cutoff
        dict(chain, name="md-chains-48", chains=48, lo=200, atoms=2000, steps=20),
        # learned Born radii (judged and trained every 50 steps) on large chains
        dict(chain, name="md-chains-learned-3x5000", chains=3, lo=5000, atoms=5000, steps=50,
             learned=True),
        # one large chain with a cutoff, forces for an outside program
        dict(chain, kind="force_chain", name="force-chain-cutoff-4999", atoms=4999, cutoff=2.0),
        # the network alone on the features of 80,000 particles (16 chains of 5,000 atoms)
        dict(kind="mlp", name="mlp-80000", rows=80000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_box(rng, lo, hi):
    k = _log_int(rng, lo ** 3, hi ** 3) ** (1.0 / 3.0)
    kx = max(3, min(hi, int(round(k)) + rng.choice((-1, 0, 0, 1))))
    ky = max(3, min(hi, int(round(k)) + rng.choice((0, 0, 1))))
    kz = max(3, min(hi, int(round(k))))
    return dict(kx=kx, ky=ky, kz=kz, vacant=rng.randrange(1, 4 + kx * ky * kz // 20))


def draw(rng):
    kind = rng.choice(("md_water", "md_water", "force_water", "md_chain", "force_chain", "mlp"))
    if kind == "mlp":
        return dict(kind=kind, rows=_log_int(rng, 300, 80000))
    if kind == "force_water":
        return dict(kind=kind, precision=rng.choice(("mixed", "mixed", "double")),
                    method=rng.choice(("PME", "PME", "RF")), **_draw_box(rng, 4, 13))
    if kind == "md_water":
        form = rng.choice(("nvt", "nvt", "npt", "double"))
        box = _draw_box(rng, 4, 20 if form == "nvt" else 8)
        steps = rng.choice((20, 50, 60)) if box["kx"] <= 13 else 20
        return dict(kind=kind, precision="double" if form == "double" else "mixed",
                    barostat=form == "npt", steps=steps, **box)
    chains = rng.choice((1, 1, _log_int(rng, 2, 40)))
    atoms = _log_int(rng, 200, 5000 if chains == 1 else 2000)
    case = dict(kind=kind, chains=chains, lo=max(50, atoms // 3) if chains > 1 else 0, atoms=atoms,
                cutoff=rng.choice((0.0, 0.0, 1.5, 2.0)), learned=False)
    if kind == "md_chain":
        case.update(steps=rng.choice((20, 50)) if chains == 1 else 20, cutoff=0.0)
    return case


# ---- inputs -------------------------------------------------------------------------------
def _box(case):
    return np.array([case["kx"], case["ky"], case["kz"]]) * ICE_CELL


def _n_waters(case):
    return 8 * case["kx"] * case["ky"] * case["kz"] - case["vacant"]


def ice_box(case, seed):
    """Waters on the diamond lattice: sublattice A donates along bonds 0 and 1, sublattice B
    along bonds 2 and 3, so every bond holds one hydrogen."""
    rng = np.random.default_rng(seed)
    fcc = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    sites = np.concatenate([fcc, fcc + 0.25])
    cells = np.stack(np.meshgrid(*[np.arange(case[k]) for k in ("kx", "ky", "kz")], indexing="ij"),
                     -1).reshape(-1, 1, 3)
    o = ((cells + sites).reshape(-1, 3) + 0.125) * ICE_CELL
    bonds = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]]) / math.sqrt(3.0)
    pair = np.where(np.arange(len(o))[:, None] % 8 < 4, np.array([[0, 1]]), np.array([[2, 3]]))
    d = bonds[pair] * np.where(np.arange(len(o)) % 8 < 4, 1.0, -1.0)[:, None, None]
    keep = np.sort(rng.permutation(len(o))[:len(o) - case["vacant"]])
    o, d = o[keep] + rng.uniform(-0.01, 0.01, (len(keep), 3)), d[keep]
    mid = d[:, 0] + d[:, 1] + 0.3 * rng.normal(size=(len(keep), 3))  # tilted at random
    mid /= np.linalg.norm(mid, axis=1, keepdims=True)
    side = d[:, 0] - d[:, 1]
    side -= (side * mid).sum(1, keepdims=True) * mid
    side /= np.linalg.norm(side, axis=1, keepdims=True)
    half = synth.ANGLE_HOH / 2
    pos = np.stack([o, o + synth.D_OH * (math.cos(half) * mid + math.sin(half) * side),
                    o + synth.D_OH * (math.cos(half) * mid - math.sin(half) * side)], 1)
    return synth.WaterBox(positions=pos.reshape(-1, 3), box=np.diag(_box(case)),
                          n_waters=len(keep))


def _water_system(case, w):
    if case.get("method", "PME") == "PME":
        s = systems.water_system(w, cutoff=CUTOFF, ewald_tolerance=TOL)
    else:
        s = systems.water_system(w, cutoff=CUTOFF, method="CutoffPeriodic",
                                 dispersion_correction=False, switching_distance=0.8)
    if case.get("barostat"):
        bar = ommb200.MonteCarloBarostat(1.0, 300.0, 25)
        bar.set_random_number_seed(11)
        s.add_force(bar)
    return s


def _chain_sizes(case):
    """The sizes come from the case alone, so that the inputs of every seed have the same shapes."""
    if not case["lo"]:
        return np.full(case["chains"], case["atoms"])
    rng = np.random.default_rng(case["chains"] * 10007 + case["atoms"])
    return rng.integers(case["lo"], case["atoms"] + 1, case["chains"])


def chain_list(case, seed):
    rng = np.random.default_rng(seed)
    return [synth.chain(int(s), seed=int(rng.integers(1 << 30))) for s in _chain_sizes(case)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        g = torch.Generator(device="cuda").manual_seed(seed)

        def normal(*shape):
            return torch.randn(*shape, generator=g, device="cuda")

        features = (2.0 + 1.5 * normal(case["rows"], 32)).abs()
        params = torch.cat([
            normal(2048) / math.sqrt(32), 0.1 * normal(64), normal(4096) / 8.0, 0.1 * normal(64),
            normal(64) / 8.0, torch.tensor([0.05], device="cuda"),
            torch.full((32,), 2.1, device="cuda"), torch.full((32,), 1.0 / 1.35, device="cuda"),
            torch.tensor([0.01, 0.02], device="cuda")])
        return dict(kind=kind, features=features, params=params)
    if kind.endswith("water"):
        w = ice_box(case, seed)
        x = w.positions
        ctx = ommb200.Context(_water_system(case, w), systems.langevin(seed=seed % 100003 + 1),
                              precision=case["precision"])
    else:
        chs = chain_list(case, seed)
        x = np.concatenate([c.positions for c in chs])
        learned = dict(judge_interval=50) if case["learned"] else None
        built = [systems.chain_system(c, cutoff=case["cutoff"] or None, learned_radii=learned)
                 for c in chs]
        integ = systems.langevin(step_size=0.001, seed=seed % 100003 + 1)
        ctx = (ommb200.Context(built[0], integ) if len(built) == 1
               else ommb200.BatchContext(built, integ))
    if kind.startswith("md"):
        ctx.set_positions(x)
        ctx.set_velocities_to_temperature(300.0, seed=seed % 100003 + 1)
    return dict(kind=kind, ctx=ctx, x=x, steps=case.get("steps", 0))


def run(state):
    if state["kind"] == "mlp":
        tail, gradient = ommb200.radii_mlp_forward(state["features"], state["params"])
        return {"tail": tail, "gradient": gradient}
    ctx = state["ctx"]
    if state["kind"].startswith("force"):
        ctx.set_positions(state["x"])
        st = ctx.get_state(forces=True, energy=True)
        return {"forces": st.forces, "energy": st.potential_energy}
    ctx.step(state["steps"])
    st = ctx.get_state(positions=True, velocities=True, energy=True)
    return {"positions": st.positions, "velocities": st.velocities,
            "potential": st.potential_energy, "kinetic": st.kinetic_energy}


# ---- what a pass cannot do without ----------------------------------------------------------
def _chain_pairs(case):
    sizes = _chain_sizes(case)
    n = int(sizes.sum())
    if not case["cutoff"]:
        return n, float((sizes.astype(float) * (sizes - 1) / 2).sum())
    # a self-avoiding walk is loose: about 6 particles per nm^3 within the cutoff of one
    return n, float(n) * min(float(sizes.mean()) / 2, 0.5 * 6.0 * 4.2 * case["cutoff"] ** 3)


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        # 32 -> 64 -> 64 -> 1 forward and input gradient
        return {"bytes": case["rows"] * 4.0 * 65, "flops": case["rows"] * 4.0 * (32 * 64 + 64 * 64 + 64)}
    real = 8 if case.get("precision") == "double" else 4
    if kind.endswith("water"):
        n = 3 * _n_waters(case)
        density = n / float(np.prod(_box(case)))
        flops = n * 0.5 * density * 4.0 / 3.0 * math.pi * CUTOFF ** 3 * FLOPS_PAIR
        evaluation = n * (24 + 24 + 20)  # positions in, forces out, charge and LJ parameters
        if case.get("method", "PME") == "PME":
            g = float(np.prod(_grid(_box(case))))
            flops += n * 125 * 20.0 + 5.0 * g * math.log2(g)
            evaluation += 2 * real * g  # the charge grid written, the potential grid read
    else:
        n, pairs = _chain_pairs(case)
        flops = pairs * FLOPS_GB
        evaluation = n * (24 + 24 + 44)
    if kind.startswith("force"):
        return {"bytes": evaluation, "flops": flops}
    # the integrator reads positions, velocities and forces and writes positions, velocities;
    # the state that is returned needs one more evaluation, of the energy
    passes = case["steps"] + 1 + (2 * (case["steps"] // 25) if case.get("barostat") else 0)
    return {"bytes": case["steps"] * n * 120.0 + passes * evaluation + n * 48.0,
            "flops": passes * flops}


def tolerance(case):
    """About four times what the engine differs by from itself with its sums in another order
    (another list, the culling kernel) or, chains, with 64-bit pair arithmetic."""
    kind = case["kind"]
    if kind == "mlp":
        return {"rel": 4e-3, "max": 0.1}  # bf16 operands
    if case.get("precision") == "double":
        return {"rel": 1e-10, "max": 1e-8}
    if kind == "force_water":
        return {"rel": 4e-6, "max": 3e-5}
    if kind == "force_chain":
        return {"rel": 1e-5, "max": 4e-4}
    if kind == "md_chain":
        return {"rel": 2e-5, "max": 1e-3}
    # 32-bit forces of a liquid: a trajectory carries their rounding forward (measured after two
    # passes: 2e-4 in the velocities after 200 steps, 8e-6 after 100, 2e-6 after 40)
    if case["steps"] >= 100:
        return {"rel": 1e-3, "max": 0.03}
    return {"rel": 2e-4, "max": 6e-3} if case["steps"] >= 50 else {"rel": 2e-5, "max": 2e-3}


# ---- the same results in 64 bits --------------------------------------------------------------
def _grid(box):
    a = math.sqrt(-math.log(2.0 * TOL)) / CUTOFF
    return [max(6, math.ceil(2.0 * a * b / (3.0 * TOL ** 0.2))) for b in box]


def _spline(f, order):
    """B-spline weights of the given order at fractions f: [n, order]."""
    w = [1.0 - f, f]
    for n in range(3, order + 1):
        new = []
        for i in range(n):
            left = (f + (n - 1 - i)) * w[i - 1] if i > 0 else 0.0
            right = ((i + 1) - f) * w[i] if i < n - 1 else 0.0
            new.append((left + right) / (n - 1))
        w = new
    return torch.stack(w, -1)


def _reciprocal(x, q, box, alpha, grid):
    """Smooth particle-mesh Ewald, order 5: energy and forces."""
    dev, n = x.device, len(x)
    frac = x / box
    u = (frac - torch.floor(frac)) * torch.tensor(grid, dtype=torch.float64, device=dev)
    base = torch.floor(u)
    f = u - base
    w = _spline(f, 5)                                   # [n, 3, 5]
    w4 = _spline(f, 4)
    zero = torch.zeros_like(w4[..., :1])
    dw = torch.cat([zero, w4], -1) - torch.cat([w4, zero], -1)
    k = torch.arange(5, device=dev)
    at = [(base[:, a, None].long() + k) % grid[a] for a in range(3)]
    idx = ((at[0][:, :, None, None] * grid[1] + at[1][:, None, :, None]) * grid[2]
           + at[2][:, None, None, :]).reshape(n, -1)

    def outer(a, b, c):
        return (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(n, -1)

    rho = torch.zeros(grid[0] * grid[1] * grid[2], dtype=torch.float64, device=dev)
    rho.index_add_(0, idx.reshape(-1), (q[:, None] * outer(w[:, 0], w[:, 1], w[:, 2])).reshape(-1))
    s = torch.fft.fftn(rho.view(*grid))
    kk, mod = [], []
    w0 = _spline(torch.zeros((), dtype=torch.float64, device=dev), 5)
    for a in range(3):
        m = torch.arange(grid[a], device=dev, dtype=torch.float64)
        kk.append(torch.where(m < (grid[a] + 1) // 2, m, m - grid[a]) / box[a])
        ang = 2.0 * math.pi * m[:, None] * k / grid[a]
        b2 = (w0 * torch.cos(ang)).sum(1) ** 2 + (w0 * torch.sin(ang)).sum(1) ** 2
        # the modulus vanishes at the middle of an even grid: the mean of its neighbours there
        mod.append(torch.where(b2 < 1e-7, 0.5 * (b2.roll(1) + b2.roll(-1)), b2))
    k2 = kk[0][:, None, None] ** 2 + kk[1][None, :, None] ** 2 + kk[2][None, None, :] ** 2
    b2 = mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :]
    k2[0, 0, 0] = 1.0
    g = KE * torch.exp(-math.pi ** 2 * k2 / alpha ** 2) / (math.pi * box.prod() * k2 * b2)
    g[0, 0, 0] = 0.0
    energy = 0.5 * (g * (s.real ** 2 + s.imag ** 2)).sum()
    phi = (torch.fft.ifftn(s * g).real * rho.numel()).reshape(-1)[idx]
    scale = torch.tensor(grid, dtype=torch.float64, device=dev) / box
    grad = torch.stack([(phi * outer(dw[:, 0], w[:, 1], w[:, 2])).sum(1),
                        (phi * outer(w[:, 0], dw[:, 1], w[:, 2])).sum(1),
                        (phi * outer(w[:, 0], w[:, 1], dw[:, 2])).sum(1)], 1)
    return energy, -q[:, None] * grad * scale


def _exact_water(case, seed):
    w = ice_box(case, seed)
    pme = case["method"] == "PME"
    dev = "cuda"
    x = torch.tensor(w.positions, device=dev)
    q = torch.tensor(w.charges(), device=dev)
    box = torch.tensor(_box(case), device=dev)
    n = len(x)
    alpha = math.sqrt(-math.log(2.0 * TOL)) / CUTOFF
    forces = torch.zeros_like(x)
    energy = torch.zeros((), dtype=torch.float64, device=dev)
    mol = torch.arange(n, device=dev) // 3
    oxygen = torch.arange(n, device=dev) % 3 == 0
    eps4, sig2 = 4.0 * synth.EPS_O, synth.SIGMA_O ** 2
    krf = (78.3 - 1.0) / (2.0 * 78.3 + 1.0) / CUTOFF ** 3
    crf = 3.0 * 78.3 / (2.0 * 78.3 + 1.0) / CUTOFF
    step = max(1, 40_000_000 // n)
    for i in range(0, n, step):
        d = x[None, :] - x[i:i + step, None]
        d -= torch.round(d / box) * box
        r2 = (d * d).sum(-1)
        use = (r2 < CUTOFF ** 2) & (mol[i:i + step, None] != mol[None, :])
        row, col = use.nonzero(as_tuple=True)
        d, r2 = d[row, col], r2[row, col]
        row = row + i
        r = r2.sqrt()
        qq = KE * q[row] * q[col]
        if pme:
            erfc = torch.special.erfc(alpha * r)
            e = qq * erfc / r
            f = -qq * (erfc / r + 2.0 * alpha / math.sqrt(math.pi)
                       * torch.exp(-alpha ** 2 * r2)) / r2
        else:
            e = qq * (1.0 / r + krf * r2 - crf)
            f = qq * (-1.0 / (r2 * r) + 2.0 * krf)
        lj = oxygen[row] & oxygen[col]
        s6 = (sig2 / r2) ** 3
        le = eps4 * (s6 * s6 - s6)
        lf = eps4 * (-12.0 * s6 * s6 + 6.0 * s6) / r2
        if not pme:
            t = ((r - 0.8) / 0.1).clamp(min=0.0)
            s = 1.0 + t ** 3 * (-10.0 + t * (15.0 - 6.0 * t))
            lf = s * lf - le * 30.0 * t * t * (1.0 - t) ** 2 / 0.1 / r
            le = s * le
        e = torch.where(lj, e + le, e)
        f = torch.where(lj, f + lf, f)
        energy += 0.5 * e.sum()
        forces.index_add_(0, row, f[:, None] * d)
    if pme:
        er, fr = _reciprocal(x, q, box, alpha, _grid(_box(case)))
        energy += er - KE * alpha / math.sqrt(math.pi) * (q * q).sum()
        forces += fr
        m = x.view(-1, 3, 3)
        for a, b, qq in ((0, 1, synth.Q_O * synth.Q_H), (0, 2, synth.Q_O * synth.Q_H),
                         (1, 2, synth.Q_H ** 2)):  # the excluded pairs of each molecule
            d = m[:, b] - m[:, a]
            r = d.norm(dim=1)
            erf = torch.special.erf(alpha * r)
            energy -= KE * qq * (erf / r).sum()
            f = -KE * qq * (2.0 * alpha / math.sqrt(math.pi) * torch.exp(-(alpha * r) ** 2)
                            - erf / r) / r ** 2
            forces.view(-1, 3, 3)[:, a] += f[:, None] * d
            forces.view(-1, 3, 3)[:, b] -= f[:, None] * d
        nw = n // 3  # dispersion tail: mean of 4 eps sigma^k over ordered pairs, self included
        moment = [(4.0 * synth.EPS_O * synth.SIGMA_O ** p) * nw * (nw + 1) / (n * (n + 1.0))
                  for p in (12, 6)]
        energy += 8.0 * math.pi * n * n / float(box.prod()) / 4.0 * (
            moment[0] / (9.0 * CUTOFF ** 9) - moment[1] / (3.0 * CUTOFF ** 3))
    return {"forces": forces, "energy": energy}


def _descreening(ri, sj, r):
    """Pairwise descreening integral of a sphere sj at distance r outside radius ri."""
    lower = 1.0 / torch.maximum(ri, (r - sj).abs())
    upper = 1.0 / (r + sj)
    h = (lower - upper + 0.25 * r * (upper ** 2 - lower ** 2) + 0.5 / r * torch.log(upper / lower)
         + 0.25 * sj ** 2 / r * (lower ** 2 - upper ** 2))
    h = h + torch.where(ri < sj - r, 2.0 * (1.0 / ri - lower), torch.zeros_like(h))
    return torch.where(ri >= r + sj, torch.zeros_like(h), h)


def _chain_energy(ch, x, cutoff):
    n = len(x)
    dev = x.device
    q = torch.tensor(ch.charges, device=dev)
    rad = torch.tensor(ch.radii, device=dev)
    off = rad - 0.009
    scaled = off * ch.gb_scale
    i, j = torch.triu_indices(n, n, 1, device=dev)
    if cutoff:
        near = (x[i] - x[j]).detach().norm(dim=1)
        keep = (near <= cutoff) | (j - i <= 3)
        i, j = i[keep], j[keep]
    r = (x[j] - x[i]).norm(dim=1)
    inside = r.detach() < cutoff if cutoff else torch.ones_like(r, dtype=torch.bool)
    zero = torch.zeros_like(r)
    # NonbondedForce: 1-2 and 1-3 excluded, 1-4 without the cutoff
    qq = KE * q[i] * q[j]
    s6 = (ch.sigma / r) ** 6
    lj = 4.0 * ch.epsilon * (s6 * s6 - s6)
    coulomb = qq / r
    if cutoff:
        krf = (78.3 - 1.0) / (2.0 * 78.3 + 1.0) / cutoff ** 3
        crf = 3.0 * 78.3 / (2.0 * 78.3 + 1.0) / cutoff
        far = qq * (1.0 / r + krf * r * r - crf)
    else:
        far = coulomb
    sep = j - i
    e = torch.where((sep > 3) & inside, far + lj, zero).sum()
    e = e + torch.where(sep == 3, coulomb + lj, zero).sum()
    # GBSAOBCForce
    born = torch.zeros(n, dtype=torch.float64, device=dev)
    born = born.index_add(0, i, torch.where(inside, _descreening(off[i], scaled[j], r), zero))
    born = born.index_add(0, j, torch.where(inside, _descreening(off[j], scaled[i], r), zero))
    psi = 0.5 * off * born
    born = 1.0 / (1.0 / off - torch.tanh(psi - 0.8 * psi ** 2 + 4.85 * psi ** 3) / rad)
    pre = -KE * (1.0 - 1.0 / 78.5)
    e = e + (0.5 * pre * q * q / born).sum()
    e = e + (4.0 * math.pi * 2.25936 * (rad + 0.14) ** 2 * (rad / born) ** 6).sum()
    bb = born[i] * born[j]
    gb = pre * q[i] * q[j] / torch.sqrt(r * r + bb * torch.exp(-r * r / (4.0 * bb)))
    if cutoff:
        gb = gb - pre * q[i] * q[j] / cutoff
    e = e + torch.where(inside, gb, zero).sum()
    b = x[1:] - x[:-1]
    length = b.norm(dim=1)
    e = e + (0.5 * ch.bond_k * (length - ch.bond_length) ** 2).sum()
    cos = -(b[1:] * b[:-1]).sum(1) / (length[1:] * length[:-1])
    return e + (0.5 * ch.angle_k * (torch.acos(cos) - ch.angle) ** 2).sum()


def exact(case, seed):
    kind = case["kind"]
    if kind == "force_water":
        return _exact_water(case, seed)
    if kind == "force_chain":
        forces, energy = [], 0.0
        for ch in chain_list(case, seed):
            x = torch.tensor(ch.positions, device="cuda", requires_grad=True)
            e = _chain_energy(ch, x, case["cutoff"])
            forces.append(-torch.autograd.grad(e, x)[0])
            energy = energy + e.detach()
        return {"forces": torch.cat(forces), "energy": energy}
    if kind == "mlp":
        st = prepare(case, seed)
        p = st["params"].double()
        x = st["features"].double().requires_grad_(True)
        h = torch.tanh((x - p[6337:6369]) * p[6369:6401] @ p[:2048].view(32, 64) + p[2048:2112])
        h = torch.tanh(h @ p[2112:6208].view(64, 64) + p[6208:6272])
        tail = (h @ p[6272:6336] + p[6336]) * p[6402] + p[6401]
        return {"tail": tail.detach(), "gradient": torch.autograd.grad(tail.sum(), x)[0]}
    return None  # a trajectory of the engine's own random stream
