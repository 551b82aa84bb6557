"""What the performance of this framework is measured on: calls through its public
entry points, as programs that use it make them.

Every system is a seeded water box (the 23,558-atom box's density) around one or two
ligand chains, with 1-2 and 1-3 exclusions and scaled 1-4 exceptions in the ligand.
The replicas of one batch share the System, as in replica exchange over one alchemical
schedule, and differ in their positions and their state of the schedule.

Kinds of calls:
  context   one Context, as a plugin host drives it: new positions in, energy, forces
            and perturbation energy out, host arrays
  batch     ReplicaBatch.evaluateDevice on device tensors: the inner step of a sampler
            whose state lives on the GPU
  exchange  ReplicaBatch.evaluate with page-locked host buffers and the replicas x
            states matrix: a replica-exchange attempt of a host program
  gradient  W and its gradients with respect to positions, displacements and softplus
            parameters (autograd), fixed force field
  training  one step of fitting the ligand's charges, sigmas and epsilons and the
            softplus parameters: forward, backward, update of the parameters
  md        Langevin steps of one or many replicas and the state afterwards
  noalloc   the allocation-free reaction-field entry point
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "openmm-atmmetaforce-plugin_gb300"))

import atmmetaforce as atm  # noqa: E402
from atmmetaforce import autograd, synthetic  # noqa: E402
from atmmetaforce._lib import call  # noqa: E402

DENSITY = 23558 / 6.2 ** 3  # atoms per nm^3
METHODS = {"none": synthetic.NOCUTOFF, "rf": synthetic.CUTOFF_PERIODIC, "pme": synthetic.PME}
KE = 138.935456
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, atoms, ligand, method="pme", replicas=1, ligands=1, cutoff=0.9, triclinic=False,
          dispersion=True, difference=True, direction=1, steps=0, sizes=1):
    return {"name": name, "kind": kind, "atoms": atoms, "ligand": ligand, "method": method, "replicas": replicas,
            "ligands": ligands, "cutoff": cutoff, "triclinic": triclinic, "dispersion": dispersion,
            "difference": difference, "direction": direction, "steps": steps, "sizes": sizes}


def listed():
    return [
        # the smallest drop-in call: a host-guest sized box under a plugin host, both
        # end states in full, as the reference evaluates them
        _case("context-rf-2394", "context", 2394, 24, "rf", difference=False),
        # the drop-in call at the size the reference is quoted on, OpenMM's defaults
        _case("context-pme-23558", "context", 23558, 44, difference=False),
        # a few replicas of a small ragged box in a rhombic dodecahedral cell
        _case("batch-triclinic-8009x4", "batch", 8009, 29, replicas=4, triclinic=True),
        # the headline batch: a 22-state schedule of the 23,558-atom box
        _case("batch-pme-23558x22", "batch", 23558, 44, replicas=22, dispersion=False),
        # relative binding free energies: two ligands swapped, the largest box
        _case("batch-rbfe-60000x8", "batch", 60000, 36, replicas=8, ligands=2, cutoff=1.0, dispersion=False),
        # exchange attempts of a host program over boxes of several sizes
        _case("exchange-mixed-12000x8", "exchange", 12000, 30, replicas=8, sizes=3),
        # gradients through W at a fixed force field
        _case("gradient-12000x8", "gradient", 12000, 30, replicas=8, dispersion=False),
        # fitting a ligand's parameters: every step has new ones
        _case("training-5000x4", "training", 5000, 18, replicas=4, dispersion=False),
        # one trajectory, as the reference's own test and example run it
        _case("md-23558", "md", 23558, 44, steps=50, dispersion=False),
        # a batch of trajectories, records and matrix at every tenth step
        _case("md-12000x8", "md", 12000, 30, replicas=8, steps=20),
        # a caller whose own pool holds all device memory
        _case("noalloc-rf-12000", "noalloc", 12000, 30, "rf", dispersion=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["context", "batch", "batch", "exchange", "gradient", "training", "md", "noalloc"])
    method = rng.choice(["rf", "pme", "pme"])
    replicas, steps, sizes, ligands, cutoff = 1, 0, 1, 1, 0.9
    triclinic = rng.random() < 0.25
    difference = True
    if kind == "context":
        atoms = _log_int(rng, 900, 60000)
        difference = rng.random() < 0.4
        if atoms <= 3000 and rng.random() < 0.25:
            method, triclinic = "none", False
    elif kind == "batch":
        atoms = _log_int(rng, 900, 60000)
        replicas = max(1, min(32, _log_int(rng, 1, 500000 / atoms)))
        if atoms > 8000 and rng.random() < 0.4:
            ligands, cutoff = 2, 1.0
    elif kind == "exchange":
        atoms = _log_int(rng, 2500, 20000)
        replicas = max(2, min(24, _log_int(rng, 2, 250000 / atoms)))
        sizes = rng.randint(1, 3)
    elif kind in ("gradient", "training"):
        atoms = _log_int(rng, 900, 12000)
        replicas = max(1, min(8, _log_int(rng, 1, 60000 / atoms)))
    elif kind == "md":
        atoms = _log_int(rng, 2000, 24000)
        replicas = max(1, min(8, _log_int(rng, 1, 120000 / atoms)))
        steps = rng.randint(10, 60)
        triclinic = False
    else:
        atoms = _log_int(rng, 700, 16384)
        method, triclinic = "rf", False
    if triclinic:
        atoms = max(atoms, 1500)
    ligand = min(44, max(8, atoms // 150 + rng.randint(0, 9)))
    c = _case("", kind, atoms, ligand, method, replicas, ligands, cutoff, triclinic,
              rng.random() < 0.5 and kind not in ("gradient", "training", "noalloc"), difference,
              rng.choice([1, 1, -1]), steps, sizes)
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------------


def _boxes(case):
    """Atom count of each of the case's distinct systems: one, or several around `atoms`."""
    scale = [[1.0], [0.6, 1.4], [0.42, 1.0, 2.5]][case["sizes"] - 1]
    return [max(900, int(case["atoms"] * f)) for f in scale]


@functools.lru_cache(maxsize=4)
def _base(atoms, ligand, ligands, method, cutoff, triclinic, dispersion, direction, seed, even_grid):
    """One system and its starting positions."""
    sizes = [ligand] if ligands == 1 else [ligand - 4, ligand]
    volume = atoms / DENSITY
    if triclinic:  # a rhombic dodecahedral cell
        L = (volume / math.sqrt(0.5)) ** (1.0 / 3.0)
        box, tilt = [L, L, L * math.sqrt(0.5)], (0.0, 0.5 * L, 0.5 * L)
        edge = box[2]
    else:
        edge = volume ** (1.0 / 3.0)
    d = (0.5 if ligands == 1 else 0.3) * edge
    displ = [(d, d, d)] if ligands == 1 else [(d, d, d), (-d, -d, -d)]
    params = synthetic.default_params(0.25, 0.25, 0.1, 110.0, 0.0, 200.0, 100.0, 0.0625, float(direction))
    if triclinic:
        c = synthetic.triclinic_water_ligand_box(atoms, box, tilt, sizes, displ, METHODS[method], cutoff, seed, params)
    else:
        c = synthetic.water_ligand_box(atoms, edge, sizes, displ, METHODS[method], cutoff, seed, params)
    s = c.spec
    s.use_disp_corr = dispersion
    if even_grid:
        s.grid = tuple(k + k % 2 for k in s.grid)
    i = np.concatenate([lig[:-3] for lig in c.ligands])  # scaled 1-4 pairs
    j = i + 3
    s.exc_i = np.concatenate([s.exc_i, i]).astype(np.int32)
    s.exc_j = np.concatenate([s.exc_j, j]).astype(np.int32)
    s.exc_qq = np.concatenate([s.exc_qq, s.charge[i] * s.charge[j] / 1.2])
    s.exc_sig = np.concatenate([s.exc_sig, 0.5 * (s.sigma[i] + s.sigma[j])])
    s.exc_eps = np.concatenate([s.exc_eps, 0.5 * np.sqrt(s.epsilon[i] * s.epsilon[j])])
    return c


def _shaken(c, rng):
    """Another configuration of the same system: waters turned about and shifted, the ligand's atoms shifted."""
    n_lig = sum(len(x) for x in c.ligands)
    pos = c.pos.copy()
    w = pos[: c.n - n_lig].reshape(-1, 3, 3)
    q = rng.normal(size=(len(w), 4))
    a, b, g, d = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    rot = np.array([[a * a + b * b - g * g - d * d, 2 * (b * g - a * d), 2 * (b * d + a * g)],
                    [2 * (b * g + a * d), a * a - b * b + g * g - d * d, 2 * (g * d - a * b)],
                    [2 * (b * d - a * g), 2 * (g * d + a * b), a * a - b * b - g * g + d * d]])
    o = w[:, :1].copy()
    w[:] = o + np.einsum("xyw,wky->wkx", rot, w - o) + rng.uniform(-0.005, 0.005, (len(w), 1, 3))
    pos[c.n - n_lig:] += rng.normal(scale=0.001, size=(n_lig, 3))
    return pos


def _inputs(case, seed):
    """The case's distinct systems, which of them each replica is, positions and softplus parameters of each replica."""
    seed = int(seed) % (1 << 31)
    # OpenMM's own grids (odd ones among them); boxes of several sizes in one batch have even ones
    bases = [_base(n, case["ligand"], case["ligands"], case["method"], case["cutoff"], case["triclinic"],
                   case["dispersion"], case["direction"], seed + 7919 * k, case["sizes"] > 1)
             for k, n in enumerate(_boxes(case))]
    rng = np.random.default_rng(seed)
    which = [r % len(bases) for r in range(case["replicas"])]
    pos = [_shaken(bases[k], rng) for k in which]
    params = []
    for r in range(case["replicas"]):
        l1, l2 = synthetic.SCHEDULE_22[(5 + 3 * r) % 22 if case["replicas"] < 22 else r % 22]
        p = bases[which[r]].params.copy()
        p[0], p[1] = l1, l2
        params.append(p)
    return bases, which, pos, params


def prepare(case, seed):
    bases, which, pos, params = _inputs(case, seed)
    kind, R = case["kind"], case["replicas"]
    st = {"case": case}
    if kind == "noalloc":
        s = bases[0].spec
        lists = [[] for _ in range(s.n)]
        for i, j in zip(s.exc_i.tolist(), s.exc_j.tolist()):
            lists[i].append(j)
            lists[j].append(i)
        start = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int32)
        t = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=DEVICE)  # noqa: E731
        st["args"] = [t(pos[0]), t(s.charge), t(s.sigma), t(s.epsilon), t(start),
                      t(np.array([j for x in lists for j in x], dtype=np.int32))]
        st["out"] = [torch.zeros(1, dtype=torch.float64, device=DEVICE),
                     torch.zeros(s.n, 3, dtype=torch.float64, device=DEVICE)]
        st["box"] = (ctypes.c_double * 3)(*s.box)
        st["n"], st["cutoff"], st["eps_rf"] = s.n, s.cutoff, s.eps_rf
        return st
    if kind == "md":
        made = []
        for c in bases:
            terms, _ = synthetic.md_terms_ligand_centroid(c)
            made.append(atm.md_system_from_case(c, terms))
        integrator = atm.LangevinIntegrator(300.0, 1.0, 0.002)
        integrator.setRandomNumberSeed(int(seed))
        sim = atm.ReplicaSimulation([made[k][0] for k in which], integrator, 0, {"ListSkin": 0.1})
        sim.setPositions(np.concatenate(pos))
        sim.setVelocitiesToTemperature(300.0, int(seed))
        for r in range(R):
            for name, v in zip(synthetic.PARAM_NAMES, params[r]):
                sim.setParameter(r, name, float(v))
        if R > 1:
            sim.setRecording(10, 64)
        st.update(systems=made, sim=sim)
        return st
    made = [atm.system_from_case(c) for c in bases]
    st["systems"] = made
    if kind == "context":
        ctx = atm.Context(made[0][0], 0, {"DifferencePath": int(case["difference"])})
        for name, v in zip(synthetic.PARAM_NAMES, params[0]):
            ctx.setParameter(name, float(v))
        st.update(context=ctx, force=made[0][2], pos=pos[0])
        return st
    props = {"DifferencePath": 1}
    if kind in ("gradient", "training"):
        props["Adjoint"] = 1
    batch = atm.ReplicaBatch([made[k][0] for k in which], 0, props)
    for r in range(R):
        for name, v in zip(synthetic.PARAM_NAMES, params[r]):
            batch.setParameter(r, name, float(v))
    st["batch"] = batch
    allpos = np.concatenate(pos)
    if kind == "exchange":
        st["pos"] = torch.from_numpy(allpos).pin_memory().numpy()
        st["forces"] = torch.zeros(allpos.shape, dtype=torch.float64).pin_memory().numpy()
        return st
    dev = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=DEVICE)  # noqa: E731
    st["pos"] = dev(allpos)
    if kind == "batch":
        st["forces"] = torch.empty_like(st["pos"])
        st["results"] = torch.empty(R, atm.NUM_RES, dtype=torch.float64, device=DEVICE)
        return st
    st["displ"] = dev(np.concatenate([bases[k].displ for k in which]))
    st["params"] = dev(np.stack([p[:5] for p in params]))
    st["nb"] = [dev(np.concatenate([getattr(bases[k].spec, a) for k in which])) for a in ("charge", "sigma", "epsilon")]
    if kind == "training":
        lig = np.concatenate(bases[0].ligands)
        st["where"] = torch.as_tensor(np.concatenate([r * bases[0].n + lig for r in range(R)]), device=DEVICE)
        st["leaves"] = [v[st["where"][: len(lig)]].clone().requires_grad_() for v in st["nb"]]
        st["leaves"].append(st["params"].clone().requires_grad_())
        st["target"] = torch.full((R,), 50.0, dtype=torch.float64, device=DEVICE)
    return st


# steps of the parameters' update per unit of gradient (charge, sigma, epsilon, softplus parameters)
RATES = (1e-13, 1e-14, 1e-13, 1e-14)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "context":
        ctx = st["context"]
        ctx.setPositions(st["pos"])
        state = ctx.getState(getEnergy=True, getForces=True, groups={0, 2})
        return {"energy": state.getPotentialEnergy(), "forces": state.getForces(),
                "perturbation": st["force"].getPerturbationEnergy(ctx)}
    if kind == "batch":
        st["batch"].evaluateDevice(st["pos"].data_ptr(), st["forces"].data_ptr(), st["results"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        return {"forces": st["forces"], "results": st["results"]}
    if kind == "exchange":
        e, f, res = st["batch"].evaluate(st["pos"], out=st["forces"], as_array=True)
        return {"energies": e, "forces": f, "results": res, "matrix": st["batch"].energyMatrix(1.0 / 2.479)}
    if kind == "gradient":
        leaves = [v.detach().requires_grad_() for v in (st["pos"], st["displ"], st["params"])]
        w = autograd.atm_softplus_energy(st["batch"], *leaves, *st["nb"])
        w.sum().backward()
        return {"w": w.detach(), "positions": leaves[0].grad, "displacements": leaves[1].grad, "params": leaves[2].grad}
    if kind == "training":
        R = case["replicas"]
        nb = [v.index_copy(0, st["where"], leaf.repeat(R)) for v, leaf in zip(st["nb"], st["leaves"])]
        w = autograd.atm_softplus_energy(st["batch"], st["pos"], st["displ"], st["leaves"][3], *nb)
        grads = torch.autograd.grad(((w - st["target"]) ** 2).mean(), st["leaves"])
        with torch.no_grad():
            for leaf, g, rate in zip(st["leaves"], grads, RATES):
                leaf -= rate * g
        return {"w": w.detach(), "gradients": list(grads), "updated": [leaf.detach().clone() for leaf in st["leaves"]]}
    if kind == "md":
        sim = st["sim"]
        sim.step(case["steps"])
        state = sim.getState(getPositions=True, getVelocities=True, getEnergy=True)
        out = {"positions": state.getPositions(), "velocities": state.getVelocities(),
               "potential": state.getPotentialEnergy(), "kinetic": state.getKineticEnergy()}
        if case["replicas"] > 1:
            rec = sim.getRecords()
            out.update(steps=rec["steps"], records=rec["results"], matrices=rec["matrices"])
        return out
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    call("atm_rf_nonbonded_noalloc", st["n"], *(p(t) for t in st["args"]), st["box"], float(st["cutoff"]),
         float(st["eps_rf"]), *(p(t) for t in st["out"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return {"energy": st["out"][0], "forces": st["out"][1]}


def work(case):
    """Positions and force-field parameters in, forces (and gradients or state) out; 55 operations per pair within
    the cutoff (both end states' ligand pairs neglected), 500 per atom and 5 log2 per grid point for the grids."""
    counts = _boxes(case)
    atoms = sum(counts[r % len(counts)] for r in range(case["replicas"]))
    states = 2 if case["kind"] == "context" and not case["difference"] else 1
    pairs = 0.5 * atoms * (counts[0] if case["method"] == "none" else DENSITY * 4.19 * case["cutoff"] ** 3)
    flops = 55.0 * pairs * states
    if case["method"] == "pme":
        points = atoms / DENSITY * (56 / 6.2) ** 3
        flops += states * (500.0 * atoms + 10.0 * points * math.log2(points))
    flops *= max(1, case["steps"])
    per_atom = {"gradient": 24 + 24 + 48 + 24, "training": 24 + 24 + 24 + 24, "md": 24 + 24 + 48 + 48}
    return {"bytes": float(atoms * per_atom.get(case["kind"], 24 + 24 + 24)), "flops": float(flops)}


# ---- the same results in 64 bits ---------------------------------------------------


def _image(d, s):
    """Minimum image in a reduced box: c, then b, then a."""
    if s.method == synthetic.NOCUTOFF:
        return d
    v = torch.as_tensor(synthetic.box_vectors(s.box, s.tilt), dtype=d.dtype, device=d.device)
    for k in (2, 1, 0):
        d = d - torch.round(d[..., k:k + 1] / s.box[k]).detach() * v[k]
    return d


def _pairs(s, x):
    """Pairs i < j within the cutoff that are no exceptions."""
    n = len(x)
    lo, hi = np.minimum(s.exc_i, s.exc_j).astype(np.int64), np.maximum(s.exc_i, s.exc_j)
    skip = torch.as_tensor(np.sort(lo * n + hi), device=x.device)
    found = []
    for a in range(0, n, 512):
        d = _image(x[a:a + 512, None] - x[None], s)
        near = (d * d).sum(-1) < (1e20 if s.method == synthetic.NOCUTOFF else s.cutoff ** 2)
        i, j = torch.nonzero(near, as_tuple=True)
        key = (i + a) * n + j
        at = torch.searchsorted(skip, key).clamp(max=len(skip) - 1)
        ok = (j > i + a) & (skip[at] != key)
        found.append(torch.stack([i[ok] + a, j[ok]]))
    return torch.cat(found, 1)


def _splines(t):
    """Order-5 cardinal B-spline at t, t + 1, .. t + 4 (0 <= t < 1)."""
    m = [t, 1 - t]
    for o in range(3, 6):
        z = torch.zeros_like(t)
        m = [((t + k) * (m[k] if k < o - 1 else z) + (o - t - k) * (m[k - 1] if k else z)) / (o - 1) for k in range(o)]
    return torch.stack(m, -1)


def _reciprocal(s, x, q):
    v = torch.as_tensor(synthetic.box_vectors(s.box, s.tilt), dtype=x.dtype, device=x.device)
    inv = torch.linalg.inv(v)
    K = [int(k) for k in s.grid]
    u = (x @ inv) * torch.tensor(K, dtype=x.dtype, device=x.device)
    base = torch.floor(u).detach()
    w = [_splines(u[:, d] - base[:, d]) for d in range(3)]
    k5 = torch.arange(5, device=x.device)
    at = [(base[:, d].long()[:, None] - k5) % K[d] for d in range(3)]
    cell = (at[0][:, :, None, None] * K[1] + at[1][:, None, :, None]) * K[2] + at[2][:, None, None, :]
    val = q[:, None, None, None] * w[0][:, :, None, None] * w[1][:, None, :, None] * w[2][:, None, None, :]
    grid = torch.zeros(K[0] * K[1] * K[2], dtype=x.dtype, device=x.device).index_add(0, cell.reshape(-1), val.reshape(-1))
    m, mod = [], []
    for d in range(3):
        k = torch.arange(K[d], device=x.device, dtype=x.dtype)
        m.append(torch.where(k <= K[d] // 2, k, k - K[d]))
        ph = torch.exp(2j * math.pi * k[:, None] * torch.arange(4, device=x.device) / K[d])
        b = (ph * torch.tensor([1, 11, 11, 1], device=x.device) / 24).sum(1).abs() ** 2
        mod.append(torch.where(b < 1e-7, 0.5 * (b.roll(1) + b.roll(-1)), b))
    mv = [m[0][:, None, None] * inv[d, 0] + m[1][None, :, None] * inv[d, 1] + m[2][None, None, :] * inv[d, 2]
          for d in range(3)]
    m2 = mv[0] ** 2 + mv[1] ** 2 + mv[2] ** 2
    B = mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :]
    G = torch.exp(-math.pi ** 2 * m2 / s.alpha ** 2) / (math.pi * float(np.prod(s.box)) * m2 * B)
    G[0, 0, 0] = 0.0
    return 0.5 * (G * torch.fft.fftn(grid.reshape(K)).abs() ** 2).sum()


def _energy(s, x, q, sig, eps):
    """NonbondedForce energy of positions x in 64 bits, differentiable."""
    i, j = _pairs(s, x.detach())
    d = _image(x[j] - x[i], s)
    r2 = (d * d).sum(-1)
    r = torch.sqrt(r2)
    s6 = (0.5 * (sig[i] + sig[j])) ** 6 / r2 ** 3
    qq = KE * q[i] * q[j]
    e = (4 * torch.sqrt(eps[i] * eps[j]) * (s6 * s6 - s6)).sum()
    if s.method == synthetic.PME:
        e = e + (qq * torch.erfc(s.alpha * r) / r).sum()
    elif s.method == synthetic.CUTOFF_PERIODIC:
        k = (s.eps_rf - 1) / (2 * s.eps_rf + 1) / s.cutoff ** 3
        c = 3 * s.eps_rf / (2 * s.eps_rf + 1) / s.cutoff
        e = e + (qq * (1 / r + k * r2 - c)).sum()
    else:
        e = e + (qq / r).sum()
    t = lambda v: torch.as_tensor(v, device=x.device)  # noqa: E731
    on = np.nonzero((s.exc_qq != 0) | (s.exc_eps != 0))[0]
    d = x[t(s.exc_j[on]).long()] - x[t(s.exc_i[on]).long()]
    r2 = (d * d).sum(-1)
    s6 = t(s.exc_sig[on]) ** 6 / r2 ** 3
    e = e + (KE * t(s.exc_qq[on]) / torch.sqrt(r2) + 4 * t(s.exc_eps[on]) * (s6 * s6 - s6)).sum()
    if s.method == synthetic.PME:
        a, b = t(s.exc_i).long(), t(s.exc_j).long()
        r = _image(x[b] - x[a], s).norm(dim=-1)
        e = e - (KE * q[a] * q[b] * torch.erf(s.alpha * r) / r).sum() - KE * s.alpha / math.sqrt(math.pi) * (q * q).sum()
        e = e + KE * _reciprocal(s, x, q)
    if s.use_disp_corr and s.method != synthetic.NOCUTOFF:
        kinds, count = np.unique(np.stack([s.sigma, s.epsilon]), axis=1, return_counts=True)
        total = [0.0, 0.0]
        for a in range(len(count)):
            for b in range(a, len(count)):
                sg, ep = 0.5 * (kinds[0, a] + kinds[0, b]), math.sqrt(kinds[1, a] * kinds[1, b])
                m = count[a] * (count[a] + 1) / 2 if a == b else count[a] * count[b]
                total = [total[0] + m * ep * sg ** 12, total[1] + m * ep * sg ** 6]
        n2 = s.n * (s.n + 1) / 2
        e = e + 8 * math.pi * s.n ** 2 / float(np.prod(s.box)) * (
            total[0] / n2 / (9 * s.cutoff ** 9) - total[1] / n2 / (3 * s.cutoff ** 3))
    return e


def _merge(e1, e2, p):
    """The result record of end-state energies e1, e2 (plain numbers) under parameters p."""
    l1, l2, al, u0, w0, umax, ub, ac, direction = p
    u, e0 = (e2 - e1, e1) if direction > 0 else (e1 - e2, e2)
    usc, fp = u, 1.0
    if u > ub:
        g = (u - ub) / (ac * (umax - ub))
        z = 1 + 2 * g * (g + 1)
        za = z ** ac
        usc, fp = (umax - ub) * (za - 1) / (za + 1) + ub, 4 * (2 * g + 1) / z * za / (1 + za) ** 2
    x = math.exp(-al * (usc - u0))
    L = math.log1p(x)
    W = (l2 - l1) / al * L + l2 * usc + w0
    b = (l2 - l1) / (1 + x) + l1
    dalpha = -(l2 - l1) * L / al ** 2 - (l2 - l1) / al * (usc - u0) * x / (1 + x)
    return [e0 + W, usc, b * fp, W, u, e0, b, fp, e1, e2, -L / al, L / al + usc, dalpha, (l2 - l1) * x / (1 + x), 1.0,
            0.0, b * fp]


def _states(case, c, pos, p, gradients=False):
    """Energies at x and x + d, their gradients, and the record of one replica."""
    s = c.spec
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=DEVICE)  # noqa: E731
    got = []
    for d in (0.0, 1.0):
        leaves = [(t(pos) + d * t(c.displ)).requires_grad_(), t(s.charge), t(s.sigma), t(s.epsilon)]
        for v in leaves[1:]:
            v.requires_grad_(gradients)
        e = _energy(s, *leaves)
        got.append((e.item(), torch.autograd.grad(e, leaves if gradients else leaves[:1])))
    return got[0], got[1], _merge(got[0][0], got[1][0], p)


def exact(case, seed):
    kind = case["kind"]
    if kind == "md":  # a trajectory
        return None
    bases, which, pos, params = _inputs(case, seed)
    if kind == "noalloc":
        s = bases[0].spec
        s = type(s)(**{**s.__dict__, "exc_qq": 0 * s.exc_qq, "exc_eps": 0 * s.exc_eps, "use_disp_corr": False})
        t = lambda v: torch.as_tensor(v, device=DEVICE)  # noqa: E731
        x = t(pos[0]).requires_grad_()
        e = _energy(s, x, t(s.charge), t(s.sigma), t(s.epsilon))
        return {"energy": e.detach().reshape(1), "forces": -torch.autograd.grad(e, x)[0]}
    forces, results, ends = [], [], []
    fit = kind in ("gradient", "training")
    d_nb, d_pos, d_displ, d_params, w = [[], [], []], [], [], [], []
    for r in range(case["replicas"]):
        one, two, rec = _states(case, bases[which[r]], pos[r], params[r], fit)
        sign = 1.0 if case["direction"] > 0 else -1.0
        f1, f2 = -one[1][0], -two[1][0]
        forces.append(f1 + (rec[2] if sign > 0 else 1 - rec[2]) * (f2 - f1))
        results.append(rec)
        ends.append((one[0], two[0]))
        if fit:
            k = sign * rec[16]
            w.append(rec[3])
            d_pos.append(-k * (f2 - f1))
            d_displ.append(-k * f2)
            d_params.append(rec[10:15])
            for a in range(3):
                d_nb[a].append(k * (two[1][1 + a] - one[1][1 + a]))
    t = lambda v: torch.tensor(v, dtype=torch.float64, device=DEVICE)  # noqa: E731
    if kind == "context":
        return {"energy": results[0][0], "forces": forces[0], "perturbation": results[0][1]}
    if kind == "batch":
        return {"forces": torch.cat(forces), "results": t(results)}
    if kind == "exchange":
        m = [[_merge(*e, p)[0] / 2.479 for p in params] for e in ends]
        return {"energies": t([x[0] for x in results]), "forces": torch.cat(forces), "results": t(results),
                "matrix": t(m)}
    if kind == "gradient":
        return {"w": t(w), "positions": torch.cat(d_pos), "displacements": torch.cat(d_displ), "params": t(d_params)}
    R = case["replicas"]
    lig = torch.as_tensor(np.concatenate(bases[0].ligands), device=DEVICE)
    g = 2.0 * (t(w) - 50.0) / R
    grads = [sum(g[r] * d_nb[a][r][lig] for r in range(R)) for a in range(3)] + [g[:, None] * t(d_params)]
    start = [torch.as_tensor(v, device=DEVICE)[lig] for v in (bases[0].spec.charge, bases[0].spec.sigma, bases[0].spec.epsilon)]
    start.append(t([p[:5] for p in params]))
    return {"w": t(w), "gradients": grads, "updated": [a - k * b for a, b, k in zip(start, grads, RATES)]}
