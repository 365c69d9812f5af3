"""Performance cases of the rigid-body integrator: what a program has the library do.

Four kinds of call, each through the package's public classes:

* ``replicas``   -- ``BatchedSystems.step``: one or many periodic boxes advance by ``steps`` steps with
  the library's own forces; then the energies and the frame are read, as a production run does at
  its reporting interval. Frames and logged energies are single precision, as trajectory formats
  and logs hold them.
* ``forces``     -- ``BatchedSystems.forces``: forces and potential energies at the current positions
  (a single-point evaluation, or the force call of a foreign integrator), handed on in single
  precision, the precision they are formed in.
* ``integrate``  -- ``IntegratorKernel`` on device buffers in the OpenMM layout: the drop-in use. One
  pass is two steps of the integrator, part1, fused (second half kick, first half kick) and part2,
  each with the force array the host program has then.
* ``host``       -- ``IntegratorKernel.step_host``: whole steps on pinned host arrays, forces in,
  positions and velocities out.

Boxes hold rigid 3-site waters or the 70/20/10 mix of waters, tetrahedra and six-membered rings at
about liquid density, optionally with free argon atoms and one rigid 64-atom solute whose partial
charges all differ (so that the force field has more than 32 atom types). Molecules sit on a
lattice that keeps them out of each other's Lennard-Jones cores, in random order and orientation,
with velocities at 300 K.
"""
import copy
import math

import numpy as np
import torch

from openmm_rigidbody_plugin_gb300 import batch, kernel
from openmm_rigidbody_plugin_gb300 import workloads as W

DT = 0.002            # ps
FORCE_SD = 50.0       # kJ/mol/nm, of the force arrays that a host program supplies
SITE = 0.317          # nm, edge of the lattice cell of one water
EPS_RF = 1e9          # reaction field of a conducting boundary: the Coulomb force ends at zero at the
                      # cutoff, so that a run conserves energy as pairs cross it
K_COULOMB = 138.935456
SOLUTE_EDGE, SOLUTE_SPACING = 4, 0.14

WATER, TETRA, RING, ARGON, SOLUTE = range(5)
MIX = {"water": (1.0, 0.0, 0.0), "mix": (0.7, 0.2, 0.1)}


def listed():
    return [
        # The plain single-box run: 512 waters, steps replayed from a captured graph. Every kernel is
        # small, so launches and their gaps count.
        dict(name="water512", kind="replicas", systems=1, lo=512, hi=512, mix="water", argon=0, solute=False,
             precision="mixed", mode=0, steps=21, graph=10),
        # A handful of the smallest replicas, stepped without a graph.
        dict(name="replicas24_small", kind="replicas", systems=24, lo=64, hi=190, mix="mix", argon=0, solute=False,
             precision="mixed", mode=0, steps=20, graph=0),
        # The batched workload: replicas of 64 to 4096 bodies of the mix, the default options.
        dict(name="replicas256_mix", kind="replicas", systems=256, lo=64, hi=4096, mix="mix", argon=0, solute=False,
             precision="mixed", mode=0, steps=20, graph=0),
        # Waters with some argon in single precision under NO-SQUISH, the cheap option of a screening run.
        dict(name="replicas60_single", kind="replicas", systems=60, lo=300, hi=2500, mix="water", argon=11,
             solute=False, precision="single", mode=4, steps=20, graph=0),
        # The largest box a simulation service takes: 200,000 atoms of water.
        dict(name="water66666", kind="replicas", systems=1, lo=66666, hi=66666, mix="water", argon=0, solute=False,
             precision="mixed", mode=0, steps=20, graph=0),
        # Single-point forces of solvated rigid solutes: every solute atom a type of its own.
        dict(name="forces_solutes40", kind="forces", systems=40, lo=700, hi=3100, mix="water", argon=0, solute=True,
             precision="mixed", mode=0),
        # Single-point forces of one mid-sized box of the mix in double precision (the precision study).
        dict(name="forces_double", kind="forces", systems=1, lo=15001, hi=15001, mix="mix", argon=300, solute=False,
             precision="double", mode=0),
        # The drop-in use on a small solvated system: latency.
        dict(name="integrate_333", kind="integrate", bodies=333, argon=21, domains=0, mix="mix", precision="mixed",
             mode=0, reorder=False),
        # NO-SQUISH with 10 substeps in single precision, a mid-sized water box.
        dict(name="integrate_21k_single", kind="integrate", bodies=21017, argon=1900, domains=0, mix="water",
             precision="single", mode=10, reorder=False),
        # Double precision, atoms in the slot order that the host program's reordering left, and rigid
        # protein domains of 33 to 120 atoms among the molecules.
        dict(name="integrate_50k_double", kind="integrate", bodies=50021, argon=1003, domains=97, mix="mix",
             precision="double", mode=0, reorder=True),
        # The large single system: 1,000,000 bodies and 100,000 free atoms.
        dict(name="integrate_1m", kind="integrate", bodies=1000000, argon=100000, domains=0, mix="mix",
             precision="mixed", mode=0, reorder=False),
        # Whole steps on pinned host arrays.
        dict(name="host_30k", kind="host", bodies=30011, argon=700, domains=0, mix="mix", precision="mixed", mode=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["replicas", "replicas", "forces", "integrate", "integrate", "host"])
    mode = rng.choice([0, 0, 0, 1, 4, 10])
    mix = "water" if mode else rng.choice(["mix", "water"])
    if kind in ("replicas", "forces"):
        precision = rng.choice(["mixed", "mixed", "single", "double"])
        systems = _log(rng, 1, 200)
        most = min(60000, 200000 // systems)  # no dearer than the listed batches
        lo = _log(rng, 64, min(most, 2000))
        hi = _log(rng, lo, max(lo, min(most, 16 * lo)))
        case = dict(kind=kind, systems=systems, lo=lo, hi=hi, mix=mix, argon=rng.choice([0, 0, rng.randrange(1, 40)]),
                    solute=lo >= 500 and rng.random() < 0.3, precision=precision, mode=mode)
        if kind == "replicas":
            graph = rng.choice([0, 0, 5, 10])
            case.update(steps=2 * graph + 1 if graph else rng.randrange(10, 21), graph=graph)
        return case
    bodies = _log(rng, 100, 100000 if mode or kind == "host" else 700000)
    precision = rng.choice(["mixed", "mixed", "single", "double"])
    if precision == "double":
        bodies = min(bodies, 40000 + bodies % 20000)
    case = dict(kind=kind, bodies=bodies, argon=rng.randrange(0, bodies // 10 + 2),
                domains=0 if mode else rng.choice([0, 0, rng.randrange(1, 100)]), mix=mix, precision=precision, mode=mode)
    if kind == "integrate":
        case["reorder"] = rng.random() < 0.4
    return case


# Molecules -----------------------------------------------------------------------------------
def _templates():
    """Per kind: atom coordinates about the centre of mass, masses, charges, sigmas, epsilons."""
    out = []
    for name in ("water", "tetra", "ring"):
        m = np.asarray(W.MASSES[name], dtype=np.float64)
        t = W.TEMPLATES[name] - (m[:, None] * W.TEMPLATES[name]).sum(0) / m.sum()
        q, s, e = (np.array(c) for c in zip(*(W.NONBONDED[k] for k in W.SPECIES[name])))
        out.append((t, m, q, s, e))
    q, s, e = W.NONBONDED[W.ARGON]
    out.append((np.zeros((1, 3)), np.array([W.ARGON_MASS]), np.array([q]), np.array([s]), np.array([e])))
    g = (np.arange(SOLUTE_EDGE) - 0.5 * (SOLUTE_EDGE - 1)) * SOLUTE_SPACING
    t = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3) * np.array([1.0, 1.02, 1.05])
    n = len(t)
    q = 0.3 * np.cos(1.7 * np.arange(n)) + 0.002 * np.arange(n)
    out.append((t, np.full(n, 13.0), q - q.mean(), np.full(n, 0.33), np.full(n, 0.35)))
    return out


TEMPLATES = _templates()
SIZES = np.array([len(t[1]) for t in TEMPLATES])


def _pad(column):
    out = np.zeros((len(TEMPLATES), SIZES.max()) + TEMPLATES[0][column].shape[1:])
    for k, t in enumerate(TEMPLATES):
        out[k, :SIZES[k]] = t[column]
    return out


XYZ, MASS, CHARGE, SIGMA, EPSILON = (_pad(c) for c in range(5))


def _split(bodies, mix):
    w, t, _ = MIX[mix]
    nw, nt = int(round(w * bodies)), int(round(t * bodies))
    return nw, nt, bodies - nw - nt


def _counts(case):
    """Body counts of the replicas, evenly spaced over the logarithm of their range."""
    S, lo, hi = case["systems"], case["lo"], case["hi"]
    return [int(round(lo * (hi / lo) ** ((i + 0.5) / S))) for i in range(S)]


def _lattice(rng, singles, rings, solute):
    """Box edge and the sites of `singles` one-site molecules and of `rings` flat molecules (a block of
    2 x 2 sites of a layer each), with room for the solute at the box centre."""
    room = 0.5 * (SOLUTE_EDGE - 1) * SOLUTE_SPACING * 1.05 + 0.3 if solute else 0.0
    edge = ((singles + 4 * rings) * SITE ** 3 + 8 * room ** 3) ** (1.0 / 3.0)
    while True:
        k = int(edge / 0.306)
        step = edge / max(k, 1)
        i = np.arange(k ** 3)
        site = np.stack([i % k, i // k % k, i // (k * k)], axis=1)
        x = (site + 0.5) * step
        free = (np.abs(x - 0.5 * edge) > room).any(axis=1) if solute else np.ones(len(x), dtype=bool)
        corner = np.nonzero((site[:, 0] % 2 == 0) & (site[:, 1] % 2 == 0) & (site[:, :2] < k - 1).all(axis=1))[0]
        block = corner[:, None] + np.array([0, 1, k, k + 1])
        block = block[free[block].all(axis=1)]
        if len(block) >= rings and int(free.sum()) >= singles + 4 * rings:
            break
        edge *= 1.01
    block = block[rng.permutation(len(block))[:rings]]
    free[block.ravel()] = False
    left = np.nonzero(free)[0]
    return edge, x[left[rng.permutation(len(left))[:singles]]], x[block].mean(axis=1)


def _atoms(rng, kinds, centres, system):
    """Atom arrays of molecules of the given kinds, centres and systems."""
    n = len(kinds)
    rot = W.random_rotations(rng, n)
    flat = np.nonzero(kinds == RING)[0]  # rings lie flat in their blocks
    angle = rng.uniform(0.0, 2.0 * np.pi, len(flat))
    rot[flat] = 0.0
    rot[flat, 0, 0] = rot[flat, 1, 1] = np.cos(angle)
    rot[flat, 1, 0] = np.sin(angle)
    rot[flat, 0, 1] = -rot[flat, 1, 0]
    rot[flat, 2, 2] = 1.0
    rot[kinds == SOLUTE] = np.eye(3)
    size = SIZES[kinds]
    mol = np.repeat(np.arange(n), size)
    first = np.cumsum(size) - size
    a = np.arange(len(mol)) - first[mol]
    k = kinds[mol]
    pos = centres[mol] + np.einsum("aij,aj->ai", rot[mol], XYZ[k, a])
    masses = MASS[k, a]
    vel = rng.standard_normal((len(mol), 3)) * np.sqrt(W.KB * 300.0 / masses)[:, None]
    body = np.where(k == ARGON, 0, mol + 1).astype(np.int32)
    return dict(masses=masses, body=body, system=system[mol], x=pos, v=vel, charge=CHARGE[k, a], sigma=SIGMA[k, a],
                epsilon=EPSILON[k, a])


def _boxes(case, seed):
    """The replicas of a case: concatenated atom arrays, atom offsets, box edges, cutoffs."""
    rng = np.random.default_rng(seed)
    kinds, centres, system, edges = [], [], [], []
    for s, n in enumerate(_counts(case)):
        nw, nt, nr = _split(n, case["mix"])
        edge, sites, blocks = _lattice(rng, nw + nt + case["argon"], nr, case["solute"])
        k = np.concatenate([np.repeat([WATER, TETRA, ARGON, RING], [nw, nt, case["argon"], nr]),
                            [SOLUTE] * case["solute"]]).astype(np.int64)
        c = np.concatenate([sites, blocks, np.full((int(case["solute"]), 3), 0.5 * edge)])
        order = rng.permutation(len(k))
        kinds.append(k[order])
        centres.append(c[order])
        system.append(np.full(len(k), s))
        edges.append(edge)
    a = _atoms(rng, np.concatenate(kinds), np.concatenate(centres), np.concatenate(system))
    a["offsets"] = np.concatenate([[0], np.cumsum(np.bincount(a["system"], minlength=len(edges)))])
    a["edges"] = np.array(edges)
    a["cutoffs"] = np.array([W.cutoff_for(L) for L in edges])
    return a


def _single(case, seed):
    """One large system for the integrator alone, with the force array of each half step."""
    rng = np.random.default_rng(seed)
    nw, nt, nr = _split(case["bodies"], case["mix"])
    _, sites, blocks = _lattice(rng, nw + nt + case["argon"], nr, False)
    k = np.repeat([WATER, TETRA, ARGON, RING], [nw, nt, case["argon"], nr])
    order = rng.permutation(len(k))
    a = _atoms(rng, k[order], np.concatenate([sites, blocks])[order], np.zeros(len(k), dtype=np.int64))
    if case["domains"]:  # rigid domains of 33 to 120 atoms
        size = 33 + 37 * np.arange(case["domains"]) % 88
        n = int(size.sum())
        centre = np.repeat(rng.uniform(0.0, 5.0, (case["domains"], 3)), size, axis=0)
        masses = rng.choice([1.008, 12.011, 14.007, 15.999], n)
        add = dict(masses=masses, body=np.repeat(a["body"].max() + 1 + np.arange(case["domains"]), size).astype(np.int32),
                   x=centre + 0.3 * rng.standard_normal((n, 3)),
                   v=rng.standard_normal((n, 3)) * np.sqrt(W.KB * 300.0 / masses)[:, None])
        a = {c: np.concatenate([a[c], add[c]]) for c in add}
    a["f"] = FORCE_SD * rng.standard_normal((len(a["masses"]), 3))
    a["location"] = None
    if case.get("reorder"):  # neighbourhoods of 64 atoms move together, as a spatial reordering leaves them
        n = len(a["masses"])
        blocks = rng.permutation(-(-n // 64))
        slots = (blocks[:, None] * 64 + np.arange(64)).ravel()
        a["location"] = np.argsort(slots[slots < n])
    return a


# The calls -----------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] in ("replicas", "forces"):
        a = _boxes(case, seed)
        b = batch.BatchedSystems(a["masses"], a["body"], a["offsets"], a["edges"], a["cutoffs"], a["charge"], a["sigma"],
                                 a["epsilon"], rotation_mode=case["mode"], precision=case["precision"],
                                 eps_solvent=EPS_RF)
        b.set_state(a["x"], a["v"])
        if case.get("graph"):
            b.set_graph_steps(case["graph"])
        return dict(case=case, batch=b)
    a = _single(case, seed)
    k = kernel.IntegratorKernel(a["masses"], a["body"], rotation_mode=case["mode"], precision=case["precision"])
    if case["kind"] == "host":
        k.context_set_state(a["x"], a["v"])
        pinned = [torch.empty(a["x"].shape, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
        pinned[0][:] = a["f"]
        pinned[1][:] = -a["f"]
        return dict(case=case, kernel=k, arrays=pinned)
    buf = kernel.DeviceBuffers(len(a["masses"]), precision=case["precision"])
    if a["location"] is not None:
        buf.location = a["location"]
        k.set_atom_locations(a["location"])
    buf.set_positions(a["x"])
    buf.set_velocities(a["v"], a["masses"])
    buf.set_forces(a["f"])
    k.upload_state_device(buf)
    # the force array after a step: opposed, so that a state that is stepped many times keeps its energy
    after = copy.copy(buf)
    after.force = -buf.force
    return dict(case=case, kernel=k, buffers=(buf, after))


def _f32(a):
    return torch.from_numpy(a).float()


def run(state):
    case = state["case"]
    if case["kind"] == "replicas":
        b = state["batch"]
        b.step(case["steps"], DT)
        e = b.energies()
        x, v = b.get_state()
        return dict(energies=_f32(e), x=_f32(x), v=_f32(v))
    if case["kind"] == "forces":
        f, e = state["batch"].forces()
        return dict(energies=_f32(e), f=_f32(f))
    k = state["kernel"]
    if case["kind"] == "host":
        f0, f1, x, v = state["arrays"]
        k.step_host(1, DT, f0, x, v)
        k.step_host(1, DT, f1, x, v)
        return dict(x=x, v=v)
    now, after = state["buffers"]
    k.part1(now, DT)
    k.fused(after, DT)
    k.part2(now, DT)
    out = dict(posq=now.posq, velm=now.velm)
    if now.corr is not None:
        out["corr"] = now.corr
    return out


def work(case):
    if case["kind"] in ("replicas", "forces"):
        body = atoms = free = pairs = 0
        per = np.array(MIX[case["mix"]])
        for n in _counts(case):
            na = float(n * (per * SIZES[:3]).sum()) + case["argon"] + 64 * case["solute"]
            ni = float(n * (per * np.array([3, 1, 6])).sum()) + case["argon"] + 64 * case["solute"]
            sites = float(n * (per * np.array([1, 1, 4])).sum()) + case["argon"] + 10 * case["solute"]
            volume = sites * SITE ** 3
            rc = W.cutoff_for(volume ** (1.0 / 3.0))
            pairs += 0.5 * ni * ni / volume * 4.0 / 3.0 * math.pi * rc ** 3
            body += n + int(case["solute"])
            atoms += na
            free += case["argon"]
        steps = case.get("steps", 1)
        flops = 28.0 * pairs + (350.0 * body + 40.0 * atoms if case["kind"] == "replicas" else 0.0)
        per_step = 40.0 * atoms  # positions read, forces written
        if case["kind"] == "replicas":
            per_step += 273.0 * body + 64.0 * (atoms - free) + 128.0 * free
        return dict(bytes=steps * per_step + 24.0 * atoms, flops=steps * flops)
    n = case["bodies"]
    nw, nt, nr = _split(n, case["mix"])
    atoms = nw * 3 + nt * 5 + nr * 12 + 76 * case["domains"]
    wide = 2 if case["precision"] == "double" else 1
    # per launch: body state in and out, constants; per atom: body-frame coordinates, slot, force,
    # position (or velocity) out; per free atom: force, velocity and position in and out
    launch = 273.0 * (n + case["domains"]) + (52.0 + 12.0 * wide) * atoms + 128.0 * case["argon"]
    launches = 3 if case["kind"] == "integrate" else 4
    rotate = 2 * (350.0 if case["mode"] == 0 else 150.0 * case["mode"]) * n
    host = 2 * 72.0 * (atoms + case["argon"]) if case["kind"] == "host" else 0.0
    return dict(bytes=launches * launch + host, flops=rotate + launches * (60.0 * atoms + 100.0 * n))


# The same in 64 bits, without the library -------------------------------------------------------
def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(dtype)


class _Rigid:
    """Rigid bodies and free atoms in FP64: kicks, drift and free rotation (by a fourth-order
    integration of the rotation at constant angular momentum, or NO-SQUISH on the principal axes)."""

    def __init__(self, a, mode):
        body = _t(a["body"], torch.int64)
        _, ids, counts = torch.unique(body, return_inverse=True, return_counts=True)
        self.m = _t(a["masses"])
        free = body <= 0
        # a free atom is a body of its own, without rotation
        nb = int(ids.max()) + 1
        ids = torch.where(free, nb + torch.cumsum(free, 0) - 1, ids)
        ids = torch.unique(ids, return_inverse=True)[1]
        self.ids, self.n, self.mode = ids, int(ids.max()) + 1, mode
        self.is_free = torch.zeros(self.n, dtype=torch.bool, device="cuda")
        self.is_free[ids[free]] = True
        # the atoms of each body, body by body
        order = torch.argsort(ids, stable=True)
        size = torch.bincount(ids, minlength=self.n)
        first = torch.cumsum(size, 0) - size
        self.order, self.size, self.first = order, size, first
        x, v = _t(a["x"]), _t(a["v"])
        self.M = self.sum(self.m)
        self.r = self.sum(self.m[:, None] * x) / self.M[:, None]
        self.p = self.sum(self.m[:, None] * v)
        d = x - self.r[ids]
        self.L = self.sum(self.m[:, None] * torch.linalg.cross(d, v))
        d2 = (d * d).sum(1)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        inertia = self.sum(self.m[:, None, None] * (d2[:, None, None] * eye - d[:, :, None] * d[:, None, :]))
        inertia[self.is_free] = eye
        self.L[self.is_free] = 0.0
        if mode:
            w, axes = torch.linalg.eigh(inertia.cpu())
            self.I = w.flip(1).cuda()
            axes = axes.flip(2)  # columns: principal axes, moments descending, right-handed
            self.A = (axes * torch.linalg.det(axes)[:, None, None]).cuda()
            self.d = torch.einsum("aji,aj->ai", self.A[ids], d)
        else:
            self.inv = torch.linalg.inv(inertia.cpu()).cuda()
            self.A = eye.expand(self.n, 3, 3).contiguous()
            self.d = d

    def sum(self, values):
        flat = values[self.order].reshape(len(self.ids), -1)
        out = torch.zeros(self.n, flat.shape[1], dtype=flat.dtype, device=flat.device)
        for k in range(int(self.size.max())):
            has = self.size > k
            out[has] += flat[self.first[has] + k]
        return out.reshape((self.n,) + values.shape[1:])

    def positions(self):
        return self.r[self.ids] + torch.einsum("aij,aj->ai", self.A[self.ids], self.d)

    def omega(self, A):
        if self.mode:
            body = torch.einsum("aji,aj->ai", A, self.L) / self.I
        else:
            body = torch.einsum("aij,aj->ai", self.inv, torch.einsum("aji,aj->ai", A, self.L))
        return torch.einsum("aij,aj->ai", A, body)

    def velocities(self):
        delta = torch.einsum("aij,aj->ai", self.A[self.ids], self.d)
        return (self.p / self.M[:, None])[self.ids] + torch.linalg.cross(self.omega(self.A)[self.ids], delta)

    def kick(self, f, h):
        delta = torch.einsum("aij,aj->ai", self.A[self.ids], self.d)
        self.p = self.p + h * self.sum(f)
        L = self.L + h * self.sum(torch.linalg.cross(delta, f))
        self.L = torch.where(self.is_free[:, None], torch.zeros_like(L), L)

    def drift(self, h):
        self.r = self.r + h * self.p / self.M[:, None]
        if self.mode:
            Lb = torch.einsum("aji,aj->ai", self.A, self.L)
            A, sub = self.A, h / self.mode
            for _ in range(self.mode):
                for axis, t in ((2, 0.5 * sub), (1, 0.5 * sub), (0, sub), (1, 0.5 * sub), (2, 0.5 * sub)):
                    angle = Lb[:, axis] / self.I[:, axis] * t
                    c, s = torch.cos(angle), torch.sin(angle)
                    i, j = (axis + 1) % 3, (axis + 2) % 3
                    Ai, Aj = A[:, :, i].clone(), A[:, :, j].clone()
                    A = A.clone()
                    A[:, :, i] = c[:, None] * Ai + s[:, None] * Aj
                    A[:, :, j] = c[:, None] * Aj - s[:, None] * Ai
                    Li, Lj = Lb[:, i].clone(), Lb[:, j].clone()
                    Lb = Lb.clone()
                    Lb[:, i] = c * Li + s * Lj
                    Lb[:, j] = c * Lj - s * Li
            self.A = A
            self.L = torch.einsum("aij,aj->ai", A, Lb)
            return
        n = 8
        t = h / n
        rate = lambda A: torch.linalg.cross(self.omega(A)[:, :, None].expand(-1, 3, 3), A, dim=1)  # noqa: E731
        for _ in range(n):
            k1 = rate(self.A)
            k2 = rate(self.A + 0.5 * t * k1)
            k3 = rate(self.A + 0.5 * t * k2)
            k4 = rate(self.A + t * k3)
            self.A = self.A + (t / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)

    def kinetic(self, system, S):
        t = 0.5 * (self.p * self.p).sum(1) / self.M
        r = 0.5 * (self.omega(self.A) * self.L).sum(1)
        owner = torch.zeros(self.n, dtype=torch.int64, device="cuda")
        owner[self.ids] = _t(system, torch.int64)
        out = torch.zeros(S, 2, dtype=torch.float64, device="cuda")
        for c, e in enumerate((t, r)):
            out[:, c] = torch.zeros(S, dtype=torch.float64, device="cuda").index_add(0, owner, e)
        return out


class _Field:
    """Cutoff Lennard-Jones and reaction-field forces of every box, all pairs."""

    def __init__(self, a):
        self.boxes = []
        active = (a["charge"] != 0.0) | (a["epsilon"] != 0.0)
        for s in range(len(a["edges"])):
            lo, hi = int(a["offsets"][s]), int(a["offsets"][s + 1])
            i = lo + np.nonzero(active[lo:hi])[0]
            body = np.where(a["body"][i] > 0, a["body"][i].astype(np.int64), -1 - i)
            rc = float(a["cutoffs"][s])
            krf = (EPS_RF - 1.0) / ((2.0 * EPS_RF + 1.0) * rc ** 3)
            self.boxes.append((_t(i, torch.int64), _t(body, torch.int64), _t(a["charge"][i]), _t(a["sigma"][i]),
                               _t(a["epsilon"][i]).sqrt(), float(a["edges"][s]), rc, krf, 1.0 / rc + krf * rc * rc))

    def pairs(self):
        return sum(float(len(b[0])) ** 2 for b in self.boxes)

    def __call__(self, x):
        f, energy = torch.zeros_like(x), torch.zeros(len(self.boxes), dtype=torch.float64, device="cuda")
        for s, (i, body, q, sigma, root, L, rc, krf, crf) in enumerate(self.boxes):
            p = x[i]
            rows = max(1, min(len(i), 20_000_000 // max(1, len(i))))
            for lo in range(0, len(i), rows):
                hi = min(len(i), lo + rows)
                d = p[lo:hi, None, :] - p[None, :, :]
                d -= L * torch.round(d / L)
                r2 = (d * d).sum(2)
                a, b = torch.nonzero((r2 < rc * rc) & (body[lo:hi, None] != body[None, :]), as_tuple=True)
                d, r2 = d[a, b], r2[a, b]
                a = a + lo
                inv2 = 1.0 / r2
                inv = inv2.sqrt()
                qq = K_COULOMB * q[a] * q[b]
                s6 = (0.25 * (sigma[a] + sigma[b]) ** 2 * inv2) ** 3
                e4 = 4.0 * root[a] * root[b]
                g = qq * (inv * inv2 - 2.0 * krf) + e4 * (12.0 * s6 * s6 - 6.0 * s6) * inv2
                f.index_add_(0, i[a], g[:, None] * d)
                energy[s] += 0.5 * (qq * (inv + krf * r2 - crf) + e4 * (s6 * s6 - s6)).sum()
        return f, energy


def exact(case, seed):
    if case["kind"] in ("replicas", "forces"):
        a = _boxes(case, seed)
        field = _Field(a)
        steps = case.get("steps", 0)
        if field.pairs() * (steps + 1) > 6e10:  # minutes of all-pairs FP64
            return None
        body = _Rigid(a, case["mode"])
        f, u = field(body.positions())
        if case["kind"] == "forces":
            return dict(energies=u.cpu(), f=f.cpu())
        for _ in range(steps):
            body.kick(f, 0.5 * DT)
            body.drift(DT)
            f, u = field(body.positions())
            body.kick(f, 0.5 * DT)
        e = torch.cat([u[:, None], body.kinetic(a["system"], len(a["edges"]))], dim=1)
        return dict(energies=e.cpu(), x=body.positions().cpu(), v=body.velocities().cpu())
    a = _single(case, seed)
    body, f = _Rigid(a, case["mode"]), _t(a["f"])
    if case["kind"] == "host":
        for g in (f, -f):
            body.kick(g, 0.5 * DT)
            body.drift(DT)
            body.kick(g, 0.5 * DT)
        return dict(x=body.positions().cpu(), v=body.velocities().cpu())
    body.kick(f, 0.5 * DT)
    body.drift(DT)
    body.kick(-f, DT)
    body.drift(DT)
    body.kick(f, 0.5 * DT)
    n = len(a["masses"])
    stride = (n + 31) // 32 * 32
    loc = torch.arange(n, device="cuda") if a["location"] is None else _t(a["location"], torch.int64)
    posq = torch.zeros(stride, 4, dtype=torch.float64, device="cuda")
    velm = torch.zeros_like(posq)
    posq[loc, :3] = body.positions()
    velm[loc, :3] = body.velocities()
    velm[loc, 3] = 1.0 / body.m
    out = dict(posq=posq, velm=velm)
    if case["precision"] == "mixed":
        out["corr"] = None  # the rounding residue of posq: no value of its own
    return out
