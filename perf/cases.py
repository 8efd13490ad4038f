"""The calls whose speed matters to a user of this framework, over the range of sizes they come in.

A case says through which entry point (one molecule, a ragged batch of host arrays, a batch of
device tensors, a fixed-topology plan, a differentiable torch function), with which model and
options, and how many molecules of which size.  Molecules are made from a seed: saturated chains
C_n with some interior CH2 replaced by O or NH, drawn as self-avoiding conformers (so that the
self-consistent cycle settles as it does for sound geometries), radicals of them, and water
clusters.  ``exact`` is GFN2-xTB written out in torch, in 64 bits, for closed shells of H, C, N, O.
"""
from __future__ import annotations

import math
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

import xtbloom_b200
from xtbloom_b200 import abi, autograd, interface
from xtbloom_b200.workloads import water_cluster

KT = 300.0 * abi.KELVIN_TO_HARTREE


def _case(name, api, model, kind, count, low, high, **more):
    """count molecules of kind, of low to high backbone atoms (chain) or waters (water)."""
    c = {"api": api, "model": model, "kind": kind, "count": count, "low": low, "high": high,
         "spin": 1, "mixed": False, "point_charges": 0}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # the smallest call there is: the latency of a single point, as in a loop over small molecules
        _case("one water", "calculator", "gfn2", "water", 1, 1, 1),
        # one organic molecule of ordinary size, as in a geometry optimisation
        _case("one C20 chain", "calculator", "gfn2", "chain", 1, 20, 20),
        # one large molecule (240 orbitals)
        _case("one C31 chain, GFN1", "calculator", "gfn1", "chain", 1, 31, 31),
        # conformers of one molecule through a plan, as in a conformer search or dynamics
        _case("64 conformers of C10", "plan", "gfn2", "chain", 64, 10, 10),
        # screening of different molecules, host arrays in and out
        _case("256 chains C3-C40", "batch", "gfn2", "chain", 256, 3, 40),
        # the throughput workload: a large ragged batch resident on the device, graph replay on
        _case("2048 chains C3-C40", "device", "gfn2", "chain", 2048, 3, 40),
        # the other model over a ragged batch (more orbitals per hydrogen)
        _case("300 chains C3-C30, GFN1", "batch", "gfn1", "chain", 300, 3, 30),
        # open shells: doublets with two spin channels
        _case("200 radicals C4-C30", "device", "gfn2", "chain", 200, 4, 30, spin=2),
        # QM/MM training: energies and their derivatives through torch, forward and backward
        _case("128 C20 in 200 charges", "torch", "gfn2", "chain", 128, 20, 20, point_charges=200),
        # the split-precision execution form
        _case("150 chains C5-C35, split", "device", "gfn2", "chain", 150, 5, 35, mixed=True),
        # large systems: water clusters of 600 to 1200 orbitals
        _case("12 clusters of 100-200 water", "batch", "gfn2", "water", 12, 100, 200),
    ]


def draw(rng):
    pick = rng.randrange(9)
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if pick == 0:
        n = spread(1, 40)
        return _case(None, "calculator", "gfn2", "water", 1, n, n)
    if pick == 1:
        n = rng.randint(3, 42)
        return _case(None, "calculator", rng.choice(["gfn2", "gfn1"]), "chain", 1, n, n)
    if pick == 2:
        n = rng.randint(3, 25)
        return _case(None, "plan", "gfn2", "chain", spread(4, 300), n, n)
    low = rng.randint(3, 20)
    high = rng.randint(low + 5, 42)
    if pick == 3:
        return _case(None, "batch", "gfn2", "chain", spread(10, 600), low, high)
    if pick == 4:
        return _case(None, "device", "gfn2", "chain", spread(100, 1500), low, high)
    if pick == 5:
        return _case(None, "batch", "gfn1", "chain", spread(10, 400), low, min(high, 34))
    if pick == 6:
        return _case(None, "device", "gfn2", "chain", spread(5, 200), min(low, 12), min(high, 30), spin=2)
    if pick == 7:
        n = rng.randint(5, 30)
        return _case(None, "torch", "gfn2", "chain", spread(4, 128), n, n, point_charges=rng.randint(20, 300))
    low = rng.randint(30, 150)
    return _case(None, "batch", "gfn2", "water", rng.randint(1, 8), low, rng.randint(low, 200))


# ---------------------------------------------------------------------------
# Molecules
# ---------------------------------------------------------------------------
TETRA = math.acos(-1.0 / 3.0)
BOND = {frozenset((6,)): 2.91, frozenset((6, 8)): 2.70, frozenset((6, 7)): 2.77,
        frozenset((6, 1)): 2.06, frozenset((7, 1)): 1.91}


def _sizes(case):
    """Molecule sizes of a case: spread evenly over its range."""
    return np.linspace(case["low"], case["high"], case["count"]).round().astype(int)


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _chains(backbones, rng):
    """Self-avoiding conformers of several chains at once: per chain the positions of its backbone,
    each dihedral near 60, 180 or 300 degrees, atoms five bonds apart or more at least 7 bohr apart."""
    B, L = len(backbones), max(len(b) for b in backbones)
    elem = np.full((B, L), 6)
    for i, b in enumerate(backbones):
        elem[i, :len(b)] = b
    table = np.zeros((9, 9))
    for pair, length in BOND.items():
        a, b = (list(pair) * 2)[:2]
        table[a, b] = table[b, a] = length
    bond = table[elem[:, :-1], elem[:, 1:]]
    pos = np.zeros((B, L, 3))
    pos[:, 1, 0] = bond[:, 0]
    turn = math.pi - TETRA
    pos[:, 2] = pos[:, 1] + bond[:, 1, None] * np.array([math.cos(turn), math.sin(turn), 0.0])
    for k in range(3, L):
        a, b, c = pos[:, k - 3], pos[:, k - 2], pos[:, k - 1]
        bc = _unit(c - b)
        n = _unit(np.cross(b - a, bc))
        m = np.cross(n, bc)
        dih = np.radians(rng.permuted(np.tile([60.0, 180.0, 300.0], (B, 1)), axis=1) + rng.normal(0.0, 10.0, (B, 3)))
        r = bond[:, k - 1, None, None]
        new = c[:, None] + r * (math.cos(turn) * bc[:, None] + math.sin(turn) * (
            np.cos(dih)[..., None] * m[:, None] + np.sin(dih)[..., None] * n[:, None]))
        if k > 3:
            near = np.linalg.norm(new[:, :, None] - pos[:, None, :k - 3], axis=-1).min(-1)
            first = np.where((near > 7.0).any(1), (near > 7.0).argmax(1), near.argmax(1))
        else:
            first = np.zeros(B, int)
        pos[:, k] = new[np.arange(B), first]
    return [pos[i, :len(b)] for i, b in enumerate(backbones)]


def _saturate(backbone, pos, rng, radical):
    """Atomic numbers and positions with the hydrogens; None where two atoms meet."""
    z = np.array(backbone)
    missing = int(rng.choice(np.flatnonzero(z == 6))) if radical else -1
    bis, nrm = -(_unit(pos[:-2] - pos[1:-1]) + _unit(pos[2:] - pos[1:-1])), np.cross(pos[:-2] - pos[1:-1], pos[2:] - pos[1:-1])
    half = 0.5 * TETRA
    spokes = math.cos(half) * _unit(bis)[:, None] + math.sin(half) * _unit(nrm)[:, None] * np.array([[1.0], [-1.0]])
    ends = []
    for u in _unit(np.stack([pos[1] - pos[0], pos[-2] - pos[-1]])):
        t = np.array([1.0, 0.0, 0.0]) if abs(u[0]) < 0.9 else np.array([0.0, 1.0, 0.0])
        e1 = _unit(np.cross(u, t))
        phi = rng.uniform(0, 2 * math.pi) + np.arange(3)[:, None] * (2 * math.pi / 3)
        ends.append(math.cos(TETRA) * u + math.sin(TETRA) * (np.cos(phi) * e1 + np.sin(phi) * np.cross(u, e1)))
    dirs = np.concatenate([ends[0], spokes.reshape(-1, 3), ends[1]])
    owner = np.concatenate([[0] * 3, np.repeat(np.arange(1, len(z) - 1), 2), [len(z) - 1] * 3])
    place = np.concatenate([np.arange(3), np.tile([0, 1], len(z) - 2), np.arange(3)])
    keep = (z[owner] == 6) | (z[owner] == 7) & (place < 1)
    keep &= (owner != missing) | (place > 0)
    owner, dirs = owner[keep], dirs[keep]
    length = np.where(z[owner] == 6, BOND[frozenset((6, 1))], BOND[frozenset((7, 1))])
    numbers, coords = np.concatenate([z, np.ones(len(owner))]), [pos, pos[owner] + length[:, None] * dirs]
    numbers, xyz = numbers.astype(np.int32), np.concatenate(coords)
    d2 = ((xyz[:, None] - xyz[None]) ** 2).sum(-1) + 1e3 * np.eye(len(xyz))
    hydrogen = numbers == 1
    if d2[np.ix_(hydrogen, hydrogen)].min() < 2.9 ** 2 or (d2[np.ix_(~hydrogen, hydrogen)] < 3.3 ** 2).sum() != hydrogen.sum():
        return None
    return numbers, xyz + rng.normal(0.0, 0.03, xyz.shape)


def _molecules(case, seed):
    rng = np.random.default_rng([seed, 7])
    sizes = _sizes(case)
    if case["kind"] == "water":
        return [water_cluster(int(k), rng) for k in sizes]
    # the atoms belong to the case; which system has which molecule, and every position, to the seed
    conformers = case["low"] == case["high"]   # of one molecule: the same atoms in every system
    backbones = []
    for i, c in enumerate(sizes):
        r = np.random.default_rng([int(c), 0 if conformers else i])
        one = [6] * int(c)
        for k in range(1, int(c) - 1):
            if r.random() < 0.10 and one[k - 1] == 6:
                one[k] = 8 if r.random() < 0.5 else 7
        backbones.append(one)
    rng.shuffle(backbones)
    out = [None] * len(backbones)
    todo = list(range(len(backbones)))
    while todo:
        for i, pos in zip(todo, _chains([backbones[i] for i in todo], rng)):
            out[i] = _saturate(backbones[i], pos, rng, case["spin"] == 2)
        todo = [i for i in todo if out[i] is None]
    return out


def _charges_around(mols, npc, rng):
    """npc point charges per molecule in a shell around it, at least 6 bohr from every atom."""
    pos, val = [], []
    for _, xyz in mols:
        got = np.zeros((0, 3))
        while len(got) < npc:
            d = _unit(rng.normal(size=(4 * npc, 3)))
            p = xyz[rng.integers(0, len(xyz), 4 * npc)] + d * rng.uniform(6.0, 14.0, (4 * npc, 1))
            near = np.sqrt(((p[:, None] - xyz[None]) ** 2).sum(-1)).min(1)
            got = np.concatenate([got, p[near > 6.0]])
        q = rng.uniform(-0.5, 0.5, npc)
        pos.append(got[:npc])
        val.append(q - q.mean())
    return np.concatenate(pos), np.concatenate(val)


# ---------------------------------------------------------------------------
# The calls
# ---------------------------------------------------------------------------
@lru_cache(maxsize=None)
def _library(mixed, graphs):
    lib = abi.Library(xtbloom_b200.library_path(), backend=abi.BACKEND_CUDA, device_id=torch.cuda.current_device())
    lib.set_execution(abi.PRECISION_MIXED if mixed else abi.PRECISION_FP64, 0.0, graphs)
    return lib


def prepare(case, seed):
    mols = _molecules(case, seed)
    numbers, positions = [m[0] for m in mols], [m[1] for m in mols]
    method = case["model"] + "-xtb"
    state = {"case": case}
    uhf = [case["spin"] - 1] * len(mols)
    if case["api"] == "calculator":
        state["calculator"] = interface.Calculator(method, numbers[0], positions[0])
        return state
    if case["api"] == "batch":
        state["calculator"] = interface.BatchCalculator(method, numbers, positions)
        return state
    host = abi.ragged_from_lists(numbers, positions, uhf=uhf,
                                 spin_channels=[2] * len(mols) if case["spin"] == 2 else None)
    if case["api"] == "plan":
        state["plan"] = abi.Plan(_library(case["mixed"], True), host)
        state["batch"] = host
        return state
    put = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    if case["api"] == "torch":
        p, q = _charges_around(mols, case["point_charges"], np.random.default_rng([seed, 8]))
        off = np.arange(len(mols) + 1, dtype=np.int64) * case["point_charges"]
        state["args"] = [put(host.atomic_numbers), put(host.atom_offsets),
                         put(host.positions.reshape(-1, 3)).requires_grad_(True), put(off),
                         put(p).requires_grad_(True), put(q).requires_grad_(True), put(np.full(len(q), 999.0))]
        return state
    names = ("atom_offsets", "atomic_numbers", "positions", "molecular_charges", "unpaired_electrons", "spin_channels")
    state["batch"] = abi.RaggedBatch(**{n: put(getattr(host, n)) for n in names})
    nb, na = host.batch_size, host.total_atoms
    f64 = {"dtype": torch.float64, "device": "cuda"}
    state["outputs"] = {"energies": torch.empty(nb, **f64), "forces": torch.empty(3 * na, **f64),
                        "atomic_charges": torch.empty(na, **f64),
                        "scc_iterations": torch.empty(nb, dtype=torch.int32, device="cuda"),
                        "scc_converged": torch.empty(nb, dtype=torch.uint8, device="cuda"),
                        "per_system_status": torch.empty(nb, dtype=torch.int32, device="cuda")}
    state["library"] = _library(case["mixed"], True)
    state["options"] = state["library"].make_options(
        model=abi.MODEL_GFN1 if case["model"] == "gfn1" else abi.MODEL_GFN2)
    return state


def run(state):
    case = state["case"]
    if case["api"] == "calculator":
        r = state["calculator"].singlepoint()
        return {"energies": np.array([r.get("energy")]), "forces": r.get("forces"), "charges": r.get("charges")}
    if case["api"] == "batch":
        r = state["calculator"].singlepoint()
        return {"energies": r.get("energies"), "forces": np.concatenate(r.get("forces")),
                "charges": np.concatenate(r.get("charges")), "status": r.get("status")}
    if case["api"] == "torch":
        args = state["args"]
        e = autograd.gfn2_energy(*args)
        g = torch.autograd.grad(e.sum(), [args[2], args[4], args[5]])
        return {"energies": e.detach(), "positions": g[0], "pc_positions": g[1], "pc_charges": g[2]}
    if case["api"] == "plan":
        o = state["plan"].compute(state["batch"])
    else:
        o = state["library"].compute(state["batch"], state["options"], state["outputs"])
    return {"energies": o["energies"], "forces": o["forces"].reshape(-1, 3), "charges": o["atomic_charges"],
            "status": o["per_system_status"]}


def _orbitals(case):
    """Per molecule: orbitals, occupied orbitals and atoms."""
    s = _sizes(case).astype(float)
    if case["kind"] == "water":
        return 6 * s, 4 * s, 3 * s
    h = 2 * s + 2
    return (4 * s + h * (2 if case["model"] == "gfn1" else 1)), (2 * s + 0.5 * h), s + h


def work(case):
    """A single point of n orbitals, m occupied, cannot do without an eigensolver's work for each of
    about 12 cycles and one overlap factorisation: the basis transforms, a tridiagonal form, the
    occupied vectors and their density; all n vectors once."""
    n, m, atoms = _orbitals(case)
    cycle = (3 + 4 / 3) * n ** 3 + 5 * n * n * m
    once = (4 / 3 + 2 + 1) * n ** 3
    bytes_ = 8 * (7 * atoms.sum() + case["count"]) + 56 * case["count"] * case["point_charges"]
    return {"bytes": float(bytes_), "flops": float((12 * case["spin"] * cycle + once).sum())}


def tolerance(case):
    # The cycle stops inside a gate (charge residual 1e-6): charges end about 1e-5 from the fixed
    # point, and another path to the gate ends elsewhere in it.  The split form goes on to a gate 100
    # times tighter.
    return {"rel": 2e-6, "max": 4e-5} if case["mixed"] else {"rel": 5e-5, "max": 1e-3}


# ---------------------------------------------------------------------------
# GFN2-xTB in torch, 64 bits: closed shells of H, C, N and O
# ---------------------------------------------------------------------------
_NAMES = ("wexp", "enscale", "kpol", "pair_scale_default", "rep_kexp", "rep_klight", "es3_s", "es3_p", "es3_d",
          "mp_dmp3", "mp_dmp5", "mp_kexp", "mp_shift", "mp_rmax", "d4_a1", "d4_a2", "d4_s6", "d4_s8", "d4_s9")
_BOHR, _EV = 1.8897261246204404, 1.0 / 27.21138505
_QUAD = ((0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2))


@lru_cache(maxsize=1)
def _tables():
    raw = np.load(Path(xtbloom_b200.__file__).parent / "data" / "params.npz")
    p = {k: raw[k] for k in raw.files}
    p.update(zip(_NAMES, p["gfn2_globals"].tolist()))
    return p


class _Molecule:
    """One molecule's parameters as torch arrays, and its energy terms as functions of the positions."""

    def __init__(self, numbers, dev):
        p = _tables()
        z = np.asarray(numbers) - 1
        put = lambda a: torch.as_tensor(np.asarray(a, float), device=dev)  # noqa: E731
        self.dev, self.p, self.n = dev, p, len(z)
        shells = [(a, s) for a in range(len(z)) for s in range(int(p["gfn2_nshell"][z[a]]))]
        at = np.array([a for a, _ in shells])
        lo = np.array([s for _, s in shells])
        l = p["gfn2_shell_l"][z[at], lo]
        ao_sh = np.repeat(np.arange(len(shells)), 2 * l + 1)
        # orbitals of a p shell in the order y, z, x
        axis = np.concatenate([[-1] if k == 0 else [1, 2, 0] for k in l])
        alpha, coeff = np.ones((len(shells), 4)), np.zeros((len(shells), 4))
        for i, (a, s) in enumerate(shells):
            ng, n = int(p["gfn2_shell_ngauss"][z[a], s]), int(p["gfn2_shell_n"][z[a], s])
            typ = n - 1 if l[i] == 0 else n + 3
            al = p["sto_alpha%d" % ng][typ] * p["gfn2_shell_slater"][z[a], s] ** 2
            alpha[i, :ng] = al
            coeff[i, :ng] = p["sto_coeff%d" % ng][typ] * (2 / math.pi * al) ** 0.75 * np.sqrt(4 * al) ** l[i]
        idx = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
        self.sh_at, self.ao_sh, self.ao_at, self.axis = idx(at), idx(ao_sh), idx(at[ao_sh]), idx(axis)
        self.alpha, self.coeff = put(alpha[ao_sh]), put(coeff[ao_sh])
        self.refocc = put(p["gfn2_shell_refocc"][z[at], lo])
        self.level = put(p["gfn2_shell_level"][z[at], lo] * _EV)
        self.kcn = put(p["gfn2_shell_kcn"][z[at], lo] * _EV)
        self.poly = put(p["gfn2_shell_shpoly"][z[at], lo])
        self.rad = put(p["atomic_radii_angstrom"][z] * _BOHR)
        self.rcov = put(4 / 3 * _BOHR * p["covalent_radii_angstrom"][z])
        zeta, en = p["gfn2_shell_slater"][z[at], lo], p["gfn2_en"][z[at]]
        self.scale = put((2 * np.sqrt(np.outer(zeta, zeta)) / np.add.outer(zeta, zeta)) ** p["wexp"]
                         * (1 + p["enscale"] * np.subtract.outer(en, en) ** 2)
                         * p["gfn2_shell_pair_scale"][np.ix_(l, l)] * p["pair_scale_default"])
        self.eta = put(p["gfn2_gam"][z[at]] * p["gfn2_shell_hubbard_scale"][z[at], lo])
        self.g3 = put(p["gfn2_gam3"][z[at]] * np.array([p["es3_s"], p["es3_p"]])[l])
        self.mprad, self.mpvcn = put(p["gfn2_mprad"][z]), put(p["gfn2_mpvcn"][z])
        self.dk, self.qk = put(p["gfn2_dkernel"][z]), put(p["gfn2_qkernel"][z])
        self.rep_a, self.rep_z = put(np.sqrt(p["gfn2_arep"][z])), put(p["gfn2_zeff"][z])
        self.light = idx(z < 2)
        self.d4_rcov, self.d4_en, self.r4r2 = put(p["d4_rcov"][z]), put(p["d4_en"][z]), put(p["d4_r4r2"][z])
        self.d4_zeff, self.d4_eta = put(p["d4_zeff"][z]), put(p["d4_eta"][z])
        ref = np.array([[p["d4_ref_offset"][k] + min(r, p["d4_ref_count"][k] - 1) for r in range(7)] for k in z])
        self.has = put([[r < p["d4_ref_count"][k] for r in range(7)] for k in z])
        self.ref_cn, self.ref_q, self.ref_ng = put(p["d4_ref_cn"][ref]), put(p["d4_ref_q"][ref]), put(p["d4_ref_ngauss"][ref])
        self.ref_c6 = put(p["d4_ref_c6"][ref.reshape(-1)][:, ref.reshape(-1)]).reshape(self.n, 7, self.n, 7)
        self.off = ~torch.eye(self.n, dtype=torch.bool, device=dev)

    def geometry(self, x):
        """Everything that depends on the positions alone."""
        p, g = self.p, {}
        d = x[:, None] - x[None]
        r2 = (d * d).sum(-1) + torch.where(self.off, 0.0, 1.0)
        r = r2.sqrt()
        near = lambda c: self.off & (r2 <= c * c)  # noqa: E731
        g["d"], g["r"], g["r2"] = d, r, r2
        rc = self.rcov[:, None] + self.rcov[None]
        cn = (near(25.0) * torch.sigmoid(10 * (rc / r - 1)) * torch.sigmoid(20 * ((rc + 2) / r - 1))).sum(1)
        lev = self.level - self.kcn * cn[self.sh_at]
        rr = (r / (self.rad[:, None] + self.rad[None])).sqrt()[self.sh_at][:, self.sh_at]
        other = self.sh_at[:, None] != self.sh_at[None]
        spat = torch.where(other, self.scale * (1 + self.poly[:, None] * rr) * (1 + self.poly[None] * rr), 1.0)
        fac = 0.5 * (lev[:, None] + lev[None]) * spat
        g["S"], g["D"], g["Q"] = self.integrals(x)
        g["H0"] = g["S"] * fac[self.ao_sh][:, self.ao_sh]
        avg = 0.5 * (self.eta[:, None] + self.eta[None])
        g["gam"] = torch.where(other, (torch.where(other, r2[self.sh_at][:, self.sh_at], 1.0) + avg ** -2).rsqrt(), avg)
        rad = self.mprad + (p["mp_rmax"] - self.mprad) * torch.sigmoid(p["mp_kexp"] * (cn - self.mpvcn - p["mp_shift"]))
        sc = 0.5 * (rad[:, None] + rad[None]) / r
        g["k3"] = self.off / (r ** 3 * (1 + 6 * sc ** 3))
        g["k5"] = self.off / (r ** 5 * (1 + 6 * sc ** 4))
        rc = self.d4_rcov[:, None] + self.d4_rcov[None]
        enf = 4.10451 * torch.exp(-((self.d4_en[:, None] - self.d4_en[None]).abs() + 19.08857) ** 2 / (2 * 11.28174 ** 2))
        cn4 = (near(30.0) * 0.5 * enf * torch.erfc(7.5 * (r - rc) / rc)).sum(1)
        rrij = 3 * self.r4r2[:, None] * self.r4r2[None]
        r0 = p["d4_a1"] * rrij.sqrt() + p["d4_a2"]
        g["damp"] = near(50.0) * (p["d4_s6"] / (r2 ** 3 + r0 ** 6) + p["d4_s8"] * rrij / (r2 ** 4 + r0 ** 8))
        dl2 = (cn4[:, None] - self.ref_cn) ** 2
        num = sum((self.ref_ng >= k) * torch.exp(-6.0 * k * dl2) for k in range(1, int(self.ref_ng.max()) + 1)) * self.has
        g["cw"] = num / num.sum(1, keepdim=True)
        lp = self.light[:, None] & self.light[None]
        pa = self.rep_a[:, None] * self.rep_a[None]
        rep = near(25.0) * self.rep_z[:, None] * self.rep_z[None] * torch.exp(-pa * torch.where(lp, r, r ** 1.5)) / r
        g["rep"] = 0.5 * rep.sum()
        # three-body dispersion at charge zero
        w = g["cw"] * self.charge_scale(torch.zeros_like(cn))
        c6 = torch.einsum("ar,arbs,bs->ab", w, self.ref_c6, w)
        i, j, k = (t for t in torch.combinations(torch.arange(self.n, device=self.dev), 3).T) if self.n > 2 else [torch.zeros(0, dtype=torch.long, device=self.dev)] * 3
        ok = near(25.0)
        keep = ok[i, j] & ok[i, k] & ok[j, k]
        i, j, k = i[keep], j[keep], k[keep]
        a, b, c = r2[i, j], r2[j, k], r2[i, k]
        r3 = (a * b * c) ** 1.5
        ang = 0.375 * (a + b - c) * (a - b + c) * (b + c - a) / (r3 * a * b * c) + 1 / r3
        f = 1 / (1 + 6 * ((r0[i, j] * r0[i, k] * r0[j, k]) / r3 ** (1 / 3)) ** (16 / 3))
        g["atm"] = (ang * f * p["d4_s9"] * (c6[i, j] * c6[i, k] * c6[j, k]).abs().sqrt()).sum()
        return g

    def integrals(self, x):
        """Overlap, dipole and traceless quadrupole matrices, the operators at the column's atom."""
        v = x[self.ao_at][None] - x[self.ao_at][:, None]        # row (bra) to column (ket)
        ab, ak = self.alpha[:, None, :, None], self.alpha[None, :, None, :]
        inv = 1 / (ab + ak)
        est = ab * ak * inv * (v * v).sum(-1)[..., None, None]
        pref = torch.where(est <= 25.0, torch.exp(-est), 0.0) * (math.pi * inv) ** 1.5 * self.coeff[:, None, :, None] * self.coeff[None, :, None, :]
        one, half, axes = torch.ones_like(pref), 0.5 * inv, []
        for c in range(3):
            vc = v[..., c, None, None]
            pk, pb = -vc * ab * inv, vc * ak * inv
            t = [[one, pb]]                                       # t[a][b]: a on the ket, b on the bra
            for a in range(1, 4):
                t.append([pk * t[a - 1][0] + ((a - 1) * half * t[a - 2][0] if a > 1 else 0.0), None])
                t[a][1] = pb * t[a][0] + a * half * t[a - 1][0]
            bra = (self.axis == c)[:, None, None, None]
            ket = (self.axis == c)[None, :, None, None]
            sel = [torch.where(bra, t[a][1], t[a][0]) for a in range(4)]
            axes.append([torch.where(ket, sel[a + 1], sel[a]) for a in range(3)])
        full = lambda e: (pref * axes[0][e[0]] * axes[1][e[1]] * axes[2][e[2]]).sum((-1, -2))  # noqa: E731
        S = full((0, 0, 0))
        D = torch.stack([full(tuple(int(c == k) for c in range(3))) for k in range(3)])
        raw = [full(tuple(int(c == k) + int(c == m) for c in range(3))) for k, m in _QUAD]
        tr = 0.5 * (raw[0] + raw[2] + raw[5])
        return S, D, torch.stack([1.5 * q - (tr if k == m else 0.0) for q, (k, m) in zip(raw, _QUAD)])

    def charge_scale(self, q):
        ref = self.ref_q + self.d4_zeff[:, None]
        return torch.exp(3.0 * (1 - torch.exp(2 * self.d4_eta[:, None] * (1 - ref / (q + self.d4_zeff)[:, None]))))

    def interaction(self, g, qsh, dip, quad, vpc):
        """The energy that depends on the charges and multipoles."""
        q = torch.zeros_like(dip[:, 0]).index_add(0, self.sh_at, qsh)
        e = 0.5 * qsh @ g["gam"] @ qsh + (self.g3 * qsh ** 3).sum() / 3 + qsh @ vpc
        weight = torch.tensor([1.0, 2.0, 1.0, 2.0, 2.0, 1.0], dtype=torch.float64, device=self.dev)
        e = e + (self.dk * (dip * dip).sum(1)).sum() + (self.qk * (weight * quad * quad).sum(1)).sum()
        d, k3, k5 = g["d"], g["k3"], g["k5"]
        dd = torch.einsum("fsc,sc->fs", d, dip)                    # (R_f - R_s) . mu_s
        df = torch.einsum("fsc,fc->fs", d, dip)
        e = e + (k3 * q[:, None] * dd).sum() + 0.5 * (k5 * (g["r2"] * (dip @ dip.T) - 3 * dd * df)).sum()
        sq = sum(w * d[..., k] * d[..., m] * quad[None, :, c] for c, ((k, m), w) in enumerate(zip(_QUAD, (1, 2, 1, 2, 2, 1))))
        e = e + (k5 * q[:, None] * sq).sum()
        w = g["cw"] * self.charge_scale(q)
        return e - 0.5 * (torch.einsum("ar,arbs,bs->ab", w, self.ref_c6, w) * g["damp"]).sum()

    def populations(self, g, P):
        qsh = self.refocc - torch.zeros_like(self.refocc).index_add(0, self.ao_sh, (P * g["S"]).sum(0))
        atoms = lambda m: torch.zeros((self.n, len(m)), dtype=torch.float64, device=self.dev).index_add(0, self.ao_at, -(P * m).sum(1).T)  # noqa: E731
        return qsh, atoms(g["D"]), atoms(g["Q"])

    def solve(self, x, pc_x=None, pc_q=None, pc_gam=999.0):
        """Energy, charges and the derivatives by the positions (and by the point charges')."""
        x = torch.as_tensor(x, dtype=torch.float64, device=self.dev).requires_grad_(True)
        points = [] if pc_x is None else [torch.as_tensor(a, dtype=torch.float64, device=self.dev).requires_grad_(True) for a in (pc_x, pc_q)]
        live = self.geometry(x)
        g = {k: v.detach() for k, v in live.items()}

        def potential():
            if not points:
                return torch.zeros_like(self.eta)
            d = x[self.sh_at][:, None] - points[0][None]
            return ((d * d).sum(-1) + (2 / (self.eta[:, None] + pc_gam)) ** 2).rsqrt() @ points[1]

        vpc = potential().detach()
        s, u = torch.linalg.eigh(g["S"])
        X = u * s.rsqrt() @ u.T
        ns, pairs = len(self.eta), float(self.refocc.sum()) / 2

        def cycle(vec):
            parts = [vec[:ns], vec[ns:ns + 3 * self.n].reshape(-1, 3), vec[ns + 3 * self.n:].reshape(-1, 6)]
            parts = [t.detach().requires_grad_(True) for t in parts]
            v = torch.autograd.grad(self.interaction(g, *parts, vpc), parts)
            H = g["H0"] - 0.5 * g["S"] * (v[0][self.ao_sh][:, None] + v[0][self.ao_sh][None])
            for m, pot in ((g["D"], v[1]), (g["Q"], v[2])):
                half = 0.5 * torch.einsum("cmn,nc->mn", m, pot[self.ao_at])
                H = H - half - half.T
            # the interaction's atomic charge potential comes through the shells' (dE/dq_shell)
            eps, C = torch.linalg.eigh(X @ H @ X)
            C = X @ C
            lo, hi = eps[0] - 1, eps[-1] + 1
            for _ in range(200):
                mu = 0.5 * (lo + hi)
                if torch.sigmoid((mu - eps) / KT).sum() < pairs:
                    lo = mu
                else:
                    hi = mu
            f = torch.sigmoid((mu - eps) / KT)
            ent = -2 * (torch.special.xlogy(f, f) + torch.special.xlogy(1 - f, 1 - f)).sum()
            P, W = (C * (2 * f)) @ C.T, (C * (2 * f * eps)) @ C.T
            return torch.cat([t.reshape(-1) for t in self.populations(g, P)]), P, W, ent

        cur, hx, hr = torch.zeros(ns + 9 * self.n, dtype=torch.float64, device=self.dev), [], []
        for _ in range(150):
            raw, P, W, ent = cycle(cur)
            res = raw - cur
            if float(res.norm()) / math.sqrt(len(res)) < 1e-11:
                break
            hx, hr = (hx + [cur])[-9:], (hr + [res])[-9:]
            nxt = cur + 0.4 * res
            if len(hx) > 1:
                dr = torch.stack([hr[-1] - t for t in hr[:-1]], 1)
                dx = torch.stack([hx[-1] - t for t in hx[:-1]], 1)
                c = torch.linalg.lstsq(dr.cpu(), res[:, None].cpu(), driver="gelsd").solution.to(self.dev)
                nxt = nxt - ((dx + 0.4 * dr) @ c)[:, 0]
            cur = nxt
        pop = self.populations(live, P)
        e = (P * live["H0"]).sum() + self.interaction(live, *pop, potential()) + live["rep"] + live["atm"]
        grads = torch.autograd.grad(e - (W * live["S"]).sum(), [x] + points)
        q = torch.zeros(self.n, dtype=torch.float64, device=self.dev).index_add(0, self.sh_at, pop[0].detach())
        return float(e.detach()) - KT * float(ent), q, grads


def exact(case, seed):
    n = float((_orbitals(case)[0] ** 2).sum())
    if case["model"] != "gfn2" or case["spin"] != 1 or case["count"] > 64 or n > 3e5 or _orbitals(case)[0].max() > 256:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    mols, npc = _molecules(case, seed), case["point_charges"]
    pc = _charges_around(mols, npc, np.random.default_rng([seed, 8])) if npc else None
    got, built = [], {}
    for i, (z, xyz) in enumerate(mols):
        key = tuple(int(a) for a in z)
        if key not in built:
            built = {key: _Molecule(z, dev)}
        at = slice(i * npc, (i + 1) * npc)
        got.append(built[key].solve(xyz, *((pc[0][at], pc[1][at]) if npc else ())))
    energies = torch.tensor([g[0] for g in got], dtype=torch.float64)
    by = lambda k: torch.cat([g[2][k] for g in got])  # noqa: E731
    if case["api"] == "torch":
        return {"energies": energies, "positions": by(0), "pc_positions": by(1), "pc_charges": by(2)}
    return {"energies": energies, "forces": -by(0), "charges": torch.cat([g[1] for g in got]), "status": None}
