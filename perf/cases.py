"""The engine's work as its callers ask for it: evaluations on device and host arrays,
atom-level calls, batches of molecules, short MD trajectories and LAMMPS pair-style steps.

Each case names an entry point, a model shape, a precision form and the sizes.  Models are
the seeded synthetic ones the repository's own configurations use (synth/model.py);
structures are jittered lattices, made from the seed.  A model, its engine and its
workspace are what a program keeps between calls, so they are kept per case here too;
inputs are new for every seed.

The engine computes in float32 (its BF16 form with bf16 split operands in the
channel-mixing GEMMs) and widens the sums to float64 on output.  `run` hands the results
on as float32, the precision that they carry, as a float32 simulation program takes them;
rows per edge or per ghost atom are buffers of a fixed capacity, zero behind the last one.
`exact` evaluates the same model in float64 with plain torch operations.
"""
import hashlib
import json
import math
import os
import tempfile

import numpy as np
import torch

import symmetrix_gb300
from symmetrix_gb300 import MACE, save_model_cache
from symmetrix_gb300.lammps import PairAdapter
from symmetrix_gb300.md import MD
from symmetrix_gb300.synth.model import make_model
from symmetrix_gb300.synth.structures import lammps_rank

# Model shapes: the repository's workload models (32 channels: the CPU-runnable case; 64:
# the molecule model; 128: the headline), a 96-channel one (no tensor-core GEMM shape), the
# L_max = 2 form of the precision workload with fewer species, and a model with ZBL
# repulsion and density-normalised blocks.
MODELS = {
    "c32": dict(num_channels=32, species=("H", "C", "O"), r_cut=5.0),
    "c64": dict(num_channels=64, species=("H", "C", "N", "O", "F", "S", "Cl"), r_cut=5.0),
    "c64zd": dict(num_channels=64, species=("H", "C", "O"), r_cut=5.0, zbl=True, density_scaled=True),
    "c96": dict(num_channels=96, species=("H", "C", "O"), r_cut=5.0),
    "c128": dict(num_channels=128, species=("H", "C", "N", "O"), r_cut=5.0),
    "c128l2": dict(num_channels=128, species=("H", "C", "N", "O"), r_cut=6.0, L_max=2),
}
MODEL_SEED = 1
DEVICE = "cuda"
PRECISIONS = ("float32", "bfloat16")
PAIR_MODES = ("no_domain_decomposition", "mpi_message_passing", "no_mpi_message_passing")
MD_STEPS = 10
DT_FS = 0.5
SKIN = 1.0
MASS = {1: 1.008, 6: 12.011, 7: 14.007, 8: 15.999, 9: 18.998, 16: 32.06, 17: 35.45}
KB_EV, ACCEL = 8.617333262e-5, 9.648533212331e-3  # eV/K; (eV/A)/amu in A/fs^2


def listed():
    def case(name, entry, model, precision, atoms, **more):
        return dict(name=name, entry=entry, model=model, precision=precision, atoms=atoms,
                    density=more.pop("density", 0.10), **more)

    return [
        # a small periodic cell stepped by a GPU-resident program: latency of every launch counts
        case("device_64_c32_f32", "device", "c32", "float32", 64, density=0.064),
        # an ordinary box of the molecule model, ragged size
        case("device_999_c64_bf16", "device", "c64", "bfloat16", 999),
        # the headline box in both forms
        case("device_4096_c128_bf16", "device", "c128", "bfloat16", 4096),
        case("device_4096_c128_f32", "device", "c128", "float32", 4096),
        # L_max = 2, cut-off 6 A (the precision workload's model shape), a small and an ordinary box
        case("device_300_c128l2_f32", "device", "c128l2", "float32", 300, density=0.09),
        case("device_2197_c128l2_bf16", "device", "c128l2", "bfloat16", 2197, density=0.09),
        # a large box, a prime number of atoms
        case("device_30011_c128_bf16", "device", "c128", "bfloat16", 30011),
        # the reference evaluator's own call on host arrays
        case("host_4096_c128_bf16", "host", "c128", "bfloat16", 4096),
        # an ASE-like caller: positions in, energy, forces and virial out (neighbour list on the GPU)
        case("atoms_500_c64zd_f32", "atoms", "c64zd", "float32", 500, periodic=True),
        # screening many molecules in one call
        case("molecules_512_c64_bf16", "molecules", "c64", "bfloat16", 512, mol_min=9, mol_max=118),
        # a short trajectory: set-up, neighbour builds, captured steps, state read-out
        case("md_4096_c128_bf16", "md", "c128", "bfloat16", 4096),
        # a LAMMPS step between list rebuilds, the mode with ghost evaluation
        case("pair_1728_c128_f32", "pair", "c128", "float32", 1728, mode="no_mpi_message_passing"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    entry = rng.choice(["device"] * 6 + ["host", "atoms", "molecules", "md", "pair"])
    case = dict(entry=entry, precision=rng.choice(PRECISIONS), density=round(rng.uniform(0.05, 0.12), 4))
    if entry == "device":
        case["model"] = rng.choice(["c32", "c64", "c64zd", "c96", "c128", "c128", "c128l2"])
        case["atoms"] = size(20, 4000 if case["model"] == "c128l2" else 24000)
    elif entry == "host":
        case["model"] = rng.choice(["c32", "c64", "c128"])
        case["atoms"] = size(20, 6000)
    elif entry == "atoms":
        case["model"] = rng.choice(["c32", "c64", "c64zd", "c128"])
        case["atoms"] = size(20, 6000)
        case["periodic"] = rng.random() < 0.7
    elif entry == "molecules":
        case["model"] = rng.choice(["c32", "c64"])
        case["mol_min"] = rng.randint(3, 20)
        case["mol_max"] = rng.randint(30, 120)
        case["atoms"] = size(4, 600)  # molecules
    elif entry == "md":
        case["model"] = rng.choice(["c64", "c128"])
        case["atoms"] = size(200, 5000)
    else:
        case["model"] = rng.choice(["c32", "c64", "c128"])
        case["atoms"] = size(300, 2500)
        case["mode"] = rng.choice(PAIR_MODES)
    return case


# ---------------------------------------------------------------------------
# models and engines
# ---------------------------------------------------------------------------
_models, _engines = {}, {}


def _model(name):
    if name not in _models:
        while len(_models) >= 2:
            _models.pop(next(iter(_models)))
        _models[name] = make_model(seed=MODEL_SEED, **MODELS[name])
    return _models[name]


def _model_file(name):
    """The model's binary cache, written once per machine and package location."""
    where = os.path.join(tempfile.gettempdir(), "smx_perf_models_%d" % os.getuid())
    os.makedirs(where, mode=0o700, exist_ok=True)
    text = os.path.join(where, name + ".json")
    package = hashlib.sha1(os.path.abspath(symmetrix_gb300.__file__).encode()).hexdigest()[:12]
    binary = os.path.join(where, "%s_%s_%d.smxb" % (name, package, os.getpid()))
    if not os.path.exists(text):
        with open(text + ".%d" % os.getpid(), "w") as f:
            f.write(json.dumps(_model(name)))
        os.replace(f.name, text)
    save_model_cache(text, binary)
    return binary


_files = {}


def _engine(case):
    """The engine a program with this work keeps (its schedules are tuned to the work)."""
    key = json.dumps(case, sort_keys=True)
    if key not in _engines:
        while len(_engines) >= 2:
            _engines.pop(next(iter(_engines)))
        name = case["model"]
        if name not in _files:
            _files[name] = _model_file(name)
        _engines[key] = MACE(_files[name], precision=case["precision"])
    return _engines[key]


# ---------------------------------------------------------------------------
# structures
# ---------------------------------------------------------------------------
def _lattice(n, density, g):
    """n random sites of a cubic lattice, jittered: (positions, box length); pairs stay
    about half a lattice constant apart."""
    L = (n / density) ** (1.0 / 3.0)
    m = int(math.ceil(round(n ** (1.0 / 3.0), 9)))
    a = L / m
    site = torch.randperm(m ** 3, generator=g)[:n]
    ijk = torch.stack([site // (m * m), site // m % m, site % m], 1).double()
    return (ijk + 0.5 + (torch.rand(n, 3, generator=g, dtype=torch.float64) - 0.5) * 0.54) * a, L


def _structure(case, seed):
    g = torch.Generator().manual_seed(seed * 1000003 + 17)
    S = len(MODELS[case["model"]]["species"])
    if case["entry"] == "molecules":
        counts = torch.linspace(case["mol_min"], case["mol_max"], case["atoms"]).round().long()
        counts = counts[torch.randperm(len(counts), generator=g)]
        pos = [_lattice(int(c), case["density"], g)[0] for c in counts]
        L = None
        first = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)])
        pos = torch.cat(pos)
    else:
        pos, L = _lattice(case["atoms"], case["density"], g)
        first = None
        if case["entry"] == "atoms" and not case["periodic"]:
            L = None
    species = torch.randint(0, S, (len(pos),), generator=g)
    velocity = torch.randn(len(pos), 3, generator=g, dtype=torch.float64)
    return pos, L, species, velocity, first


def _edges(pos, rc, L=None, mol=None):
    """Full directed neighbour list on the GPU: (i, j, x_j - x_i), grouped by centre."""
    x = pos.to(DEVICE)
    n = len(x)
    if L is not None:
        x = x - L * torch.floor(x / L)
    k = 0 if L is None or L >= 2 * rc else int(math.ceil(rc / L))
    s = torch.arange(-k, k + 1, device=DEVICE, dtype=torch.float64)
    shifts = torch.cartesian_prod(s, s, s) * (L or 0.0)
    out = []
    rows = max(1, int(3e7) // (n * len(shifts)))
    for a in range(0, n, rows):
        d = x[None, :, :] - x[a:a + rows, None, :]
        if L is not None and k == 0:
            d = d - L * torch.round(d / L)
        d = d[:, :, None, :] + shifts
        r2 = (d * d).sum(-1)
        near = (r2 < rc * rc) & (r2 > 1e-16)
        if mol is not None:
            near &= (mol[a:a + rows, None] == mol[None, :])[:, :, None]
        i, j, q = near.nonzero(as_tuple=True)
        out.append((i + a, j, d[i, j, q]))
    return tuple(torch.cat(t) for t in zip(*out))


def _ghost_shell(case):
    rc = MODELS[case["model"]]["r_cut"]
    return (2 * rc if case["mode"] == "no_mpi_message_passing" else rc) + SKIN


def _capacity(case):
    """Rows that a program with this work allocates, the density's count and a margin: edges,
    or for the pair style local and ghost atoms."""
    m = MODELS[case["model"]]
    if case["entry"] == "pair":
        L = (case["atoms"] / case["density"]) ** (1.0 / 3.0)
        return 256 + int(1.3 * case["density"] * (L + 2 * _ghost_shell(case)) ** 3)
    return 256 + int(1.5 * case["atoms"] * case["density"] * 4.0 / 3.0 * math.pi * m["r_cut"] ** 3)


def _pair_graph(case, inputs):
    """Nodes and edges of a pair-style step: node atoms, per edge (node, node of the row
    read, neighbour atom, atom whose force row takes the neighbour's share)."""
    rc = MODELS[case["model"]]["r_cut"]
    x, owner, lists, n = inputs["x"], inputs["local_of"], inputs["lists"], inputs["n"]
    ai = np.repeat(np.arange(len(lists)), [len(v) for v in lists])
    aj = np.concatenate(lists).astype(np.int64)
    d = x[aj] - x[ai]
    near = (d * d).sum(1) < rc * rc
    ai, aj = ai[near], aj[near]
    if case["mode"] != "no_mpi_message_passing":
        target = owner[aj] if case["mode"] == "no_domain_decomposition" else aj
        return np.arange(n), n, ai, owner[aj].astype(np.int64), aj, target
    ghosts = np.unique(aj[(ai < n) & (aj >= n)])
    node_atom = np.concatenate([np.arange(n), ghosts])
    node_of = np.full(len(x), -1)
    node_of[node_atom] = np.arange(len(node_atom))
    keep = node_of[ai] >= 0
    ai, aj = ai[keep], aj[keep]
    return node_atom, n, node_of[ai], np.maximum(node_of[aj], 0), aj, aj


def _pair_inputs(case, seed):
    pos, L, species, _, _ = _structure(case, seed)
    rc = MODELS[case["model"]]["r_cut"]
    ghosts = case["mode"] == "no_mpi_message_passing"
    x, local_of, lists = lammps_rank(pos.numpy(), L, rc + SKIN, _ghost_shell(case), ghost_lists=ghosts)
    return dict(x=x, local_of=local_of, lists=lists, n=len(pos), species=species.numpy()[local_of].astype(np.int32))


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    eng = _engine(case)
    entry = case["entry"]
    state = dict(entry=entry, eng=eng)
    rc = MODELS[case["model"]]["r_cut"]
    if entry == "pair":
        inp = _pair_inputs(case, seed)
        state["pair"] = PairAdapter(eng, np.arange(eng.num_elements, dtype=np.int32), case["mode"])
        ghosts = case["mode"] == "no_mpi_message_passing"
        n, nall = inp["n"], len(inp["x"])
        state["args"] = (inp["x"], inp["species"] + 1, None if ghosts else inp["local_of"],
                         np.arange(nall if ghosts else n), inp["lists"])
        state["gnum"] = nall - n if ghosts else 0
        state["forces"] = np.zeros((_capacity(case), 3), dtype=np.float32)
        # LAMMPS's setup step hands the lists over; the steps that follow keep them
        state["pair"].compute(*state["args"], neigh_changed=True, eflag_atom=True, gnum=state["gnum"])
        return state
    pos, L, species, velocity, first = _structure(case, seed)
    sp = species.numpy().astype(np.int32)
    if entry in ("device", "host"):
        i, j, d = _edges(pos, rc, L)
        n = len(pos)
        t = species.to(DEVICE).int()
        count = torch.bincount(i, minlength=n).int()
        arrays = [t, count, j.int(), t[j].contiguous(), d.contiguous(), d.norm(dim=1)]
        if entry == "host":
            state["args"] = [n] + [a.cpu().numpy() for a in arrays]
            state["forces"] = np.zeros(3 * _capacity(case), dtype=np.float32)
            return state
        state.update(n=n, E=len(j), arrays=arrays, stream=torch.cuda.ExternalStream(eng.stream),
                     energies=torch.empty(n, dtype=torch.float64, device=DEVICE),
                     forces=torch.zeros(_capacity(case), 3, dtype=torch.float64, device=DEVICE))
        return state
    if entry == "atoms":
        state["args"] = (pos.numpy(), sp, L)
    elif entry == "molecules":
        cut = first.tolist()
        x = pos.numpy()
        state["args"] = [(x[a:b], sp[a:b]) for a, b in zip(cut[:-1], cut[1:])]
    else:
        mass = np.array([MASS[z] for z in eng.atomic_numbers])[sp]
        v = velocity.numpy() * np.sqrt(KB_EV * 300.0 / mass * ACCEL)[:, None]
        state["args"] = dict(positions=pos.numpy(), species=sp, masses=mass, box=np.full(3, L), velocities=v,
                             dt=DT_FS, skin=SKIN, rebuild_every=MD_STEPS)
    return state


def run(state):
    eng, entry = state["eng"], state["entry"]
    if entry == "device":
        e, f = state["energies"], state["forces"]
        t, count, j, tj, d, r = (a.data_ptr() for a in state["arrays"])
        eng.compute_device(state["n"], t, count, j, tj, state["E"], d, r, e.data_ptr(), f.data_ptr())
        with torch.cuda.stream(state["stream"]):
            return {"node_energies": e.float(), "node_forces": f.float()}
    if entry == "host":
        eng.compute_node_energies_forces(*state["args"])
        f = state["forces"]
        f[:len(eng.node_forces)] = eng.node_forces
        return {"node_energies": eng.node_energies.astype(np.float32), "node_forces": f}
    if entry == "atoms":
        energy, node, forces, virial = eng.compute_atoms(*state["args"])
        return {"energy": np.float32(energy), "node_energies": node.astype(np.float32),
                "forces": forces.astype(np.float32), "virial": virial.astype(np.float32)}
    if entry == "molecules":
        energy, node, forces = eng.compute_molecules(state["args"])
        return {"energies": energy.astype(np.float32), "node_energies": np.concatenate(node).astype(np.float32),
                "forces": np.concatenate(forces).astype(np.float32)}
    if entry == "md":
        md = MD(eng, **state["args"])
        md.run(MD_STEPS)
        md.sync()
        s = md.state()
        return {"energy": np.float32(s["potential_energy"]),
                **{k: s[k].astype(np.float32) for k in ("positions", "velocities", "forces", "virial")}}
    energy, f, eatom, virial = state["pair"].compute(*state["args"], neigh_changed=False, eflag_atom=True,
                                                     gnum=state["gnum"])
    state["forces"][:len(f)] = f
    return {"energy": np.float32(energy), "forces": state["forces"], "node_energies": eatom.astype(np.float32),
            "virial": virial.astype(np.float32)}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _shape(case):
    """(layer-0 nodes, layer-0 edges, layer-1 nodes, layer-1 edges) of one evaluation, from the density."""
    rc = MODELS[case["model"]]["r_cut"]
    n = case["atoms"]
    per = case["density"] * 4.0 / 3.0 * math.pi * rc ** 3
    if case["entry"] == "molecules":
        n *= (case["mol_min"] + case["mol_max"]) / 2.0
        per = min(per, (case["mol_min"] + case["mol_max"]) / 2.0) * 0.6
    n0 = n
    if case["entry"] == "pair" and case["mode"] == "no_mpi_message_passing":
        L = (n / case["density"]) ** (1.0 / 3.0)
        n0 = n * ((L + 2 * rc) / L) ** 3
    return n0, n0 * per, n, n * per


def work(case):
    """Bytes: every input, table and weight once, every output once.  Operations: the
    per-edge radials, harmonics products and tensor products with their adjoints, the
    symmetric contractions and the channel mixing, of both directions."""
    m = MODELS[case["model"]]
    C, S, L2 = m["num_channels"], len(m["species"]), m.get("L_max", 1) == 2
    nLM, n_lme, ni, npth, T0 = (9, 71, 17, 243, 850) if L2 else (4, 40, 10, 88, 400)
    n0, e0, n1, e1 = _shape(case)
    passes = MD_STEPS + 1 if case["entry"] == "md" else 1
    flops = e0 * C * (56 + 198) + e1 * C * (24 * ni + 6 * npth) + n0 * C * 14 * T0
    flops += n1 * C * C * 4 * n_lme + n0 * C * C * 4 * nLM + n1 * C * 8 * C
    tables = (S * S * 4 + S * (S + 1) // 2 * ni) * 199 * C * 16 + S * (T0 + 111) * C * 4 + (n_lme + 2 * nLM + S) * C * C * 4
    if case["entry"] in ("device", "host"):
        io = e0 * (8 + 32 + 24) + n0 * (8 + 8)
    else:
        io = (n0 if case["entry"] == "pair" else n1) * (24 + 4 + 24 + 8)
        io += e1 * 4 * 1.7 if case["entry"] == "pair" else 0
    return {"bytes": float(tables + io), "flops": float(flops * passes)}


# ---------------------------------------------------------------------------
# the same model in float64, in plain torch
# ---------------------------------------------------------------------------
def _harmonics(v):
    """Real spherical harmonics up to l = 3 in the (z, x, y) axes, |Y_00| = 1, [E, 16]."""
    u = v / v.norm(dim=1, keepdim=True)
    y, z, x = u.unbind(1)
    s = math.sqrt
    xx, yy, zz = x * x, y * y, z * z
    return torch.stack([
        torch.ones_like(x), s(3) * y, s(3) * z, s(3) * x, s(15) * x * y, s(15) * y * z, s(5) / 2 * (2 * zz - xx - yy),
        s(15) * x * z, s(15) / 2 * (xx - yy), s(35 / 8) * y * (3 * xx - yy), s(105) * x * y * z,
        s(21 / 8) * y * (4 * zz - xx - yy), s(7) / 2 * z * (2 * zz - 3 * xx - 3 * yy), s(21 / 8) * x * (4 * zz - xx - yy),
        s(105) / 2 * z * (xx - yy), s(35 / 8) * x * (xx - 3 * yy)], 1)


class _Float64:
    def __init__(self, name):
        m = _model(name)

        def t(v, *shape):
            v = torch.tensor(v, dtype=torch.float64, device=DEVICE)
            return v.reshape(shape) if shape else v

        self.m = m
        S, C = m["num_elements"], m["num_channels"]
        self.S, self.C, self.L = S, C, m["L_max"]
        self.h = m["radial_spline_h"]
        self.spline = [tuple(t(m["radial_spline_%s_%d" % (k, q)]).transpose(1, 2).contiguous()
                             for k in ("values", "derivs")) for q in (0, 1)]  # [pair][knot][spline]
        self.H0, self.A0 = t(m["H0_weights"], S, C), t(m["A0_weights"], S, 4, C, C)
        self.H1 = t(m["H1_weights"], self.L + 1, C, C)
        self.P0 = [self._poly(m["M0_monomials"][str(q)], [m["M0_weights"][str(s)][str(q)] for s in range(S)])
                   for q in range((self.L + 1) ** 2)]
        self.P1 = self._poly(m["M1_monomials"], [m["M1_weights"][str(s)] for s in range(S)])
        self.l, self.l1, self.l2 = m["Phi1_l"], m["Phi1_l1"], m["Phi1_l2"]
        n_lme = sum(2 * l + 1 for l in self.l)
        n_p = sum((2 * a + 1) * (2 * b + 1) for a, b in zip(self.l1, self.l2))
        self.cg = torch.zeros(n_lme, n_p, dtype=torch.float64, device=DEVICE)
        for r, p, v in zip(m["Phi1_lme"], m["Phi1_lelm1lm2"], m["Phi1_clebsch_gordan"]):
            self.cg[r, p] += v
        self.ne = [self.l.count(q) for q in range(4)]
        self.A1 = [t(m["A1_weights"][q], self.ne[q] * C, C) for q in range(4)]
        self.H2a, self.H2b = t(m["H2_weights_for_H1"], S, C, C), t(m["H2_weights_for_M1"], C, C)
        self.r1, self.w1, self.w2 = t(m["readout_1_weights"], C), t(m["readout_2_weights_1"], -1, C), t(m["readout_2_weights_2"], -1)
        self.e0 = t(m["atomic_energies"], S)
        self.density = [tuple(t(m["A%d_spline_%s" % (q, k)])[..., None] for k in ("values", "derivs"))
                        if m["A%d_scaled" % q] else None for q in (0, 1)]

    def _poly(self, monomials, weights):
        index = torch.tensor([list(k) + [16] * (3 - len(k)) for k in monomials], device=DEVICE)
        c = torch.tensor([[w[str(k)] for k in range(self.C)] for w in weights], dtype=torch.float64, device=DEVICE)
        return index, c.transpose(1, 2).contiguous()  # [S][T][C]

    def poly(self, P, x, t):
        x = torch.cat([x, torch.ones_like(x[:, :1])], 1)
        i, c = P
        return (c[t] * x[:, i[:, 0]] * x[:, i[:, 1]] * x[:, i[:, 2]]).sum(1)

    def radial(self, table, a, b, r):
        """Hermite cubics on uniform knots of the unordered species pair at r."""
        v, d = table
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        p = lo * (2 * self.S - lo - 1) // 2 + hi
        n = (r.detach() / self.h).long().clamp(0, v.shape[1] - 2)
        x = (r / self.h - n.to(r.dtype))[:, None]
        return ((1 + 2 * x) * (1 - x) ** 2 * v[p, n] + x * (1 - x) ** 2 * self.h * d[p, n]
                + x * x * (3 - 2 * x) * v[p, n + 1] + x * x * (x - 1) * self.h * d[p, n + 1])

    def edges0(self, n, t, i, tj, v):
        """Layer-0 sums [n, 16, C] of edges (centre i of n nodes, neighbour species tj, vector v)."""
        r, Y = v.norm(dim=1), _harmonics(v)
        R = self.radial(self.spline[0], t[i], tj, r).reshape(-1, 4, self.C) * self.H0[tj][:, None]
        out = []
        for l in range(4):
            phi = torch.zeros(n, 2 * l + 1, self.C, dtype=torch.float64, device=DEVICE).index_add(
                0, i, Y[:, l * l:(l + 1) ** 2, None] * R[:, None, l])
            mixed = torch.zeros_like(phi)
            for s in range(self.S):
                mixed = torch.where((t == s)[:, None, None], phi @ self.A0[s, l], mixed)
            out.append(mixed)
        return torch.cat(out, 1) / self.scale(0, n, t, i, tj, r)

    def scale(self, layer, n, t, i, tj, r):
        if self.density[layer] is None:
            return 1.0
        s = self.radial(self.density[layer], t[i], tj, r)[:, 0]
        return (1.0 + torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add(0, i, s))[:, None, None]

    def nodes0(self, t, A0):
        M0 = torch.stack([self.poly(P, A0, t) for P in self.P0], 1)
        return torch.cat([M0[:, l * l:(l + 1) ** 2] @ self.H1[l] for l in range(self.L + 1)], 1)

    def edges1(self, n, t, i, tj, v, h):
        """Node energies of n nodes' layer 1 without the linear readout: A1 [n, 16, C]; h: the neighbours' H1."""
        r, Y = v.norm(dim=1), _harmonics(v)
        R = self.radial(self.spline[1], t[i], tj, r).reshape(-1, len(self.l), self.C)
        rows = []
        for q, (a, b) in enumerate(zip(self.l1, self.l2)):
            y, g = Y[:, a * a:(a + 1) ** 2], R[:, None, q] * h[:, b * b:(b + 1) ** 2]
            rows.append(torch.zeros(n, 2 * a + 1, 2 * b + 1, self.C, dtype=torch.float64, device=DEVICE).index_add(
                0, i, y[:, :, None, None] * g[:, None]).reshape(n, -1, self.C))
        phi = torch.einsum("rp,npc->nrc", self.cg, torch.cat(rows, 1))
        A, at = [], 0
        for l in range(4):
            k = (2 * l + 1) * self.ne[l]
            A.append(phi[:, at:at + k].reshape(n, 2 * l + 1, -1) @ self.A1[l])
            at += k
        return torch.cat(A, 1) / self.scale(1, n, t, i, tj, r)

    def energies(self, t, A1, H10):
        M1 = self.poly(self.P1, A1, t)
        H2 = M1 @ self.H2b
        for s in range(self.S):
            H2 = H2 + torch.where((t == s)[:, None], H10 @ self.H2a[s], torch.zeros_like(H10))
        act = self.m["readout_2_scale_factor"] * torch.nn.functional.silu(H2 @ self.w1.T)
        return self.e0[t] + H10 @ self.r1 + act @ self.w2

    def zbl(self, n, t, i, tj, v):
        m = self.m
        if not m["has_zbl"]:
            return 0.0
        Z = torch.tensor(m["atomic_numbers"], device=DEVICE)
        zi, zj = Z[t[i]].double(), Z[tj].double()
        radius = torch.tensor(m["zbl_covalent_radii"], dtype=torch.float64, device=DEVICE)
        r = v.norm(dim=1)
        a = m["zbl_a_prefactor"] * 0.529 / (zi ** m["zbl_a_exp"] + zj ** m["zbl_a_exp"])
        phi = sum(c * torch.exp(k * r / a) for c, k in zip(m["zbl_c"], (-3.2, -0.9423, -0.4028, -0.2016)))
        rm, p = radius[Z[t[i]]] + radius[Z[tj]], m["zbl_p"]
        x = r / rm
        env = 1 - (p + 1) * (p + 2) / 2 * x ** p + p * (p + 2) * x ** (p + 1) - p * (p + 1) / 2 * x ** (p + 2)
        e = torch.where(x < 1, 0.5 * 14.3996 * zi * zj / r * phi * env, torch.zeros_like(r))
        return torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add(0, i, e)

    def evaluate(self, t, i, j, tj, v, n1=None):
        """Node energies of the first n1 nodes and -dE/dv of every edge (edges grouped by centre i)."""
        n = len(t)
        n1 = n if n1 is None else n1
        first = torch.searchsorted(i, torch.arange(n + 1, device=DEVICE)).tolist()
        budget = int(2.0e9 / (self.C * 8 * len(self.cg.T)))  # edges whose widest rows take about 2 GB
        cuts, a = [], 0
        while a < n:
            b = a + 1
            while b < n and b - a < 1500 and first[b + 1] - first[a] <= budget:
                b += 1
            cuts.append((a, b))
            a = b
        # the layer-1 cuts end at n1
        cuts1 = [(a, min(b, n1)) for a, b in cuts if a < n1]
        force = torch.zeros_like(v)
        H1 = torch.zeros(n, (self.L + 1) ** 2, self.C, dtype=torch.float64, device=DEVICE)
        with torch.no_grad():
            for a, b in cuts:
                e = slice(first[a], first[b])
                H1[a:b] = self.nodes0(t[a:b], self.edges0(b - a, t[a:b], i[e] - a, tj[e], v[e]))
        E, dH1 = torch.zeros(n1, dtype=torch.float64, device=DEVICE), torch.zeros_like(H1)
        for a, b in cuts1:
            e = slice(first[a], first[b])
            w, h = v[e].clone().requires_grad_(), H1[j[e]].requires_grad_()
            own = H1[a:b, 0].clone().requires_grad_()
            A1 = self.edges1(b - a, t[a:b], i[e] - a, tj[e], w, h)
            en = self.energies(t[a:b], A1, own) + self.zbl(b - a, t[a:b], i[e] - a, tj[e], w)
            gw, gh, go = torch.autograd.grad(en.sum(), (w, h, own), allow_unused=True)
            E[a:b] = en.detach()
            if gw is not None:
                force[e] -= gw
                dH1.index_add_(0, j[e], gh)
            dH1[a:b, 0] += go
        for a, b in cuts:
            e = slice(first[a], first[b])
            w = v[e].clone().requires_grad_()
            out = self.nodes0(t[a:b], self.edges0(b - a, t[a:b], i[e] - a, tj[e], w))
            force[e] -= torch.autograd.grad((out * dH1[a:b]).sum(), w)[0]
        return E, force


_float64 = {}


def exact(case, seed):
    entry = case["entry"]
    if case["model"] not in _float64:
        _float64.clear()
        _float64[case["model"]] = _Float64(case["model"])
    ref = _float64[case["model"]]
    rc = MODELS[case["model"]]["r_cut"]
    cuda = lambda a: torch.as_tensor(a).to(DEVICE)  # noqa: E731
    if entry == "pair":
        inp = _pair_inputs(case, seed)
        node_atom, n1, i, row, aj, target = (cuda(a) for a in _pair_graph(case, inp))
        x, sp = cuda(inp["x"]), cuda(inp["species"]).long()
        v = x[aj] - x[node_atom[i]]
        E, f = ref.evaluate(sp[node_atom], i, row, sp[aj], v, int(n1))
        F = x.new_zeros(_capacity(case), 3).index_add(0, target, f).index_add(0, node_atom[i], -f)
        W = v.T @ f
        virial = torch.stack([W[0, 0], W[1, 1], W[2, 2], (W[0, 1] + W[1, 0]) / 2, (W[0, 2] + W[2, 0]) / 2,
                              (W[1, 2] + W[2, 1]) / 2])
        return {"energy": E.sum(), "forces": F, "node_energies": E, "virial": virial}
    pos, L, species, velocity, first = _structure(case, seed)
    t = species.to(DEVICE)
    n = len(t)
    mol = None
    if first is not None:
        mol = torch.repeat_interleave(torch.arange(len(first) - 1), first[1:] - first[:-1]).to(DEVICE)

    def atoms(x):
        i, j, v = _edges(x, rc, L, mol)
        E, f = ref.evaluate(t, i, j, t[j], v)
        F = torch.zeros(n, 3, dtype=torch.float64, device=DEVICE).index_add(0, j, f).index_add(0, i, -f)
        return E, f, F, v.T @ f

    if entry == "md":
        mass = torch.tensor([MASS[z] for z in ref.m["atomic_numbers"]], dtype=torch.float64, device=DEVICE)[t][:, None]
        x = pos.to(DEVICE)
        vel = velocity.to(DEVICE) * torch.sqrt(KB_EV * 300.0 / mass * ACCEL)
        E, _, F, W = atoms(x)
        for _ in range(MD_STEPS):
            vel = vel + 0.5 * DT_FS * ACCEL * F / mass
            x = x + DT_FS * vel
            E, _, F, W = atoms(x)
            vel = vel + 0.5 * DT_FS * ACCEL * F / mass
        return {"energy": E.sum(), "positions": None, "velocities": vel, "forces": F, "virial": W}
    E, f, F, W = atoms(pos)
    if entry in ("device", "host"):
        f = torch.cat([f, f.new_zeros(_capacity(case) - len(f), 3)])
        return {"node_energies": E, "node_forces": f if entry == "device" else f.reshape(-1)}
    if entry == "atoms":
        return {"energy": E.sum(), "node_energies": E, "forces": F, "virial": W}
    return {"energies": torch.zeros(len(first) - 1, dtype=torch.float64, device=DEVICE).index_add(0, mol, E),
            "node_energies": E, "forces": F}
