"""The calls that programs built on this framework spend their time in, as timed cases.

Each case is one pass through the public entry points, over the range of sizes, modes and options that the
repository's own configurations use:

  forces    an external integrator or a force-matching set asks for the forces of one structure
  energy    a line search or a scoring run asks for the energy terms of one structure
  minimize  L-BFGS iterations on one structure (what co-translational growth does after every residue)
  dynamics  a block of BAOAB steps of one structure or of an ensemble, from a restored state to the frame written
            after it (plain or learned Born radii, with and without cutoffs, surface term, SHAKE, exit tunnel)
  remd      rounds of device-side replica exchange

Structures.  "coil" systems are windows of the benchmark's relaxed 300-residue chain (several windows joined by
superposing the backbone of the residue they share, for longer chains); "fold" systems are the native NMR folds that the
tests use: Trp-cage (20 residues) and insulin (51 residues in two chains), the latter also as assemblies of several copies
packed side by side.  A case's sizes fix its windows; every seed gives other orientations, thermal displacements,
velocities and noise.

Pair forces are single-precision sums by design, and frames and force sets are stored in single precision, so forces and
frames are returned as float32; energies are double precision throughout and stay so.
"""
import functools
import math
import os

import numpy as np
import torch

import origami_b200 as og
from origami_b200 import lgb
from origami_b200.cotranslate import CylindricalTunnel
from origami_b200.minimize import MinimizeOptions, lbfgs

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")


def _case(name, kind, system, residues, replicas=1, cutoff=False, sasa=False, shake=False, dt=1.0, steps=0,
          radii="plain", tunnel=False, uneven=False, tuned=False):
    return {"name": name, "kind": kind, "system": system, "residues": residues, "replicas": replicas,
            "cutoff": cutoff, "sasa": sasa, "shake": shake, "dt": dt, "steps": steps, "radii": radii,
            "tunnel": tunnel, "uneven": uneven, "tuned": tuned}


def listed():
    return [
        # the smallest call there is: forces of a 300-atom miniprotein with the reference's cutoffs (the defaults)
        _case("force_trpcage", "forces", "fold", 20, cutoff=True),
        # forces of a mid-sized chain, every pair
        _case("force_coil_120", "forces", "coil", 120),
        # one line-search trial: the FP64 energy of a 4.7k-atom chain
        _case("energy_coil_300", "energy", "coil", 300),
        # ten L-BFGS iterations on that chain: what dominates a co-translational run
        _case("minimize_coil_300", "minimize", "coil", 300, steps=10),
        # a single small trajectory (the 20-residue configuration): a launch-bound step
        _case("langevin_trpcage", "dynamics", "fold", 20, dt=1.0, steps=100),
        # a single folded protein with cutoffs, surface term and SHAKE (the 60-residue configuration)
        _case("langevin_insulin", "dynamics", "fold", 51, cutoff=True, sasa=True, shake=True, dt=2.0, steps=50),
        # a whole chain in the exit tunnel (the 1 000-residue co-translation configuration)
        _case("growth_coil_1000", "dynamics", "coil", 1000, sasa=True, dt=1.0, steps=10, tunnel=True),
        # parallel tempering, 64 replicas of 40 residues, swaps on the device
        _case("remd_64x40", "remd", "coil", 40, replicas=64, shake=True, dt=2.0, steps=50, tuned=True),
        # 256 unequal chains of 10 to 80 residues in one engine
        _case("chains_256", "dynamics", "coil", 80, replicas=256, shake=True, dt=2.0, steps=10, uneven=True, tuned=True),
        # assemblies of six insulins (4.7k atoms, compact), the reference's cutoffs and the surface term
        _case("assembly_16x306_cutoff", "dynamics", "fold", 306, replicas=16, cutoff=True, sasa=True, shake=True, dt=2.0,
              steps=4, tuned=True),
        # the benchmark's workload, plain Born radii
        _case("ensemble_64x300", "dynamics", "coil", 300, replicas=64, sasa=True, shake=True, dt=2.0, steps=3, tuned=True),
        # the benchmark's workload, learned Born radii
        _case("learned_64x300", "dynamics", "coil", 300, replicas=64, sasa=True, shake=True, dt=2.0, steps=3,
              radii="learned", tuned=True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["forces", "energy", "minimize", "dynamics", "dynamics", "dynamics", "dynamics", "remd"])
    cutoff = rng.random() < 0.4
    if rng.random() < 0.3:
        system, residues = "fold", rng.choice([20, 51, 102, 153, 204, 255, 306])
    else:
        system, residues = "coil", _log_int(rng, 10, 300)
    if kind in ("forces", "energy", "minimize"):
        if system == "coil" and kind != "energy":
            residues = _log_int(rng, 10, 600)
        c = _case("", kind, system, residues, cutoff=cutoff, sasa=rng.random() < 0.3,
                  steps=rng.randint(4, 10) if kind == "minimize" else 0)
    elif kind == "remd":
        residues = 20 if system == "fold" else _log_int(rng, 10, 60)
        c = _case("", kind, system, residues, replicas=rng.randint(4, 64), cutoff=cutoff, shake=True, dt=2.0,
                  steps=rng.randint(20, 50), tuned=rng.random() < 0.5)
    else:
        # replicas x atoms^2 stays below the benchmark's
        most = max(1, min(64, int(64 * (300 / residues) ** 2)))
        replicas = _log_int(rng, 1, most)
        shake = rng.random() < 0.6
        c = _case("", kind, system, residues, replicas=replicas, cutoff=cutoff, sasa=rng.random() < 0.5, shake=shake,
                  dt=2.0 if shake else 1.0, steps=rng.randint(2, 3) if replicas * residues > 2000 else rng.randint(5, 20),
                  radii="learned" if rng.random() < 0.25 else "plain", tunnel=replicas == 1 and rng.random() < 0.3,
                  uneven=system == "coil" and rng.random() < 0.3, tuned=replicas > 1 and rng.random() < 0.5)
    del c["name"]
    return c


# ------------------------------------------------------------ structures

@functools.lru_cache(maxsize=None)
def _bench_chain():
    """(sequence, atoms per residue, names, coordinates) of the benchmark's relaxed chain."""
    z = np.load(os.path.join(GOLDEN, "bench_chain_300.npz"))
    seq, xyz = str(z["seq"]), z["xyz"]
    chain = og.Chain.build(seq)
    info = [chain.atom_info(i) for i in range(chain.n_atoms)]
    counts = np.bincount([r for r, _, _ in info], minlength=len(seq))
    return seq, counts, [n for _, _, n in info], xyz


@functools.lru_cache(maxsize=None)
def _native(name):
    z = np.load(os.path.join(GOLDEN, "host_model.npz"))
    g = {k: z["%s/%s" % (name, k)] for k in ("seq", "chains", "counts", "names", "elements", "xyz")}
    return str(g["seq"]), str(g["chains"]), g["counts"], [str(n) for n in g["names"]], g["elements"], g["xyz"]


def _rotation(rng):
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    q = q * np.sign(np.diag(r))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return q


def _superpose(mobile, target):
    """(rotation, shift): mobile @ rotation + shift is nearest to target (least squares)."""
    cm, ct = mobile.mean(0), target.mean(0)
    u, _, vt = np.linalg.svd((mobile - cm).T @ (target - ct))
    d = np.diag([1.0, 1.0, np.sign(np.linalg.det(u @ vt))])
    rot = u @ d @ vt
    return rot, ct - cm @ rot


def _coil(n, rng):
    """A relaxed chain of n residues: (residues, chains, atoms per residue, names, elements, coordinates)."""
    seq, counts, names, xyz = _bench_chain()
    ends = np.concatenate([[0], np.cumsum(counts)])
    out_seq, out_counts, out_names, out_xyz = "", [], [], np.zeros((0, 3))
    back = None  # N, CA, C of the last residue so far
    while len(out_seq) < n:
        # a joined window brings one residue more than it adds: the shared one
        want = min(n - len(out_seq) + (back is not None), 250 if n > len(seq) else len(seq))
        a = int(rng.integers(0, len(seq) - want + 1))
        x = xyz[ends[a]:ends[a + want]]
        nm = names[ends[a]:ends[a + want]]
        first = 0
        if back is not None:
            head = {m: x[k] for k, m in enumerate(nm[:counts[a]])}
            rot, shift = _superpose(np.array([head["N"], head["CA"], head["C"]]), back)
            x = x @ rot + shift
            first = 1
        skip = int(counts[a]) if first else 0
        out_seq += seq[a + first:a + want]
        out_counts += [int(c) for c in counts[a + first:a + want]]
        out_names += nm[skip:]
        out_xyz = np.concatenate([out_xyz, x[skip:]])
        tail = {m: out_xyz[len(out_xyz) - out_counts[-1] + k] for k, m in enumerate(out_names[-out_counts[-1]:])}
        back = np.array([tail["N"], tail["CA"], tail["C"]])
    return out_seq, "A" * len(out_seq), np.array(out_counts), out_names, None, out_xyz


def _fold(n, rng):
    """Trp-cage for 20 residues, else n / 51 insulins side by side, each in its own orientation."""
    if n == 20:
        return _native("1L2Y")
    seq, chains, counts, names, elements, xyz = _native("2HIU")
    copies = max(1, n // len(seq))
    x0 = xyz - xyz.mean(0)
    radius = np.sqrt((x0 ** 2).sum(1)).max()
    side = int(math.ceil(copies ** (1.0 / 3.0)))
    ids = [chr(ord("A") + k) if k < 26 else chr(ord("a") + k - 26) for k in range(52)]
    letters = sorted(set(chains))
    xs, ch = [], ""
    for k in range(copies):
        cell = np.array([k % side, (k // side) % side, k // (side * side)])
        xs.append(x0 @ _rotation(rng) + cell * (2.0 * radius + 1.0))
        ch += "".join(ids[(k * len(letters) + letters.index(c)) % 52] for c in chains)
    return (seq * copies, ch, np.tile(counts, copies), list(names) * copies, np.tile(elements, copies),
            np.concatenate(xs))


def _systems(case, seed):
    """The case's systems: [(chain, coordinates)]."""
    rng = np.random.default_rng([int(seed) & 0x7FFFFFFF, case["residues"], case["replicas"]])
    pick = np.random.default_rng([case["residues"], case["replicas"]])  # the atom counts are the case's, not the seed's
    build = _coil if case["system"] == "coil" else _fold
    out, chain = [], None
    for _ in range(case["replicas"]):
        if chain is None or case["uneven"]:
            n = int(pick.integers(min(10, case["residues"]), case["residues"] + 1)) if case["uneven"] else case["residues"]
            s, ch, counts, names, elements, base = build(n, pick)
            chain = og.Chain.from_structure(s, counts, names, base, elements=elements, chains=ch)
        x = (base - base.mean(0)) @ _rotation(rng) + 0.004 * rng.standard_normal(base.shape)
        out.append((chain, np.ascontiguousarray(x)))
    return out


def _params(case, seed):
    make = og.Params if case["cutoff"] else og.Params.all_pairs
    return make(dt_fs=case["dt"], friction_ps_inv=2.0, constrain_h_bonds=case["shake"], include_sasa=case["sasa"],
                sasa_gamma_scale=0.25, born_mode=1 if case["radii"] == "learned" else 0, seed=int(seed) & 0xFFFF)


def _network(seed):
    """Network parameters like a trained one's: the linear path carries log(rho~ / R_cfa), the hidden layers a small
    correction."""
    p = lgb.init_params(seed)
    rng = np.random.default_rng(seed)
    p[lgb.OFF_W4:lgb.OFF_B4] = 1e-5 * rng.standard_normal(lgb.HIDDEN).astype(np.float32)
    p[lgb.OFF_V + 9] = 1.0
    return p


def _pinned(shape, dtype):
    return torch.empty(shape, dtype={np.dtype(np.float64): torch.float64, np.dtype(np.int64): torch.int64,
                                     np.dtype(np.int32): torch.int32}[np.dtype(dtype)], pin_memory=True).numpy()


# ------------------------------------------------------------ the cases

def prepare(case, seed):
    systems = _systems(case, seed)
    eng = og.Engine(_params(case, seed))
    n = len(systems)
    for k, (chain, x) in enumerate(systems):
        t = 280.0 * (420.0 / 280.0) ** (k / max(n - 1, 1)) if case["kind"] == "remd" else 310.0
        eng.add_system(chain, x, t)
    eng.finalize()
    state = {"case": case, "engine": eng, "chains": [c for c, _ in systems], "x": systems[0][1]}
    if case["radii"] == "learned":
        lgb.set_params(eng, _network(int(seed) & 0xFFFF))
        lgb.set_judge(eng, 500, 1e-3)
    if case["tunnel"]:
        _tunnel(systems[0][1]).apply_to(eng)
    if case["kind"] in ("dynamics", "remd"):
        for k in range(n):
            eng.init_velocities(k, int(seed) + k * 0xC0FFEE, remove_com=False)
        parts = ("positions", "velocities")
        whole = eng.state_buffers(alloc=_pinned)
        state["start"] = {k: whole[k] for k in parts}
        eng.get_state(out=state["start"], parts=parts)
        whole = eng.state_buffers(alloc=_pinned)
        state["frame"] = {k: whole[k] for k in parts}
    if case["tuned"]:
        eng.autotune()
    return state


def _tunnel(x):
    """The ribosome's exit tunnel (radius 10 A, length 80 A) around the chain's end."""
    end = x[-40:].mean(0)
    axis = end - x[-400:].mean(0)
    axis = axis / max(float(np.linalg.norm(axis)), 1e-9)
    return CylindricalTunnel(tuple(end - 20.0 * axis), tuple(axis), 10.0, 80.0, 0.1)


def run(state):
    case, eng = state["case"], state["engine"]
    if case["kind"] == "forces":
        eng.set_positions(0, state["x"])
        return eng.total_force(0).astype(np.float32)
    if case["kind"] == "energy":
        eng.set_positions(0, state["x"])
        return eng.energies(0)
    if case["kind"] == "minimize":
        eng.set_positions(0, state["x"])
        r = lbfgs(eng, 0, MinimizeOptions(max_steps=case["steps"]))
        return {"positions": eng.positions(0).astype(np.float32), "initial_energy": r.initial_energy,
                "final_energy": np.float32(r.final_energy), "max_force": np.float32(r.max_force), "steps": r.steps}
    eng.set_state(state["start"])
    out = {}
    if case["kind"] == "remd":
        out = eng.remd_run(2, case["steps"], 0xDEADBEEF)
    else:
        eng.step(case["steps"])
    eng.get_state(out=state["frame"], parts=("positions", "velocities"))
    out.update({k: v.astype(np.float32) for k, v in state["frame"].items()})
    return out


# atoms per residue, C and S atoms per residue, atoms within 10 and 20 A of one
ATOMS, SURFACE, NEAR_10, NEAR_20 = 15.5, 5.2, 220, 900


def work(case):
    n = case["residues"] * ATOMS
    if case["uneven"]:
        n *= 0.5 + 5.0 / case["residues"]
    reps = case["replicas"]
    pairs = n * (n - 1) / 2
    near10, near20 = (min(pairs, n * NEAR_10 / 2), min(pairs, n * NEAR_20 / 2)) if case["cutoff"] else (pairs, pairs)
    # per force evaluation: descreening and pair force (the repository's flop convention), bonded terms, surface term,
    # learned radii (the network's products) in place of the descreening pass
    force = 55 * near10 + 400 * n + (2e4 * n * SURFACE / ATOMS if case["sasa"] else 0.0)
    force += 86e3 * n if case["radii"] == "learned" else 60 * near20
    energy = 100 * near20 + 60 * pairs + 300 * n + (2e4 * n * SURFACE / ATOMS if case["sasa"] else 0.0)
    evals = {"forces": (1, 0), "energy": (0, 1), "minimize": (case["steps"], case["steps"] + 1),
             "dynamics": (case["steps"] + 1, 0), "remd": (2 * case["steps"] + 1, 2)}[case["kind"]]
    flops = reps * (evals[0] * force + evals[1] * energy)
    # positions and parameters in, forces out, per evaluation; 176 bytes an atom for a step's state
    moved = reps * n * (evals[0] * (24 + 72 + 24) + evals[1] * (24 + 72 + 40))
    if case["kind"] in ("dynamics", "remd"):
        moved += reps * n * (case["steps"] * 176 + 2 * 48)
    return {"bytes": float(moved), "flops": float(flops)}


# ------------------------------------------------------------ 64-bit values

KCAL, COULOMB, EPS_W = 4.184, 332.0637, 78.5


def _angle(a, b, c):
    u, v = a - b, c - b
    u, v = u / u.norm(dim=1, keepdim=True), v / v.norm(dim=1, keepdim=True)
    return torch.acos((u * v).sum(1).clamp(-1.0, 1.0))


def _dihedral(a, b, c, d):
    b0, b1, b2 = a - b, c - b, d - c
    b1 = b1 / b1.norm(dim=1, keepdim=True)
    v = b0 - b1 * (b0 * b1).sum(1, keepdim=True)
    w = b2 - b1 * (b2 * b1).sum(1, keepdim=True)
    return torch.atan2((torch.linalg.cross(b1, v) * w).sum(1), (v * w).sum(1))


def _bonded(t, x, dev):
    def f(a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)

    def ix(a):
        return torch.as_tensor(np.asarray(a, dtype=np.int64), device=dev)

    def at(idx):
        i = ix(idx)
        return [x[i[:, k]] for k in range(i.shape[1])]

    p, q = at(t.bonds)
    e = {"bond": (f(t.bond_k) * ((q - p).norm(dim=1) - f(t.bond_r0)) ** 2).sum()}
    e["angle"] = (f(t.angle_k) * (_angle(*at(t.angles)) - torch.deg2rad(f(t.angle_theta0))) ** 2).sum()
    start = np.asarray(t.dihedral_term_start)
    owner = ix(np.repeat(np.arange(len(start) - 1), np.diff(start)))
    chi = _dihedral(*at(t.dihedrals))[owner]
    e["dihedral"] = (f(t.term_k) * (1.0 + torch.cos(f(t.term_n) * chi - torch.deg2rad(f(t.term_delta))))).sum()
    if len(t.improper_k):
        om = _dihedral(*at(t.impropers)) - torch.deg2rad(f(t.improper_psi0))
        om = torch.remainder(om + math.pi, 2.0 * math.pi) - math.pi
        e["improper"] = (f(t.improper_k) * om ** 2).sum()
    else:
        e["improper"] = x.sum() * 0.0
    return {k: v * KCAL for k, v in e.items()}


def _rows(n):
    step = max(1, int(4e6 // n))
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _born(t, x, cutoff, dev):
    rho = torch.as_tensor(t.gb_rho, device=dev)
    rt = rho - 0.09
    s = torch.as_tensor(t.gb_scale, device=dev) * rt
    n = x.shape[0]
    total = torch.zeros(n, dtype=torch.float64, device=dev)
    for a, b in _rows(n):
        d = x[None, :, :] - x[a:b, None, :]
        r = (d * d).sum(-1).sqrt()
        on = torch.ones_like(r, dtype=torch.bool)
        on[torch.arange(b - a, device=dev), torch.arange(a, b, device=dev)] = False
        on &= r <= cutoff
        r = torch.where(on, r, 1.0)
        ri, sj = rt[a:b, None], s[None, :]
        low = torch.where(r - sj < ri, ri.expand_as(r), r - sj)
        up = r + sj
        on &= (r + sj > ri) & (low > 0)
        low = torch.where(on, low, 1.0)
        k = 1.0 / up ** 2 - 1.0 / low ** 2
        h = 0.5 * (1.0 / low - 1.0 / up) + 0.25 * r * k + torch.log(low / up) / (2.0 * r) + (sj ** 2 - r ** 2) / (4.0 * r) * k
        total[a:b] = torch.where(on, h, 0.0).sum(1)
    psi = total * rt
    inv = 1.0 / rt - torch.tanh(psi - 0.8 * psi ** 2 + 4.85 * psi ** 3) / rho
    floor = rt.clamp(min=0.5)
    return torch.where(inv > 0, torch.maximum(1.0 / torch.where(inv > 0, inv, 1.0), floor), floor)


def _pair_rows(t, x, born, nb, gb_cut, a, b, dev):
    """(LJ, Coulomb, GB pair) energies of rows a..b, each unordered pair counted from both ends (kcal/mol, halved)."""
    def f(v):
        return torch.as_tensor(np.asarray(v, dtype=np.float64), device=dev)

    n = x.shape[0]
    d = x[None, :, :] - x[a:b, None, :]
    self_pair = torch.zeros((b - a, n), dtype=torch.bool, device=dev)
    self_pair[torch.arange(b - a, device=dev), torch.arange(a, b, device=dev)] = True
    kind = torch.zeros((b - a, n), dtype=torch.int8, device=dev)
    ex, kd = np.asarray(t.exclusions), np.asarray(t.exclusion_kind)
    for p, q in ((0, 1), (1, 0)):
        sel = (ex[:, p] >= a) & (ex[:, p] < b)
        kind[torch.as_tensor(ex[sel, p] - a, dtype=torch.int64, device=dev),
             torch.as_tensor(ex[sel, q], dtype=torch.int64, device=dev)] = torch.as_tensor(kd[sel], device=dev)
    r2 = torch.where(self_pair, 1.0, (d * d).sum(-1))
    q = f(t.charge)
    qq = q[a:b, None] * q[None, :]
    on = ~self_pair & (kind != 1) & (r2 <= nb * nb)
    rm, ep, rm14, ep14 = f(t.rmin_half), f(t.epsilon), f(t.rmin_half_14), f(t.epsilon_14)
    is14 = kind == 2
    rmin = torch.where(is14, rm14[a:b, None] + rm14[None, :], rm[a:b, None] + rm[None, :])
    eps = torch.where(is14, (ep14[a:b, None] * ep14[None, :]).sqrt(), (ep[a:b, None] * ep[None, :]).sqrt())
    safe = torch.where(on, r2, 25.0)
    r6 = (rmin ** 2 / safe) ** 3
    lj = 0.5 * torch.where(on, eps * (r6 * r6 - 2.0 * r6), 0.0).sum()
    r = safe.sqrt()
    rf = safe / (2.0 * nb ** 3) - 1.5 / nb if math.isfinite(nb) else 0.0
    coul = 0.5 * torch.where(on, COULOMB * qq * (1.0 / r + rf), 0.0).sum()
    rp = born[a:b, None] * born[None, :]
    fgb = (r2 + rp * torch.exp(-r2 / (4.0 * rp))).sqrt()
    pref = -(1.0 - 1.0 / EPS_W) * COULOMB
    gb = 0.5 * torch.where(~self_pair & (r2 <= gb_cut * gb_cut), pref * qq / fgb, 0.0).sum()
    return lj, coul, gb


def exact(case, seed):
    """Forces and energy terms in 64 bits from the model's formulas; trajectories, minimisations and surface terms have no
    value here."""
    if case["kind"] not in ("forces", "energy") or case["sasa"]:
        return None
    chain, xyz = _systems(case, seed)[0]
    t = chain.topology()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nb, born_cut, gb_cut = (10.0, 20.0, 10.0) if case["cutoff"] else (math.inf,) * 3
    x = torch.tensor(xyz, dtype=torch.float64, device=dev)
    with torch.no_grad():
        born = _born(t, x, born_cut, dev)
    if case["kind"] == "energy":
        with torch.no_grad():
            e = {k: float(v) for k, v in _bonded(t, x, dev).items()}
            sums = [0.0, 0.0, 0.0]
            for a, b in _rows(x.shape[0]):
                for k, v in enumerate(_pair_rows(t, x, born, nb, math.inf, a, b, dev)):
                    sums[k] += float(v) * KCAL
            q = torch.as_tensor(t.charge, device=dev)
            own = float((-0.5 * (1.0 - 1.0 / EPS_W) * COULOMB * q * q / born).sum()) * KCAL
        e.update(lj=sums[0], coulomb=sums[1], gb_pair=sums[2], gb_self=own, gb=sums[2] + own, sasa=0.0)
        e["total"] = sum(e[k] for k in ("bond", "angle", "dihedral", "improper", "lj", "coulomb", "gb"))
        e.update(born_clamped=None, nb_pairs=None)
        return e
    grad = torch.zeros_like(x)
    y = x.clone().requires_grad_(True)
    grad += torch.autograd.grad(sum(_bonded(t, y, dev).values()), y)[0]
    for a, b in _rows(x.shape[0]):
        y = x.clone().requires_grad_(True)
        grad += torch.autograd.grad(KCAL * sum(_pair_rows(t, y, born, nb, gb_cut, a, b, dev)), y)[0]
    return (-grad).cpu().numpy()
