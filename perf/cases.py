"""The work this framework is used for, as cases that can be timed and compared.

Each case is a dict of plain values; `prepare` builds what a user's program
holds before the call (engine, replicas, device buffers, parameters), `run`
makes one pass through the public entry points of `rbmd_b200.rbx` /
`rbmd_b200.autograd`, and `exact` gives the same outputs from plain torch in
64 bits where a few lines can restate the path.

Kinds:
  md      velocity-Verlet steps of the LJ electrolyte (RBL or Verlet-SOG real
          space, RBE or RBSOG k-space) and the state read back
  thermo  Verlet-List steps and then a thermo output: pair energies, virial
          and the exact reciprocal energy
  water   rigid water: RBL with special bonds, RBE, SHAKE, Nose-Hoover
  batch   independent replicas advanced together
  fit     one force-field-fitting step: force, loss and its gradients
  kspace  the FP64 RBE functors on a caller's device buffers
  dropin  a whole force evaluation through the float functors on a caller's
          device buffers (RBL filter, pair force, mean removal, RBE)
  lists   linked cells and the full neighbour list on a caller's buffers
"""
from __future__ import annotations

import math

import numpy as np
import torch

from rbmd_b200 import autograd, rbx, systems

ALPHA = 0.16                       # hyper_parameters.coulomb.alpha
R_CORE, CUT_OFF, SKIN = 2.5, 5.0, 0.3
EPSILON = 1e-4                     # the lists' margin on squared radii
SAMPLES = 100                      # neighbor_sample_num
SEED = 77                          # k-sampler seed of the engines


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest production run: 4,000 atoms, where launches count
        {"name": "md_4k_mixed", "kind": "md", "n": 4000, "p": 100, "neighbor": "RBL",
         "precision": "mixed", "steps": 100},
        # the headline electrolyte in both precision forms
        {"name": "md_200k_mixed", "kind": "md", "n": 200000, "p": 100, "neighbor": "RBL",
         "precision": "mixed", "steps": 50},
        {"name": "md_200k_fp64", "kind": "md", "n": 200000, "p": 100, "neighbor": "RBL",
         "precision": "fp64", "steps": 50},
        # a mid-size box with an odd atom count and the large k-sample, FP64
        {"name": "md_60k_p400_fp64", "kind": "md", "n": 59999, "p": 400, "neighbor": "RBL",
         "precision": "fp64", "steps": 40},
        # sum-of-Gaussians electrostatics on a Verlet list
        {"name": "md_50k_sog_mixed", "kind": "md", "n": 50021, "p": 112, "neighbor": "VERLET-SOG",
         "precision": "mixed", "steps": 40},
        # Verlet list with a thermo output every ten steps
        {"name": "thermo_20k_fp64", "kind": "thermo", "n": 20011, "p": 100, "precision": "fp64",
         "steps": 10, "kmax": 8},
        # rigid water, 300 K thermostat, SHAKE (8 copies of 3,041 molecules)
        {"name": "water_73k_mixed", "kind": "water", "mols": 3041, "copies": 2, "p": 300,
         "precision": "mixed", "steps": 40},
        # independent replicas of uneven sizes advanced together
        {"name": "batch_48", "kind": "batch", "replicas": 48, "nmin": 1000, "nmax": 10000,
         "p": 100, "steps": 50},
        # one force-field-fitting step, forward and backward
        {"name": "fit_20k", "kind": "fit", "n": 20000, "p": 100, "precision": "mixed"},
        # the FP64 k-space functors
        {"name": "kspace_100k", "kind": "kspace", "n": 100003, "p": 100},
        # the float functors of one whole force evaluation
        {"name": "dropin_50k_f32", "kind": "dropin", "n": 50000, "p": 100},
        # cell sort and neighbour list of a large box
        {"name": "lists_200k", "kind": "lists", "n": 200000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["md", "md", "md", "thermo", "water", "batch", "fit", "kspace", "dropin",
                       "lists"])
    precision = rng.choice(["mixed", "fp64"])
    if kind == "md":
        nb = rng.choice(["RBL", "RBL", "VERLET-SOG"])
        return {"kind": kind, "n": _log_int(rng, 1000, 200000 if nb == "RBL" else 100000),
                "p": rng.choice([100, 144, 200] if nb == "RBL" else [112, 208]), "neighbor": nb,
                "precision": precision, "steps": rng.randint(10, 40)}
    if kind == "thermo":
        return {"kind": kind, "n": _log_int(rng, 4000, 40000), "p": rng.choice([100, 200]),
                "precision": precision, "steps": rng.randint(5, 15), "kmax": rng.randint(4, 8)}
    if kind == "water":
        side = rng.randint(9, 14)  # close to a full lattice, as a liquid's density needs
        return {"kind": kind, "mols": side ** 3 - rng.randint(0, side ** 3 // 10),
                "copies": rng.choice([1, 2]),
                "p": rng.choice([100, 200, 300]), "precision": precision, "steps": rng.randint(10, 40)}
    if kind == "batch":
        return {"kind": kind, "replicas": rng.randint(8, 64), "nmin": 1000,
                "nmax": _log_int(rng, 2000, 8000), "p": 100, "steps": rng.randint(10, 40)}
    if kind == "fit":
        return {"kind": kind, "n": _log_int(rng, 4000, 40000), "p": rng.choice([100, 200]),
                "precision": precision}
    if kind == "kspace":
        return {"kind": kind, "n": _log_int(rng, 1000, 200000), "p": rng.randint(50, 400)}
    if kind == "dropin":
        return {"kind": kind, "n": _log_int(rng, 4000, 100000), "p": rng.choice([100, 200])}
    return {"kind": kind, "n": _log_int(rng, 4000, 200000)}


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _prec(case):
    return rbx.MIXED if case["precision"] == "mixed" else rbx.PLAIN_FP64


def _lj(case, seed, n=None):
    return systems.lj_electrolyte(n or case["n"], seed=seed, kspace_p=case.get("p", 100))


def _electrolyte_engine(case, seed, neighbor="RBL", n=None):
    sog = neighbor == "VERLET-SOG"
    e = rbx.Engine(_lj(case, seed, n), precision=_prec(case), neighbor=neighbor,
                   coulomb="RBSOG" if sog else "RBE", seed=SEED)
    e.compute_forces(0)
    return e


def _water_system(case, seed):
    """copies^3 periodic images of one water box, each with velocities of its own."""
    s = systems.water(case["mols"], seed=seed, kspace_p=case["p"], dt=0.5)
    c = case["copies"]
    if c == 1:
        return s
    n, L = s["n"], np.asarray(s["hi"])
    k = np.arange(c ** 3)
    shift = np.stack([k % c, (k // c) % c, k // (c * c)], 1) * L
    rep = lambda a: np.concatenate([a + n * r for r in k])  # noqa: E731
    tile = lambda a: np.tile(a, len(k))  # noqa: E731
    p, rng = s["params"], np.random.default_rng(seed + 1)
    typ = tile(s["type"])
    m = s["mass"][typ]
    vel = rng.normal(size=(n * len(k), 3)) * np.sqrt(p["kb"] * 298.0 / (m * p["mvv2e"]))[:, None]
    vel -= (m[:, None] * vel).sum(0) / m.sum()
    pos = (s["pos"][None] + shift[:, None]).reshape(-1, 3)
    return dict(s, n=n * len(k), hi=L * c, pos=pos, vel=vel, q=tile(s["q"]), type=typ,
                gid=np.arange(n * len(k), dtype=np.int32),
                clusters=rep(s["clusters"]).astype(np.int32), bonds=rep(s["bonds"]),
                angles=rep(s["angles"]))


def _water_engine(case, seed):
    s = _water_system(case, seed)
    p = s["params"]
    ns, sp = rbx.special_build(s["n"], s["bonds"], s["angles"])
    e = rbx.Engine(s, precision=_prec(case), seed=SEED)
    e.set_shake(s["clusters"], systems.WATER_BOND, systems.WATER_ANGLE)
    e.set_special(ns, sp, (0.0, 0.0, 0.0))
    e.compute_forces(0)
    e.set_nose_hoover(298.0, 298.0, 10.0, kb=p["kb"], mvv2e=p["mvv2e"], tdof=2.0 * s["n"] - 3)
    return e


def _replica_sizes(case):
    rng = np.random.default_rng([case["replicas"], case["nmax"]])
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    return np.exp(rng.uniform(lo, hi, case["replicas"])).astype(int)


def _fit_inputs(case, seed):
    """Positions off the lattice, k-samples, target forces of the unperturbed
    parameters and the perturbed parameters of a fitting step."""
    s = _lj(case, seed)
    rng = np.random.default_rng(seed + 5)
    L = s["hi"][0]
    pos = np.mod(s["pos"] + rng.normal(0.0, 0.02, size=s["pos"].shape), L)
    m = _k_samples(L, ALPHA, case["p"], SEED, 0)
    th = {k: torch.tensor(1.0 + rng.uniform(-0.05, 0.05, 3)) for k in ("eps", "sigma")}
    th["charge"] = torch.tensor(s["q"] * (1.0 + rng.uniform(-0.05, 0.05)))
    th["alpha"] = torch.tensor(ALPHA * (1.0 + rng.uniform(-0.05, 0.05)), dtype=torch.float64)
    th["pos"] = torch.tensor(pos)
    d = _device()
    x = torch.tensor(pos, device=d)
    ref = _forces(s, x, torch.tensor(s["q"], device=d), 0, _pairs(x, L, CUT_OFF), m).cpu()
    return s, m, th, ref


def _f(a, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def _int(*shape, fill=0):
    return torch.full(shape, fill, dtype=torch.int32, device="cuda")


def _row_capacity():
    return 32 * math.ceil((1.3 * 0.8 * 4 / 3 * math.pi * (CUT_OFF + SKIN) ** 3 + 64) / 32)


def _list_buffers(s):
    n, box = s["n"], rbx.Box.make(s["lo"], s["hi"])
    dims = rbx.cell_grid(box, CUT_OFF + SKIN)
    ncell = dims[0] * dims[1] * dims[2]
    cap = _row_capacity()
    return {"box": box, "perm": _int(n), "cell": _int(n), "start": _int(ncell + 1),
            "scratch": torch.empty(rbx.cells_scratch_bytes(n, ncell), dtype=torch.uint8,
                                   device="cuda"),
            "cap": cap, "count": _int(n), "nbrs": _int(n, cap, fill=-1), "overflow": _int(1)}


def _build_lists(b, xyz):
    """Cell order, the positions in that order and their neighbour rows."""
    rbx.cells_sort(b["box"], CUT_OFF + SKIN, *xyz, b["perm"], b["cell"], b["start"], b["scratch"],
                   stream=torch.cuda.current_stream())
    order = b["perm"].long()
    xs = [c[order] for c in xyz]
    rbx.full_list(b["box"], CUT_OFF + SKIN, *xs, b["start"], b["cap"], b["count"], b["nbrs"],
                  b["overflow"], stream=torch.cuda.current_stream())
    return order, xs


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "md":
        st["engine"] = _electrolyte_engine(case, seed, case["neighbor"])
    elif kind == "thermo":
        st["engine"] = _electrolyte_engine(case, seed, "VERLET")
    elif kind == "water":
        st["engine"] = _water_engine(case, seed)
    elif kind == "batch":
        c = dict(case, precision="mixed")
        st["engines"] = [_electrolyte_engine(c, 1000 * seed + r, n=int(n))
                         for r, n in enumerate(_replica_sizes(case))]
        st["batch"] = rbx.Batch(st["engines"])
    elif kind == "fit":
        s, m, st["theta"], st["target"] = _fit_inputs(case, seed)
        st["engine"] = rbx.Engine(s, precision=_prec(case), seed=SEED)
        st["engine"].set_k_samples(*m)
    elif kind == "kspace":
        s = _lj(case, seed)
        L = s["hi"][0]
        st["box"] = rbx.Box.make(s["lo"], s["hi"])
        st["S"] = rbx.rbe_gauss_sum(st["box"], ALPHA)
        st["q"] = _f(s["q"], torch.float64)
        st["qsq"], st["qsum"] = float((s["q"] ** 2).sum()), float(s["q"].sum())
        st["m"] = [_f(v, torch.float64) for v in _k_samples(L, ALPHA, case["p"], seed, 1)]
        st["x"] = [_f(s["pos"][:, d], torch.float64) for d in range(3)]
        st["rho"] = [torch.zeros_like(st["m"][0]) for _ in range(2)]
        st["f"] = [torch.zeros_like(st["q"]) for _ in range(3)]
        st["virial"], st["energy"] = _f(np.zeros(6), torch.float64), _f(np.zeros(1), torch.float64)
    elif kind == "dropin":
        s = _lj(case, seed)
        n = s["n"]
        b = _list_buffers(s)
        order, _ = _build_lists(b, [_f(s["pos"][:, d], torch.float64) for d in range(3)])
        if int(b["overflow"].item()):
            raise RuntimeError("neighbour rows overflow")
        o = order.cpu().numpy()
        cap = b["cap"]
        st.update(n=n, box=b["box"], cap=cap, cand=b["nbrs"].reshape(-1))
        st["x"] = [_f(s["pos"][o, d]) for d in range(3)]
        st["q"], st["type"] = _f(s["q"][o]), _f(s["type"][o], torch.int32)
        st["gid"] = _f(s["gid"][o], torch.int32)
        st["start"] = torch.arange(n, dtype=torch.int32, device="cuda") * cap
        st["end"] = st["start"] + b["count"]
        st["sigma"], st["eps"] = _f(s["sigma"]), _f(s["eps"])
        st["freq"] = rbx.rbl_params(n, b["box"], R_CORE, CUT_OFF, SAMPLES)
        core_cap, shell_cap = 128, 192
        st["core_cap"], st["shell_cap"] = _int(n, fill=core_cap), shell_cap
        st["core_start"] = torch.arange(n, dtype=torch.int32, device="cuda") * core_cap
        st["core_end"], st["core"] = _int(n), _int(n * core_cap, fill=-1)
        st["shell"], st["shell_num"] = _int(shell_cap * n, fill=-1), _int(n)
        st["need"], st["realloc"] = _int(1), _int(1)
        st["S"] = rbx.rbe_gauss_sum(b["box"], ALPHA)
        st["qsq"], st["qsum"] = float((s["q"] ** 2).sum()), float(s["q"].sum())
        st["m"] = [_f(v) for v in _k_samples(s["hi"][0], ALPHA, case["p"], seed, 1)]
        st["rho"] = [torch.zeros_like(st["m"][0]) for _ in range(2)]
        st["f"] = [torch.zeros_like(st["q"]) for _ in range(3)]
        st["fk"] = [torch.zeros_like(st["q"]) for _ in range(3)]
        st["virial"], st["energy"] = _f(np.zeros(6)), _f(np.zeros(1))
    else:
        s = _lj(case, seed)
        st["lists"] = _list_buffers(s)
        st["x"] = [_f(s["pos"][:, d], torch.float64) for d in range(3)]
    return st


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind in ("md", "water"):
        st["engine"].step(case["steps"])
        return st["engine"].get_state()
    if kind == "thermo":
        e = st["engine"]
        e.step(case["steps"])
        lj, coul, virial = e.pair_energy()
        out = e.get_state()
        out.update(e_lj=float(lj), e_coul=float(coul), virial=virial,
                   e_k=e.kspace_energy_exact([case["kmax"]] * 3))
        return out
    if kind == "batch":
        st["batch"].step(case["steps"])
        states = [e.get_state() for e in st["engines"]]
        return {k: np.concatenate([s[k] for s in states]) for k in ("pos", "vel", "force")}
    if kind == "fit":
        th = {k: v.clone().requires_grad_(True) for k, v in st["theta"].items()}
        force = autograd.force(st["engine"], th["eps"], th["sigma"], th["charge"], th["alpha"],
                               th["pos"])
        loss = ((force - st["target"]) ** 2).sum() / len(force)
        loss.backward()
        return {"loss": float(loss.detach()), "force": force.detach(),
                **{k: v.grad for k, v in th.items()}}
    stream = torch.cuda.current_stream()
    if kind == "kspace":
        a = (st["box"],)
        rbx.rbe_structure_factor(*a, st["q"], *st["m"], *st["x"], *st["rho"], stream=stream)
        rbx.rbe_force(*a, ALPHA, st["S"], 1.0, *st["rho"], st["q"], *st["m"], *st["x"], *st["f"],
                      stream=stream)
        rbx.rbe_energy_virial(*a, ALPHA, st["S"], 1.0, st["qsq"], st["qsum"], *st["rho"], *st["m"],
                              st["virial"], st["energy"], stream=stream)
        return {k: st[k] for k in ("rho", "f", "virial", "energy")}
    if kind == "dropin":
        box, freq = st["box"], st["freq"]
        rbx.rbl_filter_f32(float(np.float32(R_CORE * R_CORE) - np.float32(EPSILON)),
                           float(np.float32(CUT_OFF * CUT_OFF) - np.float32(EPSILON)), st["gid"],
                           *st["x"], st["start"], st["end"], st["cand"], st["core_cap"],
                           st["core_start"], st["core_end"], st["core"], st["shell_cap"],
                           st["shell"], st["shell_num"], st["need"], box, st["realloc"], freq, 1,
                           stream=stream)
        rbx.pair_force_rbl_f32(box, R_CORE, CUT_OFF, SAMPLES, freq, ALPHA, 1.0, st["type"],
                               st["sigma"], st["eps"], st["core_start"], st["core_end"],
                               st["core"], st["shell"], st["shell_num"], st["q"], *st["x"],
                               *st["f"], stream=stream)
        rbx.fix_rbl_force_f32(*st["f"], stream=stream)
        rbx.rbe_structure_factor_f32(box, st["q"], *st["m"], *st["x"], *st["rho"], stream=stream)
        rbx.rbe_force_f32(box, ALPHA, st["S"], 1.0, *st["rho"], st["q"], *st["m"], *st["x"],
                          *st["fk"], stream=stream)
        rbx.rbe_energy_virial_f32(box, ALPHA, st["S"], 1.0, st["qsq"], st["qsum"], *st["rho"],
                                  *st["m"], st["virial"], st["energy"], stream=stream)
        return {k: st[k] for k in ("core_end", "core", "shell_num", "shell", "need", "realloc",
                                   "f", "rho", "fk", "virial", "energy")}
    b = st["lists"]
    _build_lists(b, st["x"])
    return {k: b[k] for k in ("perm", "cell", "start", "count", "nbrs", "overflow")}


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------
def work(case):
    """Per atom and step: the state (x, v, f: 72 bytes) read and written once,
    charge and type read; 40 operations a force-carrying pair, 20 a phase."""
    kind = case["kind"]
    n, p, steps = case.get("n", 0), case.get("p", 0), case.get("steps", 1)
    core = 0.8 * 4 / 3 * math.pi * R_CORE ** 3
    cut = 0.8 * 4 / 3 * math.pi * CUT_OFF ** 3
    full = 0.8 * 4 / 3 * math.pi * (CUT_OFF + SKIN) ** 3
    rbl = core + (cut - core) / 4
    pairs = rbl
    if kind == "water":
        n = 3 * case["mols"] * case["copies"] ** 3
        core, cut = 0.1002 * 4 / 3 * math.pi * 6.5 ** 3, 0.1002 * 4 / 3 * math.pi * 1000.0
        pairs = core + (cut - core) / 4
    elif kind == "batch":
        r = math.log(case["nmax"] / case["nmin"])
        n = case["replicas"] * (case["nmax"] - case["nmin"]) / r
    elif kind == "thermo" or case.get("neighbor") == "VERLET-SOG":
        pairs = cut
    if kind == "lists":
        return {"bytes": n * (24 + 12 + 4 * full), "flops": n * full * 8}
    if kind == "kspace":
        return {"bytes": n * (2 * 32 + 24) + 40 * p, "flops": 2.0 * n * p * 20}
    if kind == "dropin":
        return {"bytes": n * (4 * full + 8 * rbl + 3 * 16 + 12 + 24),
                "flops": n * (full * 8 + rbl * 40 + 2 * p * 20)}
    if kind == "fit":
        return {"bytes": n * 200.0, "flops": 3.0 * n * (rbl * 40 + 2 * p * 20)}
    flops = n * steps * (pairs * 40 + 2 * p * 20)
    if kind == "thermo":
        flops += n * (pairs * 40 + (2 * case["kmax"] + 1) ** 3 * 20)
    return {"bytes": n * steps * 156.0, "flops": flops}


def tolerance(case):
    """About four times what other launch shapes (other orders of the same
    sums) and the 64-bit restatement differ by; steps amplify a rounding, and
    one pair at a list radius that enters a step earlier moves an atom's force
    by up to 0.02 of the root mean square."""
    kind = case["kind"]
    mixed = case.get("precision", "mixed") == "mixed"
    if kind == "lists":
        return "exact"
    if kind == "kspace":
        return {"rel": 1e-12, "max": 1e-10}
    if kind == "dropin":
        return {"rel": 4e-5, "max": 1.6e-3}
    if kind == "fit":
        return {"rel": 1e-4, "max": 4e-3} if mixed else {"rel": 1e-9, "max": 4e-8}
    return {"rel": 2e-4, "max": 2e-2} if mixed else {"rel": 1e-9, "max": 1e-7}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _philox(c, key):
    """Philox4x32-10 (Salmon et al., SC'11) on arrays of 32-bit counters."""
    c = [np.asarray(v, dtype=np.uint64) for v in c]
    k0, k1 = key & 0xffffffff, key >> 32
    mask, s32 = np.uint64(0xffffffff), np.uint64(32)
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> s32) ^ c[1] ^ np.uint64(k0), b & mask, (a >> s32) ^ c[3] ^ np.uint64(k1),
             a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return c


def _k_samples(L, alpha, p, seed, step):
    """p integer k-vectors of density exp(-(pi m / L)^2 / alpha), m = 0 left out."""
    c = math.pi ** 2 / (alpha * L * L)
    w = [1.0]
    while math.exp(-c * (len(w) // 2 + 1) ** 2) >= 1e-20:
        w += [math.exp(-c * (len(w) // 2 + 1) ** 2)] * 2
    cdf = np.cumsum(w)
    m = np.zeros((3, p))
    todo = np.arange(p)
    for a in range(64):
        if not len(todo):
            break
        s = todo.astype(np.uint64)
        one = np.ones_like(s)
        st = int(step)
        lo, hi = one * np.uint64(st & 0xffffffff), one * np.uint64(st >> 32)
        u = _philox([s, one * np.uint64(2 * a), lo, hi], seed)
        v = _philox([s, one * np.uint64(2 * a + 1), lo, hi], seed)
        for d, (h, l) in enumerate(((u[0], u[1]), (u[2], u[3]), (v[0], v[1]))):
            r = (((h << np.uint64(32)) | l) >> np.uint64(11)).astype(np.float64) / 2.0 ** 53
            i = np.minimum(np.searchsorted(cdf, r * cdf[-1], side="right"), len(cdf) - 1)
            m[d, todo] = np.where(i % 2 == 1, (i + 1) // 2, -(i // 2))
        todo = todo[(m[:, todo] == 0).all(0)]
    return m


def _gauss_sum(L, alpha):
    """prod_d sqrt(alpha L^2 / pi) sum_m exp(-alpha L^2 m^2) - 1."""
    a = torch.as_tensor(alpha, dtype=torch.float64) * L * L
    h = sum(torch.exp(-a * float(m * m)) for m in range(-10, 11)) * torch.sqrt(a / math.pi)
    return h ** 3 - 1.0


def _freq(n, L):
    rho = n / L ** 3
    c = round(1.0 + (0.05 / rho - 0.05))
    rs, rc = (int(c * rho * math.ceil(4 / 3 * math.pi * r ** 3) + 1) for r in (R_CORE, CUT_OFF))
    return 1 if rc - rs <= SAMPLES else math.ceil((rc - rs) / SAMPLES)


def _shr(v, k):
    return (v >> k) & ((1 << (64 - k)) - 1)


def _i64(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _mix(v):
    v = v + _i64(0x9e3779b97f4a7c15)
    v = (v ^ _shr(v, 30)) * _i64(0xbf58476d1ce4e5b9)
    v = (v ^ _shr(v, 27)) * _i64(0x94d049bb133111eb)
    return v ^ _shr(v, 31)


def _selected(gid, i, j, epoch, freq):
    key = _mix(gid)[i] ^ _mix(gid + _i64(0xd1b54a32d192ed03))[j] ^ epoch
    h = _mix(key)
    low, high = h & 0xffffffff, _shr(h, 32)
    return ((high % freq) * ((1 << 32) % freq) + low % freq) % freq == 0


def _pairs(x, L, r):
    """Every ordered pair (i, j), i != j, within r (minimum image)."""
    n, nc = len(x), int(L / r)
    d = x.device
    if nc < 3:
        e = x[:, None] - x[None]
        e = e - L * torch.round(e / L)
        near = (e * e).sum(-1) < r * r
        near.fill_diagonal_(False)
        return near.nonzero(as_tuple=True)
    c = torch.clamp((x / (L / nc)).long(), max=nc - 1)
    flat = (c[:, 2] * nc + c[:, 1]) * nc + c[:, 0]
    order = torch.argsort(flat)
    count = torch.bincount(flat, minlength=nc ** 3)
    first = torch.cumsum(count, 0) - count
    width = int(count.max())
    slot = torch.full((nc ** 3, width), -1, dtype=torch.long, device=d)
    slot[flat[order], torch.arange(n, device=d) - first[flat[order]]] = order
    ids = torch.arange(nc ** 3, device=d)
    cz, cy, cx = ids // (nc * nc), (ids // nc) % nc, ids % nc
    part = max(1, 60_000_000 // (width * width))
    ii, jj = [], []
    for s in range(27):
        o = (((cz + s // 9 - 1) % nc) * nc + (cy + (s // 3) % 3 - 1) % nc) * nc + \
            (cx + s % 3 - 1) % nc
        for b in range(0, nc ** 3, part):
            u, v = slot[b:b + part], slot[o[b:b + part]]
            r2 = 0.0
            for k in range(3):
                e = x[u.clamp(min=0), k][:, :, None] - x[v.clamp(min=0), k][:, None, :]
                r2 = r2 + (e - L * torch.round(e / L)) ** 2
            ok = (r2 < r * r) & (u >= 0)[:, :, None] & (v >= 0)[:, None, :]
            ok &= u[:, :, None] != v[:, None, :]
            w = ok.nonzero(as_tuple=True)
            ii.append(u[w[0], w[1]])
            jj.append(v[w[0], w[2]])
    return torch.cat(ii), torch.cat(jj)


def _cell_order(s):
    """Atoms by cell of edge >= CUT_OFF + SKIN, then by 4 x 4 x 4 Morton
    sub-cell, then by index: the order the cell sort documents."""
    nc = int(s["hi"][0] / (CUT_OFF + SKIN))
    f = s["pos"] * (nc / s["hi"][0])
    c = np.clip(np.floor(f), 0, nc - 1).astype(int)
    b = np.clip(np.floor((f - c) * 4), 0, 3).astype(int)
    code = sum(((b[:, d] >> k) & 1) << (3 * k + d) for k in range(2) for d in range(3))
    return np.argsort((((c[:, 2] * nc + c[:, 1]) * nc + c[:, 0]) << 6) + code, kind="stable")


def _separations(x, L, i, j):
    e = x[j] - x[i]
    return e - L * torch.round(e / L)


def _pair_force(d, r2, eps, sigma, qq, alpha, scale):
    """Force on i of pairs with separation d = r_j - r_i."""
    u = sigma ** 6 / r2 ** 3
    r = torch.sqrt(r2)
    b = torch.as_tensor(alpha, dtype=torch.float64, device=d.device).sqrt()
    coul = (torch.erfc(b * r) / r2 + 2 * b * torch.exp(-alpha * r2) / (math.sqrt(math.pi) * r)) / r
    return d * (scale * (-24 * eps * (2 * u * u - u) / r2 - qq * coul))[:, None]


def _rbl(s, x, epoch, pairs, gid=None):
    """The core pairs and the batch-selected shell pairs, with their weights."""
    L = s["hi"][0]
    freq = _freq(s["n"], L)
    i, j = pairs
    r2 = sum(((e := x[j, k] - x[i, k]) - L * torch.round(e / L)) ** 2 for k in range(3))
    core = (r2 < R_CORE ** 2 - EPSILON) & (r2 > EPSILON)
    shell = (r2 < CUT_OFF ** 2 - EPSILON) & (r2 > R_CORE ** 2)
    ci, cj, si, sj = i[core], j[core], i[shell], j[shell]
    gid = torch.tensor(np.asarray(s["gid"], np.int64), device=x.device) if gid is None else gid
    sel = _selected(gid, si, sj, epoch, freq)
    si, sj = si[sel], sj[sel]
    w = torch.cat([torch.ones(len(ci)), torch.full((len(si),), float(freq))]).to(x)
    return torch.cat([ci, si]), torch.cat([cj, sj]), w


def _kspace(L, x, q, m, alpha, want="force"):
    """RBE structure factor and force of integer k-vectors m [3, p]."""
    p = len(m[0])
    k = 2 * math.pi * torch.as_tensor(np.asarray(m), dtype=torch.float64, device=x.device) / L
    c = -4 * math.pi * _gauss_sum(L, alpha).to(x.device) / (p * L ** 3 * (k * k).sum(0))
    re, im = [], []
    for a in range(0, p, 32):
        ph = x @ k[:, a:a + 32]
        re.append((q[:, None] * torch.cos(ph)).sum(0))
        im.append((q[:, None] * torch.sin(ph)).sum(0))
    re, im = torch.cat(re), torch.cat(im)
    f = 0.0
    for a in range(0, p, 32):
        ka = k[:, a:a + 32]
        ph = x @ ka
        f = f + (c[a:a + 32] * (torch.cos(ph) * im[a:a + 32] - torch.sin(ph) * re[a:a + 32])) @ ka.T
    return f * q[:, None], re, im, k


def _forces(s, x, q, epoch, pairs, m, eps=None, sigma=None, alpha=ALPHA, verlet=False):
    L = s["hi"][0]
    if verlet:
        i, j = pairs
        near = (_separations(x, L, i, j) ** 2).sum(1) < CUT_OFF ** 2
        i, j = i[near], j[near]
        w = torch.ones(len(i), dtype=x.dtype, device=x.device)
    else:
        with torch.no_grad():
            i, j, w = _rbl(s, x, epoch, pairs)
    if eps is None:
        e, g = 1.0, torch.ones((), dtype=x.dtype, device=x.device)
    else:
        t = torch.as_tensor(np.asarray(s["type"], np.int64), device=x.device)
        e, g = torch.sqrt(eps[t[i]] * eps[t[j]]), (sigma[t[i]] + sigma[t[j]]) / 2
    f = torch.zeros_like(x)
    for a in range(0, len(i), 1 << 25):
        ia, ja = i[a:a + (1 << 25)], j[a:a + (1 << 25)]
        d = _separations(x, L, ia, ja)
        part = slice(a, a + (1 << 25))
        ea, ga = (e, g) if eps is None else (e[part], g[part])
        f = f.index_add(0, ia, _pair_force(d, (d * d).sum(1), ea, ga, q[ia] * q[ja], alpha,
                                           w[part]))
    if not verlet:
        f = f - f.mean(0)
    return f + _kspace(L, x, q, m, alpha)[0]


def _md(case, seed, n=None, verlet=False):
    s = _lj(case, seed, n)
    L, dt, d = s["hi"][0], s["params"]["dt"], _device()
    x, v, q = (torch.tensor(s[k], device=d) for k in ("pos", "vel", "q"))
    state = {}

    def force(epoch):
        moved = "at" in state and _separations(torch.cat([state["at"], x]), L,
                                               slice(0, len(x)), slice(len(x), None))
        if "at" not in state or float((moved ** 2).sum(1).max()) > (SKIN / 2) ** 2:
            state["at"], state["pairs"] = x.clone(), _pairs(x, L, CUT_OFF + SKIN)
        m = _k_samples(L, ALPHA, case["p"], SEED, epoch)
        return _forces(s, x, q, epoch, state["pairs"], m, verlet=verlet)

    f = force(0)
    for t in range(case["steps"]):
        v = v + f * (0.5 * dt)
        x = x + v * dt
        x = torch.where(x >= L, x - L, x)
        x = torch.where(x < 0, x + L, x)
        f = force(t + 1)
        v = v + f * (0.5 * dt)
    return s, x, v, f, q


def _trajectory(case, x, v, f):
    """What steps are compared by.  In the mixed form positions alone: after
    tens of steps the velocities and forces of two correct runs differ by the
    one or two pairs that crossed r_core a step earlier in one of them (up to
    1e-5 of the norm each), not by their rounding; the fit case compares the
    mixed form's forces."""
    if case.get("precision", "mixed") == "mixed":
        return {"pos": x, "vel": None, "force": None}
    return {"pos": x, "vel": v, "force": f}


def exact(case, seed):
    kind = case["kind"]
    if kind == "md" and case["neighbor"] == "RBL":
        _, x, v, f, _ = _md(case, seed)
        return _trajectory(case, x, v, f)
    if kind == "thermo":
        s, x, v, f, q = _md(case, seed, verlet=True)
        L = s["hi"][0]
        i, j = _pairs(x, L, CUT_OFF)
        d = _separations(x, L, i, j)
        r2 = (d * d).sum(1)
        r, u, qq = torch.sqrt(r2), 1 / r2 ** 3, q[i] * q[j]
        e_coul = 0.5 * (qq * torch.erfc(math.sqrt(ALPHA) * r) / r).sum()
        fd = _pair_force(d, r2, 1.0, torch.ones_like(r), qq, ALPHA, 1.0)
        vir = [-0.5 * (d[:, a] * fd[:, b]).sum() for a, b in ((0, 0), (1, 1), (2, 2), (0, 1),
                                                             (0, 2), (1, 2))]
        g = np.arange(-case["kmax"], case["kmax"] + 1)
        m = np.stack(np.meshgrid(g, g, g, indexing="ij")).reshape(3, -1)
        m = m[:, (m != 0).any(0)]
        k = 2 * math.pi * torch.tensor(m, dtype=torch.float64, device=x.device) / L
        k2, rho2 = (k * k).sum(0), []
        for a in range(0, k.shape[1], 512):
            ph = x @ k[:, a:a + 512]
            rho2.append((q[:, None] * torch.cos(ph)).sum(0) ** 2 +
                        (q[:, None] * torch.sin(ph)).sum(0) ** 2)
        e_k = (2 * math.pi / L ** 3) * (torch.exp(-k2 / (4 * ALPHA)) / k2 * torch.cat(rho2)).sum()
        return {"pos": x, "vel": v, "force": f, "e_lj": float((2 * (u * u - u)).sum()),
                "e_coul": float(e_coul), "virial": torch.stack(vir),
                "e_k": float(e_k - math.sqrt(ALPHA / math.pi) * (q * q).sum())}
    if kind == "batch":
        out = [_md(case, 1000 * seed + r, n=int(n))[1:4]
               for r, n in enumerate(_replica_sizes(case))]
        return _trajectory(case, *(torch.cat([o[c] for o in out]) for c in range(3)))
    if kind == "fit":
        s, m, theta, target = _fit_inputs(case, seed)
        d = _device()
        th = {k: v.clone().to(d).requires_grad_(True) for k, v in theta.items()}
        pairs = _pairs(th["pos"].detach(), s["hi"][0], CUT_OFF)
        f = _forces(s, th["pos"], th["charge"], 0, pairs, m, th["eps"], th["sigma"], th["alpha"])
        loss = ((f - target.to(d)) ** 2).sum() / len(f)
        loss.backward()
        return {"loss": float(loss.detach()), "force": f.detach(),
                **{k: v.grad for k, v in th.items()}}
    if kind in ("kspace", "dropin"):
        real = torch.float64 if kind == "kspace" else torch.float32
        s = _lj(case, seed)
        L, d = s["hi"][0], _device()
        pos, q = (torch.tensor(s[k], device=d) for k in ("pos", "q"))
        out = {}
        if kind == "dropin":  # the atoms in the cell order that prepare() gave them
            o = _cell_order(s)
            pos, q, s = pos[o].to(real).double(), q[o], dict(s, gid=s["gid"][o])
            i, j, w = _rbl(s, pos, 1, _pairs(pos, L, CUT_OFF))
            f = torch.zeros_like(pos)
            e = _separations(pos, L, i, j)
            f.index_add_(0, i, _pair_force(e, (e * e).sum(1), 1.0, torch.ones_like(w), q[i] * q[j],
                                           ALPHA, w))
            out["f"] = list((f - f.mean(0)).T.contiguous())
        m = _k_samples(L, ALPHA, case["p"], seed, 1)
        fk, re, im, k = _kspace(L, pos, q, m, ALPHA)
        S, V, k2 = float(_gauss_sum(L, ALPHA)), L ** 3, (k * k).sum(0)
        base = 2 * math.pi * S / (case["p"] * V) * (re * re + im * im) / k2
        inner = 2 * (1 / (4 * ALPHA) + 1 / k2)
        vir = [(base * ((1.0 if a == b else 0.0) - inner * k[a] * k[b])).sum()
               for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))]
        self_e = math.sqrt(ALPHA / math.pi) * (q * q).sum() + \
            0.5 * math.pi * q.sum() ** 2 / (ALPHA * V)
        fk = list(fk.T.contiguous())
        out.update(rho=[re, im], virial=torch.stack(vir), energy=(base.sum() - self_e).reshape(1))
        out["f" if kind == "kspace" else "fk"] = fk
        return {key: out.get(key) for key in
                (("rho", "f", "virial", "energy") if kind == "kspace" else
                 ("core_end", "core", "shell_num", "shell", "need", "realloc", "f", "rho", "fk",
                  "virial", "energy"))}
    # water (constraints, thermostat) and the sum-of-Gaussians engine (its
    # set-up tables) are not a few lines of restatement, and lists are whole
    # numbers
    return None
