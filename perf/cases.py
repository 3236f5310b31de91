"""Performance cases of the force-and-integrate engine: what a simulation
program asks of it, from one 60-bead protein to a 200,000-bead condensate and
ensembles of over a thousand chains.

Three kinds of call:
* "frame": one system in a ``Context``; a pass advances it by the steps
  between two trajectory frames and reads the frame (positions, velocities).
* "state": a trajectory frame is handed to a ``Context`` and its forces and
  per-group energies come back (reweighting, energy files, minimisation).
* "batch": an ensemble in a ``Batch``; a pass advances every replica by one
  launch and reads all positions.

Three force fields: "go" (harmonic bonds, Go contacts, flexible-local angles
and dihedrals, excluded volume, Debye-Hueckel), "aicg" (the same with the
AICG2+ Gaussian bonds and dihedrals), "hps" (disordered chains: Ashbaugh-Hatch
Lennard-Jones and Debye-Hueckel; a periodic condensate slab in a Context,
single chains in a Batch).

The engine computes forces and velocities in single precision and trajectory
files hold single-precision frames, so that is what a pass returns.
"""
import math

import numpy as np
import torch

import opencafemol_gb300 as ocm
from opencafemol_gb300 import synth

KCAL = synth.KJ_PER_KCAL
K_BOND = 2.0 * 110.0 * KCAL * 100.0     # folded chains, 110 kcal/mol/A^2
K_BOND_HPS = 2.0 * 10.0 * KCAL * 100.0  # disordered chains, 10 kcal/mol/A^2
SIGMA_MAX = 0.75                        # nm, largest HPS bead
AREA = {"small": 15.0, "large": 30.0}   # box edge in x and y of the slabs, nm
FRICTION, DT = 0.1, 0.01                # 1/ps, ps


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small protein between two saved frames: the latency of short runs
        {"name": "go60_frame", "kind": "frame", "field": "go", "beads": 60, "steps": 50},
        # forces and energies of a mid-sized protein, frame by frame (an odd size)
        {"name": "go317_state", "kind": "state", "field": "go", "beads": 317},
        # a large multi-domain protein with the AICG2+ terms, non-periodic
        {"name": "aicg1511_frame", "kind": "frame", "field": "aicg", "beads": 1511, "steps": 50},
        # a small condensate (31 chains of 97): a run that few SMs could hold
        {"name": "slab3007_frame", "kind": "frame", "field": "hps", "chains": 31, "length": 97, "box": "small",
         "steps": 50},
        # the 100 x 200 condensate slab in a 15 x 15 x 150 nm box
        {"name": "slab20000_frame", "kind": "frame", "field": "hps", "chains": 100, "length": 200, "box": "small",
         "steps": 50},
        # forces and energies of that slab
        {"name": "slab20000_state", "kind": "state", "field": "hps", "chains": 100, "length": 200, "box": "small"},
        # the 1000 x 200 slab in a 30 x 30 x 300 nm box
        {"name": "slab200000_frame", "kind": "frame", "field": "hps", "chains": 1000, "length": 200, "box": "large",
         "steps": 20},
        # a handful of replicas of small proteins: fewer systems than SMs
        {"name": "batch24_small", "kind": "batch", "field": "go", "systems": 24, "lo": 30, "hi": 200, "proteins": 6,
         "steps": 100},
        # the 512-replica ensemble of 50..800-bead proteins
        {"name": "batch512_mix", "kind": "batch", "field": "go", "systems": 512, "lo": 50, "hi": 800,
         "proteins": 32, "steps": 100},
        # many peptides: the smallest systems of a serving stream, several per SM
        {"name": "batch1400_peptides", "kind": "batch", "field": "go", "systems": 1400, "lo": 30, "hi": 80,
         "proteins": 16, "steps": 100},
        # the largest systems of a serving stream
        {"name": "batch160_large", "kind": "batch", "field": "aicg", "systems": 160, "lo": 800, "hi": 2000,
         "proteins": 12, "steps": 50},
        # disordered single chains: the Lennard-Jones terms in the batched path
        {"name": "batch300_idr", "kind": "batch", "field": "hps", "systems": 300, "lo": 50, "hi": 400,
         "proteins": 16, "steps": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["go_frame", "go_state", "slab_frame", "slab_state", "batch", "batch", "batch_idr"])
    if kind == "go_frame":
        return {"kind": "frame", "field": rng.choice(["go", "aicg"]), "beads": _log_int(rng, 31, 1999),
                "steps": rng.choice([20, 50])}
    if kind == "go_state":
        return {"kind": "state", "field": rng.choice(["go", "aicg"]), "beads": _log_int(rng, 31, 1999)}
    if kind.startswith("slab"):
        length = rng.randint(60, 220)
        chains = max(2, _log_int(rng, 2100, 60000) // length)
        box = "small" if chains * length < 30000 else "large"
        case = {"kind": kind[5:], "field": "hps", "chains": chains, "length": length, "box": box}
        return dict(case, steps=rng.choice([20, 50])) if kind == "slab_frame" else case
    lo = _log_int(rng, 30, 700)
    if kind == "batch_idr":
        lo = min(lo, 150)
        return {"kind": "batch", "field": "hps", "systems": _log_int(rng, 8, 400), "lo": lo, "hi": 3 * lo,
                "proteins": 8, "steps": 50}
    most = max(16, min(1400, 200000 // (2 * lo)))
    return {"kind": "batch", "field": rng.choice(["go", "aicg"]), "systems": _log_int(rng, 8, most), "lo": lo,
            "hi": min(2000, 3 * lo), "proteins": 8, "steps": 50}


# ---------------------------------------------------------------------------
# Inputs: chains grown as random walks and pushed off each other, so that a
# run starts near the structures that a simulation visits
# ---------------------------------------------------------------------------
def _orthonormal(b):
    t = torch.zeros_like(b)
    near_x = b[..., 0].abs() > 0.9
    t[..., 0] = (~near_x).to(b.dtype)
    t[..., 1] = near_x.to(b.dtype)
    u = torch.linalg.cross(b, t)
    u = u / u.norm(dim=-1, keepdim=True)
    return u, torch.linalg.cross(b, u)


def _grow(count, length, gen, tries=16, bond=0.38, min_dist=0.45):
    """``count`` random walks of ``length`` beads: bond angles of 1.75 to 2.6
    rad, each bead the first of ``tries`` candidates that keeps ``min_dist``
    from the earlier beads of its chain, or the one that comes nearest to it
    (tries = 1: no such test)."""
    dev = device()
    x = torch.zeros(count, length, 3, dtype=torch.float64, device=dev)
    rnd = torch.rand(length, count, tries, 2, generator=gen, dtype=torch.float64).to(dev)
    start = torch.randn(count, 3, generator=gen, dtype=torch.float64).to(dev)
    d = start / start.norm(dim=-1, keepdim=True)
    if length > 1:
        x[:, 1] = bond * d
    rows = torch.arange(count, device=dev)
    for i in range(2, length):
        u, w = _orthonormal(d)
        th = 1.75 + 0.85 * rnd[i, :, :, :1]
        ph = 2.0 * math.pi * rnd[i, :, :, 1:]
        step = -torch.cos(th) * d[:, None] + torch.sin(th) * (torch.cos(ph) * u[:, None] + torch.sin(ph) * w[:, None])
        pick = torch.zeros(count, dtype=torch.int64, device=dev)
        if tries > 1 and i >= 3:
            cand = x[:, i - 1:i] + bond * step
            near = torch.cdist(cand, x[:, : i - 1], compute_mode="donot_use_mm_for_euclid_dist").amin(dim=2)
            ok = near >= min_dist
            pick = torch.where(ok.any(dim=1), ok.to(torch.int8).argmax(dim=1), near.argmax(dim=1))
        d = step[rows, pick]
        x[:, i] = x[:, i - 1] + bond * d
    return x


def _min_image(d, box):
    return d if box is None else d - box * torch.round(d / box)


def _neighbours(x, box, rc):
    """[n, k] indices of the beads within rc of each bead (-1: none), by a
    cell grid when the box holds one and over all beads otherwise."""
    n, dev = x.shape[0], x.device
    dims = [int(v // rc) for v in box.tolist()] if box is not None else [0, 0, 0]
    gridded = min(dims) >= 3
    if gridded:
        nd = torch.tensor(dims, device=dev)
        c = torch.minimum(((x - box * torch.floor(x / box)) / box * nd).long(), nd - 1)
        key = (c[:, 0] * nd[1] + c[:, 1]) * nd[2] + c[:, 2]
        order = torch.argsort(key, stable=True)
        cells = dims[0] * dims[1] * dims[2]
        counts = torch.bincount(key, minlength=cells)
        first = torch.cumsum(counts, 0) - counts
        table = torch.full((cells, int(counts.max())), -1, dtype=torch.int64, device=dev)
        table[key[order], torch.arange(n, device=dev) - first[key[order]]] = order
        off = torch.tensor([(a, b, g) for a in (-1, 0, 1) for b in (-1, 0, 1) for g in (-1, 0, 1)], device=dev)
    rows, width = [], 1
    chunk = max(1, 40_000_000 // (27 * table.shape[1] if gridded else n))
    for s in range(0, n, chunk):
        e = min(n, s + chunk)
        if gridded:
            around = torch.remainder(c[s:e, None, :] + off, nd)
            cand = table[(around[..., 0] * nd[1] + around[..., 1]) * nd[2] + around[..., 2]].reshape(e - s, -1)
        else:
            cand = torch.arange(n, device=dev).expand(e - s, n)
        r2 = _min_image(x[cand.clamp(min=0)] - x[s:e, None], box).square().sum(-1)
        near = (r2 < rc * rc) & (cand >= 0) & (cand != torch.arange(s, e, device=dev)[:, None])
        k = max(1, int(near.sum(1).max()))
        at = torch.argsort(near.to(torch.int8), dim=1, descending=True, stable=True)[:, :k]
        rows.append(torch.where(near.gather(1, at), cand.gather(1, at), -1))
        width = max(width, k)
    return torch.cat([torch.nn.functional.pad(r, (0, width - r.shape[1]), value=-1) for r in rows])


def _push_off(x, want, next_bond, bond, box, rounds=120, reach=0.45):
    """Moves beads apart until every pair is about ``want(i, j)`` nm apart (0:
    the pair is left alone), keeping the bonds i, i + 1 of ``next_bond``."""
    n = x.shape[0]
    has = next_bond.to(x.dtype)[:, None]
    for it in range(rounds):
        if it % 80 == 0 or it in (10, 20, 40):  # beads travel most at the beginning
            nb = _neighbours(x, box, 2 ** (1 / 6) * SIGMA_MAX + reach)
            j = nb.clamp(min=0)
            w = torch.where(nb >= 0, want(torch.arange(n, device=x.device)[:, None], j), 0.0)
        d = _min_image(x[j] - x[:, None], box)
        r = d.norm(dim=-1).clamp(min=1e-6)
        move = -(0.25 * (w - r).clamp(min=0.0) / r)[..., None] * d
        move = move.sum(dim=1)
        b = _min_image(torch.roll(x, -1, 0) - x, box)
        rb = b.norm(dim=-1, keepdim=True).clamp(min=1e-6)
        pull = 0.45 * (rb - bond) / rb * b * has
        move = move.clamp(-0.05, 0.05) + pull - torch.roll(pull, 1, 0)
        x = x + move
    return x


def _f32(a):
    return np.asarray(a, np.float32).astype(np.float64)


def _maxwell(masses, temperature, rng):
    return _f32(rng.normal(size=(len(masses), 3)) * np.sqrt(synth.BOLTZ * temperature / masses)[:, None])


def _charges(n, fraction, rng):
    q = np.full(n, np.nan)
    pick = rng.choice(n, max(2, int(round(fraction * n))), replace=False)
    q[pick] = rng.choice([-1.0, 1.0], len(pick))
    return q


def _proteins(sizes, seed, aicg):
    """Go-model proteins of the given sizes: a grown chain, relaxed against
    its excluded volume, is the native structure."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator().manual_seed(seed)
    grown = _grow(len(sizes), max(sizes), gen)
    specs = []
    for k, n in enumerate(sizes):
        seq = rng.integers(0, 20, n).astype(np.int32)
        radius = rng.uniform(0.2, 0.4, n)
        x = grown[k, :n]
        rad = torch.from_numpy(radius).to(x.device)
        native = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist") < 0.65

        def want(i, j):
            return torch.where((torch.abs(i - j) > 3) & ~native[i, j], rad[i] + rad[j], 0.0)

        bonded = torch.arange(n, device=x.device) < n - 1
        pos = _f32(_push_off(x, want, bonded, 0.38, None).cpu().numpy())
        native = native.cpu().numpy()
        s = synth.CGSpec(n=n, pos=pos, masses=synth.RESIDUE_MASS[seq].copy(), friction=FRICTION, dt=DT)
        c = np.arange(n)
        s.bonds = np.stack([c[:-1], c[1:]], 1)
        s.bond_v0 = np.linalg.norm(pos[1:] - pos[:-1], axis=1)
        s.bond_k = np.full(n - 1, K_BOND)
        ii, jj = np.nonzero(np.triu(native, k=4))
        s.contacts = np.stack([ii, jj], 1).astype(np.int64)
        s.go_k = rng.uniform(0.2, 1.0, len(ii)) * KCAL
        s.go_r0 = np.linalg.norm(pos[ii] - pos[jj], axis=1)
        s.fla_idx = np.stack([c[:-2], c[1:-1], c[2:]], 1)
        s.fla_k = np.full(n - 2, KCAL)
        s.fla_aa = seq[1:-1]
        s.fld_idx = np.stack([c[:-3], c[1:-2], c[2:-1], c[3:]], 1)
        s.fld_k = np.full(n - 3, KCAL)
        s.fld_aa1, s.fld_aa2 = seq[1:-2], seq[2:-1]
        if aicg:
            synth.add_aicg_gaussians(s, seed + 17 * k)
        top = np.sort(radius)[::-1]
        s.exv = synth.PairTerm(ratio=2.0 / (top[0] + top[1]), p0=radius, eps=0.6 * KCAL, ign_bond=3, ign_contact=1)
        s.dh = synth.PairTerm(ratio=2.0 / _debye(300.0, 0.15)[0], p0=_charges(n, 0.25, rng), ign_bond=3)
        specs.append(s)
    return specs


def _hps(chains, length, edge, seed):
    """Disordered chains: ``chains`` of them in a periodic slab of 3 beads
    per nm^3 (box edge x edge x 10 edge), or one alone (edge = None)."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator().manual_seed(seed)
    n, dev = chains * length, device()
    types = rng.integers(0, 20, n)
    sig = rng.uniform(0.45, SIGMA_MAX, 20)[types]
    lam = rng.uniform(0.0, 1.0, 20)[types]
    if edge is None:
        box = L = None
        x = _grow(1, length, gen)[0]
    else:
        box = (edge, edge, 10.0 * edge)
        L = torch.tensor(box, dtype=torch.float64, device=dev)
        wide = n / (3.0 * edge * edge)
        x = _grow(chains, length, gen, tries=1)
        x = x - x.mean(dim=1, keepdim=True) + torch.rand(chains, 1, 3, generator=gen, dtype=torch.float64).to(dev) * L
        x = x.reshape(n, 3)
        z = torch.remainder(x[:, 2], 2.0 * wide)  # folded into the slab
        x[:, 2] = 0.5 * (L[2] - wide) + torch.where(z > wide, 2.0 * wide - z, z)
    s64 = torch.from_numpy(sig).to(dev)
    idx = torch.arange(n, device=dev)
    bonded = (idx % length) < length - 1

    def want(i, j):
        near = (torch.abs(i - j) == 1) & (torch.minimum(i, j) % length < length - 1)
        return torch.where(near, 0.0, 1.05 * 0.5 * (s64[i] + s64[j]))

    x = _push_off(x, want, bonded, 0.38, L, rounds=400)
    if L is not None:
        x = x - L * torch.floor(x / L)
    pos = _f32(x.cpu().numpy())
    if box is not None:
        pos = np.where(pos >= np.array(box), pos - np.array(box), pos)
    s = synth.CGSpec(n=n, pos=pos, masses=synth.RESIDUE_MASS[types].copy(), periodic=box is not None, box=box,
                     friction=FRICTION, dt=DT)
    b0 = np.nonzero(bonded.cpu().numpy())[0]
    s.bonds = np.stack([b0, b0 + 1], 1)
    s.bond_v0 = np.full(len(b0), 0.38)
    s.bond_k = np.full(len(b0), K_BOND_HPS)
    ratio = 2.0 / (0.5 * (np.sort(sig)[-1] + np.sort(sig)[-2]))
    s.ljr = synth.PairTerm(ratio=ratio, p0=np.full(n, 0.2 * KCAL), p1=sig, ign_bond=1)
    s.lja = synth.PairTerm(ratio=ratio, p0=0.2 * KCAL * lam, p1=sig, ign_bond=1)
    s.dh = synth.PairTerm(ratio=3.5 / _debye(300.0, 0.15)[0], p0=_charges(n, 0.2, rng), ign_bond=3)
    return s


def _sizes(case):
    """Beads of the case's distinct proteins: even over the logarithm."""
    m = min(case["proteins"], case["systems"])
    return [int(v) for v in np.geomspace(case["hi"], case["lo"], m).round()]


def _inputs(case, seed):
    """(specs, replicas): the distinct systems and, for every replica, which
    one it is, its temperature, velocities and noise seed."""
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "batch":
        sizes = _sizes(case)
        specs = ([_hps(1, n, None, 1000 * seed + k) for k, n in enumerate(sizes)] if case["field"] == "hps"
                 else _proteins(sizes, seed, case["field"] == "aicg"))
        of = [k % len(specs) for k in range(case["systems"])]
        temps = rng.uniform(280.0, 360.0, case["systems"])
    else:
        specs = ([_hps(case["chains"], case["length"], AREA[case["box"]], seed)] if case["field"] == "hps"
                 else _proteins([case["beads"]], seed, case["field"] == "aicg"))
        of, temps = [0], [300.0]
    replicas = [(k, float(t), _maxwell(specs[k].masses, t, rng), 1000 + r) for r, (k, t) in enumerate(zip(of, temps))]
    return specs, replicas


def prepare(case, seed):
    specs, replicas = _inputs(case, seed)
    systems = [synth.build_system(s) for s in specs]
    if case["kind"] == "batch":
        beads = sum(specs[k].n for k, _, _, _ in replicas)
        batch = ocm.Batch(max_systems=len(replicas), max_total_beads=beads + 1024,
                          max_beads_per_system=max(s.n for s in specs))
        slots = [batch.admit(systems[k], specs[k].pos, velocities=v, temperature=t, friction=FRICTION, step_size=DT,
                             seed=sd, n_steps=10 ** 12) for k, t, v, sd in replicas]
        return {"kind": "batch", "batch": batch, "slots": np.array(slots, np.int64), "steps": case["steps"],
                "frame": np.zeros((beads, 3))}
    k, t, v, sd = replicas[0]
    ctx = ocm.Context(systems[k], ocm.LangevinIntegrator(t, FRICTION, DT, sd))
    ctx.setPositions(specs[k].pos)
    ctx.setVelocities(v)
    return {"kind": case["kind"], "context": ctx, "frame": specs[k].pos, "steps": case.get("steps"),
            "groups": len(systems[k].group_names())}


def run(state):
    if state["kind"] == "batch":
        batch = state["batch"]
        batch.run(state["steps"])
        return {"positions": batch.get_positions_many(state["slots"], out=state["frame"]).astype(np.float32)}
    ctx = state["context"]
    if state["kind"] == "state":
        ctx.setPositions(state["frame"])
        forces, total = ctx.getState()
        energies = ctx.getGroupEnergies()[: state["groups"]]
        return {"forces": forces.astype(np.float32), "energies": np.append(energies, total).astype(np.float32)}
    ctx.step(state["steps"])
    return {"positions": ctx.getPositions().astype(np.float32), "velocities": ctx.getVelocities().astype(np.float32)}


def work(case):
    """State in and out once a pass and parameters once; operations per MD
    step from the pairs within the cutoffs (coils: a few per bead, slab: 3
    beads per nm^3) and the bonded terms."""
    hps = case["field"] == "hps"
    if case["kind"] == "batch":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        beads = case["systems"] * mean
    else:
        mean = beads = case["chains"] * case["length"] if hps else case["beads"]
    steps = case.get("steps", 1)
    slab = case["kind"] != "batch" and hps
    pairs = 50.0 + 0.2 * 0.2 * 270.0 if slab else min(0.45 * mean, 15.0)
    bonded = 70.0 if hps else 300.0 + (110.0 if case["field"] == "aicg" else 0.0)
    params = 36.0 + (24.0 if hps else 120.0)
    return {"bytes": beads * (24.0 + 12.0 + 4.0 + 24.0 + 12.0 + params),
            "flops": beads * steps * (62.0 * pairs + bonded + 40.0)}


# ---------------------------------------------------------------------------
# The same passes in 64 bits, from the force field's expressions
# ---------------------------------------------------------------------------
def _debye(temperature, ionic):
    """Debye length (nm) and 1 / (4 pi eps0 eps_r) (kJ nm / mol / e^2)."""
    na, kb, e = 6.02214076e23, 1.380649e-23, 1.6021766208e-19
    eps_r = (249.4 - 0.788 * temperature + 7.2e-4 * temperature ** 2) * \
        (1.0 - 2.551e-1 * ionic + 5.151e-2 * ionic ** 2 - 6.889e-3 * ionic ** 3)
    eps0 = 8.854187817e-12 * 1.0e-6 / na / e / e
    lam = math.sqrt(eps0 * eps_r * kb * 1.0e-3 * temperature / (2.0 * ionic * 1.0e-24))
    return lam, 1.0 / (4.0 * math.pi * eps0 * eps_r)


def _spline_coefficients(y, h):
    """Natural cubic spline: second derivatives at the nodes."""
    m = len(y)
    a = np.zeros((m, m))
    r = np.zeros(m)
    a[0, 0] = a[-1, -1] = 1.0
    for k in range(1, m - 1):
        a[k, k - 1:k + 2] = 1.0, 4.0, 1.0
        r[k] = 6.0 * (y[k + 1] - 2.0 * y[k] + y[k - 1]) / (h * h)
    return np.linalg.solve(a, r)


class _Exact:
    """Energy of one or more independent systems in FP64, forces by automatic
    differentiation, pairs from neighbour lists with a wide skin."""

    SKIN = 0.8
    TH0, TH1 = 1.30900, 2.87979
    NODES = np.array([1.30900, 1.48353, 1.65806, 1.83260, 2.00713, 2.18166, 2.35619, 2.53073, 2.70526, 2.87979])

    def __init__(self, specs):
        self.dev = device()
        self.specs = specs
        self.n = sum(s.n for s in specs)
        self.starts = np.cumsum([0] + [s.n for s in specs])
        self.box = None if specs[0].box is None else self.t(specs[0].box)
        self.hps = specs[0].ljr is not None
        cat = self.cat
        self.bonds, self.v0, self.kb = cat("bonds", True), cat("bond_v0"), cat("bond_k")
        self.go, self.gok, self.gor = cat("contacts", True), cat("go_k"), cat("go_r0")
        self.gb, self.gbk, self.gbv, self.gbs = cat("gb_idx", True), cat("gb_k"), cat("gb_v0"), cat("gb_sigma")
        self.gd, self.gdk, self.gdt, self.gds = cat("gd_idx", True), cat("gd_k"), cat("gd_theta0"), cat("gd_sigma")
        self.fla, self.flak = cat("fla_idx", True), cat("fla_k")
        self.fld, self.fldk = cat("fld_idx", True), cat("fld_k")
        if not self.hps:
            self._tables()
        self._pair_parameters()

    def t(self, a):
        return torch.as_tensor(np.ascontiguousarray(a), device=self.dev)

    def cat(self, name, index=False):
        parts = [np.asarray(getattr(s, name)) + (self.starts[k] if index else 0) for k, s in enumerate(self.specs)]
        return self.t(np.concatenate(parts))

    def _tables(self):
        h = (self.TH1 - self.TH0) / 9.0
        aa = np.concatenate([s.fla_aa for s in self.specs])
        y = np.stack([ocm.fla_spline_table(a) for a in ocm.AMINO_ACIDS])
        self.y, self.m2 = self.t(y)[aa], self.t(np.stack([_spline_coefficients(v, h) for v in y]))[aa]
        grid = np.arange(self.TH0, self.TH1, 1e-4)
        emin = []
        for k, a in enumerate(ocm.AMINO_ACIDS):
            # the lowest point of the published spline, on its nodes and second derivatives as printed
            d2 = ocm.fla_second_derivative_table(a)
            q = np.minimum(8, ((grid - self.TH0) / h).astype(int))
            q = np.where(self.NODES[q + 1] < grid, q + 1, np.where(grid < self.NODES[q], q - 1, q))
            c, b = (self.NODES[q + 1] - grid) / h, (grid - self.NODES[q]) / h
            emin.append(min(y[k][0], np.min(c * y[k][q] + b * y[k][q + 1] + ((c ** 3 - c) * d2[q] + (b ** 3 - b)
                                                                             * d2[q + 1]) * h * h / 6.0)))
        self.fla_min = self.t(np.array(emin))[aa]
        # the Fourier tables that a pair of residues selects
        a1 = np.concatenate([s.fld_aa1 for s in self.specs])
        a2 = np.concatenate([s.fld_aa2 for s in self.specs])
        names = np.array(ocm.AMINO_ACIDS)
        n1, n2 = names[a1], names[a2]
        phi = np.arange(-math.pi, math.pi, 1e-4)
        base = np.stack([np.ones_like(phi), np.cos(phi), np.sin(phi), np.cos(2 * phi), np.sin(2 * phi),
                         np.cos(3 * phi), np.sin(3 * phi)])
        coef = np.zeros((len(a1), 7))
        low = np.zeros(len(a1))
        for key in ocm.fld_table_keys():
            first, second = key.split("-")
            if second == "GLY":
                sel = n2 == "GLY"
            elif second == "PRO":
                sel = (n2 == "PRO") & ((n1 == "GLY") if first == "GLY" else True)
            else:
                sel = ~np.isin(n2, ("GLY", "PRO")) & (n1 == first)
            tab = ocm.fld_fourier_table(key)
            coef[sel] += tab
            low[sel] += np.min(tab @ base)
        self.fldc, self.fld_min = self.t(coef), self.t(low)

    def _pair_parameters(self):
        s0 = self.specs[0]
        q = np.concatenate([np.nan_to_num(s.dh.p0) for s in self.specs])
        self.q = self.t(q)
        lam = [_debye(300.0, s.dh.ionic_strength) for s in self.specs]
        self.lam, self.ke = lam[0]
        self.dh_rc = s0.dh.ratio * self.lam
        rep = lambda v: self.t(np.repeat(np.array(v), [s.n for s in self.specs]))  # noqa: E731
        if self.hps:
            self.sig = self.t(np.concatenate([s.ljr.p1 for s in self.specs]))
            self.ea = self.t(np.concatenate([s.lja.p0 for s in self.specs]))
            self.er = float(s0.ljr.p0[0])
            self.lj_rc = rep([s.ljr.ratio * 0.5 * np.sort(s.ljr.p1)[-2:].sum() for s in self.specs])
        else:
            self.rad = self.t(np.concatenate([s.exv.p0 for s in self.specs]))
            self.exv_rc = rep([s.exv.ratio * np.sort(s.exv.p0)[-2:].sum() for s in self.specs])
        # chain position and chain of every bead (exclusions count bonds)
        self.chain = torch.zeros(self.n, dtype=torch.int64, device=self.dev)
        link = torch.zeros(self.n, dtype=torch.int64, device=self.dev)
        link[self.bonds[:, 1]] = 1
        self.chain = torch.cumsum(1 - link, 0)
        self.native = torch.sort(self.go.min(1).values * self.n + self.go.max(1).values).values

    def lists(self, x):
        """Pairs within reach of each cutoff, without the excluded ones."""
        def pairs(sel, rc):
            out = []
            if self.box is not None:
                ids = torch.nonzero(sel)[:, 0]
                groups = [(ids, x[ids])]
            else:
                groups = []
                for k in range(len(self.specs)):
                    ids = torch.nonzero(sel[self.starts[k]:self.starts[k + 1]])[:, 0] + int(self.starts[k])
                    groups.append((ids, x[ids]))
            for ids, xs in groups:
                if self.box is None:
                    d = torch.cdist(xs, xs, compute_mode="donot_use_mm_for_euclid_dist")
                    p = torch.nonzero(torch.triu(d < rc + self.SKIN, 1))
                else:
                    nb = _neighbours(xs, self.box, rc + self.SKIN)
                    row, col = torch.nonzero(nb >= 0, as_tuple=True)
                    to = nb[row, col]
                    p = torch.stack([row[row < to], to[row < to]], 1)
                out.append(ids[p])
            p = torch.cat(out)
            return p.min(1).values, p.max(1).values

        def apart(i, j, bonds):
            return (self.chain[i] != self.chain[j]) | (j - i > bonds)

        i, j = pairs(torch.ones(self.n, dtype=torch.bool, device=self.dev), 2.0)
        if self.hps:
            keep = apart(i, j, 1)
        else:
            keep = apart(i, j, 3)
            if len(self.native):
                at = torch.searchsorted(self.native, i * self.n + j).clamp(max=len(self.native) - 1)
                keep &= self.native[at] != i * self.n + j
        self.pi, self.pj = i[keep], j[keep]
        i, j = pairs(self.q != 0, self.dh_rc)
        keep = apart(i, j, 3)
        self.ci, self.cj = i[keep], j[keep]

    def sep(self, x, i, j):
        return _min_image(x[j] - x[i], self.box)

    def energies(self, x):
        """Energy per force group, in the order the groups are made."""
        out = [0.5 * (self.kb * (self.sep(x, self.bonds[:, 0], self.bonds[:, 1]).norm(dim=1) - self.v0) ** 2).sum()]
        if len(self.go):
            t2 = self.gor ** 2 / self.sep(x, self.go[:, 0], self.go[:, 1]).square().sum(1)
            out.append((self.gok * (5.0 * t2 ** 6 - 6.0 * t2 ** 5)).sum())
        if len(self.gb):
            r = self.sep(x, self.gb[:, 0], self.gb[:, 1]).norm(dim=1)
            out.append((self.gbk * torch.exp(-0.5 * ((r - self.gbv) / self.gbs) ** 2)).sum())
        if len(self.fla):
            out.append(self._angles(x))
        if len(self.gd):
            d = self._phi(x, self.gd) - self.gdt
            d = d - 2.0 * math.pi * torch.floor((d + math.pi) / (2.0 * math.pi))
            out.append((self.gdk * torch.exp(-0.5 * (d / self.gds) ** 2)).sum())
        if len(self.fld):
            p, c = self._phi(x, self.fld), self.fldc
            e = c[:, 0] + c[:, 1] * torch.cos(p) + c[:, 2] * torch.sin(p) + c[:, 3] * torch.cos(2 * p) + \
                c[:, 4] * torch.sin(2 * p) + c[:, 5] * torch.cos(3 * p) + c[:, 6] * torch.sin(3 * p) - self.fld_min
            out.append((self.fldk * e).sum())
        with torch.no_grad():
            rc = self.lj_rc if self.hps else self.exv_rc
            near = self.sep(x, self.pi, self.pj).square().sum(1) < rc[self.pi] ** 2
            i, j = self.pi[near], self.pj[near]
            near = self.sep(x, self.ci, self.cj).square().sum(1) < self.dh_rc ** 2
            a, b = self.ci[near], self.cj[near]
        r2 = self.sep(x, i, j).square().sum(1)
        if self.hps:
            sg = 0.5 * (self.sig[i] + self.sig[j])
            s6 = (sg * sg / r2) ** 3
            core = r2 <= 2.0 ** (1.0 / 3.0) * sg * sg
            out.append((torch.where(core, self.er * (4.0 * (s6 * s6 - s6) + 1.0), 0.0)).sum())
            r, rc = torch.sqrt(r2), self.lj_rc[i]
            w = ((r - 0.9 * rc) / (0.1 * rc)).clamp(min=0.0)
            sw = 1.0 - 10.0 * w ** 3 + 15.0 * w ** 4 - 6.0 * w ** 5
            ea = 0.5 * (self.ea[i] + self.ea[j])
            out.append((ea * torch.where(core, -torch.ones_like(r2), 4.0 * (s6 * s6 - s6)) * sw).sum())
        else:
            sg2 = (self.rad[i] + self.rad[j]) ** 2
            out.append(0.6 * KCAL * ((sg2 / r2) ** 6 - (sg2 / self.exv_rc[i] ** 2) ** 6).sum())
        r = self.sep(x, a, b).norm(dim=1)
        shift = math.exp(-self.dh_rc / self.lam) / self.dh_rc
        out.append((self.ke * self.q[a] * self.q[b] * (torch.exp(-r / self.lam) / r - shift)).sum())
        return out

    def _angles(self, x):
        h = (self.TH1 - self.TH0) / 9.0
        u = self.sep(x, self.fla[:, 1], self.fla[:, 0])
        v = self.sep(x, self.fla[:, 1], self.fla[:, 2])
        th = torch.atan2(torch.linalg.cross(u, v).norm(dim=1), (u * v).sum(1))
        k = ((th.detach() - self.TH0) / h).floor().clamp(0, 8).long()[:, None]
        b = (th - self.TH0) / h - k[:, 0]
        a = 1.0 - b
        g = lambda tab, o: tab.gather(1, k + o)[:, 0]  # noqa: E731
        s = a * g(self.y, 0) + b * g(self.y, 1) + ((a ** 3 - a) * g(self.m2, 0) + (b ** 3 - b) * g(self.m2, 1)) * h * h / 6
        s = torch.where(th < self.TH0, 30.0 * (self.TH0 - th) + self.y[:, 0], s)
        s = torch.where(th > self.TH1, 30.0 * (th - self.TH1) + self.y[:, 9], s)
        return (self.flak * (s - self.fla_min)).sum()

    def _phi(self, x, q):
        b1, b2, b3 = (self.sep(x, q[:, k], q[:, k + 1]) for k in range(3))
        n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
        return torch.atan2(b2.norm(dim=1) * (b1 * n2).sum(1), (n1 * n2).sum(1))

    def forces(self, x):
        x = x.detach().requires_grad_(True)
        e = self.energies(x)
        f = -torch.autograd.grad(sum(e), x)[0]
        return f, [float(v.detach()) for v in e]


def _noise(beads, seeds, step):
    """Three normals per bead: Philox4x32-10 of (bead, step) under each
    replica's seed, Box-Muller from 24-bit uniforms."""
    lo, m32 = np.uint64(0xFFFFFFFF), np.uint64(32)
    c = [beads.astype(np.uint64), np.full(len(beads), step & 0xFFFFFFFF, np.uint64),
         np.zeros(len(beads), np.uint64), np.zeros(len(beads), np.uint64)]
    k0, k1 = seeds.astype(np.uint64), np.uint64(0x6F636D31)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> m32) ^ c[1] ^ k0, p1 & lo, (p0 >> m32) ^ c[3] ^ k1, p0 & lo]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & lo, (k1 + np.uint64(0xBB67AE85)) & lo
    u = [((v >> np.uint64(8)) + np.uint64(1)).astype(np.float64) / 16777216.0 for v in c]
    a, b = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    p, q = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return np.stack([a * np.cos(p), a * np.sin(p), b * np.cos(q)], 1)


def exact(case, seed):
    specs, replicas = _inputs(case, seed)
    all_specs = [specs[k] for k, _, _, _ in replicas]
    model = _Exact(all_specs)
    x = model.t(np.concatenate([s.pos for s in all_specs]))
    model.lists(x)
    if case["kind"] == "state":
        f, e = model.forces(x)
        return {"forces": f.cpu().numpy(), "energies": np.array(e + [sum(e)])}
    beads = np.concatenate([np.arange(s.n) for s in all_specs])
    noise_seeds = np.concatenate([np.full(specs[k].n, sd) for k, _, _, sd in replicas])
    kt = model.t(np.concatenate([np.full(specs[k].n, synth.BOLTZ * t) for k, t, _, _ in replicas]))[:, None]
    im = model.t(1.0 / np.concatenate([s.masses for s in all_specs]))[:, None]
    v = model.t(np.concatenate([w for _, _, w, _ in replicas]))
    keep = math.exp(-FRICTION * DT)
    kick = (1.0 - keep) / FRICTION
    sq = torch.sqrt(kt * (1.0 - keep * keep) * im)
    for step in range(case["steps"]):
        f, _ = model.forces(x)
        v = keep * v + kick * im * f + sq * model.t(_noise(beads, noise_seeds, step))
        x = x + v * DT
    if case["kind"] == "batch":
        return {"positions": x.cpu().numpy()}
    return {"positions": x.cpu().numpy(), "velocities": v.cpu().numpy()}
