"""The batched kernel's classes of systems (excluded volume + Debye-Hueckel;
Lennard-Jones + Debye-Hueckel with a longer Debye-Hueckel cutoff; everything
else): forces and energies against the FP64 oracle, and trajectories that do
not depend on which classes a launch holds nor on list overflow."""
import numpy as np
import pytest

from conftest import rel_force_err

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-4   # FP32 pair arithmetic, the bar of the parity tests
ENERGY_TOL = 1e-5


def _chain(kind, n, seed):
    """A coil of n beads: "go" is the Go protein; "hps" swaps the excluded
    volume for both Lennard-Jones terms and lets Debye-Hueckel reach 3.5 nm;
    "general" gives one bead another attractive sigma; "dh" keeps
    Debye-Hueckel alone; "neutral" has no charge at all."""
    from opencafemol_gb300 import synth
    s = synth.go_protein(n, seed)
    if kind in ("hps", "general"):
        rng = np.random.default_rng(seed)
        sig = rng.uniform(0.35, 0.45, n)
        ratio = 2.0 / np.sort(sig)[-2:].mean()
        s.exv = None
        s.ljr = synth.PairTerm(ratio=ratio, p0=np.full(n, 0.8), p1=sig, ign_bond=3)
        s.lja = synth.PairTerm(ratio=ratio, p0=rng.uniform(0.0, 0.8, n), p1=sig.copy(), ign_bond=3)
        s.dh.ratio = 3.5 / synth.debye_length(300.0, 0.15)
        if kind == "general":
            s.lja.p1[n // 2] = s.ljr.p1[n // 2] * 0.99
    elif kind == "dh":
        s.exv = None
    elif kind == "neutral":
        s.dh = None
    return s


def _check_state(batch, slot, system, spec):
    from oracle import oracle
    f, e = batch.state(slot)
    f_ref, e_ref = oracle.evaluate(spec)
    assert rel_force_err(f, f_ref) <= FORCE_TOL
    for g, name in enumerate(system.group_names()):
        assert abs(e[g] - e_ref[name]) <= ENERGY_TOL * max(1.0, abs(e_ref[name])), name


@pytest.mark.parametrize("kind", ["go", "hps", "general", "dh", "neutral"])
@pytest.mark.parametrize("n", [5, 33, 64, 129, 257, 513, 800])
def test_class_forces_and_group_masks(gpu, kind, n):
    """Sizes around the edges of the pair split and of a cluster."""
    from opencafemol_gb300 import synth
    spec = _chain(kind, n, 40 + n)
    system = synth.build_system(spec)
    b = gpu.Batch(max_systems=1, max_total_beads=1024, max_beads_per_system=1024)
    slot = b.admit(system, spec.pos, seed=1, n_steps=1)
    _check_state(b, slot, system, spec)
    total, masked = b.state(slot)[0], np.zeros((n, 3))
    for g in range(len(system.group_names())):
        masked += b.state(slot, groups=1 << g)[0]
    assert np.allclose(masked, total, rtol=0, atol=1e-5 * max(1.0, np.abs(total).max()))


def test_same_alone_and_among_other_classes(gpu):
    """The kernel is chosen by the classes of the whole launch, the inner
    loops by each system's own class: a system's bits are the same alone and
    with any other class, in any launch shape, for any chunking."""
    from opencafemol_gb300 import synth
    kinds = [("go", 70), ("hps", 150), ("general", 90), ("hps", 400), ("go", 300), ("neutral", 40)]
    specs = [_chain(k, n, 60 + n) for k, n in kinds]
    systems = [synth.build_system(s) for s in specs]
    def run(which, threads, chunks):
        b = gpu.Batch(max_systems=len(which), max_total_beads=2048, max_beads_per_system=512)
        b.set_threads(threads)
        slots = [b.admit(systems[k], specs[k].pos, seed=5 + k, n_steps=120) for k in which]
        for c in chunks:
            b.run(c)
        return {k: (b.positions(s), b.velocities(s)) for k, s in zip(which, slots)}
    mix = run(range(len(kinds)), 512, [120])
    again = run([0, 1, 3, 4], 256, [7, 50, 63])  # without the general class
    for k in range(len(kinds)):
        alone = run([k], 512, [60, 60])[k]
        for other in (mix[k],) + ((again[k],) if k in again else ()):
            assert np.array_equal(alone[0], other[0]) and np.array_equal(alone[1], other[1]), kinds[k]


@pytest.mark.parametrize("kind", ["go", "hps", "general"])
@pytest.mark.parametrize("n", [60, 200, 600])
def test_overflow_scan_is_bit_identical(gpu, kind, n):
    """Lists sized from a straight chain overflow on the coil's positions:
    that launch scans, with the bits of a run whose lists were large enough."""
    from opencafemol_gb300 import synth
    spec = _chain(kind, n, 80 + n)
    system = synth.build_system(spec)
    straight = np.zeros((n, 3))
    straight[:, 0] = 0.38 * np.arange(n)
    v0 = np.random.default_rng(2).normal(scale=0.2, size=(n, 3)).astype(np.float32).astype(np.float64)
    out = []
    for start in (straight, spec.pos):
        b = gpu.Batch(max_systems=1, max_total_beads=1024, max_beads_per_system=1024)
        slot = b.admit(system, start, temperature=300.0, seed=9, n_steps=60)
        b.set_positions_many([slot], spec.pos, v0)
        b.run(30)
        b.run(30)
        out.append((b.positions(slot), b.velocities(slot)))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("kind", ["hps", "general"])
def test_bead_limit_of_a_batch(gpu, kind):
    """A batch for up to 1,888 beads per system takes a system of any class,
    the largest included."""
    from opencafemol_gb300 import synth
    b = gpu.Batch(max_systems=2, max_total_beads=4096, max_beads_per_system=1888)
    for n in (60, 1888):
        spec = _chain(kind, n, 90 + n)
        system = synth.build_system(spec)
        slot = b.admit(system, spec.pos, seed=1, n_steps=5)
        _check_state(b, slot, system, spec)
    b.run(5)
    assert all(b.status(s) == 0 and b.steps_done(s) == 5 for s in range(2))


@pytest.mark.parametrize("terms", ["all", "wca_exv", "uniform_dh", "lja"])
@pytest.mark.parametrize("n", [7, 65, 256, 600])
def test_general_terms(gpu, terms, n):
    """The General class with every pair term at once and with subsets (each
    term is a block of its own in the inner loop): forces, energies and the
    groups one at a time; the scan gives the list's bits."""
    from opencafemol_gb300 import synth
    spec = _chain("go", n, 700 + n)
    rng = np.random.default_rng(n)
    side = np.zeros(n, np.int8)
    side[: max(1, n // 2)] |= 1
    side[n // 3:] |= 2
    if terms in ("all", "lja"):
        sig = rng.uniform(0.35, 0.45, n)
        spec.lja = synth.PairTerm(ratio=2.0 / np.sort(sig)[-2:].mean(), p0=rng.uniform(0.0, 0.8, n), p1=sig, ign_bond=2)
    if terms == "all":
        spec.ljr = synth.PairTerm(ratio=4.0, p0=np.full(n, 0.8), p1=rng.uniform(0.35, 0.45, n), ign_bond=1)
    elif terms == "lja":
        spec.exv = spec.dh = None
    elif terms == "wca_exv":
        spec.dh = None
        spec.ljr = synth.PairTerm(ratio=0.0, p0=rng.uniform(0.3, 1.5, n), p1=rng.uniform(0.35, 0.55, n), kind="wca",
                                  ign_bond=1)
    else:
        spec.exv = None
        spec.lja = synth.PairTerm(ratio=3.0, p0=np.full(n, 0.6), p1=np.full(n, 0.4), kind="uniform", side=side, ign_bond=1)
    system = synth.build_system(spec)
    b = gpu.Batch(max_systems=2, max_total_beads=2048, max_beads_per_system=1024)
    slot = b.admit(system, spec.pos, seed=1, n_steps=1)
    _check_state(b, slot, system, spec)
    f, _ = b.state(slot)
    parts = sum(b.state(slot, groups=1 << g)[0] for g in range(len(system.group_names())))
    assert np.allclose(parts, f, rtol=0, atol=1e-5 * max(1.0, np.abs(f).max()))
    straight = np.zeros((n, 3))
    straight[:, 0] = 0.38 * np.arange(n)  # too short lists for the coil: the scan
    other = b.admit(system, straight, seed=1, n_steps=1)
    b.set_positions_many([other], spec.pos)
    assert np.array_equal(b.state(other)[0], f)


@pytest.mark.parametrize("kind", ["go", "hps", "general"])
@pytest.mark.parametrize("n", [64, 200, 400])
def test_list_capacity_is_per_bead(gpu, kind, n):
    """slot_stats counts the entries of a bead, however many units share
    them: room for every partner that the positions at admission have."""
    from opencafemol_gb300 import synth
    spec = _chain(kind, n, 20 + n)
    b = gpu.Batch(max_systems=1, max_total_beads=1024, max_beads_per_system=512)
    slot = b.admit(synth.build_system(spec), spec.pos, seed=1, n_steps=1)
    reach = 3.5 if kind == "general" else 2.0  # the main list's cutoff
    d = np.linalg.norm(spec.pos[:, None] - spec.pos[None], axis=2)
    partners = int((d < reach).sum(axis=1).max()) - 1
    capacity = b.slot_stats(slot)["list_capacity"]
    assert partners <= capacity <= n + 32
