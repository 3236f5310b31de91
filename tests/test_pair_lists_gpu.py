"""The per-bead pair lists of the plain path (both Lennard-Jones terms of a
large periodic system) where they can go wrong: against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_force_err

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-4   # FP32 pair arithmetic, the bar of the parity tests
ENERGY_TOL = 1e-5


def _slab(kind):
    from opencafemol_gb300 import synth
    if kind == "narrow":  # 6 nm wide: neighbour shifts near half the box need the minimum image
        spec = synth.hps_slab(23, 97, (6.0, 6.5, 110.0), slab_width=40.0, seed=3, dh_cutoff=2.2)
        spec.dh = None
        return spec
    cutoff = {"far": 4.0}.get(kind, 2.0)  # 4 nm: more neighbour clusters than a block stages, so tiles
    spec = synth.hps_slab(23, 97, (15.0, 15.0, 50.0), slab_width=14.0, seed=5, hps_cutoff=cutoff)
    if kind == "sigmas":  # the two terms' sigmas differ, and with them the cutoffs
        spec.lja.p1 = spec.lja.p1 * np.random.default_rng(1).uniform(0.9, 1.1, spec.n)
    elif kind == "molecules":  # exclusion rows of 96 partners
        spec.ljr.ign_molecule = spec.lja.ign_molecule = True
    elif kind == "empty":  # no attraction: zero epsilons
        spec.lja.p0 = np.zeros(spec.n)
    return spec


@pytest.mark.parametrize("kind", ["plain", "sigmas", "molecules", "empty", "narrow", "far"])
def test_forces_and_energies(gpu, kind):
    from opencafemol_gb300 import synth
    from oracle import oracle
    spec = _slab(kind)
    system = synth.build_system(spec)
    ctx = gpu.Context(system, gpu.LangevinIntegrator(spec.temperature, 5.0, 0.002, 7))
    ctx.setPositions(spec.pos)
    ctx.setVelocitiesToTemperature(spec.temperature, 3)
    L = np.asarray(spec.box)
    for _ in range(2):  # as packed, and after the lists were rebuilt during a run
        f, _ = ctx.getState(energy=False)
        x = ctx.getPositions()
        f_ref, e_ref = oracle.evaluate(spec, pos=x)
        assert rel_force_err(f, f_ref) <= FORCE_TOL
        e = ctx.getGroupEnergies()
        for g, name in enumerate(system.group_names()):
            assert abs(e[g] - e_ref[name]) <= ENERGY_TOL * max(1.0, abs(e_ref[name])), name
        ctx.step(200)
        x = ctx.getPositions()
        x = (x - L * np.floor(x / L)).astype(np.float32).astype(np.float64)
        ctx.setPositions(np.where(x >= L, x - L, x))  # FP32-exact for both sides
    assert ctx.stats()["reordered"] == 1


def test_repeated_runs_are_bit_identical(gpu):
    """List order and sums do not depend on the timing of the build."""
    from opencafemol_gb300 import synth
    spec = _slab("plain")
    system = synth.build_system(spec)
    out = []
    for _ in range(2):
        ctx = gpu.Context(system, gpu.LangevinIntegrator(spec.temperature, 5.0, 0.002, 7))
        ctx.setPositions(spec.pos)
        ctx.setVelocitiesToTemperature(spec.temperature, 3)
        ctx.step(120)
        out.append((ctx.getPositions(), ctx.getVelocities()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_globule_with_nearly_every_bead_in_range(gpu):
    """3,007 beads in a ball of 4.2 nm under a 4 nm cutoff: about 375 entries
    per unit, so the head-room reaches the most that a unit can hold (every
    staged bead, 512), and that is where it stops."""
    from opencafemol_gb300 import synth
    from oracle import oracle
    spec = synth.hps_slab(31, 97, (20.0, 20.0, 20.0), slab_width=18.0, seed=9, hps_cutoff=4.0)
    spec.dh = None
    side = 0.47 * np.arange(-10, 11)
    grid = np.array([(x, y, z) for a, z in enumerate(side) for b, y in enumerate(side[:: 1 - 2 * (a % 2)])
                     for x in side[:: 1 - 2 * (b % 2)]])  # neighbours in the chain are neighbours in space
    r = np.linalg.norm(grid, axis=1)
    ball = grid[np.sort(np.argsort(r, kind="stable")[: spec.n])]
    spec.pos = (10.0 + ball + np.random.default_rng(4).normal(scale=0.01, size=ball.shape)).astype(np.float32).astype(np.float64)
    spec.bond_v0 = np.linalg.norm(np.diff(spec.pos, axis=0), axis=1)[spec.bonds[:, 0]]
    assert (np.linalg.norm(spec.pos - 10.0, axis=1) < 4.25).mean() > 0.95  # partners of the middle bead
    system = synth.build_system(spec)
    ctx = gpu.Context(system, gpu.LangevinIntegrator(spec.temperature, 5.0, 0.001, 7))
    ctx.setPositions(spec.pos)
    f, _ = ctx.getState(energy=False)
    f_ref, _ = oracle.evaluate(spec)
    assert rel_force_err(f, f_ref) <= FORCE_TOL
    st = ctx.stats()
    assert st["masked_tiles"] == 0 and st["tiles"] > 0  # the lists, not the tiles
    ctx.step(20)
    assert np.all(np.isfinite(ctx.getPositions()))


def test_neighbourhood_of_many_columns(gpu):
    """A rod of 17,000 beads along z in a box of 23 x 23 columns, all within
    the 19 nm cutoff of each other: few of them hold a cluster."""
    from opencafemol_gb300 import synth
    from oracle import oracle
    chains, length = 170, 100
    n, a = chains * length, 0.47
    spec = synth.hps_slab(30, 100, (15.0, 15.0, 60.0), slab_width=20.0, seed=6, hps_cutoff=19.0)
    k = np.arange(n)
    layer, site = k // 16, k % 16
    site = np.where(layer % 2, 15 - site, site)
    y = site // 4
    x = np.where(y % 2, 3 - site % 4, site % 4)
    spec.n, spec.box = n, (44.0, 44.0, 520.0)
    pos = np.stack([21.3 + a * x, 21.3 + a * y, 3.0 + a * layer], 1)
    spec.pos = (pos + np.random.default_rng(8).normal(scale=0.01, size=pos.shape)).astype(np.float32).astype(np.float64)
    tile = lambda v: np.resize(v, n)
    spec.masses = tile(spec.masses)
    for t in (spec.ljr, spec.lja):
        t.p0, t.p1 = tile(t.p0), tile(t.p1)
    spec.dh = None
    b0 = (np.arange(chains)[:, None] * length + np.arange(length - 1)[None]).ravel()
    spec.bonds = np.stack([b0, b0 + 1], 1)
    spec.bond_v0 = np.linalg.norm(spec.pos[b0 + 1] - spec.pos[b0], axis=1)
    spec.bond_k = np.full(len(b0), spec.bond_k[0])
    ctx = gpu.Context(synth.build_system(spec), gpu.LangevinIntegrator(spec.temperature, 5.0, 0.001, 7))
    ctx.setPositions(spec.pos)
    f, _ = ctx.getState(energy=False)
    f_ref, _ = oracle.evaluate(spec, cells=0)
    assert rel_force_err(f, f_ref) <= FORCE_TOL
    assert ctx.stats()["masked_tiles"] == 0  # the lists
    ctx.step(10)
    assert np.all(np.isfinite(ctx.getPositions()))
