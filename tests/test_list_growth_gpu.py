"""Lists that outgrow their buffers: in the middle of a step call (pair
lists, and the way from them to the tiles), at the first evaluation (tiles and
masks), and in a batch; which pair path a periodic system takes; and steps
whose kernels overlap, against the oracle's trajectory."""
import numpy as np
import pytest

from conftest import rel_force_err

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-4   # FP32 pair arithmetic, the bar of the parity tests


def _cube(spec, spacing, edge):
    """The beads on a cubic lattice, row by row."""
    side = int(np.ceil(spec.n ** (1 / 3)))
    k = np.arange(spec.n)
    pos = 10.0 + spacing * np.stack([k % side, k // side % side, k // side ** 2], 1)
    pos += np.random.default_rng(3).normal(scale=0.01, size=pos.shape)
    assert pos.max() < edge
    return pos.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("cutoff,lists", [(2.0, True), (4.0, False)])
def test_growth_inside_step(gpu, cutoff, lists):
    """Lists sized on a sparse lattice, then a dense one at the same column
    layout: that step call overflows (27 -> 95 neighbour clusters, or more than
    a block stages, and 4 -> 40 entries per unit), restores its state, makes
    room and runs, with the bits of a context that never saw the sparse one."""
    from opencafemol_gb300 import synth
    edge = 56.0
    spec = synth.hps_slab(46, 97, (15.0, 15.0, 60.0), slab_width=30.0, seed=7, hps_cutoff=cutoff)
    spec.dh, spec.box = None, (edge, edge, edge)
    sparse, dense = _cube(spec, 1.2, edge), _cube(spec, 0.55, edge)
    b = spec.bonds
    spec.bond_v0 = np.linalg.norm(dense[b[:, 1]] - dense[b[:, 0]], axis=1)
    system = synth.build_system(spec)
    out, interval = [], 0
    for first in (sparse, None):
        ctx = gpu.Context(system, gpu.LangevinIntegrator(0.0, 1.0, 0.002, 7))  # no noise: no step counter either
        if first is not None:
            ctx.setPositions(first)
            ctx.setVelocities(np.zeros((spec.n, 3)))
            ctx.step(10)
            st = ctx.stats()
            assert st["masked_tiles"] == 0
            interval = st["rebuild_interval"]  # the stretched bonds may have halved it
        else:
            ctx.set_list_options(rebuild_interval=interval)
        ctx.setPositions(dense)
        ctx.setVelocities(np.zeros((spec.n, 3)))
        builds = ctx.stats()["list_builds"]
        ctx.step(10)
        st = ctx.stats()
        assert st["rebuild_interval"] == interval
        assert st["list_builds"] > builds + 10 // interval  # more than the chunks' own builds
        assert (st["masked_tiles"] == 0) == lists
        out.append((ctx.getPositions(), ctx.getVelocities()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert not np.array_equal(out[0][0], dense)


def test_tiles_and_masks_grow(gpu):
    """A 20,000-bead slab of excluded volume under a 5 nm cutoff, excluded
    inside its chains: with a quarter to spare, more tiles than 48 and more
    masked ones than 8 per cluster, which is what the buffers start with."""
    from opencafemol_gb300 import synth
    from oracle import oracle
    spec = synth.hps_slab(100, 200, (15.0, 15.0, 150.0), slab_width=30.0, seed=31)
    radius = 0.3 * spec.ljr.p1
    top = np.sort(radius)[-2:]
    spec.exv = synth.PairTerm(ratio=5.0 / (top[0] + top[1]), p0=radius, eps=0.8, ign_molecule=True)
    spec.ljr = spec.lja = spec.dh = None
    ctx = gpu.Context(synth.build_system(spec), gpu.LangevinIntegrator(spec.temperature, 1.0, 0.002, 7))
    ctx.setPositions(spec.pos)
    f1, _ = ctx.getState(energy=False)
    f2, _ = ctx.getState(energy=False)
    assert np.array_equal(f1, f2)
    f_ref, _ = oracle.evaluate(spec, cells=1)
    assert rel_force_err(f1, f_ref) <= FORCE_TOL
    clusters, st = len(ctx.cluster_order()) // 32, ctx.stats()
    assert 1.25 * st["tiles"] > 48 * clusters and 1.25 * st["masked_tiles"] > 8 * clusters


@pytest.mark.parametrize("kind,lists", [("plain", True), ("sigmas", True), ("molecules", True), ("empty", True),
                                        ("narrow", True), ("far", False)])
def test_which_path(gpu, kind, lists):
    """The slabs of the pair-list tests: tiles of bonded chains carry
    exclusion masks, per-bead lists none."""
    from opencafemol_gb300 import synth
    from test_pair_lists_gpu import _slab
    spec = _slab(kind)
    ctx = gpu.Context(synth.build_system(spec), gpu.LangevinIntegrator(spec.temperature, 5.0, 0.002, 7))
    ctx.setPositions(spec.pos)
    ctx.step(3)
    st = ctx.stats()
    assert st["reordered"] == 1 and (st["masked_tiles"] == 0) == lists


@pytest.mark.parametrize("kind", ["go", "hps", "general"])
@pytest.mark.parametrize("n", [200, 600])
def test_straight_lists_do_overflow(gpu, kind, n):
    """Lists sized from a straight chain are too short for the coil, and are
    grown at the next run; lists sized from the coil are not."""
    from opencafemol_gb300 import synth
    from test_batch_classes_gpu import _chain
    spec = _chain(kind, n, 80 + n)
    system = synth.build_system(spec)
    straight = np.zeros((n, 3))
    straight[:, 0] = 0.38 * np.arange(n)
    grown = []
    for start in (straight, spec.pos):
        b = gpu.Batch(max_systems=1, max_total_beads=1024, max_beads_per_system=1024)
        slot = b.admit(system, start, temperature=300.0, seed=9, n_steps=60)
        before = b.slot_stats(slot)["list_capacity"]
        b.set_positions_many([slot], spec.pos)
        b.run(30)
        b.run(30)
        grown.append(b.slot_stats(slot)["list_capacity"] > before)
    assert grown == [True, False]


@pytest.mark.parametrize("kind", ["tiles", "lists"])
def test_overlapping_launches_follow_the_oracle(gpu, kind):
    """Ten steps in one chunk, whose force and integrator kernels overlap on
    grids of this size: a kernel that read its predecessor's data too early
    would be off by a good part of a step.  Forces within 1e-4 keep the
    displacements within 1e-4."""
    from opencafemol_gb300 import synth
    from oracle import oracle
    spec = (synth.go_protein(600, 21) if kind == "tiles"
            else synth.hps_slab(23, 97, (15.0, 15.0, 50.0), slab_width=14.0, seed=5))
    ctx = gpu.Context(synth.build_system(spec), gpu.LangevinIntegrator(spec.temperature, 1.0, 0.005, 12), engine="tiles")
    ctx.setPositions(spec.pos)
    rng = np.random.default_rng(4)
    v = (rng.normal(size=(spec.n, 3)) * np.sqrt(0.00831446261815324 * spec.temperature / spec.masses)[:, None])
    v = v.astype(np.float32).astype(np.float64)
    ctx.setVelocities(v)
    ctx.step(10)
    x, x0 = spec.pos.copy(), spec.pos
    for step in range(10):
        f, _ = oracle.evaluate(spec, pos=x)
        x, v = oracle.langevin_step(x, v, f, spec.masses, spec.temperature, 1.0, 0.005, 12, step)
    moved = np.abs(x - x0).max()
    assert moved > 0.02
    assert np.abs(ctx.getPositions() - x).max() <= 1e-4 * moved
    assert np.abs(ctx.getVelocities() - v).max() <= 1e-4 * np.abs(v).max()


def test_tiles_until_the_options_change(gpu):
    """A context that went to the tiles stays there for new positions, and
    goes back to the lists with its options: the same forces from both."""
    from opencafemol_gb300 import synth
    edge = 56.0
    spec = synth.hps_slab(46, 97, (15.0, 15.0, 60.0), slab_width=30.0, seed=7, hps_cutoff=4.0)
    spec.dh, spec.box = None, (edge, edge, edge)
    ctx = gpu.Context(synth.build_system(spec), gpu.LangevinIntegrator(0.0, 1.0, 0.002, 7))
    sparse = _cube(spec, 1.2, edge)
    forces = []
    for positions, options, lists in ((sparse, False, True), (_cube(spec, 0.55, edge), False, False),
                                      (sparse, False, False), (sparse, True, True)):
        if options:
            ctx.set_list_options(skin=ctx.stats()["skin"])
        ctx.setPositions(positions)
        forces.append(ctx.getState(energy=False)[0])
        assert (ctx.stats()["masked_tiles"] == 0) == lists
    assert np.array_equal(forces[0], forces[3])
    assert rel_force_err(forces[2], forces[0]) <= FORCE_TOL
