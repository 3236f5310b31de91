"""Groups evaluated one at a time on overlapping beads: a repulsion that is
switched off must not reach the other groups through its overflow."""
import dataclasses

import numpy as np
import pytest

from conftest import rel_force_err

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-4   # FP32 pair arithmetic, the bar of the parity tests
ENERGY_TOL = 1e-5


def _overlap(spec, distance):
    """The last bead moved to `distance` from bead 10: (sigma / r)^12 is
    beyond single precision."""
    spec.pos = spec.pos.copy()
    spec.pos[-1] = spec.pos[10] + np.array([distance, 0.0, 0.0])
    spec.pos = spec.pos.astype(np.float32).astype(np.float64)
    return spec


def _without_repulsion(spec):
    return dataclasses.replace(spec, ljr=None)


def _group(system, name):
    return 1 << system.group_names().index(name)


@pytest.mark.parametrize("distance", [1e-4, 0.0])
def test_batched(gpu, distance):
    from opencafemol_gb300 import synth
    from oracle import oracle
    spec = synth.go_protein(150, 31)
    spec.exv, n = None, spec.n
    spec.ljr = synth.PairTerm(ratio=5.0, p0=np.full(n, 0.8), p1=np.full(n, 0.4), ign_bond=3)
    spec.lja = synth.PairTerm(ratio=5.0, p0=np.full(n, 0.5), p1=np.full(n, 0.4), ign_bond=3)
    spec.dh.p0 = np.where(np.isin(np.arange(n), (10, n - 1)), np.nan, spec.dh.p0)  # the two carry no charge
    spec = _overlap(spec, distance)
    system = synth.build_system(spec)
    b = gpu.Batch(max_systems=1, max_total_beads=256, max_beads_per_system=256)
    slot = b.admit(system, spec.pos, seed=1, n_steps=1)
    with pytest.raises(gpu.OCMError):  # with the repulsion the force is out of range
        b.state(slot)
    rest = sum(1 << g for g, name in enumerate(system.group_names()) if name != "LennardJonesRepulsive")
    f, e = b.state(slot, groups=rest)
    if distance == 0.0:  # no direction, and no reference: the oracle divides by r
        assert np.all(np.isfinite(f)) and np.all(np.isfinite(e))
    else:
        f_ref, e_ref = oracle.evaluate(_without_repulsion(spec))
        assert rel_force_err(f, f_ref) <= FORCE_TOL
        for g, name in enumerate(system.group_names()):
            if name != "LennardJonesRepulsive":
                assert abs(e[g] - e_ref[name]) <= ENERGY_TOL * max(1.0, abs(e_ref[name])), name
    assert np.all(np.isfinite(b.state(slot, groups=_group(system, "LennardJonesAttractive"))[0]))


@pytest.mark.parametrize("sigmas", ["same", "two"])
def test_pair_lists(gpu, sigmas):
    from opencafemol_gb300 import synth
    from oracle import oracle
    spec = synth.hps_slab(23, 97, (15.0, 15.0, 50.0), slab_width=14.0, seed=5)
    if sigmas == "two":
        spec.lja.p1 = spec.lja.p1 * np.random.default_rng(1).uniform(0.9, 1.1, spec.n)
    spec.dh.p0 = np.where(np.isin(np.arange(spec.n), (10, spec.n - 1)), np.nan, spec.dh.p0)
    spec = _overlap(spec, 1e-4)
    system = synth.build_system(spec)
    ctx = gpu.Context(system, gpu.LangevinIntegrator(spec.temperature, 5.0, 0.002, 7))
    ctx.setPositions(spec.pos)
    rest = sum(1 << g for g, name in enumerate(system.group_names()) if name != "LennardJonesRepulsive")
    f_ref, e_ref = oracle.evaluate(_without_repulsion(spec))
    for energy in (False, True):
        f, e = ctx.getState(energy=energy, groups=rest)
        assert rel_force_err(f, f_ref) <= FORCE_TOL
    ref = sum(v for k, v in e_ref.items() if k != "LennardJonesRepulsive")
    assert abs(e - ref) <= ENERGY_TOL * max(1.0, sum(abs(v) for v in e_ref.values()))
    assert ctx.stats()["masked_tiles"] == 0  # the per-bead lists
