"""List options changed on a live context: a wider skin can leave too few
cells for the charged rows, and Debye-Hueckel then belongs to the tiles."""
import numpy as np
import pytest

from conftest import rel_force_err

pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-4   # FP32 pair arithmetic, the bar of the parity tests
ENERGY_TOL = 1e-5


def _check(ctx, system, spec):
    from oracle import oracle
    L = np.asarray(spec.box)
    x = ctx.getPositions()
    x = (x - L * np.floor(x / L)).astype(np.float32).astype(np.float64)
    x = np.where(x >= L, x - L, x)  # FP32-exact for both sides
    ctx.setPositions(x)
    f, _ = ctx.getState(energy=False)
    f_ref, e_ref = oracle.evaluate(spec, pos=x)
    assert rel_force_err(f, f_ref) <= FORCE_TOL
    e = ctx.getGroupEnergies()
    for g, name in enumerate(system.group_names()):
        assert abs(e[g] - e_ref[name]) <= ENERGY_TOL * max(1.0, abs(e_ref[name])), name


@pytest.mark.parametrize("box,dh_cutoff", [((9.0, 9.0, 90.0), 2.6), ((12.0, 15.0, 50.0), 3.5)])
def test_debye_hueckel_survives_a_wider_skin(gpu, box, dh_cutoff):
    from opencafemol_gb300 import synth
    spec = synth.hps_slab(23, 97, box, slab_width=0.5 * box[2], seed=6, dh_cutoff=dh_cutoff)
    assert spec.n > 2048
    system = synth.build_system(spec)
    ctx = gpu.Context(system, gpu.LangevinIntegrator(spec.temperature, 5.0, 0.002, 7))
    ctx.setPositions(spec.pos)
    ctx.setVelocitiesToTemperature(spec.temperature, 3)
    for skin, split in ((0.25, 1), (0.6, 0), (0.3, 0)):  # the split does not come back
        ctx.set_list_options(skin=skin)
        _check(ctx, system, spec)
        ctx.step(20)
        _check(ctx, system, spec)
        st = ctx.stats()
        assert st["charged_split"] == split
        # per-bead lists carry no masks; tiles of bonded chains always do
        assert (st["masked_tiles"] == 0) == bool(split)
