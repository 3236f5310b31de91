"""Launches with at least four systems per CTA run their smallest systems on
quarters of a CTA: the trajectories are those of whole CTAs, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [256, 512, 1024])
def test_quarters_keep_results(gpu, threads):
    from opencafemol_gb300 import synth
    sizes = [20, 33, 64, 95, 96, 97, 128, 300]  # around a cluster and the quarter's limit
    specs = [synth.go_protein(n, 500 + n) for n in sizes]
    systems = [synth.build_system(s) for s in specs]
    count = 760  # more than four per SM, and not a multiple of it
    runs = []
    for split in (0, 512):
        b = gpu.Batch(max_systems=count, max_total_beads=count * 110, max_beads_per_system=320)
        b.set_threads(threads)
        b.set_split(split)
        slots = [b.admit(systems[k % 8], specs[k % 8].pos, seed=k, n_steps=25 if k % 3 else 40) for k in range(count)]
        b.run(25)
        b.run(25)
        assert all(b.steps_done(s) == (25 if k % 3 else 40) for k, s in enumerate(slots))
        runs.append(b.get_positions_many(slots))
    assert np.array_equal(runs[0], runs[1])
