"""GPU tests of what the handle shows after a recorded run: the debug reads of
the last substep, the automatic mode's trials and the launch count are those of
the same substeps run by pbf_step."""
import numpy as np
import pytest

import pbf_gb300 as pg
from pbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def make(iterations=3, vorticity=True, **tuning):
    x4, v4 = scenes.block((11, 9, 10), origin=(4.0, 4.0, 4.0), seed=6, vel_uniform=0.5)
    p = scenes.dam_params((32, 32, 32), iterations, epsilon=5.0, vorticity=vorticity)
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    if tuning:
        sim.set_tuning(**tuning)
    sim.set_state(x4, v4)
    return sim


def reads(sim):
    return [*sim.get_solver(), *sim.get_sort(), *sim.get_cells(), *sim.get_state()]


@pytest.mark.parametrize("substeps,every", [(1, 1), (4, 4), (3, 8), (5, 2), (6, 2)])
@pytest.mark.parametrize("iterations,vorticity", [(3, True), (1, False), (0, True)])
def test_reads_of_the_last_substep(gpu, substeps, every, iterations, vorticity):
    stepped, recorded = make(iterations, vorticity), make(iterations, vorticity)
    stepped.step(substeps)
    recorded.forward_record(substeps, every)
    want, got = reads(stepped), reads(recorded)
    if iterations == 0:  # no sweep writes a lambda
        want, got = want[1:], got[1:]
    for a, b in zip(got, want):
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint32),
                              np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("substeps,every", [(8, 8), (8, 3), (8, 6), (7, 4)])
def test_trials_go_on_in_the_recorded_segment(gpu, substeps, every):
    # the first trial starts at substep 4 and takes three substeps; the next
    # starts at substep 9 at the earliest
    stepped, recorded = make(auto_period=4), make(auto_period=4)
    stepped.step(substeps)
    recorded.forward_record(substeps, every)
    assert stepped.sweep_choice()["trials"] == 1
    assert recorded.sweep_choice()["trials"] == 1
    for a, b in zip(recorded.get_state(), stepped.get_state()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    rng = np.random.default_rng(2)
    w = rng.standard_normal((990, 4)).astype(np.float32)
    plain = make(sweep_mode="masked")
    plain.forward_record(substeps, every)
    for a, b in zip(recorded.backward(w, w), plain.backward(w, w)):
        # (recorded lists and scans agree to rounding: test_gpu_adjoint_record.py)
        a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
