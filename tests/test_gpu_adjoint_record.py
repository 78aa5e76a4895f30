"""GPU tests of what a recorded run keeps: the forward sweeps' pair lists that
the reverse sweeps replay (whole, too short for some or all particles, or
none), the last segment recorded by the forward run, and the buffers that the
next run reuses.

The reverse sweeps add the same terms in the same order whichever way they
find their pairs; only a pair within rounding of the radius h can be in one
set and not in the other, and its terms go to zero there like (h - r) / h,
a few 1e-7 of the others.  Hence 1e-5 of the largest gradient."""
import numpy as np
import pytest

import pbf_gb300 as pg
from pbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def scene(n, floor):
    # floor: the lattice starts below the wall and moves down, so that some
    # particles are predicted outside the grid (one-way candidates)
    x4, v4 = scenes.block(n, origin=(4.0, 0.25 if floor else 4.0, 4.0), seed=3, vel_uniform=0.5)
    if floor:
        v4[:, 1] -= 160.0 * (np.arange(x4.shape[0]) % 5 == 0)
    p = scenes.dam_params((32, 32, 32), 3, epsilon=5.0)
    return p, x4, v4


def grads(sim, x4, v4, substeps, every, again=False):
    rng = np.random.default_rng(9)
    w = rng.standard_normal((x4.shape[0], 4)).astype(np.float32)
    u = rng.standard_normal((x4.shape[0], 4)).astype(np.float32)
    sim.set_state(x4, v4)
    sim.forward_record(substeps, every)
    if again:  # the second reverse pass finds another segment in the slots
        sim.backward(w, u)
    state = sim.get_state()
    return [np.asarray(a, np.float64) for a in (*sim.backward(w, u), *state)]


def close(got, want):
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-30)


@pytest.mark.parametrize("floor", [False, True])
@pytest.mark.parametrize("mode", ["masked", "coop", "auto"])
@pytest.mark.parametrize("cap", [128, 30, 1])
def test_lists_and_scans_agree(gpu, floor, mode, cap):
    p, x4, v4 = scene((13, 12, 11), floor)
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    sim.set_tuning(sweep_mode="masked", pair_list_capacity=0)  # every sweep scans
    want = grads(sim, x4, v4, 5, 2)
    sim.set_tuning(sweep_mode=mode, pair_list_capacity=cap)
    close(grads(sim, x4, v4, 5, 2), want)


@pytest.mark.parametrize("substeps,every", [(1, 1), (5, 2), (4, 4), (3, 8)])
def test_recorded_again(gpu, substeps, every):
    p, x4, v4 = scene((9, 10, 7), False)
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    sim.set_tuning(sweep_mode="masked")
    first = grads(sim, x4, v4, substeps, every)
    for got in (grads(sim, x4, v4, substeps, every, again=True),
                grads(sim, x4, v4, substeps, every)):
        for a, b in zip(got, first):
            assert np.array_equal(a, b)
    other = grads(sim, x4, v4, substeps + 1, every)  # another shape in between
    assert not np.array_equal(other[0], first[0])
    assert np.array_equal(grads(sim, x4, v4, substeps, every)[0], first[0])


def test_parameters_end_a_recorded_run(gpu):
    p, x4, v4 = scene((6, 6, 6), False)
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    grads(sim, x4, v4, 2, 1)
    sim.set_params(p)  # equal ones too
    with pytest.raises(Exception):
        sim.backward(np.zeros_like(x4), np.zeros_like(x4))
    sim.forward_record(2, 1)
    sim.release_record()
    with pytest.raises(Exception):
        sim.backward(np.zeros_like(x4), np.zeros_like(x4))
