"""GPU tests of the sweeps that share a particle among four or eight lanes:
particle counts on both sides of the lines between the lane counts and between
them and the other sweeps, lists too short for some or all particles, particles
with more candidates than a group takes, scenes with few candidates.  The direct
sweeps, which the oracle tests compare with, give the bits."""
import numpy as np
import pytest

import pbf_gb300 as pg
from pbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def run(p, x4, v4, substeps, **tuning):
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    sim.set_tuning(**tuning)
    sim.set_state(x4, v4)
    sim.step(substeps)
    x, v = sim.get_state()
    return x.view(np.uint32), v.view(np.uint32)


@pytest.mark.parametrize("lattice", [(1, 1, 1), (5, 3, 2), (29, 29, 29), (30, 29, 29),
                                     (37, 36, 36), (37, 37, 36), (51, 50, 51), (51, 51, 51)])
@pytest.mark.parametrize("cap", [128, 20, 1])
def test_quads_give_the_direct_bits(gpu, lattice, cap):
    x4, v4 = scenes.block(lattice, seed=2, vel_uniform=2.0)
    box = [max(8, l // 2 + 5) for l in lattice]
    p = scenes.dam_params(box, 3, epsilon=0.01)
    want = run(p, x4, v4, 5, sweep_mode="direct", pair_list_capacity=0)
    for tuning in (dict(sweep_mode="coop"), dict(sweep_mode="auto"),
                   dict(sweep_mode="auto", coop_candidates=100)):
        got = run(p, x4, v4, 5, pair_list_capacity=cap, **tuning)
        for a, b in zip(got, want):
            assert np.array_equal(a, b), tuning


@pytest.mark.parametrize("substeps", [12, 40])
def test_quads_with_piles_and_sparse_rows(gpu, substeps):
    # collapsing: most particles end with thousands of candidates, a few with none
    x4, v4 = scenes.block((16, 12, 14), seed=5, vel_uniform=1.0)
    p = scenes.dam_params((20, 20, 20), 3, epsilon=0.01)
    want = run(p, x4, v4, substeps, sweep_mode="direct")
    got = run(p, x4, v4, substeps, sweep_mode="coop")
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
