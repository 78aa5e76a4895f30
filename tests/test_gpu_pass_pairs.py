"""GPU tests of every pair of solver and vorticity configurations, as the
automatic mode may choose them: each gives the direct sweeps' bits, on both sides
of the particle counts where the sweeps change form, for one scene and for a
batch, stepped and recorded.  What the passes hand to each other (the scan copy
of the last iterate, the lists, the listed particles) differs from pair to pair."""
import numpy as np
import pytest

import pbf_gb300 as pg
from pbf_gb300 import _capi, scenes

pytestmark = pytest.mark.gpu

PASSES = range(5)  # PBF_PASS_MASKED .. PBF_PASS_MIXED


def single(lattice):
    x4, v4 = scenes.block(lattice, seed=4, vel_uniform=2.0)
    p = scenes.dam_params([max(8, l // 2 + 5) for l in lattice], 3, epsilon=0.01)
    return (lambda: pg.SPH(x4.shape[0], tuple(p.grid), p)), x4, v4


def batch(lattices):
    parts = [single(l) for l in lattices]
    sims = [make() for make, _, _ in parts]
    params, counts = [s.params for s in sims], [s.numparticles for s in sims]
    for s in sims:
        s.close()
    return ((lambda: pg.SPHBatch(params, counts)), np.concatenate([p[1] for p in parts]),
            np.concatenate([p[2] for p in parts]))


# below 24,576 particles (eight lanes), 49,152 (four), 131,072 (four, replays only), above
CASES = {"13k": ((24, 23, 24),), "33k": ((32, 33, 31),), "61k": ((40, 39, 39),),
         "135k": ((52, 51, 51),), "batch_20k": ((16, 15, 17), (25, 24, 25)),
         "batch_60k": ((16, 15, 17), (30, 29, 33), (27, 36, 28)),
         "batch_150k": ((30, 29, 33), (50, 47, 52))}


def bits(sim):
    return [a.view(np.uint32) for a in sim.get_state()]


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("tuning", [dict(), dict(pair_list_capacity=25), dict(pair_list_capacity=0),
                                    dict(coop_candidates=100)])
def test_pairs_give_the_direct_bits(gpu, name, tuning):
    shapes = CASES[name]
    make, x4, v4 = single(shapes[0]) if len(shapes) == 1 else batch(shapes)
    direct = make()
    direct.set_tuning(sweep_mode="direct", pair_list_capacity=0)
    direct.set_state(x4, v4)
    direct.step(4)
    want = bits(direct)
    sim = make()
    sim.set_tuning(**tuning)
    for solver in PASSES:
        for vort in PASSES:
            sim.set_state(x4, v4)
            _capi.check(gpu.pbf_debug_set_passes(sim.handle, solver, vort), sim.handle)
            sim.step(4)
            for a, b in zip(bits(sim), want):
                assert np.array_equal(a, b), (solver, vort)


@pytest.mark.parametrize("name", ["13k", "33k", "61k", "batch_20k", "batch_60k"])
def test_recorded_pairs_give_the_direct_bits(gpu, name):
    # (gradients: within rounding of the pairs at the radius, test_gpu_adjoint_record.py)
    shapes = CASES[name]
    make, x4, v4 = single(shapes[0]) if len(shapes) == 1 else batch(shapes)
    w = np.random.default_rng(1).standard_normal(x4.shape).astype(np.float32)
    sim = make()
    first = None
    for solver in PASSES:
        for vort in PASSES:
            sim.set_state(x4, v4)
            _capi.check(gpu.pbf_debug_set_passes(sim.handle, solver, vort), sim.handle)
            sim.forward_record(3, 2)
            got = bits(sim)
            grads = [np.asarray(g, np.float64) for g in sim.backward(w, w)]
            if first is None:
                direct = make()
                direct.set_tuning(sweep_mode="direct", pair_list_capacity=0)
                direct.set_state(x4, v4)
                direct.step(3)
                first = bits(direct), grads
            for a, b in zip(got, first[0]):
                assert np.array_equal(a, b), (solver, vort)
            for a, b in zip(grads, first[1]):
                assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max(), (solver, vort)


def test_bad_pass_is_refused(gpu):
    sim = single((4, 4, 4))[0]()
    with pytest.raises(pg.PbfError):
        _capi.check(gpu.pbf_debug_set_passes(sim.handle, 5, 0), sim.handle)
