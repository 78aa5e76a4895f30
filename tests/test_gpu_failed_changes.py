"""GPU tests of a change of parameters or tuning that runs out of memory
part-way (host-side fault injection): the same call, repeated with the same
values, carries it out, and the handle steps as a new one would."""
import numpy as np
import pytest
import torch

import pbf_gb300 as pg
from pbf_gb300 import _capi, scenes

pytestmark = pytest.mark.gpu

OUT_OF_MEMORY = 2


class no_memory:
    """The next device allocation of the library fails."""

    def __init__(self, lib, after=0):
        self.lib, self.after = lib, after

    def __enter__(self):
        self.lib.pbf_debug_fail_allocation(self.after)

    def __exit__(self, *exc):
        self.lib.pbf_debug_fail_allocation(-1)


def scene():
    x4, v4 = scenes.block((10, 9, 8), origin=(3.0, 3.0, 3.0), seed=8, vel_uniform=0.5)
    return x4, v4, scenes.dam_params((20, 20, 20), 2, epsilon=5.0)


def stepped(sim, x4, v4):
    sim.set_state(x4, v4)
    sim.step(3)
    return [a.view(np.uint32) for a in sim.get_state()]


def test_iteration_count_raised_again_after_out_of_memory(gpu):
    x4, v4, p = scene()
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    p.num_solver_iterations = 7
    fresh = stepped(pg.SPH(x4.shape[0], tuple(p.grid), p), x4, v4)
    with no_memory(gpu):
        with pytest.raises(pg.PbfError) as e:
            sim.set_params(p)
    assert e.value.status == OUT_OF_MEMORY
    sim.set_params(p)
    for a, b in zip(stepped(sim, x4, v4), fresh):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("scene_count", [1, 2])
@pytest.mark.parametrize("after", [0, 1])
def test_parameters_set_after_a_failed_tuning(gpu, scene_count, after):
    x4, v4, p = scene()
    x4, v4 = (np.concatenate([a] * scene_count) for a in (x4, v4))
    count = x4.shape[0] // scene_count
    make = (lambda: pg.SPH(count, tuple(p.grid), p)) if scene_count == 1 else (
        lambda: pg.SPHBatch([p] * scene_count, [count] * scene_count))
    tuning = dict(use_neighbour_lists=True, list_capacity=200, sweep_mode="direct")
    fresh = make()
    fresh.set_tuning(**tuning)
    want = stepped(fresh, x4, v4)
    sim = make()
    with no_memory(gpu, after):
        with pytest.raises(pg.PbfError) as e:
            sim.set_tuning(**tuning)
    assert e.value.status == OUT_OF_MEMORY
    if scene_count == 1:
        sim.set_params(p)
    else:
        sim.set_scene_params(1, p)
    for a, b in zip(stepped(sim, x4, v4), want):
        assert np.array_equal(a, b)


def test_a_real_out_of_memory_is_reported_once(gpu):
    # entries of 4,096 candidates for this many particles do not fit on any GPU
    x4, v4, p = scene()
    sim = pg.SPH(x4.shape[0], tuple(p.grid), p)
    want = stepped(sim, x4, v4)
    many = pg.SPH(20_000_000, tuple(p.grid), p)
    many.set_tuning(pair_list_capacity=0)

    def run_out():
        with pytest.raises(pg.PbfError) as e:
            many.set_tuning(pair_list_capacity=4096)
        assert e.value.status == OUT_OF_MEMORY

    run_out()
    new = pg.SPH(x4.shape[0], tuple(p.grid), p)
    for a, b in zip(stepped(new, x4, v4), want):  # captures its graph
        assert np.array_equal(a, b)
    run_out()
    keys = torch.tensor([0, 0, 2, 5], dtype=torch.int32, device="cuda")
    start, end = (torch.empty(6, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    _capi.check(gpu.pbf_find_cells(keys.data_ptr(), 4, 6, start.data_ptr(), end.data_ptr(), None))
    assert start.tolist() == [0, -1, 2, -1, -1, 3] and end.tolist() == [2, -1, 3, -1, -1, 4]
    many.close()
