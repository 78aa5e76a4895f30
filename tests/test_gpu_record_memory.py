"""GPU tests of the memory that recorded runs keep: an allocation of the library
that finds none takes the buffers of every handle's dropped recording, and of no
other; the handles record again as before."""
import threading

import numpy as np
import pytest
import torch

import pbf_gb300 as pg
from pbf_gb300 import scenes

pytestmark = pytest.mark.gpu

EVERY = 4
# entries of 4,096 candidates for this many particles do not fit on any GPU
MANY = 20_000_000


def recorder(seed=3):
    x4, v4 = scenes.block((32, 32, 32), origin=(4.0, 4.0, 4.0), seed=seed, vel_uniform=0.5)
    p = scenes.dam_params((40, 40, 40), 3, epsilon=5.0)
    return pg.SPH(x4.shape[0], tuple(p.grid), p), x4, v4


def gradients(sim, x4, v4):
    sim.set_state(x4, v4)
    sim.forward_record(EVERY, EVERY)
    return sim.backward(x4, v4)


def tape_bytes(n, iterations, cap=128):
    lists = (iterations + 1) * (cap + 1) * 4
    return n * (EVERY * (156 + 32 * iterations + lists) + 32 + 290)


@pytest.fixture(scope="module")
def greedy(gpu):
    p = scenes.dam_params((40, 40, 40), 2)
    sim = pg.SPH(MANY, tuple(p.grid), p)
    sim.set_tuning(pair_list_capacity=0)
    yield sim
    sim.close()


def ask_for_too_much(sim):
    with pytest.raises(pg.PbfError) as e:
        sim.set_tuning(pair_list_capacity=4096)
    status = e.value.status
    sim.set_tuning(pair_list_capacity=0)
    assert status == 2


def test_dropped_recordings_give_their_memory_back(gpu, greedy):
    sim, x4, v4 = recorder()
    want = gradients(sim, x4, v4)
    sim.set_params(sim.params)  # drops the recording
    before = torch.cuda.mem_get_info()[0]
    ask_for_too_much(greedy)
    freed = torch.cuda.mem_get_info()[0] - before
    assert freed >= tape_bytes(x4.shape[0], 3)
    for a, b in zip(gradients(sim, x4, v4), want):
        assert np.array_equal(a, b)


def test_a_recording_is_kept(gpu, greedy):
    sim, x4, v4 = recorder()
    want = gradients(sim, x4, v4)
    sim.set_state(x4, v4)
    sim.forward_record(EVERY, EVERY)
    ask_for_too_much(greedy)
    for a, b in zip(sim.backward(x4, v4), want):
        assert np.array_equal(a, b)


def test_handles_in_other_threads(gpu, greedy):
    want, got, errors = [], [], []

    def train(k):
        try:
            sim, x4, v4 = recorder(seed=k)
            for _ in range(6):
                got.append((k, gradients(sim, x4, v4)))
                sim.set_params(sim.params)
        except Exception as e:  # pragma: no cover
            errors.append(e)

    for k in range(2):
        want.append(gradients(*recorder(seed=k)))
    threads = [threading.Thread(target=train, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    while any(t.is_alive() for t in threads):
        ask_for_too_much(greedy)
    for t in threads:
        t.join()
    assert not errors
    assert len(got) == 12
    for k, g in got:
        for a, b in zip(g, want[k]):
            assert np.array_equal(a, b)
