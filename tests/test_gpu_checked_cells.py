"""GPU test of the bounds-checked build's cell passes that run without a
permutation (the standalone cell finder) or without a status word (the
diagnostics): the results of the normal build."""
import numpy as np
import pytest
import torch

import pbf_gb300 as pg
from pbf_gb300 import _capi, build, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def checked(gpu):
    build.build(check=True)
    return _capi.load_checked()


@pytest.mark.parametrize("n", [1, 31, 257, 5000])
def test_standalone_cells(checked, gpu, n):
    cells = 300
    keys = torch.from_numpy(np.sort(np.random.default_rng(n).integers(0, cells, n)).astype(np.int32)).cuda()
    out = []
    for lib in (gpu, checked):
        start, end = (torch.zeros(cells, dtype=torch.int32, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        assert lib.pbf_find_cells(keys.data_ptr(), n, cells, start.data_ptr(), end.data_ptr(),
                                  None) == 0
        out.append((start.cpu().numpy(), end.cpu().numpy()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_diagnostics(checked):
    x4, v4 = scenes.block((9, 8, 7), seed=2, vel_uniform=0.5)
    p = scenes.dam_params((16, 16, 16), 2)
    out = []
    for lib in (None, checked):
        sim = pg.SPH(x4.shape[0], tuple(p.grid), p, lib=lib)
        sim.set_state(x4, v4)
        out.append(sim.diagnostics())
        assert not (sim.device_status() & _capi.PBF_DEV_INDEX)
    assert out[0] == out[1]
