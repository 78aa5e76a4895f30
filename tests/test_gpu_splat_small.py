"""GPU tests of the depth pass where sprites are filled by a share of a warp's
lanes: boxes of one pixel up to the largest that a share fills and beyond, counts
and images on both sides of the lines where the share changes, sprites of very
different sizes in one warp."""
import math

import numpy as np
import pytest

from pbf_gb300 import splat

pytestmark = pytest.mark.gpu


def view(eye, w, h):
    return splat.View.of(splat.look_at(eye, (0.0, 3.0, 0.0), (0.0, 1.0, 0.0)),
                         splat.perspective(math.radians(45.0), w / h, 1.0, 200.0))


def cloud(n, seed=0):
    rng = np.random.default_rng(seed)
    x4 = np.zeros((n, 4), np.float32)
    x4[:, :3] = rng.uniform((44, 0, 44), (84, 30, 84), (n, 3))
    return x4


def same_as_oracle(oracle_mod, x4, v, w, h):
    want = oracle_mod.splat(splat.DEPTH, x4, *v.columns(), w, h)
    got = splat.splat(splat.DEPTH, x4, v, w, h).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
    return want


@pytest.mark.parametrize("n", [16383, 16384, 16391])
@pytest.mark.parametrize("w,h", [(64, 48), (320, 240)])
def test_many_sprites_on_a_small_image(gpu, oracle_mod, n, w, h):
    want = same_as_oracle(oracle_mod, cloud(n), view((14.0, 10.0, 12.0), w, h), w, h)
    assert (want < 1.0).any()


@pytest.mark.parametrize("w,h", [(707, 707), (1000, 500), (833, 601)])
def test_both_sides_of_the_small_image(gpu, oracle_mod, w, h):
    same_as_oracle(oracle_mod, cloud(16384, 3), view((14.0, 10.0, 12.0), w, h), w, h)


@pytest.mark.parametrize("distance", [0.5, 1.2, 3.0, 8.0, 40.0, 150.0])
@pytest.mark.parametrize("n", [5, 64])
def test_box_sizes(gpu, oracle_mod, n, distance):
    # sprites 500 pixels across at the nearest, below one at the farthest
    v = view((distance, 3.0, 0.0), 320, 200)
    x4 = np.zeros((n, 4), np.float32)
    x4[:, :3] = (64.0, 14.0, 64.0) + np.random.default_rng(n).uniform(-1.5, 1.5, (n, 3))
    same_as_oracle(oracle_mod, x4, v, 320, 200)
    x4[::3] = cloud(n, 1)[::3]  # mixed sizes
    same_as_oracle(oracle_mod, x4, v, 320, 200)
