"""GPU tests of the splat passes on small and wide images, and of the depth pass
where sprites are filled by a share of a warp's lanes: boxes of one pixel up to
the largest that a share fills and beyond, counts and images on both sides of the
lines where the share changes, sprites of very different sizes in one warp."""
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


@pytest.mark.parametrize("n", [1, 700, 1023, 1024, 1500])
@pytest.mark.parametrize("w,h", [(447, 447), (448, 447), (1023, 197), (1024, 196), (1025, 196),
                                 (2050, 101), (5, 16384), (13, 16001)])
def test_thickness_added_or_summed_along_rows(gpu, oracle_mod, n, w, h):
    # (below 1,024 sprites, or 200,000 pixels, they are added pixel by pixel); rows of one step and
    # of several, of less than a thread's four pixels
    x4 = cloud(n, 2)
    for eye in ((9.0, 6.0, 7.0), (1.0, 3.5, 1.2)):
        v = view(eye, w, h)
        want = oracle_mod.splat(splat.THICKNESS, x4, *v.columns(), w, h)
        got = splat.splat(splat.THICKNESS, x4, v, w, h).cpu().numpy()
        assert np.array_equal(got, want), eye


@pytest.mark.parametrize("n", [131071, 131072])
def test_thickness_of_many_on_a_small_image(gpu, oracle_mod, n):
    x4, v = cloud(n, 4), view((14.0, 10.0, 12.0), 300, 220)
    want = oracle_mod.splat(splat.THICKNESS, x4, *v.columns(), 300, 220)
    assert np.array_equal(splat.splat(splat.THICKNESS, x4, v, 300, 220).cpu().numpy(), want)
