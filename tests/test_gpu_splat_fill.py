"""GPU tests of how the splat passes fill sprites: groups of sprites taken in
any order (counts around the group sizes and the count where the group size
changes, a number of groups that the stepping prime divides), sprites filled by
a thread or by the warp, cut by every image edge, on images narrower than a
warp's step."""
import math

import numpy as np
import pytest

from pbf_gb300 import splat

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def view(eye, w, h):
    return splat.View.of(splat.look_at(eye, (0.0, 3.0, 0.0), (0.0, 1.0, 0.0)),
                         splat.perspective(math.radians(45.0), w / h, 1.0, 200.0))


def cloud(n, seed=0):
    rng = np.random.default_rng(seed)
    x4 = np.zeros((n, 4), np.float32)
    x4[:, :3] = rng.uniform((44, 0, 44), (84, 30, 84), (n, 3))
    return x4


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 127, 129, 2000])
@pytest.mark.parametrize("w,h", [(96, 64), (7, 5), (129, 131)])
def test_matches_oracle(gpu, oracle_mod, n, w, h):
    # the eye inside the cloud: sprites from less than a pixel to hundreds
    # across, some behind it, some cut by the near plane and the image's edges
    for eye in ((9.0, 6.0, 7.0), (1.0, 3.5, 1.2)):
        v = view(eye, w, h)
        x4 = cloud(n, n)
        for p in (splat.DEPTH, splat.THICKNESS):
            want = oracle_mod.splat(p, x4, *v.columns(), w, h)
            got = splat.splat(p, x4, v, w, h).cpu().numpy()
            assert np.array_equal(bits(got), bits(want)), (p, eye)


@pytest.mark.parametrize("n", [4 * 7919, 262143, 262144 + 5, 8 * 7919 * 5])
def test_any_order_gives_the_same_image(gpu, n):
    v = view((12.0, 9.0, 10.0), 640, 360)
    x4 = cloud(n)
    x4 = x4[np.argsort(x4[:, 0] + x4[:, 2])]  # one end nearer to the eye
    want = [bits(splat.splat(p, x4, v, 640, 360).cpu().numpy()) for p in (0, 1)]
    assert (want[0] != bits(np.float32(1.0))).any()
    for order in (slice(None, None, -1), np.random.default_rng(1).permutation(n)):
        for p in (0, 1):
            got = splat.splat(p, np.ascontiguousarray(x4[order]), v, 640, 360).cpu().numpy()
            assert np.array_equal(bits(got), want[p]), p
