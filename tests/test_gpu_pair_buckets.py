"""Long pair buckets: a platform that overlaps every box, the boxes in the
order of their x (the order the sweep finds them in), against it and at
random.  Pairs exact at the edges of the bucket sort (one thread's eight keys,
a warp's 32, the merged runs), and the pair stage's time in the number of
boxes, not its square."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0


def over_platform(scenes, n, order):
    side = int(np.ceil(np.sqrt(n)))
    at = np.zeros((n + 1, 3), np.float32)
    at[0, 1] = 1.0
    k = np.arange(n)
    at[1:] = np.stack([(k // side - side / 2) * 0.5, np.full(n, 1.199), (k % side - side / 2) * 0.5], 1)
    if order == "reversed":
        at[1:] = at[:0:-1]
    elif order == "random":
        at[1:] = at[1:][np.random.default_rng(n).permutation(n)]
    quat = np.tile(np.array([0, 0, 0, 1], np.float32), (n + 1, 1))
    mats = np.tile(np.array([0.5, 0.5, 0.0], np.float32), (n + 1, 1))
    shapes = [[scenes._box((0.25 * side + 1, 0.1, 0.25 * side + 1))]] + [[scenes._box((0.1, 0.1, 0.1))] for _ in range(n)]
    return scenes._assemble(at, quat, 0 * at, 0 * at, 1000.0, shapes, mats)


@pytest.mark.parametrize("order", ["ascending", "reversed", "random"])
@pytest.mark.parametrize("n", [7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 129, 257, 2500])
def test_bucket_of_exactly_n_partners(pkg, scenes, n, order):
    w = pkg.World(0)
    w.add_scene(over_platform(scenes, n, order))
    w.collide()
    boxes = np.arange(2, n + 2)                     # shape 0 is the floor, 1 the platform
    want = np.concatenate([np.stack([np.zeros(n + 1), np.arange(1, n + 2)], 1), np.stack([np.ones(n), boxes], 1)])
    np.testing.assert_array_equal(w.pairs(0), want.astype(np.uint32))


def test_time_grows_with_the_bucket(pkg, scenes):
    ms = {}
    for n in (4000, 16000):
        w = pkg.World(0)
        w.set_sleeping(False)
        w.set_body_kinematic(w.add_scene(over_platform(scenes, n, "random")), True)
        w.step(DT, 3)
        ms[n] = min(w.profile_step(DT)["pairs"] for _ in range(3))
    # a quadratic sort made this 10, the sweep alone about 3
    assert ms[16000] < 6 * ms[4000]
