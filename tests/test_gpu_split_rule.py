"""The narrowphase's split follows the live pairs the budget was made for: a
fitted budget above the line takes the two kernels although it is smaller
than a default budget below it, and the step stays bit-identical."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0


def test_fitted_budget_above_the_line(pkg, scenes):
    rng = np.random.default_rng(3)
    clusters, per = 104, 80                          # 104 x 3,160 overlapping pairs of boxes
    centre = np.repeat(np.stack([np.arange(clusters) * 4.0, np.full(clusters, 40.0), np.zeros(clusters)], 1), per, 0)
    at = (centre + rng.uniform(-0.1, 0.1, centre.shape)).astype(np.float32)
    n = len(at)
    mats = np.tile(np.array([0.5, 0.5, 0.0], np.float32), (n, 1))
    spec = scenes._assemble(at, scenes.random_quaternions(rng, n).astype(np.float32), 0 * at, 0 * at, 1000.0,
                            [[scenes._box((0.25, 0.25, 0.25))] for _ in range(n)], mats)
    a, b = pkg.World(0), pkg.World(0)
    for w in (a, b):
        w.add_scene(spec)
        w.collide()
    assert a.counts()["pairs"] > 300000
    assert a.fit_pair_budget(1.2) < 1 << 20
    for w in (a, b):
        w.step(DT)
    assert a.kernels_per_step() == b.kernels_per_step() + 1
    np.testing.assert_array_equal(a.read_bodies(), b.read_bodies())
    for x, y in zip(a.manifolds()[:2], b.manifolds()[:2]):
        np.testing.assert_array_equal(x, y)
