"""Many scenes with one large island each take another form of the cluster
classes' solver; a scene steps in the crowd exactly as it steps alone, and a
rollout's gradients are the same up to the order of their sums."""
import numpy as np
import pytest

from test_gpu_step_edges import towers

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0


def scene(scenes, size, joined):
    """A tower of `size` cubes; joined: its neighbours held at their distance."""
    spec = towers(scenes, [size], seed=size)
    if joined:
        spec.joints = np.stack([np.arange(0, size - 1, 3), np.arange(1, size, 3)], 1).astype(np.uint32)
        spec.joint_dist = np.full(len(spec.joints), 0.5, np.float32)
    return spec.validate()


@pytest.mark.parametrize("size,count,joined", [(513, 113, True), (1024, 112, False), (1025, 57, True), (2048, 56, False),
                                               (2049, 29, False), (4090, 28, False)])
def test_a_scene_steps_as_alone(pkg, scenes, size, count, joined):
    spec = scene(scenes, size, joined)
    alone, crowd = pkg.World(0), pkg.World(0)
    alone.add_scene(spec)
    for _ in range(count):
        crowd.add_scene(spec)
    for w in (alone, crowd):
        w.set_sleeping(False)
        w.step(DT, 3)
    n = alone.counts()["bodies"]
    want, got = alone.read_bodies(), crowd.read_bodies().reshape(count, n, -1)
    assert int(crowd.islands()[0].max()) >= size
    for k in range(count):      # in its own scene's frame: every scene has the same authored poses
        np.testing.assert_array_equal(got[k], want)


def test_a_rollout_in_the_crowd(pkg, scenes):
    spec = scene(scenes, 600, False)
    grads = []
    for count in (1, 113):
        w = pkg.World(0)
        for _ in range(count):
            w.add_scene(spec)
        w.step(DT, 2)
        w.fit_pair_budget(1.5)
        n = w.counts()["bodies"] // count
        seeds = np.tile(np.random.default_rng(1).normal(0, 1, (n, 3)).astype(np.float32), (count, 1))
        w.rollout_begin(2, 2)
        w.rollout_forward(DT)
        g = w.rollout_backward(seeds)
        grads.append({k: v.reshape(count, n, -1).astype(np.float64) for k, v in g.items() if k in ("v0", "w0", "mass")})
    for k in grads[0]:
        want = grads[0][k][0]
        for got in (grads[1][k][0], grads[1][k][-1]):
            assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
