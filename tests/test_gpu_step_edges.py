"""The step at the edges of its size classes, against the oracle.

Islands of exactly n descriptors (towers of n touching cubes) around every
class of the island solvers -- the groups of small ones, one CTA, a cluster
of CTAs, global memory -- with their partition levels exact, and chains of
joints across the classes: velocities and poses within 1e-4 (the step's
tolerance).
Endpoint sorts around the widths of the one-CTA sort, long pair buckets
under one body, and the split narrowphase of large pair budgets: exact.
"""
import numpy as np
import pytest

from test_gpu_parity import oracle_levels

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0
VEL_RTOL = 1e-4


def rel_err(got, want, floor=1e-2):
    return float(np.max(np.abs(got - want) / np.maximum(np.abs(want), floor)))


def towers(scenes, sizes, seed=0):
    rng = np.random.Generator(np.random.PCG64(seed))
    at = np.concatenate([[(2.0 * t, 0.25 + 0.5 * k, 0.0) for k in range(n)] for t, n in enumerate(sizes)])
    n = len(at)
    quat = np.tile(np.array([0, 0, 0, 1], np.float32), (n, 1))
    mats = np.tile(np.array([0.5, 0.5, 0.0], np.float32), (n, 1))
    vel = rng.normal(0, 0.2, (n, 3)).astype(np.float32)
    return scenes._assemble(at.astype(np.float32), quat, vel, 0 * vel, 1000.0,
                            [[scenes._box((0.25, 0.25, 0.25))] for _ in range(n)], mats)


def check_step(pkg, oracle, spec):
    w = pkg.World(0)
    w.add_scene(spec)
    o = oracle.OracleScene(spec)
    w.step(DT)
    o.step(DT)
    np.testing.assert_array_equal(w.pairs(0), o.pairs(0))
    ws, os_ = w.read_bodies(), o.body_states()
    assert rel_err(ws[:, 3:6], os_[:, 3:6]) <= VEL_RTOL
    assert rel_err(ws[:, 10:13], os_[:, 10:13]) <= VEL_RTOL
    assert rel_err(ws[:, 0:3], os_[:, 0:3], floor=1.0) <= VEL_RTOL
    return w, o


@pytest.mark.parametrize("sizes", [
    [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 2, 1, 7], [63, 64, 65, 127, 128, 129, 1], [255, 256, 257],
    [511, 512, 513], [1023, 1024, 1025], [2047, 2048, 2049], [4095, 4096, 4097]])
def test_islands_of_every_class(pkg, oracle, scenes, sizes):
    w, o = check_step(pkg, oracle, towers(scenes, sizes))
    np.testing.assert_array_equal(w.levels(), oracle_levels(o, 0))
    assert sorted(w.islands()[0].tolist()) == sorted(sizes)


@pytest.mark.parametrize("links", [3, 12, 40, 150])
def test_joint_chains_across_classes(pkg, oracle, scenes, links):
    check_step(pkg, oracle, scenes.joint_mechanisms(6, seed=links, links=links, height=40.0, spacing=200.0, speed=0.2))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 1023, 1025, 2047, 2048])
def test_endpoint_sort_sizes(pkg, scenes, n):
    side = max(0.5, (n / 40.0) ** 0.5)
    spec = scenes.random_boxes(n, seed=n, xz=side, y=(0.3, 2.0))
    if n > 8:
        spec.bodies[: n // 4, 0] = spec.bodies[0, 0]       # equal minima: ordered by shape id
        spec.bodies[: n // 4, 3:7] = [0, 0, 0, 1]
        spec.shape_geom[: n // 4] = spec.shape_geom[0]
    w = pkg.World(0)
    w.add_scene(spec)
    w.collide()
    lo = w.encoded_bounds()[1:, 0]
    order = np.lexsort((np.arange(1, n + 1), lo))
    v, i = w.sorted_min_x(0)
    np.testing.assert_array_equal(v, lo[order])
    np.testing.assert_array_equal(i, order + 1)


@pytest.mark.parametrize("n", [7, 9, 33, 200])
def test_long_pair_buckets(pkg, oracle, scenes, n):
    spec = scenes.random_boxes(n + 1, seed=n, xz=1.5, y=(0.75, 0.95), half=(0.05, 0.1))
    spec.bodies[0, 0:7] = [0, 0.6, 0, 0, 0, 0, 1]
    spec.shape_geom[0, :3] = [2.0, 0.1, 2.0]               # overlaps every box low enough
    w = pkg.World(0)
    w.add_scene(spec)
    w.collide()
    o = oracle.OracleScene(spec)
    o.advance_collision()
    p = w.pairs(0)
    np.testing.assert_array_equal(p, o.pairs(0))
    if n >= 33:                                            # longer than one thread sorts
        assert int((p[:, 0] == 1).sum()) > 8


def test_split_narrowphase_is_the_same_step(pkg, scenes):
    """A pair budget above the split's line changes the kernels, not the
    step: bodies, manifolds and levels stay bit-identical."""
    spec = scenes.mixed_scale(900, seed=5, region=(9.0, 6.0, 9.0))
    a, b = pkg.World(0), pkg.World(0)
    for w in (a, b):
        w.add_scene(spec)
        w.step(DT)
    assert a.set_pair_budget(1 << 20) >= 1 << 20
    for steps in (1, 30, 60):
        a.step(DT, steps)
        b.step(DT, steps)
        np.testing.assert_array_equal(a.read_bodies(), b.read_bodies())
        for x, y in zip(a.manifolds()[:2], b.manifolds()[:2]):
            np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(a.levels(), b.levels())
