"""A manifold whose cached normals sum to zero has no contact normal: the
step reports it and rolls back,
in the one-kernel narrowphase and in the split one of large pair budgets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0
K_ERR_CONTACT = 1 << 1


def stack(pkg, scenes):
    at = np.array([(0.0, 0.25 + 0.5 * k, 0.0) for k in range(3)], np.float32)
    quat = np.tile(np.array([0, 0, 0, 1], np.float32), (3, 1))
    mats = np.tile(np.array([0.5, 0.5, 0.0], np.float32), (3, 1))
    w = pkg.World(0)
    w.add_scene(scenes._assemble(at, quat, 0 * at, 0 * at, 1000.0, [[scenes._box((0.25, 0.25, 0.25))] for _ in range(3)],
                                 mats))
    w.set_sleeping(False)
    w.step(DT, 60)
    return w


@pytest.mark.parametrize("budget", [0, 1 << 20])
@pytest.mark.parametrize("steps", [0, 1, 3])        # 0: a collision pass
def test_cancelling_normals_roll_back(pkg, scenes, budget, steps):
    w = stack(pkg, scenes)
    if budget:
        assert w.set_pair_budget(budget) >= budget
    pairs, counts, _ = w.manifolds()
    assert [2, 3] in pairs.tolist() and counts.max() == 4    # shape 0 is the floor
    before = w.read_bodies()
    w.test_clear_normals(3, 2)
    with pytest.raises(OverflowError):
        w.step(DT, steps) if steps else w.collide()
    assert w.error_bits() == K_ERR_CONTACT
    np.testing.assert_array_equal(w.read_bodies(), before)


def test_hook_refuses_what_has_no_manifold(pkg, scenes):
    w = stack(pkg, scenes)
    with pytest.raises(ValueError):
        w.test_clear_normals(1, 3)                  # apart
    with pytest.raises(ValueError):
        w.test_clear_normals(0, 1)                  # the floor
