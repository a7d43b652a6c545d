"""The reverse sweep at the edges of its island classes (towers of n cubes are
islands of n descriptors): packed in a warp up to 32, one warp up to 96, one
CTA up to 512, and global memory beyond, against the FP64 model with the
tolerances of test_gpu_adjoint.  One step: in a second one the 32- and 33-high
towers pass a branch that the FP64 model takes the other way (the error is then
6e-2 in whatever kernel sweeps them).  And its sums: a sweep is linear in its seeds,
so seeds scaled by 2^-100 must give the same gradients times 2^-100 although
many of a row's terms would then be subnormal (four roundings allowed)."""
import numpy as np
import pytest

from test_gpu_adjoint import (body_props, dynamic_mask, initial_velocities, one_scene_model, rel_norm, set_velocities,
                              shape_friction)
from test_gpu_step_edges import towers

pytestmark = pytest.mark.gpu

DT = 1.0 / 120.0


@pytest.mark.parametrize("sizes,tuning", [
    ([1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 2, 1], {}), ([64, 65, 96, 97], {}),
    ([32, 33, 48, 49], {"island_warp": 48, "island_cta": 128}), ([128, 129], {"island_warp": 32, "island_cta": 128})])
def test_class_edges_match_fp64_model(pkg, scenes, sizes, tuning):
    import torch
    import diff_model as dm
    spec = towers(scenes, sizes, seed=len(sizes))
    wa, wb = pkg.World(0), pkg.World(0)
    for w in (wa, wb):
        w.add_scene(spec)
        if tuning:
            w.set_tuning(**tuning)
        w.step(DT)
    assert sorted(wa.islands()[0].tolist()) == sorted(sizes)
    steps = 1
    nb = wa.counts()["bodies"]
    dyn = dynamic_mask(wa)
    v0, w0 = (0.2 * x for x in initial_velocities(nb, dyn))
    for w in (wa, wb):
        set_velocities(w, v0, w0)
    rng = np.random.default_rng(7)
    a, b = (rng.normal(size=(nb, 3)) * dyn[:, None] for _ in range(2))
    wa.rollout_begin(steps, steps)
    wa.rollout_forward(DT)
    cK, _ = wa.read_mass_frames()
    g = wa.rollout_backward(grad_center=a, grad_velocity=b)
    c0, q0 = wb.read_mass_frames()
    recs = dm.record(wb, steps, DT)
    model = one_scene_model(dm, wb, [spec])
    props = body_props(wb)
    T = lambda x, grad=False: torch.tensor(np.asarray(x, np.float64), requires_grad=grad)  # noqa: E731
    v0t, w0t = T(v0, True), T(w0, True)
    mass = T(np.where(dyn, 1.0 / np.where(props[:, 0] > 0, props[:, 0], 1.0), 1.0), True)
    mus, mud = (T(x, True) for x in shape_friction([spec]))
    c, q, v, w = model.rollout(recs, DT, T(c0), T(q0), v0t, w0t, mass, mus, mud)
    assert np.max(np.abs(torch.stack(c).detach().numpy() - cK)[dyn]) < 1e-4
    ((torch.stack(c) * T(a)).sum() + (torch.stack(v) * T(b)).sum()).backward()
    assert rel_norm(g["v0"][dyn], v0t.grad.numpy()[dyn]) <= 1e-3
    assert rel_norm(g["w0"][dyn], w0t.grad.numpy()[dyn]) <= 1e-3
    assert rel_norm(g["mass"][dyn], mass.grad.numpy()[dyn]) <= 1e-3
    ref_mu = sum(x.grad.numpy() for x in (mus, mud) if x.grad is not None)
    assert rel_norm(g["static_friction"] + g["dynamic_friction"], ref_mu) <= 1e-3


def test_small_seeds_keep_their_precision(pkg, scenes):
    w = pkg.World(0)
    for s in scenes.loose_piles(16, 64):
        w.add_scene(s)
    w.step(DT, 60)
    w.fit_pair_budget(1.5)
    seeds = np.random.default_rng(0).normal(0, 1, (w.counts()["bodies"], 3)).astype(np.float32)
    grads = []
    for scale in (0, -100):
        w.rollout_begin(1, 1)
        w.rollout_forward(DT)
        grads.append(np.ldexp(w.rollout_backward(np.ldexp(seeds, scale))["v0"].astype(np.float64), -scale))
        w.rollout_rewind()
    assert np.abs(grads[0]).max() > 0
    assert rel_norm(grads[1], grads[0]) <= 4 * np.finfo(np.float32).eps
