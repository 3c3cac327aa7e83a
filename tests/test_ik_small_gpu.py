"""Inverse kinematics towards targets next to the initial configuration, along the frames' axes: the
joints keep FP64's relative accuracy, as in the FP64 kernel that forced settings select."""
import numpy as np
import pytest

from test_bfp_gpu import cuda, fp64_route
from test_near_equilibrium_gpu import SMALL, close, joint, link, model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["revolute", "continuous", "prismatic"])
@pytest.mark.parametrize("q0", [None, 0.0, 1e-10])
def test_target_next_to_the_initial_configuration(kind, q0):
    """One joint: each update takes the share a = dt / (1 + damp) of the error that is left."""
    pm = model(link("base") + link("tip") + joint("a", "base", "tip", "0 0 1", kind=kind), ["a"], ["base", "tip"])
    d = SMALL[np.abs(SMALL) < 2.0**-16]
    n = len(d)
    target = np.tile([0.0, 0, 0, 1, 0, 0, 0], (n, 1))
    if kind == "prismatic":
        target[:, 2] = d
    else:
        target[:, 3], target[:, 6] = np.cos(d / 2), np.sin(d / 2)
    steps, dt, damp = 12, 0.25, 0.5
    start = 0.0 if q0 is None else q0
    args = dict(eps=0.0, max_iterations=steps, dt=dt, damp=damp)
    t, i = cuda(target, np.full((n, 1), start))
    q, ok, err = pm.compute_inverse_kinematics_batched(1, t, None if q0 is None else i, **args)
    # 24 operations an update, each within half a unit of the terms |d| + |q0|
    left = (1 - dt / (1 + damp)) ** steps
    want = d + (start - d) * left
    room = 24 * steps * 2.0**-53 * (np.abs(d) + start)
    assert (np.abs(q[:, 0].cpu().numpy() - want) <= room).all()
    with fp64_route():
        q64, ok64, err64 = pm.compute_inverse_kinematics_batched(1, t, None if q0 is None else i, **args)
    assert (ok.cpu() == ok64.cpu()).all()
    assert (np.abs((err - err64).cpu().numpy()) <= room[:, None]).all()
    assert (np.abs((q - q64)[:, 0].cpu().numpy()) <= room).all()


def test_small_error_beside_large_ones():
    """Environments next to their target among others that are not: these keep their bits."""
    from sapien_gb300 import synthetic as syn
    from test_bfp_gpu import pair

    import torch

    robot = syn.arm_with_fingers(sapien_style=True)
    pm, _ = pair(robot)
    n = 70
    q, _, _, _ = robot.sample(n, seed=1)
    g, _, _, _ = robot.sample(n, seed=2)
    near = np.arange(n) % 9 == 3
    far = g.copy()
    g[near] = q[near] + 1e-9
    a, b = (pm.compute_forward_kinematics_batched(*cuda(x))[:, robot.ee_link].contiguous() for x in (far, g))
    (i,) = cuda(q)
    args = dict(eps=0.0, max_iterations=20, dt=0.1, damp=1e-3)
    plain = pm.compute_inverse_kinematics_batched(robot.ee_link, a, i, **args)
    mixed = pm.compute_inverse_kinematics_batched(robot.ee_link, b, i, **args)
    keep = torch.from_numpy(~near).cuda()
    for x, y in zip(plain, mixed):
        assert torch.equal(x[keep], y[keep])
    with fp64_route():
        want = pm.compute_inverse_kinematics_batched(robot.ee_link, b, i, **args)
    # 20 updates of some 50 roundings of terms of about 1, through an inverse of at most 1 / (2 sqrt(damp))
    for x, y in zip(mixed, want):
        assert (x[~keep].double() - y[~keep].double()).abs().max() <= 20 * 50 * 2.0**-53 * 16
