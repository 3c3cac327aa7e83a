"""Large batches of deep trees go through the FP64 kernels, where these are the faster; the
block sweep keeps the others. Both sides of each rule: whether the bits are those of the FP64
kernels."""
import contextlib

import numpy as np
import pytest

from sapien_gb300 import _native as N, synthetic as syn
from test_bfp_gpu import ROBOTS, cuda, pair, rel_per_env

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def fp64():
    L = N.load()
    try:
        assert L.sgdyn_step_split(0, None) == N.OK
        yield
    finally:
        L.sgdyn_step_split(2, None)


def robot_of(name):
    return syn.serial_chain(int(name[5:]), seed=23) if name.startswith("chain") else ROBOTS[name]()


def check(run, takes_fp64, bound=None):
    mine = [t.cpu().numpy() for t in run()]
    with fp64():
        want = [t.cpu().numpy() for t in run()]
    same = all(np.array_equal(a, b) for a, b in zip(mine, want))
    assert same == takes_fp64
    if bound is not None:
        for a, b in zip(mine, want):
            assert rel_per_env(a, b) <= bound


FK, RNEA, ABA, CRBA = N.OP_FK, N.OP_INVERSE_DYNAMICS, N.OP_FORWARD_DYNAMICS, N.OP_MASS_MATRIX


@pytest.mark.parametrize("name,n,ops,takes_fp64", [
    ("chain40", 1000, ABA, False), ("chain40", 4000, ABA, True), ("chain40", 4000, ABA | RNEA, False),
    ("chain40", 8000, ABA | RNEA, True), ("chain40", 8000, FK, False), ("chain40", 13000, FK, True),
    ("chain40", 13000, RNEA, True), ("chain40", 13000, CRBA | RNEA | ABA, True), ("chain40", 13000, CRBA, False),
    ("chain40", 13000, N.OP_ALL, True), ("chain16", 40000, ABA, False), ("humanoid", 12000, ABA, False), ("quadruped", 40000, ABA, False)])
def test_steps(name, n, ops, takes_fp64):
    robot = robot_of(name)
    pm, _ = pair(robot)
    x = cuda(*robot.sample(n, seed=4))
    check(lambda: list(pm.step_batched(*x, ops=ops).values()), takes_fp64, None if ops & ABA else 1e-10)


@pytest.mark.parametrize("name,n,takes_fp64", [("chain40", 1500, False), ("chain40", 4000, True),
                                               ("quadruped", 12000, False), ("quadruped", 20000, True),
                                               ("arm9", 33000, False)])
def test_rollouts(name, n, takes_fp64):
    """Both passes of a rollout take the same kernels."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = robot_of(name)
    pm, _ = pair(robot)
    q, qd, _, _ = robot.sample(n, seed=6)
    T, K, dt = 2, 1, 1e-4
    q, qd = cuda(q, 0.1 * qd)
    tau = torch.zeros(T, n, pm.nv, dtype=torch.float64, device="cuda")
    one = torch.ones(n, pm.nq_ext, dtype=torch.float64, device="cuda")

    def run():
        qT, qdT, qc, qdc = AD.rollout_forward(pm, q, qd, tau, dt, K)
        q0b, qd0b, _ = AD.rollout_backward(pm, qc, qdc, tau, dt, K, qT_bar=one)
        return qT, qdT, q0b, qd0b

    check(run, takes_fp64)


@pytest.mark.parametrize("name,n,which,takes_fp64", [
    ("chain40", 8000, "inverse", False), ("chain40", 10000, "inverse", True), ("humanoid", 10000, "inverse", False),
    ("chain40", 3000, "forward", False), ("chain40", 5000, "forward", True), ("arm9", 40000, "forward", False)])
def test_products(name, n, which, takes_fp64):
    from sapien_gb300 import autodiff as AD

    robot = robot_of(name)
    pm, _ = pair(robot)
    q, qd, qdd, tau = cuda(*robot.sample(n, seed=8))
    (w,) = cuda(np.random.default_rng(1).normal(size=(n, pm.nv)))
    f = AD.inverse_dynamics_vjp if which == "inverse" else AD.forward_dynamics_vjp
    check(lambda: f(pm, q, qd, qdd if which == "inverse" else tau, w), takes_fp64)


@pytest.mark.parametrize("n,takes_fp64", [(8000, False), (15000, True)])
def test_passive_forces(n, takes_fp64):
    robot = robot_of("chain40")
    pm, _ = pair(robot)
    q, qd, _, _ = robot.sample(n, seed=9)
    x = cuda(q.astype(np.float32), qd.astype(np.float32))
    mine = pm.compute_passive_force_batched(*x)
    with fp64():
        want = pm.compute_passive_force_batched(*x)
    # rounded to float32, equal results need not be of one kernel
    if takes_fp64:
        assert (mine == want).all()
    assert rel_per_env(mine.double().cpu().numpy(), want.double().cpu().numpy()) <= 2.0**-23


@pytest.mark.parametrize("what", ["rollout", "product"])
def test_first_call_under_capture(what):
    """A call that changes over to kernels compiled at run time, captured before any of them is there."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = syn.quadruped(seed=71 if what == "rollout" else 72)
    pm, _ = pair(robot)
    n = 24000
    q, qd, _, tau = cuda(*robot.sample(n, seed=6))
    pm._prepare(q.device)
    if what == "rollout":
        def run():
            return AD.rollout_forward(pm, q, qd, tau[None], 1e-4)[:2]
    else:
        def run():
            return AD.forward_dynamics_vjp(pm, q, qd, tau, qd)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = run()
    g.replay()
    direct = run()
    torch.cuda.synchronize()
    for a, b in zip(captured, direct):
        assert rel_per_env(a.cpu().numpy(), b.cpu().numpy()) <= 1e-9
