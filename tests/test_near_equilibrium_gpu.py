"""States whose results are small against the terms they are summed from, or proportional to a small
angle: the batched sweeps keep the relative accuracy of FP64 there. Robots with joint axes along
the frame's axes, so that FP64 has no larger terms to lose the small ones in, against closed
forms; tolerances are a few dozen FP64 roundings of the result itself."""
import numpy as np
import pytest

from sapien_gb300 import PinocchioModel
from sapien_gb300 import _native as N
from test_bfp_gpu import ROBOTS, cuda, fp64_route, host, pair, rel_per_env

pytestmark = pytest.mark.gpu

EPS = 2.0**-53
M, LC, IYY, G = 1.3, 0.45, 0.021, 9.81
SMALL = np.array([s * v for v in (1e-1, 1e-2, 1e-3, 1e-5, 1e-7, 1e-9, 1e-12, 1e-15, 1e-18, 1e-20) for s in (1, -1)])


def link(name, com=(0, 0, 0), mass=M, inertia=(0.03, IYY, 0.01)):
    return (f'<link name="{name}"><inertial><origin xyz="{com[0]} {com[1]} {com[2]}" rpy="0 0 0"/><mass value="{mass}"/>'
            f'<inertia ixx="{inertia[0]}" iyy="{inertia[1]}" izz="{inertia[2]}" ixy="0" ixz="0" iyz="0"/></inertial></link>')


def joint(name, parent, child, axis, xyz=(0, 0, 0), kind="continuous"):
    return (f'<joint name="{name}" type="{kind}"><origin xyz="{xyz[0]} {xyz[1]} {xyz[2]}" rpy="0 0 0"/>'
            f'<parent link="{parent}"/><child link="{child}"/><axis xyz="{axis}"/>'
            '<limit effort="0" velocity="0" lower="-3.2" upper="3.2"/></joint>')


def model(body, joints, links):
    m = PinocchioModel(f'<robot name="r">{body}</robot>', [0, 0, -G])
    m.set_joint_order(joints)
    m.set_link_order(links)
    return m


def pendulum():
    return model(link("base") + link("bob", (0, 0, -LC)) + link("tip", (0, 0, 0), 1e-9, (1e-9, 1e-9, 1e-9))
                 + joint("a", "base", "bob", "0 1 0", kind="revolute")
                 + joint("end", "bob", "tip", "0 0 1", (0, 0, -2 * LC), kind="fixed"), ["a"], ["base", "bob", "tip"])


def close(got, want, rounds):
    got, want = np.asarray(got, dtype=np.float64), np.asarray(want, dtype=np.float64)
    assert (np.abs(got - want) <= rounds * EPS * np.abs(want)).all(), np.abs(got / want - 1).max()


@pytest.mark.parametrize("n", [1, 20, 3000, 10000])
def test_pendulum_near_its_equilibrium(n):
    """Gravity torque, acceleration, passive force, link position and a step of a rollout with its
    reverse pass: everything is proportional to sin q."""
    import torch

    from sapien_gb300 import autodiff as AD

    pm = pendulum()
    q = np.resize(SMALL, n).reshape(n, 1)
    zero = np.zeros_like(q)
    out = host(pm.step_batched(*cuda(q, zero, zero, zero)))
    tip = 1e-9
    grav = (M * LC + tip * 2 * LC) * G
    inertia = M * LC**2 + IYY + tip * (2 * LC) ** 2 + tip
    s = np.sin(q)
    close(out["qf"], grav * s, 64)
    close(out["qacc"], -grav / inertia * s, 64)
    for ops, key, want in ((N.OP_INVERSE_DYNAMICS, "qf", grav * s), (N.OP_FORWARD_DYNAMICS, "qacc", -grav / inertia * s)):
        close(host(pm.step_batched(*cuda(q, zero, zero, zero), ops=ops))[key], want, 64)
    close(out["link_poses"].reshape(n, -1, 7)[:, 2, 0], -2 * LC * s[:, 0], 64)
    f = pm.compute_passive_force_batched(*cuda(q.astype(np.float32), zero.astype(np.float32))).cpu().numpy()
    assert (np.abs(f - grav * np.sin(q.astype(np.float32).astype(np.float64))) <= 2.0**-23 * np.abs(f)).all()
    # dqdd/dq and the adjoint of inverse dynamics with a velocity adjoint of 0
    w = torch.ones(n, 1, dtype=torch.float64, device="cuda")
    qb, _, tb = AD.forward_dynamics_vjp(pm, *cuda(q, zero, zero), w)
    close(qb.cpu(), -grav / inertia * np.cos(q), 64)
    close(tb.cpu(), np.full((n, 1), 1 / inertia), 64)
    # rollout: two steps by hand
    dt, T = 1e-2, 2
    qT, qdT, qc, qdc = AD.rollout_forward(pm, *cuda(q, zero, np.zeros((T, n, 1))), dt, 1)
    x, v = q.copy(), zero.copy()
    for _ in range(T):
        v = v - dt * grav / inertia * np.sin(x)
        x = x + dt * v
    close(qT.cpu(), x, 64)
    close(qdT.cpu(), v, 64)
    b = AD.rollout_backward(pm, qc, qdc, *cuda(np.zeros((T, n, 1))), dt, 1, torch.zeros_like(w), w)
    k = -grav / inertia * np.cos(qc[:, :, 0].cpu().numpy())  # (adjoint of qd_2 = sums of dt k over the way)
    q0b = dt * k[0] + dt * k[1] * (1 + dt * dt * k[0])
    close(b[0].cpu().numpy()[:, 0], q0b, 256)


def test_slow_accelerations_and_motion_across_gravity():
    """Rest at q = 0 with a small acceleration; two joints about the direction of gravity moving
    slowly, where the only torques are Coriolis forces."""
    pm = pendulum()
    n = len(SMALL)
    a = SMALL.reshape(n, 1)
    zero = np.zeros_like(a)
    inertia = M * LC**2 + IYY + 1e-9 * (2 * LC) ** 2 + 1e-9
    close(host(pm.step_batched(*cuda(zero, zero, a, zero), ops=N.OP_INVERSE_DYNAMICS))["qf"], inertia * a, 64)
    close(host(pm.step_batched(*cuda(zero, zero, zero, a), ops=N.OP_FORWARD_DYNAMICS))["qacc"], a / inertia, 64)
    l1, c2 = 0.4, 0.25
    pm = model(link("base") + link("one", (0.2, 0, 0)) + link("two", (c2, 0, 0))
               + joint("a", "base", "one", "0 0 1") + joint("b", "one", "two", "0 0 1", (l1, 0, 0)),
               ["a", "b"], ["base", "one", "two"])
    qd = np.stack([SMALL, 0.7 * SMALL], axis=1)
    q = np.tile([0.6, 0.9], (n, 1))
    tau = host(pm.step_batched(*cuda(q, qd, 0 * q, 0 * q), ops=N.OP_INVERSE_DYNAMICS))["qf"]
    h = M * l1 * c2 * np.sin(0.9)
    close(tau[:, 0], -h * (2 * qd[:, 0] * qd[:, 1] + qd[:, 1] ** 2), 128)
    close(tau[:, 1], h * qd[:, 0] ** 2, 128)


def test_small_angle_beside_a_large_one():
    """Two pendulums on one base: each element keeps its own accuracy. The block sweep serves angles
    of 2^-16 and more, exact to a few times 2^-57 of the terms."""
    pm = model(link("base") + link("one", (0, 0, -LC)) + link("two", (0, 0, -LC))
               + joint("a", "base", "one", "0 1 0") + joint("b", "base", "two", "0 1 0", (0, 0.3, 0)),
               ["a", "b"], ["base", "one", "two"])
    small = np.concatenate([SMALL, [2.0**-16, -(2.0**-16), 2.0**-15.5]])
    q = np.stack([np.ones_like(small), small], axis=1)
    out = host(pm.step_batched(*cuda(q, 0 * q, 0 * q, 0 * q)))
    close(out["qf"], M * G * LC * np.sin(q), 16 * 2.0**-57 * 2.0**16 / EPS)
    close(out["qacc"], -M * G * LC / (M * LC**2 + IYY) * np.sin(q), 16 * 2.0**-57 * 2.0**16 / EPS)


@pytest.mark.parametrize("name", ["arm9", "quadruped"])
@pytest.mark.parametrize("n", [9, 2600, 9800])
def test_neighbours_of_refused_environments_keep_their_bits(name, n):
    """Any number of environments of a block in FP64, packed side by side, for its inputs or its
    configuration; a rollout that meets such a step on its way, and its reverse pass. A small
    angle among dense rotations is no reason to refuse: FP64 has no more bits of it there."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    q, qd, qdd, tau = robot.sample(n, seed=n)
    rng = np.random.default_rng(n)
    odd = np.zeros(n, dtype=bool)
    for b in range(0, n, 32):  # 0 to 32 of each 32
        odd[b:b + 32] = rng.permutation(min(32, n - b)) < (b // 32 * 5) % 33
    odd[2] = True
    p = q.copy()
    p[odd, 0] = 1e-80
    if robot.nq_ext > robot.nv:
        p[odd, 0], p[odd, 3:7] = 0.3, [1e-7, 0.0, 0.6, 0.8]
    p[:, -3] = 1e-6
    q[:, -3] = 1e-6
    for ops in (N.OP_ALL, N.OP_FORWARD_DYNAMICS):
        clean = host(pm.step_batched(*cuda(q, qd, qdd, tau), ops=ops))
        g = host(pm.step_batched(*cuda(p, qd, qdd, tau), ops=ops))
        with fp64_route():
            w = host(pm.step_batched(*cuda(p, qd, qdd, tau), ops=ops))
        for k in g:
            assert np.array_equal(g[k][~odd], clean[k][~odd]), (ops, k)
            assert rel_per_env(g[k], w[k]) <= 1e-9, (ops, k)
    if n > 100:
        return
    T, K, dt = 7, 3, 1e-3
    qd = 0.1 * qd
    taus = np.repeat(tau[None], T, axis=0)
    bars = cuda(np.ones((n, pm.nq_ext)), np.ones((n, pm.nv)))

    def run():
        qT, qdT, qc, qdc = AD.rollout_forward(pm, *cuda(q, qd, taus), dt, K)
        return [qT, qdT, *AD.rollout_backward(pm, qc, qdc, *cuda(taus), dt, K, *bars)]

    ref = run()
    taus[2, 4, 1] = taus[5, 4, 0] = taus[3, 4:7, 0] = 1e-80
    mine = run()
    with fp64_route():
        want = run()
    keep = [e for e in range(n) if not 4 <= e < 7]
    for a, b, w in zip(mine, ref, want):
        a, b, w = (t.movedim(t.dim() - 2, 0) for t in (a, b, w))
        assert torch.equal(a[keep], b[keep])
        assert rel_per_env(a[4:7].cpu().numpy(), w[4:7].cpu().numpy()) <= 1e-9
