"""The block-floating-point sweeps (csrc/bfp_block.cuh, csrc/bfp_diff.cuh), which every batched
call takes with its settings automatic, against the oracle and against the FP64 sweeps that
forced settings select. Sizes around the edges of their blocks (4 to 32 environments, fewer per
block while there are few blocks), both layouts, and inputs that send single environments of a
block to the FP64 algebra."""
import contextlib
import ctypes

import numpy as np
import pytest

from oracle.oracle import Oracle
from sapien_gb300 import PinocchioModel, synthetic as syn
from sapien_gb300 import _native as N

pytestmark = pytest.mark.gpu

ROBOTS = {
    "slide": lambda: syn.serial_chain(1, seed=2, kinds=["prismatic"]),
    "mixed": lambda: syn.serial_chain(6, seed=11, kinds=["revolute", "continuous", "prismatic", "revolute",
                                                         "continuous", "prismatic"]),
    "arm9": lambda: syn.arm_with_fingers(sapien_style=True),
    "quadruped": syn.quadruped,
    "humanoid": lambda: syn.humanoid(sapien_style=True),
    "chain40": lambda: syn.serial_chain(40, seed=23),
}


def pair(robot):
    pm, o = PinocchioModel(robot.urdf, [0, 0, -9.81]), Oracle(robot.urdf)
    for m in (pm, o):
        m.set_joint_order(robot.joint_names)
        m.set_link_order(robot.link_names)
    return pm, o


def rel_per_env(g, o):
    g, o = g.reshape(g.shape[0], -1), o.reshape(o.shape[0], -1)
    return (np.abs(g - o).max(axis=1) / np.maximum(np.abs(o).max(axis=1), 1e-300)).max()


@contextlib.contextmanager
def fp64_route():
    """One fused FP64 launch for every batched sweep; one lane for rollouts."""
    L = N.load()
    try:
        assert L.sgdyn_step_split(0, None) == N.OK and L.sgdyn_rollout_lanes(1, None) == N.OK
        yield
    finally:
        L.sgdyn_step_split(2, None)
        L.sgdyn_rollout_lanes(0, None)


def cuda(*arrays):
    import torch

    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def host(out):
    return {k: v.cpu().numpy() for k, v in out.items()}


@pytest.mark.parametrize("name,n", [("slide", 1), ("slide", 33), ("mixed", 7), ("mixed", 2433), ("arm9", 4865),
                                    ("arm9", 9729), ("quadruped", 31), ("quadruped", 4900), ("humanoid", 9),
                                    ("chain40", 5)])
def test_sweep_at_block_edges(name, n):
    """The last environments of a batch that fills its last block partly (block sizes change at
    8, 16 and 32 environments times two blocks per multiprocessor), every op set's outputs
    against the oracle."""
    robot = ROBOTS[name]()
    pm, o = pair(robot)
    ins = robot.sample(n, seed=n)
    tail = slice(max(0, n - 40), n)
    r = o.batch_step(*(a[tail] for a in ins), nthreads=8)
    dev = cuda(*ins)
    p = r["poses"][..., :12].reshape(tail.stop - tail.start, -1, 12)[..., 9:12]
    for ops in (N.OP_ALL, N.OP_MASS_MATRIX, N.OP_INVERSE_DYNAMICS, N.OP_FORWARD_DYNAMICS, N.OP_JACOBIAN, N.OP_FK):
        g = {k: v[tail] for k, v in host(pm.step_batched(*dev, ops=ops)).items()}
        for k, w, tol in (("jacobian", r["J"], 1e-12), ("mass_matrix", r["M"], 1e-12), ("qf", r["tau"], 1e-12),
                          ("qacc", r["qdd"], 1e-8)):
            if k in g:
                assert rel_per_env(g[k], w) <= tol, (ops, k)
        if "link_poses" in g:
            assert np.abs(g["link_poses"][..., :3] - p).max() <= 1e-12 * max(1.0, np.abs(p).max())


@pytest.mark.parametrize("name", ["mixed", "arm9", "quadruped"])
def test_refused_environments_match_fp64(name):
    """Environments out of the range of block floating point (beyond 2^+-200, not finite, a
    quaternion off unit length) come from the FP64 algebra of the same kernel; their neighbours
    in the block are those of the clean batch, bit for bit."""
    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    n = 70
    q, qd, qdd, tau = robot.sample(n, seed=3)
    clean = host(pm.step_batched(*cuda(q, qd, qdd, tau)))
    qd[5] *= 1e70
    qdd[17, 0] = 1e-90
    tau[33] *= 1e75
    q[40, -1] = 1e-80
    odd = [5, 17, 33, 40]
    if robot.nq_ext > robot.nv:
        q[60, 3:7] *= 1.2
        odd.append(60)
    bad = [12, 50]
    qd[12, 0] = np.nan
    q[50, 0] = np.inf
    g = host(pm.step_batched(*cuda(q, qd, qdd, tau)))
    with fp64_route():
        w = host(pm.step_batched(*cuda(q, qd, qdd, tau)))
    rest = [e for e in range(n) if e not in odd + bad]
    for k in clean:
        assert np.array_equal(g[k][rest], clean[k][rest]), k
        assert rel_per_env(g[k][odd], w[k][odd]) <= 1e-9, k
        for e in bad:
            assert np.isfinite(g[k][e]).all() == np.isfinite(w[k][e]).all(), (k, e)


@pytest.mark.parametrize("name,n", [("mixed", 45), ("arm9", 2500), ("quadruped", 11), ("humanoid", 6)])
def test_structure_of_arrays_equals_env_major(name, n):
    import torch

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    ins = cuda(*robot.sample(n, seed=4))
    want = pm.step_batched(*ins)
    soa = [t.t().contiguous() for t in ins]
    keys = ("link_poses", "jacobian", "mass_matrix", "qf", "qacc")
    outs = [torch.full((want[k].numel() // n, n), float("nan"), dtype=torch.float64, device="cuda") for k in keys]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    N.check(N.load().sgdyn_step(pm._h, n, N.OP_ALL, *[p(t) for t in soa + outs], N.COL_MAJOR,
                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    for k, o in zip(keys, outs):
        assert torch.equal(o.t().reshape(want[k].shape), want[k]), k


@pytest.mark.parametrize("name,n", [("slide", 3), ("mixed", 37), ("arm9", 9), ("quadruped", 21), ("humanoid", 5)])
def test_gradients_match_fp64(name, n):
    """Vector-Jacobian products and a rollout over three checkpoint segments with its reverse
    pass, against the FP64 kernels; the smallest scratch (a segment at a time) gives the same
    bits as the largest."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    q, qd, qdd, tau = cuda(*robot.sample(n, seed=6))
    T, K = 8, 3
    taus = tau.unsqueeze(0).repeat(T, 1, 1).contiguous()
    g = torch.Generator(device="cuda").manual_seed(1)
    qTb = torch.randn(n, pm.nq_ext, generator=g, dtype=torch.float64, device="cuda")
    qdTb = torch.randn(n, pm.nv, generator=g, dtype=torch.float64, device="cuda")

    def run():
        qT, qdT, qc, qdc = AD.rollout_forward(pm, q, 0.1 * qd, taus, 1e-3, K)
        back = [AD.rollout_backward(pm, qc, qdc, taus, 1e-3, K, qTb, qdTb, max_scratch_bytes=b) for b in (0, 1 << 30)]
        for a, b in zip(*back):
            assert torch.equal(a, b)
        return [qT, qdT, qc, qdc, *back[0]]

    mine = run()
    with fp64_route():
        want = run()
    for i, (a, b) in enumerate(zip(mine, want)):
        assert rel_per_env(a.cpu().numpy().reshape(-1, a.shape[-1]), b.cpu().numpy().reshape(-1, b.shape[-1])) <= 1e-9, i
    # the products against a one-step central difference of the sweep along a random direction
    d = [torch.randn(n, pm.nv, generator=g, dtype=torch.float64, device="cuda") for _ in range(2)]
    w = qdTb
    for vjp, call, x in ((AD.inverse_dynamics_vjp, pm.compute_inverse_dynamics_batched, qdd),
                         (AD.forward_dynamics_vjp, pm.compute_forward_dynamics_batched, tau)):
        _, vb, xb = vjp(pm, q, qd, x, w)
        h = 1e-6
        fd = ((call(q, qd + h * d[0], x + h * d[1]) - call(q, qd - h * d[0], x - h * d[1])) * w).sum(1) / (2 * h)
        got = (vb * d[0]).sum(1) + (xb * d[1]).sum(1)
        scale = (vb.abs() * d[0].abs()).sum(1) + (xb.abs() * d[1].abs()).sum(1)
        assert float(((got - fd).abs() / scale).max()) <= 1e-6


def test_rollout_that_leaves_the_range_matches_fp64():
    """A rollout whose state overflows part way: the FP64 algebra repeats that environment from
    its start; the others keep their bits."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS["arm9"]()
    pm, _ = pair(robot)
    n, T = 20, 4
    q, qd, _, tau = robot.sample(n, seed=8)
    taus = np.repeat(tau[None], T, axis=0)
    ref = AD.rollout_forward(pm, *cuda(q, qd, taus), 1e-3, None)[:2]
    taus[2, 7] = 1e70
    mine = AD.rollout_forward(pm, *cuda(q, qd, taus), 1e-3, None)[:2]
    with fp64_route():
        want = AD.rollout_forward(pm, *cuda(q, qd, taus), 1e-3, None)[:2]
    keep = [e for e in range(n) if e != 7]
    for a, b, w in zip(mine, ref, want):
        assert torch.equal(a[keep], b[keep])
        assert np.isfinite(a[7].cpu().numpy()).all() == np.isfinite(w[7].cpu().numpy()).all()


def test_reverse_pass_that_leaves_the_range_matches_fp64():
    """An adjoint beyond the integer form's range, with one segment's scratch at a time: each
    group's reverse pass goes on from the previous one's results in place."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS["arm9"]()
    pm, _ = pair(robot)
    n, T, K = 20, 8, 3
    q, qd, _, tau = cuda(*robot.sample(n, seed=9))
    taus = tau.unsqueeze(0).repeat(T, 1, 1).contiguous()
    bars = [torch.ones(n, pm.nv, dtype=torch.float64, device="cuda") for _ in range(2)]
    bars[0][7] *= 1e70
    _, _, qc, qdc = AD.rollout_forward(pm, q, 0.1 * qd, taus, 1e-3, K)
    mine = AD.rollout_backward(pm, qc, qdc, taus, 1e-3, K, *bars, max_scratch_bytes=0)
    with fp64_route():
        _, _, qc, qdc = AD.rollout_forward(pm, q, 0.1 * qd, taus, 1e-3, K)
        want = AD.rollout_backward(pm, qc, qdc, taus, 1e-3, K, *bars, max_scratch_bytes=0)
    for a, b in zip(mine, want):
        assert rel_per_env(a.cpu().numpy().reshape(-1, a.shape[-1]), b.cpu().numpy().reshape(-1, b.shape[-1])) <= 1e-9


def test_mixed_batch_matches_fp64():
    """One launch per model on its rows of the padded arrays, with and without the Euler step,
    against the persistent FP64 kernel that a forced forward-dynamics method selects."""
    import torch

    from sapien_gb300.hetero import HeteroBatch

    robots, moe = syn.hetero_mix(83, seed=3)
    robots.append(ROBOTS["mixed"]())  # a model that no environment uses
    batch = HeteroBatch([pair(r)[0] for r in robots], moe)
    ins = [r.sample(int((moe == k).sum()), seed=k) for k, r in enumerate(robots)]
    q, qd, qdd, tau = (f([x[i] for x in ins]) for i, f in enumerate((batch.pad_q, batch.pad_v, batch.pad_v, batch.pad_v)))
    q[5, 0] = float("nan")  # its environment alone
    ops = N.OP_MASS_MATRIX | N.OP_INVERSE_DYNAMICS | N.OP_FORWARD_DYNAMICS

    def run():
        out = {k: v.zero_() for k, v in batch.alloc_outputs(ops).items()}
        batch.step(q, qd, qdd, tau, ops, out)
        q1, qd1 = q.clone(), qd.clone()
        acc = batch.alloc_outputs(N.OP_FORWARD_DYNAMICS)
        batch.rollout_step(q1, qd1, tau, 1e-3, acc)
        torch.cuda.synchronize()
        return [out["mass_matrix"], out["qf"], out["qacc"], q1, qd1]

    mine = run()
    with fp64_route():
        want = run()
    keep = [e for e in range(len(moe)) if e != 5]
    for a, b in zip(mine, want):
        a, b = a.cpu().numpy().reshape(len(moe), -1), b.cpu().numpy().reshape(len(moe), -1)
        assert rel_per_env(a[keep], b[keep]) <= 1e-9
        assert not np.isfinite(a[5]).all() and not np.isfinite(b[5]).all()


@pytest.mark.parametrize("name,n", [("slide", 1), ("mixed", 35), ("arm9", 300), ("chain40", 6)])
def test_passive_force_matches_fp64(name, n):
    """Gravity and velocity terms on float32 rows with a gap between them, one environment with a
    value that is not finite: the FP64 algebra's bits to a rounding of float32."""
    import torch

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    q, qd, _, _ = robot.sample(n, seed=4)
    rows = np.full((2, n, pm.nv + 3), 7.0, dtype=np.float32)
    rows[0, :, : pm.nv], rows[1, :, : pm.nv] = q, qd
    bad = n // 2 if n > 1 else None
    if bad is not None:
        rows[0, bad, 0] = np.inf
    x, v = cuda(rows[0], rows[1])
    wide = [torch.from_numpy(r[:, : pm.nv].astype(np.float64)).cuda() for r in rows]
    zero = torch.zeros_like(wide[0])
    pm0 = PinocchioModel(robot.urdf, [0, 0, 0])
    pm0.set_joint_order(robot.joint_names)
    with fp64_route():
        full = pm.compute_inverse_dynamics_batched(wide[0], wide[1], zero)
        still = pm.compute_inverse_dynamics_batched(wide[0], zero, zero)
        free = pm0.compute_inverse_dynamics_batched(wide[0], wide[1], zero)
    for gravity, coriolis, want in ((True, True, full), (True, False, still), (False, True, free)):
        got = pm.compute_passive_force_batched(x, v, gravity=gravity, coriolis_and_centrifugal=coriolis)
        got, want = got.cpu().numpy()[:, : pm.nv], want.cpu().numpy()
        keep = [e for e in range(n) if e != bad]
        assert rel_per_env(got[keep].astype(np.float64), want[keep]) <= 2.0**-23
        if bad is not None:
            assert not np.isfinite(got[bad]).all()


@pytest.mark.parametrize("name,n,steps", [("slide", 2, 3), ("mixed", 70, 6), ("arm9", 33, 6), ("quadruped", 5, 2),
                                          ("chain40", 3, 2)])
def test_inverse_kinematics_matches_fp64(name, n, steps):
    """A few iterations towards another pose, free and with a joint held, one environment with a
    target that is not finite, and no iteration at all (the start's own error)."""
    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    q0, _, _, _ = robot.sample(n, seed=3)
    link = len(robot.link_names) - 1
    ahead = pm.step_batched(*cuda(*robot.sample(n, seed=5)), ops=N.OP_FK)["link_poses"]
    target = ahead.cpu().numpy().reshape(n, -1, 7)[:, link].copy()
    if n > 2:
        target[1, 0] = np.nan
    mask = np.ones(pm.nv, dtype=np.int32)
    mask[-1] = 0
    start, goal = cuda(q0, target)

    def run():
        out = []
        for m, it in ((None, steps), (mask, steps), (None, 0)):
            q, ok, err = pm.compute_inverse_kinematics_batched(link, goal, start, max_iterations=it, active_qmask=m)
            out += [q.cpu().numpy(), ok.cpu().numpy(), err.cpu().numpy()]
        return out

    mine = run()
    with fp64_route():
        want = run()
    keep = [e for e in range(n) if np.isfinite(target[e]).all()]
    for i, (a, b) in enumerate(zip(mine, want)):
        if i % 3 == 1:
            assert (a == b).all()
        else:
            assert rel_per_env(a[keep], b[keep]) <= 1e-9
            assert (np.isfinite(a) == np.isfinite(b)).all()


@pytest.mark.parametrize("name", ["quadruped", "arm9"])
def test_forward_dynamics_vjp_on_both_sides_of_the_batch_size_rule(name):
    """The largest batch that stays on one warp per scheduler, one environment more, and the same
    environments in a small batch."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    edge = 32 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    q, qd, _, tau = cuda(*robot.sample(edge + 1, seed=12))
    w = torch.ones_like(qd)
    small = AD.forward_dynamics_vjp(pm, q[-40:], qd[-40:], tau[-40:], w[-40:])
    for n in (edge, edge + 1):
        got = AD.forward_dynamics_vjp(pm, q[-n:], qd[-n:], tau[-n:], w[-n:])
        for a, b in zip(got, small):
            assert rel_per_env(a[-40:].cpu().numpy(), b.cpu().numpy()) <= 1e-9


@pytest.mark.parametrize("name,n", [("quadruped", 1), ("quadruped", 37), ("mixed", 5), ("humanoid", 300)])
def test_coordinate_gradients_in_one_launch(name, n):
    """The launch behind a backward pass against the tensor operations of the public function: a
    few FP64 products and sums of unit size apart."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    (q,) = cuda(robot.sample(n, seed=1)[0])
    g = torch.randn(n, pm.nv, generator=torch.Generator().manual_seed(0), dtype=torch.float64).cuda()
    pm._prepare(q.device)
    want = AD.tangent_to_coordinate_grad(pm, q, g)
    with torch.no_grad():
        got = AD._coordinate_grad(pm, q, g)
    assert got.shape == want.shape
    assert float((got - want).abs().max()) <= 32 * 2.0**-53 * float(g.abs().max()) * 4
