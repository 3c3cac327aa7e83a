"""Calls at the edges of the block sweeps' reach."""
import ctypes

import numpy as np
import pytest

from sapien_gb300 import PinocchioModel
from sapien_gb300 import _native as N
from test_bfp_gpu import ROBOTS, cuda, fp64_route, host, pair, rel_per_env

pytestmark = pytest.mark.gpu


def test_more_checkpoint_segments_than_a_grid_has_rows():
    """A checkpoint before every one of 70000 steps of one environment, all segments in one group:
    accepted, and the bits of groups of at most 20000."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS["slide"]()
    pm, _ = pair(robot)
    T = 70000
    q, qd, _, _ = cuda(*robot.sample(1, seed=2))
    taus = 0.01 * torch.randn(T, 1, 1, generator=torch.Generator().manual_seed(5), dtype=torch.float64).cuda()
    _, _, qc, qdc = AD.rollout_forward(pm, q, qd, taus, 1e-4, 1)
    one = torch.ones(1, 1, dtype=torch.float64, device="cuda")
    need = ctypes.c_int64()
    N.check(N.load().sgdyn_rollout_scratch_bytes(pm._h, 1, 1, ctypes.byref(need)))
    groups = [AD.rollout_backward(pm, qc, qdc, taus, 1e-4, 1, one, one, max_scratch_bytes=b)
              for b in (1 << 30, 5000 * need.value)]
    for a, b in zip(*groups):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("ixz", [0.02, 0.05, 0.1, 0.503, 1.002, -2.01, 30.0])
def test_mass_matrix_that_is_not_positive_definite(ixz):
    """Products of inertia beyond the moments': M = [[a, h], [h, c]] with h^2 up to millions of times
    a c, alone and below another joint. Forward dynamics and its product as in FP64."""
    import torch

    from sapien_gb300 import autodiff as AD

    def body(name, xx, xz):
        return (f'<link name="{name}"><inertial><mass value="1"/><origin xyz="0 0 0" rpy="0 0 0"/>'
                f'<inertia ixx="{xx}" iyy="0.03" izz="0.01" ixy="0" ixz="{xz}" iyz="0"/></inertial></link>')

    def joint(name, parent, child, axis):
        return (f'<joint name="{name}" type="continuous"><origin xyz="0 0 0.1" rpy="0 0 0"/><axis xyz="{axis}"/>'
                f'<parent link="{parent}"/><child link="{child}"/></joint>')

    for axes in (["0 0 1", "1 0 0"], ["0 1 0", "0 0 1", "1 0 0"]):
        names = [f"j{k}" for k in range(len(axes))]
        links = [f"l{k}" for k in range(len(axes) + 1)]
        pm = PinocchioModel("<robot name='r'>" + "".join(body(x, 0.01, ixz if x == links[-1] else 0) for x in links)
                            + "".join(joint(names[k], links[k], links[k + 1], a) for k, a in enumerate(axes))
                            + "</robot>", [0, 0, -9.81])
        pm.set_joint_order(names)
        pm.set_link_order(links)
        rng = np.random.default_rng(1)
        q = 0.3 * rng.normal(size=(9, len(axes)))
        qd, tau = rng.normal(size=q.shape), rng.normal(size=q.shape)

        def run():
            out = [pm.step_batched(*cuda(q, qd, 0 * q, tau), ops=o)["qacc"] for o in (N.OP_ALL, N.OP_FORWARD_DYNAMICS)]
            return [x.cpu().numpy() for x in out]

        mine = run()
        with fp64_route():
            want = run()
        for a, b in zip(mine, want):
            assert rel_per_env(a, b) <= 1e-9
        w = torch.ones(q.shape, dtype=torch.float64, device="cuda")
        tb = AD.forward_dynamics_vjp(pm, *cuda(q, qd, tau), w)[2].cpu().numpy()
        M = host(pm.step_batched(*cuda(q), ops=N.OP_MASS_MATRIX))["mass_matrix"].reshape(len(q), len(axes), len(axes))
        assert rel_per_env(tb, np.linalg.solve(M, np.ones(q.shape)[..., None])[..., 0]) <= 1e-9


def test_right_angles_in_the_placements():
    """rpy="pi 0 pi/2" leaves entries of 1e-17 and 1e-32 in a rotation: the block sweep takes the model
    and matches the FP64 kernels."""
    from test_block_sweep_range import arm

    pm = arm("3.141592653589793 0 1.5707963267948966")
    assert pm.block_sweep
    pm.set_joint_order(["j", "k"])
    pm.set_link_order(["base", "a", "b"])
    ins = cuda(*np.random.default_rng(3).normal(size=(4, 37, 2)))
    got = host(pm.step_batched(*ins))
    with fp64_route():
        assert not pm.block_sweep
        want = host(pm.step_batched(*ins))
    for k in got:
        assert rel_per_env(got[k], want[k]) <= 1e-12, k


@pytest.mark.parametrize("name,n", [("arm9", 2500), ("arm9", 5000), ("arm9", 9800), ("quadruped", 5000),
                                    ("mixed", 9800)])
def test_rollout_and_reverse_pass_in_blocks_of_every_size(name, n):
    """Blocks of 8, 16 and 32 environments, a partly filled last one, two checkpoint segments: the
    FP64 kernels' results."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    q, qd, _, tau = cuda(*robot.sample(n, seed=n))
    taus = (0.1 * tau).unsqueeze(0).repeat(3, 1, 1).contiguous()
    (bar,) = cuda(np.random.default_rng(4).normal(size=qd.shape))

    def run():
        qT, qdT, qc, qdc = AD.rollout_forward(pm, q, 0.1 * qd, taus, 1e-3, 2)
        return [qT, qdT, *AD.rollout_backward(pm, qc, qdc, taus, 1e-3, 2, torch.ones_like(qT), bar)]

    mine = run()
    with fp64_route():
        want = run()
    for i, (a, b) in enumerate(zip(mine, want)):
        assert rel_per_env(*(t.cpu().numpy().reshape(-1, t.shape[-1]) for t in (a, b))) <= 1e-8, i


@pytest.mark.parametrize("name", ["arm9", "quadruped"])
def test_allocation_free_reverse_pass_agrees_with_automatic_settings(name):
    """The block sweeps of sgdyn_rollout_backward and the FP64 kernels of its allocation-free form."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    n, T, K, dt = 21, 7, 3, 1e-3
    q, qd, _, tau = robot.sample(n, seed=3)
    q, qd, tau = cuda(q, 0.1 * qd, np.repeat(tau[None], T, axis=0))
    _, _, qc, qdc = AD.rollout_forward(pm, q, qd, tau, dt, K)
    bars = cuda(np.ones((n, pm.nq_ext)), np.ones((n, pm.nv)))
    want = AD.rollout_backward(pm, qc, qdc, tau, dt, K, *bars)
    got = [torch.empty_like(t) for t in want]
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    N.check(N.load().sgdyn_rollout_backward_noalloc(pm._h, n, T, dt, K, *map(p, (qc, qdc, tau, *bars, *got)),
                                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    for g, w in zip(got, want):
        g, w = (t.movedim(t.dim() - 2, 0).cpu().numpy() for t in (g, w))
        assert rel_per_env(g, w) <= 1e-10
