"""The FP64 kernels behind the block sweeps. They serve forced settings and the models and batches that
the block sweeps leave to them, so what compares their variants runs here with FP64 asked for; the block
sweeps' gradients are compared with theirs; and models that the block sweeps cannot hold go through
every entry point."""
import ctypes

import numpy as np
import pytest

import test_hetero_gpu as hetero
import test_jit_gpu as jit
from sapien_gb300 import PinocchioModel, synthetic as syn
from sapien_gb300 import _native as N
from test_bfp_gpu import ROBOTS, cuda, fp64_route, host, pair, rel_per_env

pytestmark = pytest.mark.gpu


@pytest.fixture
def any_tree_size():
    old = ctypes.c_int()
    N.check(N.load().sgdyn_jit_max_joints(64, ctypes.byref(old)))
    yield
    N.check(N.load().sgdyn_jit_max_joints(old.value, None))


@pytest.mark.parametrize("name", ["arm9", "mixed"])
def test_specialised_rollout(name, any_tree_size):
    with fp64_route():
        jit.test_specialised_rollout_matches_generic(name)


@pytest.mark.parametrize("name", ["arm9", "humanoid"])
def test_specialised_products(name, any_tree_size):
    with fp64_route():
        jit.test_specialised_vjp_matches_generic(name)


@pytest.mark.parametrize("run", [hetero.test_hetero_graph_replay_orders_and_launch_shapes_agree,
                                 hetero.test_lanes_per_environment_agree_with_one_lane,
                                 hetero.test_hetero_rollout_graph_matches_oracle,
                                 hetero.test_fused_rollout_step_equals_step_then_integrate,
                                 hetero.test_hetero_role_warp_sweeps_match_generic_and_graph],
                         ids=lambda f: f.__name__[5:])
def test_mixed_batches(run):
    with fp64_route():
        run()


@pytest.mark.parametrize("lanes", [(1, 1, 1), (1, 2, 4), (2, 2, 4)])
def test_mixed_batch_at_full_size(lanes):
    with fp64_route():
        hetero.test_hetero_full_size_mix_matches_oracle(lanes)


@pytest.mark.parametrize("name,n", [("slide", 3), ("mixed", 37), ("arm9", 9), ("arm9", 2601), ("quadruped", 21),
                                    ("quadruped", 2500), ("humanoid", 5), ("chain40", 7)])
def test_vector_jacobian_products(name, n):
    """All three gradients of both products, both layouts, some outputs left out."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS[name]()
    pm, _ = pair(robot)
    q, qd, qdd, tau = cuda(*robot.sample(n, seed=6))
    (w,) = cuda(np.random.default_rng(1).normal(size=(n, pm.nv)))

    def run():
        return [*AD.inverse_dynamics_vjp(pm, q, qd, qdd, w), *AD.forward_dynamics_vjp(pm, q, qd, tau, w)]

    mine = run()
    with fp64_route():
        want = run()
    assert not all(torch.equal(a, b) for a, b in zip(mine, want))  # two routes
    for i, (a, b) in enumerate(zip(mine, want)):
        scale = b.abs().amax(1).clamp_min(1e-9 * float(b.abs().max()) + 1e-300)
        assert float(((a - b).abs().amax(1) / scale).max()) <= 1e-9, i
    L = N.load()
    p = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    soa = [t.t().contiguous() for t in (q, qd, qdd, tau, w)]
    for k, (fn, x) in enumerate(((L.sgdyn_compute_inverse_dynamics_vjp, soa[2]),
                                 (L.sgdyn_compute_forward_dynamics_vjp, soa[3]))):
        for keep in ((1, 1, 1), (1, 0, 0), (0, 0, 1)):
            outs = [torch.empty(pm.nv, n, dtype=torch.float64, device="cuda") if u else None for u in keep]
            N.check(fn(pm._h, n, p(soa[0]), p(soa[1]), p(x), p(soa[4]), *[p(o) for o in outs], N.COL_MAJOR,
                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
            for o, ref in zip(outs, mine[3 * k:3 * k + 3]):
                assert o is None or torch.equal(o.t(), ref)


def test_settings_reach_gradients_and_passive_forces():
    """Lanes of the model and a forward-dynamics method select the FP64 kernels there too: the bits
    of the forced route."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = ROBOTS["arm9"]()
    pm, _ = pair(robot)
    q, qd, _, tau = cuda(*robot.sample(40, seed=2))
    w = torch.ones_like(qd)

    def run():
        return [*AD.forward_dynamics_vjp(pm, q, qd, tau, w), *AD.inverse_dynamics_vjp(pm, q, qd, tau, w),
                pm.compute_passive_force_batched(q.float(), qd.float())]

    assert pm.block_sweep
    with fp64_route():
        assert not pm.block_sweep
        want = run()
    pm.set_lanes(1)
    lanes = run()
    pm.set_lanes(0)
    L = N.load()
    try:
        assert L.sgdyn_fd_method(1, None) == N.OK
        method = run()
    finally:
        L.sgdyn_fd_method(0, None)
    for a, b, c in zip(want, lanes, method):
        assert torch.equal(a, b) and torch.equal(a, c)


def refused(robot):
    """The robot with one offset of 1e-40 m, out of the block sweep's range, and as it is."""
    at = robot.urdf.index('<origin xyz="', robot.urdf.index("<joint"))
    end = robot.urdf.index('"', at + len('<origin xyz="'))
    models = []
    for xyz in ("0 0 1e-40", "0 0 0"):
        pm = PinocchioModel(robot.urdf[:at] + f'<origin xyz="{xyz}' + robot.urdf[end:], [0, 0, -9.81])
        pm.set_joint_order(robot.joint_names)
        pm.set_link_order(robot.link_names)
        models.append(pm)
    assert not models[0].block_sweep and models[1].block_sweep
    return models


@pytest.mark.parametrize("name", ["mixed", "arm9"])
def test_refused_model_through_every_entry_point(name):
    """Results of the FP64 kernels, which the model takes by itself, against the block sweeps' for the
    same robot without the offending digit."""
    import torch

    from sapien_gb300 import autodiff as AD
    from sapien_gb300.hetero import HeteroBatch

    robot = ROBOTS[name]()
    n, T, K = 35, 6, 4
    q, qd, qdd, tau = cuda(*robot.sample(n, seed=3))
    taus = tau.unsqueeze(0).repeat(T, 1, 1).contiguous()
    (w,) = cuda(np.random.default_rng(2).normal(size=qd.shape))
    link = len(robot.link_names) - 1

    def run(pm):
        out = pm.step_batched(q, qd, qdd, tau)
        r = [out[k] for k in ("link_poses", "jacobian", "mass_matrix", "qf", "qacc")]
        r += [pm.step_batched(q, qd, qdd, tau, ops=1 << b)[k]
              for b, k in enumerate(("link_poses", "jacobian", "mass_matrix", "qf", "qacc"))]
        r += [*AD.inverse_dynamics_vjp(pm, q, qd, qdd, w), *AD.forward_dynamics_vjp(pm, q, qd, tau, w)]
        qT, qdT, qc, qdc = AD.rollout_forward(pm, q, 0.1 * qd, taus, 1e-3, K)
        r += [qT, qdT, *AD.rollout_backward(pm, qc, qdc, taus, 1e-3, K, torch.ones_like(qT), w)]
        r += [pm.compute_passive_force_batched(q.float(), qd.float()).double()]
        target = out["link_poses"].reshape(n, -1, 7)[:, link].contiguous()
        r += [pm.compute_inverse_kinematics_batched(link, target, 0.9 * q, max_iterations=4)[k] for k in (0, 2)]
        return r

    other = pair(ROBOTS["slide"]())[0]

    def mixed(pm):
        moe = np.arange(2 * n) % 2
        batch = HeteroBatch([pm, other], moe)
        z = [np.zeros((n, 1))] * 4
        ins = [f([x.cpu().numpy(), y]) for f, x, y in zip((batch.pad_q, batch.pad_v, batch.pad_v, batch.pad_v),
                                                         (q, qd, qdd, tau), z)]
        out = batch.step(*ins)
        return [batch.unpad_v(out[k], 0) for k in ("qf", "qacc")] + [batch.unpad_M(out["mass_matrix"], 0)]

    bad, good = refused(robot)
    for i, (a, b) in enumerate(zip(run(bad) + mixed(bad), run(good) + mixed(good))):
        a, b = (t.cpu().numpy().reshape(-1, t.shape[-1]) for t in (a, b))
        assert rel_per_env(a, b) <= (2.0**-23 if i == 21 else 1e-9), i  # (21: passive forces in float32)


def test_tree_too_large_for_a_block():
    """A chain of 63 joints: no block holds four environments of it."""
    import torch

    from sapien_gb300 import autodiff as AD

    robot = syn.serial_chain(63, seed=8)
    pm, o = pair(robot)
    assert not pm.block_sweep
    q, qd, qdd, tau = robot.sample(9, seed=1)
    r = o.batch_step(q, qd, qdd, tau)
    dev = cuda(q, qd, qdd, tau)
    for ops in (N.OP_ALL, N.OP_MASS_MATRIX, N.OP_INVERSE_DYNAMICS, N.OP_FORWARD_DYNAMICS, N.OP_JACOBIAN):
        g = host(pm.step_batched(*dev, ops=ops))
        for k, w, tol in (("jacobian", r["J"], 1e-10), ("mass_matrix", r["M"], 1e-10), ("qf", r["tau"], 1e-10),
                          ("qacc", r["qdd"], 1e-8)):
            assert k not in g or rel_per_env(g[k], w) <= tol, (ops, k)
    f = pm.compute_passive_force_batched(dev[0].float(), dev[1].float()).cpu().numpy()
    want = pm.compute_inverse_dynamics_batched(dev[0].float().double(), dev[1].float().double(), 0 * dev[1]).cpu().numpy()
    assert rel_per_env(f, want) <= 2.0**-23
    w = torch.ones_like(dev[1])
    for vjp, dense, x in ((AD.inverse_dynamics_vjp, AD.rnea_derivatives, dev[2]),
                          (AD.forward_dynamics_vjp, AD.aba_derivatives, dev[3])):
        got, rows = vjp(pm, dev[0], dev[1], x, w), dense(pm, dev[0], dev[1], x)
        for a, D in zip(got, rows):
            assert rel_per_env(a.cpu().numpy(), D.reshape(9, 63, 63).sum(1).cpu().numpy()) <= 1e-8
    T = 3
    taus = dev[3].unsqueeze(0).repeat(T, 1, 1).contiguous()
    qT, qdT, qc, qdc = AD.rollout_forward(pm, dev[0], 0.1 * dev[1], taus, 1e-4, 2)
    x, v = q.copy(), 0.1 * qd
    for _ in range(T):
        acc = o.batch_step(x, v, qdd, tau)["qdd"]
        v = v + 1e-4 * acc
        x = x + 1e-4 * v
    assert rel_per_env(qT.cpu().numpy(), x) <= 1e-9 and rel_per_env(qdT.cpu().numpy(), v) <= 1e-8
    back = AD.rollout_backward(pm, qc, qdc, taus, 1e-4, 2, torch.ones_like(qT), torch.ones_like(qdT))
    assert all(torch.isfinite(b).all() for b in back)
