"""The work that users have this framework do, for measuring it: batched sweeps of one robot
model at several sizes, gradients, rollouts, inverse kinematics, dense derivatives and mixed
batches. Robots are the seeded synthetic ones of ``sapien_gb300.synthetic`` (float64, as every
entry point but the passive force, which reads float32 simulator state)."""
import math
import xml.etree.ElementTree as ET

import numpy as np
import torch

from sapien_gb300 import PinocchioModel, autodiff, synthetic
from sapien_gb300 import _native as N
from sapien_gb300.hetero import HeteroBatch

DYNAMICS = N.OP_MASS_MATRIX | N.OP_INVERSE_DYNAMICS | N.OP_FORWARD_DYNAMICS
GRAVITY = (0.0, 0.0, -9.81)

# kind of call: (robots, smallest and largest batch) of its range
RANGES = {
    "step": (("chain7", "arm6", "arm9", "quadruped18", "humanoid30"), 1, 131072),
    "dynamics": (("chain7", "arm6", "arm9", "quadruped18", "humanoid30"), 16, 262144),
    "forward": (("chain7", "arm9", "quadruped18", "humanoid30"), 16, 131072),
    "passive": (("chain7", "arm9"), 64, 131072),
    "gradient": (("chain7", "arm9", "quadruped18"), 64, 32768),
    "rollout": (("arm9", "arm6", "quadruped18"), 64, 4096),
    "mix": (("mix",), 256, 8192),
    "mix_rollout": (("mix",), 256, 8192),
    "ik": (("chain7", "arm9"), 16, 65536),
    "derivatives": (("arm9", "quadruped18", "humanoid30"), 32, 8192),
}


def _case(name, kind, robot, n, style=False, steps=0):
    return {"name": name, "kind": kind, "robot": robot, "n": n, "exporter_style": style, "steps": steps}


def listed():
    return [
        # a controller that asks for everything about a handful of sampled states
        _case("step_chain7_16", "step", "chain7", 16, style=True),
        # a thousand sampled configurations of a 7-DoF arm
        _case("step_chain7_1000", "step", "chain7", 1000),
        # the benchmark's batch: all five quantities for 16384 environments of a 9-DoF arm
        _case("step_arm9_16384", "step", "arm9", 16384),
        # a large training batch that needs M, inverse and forward dynamics; a ragged size
        _case("dynamics_arm9_131071", "dynamics", "arm9", 131071, style=True),
        # simulating a floating-base robot: forward dynamics alone, a ragged middle size
        _case("forward_quadruped_3001", "forward", "quadruped18", 3001),
        # a wide tree in a small batch: whole-body control of humanoids
        _case("dynamics_humanoid_1024", "dynamics", "humanoid30", 1024),
        # gravity and Coriolis compensation read from float32 simulator state
        _case("passive_arm9_4096", "passive", "arm9", 4096, style=True),
        # one optimiser step through inverse and forward dynamics, values and gradients
        _case("gradient_arm9_16384", "gradient", "arm9", 16384),
        # trajectory optimisation: a checkpointed rollout and its gradients
        _case("rollout_arm9_4096", "rollout", "arm9", 4096, steps=200),
        # robots of three kinds stepped together, by a recorded graph
        _case("mix_8192", "mix", "mix", 8192, steps=4),
        # following targets: up to 100 CLIK iterations for each
        _case("ik_arm9_65536", "ik", "arm9", 65536, steps=100),
        # linearisation of humanoid dynamics for an optimal-control solver
        _case("derivatives_humanoid_8192", "derivatives", "humanoid30", 8192),
    ]


def draw(rng):
    kind = rng.choice(sorted(RANGES))
    robots, lo, hi = RANGES[kind]
    robot = rng.choice(robots)
    if robot in ("quadruped18", "humanoid30"):
        hi = min(hi, 32768 if robot == "quadruped18" else 8192)
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if n > 4 and rng.random() < 0.5:
        n |= 1
    steps = {"rollout": rng.choice((20, 50, 100)), "mix": rng.choice((1, 3, 8)), "mix_rollout": rng.choice((2, 5, 10)),
             "ik": rng.choice((10, 30, 100))}.get(kind, 0)
    return {"kind": kind, "robot": robot, "n": max(lo, min(n, hi)),
            "exporter_style": robot != "mix" and rng.random() < 0.4, "steps": steps}


# ---- inputs ------------------------------------------------------------------------
def _robot(case):
    return synthetic.by_name(case["robot"], sapien_style=bool(case["exporter_style"]))


def _model(robot):
    m = PinocchioModel(robot.urdf, GRAVITY)
    m.set_joint_order(robot.joint_names)
    m.set_link_order(robot.link_names)
    return m


def _sample(robot, n, gen, dev):
    """q within the joint limits (floating base: a position in the unit cube and any attitude),
    velocities and accelerations of the order of one, torques of the order of ten."""
    u = lambda lo, hi, c: lo + (hi - lo) * torch.rand(n, c, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    g = lambda c, s=1.0: s * torch.randn(n, c, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    cols = []
    for kind, (lo, hi) in zip(robot.joint_kinds, robot.joint_limits):
        if kind == synthetic.FLOATING:
            quat = g(4)
            cols += [u(-1.0, 1.0, 3), quat / quat.norm(dim=1, keepdim=True)]
        else:
            cols.append(u(lo, hi, 1))
    return torch.cat(cols, dim=1).contiguous(), g(robot.nv), g(robot.nv), g(robot.nv, 10.0)


def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def _mix_parts(case):
    robots, model_of_env = synthetic.hetero_mix(case["n"])
    return robots, model_of_env, [int((model_of_env == k).sum()) for k in range(len(robots))]


def _inputs(case, seed, dev):
    """The case's inputs: one set, or for a mixed batch one per robot."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    n, kind = case["n"], case["kind"]
    if kind in ("mix", "mix_rollout"):
        robots, _, counts = _mix_parts(case)
        return [_sample(r, c, gen, dev) for r, c in zip(robots, counts)]
    robot = _robot(case)
    q, qd, qdd, tau = _sample(robot, n, gen, dev)
    if kind == "passive":
        pad = torch.zeros(n, 3, dtype=torch.float64, device=dev)
        return torch.cat([q, pad], dim=1).float().contiguous(), torch.cat([qd, pad], dim=1).float().contiguous()
    if kind == "gradient":
        w = torch.randn(n, robot.nv, generator=gen, dtype=torch.float64, device=dev)
        return q, qd, qdd, tau, w
    if kind == "rollout":
        small = torch.randn(case["steps"], n, robot.nv, generator=gen, dtype=torch.float64, device=dev)
        goal = torch.randn(n, robot.nv, generator=gen, dtype=torch.float64, device=dev)
        return q, 0.1 * qd, small, goal
    if kind == "ik":
        # following a moving target: the end effector's pose a few degrees per joint from the start
        lo = torch.tensor([a for a, _ in robot.joint_limits], dtype=torch.float64, device=dev)
        hi = torch.tensor([b for _, b in robot.joint_limits], dtype=torch.float64, device=dev)
        start = torch.minimum(torch.maximum(q + 0.05 * qd * (hi - lo) / (2 * math.pi), lo), hi)
        tree = _Tree(robot)
        R, p = tree.poses(q)[tree.links[robot.ee_link]]
        return torch.cat([p, _quaternion(R)], dim=1).contiguous(), start.contiguous()
    return q, qd, qdd, tau


def prepare(case, seed):
    dev = _device()
    kind = case["kind"]
    data = _inputs(case, seed, dev)
    state = {"kind": kind, "data": data, "case": case}
    if kind in ("mix", "mix_rollout"):
        robots, model_of_env, _ = _mix_parts(case)
        batch = HeteroBatch([_model(r) for r in robots], model_of_env)
        batch.set_launch(8, 1, 0)
        batch.set_lanes((1, 4, 4))
        place = [torch.as_tensor(np.nonzero(model_of_env == k)[0], device=dev) for k in range(len(robots))]

        def pad(i, width):
            out = torch.zeros(case["n"], width, dtype=torch.float64, device=dev)
            for rows, d in zip(place, data):
                out[rows, : d[i].shape[1]] = d[i]
            return out

        q, qd, qdd, tau = pad(0, batch.max_nq), pad(1, batch.max_nv), pad(2, batch.max_nv), pad(3, batch.max_nv)
        state.update(batch=batch, q=q, qd=qd, qdd=qdd, tau=tau, rows=place)
        if kind == "mix":
            out = batch.alloc_outputs(DYNAMICS)
            for t in out.values():
                t.zero_()  # the padding is never written
            state["graph"] = batch.capture(q, qd, qdd, tau, steps=case["steps"], ops=DYNAMICS, out=out)
        else:
            state["graph"] = batch.capture_rollout(q, qd, tau, 1e-3, case["steps"])
            state["start"] = (q.clone(), qd.clone())
        return state
    robot = _robot(case)
    state["model"] = _model(robot)
    state["ee"] = robot.ee_link
    return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "mix":
        state["graph"].replay()
        return state["graph"].outputs
    if kind == "mix_rollout":
        state["q"].copy_(state["start"][0])
        state["qd"].copy_(state["start"][1])
        state["graph"].replay()
        return state["q"], state["qd"]
    m = state["model"]
    if kind == "step":
        return m.step_batched(*state["data"])
    if kind == "dynamics":
        return m.step_batched(*state["data"], ops=DYNAMICS)
    if kind == "forward":
        q, qd, _, tau = state["data"]
        return m.compute_forward_dynamics_batched(q, qd, tau)
    if kind == "passive":
        return m.compute_passive_force_batched(*state["data"])
    if kind == "ik":
        target, start = state["data"]
        return m.compute_inverse_kinematics_batched(state["ee"], target, start, eps=1e-4, max_iterations=case["steps"])
    if kind == "derivatives":
        q, qd, _, tau = state["data"]
        return autodiff.aba_derivatives(m, q, qd, tau)
    if kind == "gradient":
        q, qd, qdd, tau, w = state["data"]
        leaves = [t.detach().requires_grad_() for t in (q, qd, qdd, tau)]
        force = autodiff.inverse_dynamics(m, leaves[0], leaves[1], leaves[2])
        acc = autodiff.forward_dynamics(m, leaves[0], leaves[1], leaves[3])
        loss = (force * w).sum() + (acc * w).sum()
        return [force.detach(), acc.detach()] + list(torch.autograd.grad(loss, leaves))
    q, qd, tau, goal = state["data"]
    leaves = [t.detach().requires_grad_() for t in (q, qd, tau)]
    qT, qdT = autodiff.rollout(m, *leaves, dt=1e-3, checkpoint_every=20)
    loss = (qT.square()).sum() + (qdT * goal).sum()
    return [qT.detach(), qdT.detach()] + list(torch.autograd.grad(loss, leaves))


# ---- the work of a pass --------------------------------------------------------------
def work(case):
    """Bytes: inputs read once, outputs written once. Operations: a floor from the textbook
    recursions per joint (mass matrix entries, Newton-Euler, articulated bodies)."""
    n, kind = case["n"], case["kind"]

    def sizes(robot):
        depth = []  # ancestors of each column, itself included
        tree = _Tree(robot)
        for j in tree.moving:
            up, a = 0, j
            while a is not None:
                up += a["nv"]
                a = tree.above(a)
            depth += [up] * j["nv"]
        return robot.nq_ext, robot.nv, len(robot.link_names), sum(depth), len(tree.moving)

    def dyn(s):  # operations of M, inverse and forward dynamics on shared kinematics
        _, nv, _, pairs, nj = s
        return 700 * nj + 11 * pairs + pairs * pairs / max(nv, 1)

    if kind in ("mix", "mix_rollout"):
        robots, _, counts = _mix_parts(case)
        b = f = 0.0
        for r, c in zip(robots, counts):
            s = sizes(r)
            nq, nv = s[0], s[1]
            b += 8.0 * c * ((nq + 3 * nv) + (nv * nv + 2 * nv) if kind == "mix" else 2 * (nq + nv) + nv)
            f += c * case["steps"] * dyn(s)
        return {"bytes": b, "flops": f}
    s = sizes(_robot(case))
    nq, nv, nl, pairs, nj = s
    if kind == "step":
        return {"bytes": 8.0 * n * (nq + 3 * nv + 7 * nl + 6 * nv + nv * nv + 2 * nv), "flops": n * (dyn(s) + 60.0 * nl)}
    if kind == "dynamics":
        return {"bytes": 8.0 * n * (nq + 3 * nv + nv * nv + 2 * nv), "flops": n * dyn(s)}
    if kind == "forward":
        return {"bytes": 8.0 * n * (nq + 3 * nv), "flops": n * dyn(s)}
    if kind == "passive":
        return {"bytes": 4.0 * n * (nq + 2 * nv), "flops": n * 500.0 * nj}
    if kind == "gradient":
        return {"bytes": 8.0 * n * (nq + 4 * nv + 2 * nv + nq + 3 * nv), "flops": n * 3.0 * dyn(s)}
    if kind == "rollout":
        T = case["steps"]
        return {"bytes": 8.0 * n * (2 * T * nv + 3 * nq + 4 * nv), "flops": n * T * 4.0 * dyn(s)}
    if kind == "ik":
        return {"bytes": 8.0 * n * (7 + 2 * nq + 6) + n, "flops": n * case["steps"] * (150.0 * nj + 42.0 * nv + 500.0)}
    return {"bytes": 8.0 * n * (nq + 2 * nv + 3 * nv * nv), "flops": n * (dyn(s) + 30.0 * pairs + 6.0 * nv * pairs)}


# ---- the same results in plain torch ---------------------------------------------------
def _skew(w):
    z = torch.zeros_like(w[..., 0])
    x, y, t = w.unbind(-1)
    return torch.stack([z, -t, y, t, z, -x, -y, x, z], dim=-1).reshape(*w.shape[:-1], 3, 3)


def _rotation(quat):  # x y z w
    quat = quat / quat.norm(dim=-1, keepdim=True)
    K = _skew(quat[..., :3])
    return torch.eye(3, dtype=quat.dtype, device=quat.device) + 2 * quat[..., 3, None, None] * K + 2 * K @ K


def _quaternion(R):
    """w x y z, with w > 0 where the trace is, else the largest of x, y, z positive."""
    d = torch.diagonal(R, dim1=-2, dim2=-1)
    t = d.sum(-1, keepdim=True)
    sq = torch.cat([1 + t, 1 + 2 * d - t], dim=-1).clamp_min(0)  # 4 w^2, 4 x^2, ...
    i = torch.where(t[..., 0] > 0, torch.zeros_like(d[..., 0], dtype=torch.long), 1 + d.argmax(-1))
    a = R - R.transpose(-1, -2)
    s = R + R.transpose(-1, -2)
    rows = torch.stack([
        torch.stack([sq[..., 0], a[..., 2, 1], a[..., 0, 2], a[..., 1, 0]], -1),
        torch.stack([a[..., 2, 1], sq[..., 1], s[..., 0, 1], s[..., 0, 2]], -1),
        torch.stack([a[..., 0, 2], s[..., 0, 1], sq[..., 2], s[..., 1, 2]], -1),
        torch.stack([a[..., 1, 0], s[..., 0, 2], s[..., 1, 2], sq[..., 3]], -1)], dim=-2)
    row = torch.gather(rows, -2, i[..., None, None].expand(*i.shape, 1, 4)).squeeze(-2)
    return row / (2 * torch.gather(sq, -1, i[..., None]).sqrt())


def _floats(text):
    return torch.tensor([float(v) for v in text.split()], dtype=torch.float64)


def _placed(el):
    rpy, xyz = torch.zeros(3, dtype=torch.float64), torch.zeros(3, dtype=torch.float64)
    if el is not None:
        xyz, rpy = _floats(el.get("xyz", "0 0 0")), _floats(el.get("rpy", "0 0 0"))
    ex, ey, ez = torch.eye(3, dtype=torch.float64)
    m = lambda axis, a: torch.eye(3, dtype=axis.dtype) + torch.sin(a) * _skew(axis) + (1 - torch.cos(a)) * (  # noqa: E731
        _skew(axis) @ _skew(axis))
    return m(ez, rpy[2]) @ m(ey, rpy[1]) @ m(ex, rpy[0]), xyz


class _Tree:
    """The robot's URDF text as a list of joints, parents first; spatial quantities in the
    world frame, (linear, angular)."""

    def __init__(self, robot):
        root = ET.fromstring(robot.urdf)
        self.body = {}
        for l in root.findall("link"):
            el = l.find("inertial")
            if el is None:
                continue
            R, c = _placed(el.find("origin"))
            g = lambda k, e=el: float(e.find("inertia").get(k))  # noqa: E731
            I = torch.tensor([[g("ixx"), g("ixy"), g("ixz")], [g("ixy"), g("iyy"), g("iyz")],
                              [g("ixz"), g("iyz"), g("izz")]], dtype=torch.float64)
            self.body[l.get("name")] = (float(el.find("mass").get("value")), c, R @ I @ R.T)
        col = {}
        qc = vc = 0
        for name, kind in zip(robot.joint_names, robot.joint_kinds):
            col[name] = (qc, vc)
            qc, vc = qc + (7 if kind == "floating" else 1), vc + (6 if kind == "floating" else 1)
        todo = {}
        for j in root.findall("joint"):
            todo.setdefault(j.find("parent").get("link"), []).append(j)
        children = {j.find("child").get("link") for js in todo.values() for j in js}
        self.base = next(l.get("name") for l in root.findall("link") if l.get("name") not in children)
        self.joints, self.into, stack = [], {}, [self.base]
        while stack:
            at = stack.pop()
            for j in todo.get(at, []):
                R, p = _placed(j.find("origin"))
                axis = j.find("axis")
                kind, child = j.get("type"), j.find("child").get("link")
                J = {"kind": kind, "parent": at, "child": child, "R": R, "p": p,
                     "axis": _floats(axis.get("xyz")) if axis is not None else None,
                     "nv": {"fixed": 0, "floating": 6}.get(kind, 1), "col": col.get(j.get("name"))}
                self.joints.append(J)
                self.into[child] = J
                stack.append(child)
        self.moving = [J for J in self.joints if J["nv"]]
        self.links, self.nv = robot.link_names, robot.nv

    def above(self, J):
        """The moving joint next towards the base, or None."""
        J = self.into.get(J["parent"])
        while J is not None and not J["nv"]:
            J = self.into.get(J["parent"])
        return J

    def poses(self, q, twist=None):
        """{link: (R, p)}; `twist` [n, 6]: a first-order displacement of the floating base."""
        n, d = q.shape[0], dict(dtype=q.dtype, device=q.device)
        out = {self.base: (torch.eye(3, **d).expand(n, 3, 3), torch.zeros(n, 3, **d))}
        for J in self.joints:
            R, p = out[J["parent"]]
            p = p + R @ J["p"].to(**d)
            R = R @ J["R"].to(**d)
            if J["kind"] == "floating":
                c = J["col"][0]
                p = p + (R @ q[:, c : c + 3, None])[..., 0]
                R = R @ _rotation(q[:, c + 3 : c + 7])
                if twist is not None:
                    p = p + (R @ twist[:, :3, None])[..., 0]
                    R = R + R @ _skew(twist[:, 3:])
            elif J["kind"] == "prismatic":
                p = p + (R @ J["axis"].to(**d)) * q[:, J["col"][0], None]
            elif J["kind"] != "fixed":
                K = _skew(J["axis"].to(**d))
                x = q[:, J["col"][0], None, None]
                R = R @ (torch.eye(3, **d) + torch.sin(x) * K + (1 - torch.cos(x)) * (K @ K))
            out[J["child"]] = (R, p)
        return out

    def columns(self, J, pose):
        """The joint's motion subspace, [n, 6, nv]."""
        R, p = pose
        if J["kind"] == "floating":
            w = R
            zero = torch.zeros_like(R)
            return torch.cat([torch.cat([R, _skew(p) @ w], -1), torch.cat([zero, w], -1)], -2)
        u = (R @ J["axis"].to(R))[..., None]
        if J["kind"] == "prismatic":
            return torch.cat([u, torch.zeros_like(u)], -2)
        return torch.cat([_skew(p) @ u, u], -2)

    def jacobian(self, q, poses=None):
        poses = poses or self.poses(q)
        S = torch.zeros(q.shape[0], 6, self.nv, dtype=q.dtype, device=q.device)
        for J in self.moving:
            S[:, :, J["col"][1] : J["col"][1] + J["nv"]] = self.columns(J, poses[J["child"]])
        return S

    def inertias(self, poses):
        """{link: 6x6 world inertia}"""
        out = {}
        for name, (m, c, I) in self.body.items():
            if name == self.base:
                continue
            R, p = poses[name]
            C = _skew(p + R @ c.to(p))
            one = m * torch.eye(3, dtype=p.dtype, device=p.device).expand_as(R)
            Iw = R @ I.to(R) @ R.transpose(-1, -2) - m * C @ C
            out[name] = torch.cat([torch.cat([one, -m * C], -1), torch.cat([m * C, Iw], -1)], -2)
        return out

    def dynamics(self, q, qd, qdd, twist=None, mass=True):
        """(M, inverse dynamics) by composite inertias and Newton-Euler."""
        poses = self.poses(q, twist)
        Y = self.inertias(poses)
        zero = torch.zeros(q.shape[0], 6, dtype=q.dtype, device=q.device)
        g = zero.clone()
        g[:, :3] = -torch.tensor(GRAVITY, dtype=q.dtype, device=q.device)
        v, a, cols = {self.base: zero}, {self.base: g}, {}
        X = lambda x: torch.cat([torch.cat([_skew(x[:, 3:]), _skew(x[:, :3])], -1),  # noqa: E731
                                 torch.cat([torch.zeros_like(_skew(x[:, 3:])), _skew(x[:, 3:])], -1)], -2)
        f, comp = {}, {}
        for J in self.joints:
            at, up = J["child"], J["parent"]
            v[at], a[at] = v[up], a[up]
            if J["nv"]:
                c = slice(J["col"][1], J["col"][1] + J["nv"])
                S = cols[at] = self.columns(J, poses[at])
                vj = (S @ qd[:, c, None])[..., 0]
                v[at] = v[up] + vj
                a[at] = a[up] + (S @ qdd[:, c, None])[..., 0] + (X(v[at]) @ vj[..., None])[..., 0]
            if at in Y:
                h = Y[at] @ v[at][..., None]
                f[at] = (Y[at] @ a[at][..., None] - X(v[at]).transpose(-1, -2) @ h)[..., 0]
                comp[at] = Y[at]
        M = torch.zeros(q.shape[0], self.nv, self.nv, dtype=q.dtype, device=q.device) if mass else None
        tau = [None] * self.nv
        for J in reversed(self.joints):
            at, up = J["child"], J["parent"]
            if J["nv"]:
                c = J["col"][1]
                t = (cols[at].transpose(-1, -2) @ f.get(at, zero)[..., None])[..., 0]
                for k in range(J["nv"]):
                    tau[c + k] = t[:, k]
                if mass and at in comp:
                    F, A = comp[at] @ cols[at], J
                    while A is not None:
                        r = slice(A["col"][1], A["col"][1] + A["nv"])
                        B = cols[A["child"]].transpose(-1, -2) @ F
                        M[:, r, c : c + J["nv"]] = B
                        M[:, c : c + J["nv"], r] = B.transpose(-1, -2)
                        A = self.above(A)
            if at in f and up != self.base:
                f[up] = f[up] + f[at] if up in f else f[at]
                comp[up] = comp[up] + comp[at] if up in comp else comp[at]
        return M, torch.stack(tau, -1)

    def forward(self, q, qd, tau):
        M, h = self.dynamics(q, qd, torch.zeros_like(qd))
        return torch.linalg.solve(M, (tau - h)[..., None])[..., 0]

    def advance(self, q, v):
        """q moved by the velocity displacement v."""
        out = list(q.unbind(-1))
        for J in self.moving:
            c, w = J["col"]
            if J["kind"] != "floating":
                out[c] = out[c] + v[:, w]
                continue
            R = _rotation(q[:, c + 3 : c + 7])
            A = torch.zeros(q.shape[0], 4, 4, dtype=q.dtype, device=q.device)
            A = torch.cat([torch.cat([_skew(v[:, w + 3 : w + 6]), v[:, w : w + 3, None]], -1), A[:, 3:]], -2)
            E = torch.matrix_exp(A)
            p = q[:, c : c + 3] + (R @ E[:, :3, 3:])[..., 0]
            t = _quaternion(R @ E[:, :3, :3])[:, [1, 2, 3, 0]]
            t = torch.where((t * q[:, c + 3 : c + 7]).sum(-1, keepdim=True) < 0, -t, t)
            for k in range(3):
                out[c + k] = p[:, k]
            for k in range(4):
                out[c + 3 + k] = t[:, k]
        return torch.stack(out, -1)


def _log(R):
    quat = _quaternion(R)
    quat = torch.where(quat[:, :1] < 0, -quat, quat)
    s = quat[:, 1:].norm(dim=-1)
    t = 2 * torch.atan2(s, quat[:, 0])
    k = torch.where(s > 1e-12, t / s.clamp_min(1e-300), 2 * torch.ones_like(s))
    return quat[:, 1:] * k[:, None], t


def _log6(R, p):
    """(linear, angular) logarithm of a placement."""
    w, t = _log(R)
    small = t < 0.02
    ts = torch.where(small, torch.ones_like(t), t)
    beta = torch.where(small, 1 / 12 + t * t / 720 + t**4 / 30240, (1 - ts / 2 / torch.tan(ts / 2)) / ts**2)
    K = _skew(w)
    v = p - 0.5 * (K @ p[..., None])[..., 0] + beta[:, None] * ((K @ K) @ p[..., None])[..., 0]
    return torch.cat([v, w], -1)


_BERNOULLI = [1.0, 0.5, 1 / 6, 0.0, -1 / 30, 0.0, 1 / 42, 0.0, -1 / 30, 0.0, 5 / 66, 0.0, -691 / 2730, 0.0, 7 / 6, 0.0,
              -3617 / 510, 0.0, 43867 / 798, 0.0, -174611 / 330, 0.0, 854513 / 138]


def _jlog6(xi):
    """Inverse of the right Jacobian of SE(3) at xi: closed form of the series
    x / (1 - exp(-x)) in the adjoint of xi, by its eigenvalues 0 and +- i t (each double)."""
    n = xi.shape[0]
    v, w = xi[:, :3], xi[:, 3:]
    A = torch.zeros(n, 6, 6, dtype=xi.dtype, device=xi.device)
    A[:, :3, :3] = A[:, 3:, 3:] = _skew(w)
    A[:, :3, 3:] = _skew(v)
    t = w.norm(dim=-1)
    small = t < 0.5
    ts = torch.where(small, torch.ones_like(t), t)
    # x / (1 - exp(-x)) = 1 + x / 2 + c1 x^2 + c2 x^4 on the minimal polynomial x (x^2 + t^2)^2;
    # h(t) = (t / 2) cot(t / 2): 1 - c1 t^2 + c2 t^4 = h and -2 c1 t + 4 c2 t^3 = h'
    h = ts / 2 / torch.tan(ts / 2)
    dh = 0.5 / torch.tan(ts / 2) - ts / 4 / torch.sin(ts / 2) ** 2
    c2 = (ts * dh - 2 * (h - 1)) / (2 * ts**4)
    c1 = (1 - h) / ts**2 + c2 * ts**2
    eye = torch.eye(6, dtype=xi.dtype, device=xi.device).expand(n, 6, 6)
    A2 = A @ A
    J = eye + 0.5 * A + c1[:, None, None] * A2 + c2[:, None, None] * (A2 @ A2)
    series, P = eye + 0.5 * A, A2
    for k in range(2, 22, 2):
        series = series + (_BERNOULLI[k] / math.factorial(k)) * P
        P = P @ A2
    return torch.where(small[:, None, None], series, J)


def _exact_ik(robot, target, start, iterations, eps=1e-4, dt=0.1, damp=1e-6):
    tree = _Tree(robot)
    ee = tree.links[robot.ee_link]
    J = tree.into[ee]
    while not J["nv"]:
        J = tree.into[J["parent"]]
    chain, A = [], J
    while A is not None:
        chain.append(A["col"][1])
        A = tree.above(A)
    q = start.clone()
    n, d = q.shape[0], dict(dtype=q.dtype, device=q.device)
    Rt, pt = _rotation(target[:, [4, 5, 6, 3]]), target[:, :3]
    at = tree.poses(q)
    (Rj, pj), (Rl, pl) = at[J["child"]], at[ee]
    Rjl, pjl = Rj.transpose(-1, -2) @ Rl, (Rj.transpose(-1, -2) @ (pl - pj)[..., None])[..., 0]
    Rd = Rt @ Rjl.transpose(-1, -2)
    pd = pt - (Rd @ pjl[..., None])[..., 0]
    best, best_err, least = q.clone(), torch.zeros(n, 6, **d), torch.full((n,), 1e10, **d)
    done = torch.zeros(n, dtype=torch.bool, device=q.device)
    mask = torch.zeros(tree.nv, **d)
    mask[chain] = 1
    for it in range(iterations + 1):
        poses = tree.poses(q)
        R, p = poses[J["child"]]
        Rt_ = R.transpose(-1, -2)
        err = _log6(Rt_ @ Rd, (Rt_ @ (pd - p)[..., None])[..., 0])
        size = err.norm(dim=-1)
        new = (size < least) & ~done
        least, best, best_err = torch.where(new, size, least), torch.where(new[:, None], q, best), torch.where(new[:, None], err, best_err)
        done = done | (size < eps)
        if it == iterations or bool(done.all()):
            break
        S = tree.jacobian(q, poses) * mask
        lin = Rt_ @ (S[:, :3] - _skew(p) @ S[:, 3:])
        Jl = -_jlog6(-err) @ torch.cat([lin, Rt_ @ S[:, 3:]], -2)
        A = Jl @ Jl.transpose(-1, -2) + damp * torch.eye(6, **d)
        v = -(Jl.transpose(-1, -2) @ torch.linalg.solve(A, err[..., None]))[..., 0]
        q = torch.where(done[:, None], q, q + dt * v)
    return best, done, best_err


def _exact_chunk(case, robot, data):
    kind = case["kind"]
    tree = _Tree(robot)
    if kind in ("step", "dynamics", "forward"):
        q, qd, qdd, tau = data
        acc = tree.forward(q, qd, tau)
        if kind == "forward":
            return acc
        M, force = tree.dynamics(q, qd, qdd)
        out = {"mass_matrix": M, "qf": force, "qacc": acc}
        if kind == "step":
            poses = tree.poses(q)
            out["jacobian"] = tree.jacobian(q, poses)
            out["link_poses"] = torch.stack([torch.cat([poses[l][1], _quaternion(poses[l][0])], -1) for l in tree.links], 1)
        return out
    if kind == "passive":
        q, qd = (t.double()[:, : robot.nv] for t in data)
        force = tree.dynamics(q, qd, torch.zeros_like(qd), mass=False)[1]
        return torch.cat([force, torch.zeros(q.shape[0], 3, dtype=force.dtype, device=q.device)], 1)
    if kind == "gradient":
        q, qd, qdd, tau, w = data
        leaves = [t.clone().requires_grad_() for t in (q, qd, qdd, tau)]
        force = tree.dynamics(*leaves[:3], mass=False)[1]
        acc = tree.forward(leaves[0], leaves[1], leaves[3])
        return [force.detach(), acc.detach()] + list(torch.autograd.grad((force * w).sum() + (acc * w).sum(), leaves))
    if kind == "derivatives":
        q, qd, _, tau = data
        acc = tree.forward(q, qd, tau)
        base = any(k == "floating" for k in robot.joint_kinds)
        shift = torch.zeros(q.shape[0], 6, dtype=q.dtype, device=q.device, requires_grad=True) if base else None
        x, v = q.clone().requires_grad_(), qd.clone().requires_grad_()
        force = tree.dynamics(x, v, acc, shift, mass=False)[1]
        rows_q, rows_v = [], []
        for i in range(robot.nv):
            g = torch.autograd.grad(force[:, i].sum(), [x, v] + ([shift] if base else []), retain_graph=True)
            cols = torch.zeros_like(qd)
            for J in tree.moving:
                c, w = J["col"]
                cols[:, w : w + J["nv"]] = g[2] if J["kind"] == "floating" else g[0][:, c : c + 1]
            rows_q.append(cols)
            rows_v.append(g[1])
        Mi = torch.linalg.inv(tree.dynamics(q, qd, acc)[0])
        return [-Mi @ torch.stack(rows_q, 1), -Mi @ torch.stack(rows_v, 1), Mi]
    q, qd, tau, goal = data  # rollout
    leaves = [t.clone().requires_grad_() for t in (q, qd, tau)]
    x, v = leaves[0], leaves[1]
    for t in range(case["steps"]):
        v = v + 1e-3 * tree.forward(x, v, leaves[2][t])
        x = tree.advance(x, 1e-3 * v)
    grads = torch.autograd.grad(x.square().sum() + (v * goal).sum(), leaves)
    return [x.detach(), v.detach()] + list(grads)


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "rollout" and (case["steps"] > 20 or case["robot"] == "quadruped18"):
        return None  # a graph of many steps in plain torch takes too long
    dev = _device()
    data = _inputs(case, seed, dev)
    if kind in ("mix", "mix_rollout"):
        if kind == "mix_rollout":
            return None
        robots, model_of_env, _ = _mix_parts(case)
        width = max(r.nv for r in robots)
        out = {k: torch.zeros(n, c, dtype=torch.float64, device=dev)
               for k, c in (("mass_matrix", width * width), ("qacc", width), ("qf", width))}
        for k, (r, d) in enumerate(zip(robots, data)):
            rows = torch.as_tensor(np.nonzero(model_of_env == k)[0], device=dev)
            if not len(rows):
                continue
            part = _exact_chunk({"kind": "dynamics"}, r, d)
            out["mass_matrix"][rows, : r.nv * r.nv] = part["mass_matrix"].reshape(len(rows), -1)
            out["qacc"][rows, : r.nv], out["qf"][rows, : r.nv] = part["qacc"], part["qf"]
        return out
    robot = _robot(case)
    if kind == "ik":
        target, start = data
        q, ok, err = _exact_ik(robot, target, start, case["steps"])
        return q, None, err
    if kind in ("rollout",):
        return _exact_chunk(case, robot, data)
    step = 2048 if kind == "derivatives" else 16384  # bounds the memory of the intermediate tensors
    parts = [_exact_chunk(case, robot, tuple(t[i : i + step] for t in data)) for i in range(0, n, step)]
    if isinstance(parts[0], dict):
        return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    if isinstance(parts[0], torch.Tensor):
        return torch.cat(parts)
    return [torch.cat(p) for p in zip(*parts)]
