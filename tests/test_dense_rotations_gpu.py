"""Small results among dense rotations, where FP64's terms are rounded as well: the block sweep keeps
them to FP64's error of the terms, without going through FP64."""
import numpy as np
import pytest

from sapien_gb300 import PinocchioModel, _native as N
from test_bfp_gpu import cuda, fp64_route, host
from test_near_equilibrium_gpu import G, SMALL, link

pytestmark = pytest.mark.gpu


def test_pendulum_about_a_dense_axis_at_its_equilibrium():
    pm = PinocchioModel('<robot name="r">' + link("base") + link("bob", (0.1, -0.2, -0.45))
                        + '<joint name="a" type="continuous"><origin xyz="0.1 0.2 0.3" rpy="0.3 0.7 -1.1"/>'
                          '<parent link="base"/><child link="bob"/><axis xyz="0.48 0.6 0.64"/></joint></robot>',
                        [0, 0, -G])
    pm.set_joint_order(["a"])
    pm.set_link_order(["base", "bob"])

    def torque(q):
        z = np.zeros((len(q), 1))
        return host(pm.step_batched(*cuda(q.reshape(-1, 1), z, z, z), ops=N.OP_INVERSE_DYNAMICS))["qf"][:, 0]

    with fp64_route():
        grid = np.linspace(-3, 3, 601)
        scale = np.abs(torque(grid)).max()
        assert scale > 0.1
        lo, hi = min((p for p in zip(grid[:-1], grid[1:]) if np.prod(torque(np.array(p))) < 0))
        for _ in range(60):
            mid = (lo + hi) / 2
            lo, hi = (mid, hi) if np.prod(torque(np.array([lo, mid]))) > 0 else (lo, mid)
        q = np.concatenate([hi + SMALL, [hi]])
        want = torque(q)
    # some 40 roundings in FP64, of terms that are the link's weight times its distance from the origin
    terms = 1.3 * G * (0.45 + 0.5)
    assert np.abs(torque(q) - want).max() <= 40 * 2.0**-53 * terms
