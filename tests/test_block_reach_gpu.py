"""Calls at the edges of the block sweeps' reach."""
import ctypes

import pytest

from sapien_gb300 import _native as N
from test_bfp_gpu import ROBOTS, cuda, pair

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
