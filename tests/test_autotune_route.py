"""The tuner times the FP64 kernels that its settings belong to, whichever kernels the batch runs
otherwise, and leaves the batch's own choice as it was."""
import json

import pytest

from sapien_gb300 import autotune
from test_autotune_logic import FakeBatch, FakeModel, cost


class RoutedBatch(FakeBatch):
    fp64 = False
    steps = ()

    def set_fp64(self, on):
        self.fp64 = on

    def step(self, *args):
        self.steps += (self.fp64,)


@pytest.fixture
def routed(monkeypatch, tmp_path):
    batch = RoutedBatch([FakeModel(6, 7), FakeModel(18, 14), FakeModel(35, 31)], [10, 6, 4])

    def fake_time(fn, reps=5):
        fn()
        # the block sweep takes the same time whatever the settings
        return cost(batch) if batch.fp64 else 1.0

    monkeypatch.setattr(autotune, "_time", fake_time)
    monkeypatch.setenv("SGDYN_AUTOTUNE_CACHE", str(tmp_path))
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda dev=None: "fake-gpu")
    return batch, tmp_path


@pytest.mark.parametrize("choice", [False, True])
def test_tuner_times_the_fp64_kernels(routed, choice):
    batch, tmp_path = routed
    batch.set_fp64(choice)
    shape, _ = autotune.tune_batch(batch, None, None, None, None, ops=28)
    assert tuple(shape) == (2, 2, 0) and batch.lanes == [1, 2, 4]
    assert all(batch.steps) and batch.fp64 is choice
    # not under the key of entries that were timed on the batch's own route
    (key,) = json.load(open(tmp_path / "autotune.json"))
    assert key.endswith("|fp64")


def test_choice_is_restored_when_a_step_fails(routed, monkeypatch):
    batch, _ = routed

    def broken(fn, reps=5):
        raise RuntimeError("launch failed")

    monkeypatch.setattr(autotune, "_time", broken)
    with pytest.raises(RuntimeError, match="launch failed"):
        autotune.tune_batch(batch, None, None, None, None, ops=28)
    assert batch.fp64 is False


@pytest.mark.gpu
def test_batch_route():
    """A batch's own FP64 choice: the bits of the process-wide one, for this batch alone."""
    import torch

    from sapien_gb300.hetero import OPS_DYNAMICS
    from test_bfp_gpu import fp64_route
    from test_hetero_gpu import setup, valid_blocks

    batch, _, _, args = setup(n=120, seed=4)
    other, _, _, _ = setup(n=120, seed=4)
    auto = valid_blocks(batch, batch.step(*args, OPS_DYNAMICS))
    assert batch.block_sweep and not batch.fp64
    with fp64_route():
        assert not batch.block_sweep and not batch.fp64
        want = valid_blocks(batch, batch.step(*args, OPS_DYNAMICS))
    batch.set_fp64(True)
    assert batch.fp64 and not batch.block_sweep and other.block_sweep
    got = valid_blocks(batch, batch.step(*args, OPS_DYNAMICS))
    same = valid_blocks(other, other.step(*args, OPS_DYNAMICS))
    batch.set_fp64(False)
    back = valid_blocks(batch, batch.step(*args, OPS_DYNAMICS))
    for a, b, c, d, e in zip(auto, want, got, same, back):
        assert torch.equal(b, c) and torch.equal(a, d) and torch.equal(a, e)
    assert not all(torch.equal(a, b) for a, b in zip(auto, want))
