"""Launches of one kernel for models of different size: the shared memory of each is its own."""
import ctypes
import threading

import pytest

from sapien_gb300 import synthetic as syn
from sapien_gb300 import _native as N
from test_bfp_gpu import cuda, pair

pytestmark = pytest.mark.gpu

ENVS = 9800  # 32 environments per block


def arms():
    """Arms whose blocks take 70 and 105 KB in one kernel, with inputs."""
    return [(pair(r)[0], cuda(*r.sample(ENVS, seed=k)))
            for k, r in enumerate((syn.serial_chain(6, seed=4), syn.arm_with_fingers()))]


def test_threads_with_blocks_of_different_size():
    """Eight host threads, some thousand calls each on a stream of their own: all succeed and give
    the first call's bits."""
    import torch

    step, errors, gate = N.load().sgdyn_step, [], threading.Barrier(8)
    work = [(pm, ins[0], pm.step_batched(*ins, ops=N.OP_JACOBIAN)["jacobian"]) for pm, ins in arms()]
    outs = [torch.empty_like(work[k % 2][2]) for k in range(8)]
    streams = [torch.cuda.Stream() for _ in range(8)]
    torch.cuda.synchronize()

    def run(k):
        pm, q, _ = work[k % 2]
        args = (pm._h, ENVS, N.OP_JACOBIAN, ctypes.c_void_p(q.data_ptr()), None, None, None, None,
                ctypes.c_void_p(outs[k].data_ptr()), None, None, None, N.ENV_MAJOR,
                ctypes.c_void_p(streams[k].cuda_stream))
        torch.cuda.set_device(0)
        gate.wait()
        for _ in range(4000):
            if step(*args) != N.OK:
                errors.append(N.last_error())
                return

    threads = [threading.Thread(target=run, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for k in range(8):
        assert torch.equal(outs[k], work[k % 2][2])


def test_smaller_model_between_capture_and_instantiation():
    """A captured step of the larger arm, a call for the smaller one before the graph is complete."""
    import torch

    (small, a), (large, b) = arms()
    want = [large.step_batched(*b, ops=N.OP_JACOBIAN)["jacobian"], small.step_batched(*a, ops=N.OP_JACOBIAN)["jacobian"]]
    torch.cuda.synchronize()
    g, stream, other = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="relaxed")
        out = large.step_batched(*b, ops=N.OP_JACOBIAN)["jacobian"]
        with torch.cuda.stream(other):
            got = small.step_batched(*a, ops=N.OP_JACOBIAN)["jacobian"]
        g.capture_end()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0]) and torch.equal(got, want[1])
