"""Calls on the library's own stream and the work queued on the caller's: calls on
host arrays do not wait for the default stream, calls on device tensors run
after what torch has queued on its current stream."""
import numpy as np
import pytest

import pacman
import pacman_b200

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CUDA = pacman_b200.execspaces.CUDA
RNG = np.random.default_rng(8)
S, T = RNG.random((3000, 3)), RNG.random((2000, 3))
V = np.sin(S @ [3, 2, 1])


def _transfer():
    return pacman_b200.rbf.interpolate(3, CUDA, 0x11, S, V, T)


def _batch():
    return pacman_b200.rbf.interpolate_batch([(3, 0x11, S, V, T)] * 3)[2]


def _nearest():
    return pacman_b200.fe.interpolate(3, CUDA, pacman_b200.fe.methods.NEAREST_NEAREST, S, V,
                                      None, None, None, T)[0]


def _mls():
    return pacman.MLS.interpolate(3, CUDA, S, V, T)


@pytest.mark.parametrize("call", [_transfer, _batch, _nearest, _mls])
def test_host_arrays_do_not_wait(call):
    want = call()  # also brings what is allocated once
    torch.cuda.synchronize()
    torch.cuda._sleep(1_500_000_000)  # the better part of a second
    after = torch.cuda.Event()
    after.record()
    got = call()
    waited = after.query()
    torch.cuda.synchronize()
    assert not waited
    assert np.array_equal(got, want)


def _gpu(*arrays):
    return [torch.tensor(a, device="cuda") for a in arrays]


@pytest.mark.parametrize("side", [False, True])
def test_plan_waits_for_device_tensors(side):
    grad = RNG.standard_normal(len(T))
    plan = pacman_b200.rbf.Plan(3, S, T)
    want = plan.execute(0x11, V, save_for_adjoint=True)
    want_v, want_t = plan.adjoint(grad)
    final = _gpu(S, T, V, grad)
    sources, targets, values, upstream = early = _gpu(
        RNG.random(S.shape), RNG.random(T.shape), np.zeros(len(S)), np.zeros(len(T)))
    stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
    torch.cuda.synchronize()

    def late(*which):
        torch.cuda._sleep(50_000_000)  # some 25 ms
        for i in which:
            early[i].copy_(final[i])
    with torch.cuda.stream(stream):
        late(0, 1)
        plan = pacman_b200.rbf.Plan(3, sources, targets)
        late(2)
        out = plan.execute(0x11, values, save_for_adjoint=True)
        late(3)
        gv, gt = plan.adjoint(upstream)
        out, gv, gt = (x.cpu().numpy() for x in (out, gv, gt))
    assert np.array_equal(out, want)
    assert np.array_equal(gv, want_v) and np.array_equal(gt, want_t)
