"""Calls on the library's own stream and the work queued on the default stream:
calls on host arrays do not wait for it."""
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
