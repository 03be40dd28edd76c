"""Calls that fail give their stream back and leave the library usable."""
import ctypes

import numpy as np
import pytest

import oracle
import pacman_b200 as pacman

pytestmark = pytest.mark.gpu

CUDA = pacman.execspaces.CUDA


def _stream_id():
    # The runtime numbers streams as they are created.
    rt = ctypes.CDLL("libcudart.so.12")
    handle, number = ctypes.c_void_p(), ctypes.c_ulonglong()
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(handle), 1) == 0
    assert rt.cudaStreamGetId(handle, ctypes.byref(number)) == 0
    assert rt.cudaStreamDestroy(handle) == 0
    return number.value


def _fails(call):
    with pytest.raises(RuntimeError, match="degenerate"):
        call()


def test_streams_come_back():
    pytest.importorskip("torch")  # brings the runtime library
    same = np.ones((40, 3))  # every source in one place: no patch radius
    rng = np.random.default_rng(1)
    S, T = rng.random((2000, 3)), rng.random((1500, 3))
    v = np.sin(S @ [3, 2, 1])
    calls = (lambda: pacman.rbf.interpolate(3, CUDA, 0x11, same, np.ones(40), T),
             lambda: pacman.rbf.Plan(3, same, T),
             lambda: pacman.rbf.interpolate_batch([(3, 0x11, S, v, T),
                                                   (3, 0x11, same, np.ones(40), T)]))
    ref = oracle.interpolate(3, 0x11, S, v, T)
    for call in calls:
        _fails(call)
        before = _stream_id()
        for _ in range(30):
            _fails(call)
        assert _stream_id() - before < 10
        out = pacman.rbf.interpolate(3, CUDA, 0x11, S, v, T)
        assert np.linalg.norm(out - ref) <= 1e-12 * np.linalg.norm(ref)
