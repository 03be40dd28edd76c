"""Calls from several threads at once share the idle streams, events and pinned
blocks of the library: each gives what it gives alone, with more plans alive than
sets of streams are kept idle, and with calls that fail among them."""
import threading

import numpy as np
import pytest

import pacman_b200 as pacman
from pacman_b200 import workloads as W

pytestmark = pytest.mark.gpu

CUDA = pacman.execspaces.CUDA
RNG = np.random.default_rng(6)
UNIFORM = (RNG.random((4000, 3)), RNG.random((3000, 3)))
_CLOUD = W.make("grid_blobs_1m", scale=0.005)
REFINED = (_CLOUD["src"], _CLOUD["tgt"])


def _values(S):
    return np.sin(S @ [3.0, 2.0, 1.0])


def _transfer(points, precision):
    S, T = points
    return pacman.rbf.interpolate(3, CUDA, 0x11, S, _values(S), T, precision=precision)


def _kept(points):
    S, T = points
    plan = pacman.rbf.Plan(3, S, T, precision="mixed")
    plan.execute(0x11, np.cos(S[:, 0]), keep_factors=True)
    out = plan.execute(0x11, _values(S), keep_factors=True)
    plan.close()
    return out


def _gradient(points):
    S, T = points
    plan = pacman.rbf.Plan(3, S, T)
    out = plan.execute(0x11, _values(S), save_for_adjoint=True)
    gv, gt = plan.adjoint(out)
    plan.close()
    return np.concatenate([out, gv, gt.ravel()])


def _batch():
    probs = [(3, 0x11, S, _values(S), T) for S, T in (UNIFORM, REFINED, UNIFORM)]
    return np.concatenate(pacman.rbf.interpolate_batch(probs, precision="mixed"))


def _fails():
    with pytest.raises(RuntimeError):
        pacman.rbf.interpolate(3, CUDA, 0x11, np.ones((50, 3)), np.ones(50), UNIFORM[1])
    return np.zeros(1)


JOBS = [lambda: _transfer(UNIFORM, "fp64"), lambda: _transfer(REFINED, "mixed"),
        lambda: _transfer(REFINED, "fp64"), lambda: _kept(UNIFORM), lambda: _kept(REFINED),
        lambda: _gradient(REFINED), _batch, _fails]


def test_threads_share_the_library():
    want = [job() for job in JOBS]
    wrong = []

    def work(first):
        for turn in range(6):
            i = (first + turn) % len(JOBS)
            try:
                if not np.array_equal(JOBS[i](), want[i]):
                    wrong.append(i)
            except Exception as e:  # noqa: BLE001 - reported by the test's thread
                wrong.append((i, repr(e)))
    for _ in range(2):  # new threads take over what the first ones left
        threads = [threading.Thread(target=work, args=(k,)) for k in range(10)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not wrong
