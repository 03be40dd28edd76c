"""Which solver takes a patch of a batch (precision mixed) depends on its own
problem alone: the members of a batch are solved as their single calls, to the
bit where the field counts agree."""
import numpy as np
import pytest

import pacman_b200 as pacman
from pacman_b200 import workloads as W

pytestmark = pytest.mark.gpu

CUDA = pacman.execspaces.CUDA
BASIS = 0x12


def _largest(S, T):
    plan = pacman.rbf.Plan(3, S, T, precision="mixed")
    n = np.diff(plan.patch_lists("source")[0])
    plan.close()
    return n.max()


@pytest.mark.parametrize("order", [(0, 1), (1, 0), (0, 2, 1), (1, 0, 1, 0)])
def test_members_are_solved_as_single_calls(order):
    # Uniform: patches up to 65..96 sources, all in the register kernel.  Refined:
    # some above 96, so those above 64 go to the tiled engine.
    rng = np.random.default_rng(3)
    S, T = rng.random((20000, 3)), rng.random((4000, 3))
    refined = W.make("grid_blobs_1m", scale=0.01)
    assert 64 < _largest(S, T) <= 96
    assert _largest(refined["src"], refined["tgt"]) > 96
    def fields(p):
        return np.stack([W.franke_3d(p), np.cos(3.0 * p[:, 0] + p[:, 2])], axis=1)
    pool = [(3, BASIS, S, fields(S), T),
            (3, BASIS, refined["src"], fields(refined["src"]), refined["tgt"]),
            (3, BASIS, S, fields(S), T[:0])]
    outs = pacman.rbf.interpolate_batch([pool[i] for i in order], precision="mixed")
    for i, out in zip(order, outs):
        dim, basis, P, v, Y = pool[i]
        one = pacman.rbf.interpolate(dim, CUDA, basis, P, v, Y, precision="mixed")
        assert np.array_equal(out, one), i
