"""Clouds whose squared distances come close to the largest double."""
import numpy as np
import pytest

import oracle
import pacman_b200 as pacman
from pacman_b200 import workloads as W
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# The transfer's specified tolerances (tests/test_gpu_parity.py).
TOL = {"fp64": 1e-12, "mixed": 1e-10}


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("exponent", [100, 470, 500])
def test_large_coordinates(exponent, precision):
    # Uniform: the register kernel; refined: the tiled engine too.
    s = 2.0 ** exponent
    rng = np.random.default_rng(1)
    refined = W.make("grid_blobs_1m", scale=0.005)
    for S, T in ((rng.random((3000, 3)), rng.random((2000, 3))), (refined["src"], refined["tgt"])):
        v = W.franke_3d(S)
        plan = pacman.rbf.Plan(3, S * s, T * s, support_radius=0.1 * s, precision=precision)
        out = plan.execute(0x11, v)
        ref = oracle.interpolate(3, 0x11, S * s, v, T * s, support_radius=0.1 * s)
        assert rel_l2(out, ref) <= TOL[precision]
        assert not (plan.patch_status() & (2 | 4 | 8 | 16)).any()
        plan.close()
