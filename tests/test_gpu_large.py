"""Tiled-engine patches whose size sits at the edges of the 64-row tiles, of the
row pairs of the int8 step and of the clusters that sweep long slots, against
the CPU oracle: forward in both precisions and kept factors, and the adjoint."""
import functools

import numpy as np
import pytest

import oracle
import pacman_b200 as pacman
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# The transfer's specified tolerances (tests/test_gpu_parity.py).
TOL = {"fp64": 1e-12, "mixed": 1e-10}
SIZES = [65, 128, 129, 192, 193, 256, 257, 704, 705, 1984, 1985, 2048, 2049]


def _problem(n, fields):
    # Nearly every patch holds the whole cloud: nodes_per_cluster = n.
    rng = np.random.default_rng(n)
    S, T = rng.random((n, 3)), rng.random((70, 3))
    x = S @ np.array([2.0, 1.0, 3.0])
    v = np.stack([np.sin(x + f) for f in range(fields)], axis=1)
    return S, T, v


@functools.lru_cache(maxsize=1)
def _reference(n):
    S, T, v = _problem(n, 8)
    return oracle.interpolate(3, 0x11, S, v, T, n)


@pytest.mark.parametrize("fields", [1, 3, 8])
@pytest.mark.parametrize("n", SIZES)
def test_sizes_match_oracle(n, fields, monkeypatch):
    monkeypatch.setenv("PACMAN_B200_BIG_N", "8")
    S, T, v = _problem(n, fields)
    ref = _reference(n)
    for precision, tol in TOL.items():
        plan = pacman.rbf.Plan(3, S, T, nodes_per_cluster=n, precision=precision)
        assert np.diff(plan.patch_lists("source")[0]).max() == n
        for keep in (False, True, True):  # plain, factoring, from the kept factors
            out = plan.execute(0x11, v, keep_factors=keep)
            for f in range(fields):
                assert rel_l2(out[:, f], ref[:, f]) <= tol, (precision, keep, f)
        assert not (plan.patch_status() & (2 | 4 | 8 | 16)).any()


@pytest.mark.parametrize("n", SIZES)
def test_adjoint_is_the_transpose(n, monkeypatch):
    monkeypatch.setenv("PACMAN_B200_BIG_N", "8")
    S, T, v = _problem(n, 2)
    G = np.random.default_rng(1).standard_normal((len(T), 2))
    plan = pacman.rbf.Plan(3, S, T, nodes_per_cluster=n)
    out = plan.execute(0x11, v, save_for_adjoint=True)
    gv, _ = plan.adjoint(G, targets=False)
    scale = np.linalg.norm(out) * np.linalg.norm(G) + np.linalg.norm(v) * np.linalg.norm(gv)
    assert abs((G * out).sum() - (v * gv).sum()) <= 1e-11 * scale
