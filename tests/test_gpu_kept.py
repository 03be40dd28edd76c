"""Kept factors of the register kernel's widest class (65 to 96 sources), where
no patch of the plan is larger: three warps take part in the substitutions.
Every execute from the kept factors against the CPU oracle and a fresh plan."""
import numpy as np
import pytest

import oracle
import pacman_b200 as pacman
from pacman_b200 import workloads as W
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# The transfer's specified tolerance, and the one of tests/test_gpu_factors.py
# between kept and fresh factors.
TOL_MIXED = 1e-10
TOL_REUSE = 1e-12


def _fields(S, count, seed):
    k = np.random.default_rng(seed).uniform(1.0, 4.0, size=(count, S.shape[1]))
    return np.stack([np.sin(S @ k[f]) + 0.3 * f for f in range(count)], axis=1)


def _check(dim, S, T, basis, npc, support, fields):
    def make():
        return pacman.rbf.Plan(dim, S, T, nodes_per_cluster=npc, support_radius=support,
                               precision="mixed")
    plan, fresh = make(), make()
    n = np.diff(plan.patch_lists("source")[0])
    m = np.diff(plan.patch_lists("target")[0])
    assert n.max() <= 96 and ((n >= 65) & (m > 0)).any()
    plan.execute(basis, _fields(S, fields, 0), keep_factors=True)
    for seed in (1, 2):
        v = _fields(S, fields, seed)
        st = {}
        out = plan.execute(basis, v, keep_factors=True, stats=st)
        assert st["factors_reused"] == np.count_nonzero(m)
        assert rel_l2(out, fresh.execute(basis, v)) <= TOL_REUSE
        for f in {0, fields - 1}:
            ref = oracle.interpolate(dim, basis, S, np.ascontiguousarray(v[:, f]), T, npc,
                                     support_radius=support)
            assert rel_l2(out[:, f], ref) <= TOL_MIXED
    plan.close()
    fresh.close()


@pytest.mark.parametrize("fields", [1, 3, 8])
@pytest.mark.parametrize("n", [65, 80, 95, 96])
def test_whole_cloud_patches(n, fields):
    rng = np.random.default_rng(n)
    _check(3, rng.random((n, 3)), rng.random((120, 3)), 0x11, n, 1.0, fields)


@pytest.mark.parametrize("fields", [1, 3, 8])
@pytest.mark.parametrize("dim,count", [(2, 5000), (3, 20000)])
def test_uniform_clouds(dim, count, fields):
    rng = np.random.default_rng(dim)
    _check(dim, rng.random((count, dim)), rng.random((4000, dim)), 0x12, 50, 0.1, fields)


@pytest.mark.parametrize("made,used", [("128", "128"), ("128", None), (None, "128"), ("8", "128")])
def test_size_line_of_the_environment(made, used, monkeypatch):
    # PACMAN_B200_BIG_N = 128 leaves patches of 97 to 128 sources to a kernel that
    # keeps nothing; the line may also differ between the two executes.
    def line(value):
        if value is None:
            monkeypatch.delenv("PACMAN_B200_BIG_N", raising=False)
        else:
            monkeypatch.setenv("PACMAN_B200_BIG_N", value)
    case = W.make("grid_blobs_1m", scale=0.01)
    S, T = case["src"], case["tgt"]
    plan = pacman.rbf.Plan(3, S, T, precision="mixed")
    n = np.diff(plan.patch_lists("source")[0])
    m = np.diff(plan.patch_lists("target")[0])
    assert ((n > 96) & (n <= 128) & (m > 0)).any() and ((n > 128) & (m > 0)).any()
    line(made)
    plan.execute(0x12, _fields(S, 1, 0), keep_factors=True)
    line(used)
    for fields, seed in ((1, 1), (2, 2)):
        v = _fields(S, fields, seed)
        st = {}
        out = plan.execute(0x12, v, keep_factors=True, stats=st)
        assert st["factors_reused"] > 0
        for f in range(fields):
            ref = oracle.interpolate(3, 0x12, S, np.ascontiguousarray(v[:, f]), T)
            assert rel_l2(out[:, f], ref) <= TOL_MIXED
    plan.close()
