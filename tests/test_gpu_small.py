"""Register-kernel patches (n <= 96): every size class and its edges, field
counts, both precisions, the adjoint, and clouds whose matrices are singular,
against the CPU oracle."""
import numpy as np
import pytest

import oracle
import pacman_b200 as pacman
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

CUDA = pacman.execspaces.CUDA
# The transfer's specified tolerances (tests/test_gpu_parity.py).
TOL = {"fp64": 1e-12, "mixed": 1e-10}


def _fields(p, count):
    x = p @ np.array([3.0, 2.0, 1.0])[: p.shape[1]]
    return np.stack([np.sin(x + f) + f * np.cos(2 * x) for f in range(count)], axis=1)


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("fields", [1, 3, 8])
def test_size_classes_match_oracle(precision, fields):
    # Enough patches that every class (32, 40, 48, 56, 64) gets its own launch.
    rng = np.random.default_rng(8)
    S, T = rng.random((110003, 3)), rng.random((90001, 3))
    v = _fields(S, fields)
    plan = pacman.rbf.Plan(3, S, T, precision=precision)
    n = np.diff(plan.patch_lists("source")[0])
    edges = {32, 33, 40, 41, 48, 49, 56, 57, 64, 65}
    assert edges <= set(n.tolist()) and n.min() < 32
    for lo, hi in ((0, 32), (32, 40), (40, 48), (48, 56), (56, 64)):
        assert ((n > lo) & (n <= hi)).sum() > 5 * 148
    out = plan.execute(0x12, v)
    for f in {0, fields - 1}:
        ref = oracle.interpolate(3, 0x12, S, np.ascontiguousarray(v[:, f]), T)
        assert rel_l2(out[:, f], ref) <= TOL[precision]
    assert not (plan.patch_status() & (2 | 4 | 16)).any()


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("n", [2, 3, 17, 31, 32, 33, 48, 63, 64, 65])
def test_whole_cloud_patches_match_oracle(precision, n):
    rng = np.random.default_rng(n)
    S = rng.random((n, 2))
    T = S.min(0) + (S.max(0) - S.min(0)) * rng.random((40, 2))
    v = _fields(S, 1)[:, 0]
    out = pacman.rbf.interpolate(2, CUDA, 0x11, S, v, T, nodes_per_cluster=64,
                                 precision=precision)
    ref = oracle.interpolate(2, 0x11, S, v, T, 64)
    assert np.array_equal(np.isfinite(out), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert rel_l2(out[ok], ref[ok]) <= TOL[precision]


def test_repeated_sources_stay_singular():
    # Two equal points make A exactly singular: the FP64 path answers what the
    # unpivoted LU answers (non-finite values at the targets of their patches).
    rng = np.random.default_rng(4)
    S = rng.random((700, 3))
    S[350] = S[20]
    T = rng.random((900, 3))
    v = _fields(S, 1)[:, 0]
    plan = pacman.rbf.Plan(3, S, T)
    out = plan.execute(0x12, v)
    ref = oracle.interpolate(3, 0x12, S, v, T)
    assert not np.isfinite(ref).all()
    assert np.array_equal(np.isfinite(out), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert rel_l2(out[ok], ref[ok]) <= TOL["fp64"]
    assert not (plan.patch_status() & (4 | 16)).any()


@pytest.mark.parametrize("fields", [1, 2, 8])
def test_adjoint_is_the_transpose(fields):
    # <G, out(v)> = <v, adjoint(G)> for random v and G, all size classes.
    rng = np.random.default_rng(9)
    S, T = rng.random((90001, 3)), rng.random((80003, 3))
    v, G = rng.standard_normal((len(S), fields)), rng.standard_normal((len(T), fields))
    plan = pacman.rbf.Plan(3, S, T)
    out = plan.execute(0x11, v, save_for_adjoint=True)
    gv, _ = plan.adjoint(G, targets=False)
    # Both sums round each of their terms once more: n eps of the larger norm.
    scale = np.linalg.norm(out) * np.linalg.norm(G) + np.linalg.norm(v) * np.linalg.norm(gv)
    assert abs((G * out).sum() - (v * gv).sum()) <= 1e-11 * scale


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("n", [65, 66, 80, 95, 96, 97])
def test_three_warp_class_matches_oracle(precision, n):
    # 65 to 96 sources: three warps, the last of them full or ragged.
    rng = np.random.default_rng(n)
    S = rng.random((n, 3))
    T = S.min(0) + (S.max(0) - S.min(0)) * rng.random((50, 3))
    plan = pacman.rbf.Plan(3, S, T, nodes_per_cluster=128, precision=precision)
    assert n in np.diff(plan.patch_lists("source")[0])
    for fields in (1, 3, 8):
        v = _fields(S, fields)
        out = plan.execute(0x11, v, save_for_adjoint=True)
        for f in range(fields):
            ref = oracle.interpolate(3, 0x11, S, np.ascontiguousarray(v[:, f]), T, 128)
            assert rel_l2(out[:, f], ref) <= TOL[precision]
        G = rng.standard_normal((len(T), fields))
        gv, _ = plan.adjoint(G, targets=False)
        scale = np.linalg.norm(out) * np.linalg.norm(G) + np.linalg.norm(v) * np.linalg.norm(gv)
        assert abs((G * out).sum() - (v * gv).sum()) <= 1e-10 * scale
    assert not (plan.patch_status() & (2 | 4 | 16)).any()


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n", [60, 200])
@pytest.mark.parametrize("ratio", [1e-3, 0.2, 0.45, 0.55, 0.99, 1.01, 3.0])
def test_axis_drop_decision_near_the_limit(dim, n, ratio):
    # The last axis is scaled so that cond([1, x]) = ratio 1e5: an axis is
    # dropped in exactly the patches above the limit (1% is far above the rounding
    # of a condition number of 1e5, about 1e-11).
    rng = np.random.default_rng(n + dim)
    S = 1.0 + rng.random((n, dim))
    T = S[:20].copy()

    def cond(h):
        P = S.copy()
        P[:, -1] = 1.5 + (P[:, -1] - 1.5) * h
        return np.linalg.cond(np.column_stack([np.ones(n), P])), P

    lo, hi = 1e-8, 1.0
    for _ in range(200):
        mid = np.sqrt(lo * hi)
        lo, hi = (mid, hi) if cond(mid)[0] > ratio * 1e5 else (lo, mid)
    c, P = cond(hi)
    assert abs(c / (ratio * 1e5) - 1) < 1e-3
    T[:, -1] = P[:20, -1]
    plan = pacman.rbf.Plan(dim, P, T, nodes_per_cluster=256)
    v = np.sin(P.sum(axis=1))
    out = plan.execute(0x12, v)
    assert np.isfinite(out).all()
    off, idx = plan.patch_lists("source")[:2]
    toff = plan.patch_lists("target")[0]
    status = plan.patch_status()
    checked = 0
    for k in range(len(off) - 1):
        own = P[idx[off[k]:off[k + 1]]]
        if toff[k + 1] > toff[k] and len(own) > dim:
            c = np.linalg.cond(np.column_stack([np.ones(len(own)), own])) / 1e5
            if abs(c - 1) > 0.005:
                assert (status[k] & 1) == (c > 1)
                checked += 1
    assert checked


def test_shards_choose_the_solver_of_the_whole_plan():
    # Patches of 65 to 96 sources go to the register kernel where the plan has no
    # larger one; shards whose own patches are all smaller answer as the whole does.
    rng = np.random.default_rng(12)
    S = np.r_[rng.random((12000, 3)), 0.02 * rng.random((150, 3))]
    T = rng.random((9000, 3))
    v = _fields(S, 1)[:, 0]

    def plan():
        return pacman.rbf.Plan(3, S, T, nodes_per_cluster=60, precision="mixed")

    full = plan()
    n = np.diff(full.patch_lists("source")[0])
    assert n.max() > 96
    ref = full.execute(0x12, v)
    total, without = np.zeros_like(ref), 0
    for rank in range(4):
        p = plan()
        p.shard(rank, 4)
        live = n[np.diff(p.patch_lists("target")[0]) > 0]
        without += live.max() <= 96 and (live > 64).any()
        total += p.execute(0x12, v)
    assert without
    assert np.array_equal(total, ref)
