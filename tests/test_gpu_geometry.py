"""Geometry kernels at their edges, bit for bit against the CPU oracle: list
lengths around the warp, block and segmented sorts, radii whose k-th distance
is shared by many sources, refined clouds, few points, targets outside the
sources' box and no targets."""
import numpy as np
import pytest

import oracle
import pacman_b200 as pacman

pytestmark = pytest.mark.gpu


def _same(dim, S, T, npc):
    plan = pacman.rbf.Plan(dim, S, T, nodes_per_cluster=npc)
    ref = oracle.build(dim, S, T, npc)
    info = plan.info()
    assert info["radius"] == ref.radius
    assert info["num_candidates"] == ref.num_candidates
    assert info["num_patches"] == ref.num_patches
    assert np.array_equal(plan.centers(), ref.centers())
    sizes = []
    for which, csr in (("source", ref.src_csr()), ("target", ref.tgt_csr())):
        off, idx = plan.patch_lists(which)
        assert np.array_equal(off, csr[0]), which
        assert np.array_equal(idx, csr[1]), which
        sizes.append(np.diff(off))
    return sizes


# Longest lists below and above a warp's sort (256), a block's (32768), and
# past it; in 1D an inner patch holds about npc sources.
@pytest.mark.parametrize("npc,lo,hi", [(110, 65, 256), (140, 129, 256), (225, 257, 512),
                                       (270, 257, 512), (4000, 2049, 8192),
                                       (14000, 8193, 16384), (24000, 16385, 32768),
                                       (34000, 32769, 70001)])
def test_list_lengths(npc, lo, hi):
    rng = np.random.default_rng(1)
    S, T = rng.random((70001, 1)), rng.random((5003, 1))
    ns, _ = _same(1, S, T, npc)
    assert lo <= ns.max() <= hi


@pytest.mark.parametrize("seed", range(6))
def test_radius_is_the_same_every_time(seed):
    # Several blocks per kernel of the radius search, built again and again.
    rng = np.random.default_rng(seed)
    S, T = rng.random((150000, 3)), rng.random((1000, 3))
    ref = oracle.build(3, S, T, 50)
    for _ in range(5):
        info = pacman.rbf.Plan(3, S, T).info()
        assert (info["radius"], info["num_patches"]) == (ref.radius, ref.num_patches)


@pytest.mark.parametrize("ring", [2000, 2049, 6000])
def test_radius_with_equal_distances(ring):
    # The central sample projects onto the centre of a ring of sources; the
    # 50th distance is the ring's, shared by more keys than are gathered.
    a = 2 * np.pi * np.arange(ring) / ring
    circle = np.stack([np.cos(a), np.sin(a)], axis=1)
    rng = np.random.default_rng(2)
    S = np.concatenate([[[0.0, 0.0]], circle, 3.0 * rng.random((500, 2)) - 1.5])
    S = np.concatenate([S, [[-1.5, -1.5], [1.5, 1.5]]])
    T = 3.0 * rng.random((2000, 2)) - 1.5
    _same(2, S, T, 50)


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("n", [2, 5, 31, 257, 4000])
def test_small_clouds(dim, n):
    rng = np.random.default_rng(n)
    _same(dim, rng.random((n, dim)), 1.4 * rng.random((n + 3, dim)) - 0.2, 20)


def test_refined_cloud_and_far_targets():
    rng = np.random.default_rng(5)
    S = np.concatenate([rng.random((20000, 3)), 0.5 + 0.003 * rng.standard_normal((30000, 3))])
    T = np.concatenate([rng.random((20000, 3)), 5.0 + rng.random((100, 3))])
    _same(3, S, T, 50)


def test_no_targets():
    rng = np.random.default_rng(6)
    S = rng.random((3000, 3))
    _same(3, S, np.zeros((0, 3)), 30)


@pytest.mark.parametrize("dim", [1, 2, 3])
def test_point_searches_at_cell_faces_and_outside(dim):
    # Sources and targets on the faces and corners of the search grid's cells,
    # targets far outside, fewer sources than one shell.
    rng = np.random.default_rng(dim)
    for n in (3, 64, 4096):
        side = int(round(n ** (1.0 / dim)))
        g = np.arange(side) / max(side, 1)
        S = np.stack(np.meshgrid(*([g] * dim), indexing="ij"), -1).reshape(-1, dim)
        T = np.concatenate([S, S + 0.5 / side, S[:50] - 3.0, S[:50] + 7.5,
                            rng.random((200, dim))])
        v = np.cos(S @ np.arange(1.0, dim + 1))
        out, _ = pacman.fe.interpolate(dim, pacman.execspaces.CUDA,
                                       pacman.fe.methods.NEAREST_NEAREST, S, v, None, None, None, T)
        assert np.array_equal(out, oracle.fe_nearest(dim, S, v, T)[0])
        mls = pacman.mls.interpolate(dim, pacman.execspaces.CUDA, S, v, T)
        assert np.array_equal(mls, oracle.mls_interpolate(dim, S, v, T, knn="brute"))


def test_mls_target_chunks():
    # More targets than one chunk of neighbour ids holds.
    rng = np.random.default_rng(3)
    S, T = rng.random((700, 1)), rng.random(((1 << 22) + 1001, 1))
    v = np.sin(5 * S[:, 0])
    out = pacman.mls.interpolate(1, pacman.execspaces.CUDA, S, v, T)
    pick = np.r_[0:2000, (1 << 22) - 500:len(T)]
    assert np.array_equal(out[pick], oracle.mls_interpolate(1, S, v, T[pick]))
    near = rng.choice(len(T), 20000, replace=False)
    assert np.array_equal(out[near], oracle.mls_interpolate(1, S, v, T[near]))
