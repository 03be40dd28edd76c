"""Point methods for targets with NaN coordinates, which have no neighbour and get
zero, and with infinite ones, among ordinary targets."""
import numpy as np
import pytest

import oracle
import pacman
import pacman_b200

pytestmark = pytest.mark.gpu

CUDA = pacman_b200.execspaces.CUDA
NN = pacman_b200.fe.methods.NEAREST_NEAREST


def _problem(dim):
    rng = np.random.default_rng(dim)
    S, T = rng.random((5000, dim)), rng.random((600, dim))
    T[::3, 0] = np.nan
    T[1::6, dim - 1] = -np.nan
    return S, T, rng.standard_normal(len(S)), np.isnan(T).any(axis=1)


@pytest.mark.parametrize("dim", [1, 2, 3])
def test_nearest(dim):
    S, T, v, nan = _problem(dim)
    T[2::60] = np.inf
    out, _ = pacman_b200.fe.interpolate(dim, CUDA, NN, S, v, None, None, None, T)
    ref, _ = oracle.fe_nearest(dim, S, v, T)
    assert np.all(out[nan] == 0.0)
    assert np.array_equal(out[~nan], ref[~nan])


@pytest.mark.parametrize("dim", [1, 2, 3])
def test_mls(dim):
    S, T, v, nan = _problem(dim)
    out = pacman.MLS.interpolate(dim, CUDA, S, v, T)
    assert np.all(out[nan] == 0.0)
    assert np.array_equal(out[~nan], oracle.mls_interpolate(dim, S, v, T[~nan]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_transfer(precision):
    S, T, v, nan = _problem(3)
    out = pacman_b200.rbf.interpolate(3, CUDA, 0x11, S, v, T, precision=precision)
    clean = pacman_b200.rbf.interpolate(3, CUDA, 0x11, S, v, T[~nan], precision=precision)
    assert np.all(out[nan] == 0.0)
    assert np.array_equal(out[~nan], clean)
