"""As many targets as a call may have: the nearest-source search takes them in
turns.  Points are limited to 2^31 - 1 in each set, not in both together."""
import pytest

import pacman_b200 as pacman

pytestmark = pytest.mark.gpu

NN = pacman.fe.methods.NEAREST_NEAREST


def test_more_points_than_an_index_holds():
    torch = pytest.importorskip("torch")
    n, m = 2000, 2 ** 31 - 1000
    turn = 2 ** 28
    gen = torch.Generator(device="cuda").manual_seed(1)
    S = torch.rand((n, 1), dtype=torch.float64, device="cuda", generator=gen)
    v = torch.arange(n, dtype=torch.float64, device="cuda")
    T = torch.rand((m, 1), dtype=torch.float64, device="cuda", generator=gen)
    out, _ = pacman.fe.interpolate(1, pacman.execspaces.CUDA, NN, S, v, None, None, None, T)
    for first in (0, turn - 500, 5 * turn - 500, 2 ** 30 + 12345, m - 1000):
        part = T[first:first + 1000]
        near = (part - S.T).abs().argmin(dim=1)
        assert torch.equal(out[first:first + 1000], v[near])
    del out, T
    torch.cuda.empty_cache()
