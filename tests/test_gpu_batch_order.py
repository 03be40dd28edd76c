"""A batch runs in order on its stream: the geometry after what the caller has
queued there, and the merged solve after every problem's lists are complete,
whichever host thread and stream built them."""
import numpy as np
import pytest

import pacman_b200 as pacman

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", ["1", "2", "5"])
def test_lists_are_complete(threads, monkeypatch):
    # Large problems (their lists take a while to fill) behind small ones, the
    # last one handed out running alone.
    monkeypatch.setenv("PACMAN_B200_BATCH_THREADS", threads)
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2)
    def problem(n, m):
        S, T = rng.random((n, 3)), rng.random((m, 3))
        return (3, 0x11) + tuple(torch.tensor(a, device="cuda") for a in (S, np.sin(S @ [3, 2, 1]), T))
    probs = [problem(n, m) for n, m in ((1500, 900), (120000, 200000), (2000, 1500), (150000, 90000))]
    single = [pacman.rbf.interpolate(d, pacman.execspaces.CUDA, b, S, v, T) for d, b, S, v, T in probs]
    for _ in range(8):
        for one, out in zip(single, pacman.rbf.interpolate_batch(probs)):
            assert torch.equal(one, out)


def test_inputs_still_on_their_way():
    # The points arrive on the caller's stream, behind a kernel of about 50 ms.
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    S, T = rng.random((4000, 3)), rng.random((3000, 3))
    v = np.sin(S @ [3, 2, 1])
    single = pacman.rbf.interpolate(3, pacman.execspaces.CUDA, 0x11, S, v, T)
    final = [torch.tensor(a, device="cuda") for a in (S, v, T)]
    early = [torch.tensor(a, device="cuda") for a in (rng.random(S.shape), v, rng.random(T.shape))]
    pacman.rbf.interpolate_batch([(3, 0x11, *early)])
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)
        for a, b in zip(early, final):
            a.copy_(b)
        out, = pacman.rbf.interpolate_batch([(3, 0x11, *early)])
    stream.synchronize()
    assert np.array_equal(out.cpu().numpy(), single)
