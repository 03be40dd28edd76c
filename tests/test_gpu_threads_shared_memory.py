"""Threads whose patches need different amounts of shared memory in the same
kernel (FP64, 97 to 128 sources a patch) do not refuse each other's launches."""
import threading

import numpy as np
import pytest

import pacman_b200 as pacman

pytestmark = pytest.mark.gpu


def _job(n):
    rng = np.random.default_rng(n)
    S, T = rng.random((n, 3)), rng.random((40, 3))
    v = np.sin(S @ [3.0, 2.0, 1.0])
    plan = pacman.rbf.Plan(3, S, T, nodes_per_cluster=n, support_radius=1.0)
    assert np.diff(plan.patch_lists("source")[0]).max() == n
    return lambda: plan.execute(0x11, v)


def test_sizes_side_by_side():
    jobs = [_job(n) for n in (97, 128, 97, 128)]
    want = [job() for job in jobs]
    wrong = []

    def work(i):
        try:
            for _ in range(400):
                if not np.array_equal(jobs[i](), want[i]):
                    wrong.append(i)
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            wrong.append((i, repr(e)))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
