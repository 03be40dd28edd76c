"""A patch whose tiles fit the memory but not its int8 slices beside them."""
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.conftest import ROOT, rel_l2

pytestmark = pytest.mark.gpu

N = 20000  # tiles 3.2 GB, slices 2.8 GB

CHILD = """
import sys
import numpy as np
import torch
import pacman_b200 as pacman
leave, path = float(sys.argv[1]), sys.argv[2]
rng = np.random.default_rng(0)
S, T = rng.random((%d, 3)), 0.5 + 0.01 * rng.random((50, 3))
v = np.sin(S @ [3.0, 2.0, 1.0])
torch.zeros(1, device="cuda")
if leave:
    free, _ = torch.cuda.mem_get_info()
    rest = torch.empty(int(free - leave * 2 ** 30), dtype=torch.uint8, device="cuda")
plan = pacman.rbf.Plan(3, S, T, nodes_per_cluster=len(S), precision="mixed")
assert np.diff(plan.patch_lists("source")[0]).max() == len(S)
np.save(path, plan.execute(0x11, v))
assert not (plan.patch_status() & (2 | 4 | 8 | 16)).any()
""" % N


def _run(leave, path):
    subprocess.run([sys.executable, "-c", CHILD, str(leave), str(path)], check=True, cwd=ROOT,
                   env=dict(os.environ, PYTHONPATH=ROOT), timeout=300)
    return np.load(path)


def test_slices_that_do_not_fit(tmp_path):
    # 5 GiB left: room for the tiles and half of the slices.
    out = _run(5.0, tmp_path / "little.npy")
    assert rel_l2(out, _run(0.0, tmp_path / "all.npy")) <= 1e-10  # the mixed path's tolerance
