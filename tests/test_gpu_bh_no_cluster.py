"""Barnes-Hut of small designs where no cluster fits the device share (FLUXION_BH_CLUSTER=0 says so
in a process of its own): the many-block sort takes over, with the same keys, order, root, forces and
iterations, bit for bit, around the sizes at which the cluster's blocks hold more points a thread."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

_SCRIPT = r"""
import sys
sys.path[:0] = [sys.argv[1]]
import numpy as np
import fluxion_b200 as fx
out = {}
ctx = fx.Context(0)
for n in (1, 2, 513, 4096, 4097, 8193, 16385, 32768, 32769):
    rng = np.random.default_rng(n)
    side = float(1.2 * np.sqrt(n) + 4)
    x, y = (rng.random((2, n)) * side).astype(np.float32)
    d = fx.Design(ctx, fx.Circuit.from_nets([[0, n - 1]] if n > 1 else [[0]], n, side, side))
    d.set_positions(x, y)
    at = ctx.kernel_launches()
    for name, v in zip(("fx", "fy", "keys", "perm", "root"), d.barnes_hut()):
        out[f"{n}_{name}"] = v
    out[f"{n}_launches"] = ctx.kernel_launches() - at
    d.force_iterate(fx.iter_cfg(density_bins=0, cong_cols=0, cong_rows=0), 3)
    out[f"{n}_x"], out[f"{n}_y"] = d.get_positions()
    d.close()
ctx.close()
np.savez(sys.argv[2], **out)
"""


def _run(path, **env):
    r = subprocess.run([sys.executable, "-c", _SCRIPT, str(ROOT / "neon-physics-fluxion_b200"),
                        str(path)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, **env))
    assert r.returncode == 0, r.stdout + r.stderr
    return np.load(path)


def test_many_block_sort_takes_over(fx, tmp_path):
    got = _run(tmp_path / "without.npz", FLUXION_BH_CLUSTER="0")
    want = _run(tmp_path / "with.npz")
    more = 0
    for k in want.files:
        if k.endswith("_launches"):
            more += int(got[k] > want[k])
        else:
            assert np.array_equal(got[k], want[k]), k
    assert more == 8  # all but 32,769 points took the cluster
