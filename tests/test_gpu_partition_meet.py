"""The power iterations of a depth wait for one another with a limit on the polls. With a limit of
one poll (FLUXION_PART_MEET_POLLS, read once per process) the wait runs out at once: the call
returns FX_ETIMEOUT, as every bounded wait does, and the context stays usable."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

_SCRIPT = r"""
import sys
sys.path[:0] = [sys.argv[1]]
import numpy as np
import fluxion_b200 as fx
from fluxion_b200 import _lib
s = fx.synth_plain(1, 9001, 10800, 115.0)
ctx = fx.Context(0)
d = fx.Design(ctx, s.circuit)
cfg = lambda tol: fx.part_cfg(mode=fx.FX_PART_FP64, power_iterations=30, tol=tol)
before = d.partition(cfg(1e-6))
try:
    d.partition(cfg(0.0))
    raise SystemExit("no wait ran out")
except fx.FluxionError as e:
    assert e.code == _lib.FX_ETIMEOUT, e
after = d.partition(cfg(1e-6))  # the stepped kernels wait for nothing
assert np.array_equal(before["leaf_gate"], after["leaf_gate"])
d.close()
ctx.close()
print("timeout ok")
"""


def test_expired_meeting_is_a_timeout(fx):
    env = dict(os.environ, FLUXION_PART_MEET_POLLS="1")
    r = subprocess.run([sys.executable, "-c", _SCRIPT, str(ROOT / "neon-physics-fluxion_b200")],
                       capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "timeout ok" in r.stdout
