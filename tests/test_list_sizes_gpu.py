"""Cell and index lists at sphere counts where the sort of long lists changes
its form or what it asks of the device."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

# In a process of its own: a larger substrate built earlier would leave the
# kernel's shared-memory limit raised.  Ascending, so that no size does that
# for the next.
FRESH = """
import numpy as np
from nozomi_b200 import engine
for S in (384_640, 384_641, 390_000, 393_216, 393_217):
    rng = np.random.default_rng(S)
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-20.0, 20.0, (3, S))
    sph[3] = 0.2
    sph[4] = rng.integers(0, 3, S)
    sub = engine.DeviceSubstrate(sph, 3, (40.0,) * 3, (6, 6, 6), np.full(4, 2.0), np.full(4, 80.0), near_margin=0.4)
    perm = sub.perm.cpu().numpy()
    for start, count, items, idx in ((sub.cell_start, sub.cell_count, sub.cell_items, sub.cell_idx),
                                     (*sub.near[:3], sub.near[5])):
        start, count, items, idx = (t.cpu().numpy() for t in (start, count, items, idx))
        for c in (0, 100, 215):
            part = slice(start[c], start[c] + count[c])
            assert count[c] > 128 and (np.diff(items[part]) > 0).all()
            assert np.array_equal(idx[part], np.sort(perm[items[part]]))
print("built")
"""


def test_lists_of_a_fresh_process():
    r = subprocess.run([sys.executable, "-c", FRESH], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "built" in r.stdout, r.stderr[-800:]
