"""The candidates' selection at the edge of the shared memory that a launch has without asking: 1,024 origins x
6 tiles are 48 KB of entries, and the kernel's own arrays come on top.  In a process of its own, since an
earlier call with more entries would have asked."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CALL = """
import sys
sys.path[:0] = [{root!r}, {root!r} + '/tests', {root!r} + '/oracle']
import numpy as np
import cryoim_gb300 as ci
from _data import small_case
p, vol, tmpl, timgs, imgs, parts, truth = small_case(P=3, T=2, step=4.0)
q = parts.copy()
for i, f in enumerate(('theta', 'phi', 'omega')):
    q[f] = truth[:, i] + 2.0
with ci.Context(0, p) as ctx:
    ctx.set_reference_map(vol)
    c = ctx.contract_search(imgs, q, origin_max=15.5, origin_step=1.0, topk=16, pick=1, want_cands=True,
                            local_range=10.0, local_step=2.0)
have = c[:, :, 5] > -1e38
assert have[:, 0].all() and np.abs(c[:, :, 5] - c[:, :, 6])[have].max() < 2e-2
"""


def test_selection_at_48_kilobytes(built):
    r = subprocess.run([sys.executable, "-c", CALL.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
