"""An indel join whose bitsets fit the free device memory only without a
cluster's layout (which rounds every CTA's slots up to 128: 2,100 cells take 4,096
slots there and 2,176 on all SMs) runs on all SMs."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_FRESH = r"""
import json, sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
import casphy_b200.lib as L
rng = np.random.default_rng(1)
ncell, nsite, ns = 2100, 400, 20000
codes = rng.integers(2, ns + 2, size=(90, nsite))[rng.integers(0, 90, size=ncell)]
codes[rng.random(codes.shape) < 0.6] = 1
codes = codes.astype(np.uint32)
w = np.ones((ns, nsite)) if sys.argv[2] == "unit" else rng.uniform(0.5, 2.0, size=(ns, nsite))
small = codes[:40]
L.join_indel(small, ns, w[:, :nsite])  # the context and its kernels
# bitsets: 4.4 GB on all SMs, 8.2 GB in the cluster's layout
free = torch.cuda.mem_get_info()[0]
keep = torch.empty(max(free - (6 << 30), 0), dtype=torch.uint8, device="cuda")
e1, s1, st1 = L.join_indel(codes, ns, w)
del keep
torch.cuda.empty_cache()
e2, s2, st2 = L.join_indel(codes, ns, w)
print(json.dumps([st1["scan_path"], st1["refreshes"], st2["scan_path"], st2["refreshes"],
                  bool(np.array_equal(e1, e2) and np.array_equal(s1, s2))]))
"""


@pytest.mark.parametrize("weights", ["unit", "half"])
def test_short_memory_leaves_the_cluster(weights):
    root = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
    out = subprocess.run([sys.executable, "-c", _FRESH, root, weights], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    path1, ref1, path2, ref2, same = json.loads(out.stdout.strip().splitlines()[-1])
    assert same and path2 == 1 and ref2 == 0      # room: a cluster
    assert path1 == (1 if weights == "unit" else 0) and ref1 > 0
