"""The one-cluster join engine at the sizes where its split can go wrong: the
edges of a CTA's range (128 slots), of a 32-slot word, of a block of 1,024
sites, and ranges of more words than a warp takes at once.  Small trees are
checked against the oracle, the largest against the column scan on all SMs."""
import numpy as np
import pytest

import oracle as O
from casphy_b200 import synth

pytestmark = pytest.mark.gpu


def _case(ncell, nsite, nallele, weights, seed):
    raw = synth.lineage_states(ncell, nsite, 16, 0.04, nallele, 1.3, 0.1, seed=seed)
    codes, ns = synth.regularize(raw)
    rng = np.random.default_rng(seed)
    w = {"unit": np.ones((ns, nsite)), "integer": rng.integers(0, 3, size=(ns, nsite)).astype(float),
         "half": rng.uniform(0.01, 4.0, size=(ns, nsite))}[weights]
    return codes, ns, w


@pytest.mark.parametrize("weights", ["unit", "integer", "half"])
@pytest.mark.parametrize("ncell,nsite,nallele", [
    (2, 1, 2), (3, 5, 3), (33, 7, 4), (128, 31, 9), (129, 64, 9), (257, 1030, 30), (1025, 40, 8), (2049, 33, 12), (700, 90, 300), (1600, 260, 200),
    (4400, 12, 5)])
def test_cluster_join_vs_oracle(gpu_lib, weights, ncell, nsite, nallele):
    codes, ns, w = _case(ncell, nsite, nallele, weights, seed=ncell + nsite)
    e1, s1, st = gpu_lib.join_indel(codes, ns, w)
    assert st["scan_path"] == 1
    e0, s0, _ = O.join_indel(codes, ns, w)
    assert np.array_equal(e1, e0) and np.array_equal(s1, s0)


@pytest.mark.parametrize("weights", ["unit", "half"])
def test_cluster_join_size_rule(gpu_lib, weights):
    codes, ns, w = _case(700, 40, 8, weights, seed=5)
    tip = np.random.default_rng(5).integers(1, 30, size=700)
    e1, s1, _ = gpu_lib.join_indel(codes, ns, w, tip, 12, 1.5)
    e0, s0, _ = O.join_indel(codes, ns, w, tip, 12, 1.5)
    assert np.array_equal(e1, e0) and np.array_equal(s1, s0)


@pytest.mark.parametrize("ncell,nsite,weights", [(17000, 24, "unit"), (40000, 16, "unit"), (9000, 20, "half")])
def test_cluster_join_vs_column_scan(gpu_lib, monkeypatch, ncell, nsite, weights):
    codes, ns, w = _case(ncell, nsite, 12, weights, seed=ncell)
    e1, s1, st1 = gpu_lib.join_indel(codes, ns, w)
    assert st1["scan_path"] == 1 and st1["compactions"] > 0
    monkeypatch.setenv("CASPHY_INDEL_SCAN", "dense")
    e0, s0, st0 = gpu_lib.join_indel(codes, ns, w)
    assert st0["scan_path"] == 0
    assert np.array_equal(e1, e0) and np.array_equal(s1, s0)


@pytest.mark.parametrize("weights", ["unit", "planes", "float"])
@pytest.mark.parametrize("ncell,nsite,atype", [
    (2, 32, 0), (3, 64, 1), (31, 32, 1), (33, 96, 0), (513, 96, 1), (1100, 1056, 0), (2500, 64, 1), (6000, 224, 1)])
def test_cluster_bit_join_vs_oracle(gpu_lib, weights, ncell, nsite, atype):
    """Bit rows: one cell to a range and several words per lane; columns that
    are resident in shared memory at once and only after a compaction."""
    words = synth.binary_workload(ncell, nsite, 14, 0.04, 0.05, seed=ncell + nsite)
    rng = np.random.default_rng(ncell)
    w = {"unit": None, "planes": rng.integers(0, 7, size=nsite).astype(float),
         "float": rng.uniform(0.01, 3.0, size=nsite)}[weights]
    e1, s1, _ = gpu_lib.join_bit(words, w, atype)
    e0, s0, _ = O.join_bit(words, w, atype)
    assert np.array_equal(e1, e0) and np.array_equal(s1, s0)
