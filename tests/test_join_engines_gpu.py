"""The greedy joins' engines: which one a call runs on, and that each gives the
oracle's tree."""
import numpy as np
import pytest

import oracle as O
from casphy_b200 import synth

pytestmark = pytest.mark.gpu


def _indel(ncell, nsite, nallele, weights, seed):
    raw = synth.lineage_states(ncell, nsite, 16, 0.04, nallele, 1.3, 0.1, seed=seed)
    codes, ns = synth.regularize(raw)
    rng = np.random.default_rng(seed)
    w = {"unit": np.ones((ns, nsite)), "integer": rng.integers(0, 3, size=(ns, nsite)).astype(float),
         "half": rng.uniform(0.01, 4.0, size=(ns, nsite))}[weights]
    return codes, ns, w


def _bit(ncell, nsite, weights, seed):
    words = synth.binary_workload(ncell, nsite, 14, 0.04, 0.05, seed=seed)
    rng = np.random.default_rng(seed)
    w = {"unit": None, "planes": rng.integers(0, 7, size=nsite).astype(float),
         "float": rng.uniform(0.01, 3.0, size=nsite)}[weights]
    return words, w


def _same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


# rows, bitsets and fill; initial scan; join; gather.  Fractional weights: the
# columns of the initial scan too.  Codes that are not resident from the start:
# the bitsets are split by CTA.
@pytest.mark.parametrize("ncell,nsite,weights,launches", [
    (900, 60, "unit", 6), (4100, 600, "unit", 7), (500, 20, "half", 7), (4500, 700, "half", 8)])
def test_indel_join_counts_its_launches(gpu_lib, ncell, nsite, weights, launches):
    codes, ns, w = _indel(ncell, nsite, 8, weights, 3)
    assert gpu_lib.join_indel(codes, ns, w)[2]["kernel_launches"] == launches


def test_bit_join_counts_its_launches(gpu_lib):
    # rows, fill, initial scan, join, gather
    words, w = _bit(300, 64, "unit", 3)
    assert gpu_lib.join_bit(words, w, 0)[2]["kernel_launches"] == 5
    # one cell: no scan and no join
    assert gpu_lib.join_bit(words[:1], w, 0)[2]["kernel_launches"] == 3
