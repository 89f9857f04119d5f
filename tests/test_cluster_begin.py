"""The cluster join's slots are visible to the whole block before a model reads
them.  Slot x is written by thread x mod 512, that is by warp (x mod 512) / 32;
the indel model's resident codes read it from warp x mod 16.  A block barrier
between the two is what orders them: without it the read is of whatever shared
memory held, and it indexes the node rows."""
import os
import re

import numpy as np
import pytest

import oracle as O
from casphy_b200 import synth

SRC = os.path.join(os.path.dirname(__file__), "..", "casphy_b200", "csrc", "join_cluster.cuh")


def test_slots_are_written_by_other_warps_than_read_them():
    x = np.arange(1024)
    assert np.mean((x % 512) // 32 != x % 16) > 0.9


def test_a_block_barrier_lies_between_the_slots_and_begin():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    init = text.index("st.idx[x] = key_node(key);")
    begin = text.index("M::begin(")
    assert init < begin and "__syncthreads();" in text[init:begin]


@pytest.mark.gpu
@pytest.mark.parametrize("weights", ["unit", "half"])
def test_resident_codes_of_trees_of_changing_size(gpu_lib, weights):
    """Codes resident from the start, in trees whose ranges fill from one to
    all sixteen warps, one after the other, so that shared memory holds another
    tree's slots when each begins."""
    for ncell, nsite in ((1024, 256), (40, 9), (1900, 150), (130, 77), (1024, 256), (515, 31)):
        raw = synth.lineage_states(ncell, nsite, 16, 0.04, 8, 1.3, 0.1, seed=ncell)
        codes, ns = synth.regularize(raw)
        w = np.ones((ns, nsite)) if weights == "unit" else \
            np.random.default_rng(ncell).uniform(0.01, 4.0, size=(ns, nsite))
        e0, s0, _ = O.join_indel(codes, ns, w)
        for _ in range(3):
            e1, s1, st = gpu_lib.join_indel(codes, ns, w)
            assert st["scan_path"] == 1
            assert np.array_equal(e1, e0) and np.array_equal(s1, s0)
