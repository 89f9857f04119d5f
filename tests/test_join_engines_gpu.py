"""The greedy joins' engines: which one a call runs on, and that each gives the
oracle's tree."""
import numpy as np
import pytest

import oracle as O
from casphy_b200 import bootstrap as B
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


# The engine of all SMs takes trees beyond the cluster; here it is asked for at
# sizes the oracle can follow: ranges of no slot, of one, and of several words,
# and enough slots for its compaction (4,096).
@pytest.mark.parametrize("weights", ["unit", "planes", "float"])
@pytest.mark.parametrize("ncell,nsite,atype", [(2, 32, 0), (149, 96, 1), (1100, 416, 0), (5000, 64, 1)])
def test_bit_join_on_all_sms(gpu_lib, monkeypatch, weights, ncell, nsite, atype):
    words, w = _bit(ncell, nsite, weights, ncell + nsite)
    want = O.join_bit(words, w, atype)
    assert _same(gpu_lib.join_bit(words, w, atype), want)
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    got = gpu_lib.join_bit(words, w, atype)
    assert got[2]["kernel_launches"] == 6 and got[2]["scan_path"] == 0
    assert _same(got, want)


@pytest.mark.parametrize("weights", ["unit", "integer", "half"])
@pytest.mark.parametrize("ncell,nsite,nallele,min_size", [
    (2, 1, 2, 0), (149, 33, 9, 0), (1100, 260, 30, 0), (700, 40, 8, 12), (5000, 24, 8, 0)])
def test_indel_join_on_all_sms(gpu_lib, monkeypatch, weights, ncell, nsite, nallele, min_size):
    """Allele bitsets for integer weights, the column scan for fractional ones."""
    codes, ns, w = _indel(ncell, nsite, nallele, weights, ncell)
    tip = np.random.default_rng(ncell).integers(1, 30, size=ncell) if min_size else None
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    got = gpu_lib.join_indel(codes, ns, w, tip, min_size, 1.5)
    assert got[2]["scan_path"] == (0 if weights == "half" else 1)
    assert got[2]["kernel_launches"] == 7
    assert _same(got, O.join_indel(codes, ns, w, tip, min_size, 1.5))


def _many_states(ncell, nsite, nstate, seed):
    """Codes 0 .. nstate + 1 drawn directly, rows alike enough to share alleles."""
    rng = np.random.default_rng(seed)
    base = rng.integers(2, nstate + 2, size=(max(ncell // 25, 2), nsite))
    codes = base[rng.integers(0, len(base), size=ncell)]
    new = rng.random(codes.shape)
    codes = np.where(new < 0.25, rng.integers(2, nstate + 2, size=codes.shape), codes)
    return np.where(new > 0.8, rng.integers(0, 2, size=codes.shape), codes).astype(np.uint32)


# Bitset rows copied to the stage.  More than 253 states never fit a byte; a
# query's 2,080 entries of eight words (2,100 x 2,600) with fractional weights are
# more than the stage holds, so the sums go on over several rounds; 4,500 x 700
# are too many bytes at first, and a compaction makes them resident.
@pytest.mark.parametrize("ncell,nsite,nstate,weights", [
    (300, 70, 254, "unit"), (1500, 1024, 400, "unit"), (2100, 2000, 300, "unit"),
    (300, 70, 254, "half"), (1500, 1024, 400, "half"), (2100, 2600, 300, "half")])
def test_staged_bitsets_of_many_states(gpu_lib, ncell, nsite, nstate, weights):
    codes = _many_states(ncell, nsite, nstate, ncell)
    w = np.ones((nstate, nsite)) if weights == "unit" else \
        np.random.default_rng(1).uniform(0.01, 4.0, size=(nstate, nsite))
    got = gpu_lib.join_indel(codes, nstate, w)
    assert got[2]["scan_path"] == 1 and got[2]["kernel_launches"] == (8 if weights == "half" else 7)
    assert got[2]["stale_recomputes"] > 0 and got[2]["compactions"] == (1 if ncell > 2048 else 0)
    assert _same(got, O.join_indel(codes, nstate, w))


def test_staged_bitsets_then_resident_codes(gpu_lib, monkeypatch):
    codes, ns, w = _indel(4500, 700, 8, "half", 4)
    got = gpu_lib.join_indel(codes, ns, w)
    assert got[2]["scan_path"] == 1 and got[2]["kernel_launches"] == 8 and got[2]["compactions"] > 0
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    assert _same(got, gpu_lib.join_indel(codes, ns, w))


# Ordered binary32 sums with the columns in global memory: too many words for
# shared memory throughout (1,100 x 8,192, compacted once), or until a
# compaction (3,500 x 2,560).
def test_bit_columns_in_global_memory(gpu_lib):
    words, w = _bit(1100, 8192, "float", 7)
    got = gpu_lib.join_bit(words, w, 1)
    assert got[2]["scan_path"] == 0 and got[2]["kernel_launches"] == 5 and got[2]["compactions"] > 0
    assert _same(got, O.join_bit(words, w, 1))


def test_bit_columns_move_to_shared_memory(gpu_lib, monkeypatch):
    words, w = _bit(3500, 2560, "float", 8)
    got = gpu_lib.join_bit(words, w, 0)
    assert got[2]["scan_path"] == 0 and got[2]["kernel_launches"] == 5 and got[2]["compactions"] > 0
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    assert _same(got, gpu_lib.join_bit(words, w, 0))


def test_bit_columns_resident_from_the_start(gpu_lib):
    words, w = _bit(1500, 320, "float", 9)
    got = gpu_lib.join_bit(words, w, 0)
    assert got[2]["scan_path"] == 1 and _same(got, O.join_bit(words, w, 0))


# The cluster's line in cells x edited sites: 26,000,000 with unit weights and
# 4,000,000 with other integers while at most 0.8 of the known sites are edited,
# falling to 6,000,000 and 1,200,000 where all are; fractional weights leave it
# where more than 0.7 are edited, beyond 35,000 cells or 18,000,000.  (Only the
# engine of all SMs has refresh phases, and only the column scan path 0.)
@pytest.mark.parametrize("ncell,nsite,weights,edited,missing,on_cluster", [
    (13500, 2048, "unit", 0.60, 0.0, True), (13500, 2048, "unit", 0.82, 0.0, True),
    (13500, 2048, "unit", 0.86, 0.0, False), (13500, 2048, "unit", 0.50, 0.5, False),
    (12000, 520, "unit", 0.94, 0.06, True),
    (5000, 1000, "integer", 0.75, 0.0, True), (5000, 1000, "integer", 0.81, 0.0, False),
    (5000, 1000, "integer", 0.30, 0.7, False), (2000, 601, "integer", 0.98, 0.02, True),
    (36000, 20, "half", 0.60, 0.1, True), (36000, 20, "half", 0.80, 0.1, False),
    (9000, 2100, "half", 0.90, 0.0, True), (9000, 2100, "half", 0.97, 0.0, False)])
def test_indel_engine_follows_the_edited_sites(gpu_lib, monkeypatch, ncell, nsite, weights, edited, missing, on_cluster):
    ns = 20
    rng = np.random.default_rng(11)
    base = rng.integers(2, ns + 2, size=(500, nsite), dtype=np.uint32)
    codes = base[rng.integers(0, len(base), size=ncell)]
    u = rng.random(codes.shape)
    codes[u >= edited] = 1
    codes[u >= 1.0 - missing] = 0
    w = {"unit": np.ones((ns, nsite)), "integer": rng.integers(1, 3, size=(ns, nsite)).astype(float),
         "half": rng.uniform(0.01, 4.0, size=(ns, nsite))}[weights]
    got = gpu_lib.join_indel(codes, ns, w)
    if weights == "half":
        assert (got[2]["scan_path"] == 1) == on_cluster
    else:
        assert got[2]["scan_path"] == 1 and (got[2]["refreshes"] == 0) == on_cluster
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    other = gpu_lib.join_indel(codes, ns, w)
    assert other[2]["refreshes"] > 0 and _same(got, other)


# Fractional weights: a cluster up to 90,000 cells.
@pytest.mark.parametrize("ncell,launches", [(90000, 5), (90001, 6)])
def test_fractional_bit_engine_follows_the_cells(gpu_lib, ncell, launches):
    rng = np.random.default_rng(2)
    words = rng.integers(0, 1 << 31, size=(2000, 1), dtype=np.uint32)[rng.integers(0, 2000, size=ncell)]
    words ^= np.uint32(1) << rng.integers(0, 32, size=(ncell, 1), dtype=np.uint32)
    got = gpu_lib.join_bit(words, rng.uniform(0.01, 3.0, size=32), 1)
    assert got[2]["kernel_launches"] == launches and got[2]["joins"] == ncell - 1


# Integer weights of several planes: a cluster up to 4,500,000 cells x planes x
# words, the words in blocks of eight.
@pytest.mark.parametrize("ncell,nsite,top,launches", [
    (9375, 992, 1 << 14, 5), (9376, 992, 1 << 14, 6), (9376, 992, (1 << 14) - 1, 5), (20000, 288, 1 << 14, 6),
    (37500, 256, 1 << 14, 5), (37501, 256, 1 << 14, 6), (300, 14368, 4, 5)])
def test_plane_bit_engine_follows_planes_and_words(gpu_lib, monkeypatch, ncell, nsite, top, launches):
    words = synth.binary_workload(ncell, nsite, 16, 0.04, 0.05, seed=ncell)
    w = np.zeros(nsite)
    w[:3] = 1, 2, top
    work = ncell * int(top).bit_length() * (-(-words.shape[1] // 8) * 8)
    assert (work <= 4500000) == (launches == 5)
    got = gpu_lib.join_bit(words, w, 1)
    assert got[2]["kernel_launches"] == launches
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    assert _same(got, gpu_lib.join_bit(words, w, 1))


# Wide rows are shared out among a query's warps (from 128 words, with planes from
# 64) while there are fewer groups of 32 slots than warps: sizes on both sides of the
# lines, rows that end within a block of eight words, groups part filled and CTAs
# without a slot, and ranges that reach fewer groups only by a compaction.
@pytest.mark.parametrize("weights,ncell,nsite", [
    ("unit", 9, 4096), ("unit", 333, 4064), ("unit", 333, 4096), ("unit", 1000, 4128), ("unit", 520, 9632),
    ("unit", 9000, 4160), ("planes", 9, 2048), ("planes", 333, 2016), ("planes", 333, 2080), ("planes", 1200, 4000),
    ("planes", 17, 30016)])
def test_wide_rows_on_a_cluster(gpu_lib, monkeypatch, weights, ncell, nsite):
    words, w = _bit(ncell, nsite, weights, ncell + nsite)
    got = gpu_lib.join_bit(words, w, 1)
    assert got[2]["kernel_launches"] == (6 if ncell == 9000 else 5)
    if ncell <= 1200:
        assert _same(got, O.join_bit(words, w, 1))
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    assert _same(got, gpu_lib.join_bit(words, w, 1))


# A replicate's columns stay in global memory at first; clusters of every size.
@pytest.mark.parametrize("mult", [1, 3])
@pytest.mark.parametrize("group", [1, 2, 8])
def test_wide_rows_of_replicates(gpu_lib, monkeypatch, mult, group):
    ncell, nsite, sizes = 1500, 12000, [2, 33, 290, 512, 700, 1500]
    words = synth.binary_workload(ncell, nsite, 14, 0.03, 0.05, seed=2)
    rng = np.random.default_rng(4)
    w = np.stack([np.bincount(rng.integers(0, nsite, nsite), minlength=words.shape[1] * 32) for _ in sizes]) * float(mult)
    cells = [np.sort(rng.permutation(ncell)[:n]) for n in sizes]
    full = gpu_lib.join_bit(words, None, 1)[0]
    monkeypatch.setenv("CASPHY_BS_GROUP", str(group))
    got = gpu_lib.bootstrap_bit(words, full, np.concatenate([[0], np.cumsum(sizes)]), np.concatenate(cells), w, raw_edges=True)
    assert got["stats"]["max_ctas_per_rep"] == group
    monkeypatch.setenv("CASPHY_JOIN_ENGINE", "grid")
    for r, n in enumerate(sizes):
        edge = gpu_lib.join_bit(np.ascontiguousarray(words[cells[r]]), w[r], 1)[0]
        ncol = (n + 31) // 32
        a = B.clade_bits(edge, n, ncol)
        b = B.clade_bits(got["raw_edges"][r].reshape(-1, 2), n, ncol)
        assert np.array_equal(np.unique(a, axis=0), np.unique(b, axis=0)), n
