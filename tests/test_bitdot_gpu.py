"""Shared-bit counts on the tensor cores (radius search, transfer distance) at
the edges of their tiles: rows around multiples of 128 and 256, words that do
not fill a 128-bit chunk, thresholds at the counts' ends, and the three kinds
of DNA codes (bases and gaps, N, other ambiguity codes)."""
import numpy as np
import pytest

import oracle as O
from casphy_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncell,nsite,radius", [
    (2, 32, 1), (127, 64, 5), (128, 128, 10), (129, 160, 11), (255, 480, 60), (257, 512, 70), (513, 544, 0),
    (641, 96, 1000), (1025, 1024, 150)])
def test_radius_bit_tiles(gpu_lib, ncell, nsite, radius):
    words = synth.binary_workload(ncell, nsite, 14, 0.03, 0.05, seed=ncell)
    bmat = np.ascontiguousarray(words.T)
    w = np.ones(bmat.shape[0] * 32)
    c1, i1 = gpu_lib.radius_bit(bmat, w, radius)
    c0, i0 = O.radius_bit(bmat, w, radius)
    assert np.array_equal(c1, c0) and np.array_equal(i1, i0)
    lo, hi = ncell // 3, ncell - ncell // 4
    c2, i2 = gpu_lib.radius_bit_rows(bmat, w, radius, lo, hi)
    off = np.concatenate([[0], np.cumsum(c0.astype(np.int64))])
    assert np.array_equal(c2, c0[lo:hi]) and np.array_equal(i2, i0[off[lo]:off[hi]])


@pytest.mark.parametrize("codes", ["bases", "n", "ambiguous"])
@pytest.mark.parametrize("ntip,nsite", [(3, 4), (130, 31), (256, 129), (515, 700)])
def test_radius_dna_codes(gpu_lib, codes, ntip, nsite):
    rng = np.random.default_rng(ntip + nsite)
    base = rng.choice([1, 2, 4, 8], size=nsite)
    b = np.where(rng.random((ntip, nsite)) < 0.2, rng.choice([1, 2, 4, 8], size=(ntip, nsite)), base)
    b = np.where(rng.random(b.shape) < 0.05, 0x10, b)
    if codes != "bases":
        b = np.where(rng.random(b.shape) < 0.2, 0x0F, b)
    if codes == "ambiguous":
        b = np.where(rng.random(b.shape) < 0.05, rng.choice([3, 5, 6, 9, 10, 12, 7, 11, 13, 14], size=b.shape), b)
    raw = np.zeros((ntip, (nsite + 3) // 4 * 4), np.uint8)
    raw[:, :nsite] = b
    raw = raw.view(np.uint32)
    for radius in (0, nsite // 2, int(0.7 * nsite), nsite):
        c1, i1 = gpu_lib.radius_dna(raw, radius)
        c0, i0 = O.radius_dna(raw, radius)
        assert np.array_equal(c1, c0) and np.array_equal(i1, i0)
    q = np.arange(0, ntip, 7, dtype=np.uint32)
    assert np.array_equal(gpu_lib.try_radius_dna(raw, nsite // 2, q), O.try_radius_dna(raw, nsite // 2, q))


@pytest.mark.parametrize("ny,nx,ntip", [(127, 129, 40), (8, 257, 100), (255, 5, 129), (256, 128, 500), (700, 513, 1000)])
def test_transfer_tiles(gpu_lib, ny, nx, ntip):
    rng = np.random.default_rng(ny + nx)
    nb = (ntip + 31) // 32
    y = rng.integers(0, 2**32, size=(ny, nb), dtype=np.uint64).astype(np.uint32)
    x = rng.integers(0, 2**32, size=(nx, nb), dtype=np.uint64).astype(np.uint32)
    x[::3] = y[rng.integers(0, ny, size=len(x[::3]))]
    if ntip % 32:  # clear the bits past the tips on most rows, keep some set
        keep = np.uint32((1 << (ntip % 32)) - 1)
        y[::2, -1] &= keep
        x[1::2, -1] &= keep
    for got, want in zip(gpu_lib.transfer_dis(y, x, ntip), O.transfer_dis(y, x, ntip)):
        assert np.array_equal(got, want)
