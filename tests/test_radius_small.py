"""DNA radius searches on either side of the line between popcounts and tensor
core tiles (16,000,000 row pairs x plane words), and calls of no rows."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _raw(ntip, nsite, codes, seed):
    rng = np.random.default_rng(seed)
    base = rng.choice([1, 2, 4, 8], size=nsite)
    b = np.where(rng.random((ntip, nsite)) < 0.2, rng.choice([1, 2, 4, 8], size=(ntip, nsite)), base)
    b = np.where(rng.random(b.shape) < 0.05, 0x10, b)
    if codes != "bases":
        b = np.where(rng.random(b.shape) < 0.2, 0x0F, b)
    if codes == "ambiguous":
        b = np.where(rng.random(b.shape) < 0.05, rng.choice([3, 5, 6, 9, 10, 12, 7, 11, 13, 14], size=b.shape), b)
    raw = np.zeros((ntip, (nsite + 3) // 4 * 4), np.uint8)
    raw[:, :nsite] = b
    return raw.view(np.uint32)


# 2,000 x 31 is the line itself; the tiles: rows about multiples of 128 and 256,
# one block of positions and several, the N positions' chunk full and not
@pytest.mark.parametrize("codes", ["bases", "n", "ambiguous"])
@pytest.mark.parametrize("ntip,nsite", [(2000, 31), (2001, 31), (2049, 129), (1023, 257), (640, 700), (1281, 514)])
def test_dna_on_both_sides_of_the_line(gpu_lib, codes, ntip, nsite):
    raw = _raw(ntip, nsite, codes, ntip + nsite)
    words = ntip * ntip * 4 * (-(-nsite // 32))
    assert (words <= 16000000) == (ntip == 2000)
    for radius in (int(0.7 * nsite), nsite):
        c1, i1 = gpu_lib.radius_dna(raw, radius)
        c0, i0 = O.radius_dna(raw, radius)
        assert np.array_equal(c1, c0) and np.array_equal(i1, i0)
    lo, hi = ntip // 3, ntip - 5
    c2, i2 = gpu_lib.radius_dna_rows(raw, nsite, lo, hi)
    off = np.concatenate([[0], np.cumsum(c0.astype(np.int64))])
    assert np.array_equal(c2, c0[lo:hi]) and np.array_equal(i2, i0[off[lo]:off[hi]])


def test_transfer_of_one_side_only(gpu_lib):
    y = np.random.default_rng(1).integers(0, 1 << 32, size=(70, 3), dtype=np.uint64).astype(np.uint32)
    none = np.zeros((0, 3), np.uint32)
    for a, b in ((y, none), (none, y), (none, none)):
        for got, want in zip(gpu_lib.transfer_dis(a, b, 90), O.transfer_dis(a, b, 90)):
            assert np.array_equal(got, want)


def test_transfer_rows_in_panels(gpu_lib):
    """520 rows of 32,768 words, more than the 64 MiB panel that rows for the tiles come
    through: so few blocks take the popcounts, which need both sides whole."""
    rng = np.random.default_rng(3)
    nb = 32768
    y = rng.integers(0, 1 << 32, size=(520, nb), dtype=np.uint64).astype(np.uint32)
    x = y[rng.integers(0, 520, size=37)].copy()
    x[::2, :100] ^= np.uint32(1)
    for got, want in zip(gpu_lib.transfer_dis(y, x, 32 * nb), O.transfer_dis(y, x, 32 * nb)):
        assert np.array_equal(got, want)
    for got, want in zip(gpu_lib.transfer_dis(x, y, 32 * nb), O.transfer_dis(x, y, 32 * nb)):
        assert np.array_equal(got, want)
