"""Host arrays on either side of the line between the driver's copies and the
copy threads (10 MiB), up and down, with slots (1 MiB) filled and part filled."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LINE = 10 << 20


@pytest.mark.parametrize("nbytes", [LINE - 4, LINE, LINE + 4, LINE + (1 << 20) + 12, 41 << 20])
def test_uploads(gpu_lib, nbytes):
    """One-word clades against the clade of no tip: a row's distance is the popcount of
    it or of its complement, and so is its size."""
    n = nbytes // 4
    y = np.random.default_rng(nbytes).integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    ymin, ysize, xmin, _ = gpu_lib.transfer_dis(y[:, None], np.zeros((1, 1), np.uint32), 32)
    pop = np.unpackbits(y.view(np.uint8)).reshape(n, 32).sum(1).astype(np.uint32)
    assert np.array_equal(ymin, np.minimum(pop, 32 - pop))
    assert np.array_equal(ysize, np.minimum(pop, 32 - pop))
    assert xmin[0] == min(pop.min(), 32 - pop.max())


@pytest.mark.parametrize("n", [1200, 1619, 1620, 3001])
def test_downloads(gpu_lib, n):
    """Lists of n neighbours of every row; 1,619^2 ids are the last below the line."""
    assert (4 * n * n >= LINE) == (n >= 1620)
    counts, idx = gpu_lib.radius_bit(np.full((1, n), 1, np.uint32), np.ones(32), 1)
    assert np.all(counts == n) and np.array_equal(idx.reshape(n, n), np.broadcast_to(np.arange(n), (n, n)))
