"""Transfer distances on either side of the lines between popcounts and tensor-core
tiles (100,000,000 row pairs x words, 240 blocks of 32 x 64 rows), and the
popcounts at the edges of their blocks."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _sides(ny, nx, nb):
    rng = np.random.default_rng(ny + nx + nb)
    y = rng.integers(0, 1 << 32, size=(ny, nb), dtype=np.uint64).astype(np.uint32)
    x = rng.integers(0, 1 << 32, size=(nx, nb), dtype=np.uint64).astype(np.uint32)
    x[::3] = y[rng.integers(0, ny, size=len(x[::3]))]
    x[::6, 0] ^= np.uint32(5)
    y[::2, -1] &= np.uint32(0x1FFFFFF)  # some rows keep bits past the tips
    return y, x, 32 * nb - 7


def _check(gpu_lib, y, x, ntip):
    for got, want in zip(gpu_lib.transfer_dis(y, x, ntip), O.transfer_dis(y, x, ntip)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("ny,nx,nb", [
    (1, 1, 1), (7, 9, 2), (64, 32, 32), (65, 33, 33), (63, 31, 31), (120, 257, 65), (3, 1000, 40), (1000, 3, 40)])
def test_popcounts(gpu_lib, ny, nx, nb):
    _check(gpu_lib, *_sides(ny, nx, nb))


@pytest.mark.parametrize("ny,nx,nb,tiles", [
    (1025, 1153, 84, False), (1025, 1153, 85, True), (10007, 999, 10, False), (10007, 1003, 10, True),
    (1024, 480, 300, False), (1025, 480, 300, True), (1024, 481, 300, True), (385, 1283, 401, True)])
def test_both_sides_of_the_lines(gpu_lib, ny, nx, nb, tiles):
    assert tiles == (ny * nx * nb > 100_000_000 and -(-nx // 32) * -(-ny // 64) > 240)
    _check(gpu_lib, *_sides(ny, nx, nb))


def test_tile_rows_in_panels(gpu_lib):
    """Rows for the tiles come through a 64 MiB panel: 2,900 rows of 6,016 words take
    two, the other side one."""
    y, x, ntip = _sides(2900, 170, 6016)
    _check(gpu_lib, y, x, ntip)
    y, x, ntip = _sides(340, 2900, 6016)
    _check(gpu_lib, y, x, ntip)
