"""Batched bootstrap where its kernels' tiles end: replicate sizes around the
128 x 256 tiles of the initial scan, and full trees past one window of the
bitmap that sorts a replicate's cells."""
import numpy as np
import pytest

import oracle as O
from casphy_b200 import bootstrap as B
from casphy_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbin", [1, 5, 9])
def test_replicate_sizes_around_tiles(gpu_lib, nbin):
    ncell, sizes = 600, [2, 3, 127, 128, 129, 255, 256, 257, 384, 385, 513, 600]
    rng = np.random.default_rng(nbin)
    words = synth.binary_workload(ncell, nbin * 32, 12, 0.03, 0.05, seed=nbin)
    words[rng.integers(0, ncell, 20)] = 0  # rows that share nothing
    full_edge, _, _ = O.join_bit(words, None, 1)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    cells = np.concatenate([np.sort(rng.permutation(ncell)[:n]) for n in sizes]).astype(np.uint32)
    ns = nbin * 32
    w = np.stack([np.bincount(rng.integers(0, ns, ns), minlength=ns) for _ in sizes]).astype(np.float64)
    got = gpu_lib.bootstrap_bit(words, full_edge, off, cells, w, raw_edges=True)
    ncol = (ncell + 31) // 32
    full_bits = B.clade_bits(full_edge, ncell, ncol)
    for r, n in enumerate(sizes):
        c = cells[off[r]:off[r + 1]]
        edge, _, _ = O.join_bit(np.ascontiguousarray(words[c]), w[r], 1)
        a = B.clade_bits(edge, n, ncol, tip_map=c)
        b = B.clade_bits(got["raw_edges"][r].reshape(-1, 2), n, ncol, tip_map=c)
        assert np.array_equal(np.unique(a, axis=0), np.unique(b, axis=0)), f"replicate of {n} cells differs"
        ymin, ysize = B.plain_replicate(O, words, full_bits, c, w[r])
        assert np.array_equal(got["ymin"][r], ymin) and np.array_equal(got["ysize"][r], ysize)


@pytest.mark.parametrize("ntip", [262144, 262145, 300001])
def test_full_tree_past_one_window(gpu_lib, ntip):
    rng = np.random.default_rng(ntip)
    words = rng.integers(0, 2**32, size=(ntip, 1), dtype=np.uint64).astype(np.uint32)
    # nodes joined first come, first served: a balanced tree over shuffled tips
    queue = np.concatenate([rng.permutation(ntip), np.arange(ntip, 2 * ntip - 1)])
    full_edge = np.empty((2 * ntip - 2, 2), np.uint32)
    full_edge[:, 0] = ntip + np.arange(2 * ntip - 2) // 2
    full_edge[:, 1] = queue[:2 * ntip - 2]
    cells = np.sort(rng.permutation(ntip)[:300]).astype(np.uint32)
    w = np.ones((1, 32))
    got = gpu_lib.bootstrap_bit(words, full_edge, [0, 300], cells, w)
    nodes = np.concatenate([np.arange(2 * ntip - 10, 2 * ntip - 2), rng.integers(ntip, 2 * ntip - 2, 20)])
    bits = np.zeros((len(nodes), (ntip + 31) // 32), np.uint32)
    for i, v in enumerate(nodes):
        front = np.array([v])
        while (front >= ntip).any():
            inner = front[front >= ntip] - ntip
            front = np.concatenate([front[front < ntip], queue[2 * inner], queue[2 * inner + 1]])
        np.bitwise_or.at(bits[i], front // 32, (1 << (front % 32)).astype(np.uint32))
    ymin, ysize = B.plain_replicate(gpu_lib, words, bits, cells, w[0])
    assert np.array_equal(got["ymin"][0, nodes - ntip], ymin)
    assert np.array_equal(got["ysize"][0, nodes - ntip], ysize)
    with pytest.raises(gpu_lib.CasphyError):
        gpu_lib.bootstrap_bit(words, full_edge, [0, 3], [cells[5], 7, cells[5]], w)


def test_replicate_past_the_shared_offsets(gpu_lib):
    """All cells with unit weights: the replicate's tree is the full tree, so
    every clade is at distance 0."""
    rng = np.random.default_rng(1)
    n = 53600
    words = synth.binary_workload(n, 64, 16, 0.03, 0.05, seed=1)
    full_edge, _, _ = gpu_lib.join_bit(words, None, 1)
    got = gpu_lib.bootstrap_bit(words, full_edge, [0, n], np.arange(n, dtype=np.uint32), np.ones((1, words.shape[1] * 32)))
    assert not got["ymin"].any() and got["ysize"].all() and (got["support"] == 1).all()
    with pytest.raises(gpu_lib.CasphyError):
        cells = np.arange(57857, dtype=np.uint32)
        edge = np.stack([57857 + np.arange(2 * 57856) // 2, np.arange(2 * 57856)], 1).astype(np.uint32)
        gpu_lib.bootstrap_bit(rng.integers(0, 9, (57857, 1)).astype(np.uint32), edge, [0, 57857], cells, np.ones((1, 32)))
