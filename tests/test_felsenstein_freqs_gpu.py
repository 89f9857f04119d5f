"""Allele frequencies and the code check of the edit model, taken on the
device: the same log L and gradient, bit for bit, as with the tips' counts
passed in, around the blocks of 32 sites and 256 tips and with more alleles
than fit the shared-memory counters."""
import numpy as np
import pytest

from casphy_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntip,nsite,nallele", [(2, 1, 1), (31, 33, 3), (257, 64, 40), (300, 31, 383), (300, 31, 384), (520, 40, 2000)])
def test_device_frequencies_equal_given_counts(gpu_lib, ntip, nsite, nallele):
    codes, (par, ch, t) = synth.edit_alignment(ntip, nsite, 1.0, nallele, 1.2, 0.1, 0.1, seed=ntip + nsite)
    codes[:, 0] = np.minimum(codes[:, 0], 1)  # a site without an allele
    edge = np.stack([par, ch], 1)
    freq = np.zeros((nsite, nallele + 1))
    for s in range(nsite):
        freq[s] = np.bincount(np.maximum(codes[:, s].astype(int) - 1, 0), minlength=nallele + 1)
    a = gpu_lib.felsenstein_loglik(edge, t, codes, model="irreversible", nallele=nallele, grad=True)
    b = gpu_lib.felsenstein_loglik(edge, t, codes, model="irreversible", nallele=nallele, allele_freq=freq, grad=True)
    assert a[0] == b[0] and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("given", [False, True])
def test_code_beyond_the_alleles(gpu_lib, given):
    codes, (par, ch, t) = synth.edit_alignment(300, 40, 1.0, 5, 1.2, 0.1, 0.1, seed=3)
    codes[299, 39] = 7
    freq = np.ones((40, 6)) if given else None
    with pytest.raises(gpu_lib.CasphyError) as e:
        gpu_lib.felsenstein_loglik(np.stack([par, ch], 1), t, codes, model="irreversible", nallele=5, allele_freq=freq)
    assert e.value.status == 2
