"""Levels near the root: one launch for all of them up to as many sites as the
device holds at once (two CTAs of 32 sites an SM), a launch each beyond; every
bit is the same."""
import numpy as np
import pytest

from casphy_b200 import synth

pytestmark = pytest.mark.gpu
PI = [0.3, 0.2, 0.2, 0.3]


def _problem(model, ntip, nsite):
    if model == "hky85":
        s, (par, ch, t) = synth.hky85_alignment(ntip, nsite, 4.0, PI, 0.05, 0.02, seed=ntip)
        return np.stack([par, ch], axis=1).astype(np.uint32), synth.dna_nibbles(s), t, dict(kappa=4.0, pi=PI)
    codes, (par, ch, t) = synth.edit_alignment(ntip, nsite, 1.0, 30, 1.5, 0.15, 0.1, seed=ntip)
    return np.stack([par, ch], axis=1).astype(np.uint32), codes, t, \
        dict(model="irreversible", rate=1.0, nallele=int(codes.max()) - 1)


@pytest.mark.parametrize("model", ["hky85", "irreversible"])
@pytest.mark.parametrize("ntip", [2, 40, 150])
def test_levels_follow_the_sites(gpu_lib, model, ntip):
    import torch
    most = 2 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    edge, codes, t, kw = _problem(model, ntip, most + 1)
    launches = []
    for nsite in (most, most + 1):
        _, st = gpu_lib.felsenstein_optimize(edge, t, codes[:, :nsite], max_iter=1, rel_tol=0.0, **kw)
        launches.append(st["launches_per_eval"])
        levels = st["levels_inside"]
    # transition matrices, log L, two sums; a launch per level and direction
    assert launches[1] == 4 + 2 * levels
    assert launches[0] == 6 if ntip <= 64 else launches[0] < launches[1]
    # site chunks below the line take the narrow levels, the whole does not
    per_site = (ntip - 1) * (36 if model == "hky85" else 32)
    a = gpu_lib.felsenstein_loglik(edge, t, codes, grad=True, **kw)
    b = gpu_lib.felsenstein_loglik(edge, t, codes, grad=True, mem_budget=per_site * 1024, **kw)
    assert a[0] == b[0] and np.array_equal(a[1], b[1])
