"""The L-BFGS steps on one cluster: every CTA that waits in a reduction is also
waited for, and the steps are the grid kernels' bit for bit.

A reduction has two buffers, one barrier each, and no flow control but this: a
CTA sends the sums of epoch e + 1 after it has received those of epoch e from
every CTA that sends any.  `_exchange` runs that protocol with one CTA held back
as long as the others can go on, and says whether it ends."""
import os
import subprocess

import numpy as np
import pytest

from casphy_b200 import synth

CSRC = os.path.join(os.path.dirname(__file__), "..", "casphy_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include "lbfgs_plan.h"
int main() {
    for (unsigned n = 1; n <= 148 * 512; n++) {
        const auto p = casphy::fel::lb_plan(n);
        std::printf("%u %u %u %u\\n", n, p.blocks, p.ctas, p.perCta);
    }
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    """n, blocks, CTAs, blocks per CTA of every problem a cluster may take."""
    d = tmp_path_factory.mktemp("lbfgs")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", str(d / "plan"), str(d / "plan.cpp")], check=True)
    out = subprocess.run([str(d / "plan")], check=True, capture_output=True, text=True).stdout
    return np.array(out.split(), np.int64).reshape(-1, 4)


def test_every_cta_owns_a_block(plans):
    n, blocks, ctas, per = plans.T
    assert np.array_equal(blocks, -(-n // 512))
    assert np.all((ctas >= 1) & (ctas <= 16) & (ctas & (ctas - 1) == 0))
    assert np.all(ctas <= blocks)  # block r belongs to CTA r
    assert np.all(ctas * per >= blocks) and np.all(ctas * (per - 1) < blocks)
    assert per.max() <= 10 and blocks.max() <= 160
    assert np.all((2 * ctas > blocks) | (ctas == 16))  # and no fewer CTAs than that allows


def _exchange(blocks, ctas, late, epochs=6):
    """True when all CTAs finish `epochs` reductions with CTA `late` running
    only while no other can.  A barrier holds (phase, arrivals, bytes owed); a
    message completes on the phase that is open when it lands."""
    senders = [r for r in range(ctas) if r < blocks]
    phase = [[0, 0] for _ in range(ctas)]       # completed phases per barrier
    armed = [[False, False] for _ in range(ctas)]
    owed = [[0, 0] for _ in range(ctas)]        # expected minus received of the open phase
    pc, sent = [0] * ctas, [False] * ctas       # epoch, whether its sums have left

    def settle(r, b):
        if armed[r][b] and owed[r][b] == 0:
            phase[r][b] += 1
            armed[r][b] = False

    def step(r):
        e = pc[r]
        if e == epochs:
            return False
        b = e & 1
        if not sent[r]:
            armed[r][b] = True
            owed[r][b] += len(senders)
            settle(r, b)
            if r in senders:
                for t in range(ctas):
                    owed[t][b] -= 1
                    settle(t, b)
            sent[r] = True
            return True
        if (phase[r][b] & 1) != (e >> 1 & 1):   # parity wait: the phase of this epoch is complete
            pc[r], sent[r] = e + 1, False
            return True
        return False

    while True:
        if any([step(r) for r in range(ctas) if r != late]):
            continue
        if not step(late):
            return all(p == epochs for p in pc)


def test_a_late_cta_without_a_block_breaks_the_exchange():
    # 2,000 tips on sixteen CTAs: eight own a block, eight would only listen
    assert _exchange(8, 8, late=3) and _exchange(16, 16, late=15)
    assert not _exchange(8, 16, late=12)


def test_the_plans_exchange_ends_whoever_is_late(plans):
    for blocks, ctas in {(int(b), int(c)) for _, b, c, _ in plans if b <= 40}:
        assert all(_exchange(blocks, ctas, late) for late in range(ctas)), (blocks, ctas)


@pytest.mark.gpu
# edges 510, 514, 1,030, 3,998, 7,680, 8,190, 8,194, 20,002, 45,002: one block and
# a part, one to ten blocks a CTA, the last ones partly absent
@pytest.mark.parametrize("ntip", [20, 200, 256, 258, 516, 2000, 3841, 4096, 4098, 10002, 22502])
def test_cluster_steps_equal_grid_steps(gpu_lib, monkeypatch, plans, ntip):
    s, (par, ch, t) = synth.hky85_alignment(ntip, 8, 4.0, [0.3, 0.2, 0.2, 0.3], 0.05, 0.02, seed=ntip)
    edge, codes = np.stack([par, ch], axis=1).astype(np.uint32), synth.dna_nibbles(s)
    t0 = np.random.default_rng(ntip).uniform(0.3, 3.0, len(t)) * np.maximum(t, 1e-4)
    kw = dict(kappa=4.0, pi=[0.3, 0.2, 0.2, 0.3], max_iter=14, rel_tol=0.0)
    t1, st1 = gpu_lib.felsenstein_optimize(edge, t0, codes, **kw)
    assert st1["step_ctas"] == plans[len(edge) - 1, 2]
    monkeypatch.setenv("CASPHY_LBFGS", "grid")
    t2, st2 = gpu_lib.felsenstein_optimize(edge, t0, codes, **kw)
    assert st2["step_ctas"] == 0
    assert st1["iterations"] == st2["iterations"] > 0 and st1["evaluations"] == st2["evaluations"]
    assert st1["loglik_end"] == st2["loglik_end"] and np.array_equal(t1, t2)
