// How the L-BFGS steps of n elements are shared out on one thread-block
// cluster: elements in blocks of 512, block b to CTA b mod ctas.
//
// Every CTA of the cluster owns at least one block.  The reductions have two
// buffers and no other flow control: a CTA may send the sums of epoch e + 2
// because it has received those of e + 1 from every CTA, so all of them are
// done with e.  A CTA without a block would send nothing, nobody would wait for
// it, and one that fell two epochs behind would find its barrier's bytes of two
// epochs mixed and wait until its limit.
#pragma once
#include <algorithm>
#include <cstdint>

namespace casphy {
namespace fel {

constexpr uint32_t kLbThreads = 512;
constexpr uint32_t kLbCluster = 16;    // CTAs, at most
constexpr uint32_t kLbMaxBlocks = 160;
constexpr uint32_t kLbMaxPerCta = 10;

struct LbPlan {
    uint32_t blocks, ctas, perCta;  // perCta: blocks of a CTA, at most
};

// The cluster for n >= 1 elements: a power of two of CTAs, no more than blocks.
inline LbPlan lb_plan(uint32_t n) {
    LbPlan p{(n + kLbThreads - 1) / kLbThreads, kLbCluster, 0};
    while (p.ctas > p.blocks) p.ctas /= 2;
    p.perCta = (p.blocks + p.ctas - 1) / p.ctas;
    return p;
}

}  // namespace fel
}  // namespace casphy
