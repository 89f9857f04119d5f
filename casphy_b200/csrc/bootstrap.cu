// Batched bootstrap of the bit join with transfer support on B200.
//
// The reference bootstraps by re-running the whole pipeline once per
// replicate from R (vignettes/CasPhy.Rmd:255-291): columns are resampled with
// replacement and, for binary data, handed to joinEdgeBitReverse as integer
// site weights (idx2weight, src/functions.cpp:4485-4492); every replicate tree
// is cut into clades (nodeDesBig, src/functions.cpp:1277-1366) and compared
// with the full-data tree by the transfer distance of TransferDisStream
// (cu/TransferDisStream.cu:22-128); the support of a full-tree clade is the
// fraction of replicates whose normalised distance is <= threshold
// (cal.abs, R/bootstrap_functions.R:190-219).
//
// Here all replicates run in one pass:
//  0. k_bs_ranks: one block per replicate looks up its cells' places in the
//     full tree and sorts them (they are distinct: a bitmap and its running
//     counts).
//  1. k_bs_prep: one warp per (replicate, tip) gathers the tip's row of the
//     full matrix and builds the replicate's slot matrix and query entries.
//     When every replicate's weights sum to at most the site count (a
//     column resample does), each resampled column is repeated as often as
//     it was drawn (k_bs_gather) and scored with unit weights: the same
//     integer scores and per-column merges as weight w on one column, with
//     one entry per word instead of one per (word, weight bit plane).
//     Otherwise the weights are integer bit planes (the single join's
//     PLANES path).
//  2. The initial all-pairs scan of every replicate.  Unit weights (repeated
//     columns): shared-bit counts on the tensor cores, all replicates' tiles in
//     one grid (InitTile).  Bit planes: k_bs_init, popcounts, tiles of all
//     replicates drawn from one queue.
//  3. k_bs_join: one thread-block cluster per replicate, largest first, running
//     the cluster join engine.  The cluster size (one for all replicates) comes
//     from a cost model whose constants are fitted to the per-replicate times of
//     the previous call on the device (the autotuner): the size with the least
//     predicted makespan when the replicates are dealt, largest first, to the
//     clusters that the device holds at once.  CTA 0 then lays out the replicate
//     tree's post-order (heavier child first, so a walk needs a stack of at most
//     log2(n)+1).
//  4. k_bs_transfer: one thread per (full-tree clade X, replicate).  X is the
//     pre-order tip interval [lo, hi] of the full tree; walking the replicate
//     tree's post-order with a stack of |X n Y| counts gives, for every
//     replicate clade Y, d = |X| + |Y| - 2|X n Y| and the transfer distance
//     min(d, n - d) over the replicate's n tips.  This is the quantity
//     TransferDisStream computes for clade bitsets restricted to the
//     replicate's tips (its pad and group-of-8 arithmetic cancel when no row
//     has bits past the tips), in O(clades x nodes) instead of
//     O(clades x clades x words).
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <numeric>
#include <queue>
#include <vector>

#include "bitdot.cuh"
#include "join_bit_cluster.cuh"
#include "runtime.h"

namespace casphy {
namespace boot {

using namespace bitjoin;

constexpr u32 kOpInternal = 0x80000000u, kOpRoot = 0x40000000u;
constexpr u32 kXThreads = 128;  // clades per transfer block
constexpr u32 kStack = 32;      // post-order stack (heavier child first: <= log2(n)+1)
constexpr u32 kOpChunk = 2048;  // ops staged in shared memory per step

struct Rep {
    joinc::Args c;
    BitClusterArgs m;
    InitArgs init;
    u32 off;        // first tip in the concatenated cell list
    u32* colT;
    u32* ops;       // 2n-1 post-order ops
    u32* eW;
    u32* eQ;
    u32* eLen;
    u32 eStride;
    uint4* chunks;  // unit weights: the rows as [128-bit chunk][tip], else null
};

// Places of the replicates' cells in the full tree's tip order, as listed and
// sorted.  Block r is replicate r; a window of kRankWords words of the bitmap is
// in shared memory at a time.  (64 replicates of 1,667 to 5,000 cells took a
// host thread 9.5 ms to sort; this takes 12 us.)
constexpr u32 kRankThreads = 512, kRankWords = 8192;
__global__ void __launch_bounds__(kRankThreads) k_bs_ranks(const u32* __restrict__ repOff, const u32* __restrict__ repN,
                                                           const u32* __restrict__ cells,
                                                           const u32* __restrict__ rank, u32 ntip, u32* repOfWarp,
                                                           u32* rankOf, u32* sortedRank, int* twice) {
    __shared__ u32 s_bits[kRankWords];
    __shared__ u32 s_warp[kRankThreads / 32];
    const u32 r = blockIdx.x, off = repOff[r], n = repN[r];
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (u32 i = tid; i < n; i += kRankThreads) {
        repOfWarp[off + i] = r;
        rankOf[off + i] = rank[cells[off + i]];
    }
    u32 done = 0;
    for (u32 lo = 0; lo < ntip; lo += 32 * kRankWords) {
        const u32 words = (min(ntip - lo, 32 * kRankWords) + 31u) / 32u;
        for (u32 w = tid; w < words; w += kRankThreads) s_bits[w] = 0u;
        __syncthreads();
        for (u32 i = tid; i < n; i += kRankThreads) {  // (each thread reads what it wrote)
            const u32 x = rankOf[off + i] - lo;
            if (x < 32 * words && (atomicOr(&s_bits[x / 32], 1u << (x & 31u)) >> (x & 31u) & 1u)) *twice = 1;
        }
        __syncthreads();
        const u32 per = (words + kRankThreads - 1) / kRankThreads;
        const u32 w0 = min(tid * per, words), w1 = min(w0 + per, words);
        u32 mine = 0;
        for (u32 w = w0; w < w1; w++) mine += (u32)__popc(s_bits[w]);
        u32 scan = mine;
        for (u32 o = 1; o < 32; o <<= 1) {
            const u32 y = __shfl_up_sync(0xFFFFFFFFu, scan, o);
            if (lane >= o) scan += y;
        }
        if (lane == 31) s_warp[warp] = scan;
        __syncthreads();
        u32 before = done, total = 0;
        for (u32 k = 0; k < kRankThreads / 32; k++) {
            if (k < warp) before += s_warp[k];
            total += s_warp[k];
        }
        u32 pos = off + before + scan - mine;
        for (u32 w = w0; w < w1; w++)
            for (u32 b = s_bits[w]; b; b &= b - 1u) sortedRank[pos++] = lo + 32 * w + (u32)__ffs(b) - 1u;
        done += total;
        __syncthreads();  // the next window clears the bitmap
    }
}

// Resampled rows: bit b of word j of (replicate r, tip) is the full row's
// bit colIdx[r][32j+b] (kNone pads).  One warp per (replicate, tip).
__global__ void k_bs_gather(const u32* __restrict__ repOfWarp, const u32* __restrict__ cells,
                            const u32* __restrict__ words, const u32* __restrict__ colIdx, u32 nbin, u32 totalTips,
                            u32* __restrict__ rows) {
    const u32 warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= totalTips) return;
    const u32* src = words + (size_t)cells[warp] * nbin;
    const u32* ci = colIdx + (size_t)repOfWarp[warp] * nbin * 32;
    for (u32 j = lane; j < nbin; j += 32) {
        u32 v = 0;
#pragma unroll 8
        for (u32 b = 0; b < 32; b++) {
            const u32 c = ci[32 * j + b];
            if (c != kNone) v |= ((__ldg(src + (c >> 5)) >> (c & 31)) & 1u) << b;
        }
        rows[(size_t)warp * nbin + j] = v;
    }
}

// One warp per (replicate, tip); rows: the resampled rows by warp, or null
// to read the full rows.
__global__ void k_bs_prep(const Rep* __restrict__ reps, const u32* __restrict__ repOfWarp,
                          const u32* __restrict__ cells, const u32* __restrict__ words, const u32* __restrict__ rows,
                          u32 nbin, u32 totalTips) {
    const u32 warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= totalTips) return;
    const u32 r = repOfWarp[warp];
    const Rep& R = reps[r];
    const u32 tip = warp - R.off;
    const u32 cell = cells[warp];
    prep_tip(rows ? rows + (size_t)warp * nbin : words + (size_t)cell * nbin, tip, nbin, R.m.nbinP,
             (R.c.ntip + 7u) & ~7u, R.m.nplanes,
             R.m.planeMask, R.m.nodeSeq, R.m.nodeBis, R.colT, R.eW, R.eQ, R.eLen, R.eStride);
    // initial local maximum: value -1, node ~0 (replaced by the initial scan)
    if ((threadIdx.x & 31) == 0) R.init.initKey[tip] = ((u64)ORD_F32_NEG1 << 32) | 0xFFFFFFFFull;
    if (R.chunks) {
        const u32* row = rows + (size_t)warp * nbin;
        u32* c = reinterpret_cast<u32*>(R.chunks + tip);
        for (u32 w = threadIdx.x & 31; w < R.m.nbinP; w += 32)
            c[(size_t)(w / 4) * R.c.ntip * 4 + (w & 3u)] = w < nbin ? row[w] : 0u;
    }
}

// Initial scan of unit-weight replicates from the shared-bit counts: every
// row's best column above it, ties to the smaller.  A thread owns a row and a
// third of the tile's columns; one 64-bit maximum per thread and tile goes to
// memory.  (64 replicates of 1,667 to 5,000 cells x 512 sites: popcounts took
// 5.8 ms, this takes 0.37 ms.)
struct InitTile {
    static constexpr bool kBatched = true;
    struct Params {
        const Rep* reps;
        const u64* tileStart;  // replicate r's tiles from tileStart[r]
        u32 nrep;
        u64 first;             // tile of block 0
        unsigned long long* key;
    };
    __device__ static u32 pick(bitdot::Args& a, Params& p, u32 block) {
        const u64 t = p.first + block;
        u32 lo = 0, hi = p.nrep;  // tileStart[lo] <= t < tileStart[hi]
        while (hi - lo > 1) {
            const u32 mid = (lo + hi) / 2;
            if (p.tileStart[mid] <= t) lo = mid;
            else hi = mid;
        }
        const Rep& R = p.reps[lo];
        a.A = a.B = R.chunks;
        a.ldA = a.ldB = a.rowsA = a.rowsB = R.c.ntip;
        a.tilesN = (R.c.ntip + bitdot::kN - 1) / bitdot::kN;
        p.key = R.init.initKey;
        return (u32)(t - p.tileStart[lo]);
    }
    __device__ static void tile(const bitdot::Args& a, const Params& p, u32 m0, u32 n0, u32 taddr, unsigned char*) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wr = warp & 3u;
        const u32 q = m0 + 32 * wr + lane;
        int best = -1;
        u32 at = 0;
        for (u32 cb = warp >> 2; cb < bitdot::kN / 32; cb += bitdot::kThreads / 128) {
            const u32 n = n0 + cb * 32;
            if (n >= a.rowsB || n + 31 <= m0 + 32 * wr) continue;  // no column above any of the warp's rows
            u32 r[32];
            bitdot::load32(taddr + (32 * wr << 16) + cb * 32, r);
            if (n > m0 + 32 * wr + 31 && n + 32 <= a.rowsB) {
#pragma unroll
                for (u32 j = 0; j < 32; j++)
                    if ((int)r[j] > best) {
                        best = (int)r[j];
                        at = n + j;
                    }
            } else {
#pragma unroll
                for (u32 j = 0; j < 32; j++)
                    if ((int)r[j] > best && n + j > q && n + j < a.rowsB) {
                        best = (int)r[j];
                        at = n + j;
                    }
            }
        }
        if (best >= 0 && q < a.rowsA)
            atomicMax(p.key + q, (unsigned long long)make_key(ord_f32((float)(best / 8)), at));
    }
};

// initial scan with bit planes: tiles of all replicates from one queue
__global__ void __launch_bounds__(kThreads) k_bs_init(const Rep* __restrict__ reps, const u64* __restrict__ tileStart,
                                                      u32 nrep, unsigned long long* counter) {
    __shared__ unsigned long long s_tile[2];
    __shared__ u64 red[32];
    const u64 total = tileStart[nrep];
    if (threadIdx.x == 0) s_tile[0] = atomicAdd(counter, 1ull);
    __syncthreads();
    int cur = 0;
    for (;;) {
        const u64 t = s_tile[cur];
        if (t >= total) break;
        if (threadIdx.x == 0) s_tile[cur ^ 1] = atomicAdd(counter, 1ull);
        u32 lo = 0, hi = nrep;  // replicate r with tileStart[r] <= t < tileStart[r+1]
        while (hi - lo > 1) {
            const u32 mid = (lo + hi) / 2;
            if (tileStart[mid] <= t) lo = mid;
            else hi = mid;
        }
        init_tile<PATH_PLANES>(reps[lo].init, t - tileStart[lo], red);
        cur ^= 1;
        __syncthreads();
    }
}

// Post-order of the replicate tree (raw join edges: node ntip+k has children
// rawEdge[4k+1], rawEdge[4k+3]; the root is 2ntip-2), heavier child first.
// Tip ops carry the tip's full-tree pre-order rank; internal ops carry their
// tip count, the root is flagged.  Offsets go from parents to children, so one
// thread walks the nodes from the root down; what it reads of them is staged
// by the whole block, kOpsStage nodes at a time (read by the walking thread
// itself, two dependent loads a node, it took about 1 us a node).
constexpr u32 kOpsStage = 512;
struct OpsNode {
    u32 a, b, ta, tb, ra, rb;  // children, their tips and, for tips, their ranks
};
__host__ __device__ inline size_t ops_smem(u32 n) { return sizeof(OpsNode) * kOpsStage + sizeof(u32) * (size_t)n; }
constexpr size_t kOpsMost = 231424;  // bytes of a replicate's offsets, at most: 57,856 cells
// The offsets s: in shared memory after the stage or, for replicates beyond
// about 53,000 cells, in memory.
template <class S>
__device__ __forceinline__ void build_ops(const joinc::Args& c, const u32* __restrict__ rankOf, u32* ops, OpsNode* stage,
                                          S s) {
    const u32 n = c.ntip, root = 2 * n - 2;
    if (threadIdx.x == 0) s[root - n] = 0;
    for (u32 top = n - 1; top > 0;) {  // nodes n + top - 1 down
        const u32 m = min(kOpsStage, top);
        __syncthreads();
        for (u32 i = threadIdx.x; i < m; i += joinc::kThreads) {
            const u32 k = top - 1 - i;
            OpsNode o;
            o.a = ld_cg_u32(c.rawEdge + 4 * k + 1);
            o.b = ld_cg_u32(c.rawEdge + 4 * k + 3);
            o.ta = o.a < n ? 1u : ld_cg_u32(c.nodeSize + o.a);
            o.tb = o.b < n ? 1u : ld_cg_u32(c.nodeSize + o.b);
            if (o.tb > o.ta) {
                const u32 x = o.a; o.a = o.b; o.b = x;
                const u32 y = o.ta; o.ta = o.tb; o.tb = y;
            }
            o.ra = o.a < n ? rankOf[o.a] : 0u;
            o.rb = o.b < n ? rankOf[o.b] : 0u;
            stage[i] = o;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (u32 i = 0; i < m; i++) {
                const u32 k = top - 1 - i, tv = stage[i].ta + stage[i].tb;
                const OpsNode o = stage[i];
                const u32 base = s[k], sb = base + 2 * o.ta - 1;
                ops[base + 2 * tv - 2] = kOpInternal | (n + k == root ? kOpRoot : 0u) | tv;
                if (o.a < n) ops[base] = o.ra;
                else s[o.a - n] = base;
                if (o.b < n) ops[sb] = o.rb;
                else s[o.b - n] = sb;
            }
        top -= m;
    }
}

// Cluster i joins replicate order[i].
template <class Model>
__global__ void __launch_bounds__(joinc::kThreads, 1) k_bs_join(const Rep* __restrict__ reps,
                                                                const u32* __restrict__ order, u32 G,
                                                                const u32* __restrict__ rankOf,
                                                                const int* __restrict__ initErr, u32 opsShared) {
    extern __shared__ __align__(16) unsigned char smem[];
    const u32 r = order[blockIdx.x / G], rank = joinc::cluster_rank();
    if (*initErr) return;  // (an earlier kernel's: the same for all)
    const joinc::Args c = reps[r].c;
    const BitClusterArgs m = reps[r].m;
    const u64 t0 = globaltimer_ns();
    joinc::cluster_join<Model>(c, m, rank, smem);
    __syncthreads();
    if (rank != 0) return;
    int err = 0;
    if (threadIdx.x == 0) err = *(volatile int*)c.err;
    if (__syncthreads_or(err)) return;
    OpsNode* stage = reinterpret_cast<OpsNode*>(smem);
    if (opsShared) {
        build_ops(c, rankOf + reps[r].off, reps[r].ops, stage, reinterpret_cast<u32*>(smem + sizeof(OpsNode) * kOpsStage));
    } else {  // (the initial keys have been read)
        build_ops(c, rankOf + reps[r].off, reps[r].ops, stage,
                  reinterpret_cast<volatile u32*>(const_cast<unsigned long long*>(c.initKey)));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        c.statsOut[6] = t0;
        c.statsOut[7] = globaltimer_ns();
    }
}

// Transfer distances: grid (clade blocks, replicates).
struct XferArgs {
    u32 nX, nrep, fill;
    const u32* Xlo;
    const u32* Xhi;
    const u32* repN;       // tips per replicate
    const u32* repOff;     // first tip (sorted ranks) per replicate
    const u32* repOpsOff;  // first op per replicate
    const u32* sortedRank;
    const u32* ops;
    double threshold;
    u32* ymin;   // nrep x nX
    u32* ysize;  // nrep x nX
    u32* support;
    int* err;
};

__device__ __forceinline__ u32 lower_bound_u32(const u32* a, u32 n, u32 v) {
    u32 lo = 0, hi = n;
    while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(kXThreads) k_bs_transfer(XferArgs a) {
    __shared__ u32 stack[kStack * kXThreads];
    __shared__ u32 sops[kOpChunk];
    const u32 r = blockIdx.y;
    const u32 x = blockIdx.x * kXThreads + threadIdx.x;
    const bool ok = x < a.nX;
    const u32 n = a.repN[r];
    const u32* srt = a.sortedRank + a.repOff[r];
    const u32* ops = a.ops + a.repOpsOff[r];
    const u32 lo = ok ? a.Xlo[x] : 1u, hi = ok ? a.Xhi[x] : 0u;
    const u32 nX = ok ? lower_bound_u32(srt, n, hi + 1) - lower_bound_u32(srt, n, lo) : 0u;
    u32 best = a.fill;
    u32 sp = 0;
    bool over = false;
    const u32 nops = 2 * n - 1;
    for (u32 o0 = 0; o0 < nops; o0 += kOpChunk) {
        const u32 m = min(kOpChunk, nops - o0);
        __syncthreads();
        for (u32 i = threadIdx.x; i < m; i += kXThreads) sops[i] = ops[o0 + i];
        __syncthreads();
        for (u32 i = 0; i < m; i++) {
            const u32 op = sops[i];
            if (!(op & kOpInternal)) {
                if (sp < kStack) stack[sp * kXThreads + threadIdx.x] = (op >= lo && op <= hi) ? 1u : 0u;
                else over = true;
                sp++;
            } else {
                if (sp < 2 || sp > kStack) {
                    over = true;
                    continue;
                }
                const u32 cnt = stack[(sp - 1) * kXThreads + threadIdx.x] + stack[(sp - 2) * kXThreads + threadIdx.x];
                sp--;
                stack[(sp - 1) * kXThreads + threadIdx.x] = cnt;
                if (!(op & kOpRoot)) {
                    const u32 sY = op & 0x3FFFFFFFu;
                    const u32 d = nX + sY - 2 * cnt;
                    const u32 t = min(d, n - d);
                    best = min(best, t);
                }
            }
        }
    }
    if (over && threadIdx.x == 0) atomicCAS(a.err, 0, CASPHY_EINTERNAL);
    if (!ok) return;
    const u32 ys = min(nX, n - nX);
    a.ymin[(size_t)r * a.nX + x] = best;
    a.ysize[(size_t)r * a.nX + x] = ys;
    if (ys > 0 && (double)best <= a.threshold * (double)ys) atomicAdd(a.support + x, 1u);
}

}  // namespace boot

using namespace boot;

static int full_tree_intervals(u32 ntip, const u32* edge, std::vector<u32>& Xlo, std::vector<u32>& Xhi,
                               std::vector<u32>& rank) {
    const u32 nn = 2 * ntip - 1, nedge = 2 * ntip - 2, none = 0xFFFFFFFFu;
    std::vector<u32> kidA(nn, none), kidB(nn, none);
    std::vector<unsigned char> isChild(nn, 0);
    for (u32 e = 0; e < nedge; e++) {
        const u32 p = edge[2 * e], c = edge[2 * e + 1];
        if (p >= nn || c >= nn || p < ntip || isChild[c]) return CASPHY_EINVAL;
        isChild[c] = 1;
        if (kidA[p] == none) kidA[p] = c;
        else if (kidB[p] == none) kidB[p] = c;
        else return CASPHY_EINVAL;
    }
    u32 root = none, nroot = 0;
    for (u32 v = 0; v < nn; v++)
        if (!isChild[v]) {
            root = v;
            nroot++;
        }
    if (nroot != 1 || root < ntip) return CASPHY_EINVAL;
    rank.assign(ntip, none);
    std::vector<u32> lo(nn, none), hi(nn, 0), stack{root}, post;
    post.reserve(nn);
    u32 next = 0;
    while (!stack.empty()) {
        const u32 v = stack.back();
        stack.pop_back();
        post.push_back(v);
        if (v < ntip) {
            rank[v] = next++;
        } else {
            if (kidB[v] == none) return CASPHY_EINVAL;
            stack.push_back(kidB[v]);
            stack.push_back(kidA[v]);
        }
        if (post.size() > nn) return CASPHY_EINVAL;
    }
    if (post.size() != nn || next != ntip) return CASPHY_EINVAL;
    for (auto it = post.rbegin(); it != post.rend(); ++it) {
        const u32 v = *it;
        if (v < ntip) {
            lo[v] = hi[v] = rank[v];
        } else {
            lo[v] = std::min(lo[kidA[v]], lo[kidB[v]]);
            hi[v] = std::max(hi[kidA[v]], hi[kidB[v]]);
        }
    }
    Xlo.clear();
    Xhi.clear();
    for (u32 v = ntip; v < nn; v++) {
        if (v == root) continue;
        Xlo.push_back(lo[v]);
        Xhi.push_back(hi[v]);
    }
    return CASPHY_OK;
}

}  // namespace casphy

namespace casphy {
namespace boot {

// Cost of joining one replicate of n cells with a cluster of G CTAs: its
// phases times (alpha + beta * n / G + gamma when G > 1) -- a fixed per-phase
// part, the scan of the slots each CTA owns, and the exchange between CTAs.
// The constants start from a B200 estimate and are refitted on every call from
// the measured replicate times, per device.
struct Tune {
    int measured = 0;
    double alpha = 2.2;        // us per phase
    double beta = 1.0e-3;      // us per phase per slot of a CTA
    double gamma = 0.6;        // us per phase for the exchange of a cluster
    double phasesPerTip = 1.5;
};
constexpr int kMaxDev = 64;
Tune g_tune[kMaxDev];  // read and written under the device's workspace lock

inline double cost_us(const Tune& T, u32 n, u32 G) {
    return T.phasesPerTip * n * (T.alpha + T.beta * (double)n / G + (G > 1 ? T.gamma : 0.0));
}

// Predicted time of all replicates, `sorted` by falling size, on `slots`
// clusters of G CTAs, each taking the next replicate when it is free.
inline double makespan_us(const Tune& T, const std::vector<u32>& sorted, u32 G, u32 slots) {
    std::priority_queue<double, std::vector<double>, std::greater<double>> freeAt;
    for (u32 i = 0; i < slots; i++) freeAt.push(0.0);
    double end = 0;
    for (u32 n : sorted) {
        const double t = freeAt.top() + cost_us(T, n, G);
        freeAt.pop();
        freeAt.push(t);
        end = std::max(end, t);
    }
    return end;
}

// Refits alpha and beta (single CTAs) or gamma and beta (clusters) by least
// squares of the per-phase time over the slots per CTA; keeps the previous
// value of a constant the measurements cannot pin down.
void refit(Tune& T, const std::vector<u32>& repN, u32 G, const std::vector<double>& us,
           const std::vector<unsigned long long>& phases) {
    double s1 = 0, sx = 0, sxx = 0, sy = 0, sxy = 0, ptot = 0, ntot = 0;
    for (size_t r = 0; r < repN.size(); r++) {
        if (phases[r] == 0 || us[r] <= 0) continue;
        ptot += (double)phases[r];
        ntot += repN[r];
        const double x = (double)repN[r] / G, y = us[r] / (double)phases[r];
        s1 += 1;
        sx += x;
        sxx += x * x;
        sy += y;
        sxy += x * y;
    }
    if (ntot > 0) T.phasesPerTip = ptot / ntot;
    const double det = s1 * sxx - sx * sx;
    if (s1 >= 8 && det > 0) {
        const double b = (s1 * sxy - sx * sy) / det, a = (sy - b * sx) / s1;
        if (a > 0 && b > 0) {
            if (G == 1) T.alpha = a;
            else T.gamma = std::max(0.1, a - T.alpha);
            T.beta = b;
            T.measured = 1;
        }
    }
}

}  // namespace boot
}  // namespace casphy

extern "C" int casphy_bootstrap_bit(uint32_t ntip, uint32_t nbin, const uint32_t* words, const uint32_t* full_edge,
                                    uint32_t nrep, const uint32_t* rep_offsets, const uint32_t* rep_cells,
                                    const double* rep_weights, int ancestralType, double threshold,
                                    uint32_t* support, uint32_t* ymin_out, uint32_t* ysize_out,
                                    uint32_t* rep_raw_edges, casphy_bootstrap_stats* stats) {
    using namespace casphy;
    int rc = require_device();
    if (rc) return rc;
    if (ntip < 3 || nbin == 0 || nbin > kMaxBin || !words || !full_edge || nrep == 0 || !rep_offsets || !rep_cells ||
        !rep_weights || !support || !(threshold >= 0)) {
        casphy_set_last_error_msg("bootstrap: bad arguments");
        return CASPHY_EINVAL;
    }
    std::vector<u32> Xlo, Xhi, rank;
    if ((rc = full_tree_intervals(ntip, full_edge, Xlo, Xhi, rank))) {
        casphy_set_last_error_msg("bootstrap: full_edge is not a binary tree over ntip tips");
        return rc;
    }
    const u32 nX = (u32)Xlo.size(), nsite = nbin * 32, nbinP = (nbin + 3u) & ~3u;
    // replicate sizes, weights -> bit planes
    std::vector<u32> repN(nrep), repOpsOff(nrep + 1, 0), nplanesOf(nrep);
    u32 nmax = 0, totalTips = rep_offsets[nrep] - rep_offsets[0];
    if (rep_offsets[0] != 0) return CASPHY_EINVAL;
    u32 P = 1;
    for (u32 r = 0; r < nrep; r++) {
        if (rep_offsets[r + 1] < rep_offsets[r]) return CASPHY_EINVAL;
        repN[r] = rep_offsets[r + 1] - rep_offsets[r];
        if (repN[r] < 2) {
            casphy_set_last_error_msg("bootstrap: every replicate needs at least 2 cells");
            return CASPHY_EINVAL;
        }
        nmax = std::max(nmax, repN[r]);
        repOpsOff[r + 1] = repOpsOff[r] + 2 * repN[r] - 1;
        double tot = 0;
        u32 maxw = 0;
        for (u32 i = 0; i < nsite; i++) {
            const double w = rep_weights[(size_t)r * nsite + i];
            if (!(w >= 0) || w != std::floor(w) || w >= 16777216.0) {
                casphy_set_last_error_msg("bootstrap: replicate weights must be non-negative integers");
                return CASPHY_EINVAL;
            }
            tot += w;
            maxw = std::max(maxw, (u32)w);
        }
        if (tot > 16777216.0) return CASPHY_ERANGE;
        u32 np = 0;
        while ((1u << np) <= maxw && np < 24) np++;
        P = std::max(P, std::max(np, 1u));
    }
    for (u32 i = 0; i < totalTips; i++)
        if (rep_cells[i] >= ntip) return CASPHY_EINVAL;
    // repeated columns when every replicate's draws fit the row, else planes
    bool repeat = true;
    for (u32 r = 0; r < nrep && repeat; r++) {
        double tot = 0;
        for (u32 i = 0; i < nsite; i++) tot += rep_weights[(size_t)r * nsite + i];
        repeat = tot <= (double)nsite;
    }
    std::vector<u32> colIdx;
    if (repeat) {
        P = 1;
        colIdx.assign((size_t)nrep * nsite, joinx::kNone);
        for (u32 r = 0; r < nrep; r++) {
            size_t pos = (size_t)r * nsite;
            for (u32 i = 0; i < nsite; i++)
                for (u32 c = (u32)rep_weights[(size_t)r * nsite + i]; c > 0; c--) colIdx[pos++] = i;
        }
    }
    const u32 nplanes = repeat ? 0u : P;
    std::vector<u32> planes((size_t)nrep * P * nbin, 0u);
    if (!repeat)
        for (u32 r = 0; r < nrep; r++)
            for (u32 i = 0; i < nsite; i++) {
                const u32 v = (u32)rep_weights[(size_t)r * nsite + i];
                for (u32 k = 0; k < P; k++)
                    if ((v >> k) & 1u) planes[((size_t)r * P + k) * nbin + i / 32] |= 1u << (i % 32);
            }
    const u32 eStride = nbin * P;
    // per-replicate layout in one arena
    DeviceScope ds;
    int nSM = 0;
    CASPHY_CUDA_TRY(cudaDeviceGetAttribute(&nSM, cudaDevAttrMultiProcessorCount, ds.dev));
    // CTAs per replicate from the device's cost model (one join CTA per SM):
    // every size whose shared memory fits the largest replicate
    boot::Tune& tune = boot::g_tune[(ds.dev >= 0 && ds.dev < boot::kMaxDev) ? ds.dev : 0];
    const int tunedBefore = tune.measured;
    int maxSmem = 0;
    CASPHY_CUDA_TRY(cudaDeviceGetAttribute(&maxSmem, cudaDevAttrMaxSharedMemoryPerBlockOptin, ds.dev));
    const size_t smemLim = (size_t)maxSmem - 6144;  // the kernel's static shared memory
    const auto joinFn = wide_rows(nbin, nplanes) ? k_bs_join<BitCluster<PATH_PLANES, true>>
                                                 : k_bs_join<BitCluster<PATH_PLANES>>;
    auto plan = [&](u32 n, u32 G, joinc::Args& a, BitClusterArgs& m, size_t* smem) {
        a.ntip = n;
        a.nnode = 2 * n - 1;
        a.G = G;
        a.R = ((n + G - 1) / G + 31u) & ~31u;
        a.deathWords = (a.nnode + 31) / 32;
        m.nbin = nbin;
        m.nbinP = nbinP;
        m.nplanes = nplanes;
        return a.R < 0xFFFFu && cluster_fit<PATH_PLANES>(a, m, smemLim, smem);
    };
    std::vector<u32> order(nrep), sorted(nrep);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](u32 a, u32 b) { return repN[a] > repN[b]; });
    for (u32 r = 0; r < nrep; r++) sorted[r] = repN[order[r]];
    if (4 * (size_t)nmax > kOpsMost) {
        casphy_set_last_error_msg("bootstrap: replicate too large");
        return CASPHY_ERANGE;
    }
    const u32 opsShared = ops_smem(nmax) <= smemLim ? 1u : 0u;
    const size_t opsBytes = opsShared ? ops_smem(nmax) : ops_smem(0);
    u32 G = 0, fixedG = 0;
    if (const char* env = std::getenv("CASPHY_BS_GROUP"))  // a fixed size, at most 8 (the cost model is bypassed)
        for (fixedG = 1; fixedG < 8 && (int)(2 * fixedG) <= std::atoi(env);) fixedG *= 2;
    double bestUs = 0;
    for (u32 g = 1; g <= joinc::kMaxG; g *= 2) {
        joinc::Args a{};
        BitClusterArgs m{};
        size_t sm = 0;
        if (!plan(nmax, g, a, m, &sm)) continue;
        sm = std::max(sm, opsBytes);
        const int slots = joinc::placeable((void*)joinFn, g, sm);
        if (slots < 1) continue;
        const double t = g == fixedG ? 0.0 : makespan_us(tune, sorted, g, (u32)slots);
        if (G == 0 || t < bestUs) {
            G = g;
            bestUs = t;
        }
    }
    if (G == 0) {
        casphy_set_last_error_msg("bootstrap: replicate too large for one cluster's shared memory");
        return CASPHY_ERANGE;
    }
    struct RepBufs {
        u32 *planeMask, *nodeSeq, *nodeBis, *colT0, *colT1, *nodeSize, *rawEdge;
        u32 *eW, *eQ, *eLen;
        uint4* chunks;
        unsigned long long* initKey;
        u64* chunkStart;
    };
    auto rep_layout = [&](Carve& c, u32 n) {
        RepBufs b{};
        const u32 Sp = (n + 7u) & ~7u, nnode = 2 * n - 1, nChunks = (n + kCap - 1) / kCap;
        b.planeMask = c.take<u32>((size_t)P * nbin);
        b.nodeSeq = c.take<u32>((size_t)nnode * nbinP);
        b.nodeBis = c.take<u32>((size_t)nnode * nbinP);
        b.colT0 = c.take<u32>((size_t)nbin * Sp);
        b.colT1 = c.take<u32>((size_t)nbin * Sp);
        b.nodeSize = c.take<u32>(nnode);
        b.rawEdge = c.take<u32>((size_t)4 * n);
        if (repeat) {
            b.chunks = c.take<uint4>((size_t)n * (nbinP / 4));
        } else {
            b.eW = c.take<u32>((size_t)n * eStride);
            b.eQ = c.take<u32>((size_t)n * eStride);
            b.eLen = c.take<u32>(n);
            b.chunkStart = c.take<u64>(nChunks + 1);
        }
        b.initKey = c.take<unsigned long long>(n);
        return b;
    };
    struct Glob {
        Rep* reps;
        u32 *repOfWarp, *cells, *words, *order, *rankOf, *sortedRank, *ops, *Xlo, *Xhi, *repN, *repOff, *repOpsOff;
        u32 *ymin, *ysize, *support;
        u64* tileStart;
        unsigned long long* counter;
        unsigned long long* stats;
        u32* rank;
        int* errs;
        int* xerr;  // post-order stack, a cell listed twice, initial scan
        u32* colIdx;
        u32* rrows;
    };
    auto glob_layout = [&](Carve& c) {
        Glob g;
        g.reps = c.take<Rep>(nrep);
        g.repOfWarp = c.take<u32>(totalTips);
        g.cells = c.take<u32>(totalTips);
        g.words = c.take<u32>((size_t)ntip * nbin);
        g.order = c.take<u32>(nrep);
        g.rankOf = c.take<u32>(totalTips);
        g.sortedRank = c.take<u32>(totalTips);
        g.ops = c.take<u32>(repOpsOff[nrep]);
        g.Xlo = c.take<u32>(nX);
        g.Xhi = c.take<u32>(nX);
        g.repN = c.take<u32>(nrep);
        g.repOff = c.take<u32>(nrep);
        g.repOpsOff = c.take<u32>(nrep);
        g.ymin = c.take<u32>((size_t)nrep * nX);
        g.ysize = c.take<u32>((size_t)nrep * nX);
        g.support = c.take<u32>(nX);
        g.tileStart = c.take<u64>(nrep + 1);
        g.counter = c.take<unsigned long long>(1);
        g.errs = c.take<int>(nrep);
        g.xerr = c.take<int>(3);
        g.stats = c.take<unsigned long long>((size_t)8 * nrep);
        g.rank = c.take<u32>(ntip);
        g.colIdx = c.take<u32>(repeat ? (size_t)nrep * nsite : 1);
        g.rrows = c.take<u32>(repeat ? (size_t)totalTips * nbin : 1);
        return g;
    };
    Carve cv;
    glob_layout(cv);
    for (u32 r = 0; r < nrep; r++) rep_layout(cv, repN[r]);
    void* base = nullptr;
    if ((rc = ds.reserve(cv.off + 256, &base))) return rc;
    Carve c2;
    c2.base = static_cast<char*>(base);
    const Glob gl = glob_layout(c2);
    std::vector<Rep> reps(nrep);
    std::vector<RepBufs> rb(nrep);
    std::vector<u64> tileStart(nrep + 1, 0), chunkAll;
    std::vector<std::vector<u64>> chunkStarts(nrep);
    size_t smem = opsBytes;
    for (u32 r = 0; r < nrep; r++) {
        rb[r] = rep_layout(c2, repN[r]);
        const u32 n = repN[r], Sp = (n + 7u) & ~7u, nChunks = (n + kCap - 1) / kCap;
        auto& cs = chunkStarts[r];
        cs.assign(nChunks + 1, 0);
        for (u32 k = 0; k < nChunks; k++) {
            const u64 end = std::min<u64>((u64)(k + 1) * kCap, n);
            cs[k + 1] = cs[k] + (end >= 1 ? end - 1 : 0);
        }
        tileStart[r + 1] = tileStart[r] + (repeat ? bitdot::tiles(n, n, true) : cs[nChunks]);
        Rep& R = reps[r];
        std::memset(&R, 0, sizeof(Rep));
        const RepBufs& b = rb[r];
        joinc::Args& c = R.c;
        size_t sm = 0;
        if (!plan(n, G, c, R.m, &sm)) return CASPHY_EINTERNAL;  // no larger than the largest, which fits
        smem = std::max(smem, sm);
        c.initKey = b.initKey;
        c.nodeSize = b.nodeSize; c.rawEdge = b.rawEdge; c.err = gl.errs + r;
        c.limitNs = 20ull * 1000 * 1000 * 1000; c.statsOut = gl.stats + (size_t)8 * r;
        c.ordNeg1 = ORD_F32_NEG1; c.compactMin = 256; c.bytesPerPairSite = 4000;
        R.m.compactAt = 12;  // a few CTAs per tree, many slots each: 8 took 31.8 ms where this takes 31.0
        c.keepSizes = 1;  // build_ops lays out clades by node size
        R.m.ancType = ancestralType ? 1 : 0;
        R.m.planeMask = b.planeMask;
        R.m.nodeSeq = b.nodeSeq; R.m.nodeBis = b.nodeBis;
        R.m.colT[0] = b.colT0; R.m.colT[1] = b.colT1;
        R.m.Sp = Sp;
        R.colT = b.colT0;
        R.init = InitArgs{n, nbin, Sp, eStride, b.colT0, b.eW, b.eQ, b.eLen, nullptr, b.chunkStart, nChunks,
                          cs[nChunks], nullptr, b.initKey};
        R.off = rep_offsets[r];
        R.ops = gl.ops + repOpsOff[r];
        R.eW = b.eW; R.eQ = b.eQ; R.eLen = b.eLen; R.eStride = eStride;
        R.chunks = b.chunks;
    }
    cudaStream_t st = 0;
    cudaEvent_t ev[4];
    for (auto& e : ev) CASPHY_CUDA_TRY(cudaEventCreate(&e));
    auto up = [&](void* d, const void* h, size_t n) { return cudaMemcpyAsync(d, h, n, cudaMemcpyHostToDevice, st); };
    // per-replicate plane masks and tile tables
    for (u32 r = 0; r < nrep && !repeat; r++) {
        const RepBufs& b = rb[r];
        const u32 nChunks = (u32)chunkStarts[r].size() - 1;
        CASPHY_CUDA_TRY(up(b.planeMask, planes.data() + (size_t)r * P * nbin, sizeof(u32) * P * nbin));
        CASPHY_CUDA_TRY(up(b.chunkStart, chunkStarts[r].data(), sizeof(u64) * (nChunks + 1)));
    }
    CASPHY_CUDA_TRY(up(gl.reps, reps.data(), sizeof(Rep) * nrep));
    CASPHY_CUDA_TRY(up(gl.cells, rep_cells, 4ull * totalTips));
    CASPHY_CUDA_TRY(up(gl.words, words, 4ull * ntip * nbin));
    CASPHY_CUDA_TRY(up(gl.order, order.data(), 4ull * nrep));
    CASPHY_CUDA_TRY(up(gl.rank, rank.data(), 4ull * ntip));
    CASPHY_CUDA_TRY(up(gl.Xlo, Xlo.data(), 4ull * nX));
    CASPHY_CUDA_TRY(up(gl.Xhi, Xhi.data(), 4ull * nX));
    CASPHY_CUDA_TRY(up(gl.repN, repN.data(), 4ull * nrep));
    CASPHY_CUDA_TRY(up(gl.repOff, rep_offsets, 4ull * nrep));
    CASPHY_CUDA_TRY(up(gl.repOpsOff, repOpsOff.data(), 4ull * nrep));
    CASPHY_CUDA_TRY(up(gl.tileStart, tileStart.data(), 8ull * (nrep + 1)));
    CASPHY_CUDA_TRY(cudaMemsetAsync(gl.support, 0, 4ull * nX, st));
    CASPHY_CUDA_TRY(cudaMemsetAsync(gl.counter, 0, sizeof(unsigned long long), st));
    CASPHY_CUDA_TRY(cudaMemsetAsync(gl.errs, 0, sizeof(int) * nrep, st));
    CASPHY_CUDA_TRY(cudaMemsetAsync(gl.xerr, 0, 3 * sizeof(int), st));
    if (repeat) CASPHY_CUDA_TRY(up(gl.colIdx, colIdx.data(), 4ull * nrep * nsite));
    k_bs_ranks<<<nrep, kRankThreads, 0, st>>>(gl.repOff, gl.repN, gl.cells, gl.rank, ntip, gl.repOfWarp, gl.rankOf,
                                              gl.sortedRank, gl.xerr + 1);
    CASPHY_CUDA_TRY(cudaGetLastError());
    int twice = 0;
    CASPHY_CUDA_TRY(cudaMemcpyAsync(&twice, gl.xerr + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    CASPHY_CUDA_TRY(cudaStreamSynchronize(st));
    if (twice) {
        for (auto& e : ev) cudaEventDestroy(e);
        casphy_set_last_error_msg("bootstrap: a replicate lists a cell twice");
        return CASPHY_EINVAL;
    }
    CASPHY_CUDA_TRY(cudaFuncSetAttribute((void*)bitdot::k_bitdot<InitTile>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bitdot::kSmemBytes));
    int perSM = 0;
    CASPHY_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_bs_init, kThreads, 0));
    // (the planned size may have shrunk to what the replicates need)
    if (joinc::placeable((void*)joinFn, G, smem) < 1) return CASPHY_EINTERNAL;
    XferArgs xa{nX, nrep, 32u * ((ntip + 31) / 32), gl.Xlo, gl.Xhi, gl.repN, gl.repOff, gl.repOpsOff, gl.sortedRank, gl.ops,
                threshold, gl.ymin, gl.ysize, gl.support, gl.xerr};
    // the whole pass: prep, initial scans, the joins, transfer
    constexpr u64 kGrid = 1ull << 30;  // tiles per launch
    const u64 nTile = tileStart[nrep];
    const u64 launches = 4 + (repeat ? 1 + (nTile + kGrid - 1) / kGrid : 1);
    auto enqueue = [&](cudaStream_t s) -> cudaError_t {
        cudaError_t e;
        if ((e = cudaEventRecordWithFlags(ev[0], s, cudaEventRecordExternal)) != cudaSuccess) return e;
        if (repeat)
            k_bs_gather<<<(totalTips + 7) / 8, 256, 0, s>>>(gl.repOfWarp, gl.cells, gl.words, gl.colIdx, nbin, totalTips,
                                                          gl.rrows);
        k_bs_prep<<<(totalTips + 7) / 8, 256, 0, s>>>(gl.reps, gl.repOfWarp, gl.cells, gl.words,
                                                      repeat ? gl.rrows : nullptr, nbin, totalTips);
        if (repeat) {
            bitdot::Args a{};
            a.chunks = a.negFrom = nbinP / 4;
            a.upper = 1;
            a.err = gl.xerr + 2;
            for (u64 t = 0; t < nTile; t += kGrid)
                bitdot::k_bitdot<InitTile><<<(u32)std::min(kGrid, nTile - t), bitdot::kThreads, bitdot::kSmemBytes, s>>>(
                    a, InitTile::Params{gl.reps, gl.tileStart, nrep, t, nullptr});
        } else {
            k_bs_init<<<nSM * std::max(perSM, 1), kThreads, 0, s>>>(gl.reps, gl.tileStart, nrep, gl.counter);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = cudaEventRecordWithFlags(ev[1], s, cudaEventRecordExternal)) != cudaSuccess) return e;
        if ((e = joinc::enqueue(joinFn, G, nrep, smem, s, (const Rep*)gl.reps, (const u32*)gl.order, G,
                                (const u32*)gl.rankOf, (const int*)(gl.xerr + 2), opsShared)) !=
            cudaSuccess)
            return e;
        if ((e = cudaEventRecordWithFlags(ev[2], s, cudaEventRecordExternal)) != cudaSuccess) return e;
        k_bs_transfer<<<dim3((nX + kXThreads - 1) / kXThreads, nrep), kXThreads, 0, s>>>(xa);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        return cudaEventRecordWithFlags(ev[3], s, cudaEventRecordExternal);
    };
    // run it as one captured CUDA graph; launch directly if capture fails
    bool graphed = false;
    {
        cudaStream_t cs = nullptr;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) == cudaSuccess &&
            cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            const cudaError_t e = enqueue(cs);
            const cudaError_t e2 = cudaStreamEndCapture(cs, &graph);
            if (e == cudaSuccess && e2 == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess)
                graphed = cudaGraphLaunch(exec, cs) == cudaSuccess && cudaStreamSynchronize(cs) == cudaSuccess;
        }
        if (!graphed) cudaGetLastError();  // a refused capture is not an error of the call
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (cs) cudaStreamDestroy(cs);
    }
    if (!graphed) CASPHY_CUDA_TRY(enqueue(st));
    std::vector<int> errs(nrep);
    int xerr[3] = {0, 0, 0};
    CASPHY_CUDA_TRY(cudaMemcpyAsync(errs.data(), gl.errs, sizeof(int) * nrep, cudaMemcpyDeviceToHost, st));
    CASPHY_CUDA_TRY(cudaMemcpyAsync(xerr, gl.xerr, sizeof(xerr), cudaMemcpyDeviceToHost, st));
    CASPHY_CUDA_TRY(cudaMemcpyAsync(support, gl.support, 4ull * nX, cudaMemcpyDeviceToHost, st));
    if (ymin_out) CASPHY_CUDA_TRY(cudaMemcpyAsync(ymin_out, gl.ymin, 4ull * nrep * nX, cudaMemcpyDeviceToHost, st));
    if (ysize_out) CASPHY_CUDA_TRY(cudaMemcpyAsync(ysize_out, gl.ysize, 4ull * nrep * nX, cudaMemcpyDeviceToHost, st));
    if (rep_raw_edges) {
        size_t o = 0;
        for (u32 r = 0; r < nrep; r++) {
            const size_t ne = (size_t)4 * (repN[r] - 1);
            CASPHY_CUDA_TRY(cudaMemcpyAsync(rep_raw_edges + o, rb[r].rawEdge, 4 * ne, cudaMemcpyDeviceToHost, st));
            o += ne;
        }
    }
    std::vector<unsigned long long> hst((size_t)8 * nrep);
    CASPHY_CUDA_TRY(cudaMemcpyAsync(hst.data(), gl.stats, sizeof(unsigned long long) * hst.size(), cudaMemcpyDeviceToHost, st));
    CASPHY_CUDA_TRY(cudaStreamSynchronize(st));
    unsigned long long phases = 0;
    std::vector<double> repUs(nrep, 0.0);
    std::vector<unsigned long long> repPhases(nrep, 0);
    double longest = 0, busy = 0;
    for (u32 r = 0; r < nrep; r++) {
        phases += hst[8 * r + 3];
        repPhases[r] = hst[8 * r + 3];
        const unsigned long long t0 = hst[8 * r + 6], t1 = hst[8 * r + 7];
        repUs[r] = t1 > t0 ? (double)(t1 - t0) * 1e-3 : 0.0;
        longest = std::max(longest, repUs[r]);
        busy += repUs[r] * G;
    }
    if (xerr[2]) {
        casphy_set_last_error_msg("bootstrap: a device-side wait timed out");
        return xerr[2];
    }
    for (u32 r = 0; r < nrep; r++)
        if (errs[r]) {
            casphy_set_last_error_msg(errs[r] == CASPHY_ETIMEOUT ? "bootstrap: a replicate join timed out"
                                                                  : "bootstrap: a replicate join failed");
            return errs[r];
        }
    if (xerr[0]) {
        casphy_set_last_error_msg("bootstrap: post-order stack overflow");
        return CASPHY_EINTERNAL;
    }
    boot::refit(tune, repN, G, repUs, repPhases);
    float tInit = 0, tJoin = 0, tX = 0, tAll = 0;
    cudaEventElapsedTime(&tInit, ev[0], ev[1]);
    cudaEventElapsedTime(&tJoin, ev[1], ev[2]);
    cudaEventElapsedTime(&tX, ev[2], ev[3]);
    cudaEventElapsedTime(&tAll, ev[0], ev[3]);
    for (auto& e : ev) cudaEventDestroy(e);
    if (stats) {
        casphy_bootstrap_stats s{};
        s.nrep = nrep;
        s.nclade = nX;
        s.prep_ms = tInit;
        s.join_ms = tJoin;
        s.transfer_ms = tX;
        s.total_ms = tAll;
        s.kernel_launches = launches;
        s.join_phases = phases;
        s.max_ctas_per_rep = G;
        s.graph = graphed ? 1u : 0u;
        s.tuned = tunedBefore ? 1u : 0u;
        s.join_longest_ms = longest * 1e-3;
        s.join_busy_ms = busy * 1e-3;
        s.cost_alpha_us = tune.alpha;
        s.cost_beta_us = tune.beta;
        s.cost_gamma_us = tune.gamma;
        *stats = s;
    }
    return CASPHY_OK;
}
