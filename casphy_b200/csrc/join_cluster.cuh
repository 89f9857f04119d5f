// Greedy-join engine on one thread-block cluster.
//
// The same loop as join_engine.cuh (cu/joinEdgeIndel.cu:376-468,
// cu/joinEdgeBitReverse.cu:404-505), the same joins in the same order, for
// trees whose slots a cluster of at most 16 CTAs can scan.  The loop is a
// chain of dependent phases, so what counts is the latency of one phase, not
// the width of the machine: on 148 CTAs a phase of a 12,000-cell tree took
// 10.3 us, of which the scan itself was a few hundred nanoseconds and the rest
// flag barriers through L2, the read of the published table, block-wide
// argmaxes and about thirty block barriers.  Here
//  * CTAs exchange their records through distributed shared memory: 16-byte
//    st.async stores that complete on the receiver's mbarrier, one trip and no
//    flag, no table read; every wait is bounded;
//  * a slot's node, maximum and partner live in its CTA's shared memory for
//    the whole join;
//  * each CTA publishes the best record of each of four thread groups, after
//    every phase: the lists are always fresh, so none runs dry.  A rescan phase
//    publishes them without the rescanned rows, whose new records every CTA
//    forms itself from the exchanged partial bests;
//  * one warp takes the decision and broadcasts it through shared memory;
//  * when enough of the slots are dead (the model says how many) every CTA
//    squeezes its own range, in the middle of a join phase; slots never move
//    between CTAs, so a compaction needs no exchange.
//
// A Model supplies the query build (and, if it likes, an early load of its
// rows), the scores of a CTA's slots and the move of slot data in a compaction.
// Rows of new nodes are written by CTA 0 and
// fenced before its records are sent, so a CTA that has received them reads
// the row from L2.
#pragma once
#include "cluster.cuh"
#include "join_engine.cuh"

namespace casphy {
namespace joinc {

using namespace clu;
using joinx::kDead;
using joinx::kMaxBatch;
constexpr int kThreads = clu::kThreads, kWarps = kThreads / 32;
constexpr u32 kLists = 4;    // records a CTA publishes per exchange, one per four warps

// One published record: larger ord, then larger inv (smaller node) is better;
// ord 0 is no record.  slot: rank of the owning CTA << 24 | slot in its range.
struct alignas(16) Rec {
    u32 ord, inv, slot, partner;
};

struct Args {
    u32 ntip, nnode, G;
    u32 R;                // slots per CTA at the start, below 65,535
    const unsigned long long* initKey;  // ntip initial (maximum, partner) keys
    const u32* tipSize;   // null: all 1
    u32* nodeSize;        // of the new nodes (needSizes, keepSizes)
    u32* rawEdge;
    int* err;
    u64 limitNs;
    unsigned long long* statsOut;  // as joinx::Common
    unsigned long long* prof;
    u32 ordNeg1, compactMin, bytesPerPairSite, maxBatch, deathWords, needSizes, keepSizes;
};

// This CTA's slots [0, n) (capacity cap), in shared memory.
struct Slots {
    u32 n, cap;
    u32* node;
    u32* ord;
    u32* idx;
};

__host__ __device__ inline size_t engine_smem(u32 G, u32 R, u32 deathWords) {
    const size_t tab = 2 * ((size_t)G * kLists * sizeof(Rec) + (size_t)G * kMaxBatch * sizeof(u64));
    return (tab + sizeof(u32) * (3 * (size_t)R + joinx::death_words_padded(deathWords)) + 15) & ~size_t(15);
}

// ---------------------------------------------------------------------------

// The maximum of the warp's (ord, inv) keys, in every lane.  NARROW: the
// scores are non-negative binary16 and the nodes below 2^17, so the key fits 32
// bits (ord's top bit is set in every record) and one reduction (about 90
// clocks) finds it instead of two.
constexpr u32 kNarrowNodes = 1u << 17;
template <bool NARROW>
__device__ __forceinline__ void warp_max2(u32& hi, u32& lo) {
    if (NARROW) {
        constexpr u32 base = 0xFFFFFFFFu - (kNarrowNodes - 1u);  // inv of the largest node
        const u32 k = __reduce_max_sync(0xFFFFFFFFu, hi ? ((hi & 0x7FFFu) << 17) | (lo - base) : 0u);
        hi = k ? 0x8000u | (k >> 17) : 0u;
        lo = k ? base + (k & (kNarrowNodes - 1u)) : 0u;
        return;
    }
    const u32 h = __reduce_max_sync(0xFFFFFFFFu, hi);
    lo = __reduce_max_sync(0xFFFFFFFFu, hi == h ? lo : 0u);
    hi = h;
}

// Best slot of a thread, kept as it walks its slots.
struct Best {
    u32 ord, inv, x;
    __device__ __forceinline__ void init() { ord = inv = x = 0u; }
    __device__ __forceinline__ void push(u32 o, u32 node, u32 at) {
        const u32 iv = ~node;
        if (o > ord || (o == ord && iv > inv)) {
            ord = o; inv = iv; x = at;
        }
    }
};

// The join loop of one cluster; every CTA of the cluster calls it with its
// rank.  smem: engine_smem bytes, then the model's.
template <class M>
__device__ __forceinline__ void cluster_join(const Args& a, const typename M::Args& m, u32 rank, unsigned char* smem) {
    const u32 G = a.G;
    Rec* tab = reinterpret_cast<Rec*>(smem);                       // 2 x G x kLists
    u64* part = reinterpret_cast<u64*>(tab + 2 * G * kLists);      // 2 x kMaxBatch x G
    Slots st;
    st.node = reinterpret_cast<u32*>(part + 2 * G * kMaxBatch);
    st.ord = st.node + a.R;
    st.idx = st.ord + a.R;
    u32* deathBits = st.idx + a.R;
    typename M::Smem ms;
    M::carve_smem(a, m, smem + engine_smem(G, a.R, a.deathWords), ms);
    ms.prof = a.prof != nullptr && rank == 0;
    __shared__ __align__(8) u64 s_bar[2];
    __shared__ Rec s_wrec[kWarps];
    __shared__ Rec s_rows[kMaxBatch];   // the rescanned rows
    __shared__ Rec s_extra[kMaxBatch];  // their new records
    __shared__ u64 s_red[kMaxBatch][kWarps];
    __shared__ u32 s_dec[6];            // -, rescanned rows, j1, slot of j1, j2, failure
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 bar0 = smem_u32(&s_bar[0]);

    joinx::Prof pf;
    pf.init(a.prof != nullptr && rank == 0);
    if (tid == 0) {
        mbar_init(bar0);
        mbar_init(bar0 + 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (G > 1) mbar_expect(bar0, G * kLists * (u32)sizeof(Rec));  // the first exchange
    }
    const u32 lo = min(rank * a.R, a.ntip);
    st.n = min(lo + a.R, a.ntip) - lo;
    st.cap = a.R;
    for (u32 x = tid; x < st.n; x += kThreads) {
        const u64 key = a.initKey[lo + x];
        st.node[x] = lo + x;
        st.ord[x] = key_ord(key);
        st.idx[x] = key_node(key);
    }
    for (u32 i = tid; i < a.deathWords; i += kThreads) deathBits[i] = 0u;
    if (tid < kMaxBatch * kWarps) (&s_red[0][0])[tid] = 0ull;
    // slot x's node is written by thread x mod 512; begin() may read it from any
    // warp (the indel model's resident codes: warp x mod 16)
    __syncthreads();
    M::begin(a, m, ms, rank, st);
    __syncthreads();
    if (G > 1) cluster_sync();

    // Every group of four warps sends its best record to every CTA.
    auto send_lists = [&](const Best& b, u32 buf) {
        u32 hi = b.ord, lw = b.inv;
        warp_max2<M::kNarrow>(hi, lw);
        if (hi == 0u) {
            if (lane == 0) s_wrec[warp] = Rec{0u, 0u, 0u, 0u};
        } else if (b.ord == hi && b.inv == lw) {
            s_wrec[warp] = Rec{b.ord, b.inv, (rank << 24) | b.x, st.idx[b.x]};
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp >> 2)) : "memory");
        if ((warp & 3) == 0) {
            const u32 o = lane < 4 ? s_wrec[warp + lane].ord : 0u, v = lane < 4 ? s_wrec[warp + lane].inv : 0u;
            u32 h2 = o, l2 = v;
            warp_max2<M::kNarrow>(h2, l2);
            const u32 w = __ballot_sync(0xFFFFFFFFu, lane < 4 && o == h2 && v == l2);
            const Rec r = s_wrec[warp + __ffs(w) - 1];
            Rec* dst = tab + (size_t)buf * G * kLists + rank * kLists + (warp >> 2);
            if (G == 1) {
                if (lane == 0) *dst = r;
            } else if (lane < G) {
                st_async16(mapa(smem_u32(dst), lane), make_uint4(r.ord, r.inv, r.slot, r.partner), mapa(bar0 + 8 * buf, lane));
            }
        }
    };
    auto list_best = [&](Best& b) {
        b.init();
        for (u32 x = tid; x < st.n; x += kThreads)
            if (st.node[x] != kDead && st.ord[x] != a.ordNeg1)
                b.push(st.ord[x], st.node[x], x);
    };

    const u32 nJoin = a.ntip - 1;
    u32 k = 0, p = 0, prevQ = 0, S = a.ntip;
    unsigned long long nStale = 0, nPairs = 0, nComp = 0, algMilli = 0;
    int fail = 0;
    {
        Best b;
        list_best(b);
        send_lists(b, 0);
    }
    pf.mark(joinx::PROF_COMPACT);
    typename M::Pre pre;
    for (; k < nJoin; p++) {
        const u32 buf = p & 1u;
        if (G == 1) __syncthreads();
        if (warp == 0) {
            // the exchange's records, from every CTA
            u32 bad = 0;
            if (G > 1) {
                bad = mbar_wait(bar0 + 8 * buf, (p >> 1) & 1u, a.err, a.limitNs) ? 0u : 1u;
                bad = __any_sync(0xFFFFFFFFu, bad);
            }
            pf.mark(joinx::PROF_BARRIER);
            // new records of the rows rescanned in the last phase
            if (prevQ) {
                const u32 q = lane >> 2;
                u64 v = 0ull;
                if (q < prevQ)
                    for (u32 r = lane & 3; r < G; r += 4) {
                        const u64 x = part[((size_t)buf * kMaxBatch + q) * G + r];
                        v = x > v ? x : v;
                    }
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    const u64 x = __shfl_xor_sync(0xFFFFFFFFu, v, o);
                    v = x > v ? x : v;
                }
                if (q < prevQ && (lane & 3) == 0) {
                    const u64 seed = make_key(a.ordNeg1, 0u);
                    if (v < seed) v = seed;
                    Rec r = s_rows[q];
                    const u32 o = key_ord(v);
                    r.partner = key_node(v);
                    if (r.slot >> 24 == rank) {
                        st.ord[r.slot & 0xFFFFFFu] = o;
                        st.idx[r.slot & 0xFFFFFFu] = r.partner;
                    }
                    r.ord = o == a.ordNeg1 ? 0u : o;
                    if (r.ord == 0u) r.inv = 0u;
                    s_extra[q] = r;
                }
                __syncwarp();
            }
            // the decision: the best of up to three records per lane is joined
            // when its partner lives; else it and the other stale records
            // above the best live one are rescanned, best first
            const u32 nList = G * kLists;
            const Rec* T = tab + (size_t)buf * nList;
            Rec rec[3];
            rec[0] = lane < nList ? T[lane] : Rec{0u, 0u, 0u, 0u};
            rec[1] = lane + 32 < nList ? T[lane + 32] : Rec{0u, 0u, 0u, 0u};
            rec[2] = lane < prevQ ? s_extra[lane] : Rec{0u, 0u, 0u, 0u};
            auto better = [](const Rec& r, u32 ord, u32 inv) { return r.ord > ord || (r.ord == ord && r.inv > inv); };
            auto is_dead = [&](const Rec& r) {
                return r.ord && r.partner < a.nnode && ((deathBits[r.partner >> 5] >> (r.partner & 31)) & 1u);
            };
            u32 top = better(rec[1], rec[0].ord, rec[0].inv) ? 1u : 0u;
            Rec mine = top ? rec[1] : rec[0];
            if (prevQ && better(rec[2], mine.ord, mine.inv)) {
                mine = rec[2];
                top = 2u;
            }
            u32 hi = mine.ord, lw = mine.inv, nq = 0;
            warp_max2<M::kNarrow>(hi, lw);
            const bool winner = hi && mine.ord == hi && mine.inv == lw;
            if (winner) {
                if ((~lw) >= a.nnode || mine.partner >= a.nnode) bad = 1;
            }
            // the rows that the decision will most likely need: their load is under
            // way while it is taken (unconditional, so that no register is moved
            // before the load is done)
            if constexpr (M::kLoadsEarly) {
                const u32 partner = __reduce_max_sync(0xFFFFFFFFu, winner ? mine.partner : 0u);
                M::load_early(m, pre, min(~lw, a.nnode - 1u), min(partner, a.nnode - 1u));
            }
            if (hi == 0u) bad = bad ? bad : 2u;  // two live rows always have a record
            bool stale = winner && is_dead(mine);
            if (!__any_sync(0xFFFFFFFFu, stale)) {
                if (winner) {
                    const u32 j1 = ~lw, j2 = mine.partner;
                    s_dec[2] = j1;
                    s_dec[3] = mine.slot;
                    s_dec[4] = j2;
                    if (!bad) {
                        atomicOr(deathBits + (j1 >> 5), 1u << (j1 & 31));
                        atomicOr(deathBits + (j2 >> 5), 1u << (j2 & 31));
                    }
                }
            } else {
                bool dead[3];
                u32 fk = 0, fi = 0;  // the best record whose partner lives
#pragma unroll
                for (u32 j = 0; j < 3; j++) {
                    dead[j] = is_dead(rec[j]);
                    if (!dead[j] && better(rec[j], fk, fi)) {
                        fk = rec[j].ord;
                        fi = rec[j].inv;
                    }
                }
                warp_max2<M::kNarrow>(fk, fi);
                while (nq < a.maxBatch) {
#pragma unroll
                    for (u32 j = 0; j < 3; j++)
                        if (dead[j] && rec[j].ord == hi && rec[j].inv == lw) {
                            s_rows[nq] = rec[j];
                            dead[j] = false;
                            if ((~lw) >= a.nnode) bad = 1;
                            // its old record leaves the lists
                            if (rec[j].slot >> 24 == rank) st.ord[rec[j].slot & 0xFFFFFFu] = a.ordNeg1;
                        }
                    nq++;
                    hi = lw = 0u;
#pragma unroll
                    for (u32 j = 0; j < 3; j++)
                        if (dead[j] && better(rec[j], fk, fi) && better(rec[j], hi, lw)) {
                            hi = rec[j].ord;
                            lw = rec[j].inv;
                        }
                    warp_max2<M::kNarrow>(hi, lw);
                    if (hi == 0u) break;
                }
            }
            const u32 badAny = __any_sync(0xFFFFFFFFu, bad == 1u) ? 1u : bad;
            if (lane == 0) {
                s_dec[1] = nq;
                s_dec[5] = badAny;
                if (G > 1) mbar_expect(bar0 + 8 * (buf ^ 1u), G * (kLists * (u32)sizeof(Rec) + nq * (u32)sizeof(u64)));
            }
        }
        __syncthreads();
        pf.mark(joinx::PROF_DECIDE);
        const u32 nq = s_dec[1];
        if (s_dec[5]) {
            if (s_dec[5] == 2u || G == 1) fail = CASPHY_EINTERNAL;
            else if (tid == 0) atomicCAS(a.err, 0, CASPHY_EINTERNAL);  // after a timeout the first code stays
            break;
        }
        if (nq) {
            const u32 nE = M::build_stale(a, m, ms, st, nq, s_rows, pre);
            pf.mark(joinx::PROF_SELECT);
            // best (score, node) key of every row over this CTA's live slots
            // other than its own; one thread calls row(q, ...) per slot
            u64 bk = 0ull;
            M::scores(m, ms, st, nq,
                      [&](u32 q, u32 x, u32 o) {
                          const u32 node = st.node[x];
                          if (node == kDead || node == ~s_rows[q].inv) return;
                          const u64 key = make_key(o, node);
                          bk = key > bk ? key : bk;
                      },
                      [&](u32 q) {  // this warp is done with row q
                          u32 hi = key_ord(bk), lw = (u32)bk;
                          warp_max2<M::kNarrow>(hi, lw);
                          if (lane == 0) s_red[q][warp] = ((u64)hi << 32) | lw;
                          bk = 0ull;
                      });
            pf.mark(joinx::PROF_STALE_SCAN);
            Best b;
            list_best(b);
            send_lists(b, buf ^ 1u);
            __syncthreads();
            if (warp < nq) {
                const u64 v = lane < kWarps ? s_red[warp][lane] : 0ull;
                u32 hi = key_ord(v), lw = (u32)v;
                warp_max2<M::kNarrow>(hi, lw);
                const u64 best = ((u64)hi << 32) | lw;
                u64* dst = part + ((size_t)(buf ^ 1u) * kMaxBatch + warp) * G + rank;
                if (G == 1) {
                    if (lane == 0) *dst = best;
                } else if (lane < G) {
                    st_async8(mapa(smem_u32(dst), lane), best, mapa(bar0 + 8 * (buf ^ 1u), lane));
                }
                __syncwarp();
                if (lane < kWarps) s_red[warp][lane] = 0ull;
            }
            nStale += nq;
            nPairs += (unsigned long long)nq * ((a.ntip - k) - 1);
            algMilli += (unsigned long long)a.bytesPerPairSite * nE * ((a.ntip - k) - 1);
            prevQ = nq;
            pf.mark(joinx::PROF_STALE_POST);
            continue;
        }
        // join j1 and j2 into node ntip + k, which takes j1's slot
        const u32 j1 = s_dec[2], slot1 = s_dec[3], j2 = s_dec[4], newNode = a.ntip + k;
        u32 sz1 = 0, sz2 = 0;
        const bool bookkeeper = rank == 0 && tid == kThreads - 1;
        if (a.needSizes || (a.keepSizes && bookkeeper)) {
            auto size_of = [&](u32 j) {
                if (j >= a.ntip) return ld_cg_u32(a.nodeSize + j);
                return a.tipSize ? a.tipSize[j] : 1u;
            };
            sz1 = size_of(j1);
            sz2 = size_of(j2);
        }
        const u32 own = slot1 >> 24 == rank ? slot1 & 0xFFFFFFu : joinx::kNone;
        const u32 nE = M::build_join(a, m, ms, st, rank, j1, j2, sz1, sz2, newNode, own, pre);
        if (bookkeeper) {
            *reinterpret_cast<uint4*>(a.rawEdge + 4 * (size_t)k) = make_uint4(newNode, j1, newNode, j2);
            if (a.needSizes || a.keepSizes) a.nodeSize[newNode] = sz1 + sz2;
        }
        pf.mark(joinx::PROF_BUILD);
        Best b;
        b.init();
        M::scores(m, ms, st, 1u,
                  [&](u32, u32 x, u32 o) {
                      const u32 node = st.node[x];
                      u32 cur = st.ord[x];
                      if (node == j1 || node == j2) {
                          st.node[x] = node == j1 ? newNode : kDead;
                          st.ord[x] = a.ordNeg1;
                      } else if (node != kDead) {
                          if (o > cur) {  // strict improvement
                              cur = o;
                              st.ord[x] = o;
                              st.idx[x] = newNode;
                          }
                          if (cur != a.ordNeg1) b.push(cur, node, x);
                      }
                  },
                  [&](u32) {});
        pf.mark(joinx::PROF_SCAN);
        nPairs += (a.ntip - k - 1) - 1;
        algMilli += (unsigned long long)a.bytesPerPairSite * nE * ((a.ntip - k - 1) - 1);
        k++;
        const u32 alive = a.ntip - k;
        if (S >= a.compactMin && 16 * alive < M::compact_at(m, S) * S && k < nJoin) {
            if (G > 1) cluster_sync();  // the model may read the row CTA 0 has just stored
            else __syncthreads();
            // squeeze this CTA's slots, in order: a slot only moves down, and
            // a chunk is read before any of it is overwritten
            u16* ranks = M::rank_space(ms);
            u32 base = 0;
            for (u32 x0 = 0; x0 < st.n; x0 += kThreads) {
                const u32 x = x0 + tid;
                u32 node = kDead, o = 0, i = 0;
                if (x < st.n) {
                    node = st.node[x];
                    o = st.ord[x];
                    i = st.idx[x];
                }
                const u32 live = __ballot_sync(0xFFFFFFFFu, node != kDead);
                if (lane == 0) s_wrec[warp].ord = __popc(live);
                __syncthreads();
                const u32 c = lane < kWarps ? s_wrec[lane].ord : 0u;
                const u32 before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? c : 0u);
                const u32 total = __reduce_add_sync(0xFFFFFFFFu, c);
                const u32 r = base + before + __popc(live & ((1u << lane) - 1u));
                if (x < st.n) ranks[x] = (u16)(node != kDead ? r : 0xFFFFu);
                if (node != kDead) {
                    st.node[r] = node;
                    st.ord[r] = o;
                    st.idx[r] = i;
                }
                base += total;
                __syncthreads();
            }
            M::compact(a, m, ms, rank, st, base, ranks);
            st.n = base;
            __syncthreads();
            S = alive;
            nComp++;
            list_best(b);
            pf.mark(joinx::PROF_COMPACT);
        }
        if (k < nJoin) {  // nothing is sent that nobody waits for
            // the new node's row, before the records without which no CTA goes on
            if (rank == 0 && G > 1) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            send_lists(b, buf ^ 1u);
        }
        prevQ = 0;
        pf.mark(joinx::PROF_POST);
    }
    if (fail && tid == 0) atomicCAS(a.err, 0, fail);
    if (rank == 0 && tid == 0) {
        a.statsOut[0] = nStale;
        a.statsOut[1] = nPairs;
        a.statsOut[2] = nComp;
        a.statsOut[3] = p;
        a.statsOut[4] = 0;
        a.statsOut[5] = algMilli / 1000ull;
    }
    if (pf.on)
        for (int i = 0; i < joinx::PROF_N; i++) a.prof[i] = joinx::prof_acc[i];
    if (G > 1) {
        // no CTA leaves while another may still write into its shared memory;
        // after a failure the stores already under way get time to land
        cluster_sync();
        if (k < nJoin) {
            const u64 t0 = globaltimer_ns();
            while (globaltimer_ns() - t0 < 20000ull) {}
        }
        cluster_sync();
    }
}

}  // namespace joinc
}  // namespace casphy
