// Bit-join model for the cluster engine (join_cluster.cuh), for the single
// join and the batched bootstrap.
//
// A CTA keeps the columns of its slots (word w of every slot) in shared
// memory when they fit, from the start or from the first compaction that makes
// them fit; until then it reads them from global memory.  Lane = slot, so
// every read is a row of consecutive words and the query words are broadcast.
// The warps are shared out among the queries of a rescan batch.
//  * integer weights: one popcount per (slot, word, plane);
//  * FLOAT: the query's set bits with their weights as a list in ascending
//    order, one predicated add each.  (Walking the set bits of every slot's
//    own intersection, with the weight loaded per bit, took 28 us a scan of a
//    2,999 x 352 tree.)
#pragma once
#include "join_bit_model.cuh"
#include "join_cluster.cuh"

namespace casphy {
namespace bitjoin {

// Rows of so many words are shared out among a query's warps where there are fewer
// groups of 32 slots than warps; a warp that takes a group alone leaves the others
// idle for as long as it walks the row, but shared sums cost a barrier and an atomic
// a slot.  Loops shared and not, one plane: 4,000 cells x 48 words 15.7 and 14.2 ms,
// x 64 16.5 and 15.6, x 96 17.5 and 17.6, x 128 18.8 and 19.9, 500 x 938 2.9 and 9.0;
// three planes: 8,000 x 32 45.8 and 45.0, 4,000 x 48 22.4 and 23.9, x 64 24.1 and
// 27.1, 500 x 938 5.0 and 21.2; bootstrap joins of 40 replicates of 100 to 300 cells x
// 3,125 words 16 and 78, of 64 of 167 to 500 x 938 13 and 37.
constexpr u32 kShareWords = 128, kShareWordsPlanes = 64;

// Whether the rows of nbin words (nplanes: 0 or 1 plane) are shared so.
inline bool wide_rows(u32 nbin, u32 nplanes) { return nbin >= (nplanes > 1 ? kShareWordsPlanes : kShareWords); }

struct BitClusterArgs {
    u32 nbin, nbinP, nplanes;
    int ancType;
    const u32* planeMask;  // nplanes x nbin
    const float* wf;       // nbin x 32 (FLOAT)
    u32* nodeSeq;
    u32* nodeBis;
    u32* colT[2];          // nbin x Sp
    u32 Sp, maxBatch;
    u32 colWords;          // shared-memory words for resident columns
    u32 compactAt;         // sixteenths of the slots still live at a compaction
};

// WIDE: rows shared out among the warps.  A kernel of its own, because that code
// beside the other takes the narrow rows' phases from 2.58 to 2.62 us.
template <int PATH, bool WIDE = false>
struct BitCluster {
    static constexpr bool kNarrow = false;  // binary32 scores
    using Args = BitClusterArgs;
    struct Smem {
        u32* sq;       // maxBatch x planes x nbinP: (plane-masked) query words
        uint2* ent;    // FLOAT: maxBatch x nbin * 32 (column offset << 5 | bit, weight), ascending
        u32* len;      // FLOAT: maxBatch list lengths
        u32* colS;     // resident columns
        u16* ranks;
        const u32* col;
        u32 stride;
        u32 next;      // global buffer the next compaction writes
        u32 rank;
        u32 par;
        bool prof;     // section times are taken
    };
    __host__ __device__ static u32 planes(const Args& m) { return PATH == PATH_PLANES && m.nplanes ? m.nplanes : 1u; }
    __host__ static size_t smem_bytes(const Args& m, u32 R) {
        // (4 words more: the last plane's words are read eight at a time)
        size_t s = sizeof(u32) * ((size_t)m.maxBatch * planes(m) * m.nbinP + 4 + m.colWords) + sizeof(u16) * (size_t)R + 32;
        if (PATH == PATH_FLOAT)
            s += (size_t)m.maxBatch * (sizeof(uint2) * m.nbin * 32 + sizeof(u32));
        return s;
    }
    __device__ static void carve_smem(const joinc::Args& a, const Args& m, unsigned char* p, Smem& s) {
        s.ent = reinterpret_cast<uint2*>(p);
        s.sq = reinterpret_cast<u32*>(s.ent + (PATH == PATH_FLOAT ? (size_t)m.maxBatch * m.nbin * 32 : 0u));
        s.colS = s.sq + (size_t)m.maxBatch * planes(m) * m.nbinP + 4;
        s.len = s.colS + m.colWords;
        s.ranks = reinterpret_cast<u16*>(s.len + (PATH == PATH_FLOAT ? m.maxBatch : 0u));
        s.par = 0;
        (void)a;
    }
    __device__ static u16* rank_space(Smem& s) { return s.ranks; }
    // non-zero (word, plane) entries of the queries being built
    __device__ static u32* entries(u32 par) {
        __shared__ u32 s_ne[2];
        return s_ne + par;
    }
    // sums of words shared out among warps, 0 between the scans
    __device__ static u32* sums() {
        __shared__ u32 s_sum[joinc::kThreads];
        return s_sum;
    }
    __device__ static void begin(const joinc::Args& a, const Args& m, Smem& s, u32 rank, const joinc::Slots& st) {
        s.rank = rank;
        if (WIDE) sums()[threadIdx.x] = 0u;
        s.col = m.colT[0] + (size_t)rank * a.R;
        s.stride = m.Sp;
        s.next = 1;
        if (threadIdx.x < 2) *entries(threadIdx.x) = 0u;
        if ((size_t)m.nbin * a.R <= m.colWords) {
            const u32 warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
            for (u32 w = warp; w < m.nbin; w += joinc::kWarps)
                for (u32 x = lane; x < st.n; x += 32) s.colS[w * a.R + x] = s.col[(size_t)w * m.Sp + x];
            s.col = s.colS;
            s.stride = a.R;
        }
    }
    // Query q's words of one row, this thread's word w (every lane of the warp
    // calls it; sq = 0 past the row).
    __device__ static void put(const Args& m, Smem& s, u32 q, u32 w, u32 sq) {
        const u32 P = planes(m);
        u32 ne = 0;
        for (u32 k = 0; k < P; k++) {
            u32 v = sq;
            if (PATH == PATH_PLANES && m.nplanes) v &= w < m.nbin ? __ldg(m.planeMask + (size_t)k * m.nbin + w) : 0u;
            if (w < m.nbinP) s.sq[((size_t)q * P + k) * m.nbinP + w] = v;
            ne += __popc(__ballot_sync(0xFFFFFFFFu, v != 0u));
        }
        if ((threadIdx.x & 31) == 0 && s.rank == 0) atomicAdd(entries(s.par), ne);
    }
    // The queries are complete.  FLOAT: their lists, a warp per (query, word),
    // lane = bit; the bits of the words before place the word's entries.
    __device__ static u32 finish(const Args& m, Smem& s, u32 nq) {
        __syncthreads();
        if (threadIdx.x == 0) *entries(s.par ^ 1u) = 0u;
        if (PATH == PATH_FLOAT) {
            const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            for (u32 q = 0; q < nq; q++) {
                const u32* sq = s.sq + (size_t)q * m.nbinP;
                for (u32 w = (warp + 16u - (q * m.nbin) % 16u) % 16u; w < m.nbin; w += joinc::kWarps) {
                    const u32 v = sq[w];
                    u32 before = 0;
                    for (u32 i = lane; i < w; i += 32) before += __popc(sq[i]);
                    before = __reduce_add_sync(0xFFFFFFFFu, before);
                    if ((v >> lane) & 1u)
                        s.ent[(size_t)q * m.nbin * 32 + before + __popc(v & ((1u << lane) - 1u))] =
                            make_uint2((w * s.stride) << 5 | lane, __float_as_uint(__ldg(m.wf + w * 32 + lane)));
                    if (w == m.nbin - 1 && lane == 0) s.len[q] = before + __popc(v);
                }
            }
            __syncthreads();
        }
        return *entries(s.par);
    }
    // The deciding warp's words of the best record's row and its partner's: it
    // merges most rows alone (10,000 x 512: 35.2 -> 34.1 ms a call; 2,999 x 352
    // fractional 18.6 -> 18.2).
    static constexpr bool kLoadsEarly = true;
    struct Pre {
        u32 j1 = joinc::kDead, j2 = joinc::kDead, s1 = 0, s2 = 0, b1 = 0, b2 = 0;
    };
    __device__ static void load_early(const Args& m, Pre& pre, u32 j1, u32 j2) {
        const u32 w = threadIdx.x < m.nbin ? threadIdx.x : 0u;
        pre.j1 = j1;
        pre.j2 = j2;
        const size_t r1 = (size_t)j1 * m.nbinP + w, r2 = (size_t)j2 * m.nbinP + w;
        pre.s1 = ld_cg_u32(m.nodeSeq + r1);
        pre.s2 = ld_cg_u32(m.nodeSeq + r2);
        pre.b1 = ld_cg_u32(m.nodeBis + r1);
        pre.b2 = ld_cg_u32(m.nodeBis + r2);
    }
    // Warps of one query: all 16 for one, down to two each for eight.
    __device__ static u32 build_stale(const joinc::Args&, const Args& m, Smem& s, const joinc::Slots&, u32 nq,
                                      const joinc::Rec* rows, const Pre& pre) {
        s.par ^= 1u;
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const u32 lgq = nq <= 1 ? 4u : (nq <= 2 ? 3u : (nq <= 4 ? 2u : 1u));
        const u32 nwq = 1u << lgq, q = warp >> lgq, wi = warp & (nwq - 1u);
        if (q < nq) {
            const u32 j = ~rows[q].inv;
            const u32* src = m.nodeSeq + (size_t)j * m.nbinP;
            for (u32 w0 = wi * 32; w0 < m.nbinP; w0 += nwq * 32) {
                const u32 w = w0 + lane;
                u32 v = 0;
                if (w < m.nbin) v = w == threadIdx.x && j == pre.j1 ? pre.s1 : ld_cg_u32(src + w);
                put(m, s, q, w, v);
            }
        }
        return finish(m, s, nq);
    }
    // ancestral rules (updateAncestralKernel / updateAncestralKernel2,
    // cu/joinEdgeBitReverse.cu:77-113)
    __device__ static u32 build_join(const joinc::Args&, const Args& m, Smem& s, const joinc::Slots&, u32 rank, u32 j1,
                                     u32 j2, u32, u32, u32 newNode, u32 own, const Pre& pre) {
        s.par ^= 1u;
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        {
            const size_t r1 = (size_t)j1 * m.nbinP, r2 = (size_t)j2 * m.nbinP, rn = (size_t)newNode * m.nbinP;
            u32* col = const_cast<u32*>(s.col);
            for (u32 w0 = warp * 32; w0 < m.nbinP; w0 += joinc::kWarps * 32) {
                const u32 w = w0 + lane;
                u32 sq = 0, bs = 0;
                if (w < m.nbin) {
                    u32 s1 = pre.s1, s2 = pre.s2, bs1 = pre.b1, bs2 = pre.b2;
                    if (w != threadIdx.x || pre.j1 != j1 || pre.j2 != j2) {
                        s1 = ld_cg_u32(m.nodeSeq + r1 + w);
                        s2 = ld_cg_u32(m.nodeSeq + r2 + w);
                        bs1 = ld_cg_u32(m.nodeBis + r1 + w);
                        bs2 = ld_cg_u32(m.nodeBis + r2 + w);
                    }
                    if (m.ancType == 0) {
                        const u32 diff = s1 ^ s2;
                        const u32 conflict = diff & (bs1 | bs2);
                        sq = (s1 | s2) & ~conflict;
                        bs = (diff & ~(bs1 ^ bs2)) | (bs1 & bs2);
                    } else {
                        sq = (s1 & s2) | (bs1 & s2) | (bs2 & s1);
                        bs = (s1 ^ s2) & ~(bs1 | bs2);
                    }
                }
                if (rank == 0 && w < m.nbinP) {
                    m.nodeSeq[rn + w] = sq;
                    m.nodeBis[rn + w] = bs;
                }
                if (own != kNone && w < m.nbin) col[(size_t)w * s.stride + own] = sq;
                put(m, s, 0u, w, sq);
            }
        }
        return finish(m, s, 1u);
    }

    // Bits set in eight words: four carry-save adders leave four words to count.
    // (10,000 x 1,024 integer weights 73.2 -> 68.5 ms a call; with one plane the
    // few words a thread has wait on their loads, not on the popcounts, and eight
    // plain ones do: a 64-replicate bootstrap 31.3 ms, 33.7 with the adders.)
    __device__ __forceinline__ static u32 popc8(u32 a, u32 b, u32 c, u32 d, u32 e, u32 f, u32 g, u32 h) {
        auto maj = [](u32 x, u32 y, u32 z) { return (x & y) | (x & z) | (y & z); };
        const u32 s0 = a ^ b ^ c, c0 = maj(a, b, c);
        const u32 s1 = s0 ^ d ^ e, c1 = maj(s0, d, e);
        const u32 s2 = s1 ^ f ^ g, c2 = maj(s1, f, g);
        return (u32)__popc(s2) + (u32)__popc(h) + 2u * (u32)__popc(c0 ^ c1 ^ c2) + 4u * (u32)__popc(maj(c0, c1, c2));
    }
    // Score of query q (words sq) against the slot whose word w is c[w * stride].
    template <bool RES>
    __device__ __forceinline__ static float score(const Args& m, const Smem& s, const u32* c, u32 q, const u32* sq) {
        const u32 stride = s.stride;
        if (PATH == PATH_FLOAT) {
            float fa = 0.f;
            const u32 n = s.len[q];
            const uint2* ent = s.ent + (size_t)q * m.nbin * 32;
            auto add = [&](u32 v, uint2 t) {
                asm("{\n .reg .pred p;\n .reg .b32 t;\n shf.r.wrap.b32 t, %1, %1, %2;\n and.b32 t, t, 1;\n"
                    " setp.ne.u32 p, t, 0;\n @p add.rn.f32 %0, %0, %3;\n}"
                    : "+f"(fa)
                    : "r"(v), "r"(t.x), "f"(__uint_as_float(t.y)));
            };
            // eight entries at a time, the next eight loaded before these are
            // added (only this CTA writes its columns, so plain loads do)
            u32 e = 0;
            if (n > 7) {
                uint2 t[8];
                u32 v[8];
#pragma unroll
                for (u32 j = 0; j < 8; j++) {
                    t[j] = ent[j];
                    v[j] = c[t[j].x >> 5];
                }
                for (; e + 15 < n; e += 8) {
                    uint2 nt[8];
                    u32 nv[8];
#pragma unroll
                    for (u32 j = 0; j < 8; j++) nt[j] = ent[e + 8 + j];
#pragma unroll
                    for (u32 j = 0; j < 8; j++) nv[j] = c[nt[j].x >> 5];
#pragma unroll
                    for (u32 j = 0; j < 8; j++) add(v[j], t[j]);
#pragma unroll
                    for (u32 j = 0; j < 8; j++) {
                        t[j] = nt[j];
                        v[j] = nv[j];
                    }
                }
#pragma unroll
                for (u32 j = 0; j < 8; j++) add(v[j], t[j]);
                e += 8;
            }
            if (e < n) {  // the rest as one batch; past the end, words of 0
                uint2 t[8];
                u32 v[8];
#pragma unroll
                for (u32 j = 0; j < 8; j++) t[j] = e + j < n ? ent[e + j] : make_uint2(0u, 0u);
#pragma unroll
                for (u32 j = 0; j < 8; j++) v[j] = e + j < n ? c[t[j].x >> 5] : 0u;
#pragma unroll
                for (u32 j = 0; j < 8; j++) add(v[j], t[j]);
            }
            return fa;
        }
        return (float)count<RES>(m, s, c, sq, 0u, m.nbin);
    }
    // Integer weights: the score's words [w0, wEnd), w0 a multiple of eight.
    template <bool RES>
    __device__ __forceinline__ static u32 count(const Args& m, const Smem& s, const u32* c, const u32* sq, u32 w0,
                                                u32 wEnd) {
        const u32 stride = s.stride, P = planes(m);
        u32 acc = 0;
        if (P == 1 && RES) {
            u32 w = w0;
#pragma unroll 4
            for (; w + 4 <= wEnd; w += 4) {
                const uint4 a = *reinterpret_cast<const uint4*>(sq + w);
                const u32 v0 = c[w * stride], v1 = c[(w + 1) * stride], v2 = c[(w + 2) * stride], v3 = c[(w + 3) * stride];
                acc += (u32)(__popc(a.x & v0) + __popc(a.y & v1)) + (u32)(__popc(a.z & v2) + __popc(a.w & v3));
            }
            for (; w < wEnd; w++) acc += (u32)__popc(sq[w] & c[w * stride]);
            return acc;
        }
        // eight words of the slot at a time against every plane's
        auto block = [&](const u32 (&v)[8]) {
            for (u32 k = 0; k < P; k++) {
                const uint4 a = *reinterpret_cast<const uint4*>(sq + k * m.nbinP + w0);
                const uint4 b = *reinterpret_cast<const uint4*>(sq + k * m.nbinP + w0 + 4);
                if (PATH == PATH_UNIT)
                    acc += (u32)(__popc(a.x & v[0]) + __popc(a.y & v[1]) + __popc(a.z & v[2]) + __popc(a.w & v[3]) +
                                 __popc(b.x & v[4]) + __popc(b.y & v[5]) + __popc(b.z & v[6]) + __popc(b.w & v[7]));
                else
                    acc += popc8(a.x & v[0], a.y & v[1], a.z & v[2], a.w & v[3], b.x & v[4], b.y & v[5], b.z & v[6], b.w & v[7])
                           << k;
            }
        };
        for (; w0 + 8 <= wEnd; w0 += 8) {
            u32 v[8];
#pragma unroll
            for (u32 j = 0; j < 8; j++) v[j] = RES ? c[(w0 + j) * stride] : ld_cg_u32(c + (size_t)(w0 + j) * stride);
            block(v);
        }
        if (w0 < wEnd) {  // words past the row are 0 on the slot's side
            u32 v[8];
#pragma unroll
            for (u32 j = 0; j < 8; j++)
                v[j] = w0 + j >= wEnd ? 0u : (RES ? c[(w0 + j) * stride] : ld_cg_u32(c + (size_t)(w0 + j) * stride));
            block(v);
        }
        return acc;
    }

    template <class F, class D>
    __device__ static void scores(const Args& m, Smem& s, const joinc::Slots& st, u32 nq, F f, D done) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const u32 lgq = nq <= 1 ? 4u : (nq <= 2 ? 3u : (nq <= 4 ? 2u : 1u));
        const u32 nwq = 1u << lgq;
        const u32 q = warp >> lgq, wi = warp & (nwq - 1u);
        const bool resident = s.col == s.colS;
        const u32 groups = (st.n + 31u) / 32u;
        if (WIDE && groups < nwq) {
            // a query's warps share the words of all groups of 32 slots evenly
            u32* acc = sums() + q * nwq * 32;
            if (q < nq) {
                const u32* sq = s.sq + (size_t)q * planes(m) * m.nbinP;
                const u32 blocks = (m.nbin + 7u) / 8u, total = groups * blocks;
                for (u32 i = wi * total / nwq, end = (wi + 1u) * total / nwq; i < end;) {
                    const u32 g = i / blocks, b = i - g * blocks, e = min(blocks, b + end - i);
                    const u32 x = 32 * g + lane, xs = x < st.n ? x : 32 * g, w1 = min(8 * e, m.nbin);
                    const u32 v = resident ? count<true>(m, s, s.colS + xs, sq, 8 * b, w1)
                                           : count<false>(m, s, s.col + xs, sq, 8 * b, w1);
                    if (x < st.n) atomicAdd(acc + x, v);
                    i += e - b;
                }
            }
            __syncthreads();
            if (q < nq) {
                const u32 x = 32 * wi + lane;
                if (x < st.n) {
                    const float v = (float)acc[x];
                    acc[x] = 0u;
                    f(q, x, ord_f32(v));
                }
                done(q);
            }
            if (s.prof) joinx::prof_mark(joinx::PROF_SC_ACC);
            return;
        }
        if (q < nq) {
            const u32* sq = s.sq + (size_t)q * planes(m) * m.nbinP;
            for (u32 x0 = wi * 32; x0 < st.n; x0 += nwq * 32) {
                const u32 x = x0 + lane, xs = x < st.n ? x : x0;
                // (two calls, so that resident columns are read as shared memory)
                const float v = resident ? score<true>(m, s, s.colS + xs, q, sq) : score<false>(m, s, s.col + xs, q, sq);
                if (x < st.n) f(q, x, ord_f32(v));
            }
            done(q);
        }
        if (s.prof) joinx::prof_mark(joinx::PROF_SC_ACC);
    }

    __device__ static u32 compact_at(const Args& m, u32) { return m.compactAt; }
    // Moves the live slots' columns to their new places; n live slots, ranks
    // by old slot.  In shared memory in place, a warp per column: a slot only
    // moves down, and 32 are read before any of them is written.
    __device__ static void compact(const joinc::Args& a, const Args& m, Smem& s, u32 rank, const joinc::Slots& st, u32 n,
                                   const u16* ranks) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const bool resident = s.col == s.colS;
        const u32 Rn = (n + 31u) & ~31u;
        u32* dst = s.colS;
        u32 stride = s.stride;
        if (!resident) {
            if ((size_t)m.nbin * Rn <= m.colWords) {
                stride = Rn;
            } else {
                dst = (s.next ? m.colT[1] : m.colT[0]) + (size_t)rank * a.R;
                s.next ^= 1u;
            }
        }
        for (u32 w = warp; w < m.nbin; w += joinc::kWarps) {
            const u32* src = s.col + (size_t)w * s.stride;
            for (u32 x0 = 0; x0 < st.n; x0 += 32) {
                const u32 x = x0 + lane;
                const u32 r = x < st.n ? ranks[x] : 0xFFFFu;
                u32 v = 0;
                if (r != 0xFFFFu) v = resident ? src[x] : ld_cg_u32(src + x);
                __syncwarp();
                if (r != 0xFFFFu) dst[(size_t)w * stride + r] = v;
                __syncwarp();
            }
        }
        s.col = dst;
        s.stride = stride;
        __syncthreads();
    }
};

template <class M>
__global__ void __launch_bounds__(joinc::kThreads, 1) k_cluster_join(joinc::Args a, typename M::Args m) {
    extern __shared__ __align__(16) unsigned char smem[];
    joinc::cluster_join<M>(a, m, joinc::cluster_rank(), smem);
}

// Shared memory of a cluster join of a.ntip cells by a.G CTAs (a.R set):
// batches of rescanned rows first, then resident columns; false when it does
// not fit.
template <int PATH>
inline bool cluster_fit(joinc::Args& a, BitClusterArgs& m, size_t lim, size_t* smem) {
    for (a.maxBatch = joinx::stale_batch_setting(); a.maxBatch >= 1; a.maxBatch--) {
        m.maxBatch = a.maxBatch;
        m.colWords = 0;
        const size_t need = joinc::engine_smem(a.G, a.R, a.deathWords) + BitCluster<PATH>::smem_bytes(m, a.R);
        if (need > lim) continue;
        m.colWords = (u32)std::min<size_t>((lim - need) / sizeof(u32), (size_t)m.nbin * a.R);
        *smem = joinc::engine_smem(a.G, a.R, a.deathWords) + BitCluster<PATH>::smem_bytes(m, a.R);
        return true;
    }
    return false;
}

}  // namespace bitjoin
}  // namespace casphy
