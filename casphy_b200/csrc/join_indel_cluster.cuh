// Indel-join model for the cluster engine (join_cluster.cuh): allele bitsets,
// as IndelBits of join_indel.cu, and on the same bitsets the ordered binary16
// sums for weights that are not small integers.
//
// A query is the list of its edited sites' bitset rows.  The words of those
// rows that cover this CTA's slots are copied to shared memory (cp.async, in
// two groups, so the first half is added while the second is in flight).
//  * Integer weights: a warp owns a few words and adds all entries of them;
//    lanes that share a word take every NG-th entry and their bit-sliced counts
//    are summed by shuffles.  No warp needs another's sums, so nothing but the
//    copies is waited for.  (Warps that split the entries instead, with a tree
//    over their counters in shared memory, took 2.9 us a phase for the tree.)
//  * HALF: a lane takes two slots and the entries in ascending site order, one
//    paired binary16 add each.  The bit test replaces the column scan's compare of 16-bit
//    codes, and the copies are issued by all threads, where the column scan
//    had one thread in flight per eight slots (27 slots a CTA at 4,000 cells)
//    and spent 6.5 us a scan.
// When a CTA's slots are few (from the start or after a compaction) their codes
// fit shared memory as bytes, [site][slot], and nothing is copied: a thread
// compares four slots (HALF: a lane two) with the query's code at a time.  A
// phase of a 1,024 x 256 tree spent 1.5 of its 4 us on the copies and on folding
// the bit-sliced counts of many lanes; loops measured with bitsets and with codes:
// 1,024 x 256 unit 5.78 and 4.94 ms, 1,000 x 300 fractional 5.73 and 4.92 us a
// join, 4,000 x 500 fractional 27.5 and 24.9 ms.
// Included by join_indel.cu after the bit-sliced adders.
#pragma once
#include "join_cluster.cuh"

namespace casphy {
namespace indel {

constexpr u32 kOneCopyWords = 4096;
constexpr u32 kResidentWords = 384;  // resident codes: words of four slots, at most
// ... and, for the integer sums, (slot, site) pairs: comparing bytes costs more
// than adding bits once a phase is not all latency (2,000 x 256 on 16 CTAs, 32,000
// pairs: 5.1 us a join resident, 5.9 with bitsets; 8,000 x 500, 250,000: 7.8 and 6.8)
constexpr u32 kResidentUnits = 80000;

template <bool HALF>
struct IndelCluster {
    // (rows of many words are loaded by all warps after the decision: loaded early
    // by the deciding warp alone or by all, waiting for the records, 5.55 -> 5.65
    // and 5.75 ms of a 1,024 x 256 call)
    static constexpr bool kLoadsEarly = false;
    struct Pre {};
    static constexpr bool kNarrow = true;  // non-negative binary16 scores; cluster_plan bounds the nodes
    struct Args {
        u32 ncol, ncolP, nState, minSize;
        float minRatio;
        int unitW;
        const u16* Wsel;
        u16* nodeRow;
        u32* bits[2];
        u32 rows;        // ncol x nState bitset rows
        u32 maxBatch;
        u32 stageWords;
    };
    struct Smem {
        u32* eRow;    // maxBatch x ncolW: bitset row of every entry, or its codes' offset << 8 | code
        u32* eW;      // maxBatch x ncolW: weights (unless all are 1); HALF: in both halves of a word
        u32* stage;   // stageWords
        u32* sums;    // HALF: maxBatch x R / 2 pairs of running sums
        u32* slab;    // else: 12 planes of 32 words per warp
        u32* B;       // this CTA's bitset rows, `pitch` words each
        u32* other;   // the same in the other buffer
        u32 pitch;
        u32 rp;       // bytes per site of the resident codes, 0 when there are none
        u32 par;      // parity of the entry counters
        bool prof;    // section times are taken
    };
    // entry counters of the current and the next query build
    __device__ static u32* counts(u32 par) {
        __shared__ u32 s_cnt[2][joinx::kMaxBatch];
        return s_cnt[par];
    }
    __host__ __device__ static u32 ncolW(u32 ncol) { return (ncol + 7u) & ~7u; }
    __host__ static size_t smem_bytes(const Args& m, u32 R) {
        return sizeof(u32) * ((size_t)m.maxBatch * ncolW(m.ncol) * (m.unitW ? 1 : 2) + m.stageWords) +
               (HALF ? sizeof(u16) * (size_t)m.maxBatch * R : sizeof(u32) * joinc::kWarps * 32 * 12) + 16;
    }
    __device__ static void carve_smem(const joinc::Args&, const Args& m, unsigned char* p, Smem& s) {
        s.stage = reinterpret_cast<u32*>(p);
        s.eRow = s.stage + m.stageWords;
        s.eW = s.eRow + (size_t)m.maxBatch * ncolW(m.ncol);
        s.sums = s.eW + (m.unitW ? 0u : (size_t)m.maxBatch * ncolW(m.ncol));
        s.slab = s.sums;
        s.par = 0;
    }
    __device__ static u16* rank_space(Smem& s) { return reinterpret_cast<u16*>(s.stage); }
    // Bytes per site of n slots' resident codes: an odd number of words, so that
    // a slot's column spreads over the banks; 0 when they do not fit (the codes
    // a byte, the stage, the partial sums in the slab).
    __host__ __device__ static u32 resident_pitch(const Args& m, u32 n) {
        const u32 nw = (n + 3u) / 4u, rp = (nw | 1u) * 4u;
        return m.nState <= 253u && nw <= kResidentWords && (HALF || (size_t)n * m.ncol <= kResidentUnits) &&
                       (size_t)m.ncol * rp <= sizeof(u32) * (size_t)m.stageWords
                   ? rp
                   : 0u;
    }
    // The resident codes of the first n slots from their nodes' rows.
    __device__ static void load_codes(const Args& m, Smem& s, const joinc::Slots& st, u32 n) {
        unsigned char* c8 = reinterpret_cast<unsigned char*>(s.stage);
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (u32 x = warp; x < ((n + 3u) & ~3u); x += joinc::kWarps) {
            const u16* row = m.nodeRow + (size_t)(x < n ? st.node[x] : 0u) * m.ncolP;
            for (u32 i = 2 * lane; i < m.ncol; i += 64) {
                const u32 c = x < n ? ld_cg_u32(reinterpret_cast<const u32*>(row + i)) : 0u;
                c8[i * s.rp + x] = (unsigned char)c;
                if (i + 1 < m.ncol) c8[(i + 1) * s.rp + x] = (unsigned char)(c >> 16);
            }
        }
    }
    // A CTA's bitset rows lie together, so that its share of the matrix stays
    // as small as its live slots: k_split_bits has laid them out in bits[1].
    __device__ static void begin(const joinc::Args& a, const Args& m, Smem& s, u32 rank, const joinc::Slots& st) {
        const size_t region = (size_t)rank * m.rows * (a.R / 32);
        s.B = m.bits[1] + region;
        s.other = m.bits[0] + region;
        s.pitch = a.R / 32;
        s.rp = resident_pitch(m, st.n);
        if (s.rp) load_codes(m, s, st, st.n);
        if (threadIdx.x < joinx::kMaxBatch) counts(0)[threadIdx.x] = counts(1)[threadIdx.x] = 0u;
    }

    // Appends the edited ones of this thread's sites (2 per thread, codes c in
    // pairs) to the nq lists; every thread of the CTA calls it.  HALF keeps
    // ascending sites, which takes the warps' counts first.
    __device__ static void append(const Args& m, Smem& s, u32 nq, u32 site, const u32 (&c)[joinx::kMaxBatch], u32* cnt) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, below = (1u << lane) - 1u;
        __shared__ u32 s_wc[joinx::kMaxBatch][joinc::kWarps];
        auto put = [&](u32 q, u32 pos, u32 st, u32 code) {
            s.eRow[(size_t)q * ncolW(m.ncol) + pos] = s.rp ? (st * s.rp) << 8 | code : st * m.nState + code - 2u;
            if (!m.unitW)
                s.eW[(size_t)q * ncolW(m.ncol) + pos] = m.Wsel[(size_t)(code - 2u) * m.ncol + st] * (HALF ? 0x10001u : 1u);
        };
        if (HALF) {
#pragma unroll
            for (u32 q = 0; q < joinx::kMaxBatch; q++) {
                if (q >= nq) break;
                const u32 n = __popc(__ballot_sync(0xFFFFFFFFu, (c[q] & 0xFFFFu) > 1u)) +
                              __popc(__ballot_sync(0xFFFFFFFFu, (c[q] >> 16) > 1u));
                if (lane == 0) s_wc[q][warp] = n;
            }
            __syncthreads();
        }
#pragma unroll
        for (u32 q = 0; q < joinx::kMaxBatch; q++) {
            if (q >= nq) break;
            const u32 c0 = c[q] & 0xFFFFu, c1 = c[q] >> 16;
            const u32 m0 = __ballot_sync(0xFFFFFFFFu, c0 > 1u), m1 = __ballot_sync(0xFFFFFFFFu, c1 > 1u);
            u32 base = 0;
            if (HALF) {
                const u32 v = lane < joinc::kWarps ? s_wc[q][lane] : 0u;
                base = cnt[q] + __reduce_add_sync(0xFFFFFFFFu, lane < warp ? v : 0u);
            } else {
                if (lane == 0) base = atomicAdd(cnt + q, __popc(m0) + __popc(m1));
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
            }
            base += __popc(m0 & below) + __popc(m1 & below);
            if (c0 > 1u) put(q, base++, site, c0);
            if (c1 > 1u) put(q, base, site + 1u, c1);
        }
        if (HALF) {
            __syncthreads();
            if (warp < nq) {
                const u32 t = __reduce_add_sync(0xFFFFFFFFu, lane < joinc::kWarps ? s_wc[warp][lane] : 0u);
                if (lane == 0) cnt[warp] += t;
            }
            if (m.ncolP > 2 * kThreads) __syncthreads();  // the next block of sites reads cnt and writes s_wc
        }
    }
    // The lists are complete and the other counters zero for the next build.
    __device__ static u32 finish(Smem& s, u32 nq) {
        __syncthreads();
        const u32* cnt = counts(s.par);
        if (threadIdx.x < joinx::kMaxBatch) counts(s.par ^ 1u)[threadIdx.x] = 0u;
        u32 t = 0;
        for (u32 q = 0; q < nq; q++) t += cnt[q];
        return t;
    }
    __device__ static u32 build_stale(const joinc::Args&, const Args& m, Smem& s, const joinc::Slots&, u32 nq,
                                      const joinc::Rec* rows, const Pre&) {
        s.par ^= 1u;
        u32* cnt = counts(s.par);
        for (u32 s0 = 0; s0 < m.ncolP; s0 += 2 * kThreads) {
            const u32 site = s0 + 2 * threadIdx.x;
            u32 c[joinx::kMaxBatch];
#pragma unroll
            for (u32 q = 0; q < joinx::kMaxBatch; q++)
                c[q] = q < nq && site < m.ncolP
                           ? ld_cg_u32(reinterpret_cast<const u32*>(m.nodeRow + (size_t)(~rows[q].inv) * m.ncolP + site))
                           : 0u;
            append(m, s, nq, site, c, cnt);
        }
        return finish(s, nq);
    }
    // minSize / minRatio rule of cu/joinEdgeIndel.cu:407-413.  CTA 0 stores the
    // new row; the owner of j1's slot (own: its local index) flips the slot's
    // bit in the rows where the two states differ.
    __device__ static u32 build_join(const joinc::Args& a, const Args& m, Smem& s, const joinc::Slots&, u32 rank,
                                     u32 j1, u32 j2, u32 s1, u32 s2, u32 newNode, u32 own, const Pre&) {
        s.par ^= 1u;
        u32* cnt = counts(s.par);
        int mode = 3;
        if (a.needSizes) {
            if (s1 < m.minSize && __uint2float_rn(s1) * m.minRatio < __uint2float_rn(s2)) mode = 1;
            else if (s2 < m.minSize && __uint2float_rn(s2) * m.minRatio < __uint2float_rn(s1)) mode = 2;
        }
        for (u32 s0 = 0; s0 < m.ncolP; s0 += 2 * kThreads) {
            const u32 site = s0 + 2 * threadIdx.x;
            u32 c[joinx::kMaxBatch] = {0u};
            if (site < m.ncolP) {
                const u32 x = ld_cg_u32(reinterpret_cast<const u32*>(m.nodeRow + (size_t)j1 * m.ncolP + site));
                const u32 y = ld_cg_u32(reinterpret_cast<const u32*>(m.nodeRow + (size_t)j2 * m.ncolP + site));
                c[0] = merge_code(mode, x & 0xFFFFu, y & 0xFFFFu) | (merge_code(mode, x >> 16, y >> 16) << 16);
                if (rank == 0) *reinterpret_cast<u32*>(m.nodeRow + (size_t)newNode * m.ncolP + site) = c[0];
                if (own != kNone && c[0] != x) {
                    const u32 word = own >> 5, bit = 1u << (own & 31);
#pragma unroll
                    for (u32 h = 0; h < 2; h++) {
                        const u32 o = (x >> (16 * h)) & 0xFFFFu, n = (c[0] >> (16 * h)) & 0xFFFFu;
                        if (o == n) continue;
                        if (s.rp) {
                            if (site + h < m.ncol)
                                reinterpret_cast<unsigned char*>(s.stage)[(site + h) * s.rp + own] = (unsigned char)n;
                            continue;
                        }
                        const size_t row = (size_t)(site + h) * m.nState;
                        if (o > 1u) atomicAnd(s.B + (row + o - 2u) * s.pitch + word, ~bit);
                        if (n > 1u) atomicOr(s.B + (row + n - 2u) * s.pitch + word, bit);
                    }
                }
            }
            append(m, s, 1u, site, c, cnt);
        }
        return finish(s, 1u);
    }

    // Copies entries [a, b) of the queries' sequence, `wst` words each from
    // word wb, into the stage at `pitch` words each, counted from r0.
    __device__ static void copy_range(const Args& m, const Smem& s, u32 nq, u32 r0, u32 a, u32 b, u32 wb, u32 wst,
                                      u32 pitch) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const u32* cnt = counts(s.par);
        const u32* B = s.B + wb;
        const u32 cpe = wst >> 2;  // 16-byte pieces per entry
        // entries a warp copies at a time, and this lane's entry and piece of
        // them: quotients by cpe <= 32, exact in this form for lane <= 32
        const u32 rcp = 1024u / cpe + 1u;
        const u32 epw = cpe <= 32u ? (32u * rcp) >> 10 : 0u, jl = (lane * rcp) >> 10, kl = lane - jl * cpe;
        u32 off = 0;
        for (u32 q = 0; q < nq; q++) {
            const u32 n = cnt[q], lo = max(a, off), hi = min(b, off + n);
            const u32* list = s.eRow + (size_t)q * ncolW(m.ncol);
            if (cpe <= 32u) {
                if (jl < epw)
#pragma unroll 4
                    for (u32 e = lo + warp * epw + jl; e < hi; e += joinc::kWarps * epw)
                        cp_async16(s.stage + (e - r0) * pitch + 4 * kl, B + (size_t)list[e - off] * s.pitch + 4 * kl);
            } else {
                for (u32 e = lo + warp; e < hi; e += joinc::kWarps) {
                    const u32* src = B + (size_t)list[e - off] * s.pitch;
                    for (u32 k = lane; k < cpe; k += 32u) cp_async16(s.stage + (e - r0) * pitch + 4 * k, src + 4 * k);
                }
            }
            off += n;
        }
    }
    // Rounds of `per` entries (what the stage holds), copied in two groups;
    // add(r0, a, b) consumes the staged entries [a, b).
    template <class F>
    __device__ static void rounds(const Args& m, Smem& s, u32 nq, u32 total, u32 per, u32 wb, u32 wst, u32 pitch, F add) {
        for (u32 r0 = 0; r0 < total; r0 += per) {
            const u32 r1 = min(total, r0 + per);
            // (a few KB arrive together: halves would only add a barrier)
            const bool halves = (r1 - r0) * wst > kOneCopyWords;
            const u32 rm = halves ? min(r1, r0 + (((r1 - r0) / 2 + 7u) & ~7u)) : r1;
            copy_range(m, s, nq, r0, r0, rm, wb, wst, pitch);
            cp_async_commit();
            if (halves) {
                copy_range(m, s, nq, r0, rm, r1, wb, wst, pitch);
                cp_async_commit();
                cp_async_wait_group<1>();
            } else {
                cp_async_wait_group<0>();
            }
            __syncthreads();
            if (s.prof) joinx::prof_mark(joinx::PROF_SC_COPY);
            add(r0, r0, rm);
            if (halves) {
                cp_async_wait_group<0>();
                __syncthreads();
                add(r0, rm, r1);
            }
            if (r1 < total) __syncthreads();  // the next round overwrites the stage
            if (s.prof) joinx::prof_mark(joinx::PROF_SC_ACC);
        }
    }

    // c += the staged words of entries first, first + step, ... < end (unit
    // weights) in N bit-sliced planes: eight words at a time through carry-save
    // adders that keep the ones, twos and fours (7 adders of two logic
    // operations), the eights rippled on.
    template <int N>
    __device__ static void add8(u32 (&c)[kPlanes], const u32 (&x)[8]) {
        u32 t0, t1, f0, f1, cy;
        fa(c[0], x[0], x[1], c[0], t0);
        fa(c[0], x[2], x[3], c[0], t1);
        fa(c[1], t0, t1, c[1], f0);
        fa(c[0], x[4], x[5], c[0], t0);
        fa(c[0], x[6], x[7], c[0], t1);
        fa(c[1], t0, t1, c[1], f1);
        fa(c[2], f0, f1, c[2], cy);
#pragma unroll
        for (int k = 3; k < N; k++) {
            const u32 t = c[k] & cy;
            c[k] ^= cy;
            cy = t;
        }
    }
    template <int N>
    __device__ static void add_unit(u32 (&c)[kPlanes], const u32* stage, u32 first, u32 end, u32 step, u32 pitch) {
        const u32 hop = step * pitch;
        const u32* p = stage + first * pitch;
        u32 e = first;
        for (; e + 7 * step < end; e += 8 * step, p += 8 * hop) {
            u32 x[8];
#pragma unroll
            for (u32 j = 0; j < 8; j++) x[j] = p[j * hop];
            add8<N>(c, x);
        }
        if (e < end) {
            u32 x[8];
#pragma unroll
            for (u32 j = 0; j < 8; j++) x[j] = e + j * step < end ? p[j * hop] : 0u;
            add8<N>(c, x);
        }
    }
    // Sum of the counts of the lanes o apart, P planes in, P + 1 out.
    template <int P>
    __device__ static void fold(u32 (&c)[kPlanes], u32 o) {
        constexpr int Q = P < kPlanes ? P : kPlanes;
        u32 carry = 0, y[Q];
#pragma unroll
        for (int k = 0; k < Q; k++) y[k] = __shfl_xor_sync(0xFFFFFFFFu, c[k], o);
#pragma unroll
        for (int k = 0; k < Q; k++) fa(c[k], y[k], carry, c[k], carry);
        if (Q < kPlanes) c[Q] = carry;
    }
    // The lanes' counts (N planes) of one word summed into all of them, then
    // f(query, slot, score) for the warp's words, lane = slot.
    template <int N, class FN>
    __device__ static void emit(u32 (&c)[kPlanes], u32* slab, u32 wpw, u32 q, u32 w0, u32 words, const joinc::Slots& st,
                                FN f) {
        const u32 lane = threadIdx.x & 31;
        if (wpw <= 16u) {
            fold<N>(c, 16u);
            if (wpw <= 8u) {
                fold<N + 1>(c, 8u);
                if (wpw <= 4u) {
                    fold<N + 2>(c, 4u);
                    if (wpw <= 2u) {
                        fold<N + 3>(c, 2u);
                        if (wpw <= 1u) fold<N + 4>(c, 1u);
                    }
                }
            }
        }
        // a word's planes go through shared memory: three 16-byte broadcasts
        // where a shuffle per plane was ten
        constexpr int F = N + 5 < kPlanes ? N + 5 : kPlanes;
        constexpr int V = (F + 3) / 4;
        if (lane < wpw) {
#pragma unroll
            for (int k = 0; k < V; k++)
                reinterpret_cast<uint4*>(slab)[lane * 3 + k] = make_uint4(c[4 * k], c[4 * k + 1], c[4 * k + 2], c[4 * k + 3]);
        }
        __syncwarp();
        for (u32 j = 0; j < words; j++) {
            u32 v = 0;
#pragma unroll
            for (int k = 0; k < V; k++) {
                const uint4 p = reinterpret_cast<const uint4*>(slab)[j * 3 + k];
                v |= ((p.x >> lane) & 1u) << (4 * k) | ((p.y >> lane) & 1u) << (4 * k + 1) |
                     ((p.z >> lane) & 1u) << (4 * k + 2) | ((p.w >> lane) & 1u) << (4 * k + 3);
            }
            const u32 x = (w0 + j) * 32 + lane;
            if (x < st.n) f(q, x, ord_f16((u16)half_bits_of_int(v)));
        }
        __syncwarp();
    }

    // Bytes of x equal to the code repeated in q4, as bit 7 of each byte.
    __device__ __forceinline__ static u32 equal_bytes(u32 x, u32 q4) {
        const u32 t = x ^ q4;
        return ~(((t & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | t);
    }
    // The scores from resident codes.
    template <class F, class D>
    __device__ static void scores_resident(const Args& m, Smem& s, const joinc::Slots& st, u32 nq, F f, D done) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const u32 lgq = nq <= 1 ? 4u : (nq <= 2 ? 3u : (nq <= 4 ? 2u : 1u));
        const u32 nwq = 1u << lgq, q = warp >> lgq, wi = warp & (nwq - 1u);
        const u32 nE = q < nq ? counts(s.par)[q] : 0u;
        const unsigned char* c8 = reinterpret_cast<const unsigned char*>(s.stage);
        const u32* list = s.eRow + (size_t)(q < nq ? q : 0u) * ncolW(m.ncol);
        const u32* wl = s.eW + (size_t)(q < nq ? q : 0u) * ncolW(m.ncol);
        if constexpr (HALF) {
            // a lane adds two neighbouring slots as a pair, the entries in order
            if (q < nq) {
                for (u32 x0 = 64 * wi; x0 < st.n; x0 += 64 * nwq) {
                    const u32 x = x0 + 2 * lane;
                    const unsigned char* c = c8 + (x < st.n ? x : x0);
                    u32 h = 0;
                    auto step = [&](u32 v, u32 en, u32 wt) {
                        const u32 eq = equal_bytes(v, __byte_perm(en, 0u, 0x4400u));
                        u32 mask;  // the two bytes' top bits over a half each
                        asm("prmt.b32 %0, %1, %1, 0x9988;" : "=r"(mask) : "r"(eq));
                        asm("add.rn.f16x2 %0, %0, %1;" : "+r"(h) : "r"(wt & mask));
                    };
                    u32 e = 0;
                    uint4 en[2], wt[2], ne[2], nw[2];
                    u32 v[8], nv[8];
                    auto load_list = [&](u32 at, uint4 (&a)[2], uint4 (&b)[2]) {
                        a[0] = *reinterpret_cast<const uint4*>(list + at);
                        a[1] = *reinterpret_cast<const uint4*>(list + at + 4);
                        b[0] = *reinterpret_cast<const uint4*>(wl + at);
                        b[1] = *reinterpret_cast<const uint4*>(wl + at + 4);
                    };
                    auto load_codes8 = [&](const uint4 (&a)[2], u32 (&to)[8]) {
                        const u32 o[8] = {a[0].x, a[0].y, a[0].z, a[0].w, a[1].x, a[1].y, a[1].z, a[1].w};
#pragma unroll
                        for (u32 k = 0; k < 8; k++) to[k] = *reinterpret_cast<const u16*>(c + (o[k] >> 8));
                    };
                    auto add8 = [&](const uint4 (&a)[2], const uint4 (&b)[2], const u32 (&x8)[8]) {
                        step(x8[0], a[0].x, b[0].x);
                        step(x8[1], a[0].y, b[0].y);
                        step(x8[2], a[0].z, b[0].z);
                        step(x8[3], a[0].w, b[0].w);
                        step(x8[4], a[1].x, b[1].x);
                        step(x8[5], a[1].y, b[1].y);
                        step(x8[6], a[1].z, b[1].z);
                        step(x8[7], a[1].w, b[1].w);
                    };
                    if (nE >= 8) {
                        load_list(0, en, wt);
                        load_codes8(en, v);
                        for (; e + 23 < nE; e += 16) {  // the next eight are loaded before these are added
                            load_list(e + 8, ne, nw);
                            load_codes8(ne, nv);
                            add8(en, wt, v);
                            load_list(e + 16, en, wt);
                            load_codes8(en, v);
                            add8(ne, nw, nv);
                        }
                        add8(en, wt, v);
                        e += 8;
                    }
                    for (; e < nE; e += 8) {  // the rest; past the end a weight of 0
                        u32 o[8], w8[8];
#pragma unroll
                        for (u32 k = 0; k < 8; k++) {
                            o[k] = e + k < nE ? list[e + k] : 0u;
                            w8[k] = e + k < nE ? wl[e + k] : 0u;
                        }
#pragma unroll
                        for (u32 k = 0; k < 8; k++) v[k] = *reinterpret_cast<const u16*>(c + (o[k] >> 8));
#pragma unroll
                        for (u32 k = 0; k < 8; k++) step(v[k], o[k], w8[k]);
                    }
                    if (x < st.n) f(q, x, ord_f16((u16)h));
                    if (x + 1 < st.n) f(q, x + 1, ord_f16((u16)(h >> 16)));
                }
                done(q);
            }
        } else {
            // lanes: words of four slots, lanes that share one when a warp has
            // more than the words; warps: 32-word chunks, then shares of the
            // entries.  Counts in 16 bits, bytes 0 and 2 of a word in one half
            // of the pair, 1 and 3 in the other.
            const u32 nw = (st.n + 3u) / 4u, chunks = (nw + 31u) / 32u;
            const u32 lgw = nw > 16u ? 5u : (nw > 8u ? 4u : (nw > 4u ? 3u : 2u));
            const u32 t = lane & ((1u << lgw) - 1u), sub = lane >> lgw;
            // warps that share a chunk's entries: a power of two, so that nothing
            // is divided
            const u32 lgc = chunks <= 1u ? 0u : 32u - __clz(chunks - 1u);
            const u32 lgg = lgc < lgq ? lgq - lgc : 0u, wg = 1u << lgg;
            const u32 NG = wg << (5u - lgw);
            u32* part = s.slab;
            if (q < nq) {
                const u32 g = wi & (wg - 1u);
                for (u32 ch = wi >> lgg; ch < chunks; ch += nwq >> lgg) {
                    const u32 word = 32 * ch + t;
                    u32 lo = 0, hi = 0;
                    if (word < nw) {
                        const unsigned char* c = c8 + 4 * word;
                        // eight entries at a time; past the end code 255, which
                        // no cell has
                        for (u32 b = g + wg * sub; b < nE; b += 8 * NG) {
                            u32 en[8], x[8], acc = 0;
#pragma unroll
                            for (u32 k = 0; k < 8; k++) en[k] = b + k * NG < nE ? list[b + k * NG] : 255u;
#pragma unroll
                            for (u32 k = 0; k < 8; k++) x[k] = *reinterpret_cast<const u32*>(c + (en[k] >> 8));
                            if (m.unitW) {
#pragma unroll
                                for (u32 k = 0; k < 8; k++)
                                    acc += (equal_bytes(x[k], __byte_perm(en[k], 0u, 0x0000u)) >> 7) & 0x01010101u;
                                lo += acc & 0x00FF00FFu;
                                hi += (acc >> 8) & 0x00FF00FFu;
                            } else {
#pragma unroll
                                for (u32 k = 0; k < 8; k++) {
                                    const u32 w = b + k * NG < nE ? wl[b + k * NG] : 0u;
                                    const u32 eq = equal_bytes(x[k], __byte_perm(en[k], 0u, 0x0000u)) >> 7;
                                    lo += (eq & 0x00010001u) * w;
                                    hi += ((eq >> 8) & 0x00010001u) * w;
                                }
                            }
                        }
                    }
                    for (u32 o = 1u << lgw; o < 32u; o <<= 1) {
                        lo += __shfl_xor_sync(0xFFFFFFFFu, lo, o);
                        hi += __shfl_xor_sync(0xFFFFFFFFu, hi, o);
                    }
                    if (sub == 0 && word < nw)
                        reinterpret_cast<uint2*>(part)[((size_t)q * wg + g) * nw + word] = make_uint2(lo, hi);
                }
            }
            __syncthreads();
            if (q < nq) {
                const u16* p16 = reinterpret_cast<const u16*>(part) + (size_t)q * wg * nw * 4;
                for (u32 x = 32 * wi + lane; x - lane < st.n; x += 32 * nwq) {
                    if (x < st.n) {
                        const u32 at = (x & ~3u) | ((x & 1u) << 1) | ((x >> 1) & 1u);
                        u32 v = 0;
#pragma unroll 8
                        for (u32 g = 0; g < wg; g++) v += p16[(size_t)g * nw * 4 + at];
                        f(q, x, ord_f16((u16)half_bits_of_int(v)));
                    }
                }
                done(q);
            }
        }
        if (s.prof) joinx::prof_mark(joinx::PROF_SC_RED);
    }

    template <class F, class D>
    __device__ static void scores(const Args& m, Smem& s, const joinc::Slots& st, u32 nq, F f, D done) {
        if (s.rp) {
            scores_resident(m, s, st, nq, f, done);
            return;
        }
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const u32 lgq = nq <= 1 ? 4u : (nq <= 2 ? 3u : (nq <= 4 ? 2u : 1u));
        const u32 nwq = 1u << lgq;  // warps per query
        const u32 q = warp >> lgq, wi = warp & (nwq - 1u);
        const u32 Wc = (st.n + 31u) / 32u, W4 = (Wc + 3u) & ~3u;
        const u32* cnt = counts(s.par);
        u32 total = 0, myOff = 0, most = 0;
        for (u32 i = 0; i < nq; i++) {
            if (i == q) myOff = total;
            total += cnt[i];
            most = max(most, cnt[i]);
        }
        const u32 myN = q < nq ? cnt[q] : 0u;
        const u32* wl = s.eW + (size_t)(q < nq ? q : 0u) * ncolW(m.ncol);
        if constexpr (HALF) {
            // two words a warp, so a lane adds the two slots of its bit as a
            // pair: one 8-byte load of the words and a quarter of a 16-byte load
            // of the weights serve both (with a load of either per word and
            // entry, the shared-memory loads set the time: 1.8 us a phase at 120
            // entries of 8 words)
            u32* sums = s.sums + (size_t)(q < nq ? q : 0u) * (st.cap / 2);
            const u32 per = total * W4 <= m.stageWords ? max(total, 1u) : m.stageWords / W4 & ~7u;
            const u32 pairs = (Wc + 1u) / 2u;
            auto walk = [&](u32 r0, u32 a, u32 b) {
                const u32 lo = max(a, myOff), hi = min(b, myOff + myN);
                if (q >= nq || lo >= hi) return;
                for (u32 pr = wi; pr < pairs; pr += nwq) {
                    u32 h = lo > myOff ? sums[pr * 32 + lane] : 0u;
                    const u32* col = s.stage + 2 * pr;
                    // adding +0 leaves a sum of non-negative weights as it is
                    auto step = [&](uint2 v, u32 wt) {
                        const u32 bits = __byte_perm(v.x >> lane, v.y >> lane, 0x5410u) & 0x00010001u;
                        const u32 w = wt & (bits * 0xFFFFu);
                        asm("add.rn.f16x2 %0, %0, %1;" : "+r"(h) : "r"(w));
                    };
                    const u32 end = hi - r0;
                    u32 e = lo - r0;
                    const u32* w = wl + (lo - myOff);  // entry e's weight, advanced with e
                    if (((lo - myOff) & 3u) == 0u) {
                        // the next eight entries are loaded before these are added
                        uint2 v[8], nv[8];
                        uint4 w0, w1, nw0, nw1;
                        auto load = [&](u32 at, const u32* wp, uint2 (&x)[8], uint4& a0, uint4& a1) {
#pragma unroll
                            for (u32 k = 0; k < 8; k++) x[k] = *reinterpret_cast<const uint2*>(col + (at + k) * W4);
                            a0 = reinterpret_cast<const uint4*>(wp)[0];
                            a1 = reinterpret_cast<const uint4*>(wp)[1];
                        };
                        auto add = [&](const uint2 (&x)[8], const uint4& a0, const uint4& a1) {
                            step(x[0], a0.x);
                            step(x[1], a0.y);
                            step(x[2], a0.z);
                            step(x[3], a0.w);
                            step(x[4], a1.x);
                            step(x[5], a1.y);
                            step(x[6], a1.z);
                            step(x[7], a1.w);
                        };
                        if (e + 7 < end) {
                            load(e, w, v, w0, w1);
                            for (; e + 23 < end; e += 16, w += 16) {
                                load(e + 8, w + 8, nv, nw0, nw1);
                                add(v, w0, w1);
                                load(e + 16, w + 16, v, w0, w1);
                                add(nv, nw0, nw1);
                            }
                            add(v, w0, w1);
                            e += 8;
                            w += 8;
                        }
                    }
                    for (; e < end; e += 8, w += 8) {  // words past the end 0
                        uint2 v[8];
                        u32 wt[8];
#pragma unroll
                        for (u32 k = 0; k < 8; k++) {
                            v[k] = e + k < end ? *reinterpret_cast<const uint2*>(col + (e + k) * W4) : make_uint2(0u, 0u);
                            wt[k] = e + k < end ? w[k] : 0u;
                        }
#pragma unroll
                        for (u32 k = 0; k < 8; k++) step(v[k], wt[k]);
                    }
                    sums[pr * 32 + lane] = h;
                }
            };
            if (Wc) rounds(m, s, nq, total, per, 0u, W4, W4, walk);
            // the same lanes that formed the sums read them
            if (q < nq) {
                for (u32 pr = wi; pr < pairs; pr += nwq) {
                    const u32 x = pr * 64 + lane, h = myN ? sums[pr * 32 + lane] : 0u;
                    if (x < st.n) f(q, x, ord_f16((u16)h));
                    if (x + 32 < st.n) f(q, x + 32, ord_f16((u16)(h >> 16)));
                }
                done(q);
            }
            if (s.prof) joinx::prof_mark(joinx::PROF_SC_RED);
        } else {
        for (u32 wb = 0; wb < Wc; wb += 32u * nwq) {
            const u32 wp = min(Wc - wb, 32u * nwq), wst = min(W4 - wb, 32u * nwq);  // words of this pass, staged
            const u32 need = (wp + nwq - 1u) >> lgq;
            const u32 lgw = need <= 1u ? 0u : 32u - __clz(need - 1u), wpw = 1u << lgw;  // words per warp
            // a stage pitch that spreads the lanes' (entry, word) reads over the banks
            const u32 pitch = wpw >= 32u ? wst : (wpw >= 4u ? wst + ((wpw - wst) & 31u) : wst + ((4u - wst) & 7u));
            const u32 t = lane & (wpw - 1u), g = lane >> lgw, NG = 32u >> lgw;
            const u32 word = wi * wpw + t;
            const bool act = q < nq && word < wp;
            const bool one = total * pitch <= m.stageWords;
            const u32 per = one ? max(total, 1u) : m.stageWords / pitch & ~7u;
            // a lane's entries, at most: a share of the two halves of every round
            const u32 mostLane = (most >> (5u - lgw)) + (one ? 2u : 2u * (total / per + 1u));
            u32 c[kPlanes];
#pragma unroll
            for (int i = 0; i < kPlanes; i++) c[i] = 0u;
            rounds(m, s, nq, total, per, wb, wst, pitch, [&](u32 r0, u32 a, u32 b) {
                const u32 lo = max(a, myOff), hi = min(b, myOff + myN);
                if (!act || lo >= hi) return;
                const u32* stage = s.stage + word;
                if (m.unitW) {
                    if (mostLane <= 7u) add_unit<3>(c, stage, lo - r0 + g, hi - r0, NG, pitch);
                    else if (mostLane <= 31u) add_unit<5>(c, stage, lo - r0 + g, hi - r0, NG, pitch);
                    else if (mostLane <= 127u) add_unit<7>(c, stage, lo - r0 + g, hi - r0, NG, pitch);
                    else add_unit<kPlanes>(c, stage, lo - r0 + g, hi - r0, NG, pitch);
                } else {
                    for (u32 e = lo - r0 + g; e < hi - r0; e += NG) vadd(c, stage[e * pitch], wl[e + r0 - myOff]);
                }
            });
            u32* slab = s.slab + warp * 32 * 12;
            const u32 mine = q < nq && wi * wpw < wp ? min(wpw, wp - wi * wpw) : 0u;
            if (m.unitW && mostLane <= 7u) emit<3>(c, slab, wpw, q, wb + wi * wpw, mine, st, f);
            else if (m.unitW && mostLane <= 31u) emit<5>(c, slab, wpw, q, wb + wi * wpw, mine, st, f);
            else if (m.unitW && mostLane <= 127u) emit<7>(c, slab, wpw, q, wb + wi * wpw, mine, st, f);
            else emit<kPlanes>(c, slab, wpw, q, wb + wi * wpw, mine, st, f);
            if (wb + 32u * nwq < Wc) __syncthreads();
        }
        if (q < nq) done(q);
        }
        if (s.prof) joinx::prof_mark(joinx::PROF_SC_RED);
    }

    // Sixteenths of the slots that are still live when the dead are squeezed
    // out; the same for all CTAs (so nothing of this CTA's slots goes in).
    // Scans of fewer dead slots pay for clearing all bitset rows, unless there
    // are many rows a slot: 40,000 x 1,024 x 256 alleles 464 ms at 8 and 433 at
    // 12, 8,000 x 500 x 64 55.0 and 52.8, but 12,345 x 777 x 256 99.7 and 101.2.
    __device__ static u32 compact_at(const Args& m, u32 S) { return m.rows <= 8u * S ? 12u : 8u; }
    // Rebuilds this CTA's words in the other buffer from the live slots' rows.
    // The engine has moved st.node already; n live slots.
    __device__ static void compact(const joinc::Args&, const Args& m, Smem& s, u32, const joinc::Slots& st, u32 n,
                                   const u16*) {
        const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        s.rp = resident_pitch(m, n);
        if (s.rp) {
            load_codes(m, s, st, n);
            __syncthreads();
            return;
        }
        u32* B = s.other;
        const u32 pitch = (n + 127u) / 128u * 4u;
        const size_t pieces = (size_t)m.rows * pitch / 4;
        for (size_t i = threadIdx.x; i < pieces; i += kThreads) reinterpret_cast<uint4*>(B)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        for (u32 x = warp; x < n; x += joinc::kWarps) {
            const u16* row = m.nodeRow + (size_t)st.node[x] * m.ncolP;
            const u32 word = x >> 5, bit = 1u << (x & 31);
            for (u32 i = 2 * lane; i < m.ncolP; i += 64) {
                const u32 c = ld_cg_u32(reinterpret_cast<const u32*>(row + i));
                if ((c & 0xFFFFu) > 1u) atomicOr(B + ((size_t)i * m.nState + (c & 0xFFFFu) - 2u) * pitch + word, bit);
                if ((c >> 16) > 1u) atomicOr(B + ((size_t)(i + 1) * m.nState + (c >> 16) - 2u) * pitch + word, bit);
            }
        }
        s.other = s.B;
        s.B = B;
        s.pitch = pitch;
        __syncthreads();
    }
};

// Bitset rows [row][Wd] -> one block of rows per CTA of the cluster,
// [rank][row][pitch] (words past the row's end are 0).
__global__ void k_split_bits(const u32* __restrict__ bits, u32 rows, u32 Wd, u32 pitch, u32* __restrict__ out) {
    const u32 p4 = pitch / 4, w0 = blockIdx.y * pitch;
    const size_t n = (size_t)rows * p4;
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.y * rows * pitch);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i / p4;
        const u32 w = w0 + 4u * (u32)(i - row * p4);
        dst[i] = w < Wd ? *reinterpret_cast<const uint4*>(bits + row * Wd + w) : make_uint4(0u, 0u, 0u, 0u);
    }
}

template <class M>
__global__ void __launch_bounds__(joinc::kThreads, 1) k_cluster_join(joinc::Args a, typename M::Args m) {
    extern __shared__ __align__(16) unsigned char smem[];
    joinc::cluster_join<M>(a, m, joinc::cluster_rank(), smem);
}

}  // namespace indel
}  // namespace casphy
