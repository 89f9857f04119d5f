// Shared-bit counts of all row pairs on the tensor cores.
//
// The number of bits set in both of two rows is the dot product of the rows
// as 0/1 vectors, so the counts of a 128 x 256 tile of pairs are one
// 128 x 256 x K integer contraction (tcgen05.mma kind::i8, 32-bit integer
// accumulators in tensor memory: the counts are exact).  Popcounts of ANDed
// words run at 16 a clock and SM, that is 512 bit pairs; the tensor core does
// 8,192.
//
// Rows are kept as bits, [chunk][row] of 128 bits, and expanded to bytes in
// shared memory, so a tile reads an eighth of a byte per element from L2: with
// byte rows the 160 MB of a 20,000 x 2,000 alignment's planes would be read at
// 3 MB a tile, and the reads, not the products, would set the time.  The
// expansion is one AND per four bytes: bit 4h + i of a byte becomes the value
// 2^i on the A side and, from the byte reversed, 2^(3-i) on the B side, so
// every pair of set bits contributes 8.  Shared memory is the bound: 48 KB
// written and 48 KB read per 128 x 256 x 128 step, 768 clocks against 512 of
// the products.  Two CTAs share an SM, so that one's epilogue runs under the
// other's products.
#pragma once
#include "common.cuh"

namespace casphy {
namespace bitdot {

constexpr u32 kM = 128, kN = 256;
constexpr u32 kThreads = kM + kN;                 // one row each
constexpr u32 kStageBytes = (kM + kN) * 128;      // one chunk of both sides as bytes
constexpr u32 kSmemBytes = 2 * kStageBytes;
constexpr u64 kLimitNs = 4ull * 1000 * 1000 * 1000;

struct Args {
    const uint4* A;      // [chunk][ldA]: rows a0 .. a0 + rowsA - 1 are the tile rows
    const uint4* B;      // [chunk][ldB]: rows 0 .. rowsB - 1 are the tile columns
    u32 ldA, ldB, a0, rowsA, rowsB;
    u32 chunks;          // 128-bit chunks; those from negFrom on count -3 a pair
    u32 negFrom;
    u32 upper;           // 1: only tiles with a column not below their rows (A = B)
    u32 tilesN;          // column tiles
    const u32* mode;     // device word or null: 0 leaves out the chunks from negFrom, above 1 does nothing
    int* err;
};

__device__ __forceinline__ u32 smem_addr(const void* p) { return static_cast<u32>(__cvta_generic_to_shared(p)); }

// Shared-memory matrix descriptor: K-major, no swizzle; 8-row x 16-byte core
// matrices, 128 bytes apart along K and 1,024 along the rows.
__device__ __forceinline__ u64 matrix_desc(u32 addr) {
    return (u64)((addr & 0x3FFFFu) >> 4) | ((u64)(128u >> 4) << 16) | ((u64)(1024u >> 4) << 32) | (1ull << 46);
}
// 32-bit integer accumulators, signed bytes, 128 x 256
constexpr u32 kInstrDesc = (2u << 4) | (1u << 7) | (1u << 10) | ((kN >> 3) << 17) | ((kM >> 4) << 24);

__device__ __forceinline__ bool bar_try(u32 bar, u32 parity) {
    u32 ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0u;
}
// Waits for the phase, at most kLimitNs; false records CASPHY_ETIMEOUT.
__device__ __forceinline__ bool bar_wait(u32 bar, u32 parity, int* err) {
    if (bar_try(bar, parity)) return true;
    const u64 t0 = globaltimer_ns();
    while (!bar_try(bar, parity))
        if (globaltimer_ns() - t0 > kLimitNs) {
            atomicCAS(err, 0, CASPHY_ETIMEOUT);
            return false;
        }
    return true;
}

// 32 accumulator columns of this warp's 32 rows.
__device__ __forceinline__ void load32(u32 addr, u32 (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// One row's 128 bits as bytes of a K-major tile row.
__device__ __forceinline__ void expand_row(unsigned char* tileRow, const uint4 v, bool sideB, bool neg) {
    const u32 w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (u32 q = 0; q < 4; q++) {
        // (the byte reversal turns bit 4h + i of a byte into bit 7 - 4h - i)
        const u32 r = sideB ? __byte_perm(__brev(w[q]), 0u, 0x0123u) : w[q];
#pragma unroll
        for (u32 h = 0; h < 2; h++) {
            const u32 src = (h == 1) == sideB ? r : r >> 4;
            u32 o[4];
#pragma unroll
            for (u32 i = 0; i < 4; i++) {
                const u32 at = sideB ? 3u - i : i;
                o[i] = src & (0x01010101u << at);
                // -3 * 2^(3-i) in a byte
                if (neg && sideB) o[i] = (o[i] >> at) * ((0x100u - 3u * (1u << at)) & 0xFFu);
            }
            *reinterpret_cast<uint4*>(tileRow + (2 * q + h) * 128) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// Tile (mb, nb) of linear index t among the tiles with nb >= mb / 2.
__device__ __forceinline__ void upper_tile(u32 t, u32 tilesN, u32& mb, u32& nb) {
    // pair p = mb / 2 starts at tile 2 (p tilesN - p (p - 1) / 2)
    u32 lo = 0, hi = tilesN;
    while (hi - lo > 1) {
        const u32 p = (lo + hi) / 2;
        if (2 * (p * tilesN - p * (p - 1) / 2) <= t) lo = p;
        else hi = p;
    }
    const u32 in = t - 2 * (lo * tilesN - (lo ? lo * (lo - 1) / 2 : 0u));
    const u32 per = tilesN - lo;
    mb = 2 * lo + in / per;
    nb = lo + in % per;
}

// One tile per CTA.  E::tile(p, m0, n0, taddr) reads the accumulators (eight
// times the counts; lane l of warp w holds row 32 (w % 4) + l) and is called by
// all warps of the CTA.  With E::kBatched the grid covers the tiles of many
// matrices: E::pick(a, p, block) fills in the rows of this block's and returns
// the tile's index there.
template <class E>
__global__ void __launch_bounds__(kThreads, 2) k_bitdot(Args a, typename E::Params p) {
    extern __shared__ __align__(128) unsigned char stage[];
    __shared__ __align__(8) u64 s_bar[2];
    __shared__ u32 s_tmem;
    const u32 tid = threadIdx.x, warp = tid >> 5;
    u32 index = blockIdx.x;
    if constexpr (E::kBatched) index = E::pick(a, p, index);
    const u32 mode = a.mode ? *a.mode : 1u;
    if (mode > 1u) return;
    const u32 chunks = mode ? a.chunks : a.negFrom;
    u32 mb, nb;
    if (a.upper) upper_tile(index, a.tilesN, mb, nb);
    else {
        mb = index / a.tilesN;
        nb = index % a.tilesN;
    }
    const u32 m0 = mb * kM, n0 = nb * kN;
    if (m0 >= a.rowsA) return;  // (an odd number of row tiles)
    const u32 bar = smem_addr(&s_bar[0]);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)), "r"(kN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 32) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const u32 tmem = s_tmem;

    const bool sideB = tid >= kM;
    const u32 row = sideB ? tid - kM : tid;
    const bool in = sideB ? n0 + row < a.rowsB : m0 + row < a.rowsA;
    const uint4* src = sideB ? a.B + n0 + row : a.A + a.a0 + m0 + row;
    const size_t ld = sideB ? a.ldB : a.ldA;
    unsigned char* mine = stage + (sideB ? kM * 128u : 0u) + (row >> 3) * 1024u + (row & 7u) * 16u;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 v = in ? src[0] : zero;
    bool ok = true;
    for (u32 c = 0; c < chunks; c++) {
        const u32 s = c & 1u;
        const uint4 next = in && c + 1 < chunks ? src[(c + 1) * ld] : zero;
        if (c >= 2) ok = bar_wait(bar + 8 * s, ((c >> 1) - 1) & 1u, a.err);  // the stage's last products are done
        expand_row(mine + s * kStageBytes, v, sideB, c >= a.negFrom);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const u32 at = smem_addr(stage) + s * kStageBytes;
#pragma unroll
            for (u32 k = 0; k < 4; k++) {  // 32 elements a step: two core matrices along K
                const u64 da = matrix_desc(at + k * 256u), db = matrix_desc(at + kM * 128u + k * 256u);
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(kInstrDesc), "r"(c + k)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar + 8 * s)
                         : "memory");
        }
        v = next;
    }
    // all products done (on failure too: the tile is then dropped)
    const u32 last = chunks - 1;
    if (ok) ok = bar_wait(bar + 8 * (last & 1u), (last >> 1) & 1u, a.err);
    ok = !__syncthreads_or(!ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) E::tile(a, p, m0, n0, tmem, stage);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kN) : "memory");
}

// Tiles of the grid.
inline u32 tiles_n(u32 rowsB) { return (rowsB + kN - 1) / kN; }
inline u64 tiles(u32 rowsA, u32 rowsB, bool upper) {
    const u64 N = tiles_n(rowsB);
    return upper ? N * (N + 1) : (u64)((rowsA + kM - 1) / kM) * N;
}

}  // namespace bitdot
}  // namespace casphy
