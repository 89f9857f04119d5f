// TransferDisStream on B200 (replaces cu/TransferDisStream.cu).
//
// For clade bitsets X (nrow_x rows) and Y (nrow_y rows) over ntip tips packed
// in ncol u32 words, the reference keeps, per x row, the minimum over y of
// min(d, c - pad) with d = popc(x ^ y), c = popc(x ^ ~y) = 32*ncol - d and
// pad = 32*ncol - ntip, but forms the two minima separately over aligned
// groups of 8 y rows before subtracting pad (u32 arithmetic), and seeds
// missing rows of a partial group with 32*ncol (cu/TransferDisStream.cu:
// 39-104); y rows symmetrically over groups of 8 x rows.  That grouping
// changes the result only when rows carry bits past ntip, and it is kept
// exactly.  Sizes are min(k, ntip - k), k = popcount of the row (:107-121).
//
// d = |x| + |y| - 2 |x n y|, so the distances of a 128 x 256 tile of pairs are
// one tensor-core contraction (bitdot.cuh) and the row popcounts; the tile's
// epilogue forms the grouped minima from them (groups of 8 columns in a thread,
// groups of 8 rows by shuffles), one atomicMin per row and column of the tile.
// 9,998 x 9,998 rows of 313 words: popcounts of the XORed words took 7 ms.  Calls
// of few row pairs and words keep to those (k_cross).
#include <algorithm>

#include "bitdot.cuh"
#include "common.cuh"
#include "runtime.h"

namespace casphy {
namespace tdis {

struct TransferTile {
    static constexpr bool kBatched = false;
    struct Params {
        u32 full, pad;  // 32 ncol, and the bits past ntip
        const u32* cx;  // popcounts of the rows
        const u32* cy;
        u32* xmin;
        u32* ymin;
    };
    // x rows are the tile's rows, y rows its columns
    __device__ static void tile(const bitdot::Args& a, const Params& p, u32 m0, u32 n0, u32 taddr, unsigned char* smem) {
        u32* s_cy = reinterpret_cast<u32*>(smem);  // kN
        u32* s_y = s_cy + bitdot::kN;              // kN
        u32* s_x = s_y + bitdot::kN;               // kM
        const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp & 3u;
        if (tid < bitdot::kN) {
            s_cy[tid] = n0 + tid < a.rowsB ? p.cy[n0 + tid] : 0u;
            s_y[tid] = 0xFFFFFFFFu;
        }
        if (tid < bitdot::kM) s_x[tid] = 0xFFFFFFFFu;
        __syncthreads();
        const u32 x = m0 + 32 * wr + lane;
        const bool xok = x < a.rowsA, gok = (x & ~7u) < a.rowsA;
        const u32 mc = xok ? p.cx[x] : 0u;
        u32 xm = 0xFFFFFFFFu;
        for (u32 cb = warp >> 2; cb < bitdot::kN / 32; cb += bitdot::kThreads / 128) {
            u32 r[32], keep = 0xFFFFFFFFu;
            bitdot::load32(taddr + (32 * wr << 16) + cb * 32, r);
            const u32 n = n0 + cb * 32;
#pragma unroll
            for (u32 g = 0; g < 4; g++) {
                u32 A = p.full, B = p.full;
#pragma unroll
                for (u32 i = 0; i < 8; i++) {
                    const u32 j = 8 * g + i;
                    const u32 d = mc + s_cy[cb * 32 + j] - (r[j] >> 2);  // the accumulator is 8 |x n y|
                    if (n + j < a.rowsB) {
                        A = min(A, d);
                        B = min(B, p.full - d);
                    }
                    u32 ya = xok ? d : p.full, yb = xok ? p.full - d : p.full;
#pragma unroll
                    for (u32 o = 1; o < 8; o <<= 1) {
                        ya = min(ya, __shfl_xor_sync(0xFFFFFFFFu, ya, o));
                        yb = min(yb, __shfl_xor_sync(0xFFFFFFFFu, yb, o));
                    }
                    u32 v = gok ? min(ya, yb - p.pad) : 0xFFFFFFFFu;
                    v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, 8));
                    v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, 16));
                    if (lane == j) keep = v;
                }
                if (n + 8 * g < a.rowsB) xm = min(xm, min(A, B - p.pad));
            }
            if (n + lane < a.rowsB) atomicMin(s_y + cb * 32 + lane, keep);
        }
        if (xok) atomicMin(s_x + 32 * wr + lane, xm);
        __syncthreads();
        if (tid < bitdot::kN && n0 + tid < a.rowsB) atomicMin(p.ymin + n0 + tid, s_y[tid]);
        if (tid < bitdot::kM && m0 + tid < a.rowsA) atomicMin(p.xmin + m0 + tid, s_x[tid]);
    }
};

// Sizes and the minima's start of both sides' rows, rows of y first: a warp a row.
__global__ void __launch_bounds__(256) k_sizes(const u32* __restrict__ Y, u32 ny, const u32* __restrict__ X, u32 nx, u32 ncol,
                                               u32 ntip, u32* __restrict__ ysize, u32* __restrict__ ymin,
                                               u32* __restrict__ xsize, u32* __restrict__ xmin) {
    const u32 i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= ny + nx) return;
    const bool isY = i < ny;
    const u32 r = isY ? i : i - ny;
    const u32* row = (isY ? Y : X) + (size_t)r * ncol;
    u32 c = 0;
    for (u32 k = lane; k < ncol; k += 32) c += (u32)__popc(row[k]);
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if (lane == 0) {
        (isY ? ysize : xsize)[r] = c > ntip - c ? ntip - c : c;
        (isY ? ymin : xmin)[r] = 32u * ncol;
    }
}

// Distances of 32 x rows (lanes) and 64 y rows (a group of eight a warp) from the
// XORed words, 32 words of both at a time in shared memory.
constexpr u32 kTX = 32, kTY = 64, kWords = 32;
__global__ void __launch_bounds__(256) k_cross(const u32* __restrict__ X, const u32* __restrict__ Y, u32 nx, u32 ny, u32 ncol,
                                               u32 ntip, u32* __restrict__ xmin, u32* __restrict__ ymin) {
    __shared__ u32 xs[kTX][kWords + 1];
    __shared__ u32 ys[kTY][kWords];
    __shared__ u32 red[8][kTX];
    const u32 lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const u32 x0 = blockIdx.x * kTX, y0 = blockIdx.y * kTY, x = x0 + lane;
    u32 d[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (u32 k0 = 0; k0 < ncol; k0 += kWords) {
        const u32 k = k0 + lane;
        for (u32 r = w; r < kTX; r += 8) xs[r][lane] = x0 + r < nx && k < ncol ? X[(size_t)(x0 + r) * ncol + k] : 0u;
        for (u32 r = w; r < kTY; r += 8) ys[r][lane] = y0 + r < ny && k < ncol ? Y[(size_t)(y0 + r) * ncol + k] : 0u;
        __syncthreads();
        const u32 kn = min(kWords, ncol - k0);
        for (u32 j = 0; j < kn; j++) {
            const u32 v = xs[lane][j];
#pragma unroll
            for (u32 i = 0; i < 8; i++) d[i] += (u32)__popc(v ^ ys[8 * w + i][j]);
        }
        __syncthreads();
    }
    const u32 full = 32u * ncol, pad = full - ntip;
    const bool xok = x < nx;
    u32 A = full, B = full;
#pragma unroll
    for (u32 i = 0; i < 8; i++) {
        const u32 yr = y0 + 8 * w + i;
        if (yr < ny) {
            A = min(A, d[i]);
            B = min(B, full - d[i]);
        }
        u32 ya = xok ? d[i] : full, yb = xok ? full - d[i] : full;
#pragma unroll
        for (u32 o = 1; o < 8; o <<= 1) {
            ya = min(ya, __shfl_xor_sync(0xFFFFFFFFu, ya, o));
            yb = min(yb, __shfl_xor_sync(0xFFFFFFFFu, yb, o));
        }
        u32 v = (x & ~7u) < nx ? min(ya, yb - pad) : 0xFFFFFFFFu;  // groups of eight x rows
        v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, 8));
        v = min(v, __shfl_xor_sync(0xFFFFFFFFu, v, 16));
        if (lane == 0 && yr < ny) atomicMin(ymin + yr, v);
    }
    red[w][lane] = min(A, B - pad);
    __syncthreads();
    if (w == 0 && xok) {
        u32 v = red[0][lane];
        for (u32 g = 1; g < 8 && y0 + 8 * g < ny; g++) v = min(v, red[g][lane]);
        atomicMin(xmin + x, v);
    }
}

// Whether the popcounts are the quicker: where row pairs x words are few, because
// the rows are not packed and the tiles' step is long, or where the blocks are too
// few to fill the device, because a step of theirs takes 0.12 us a word and one of the
// tiles 0.19.  Calls by popcounts and by tiles: 5 x 5 clades x 1 word 44 and 62 us,
// 998 x 998 x 32 (32 million) 79 and 93, 5,000 x 100 x 157 (78) 315 and 324, 1,498 x
// 1,498 x 47 (105) 150 and 153, then 20,000 x 2,000 x 4 (160) 256 and 224, 1,998 x
// 1,998 x 63 (251) 205 and 172, 100 x 10,000 x 313 (313) 883 and 814; of few blocks,
// 200 x 200 x 3,000 (120 million, 28 blocks) 748 and 905, 600 x 600 x 1,000 (360, 190
// blocks) 501 and 507, then 800 x 800 x 300 (192, 325 blocks) 231 and 223.
constexpr u64 kPopcounts = 100000000;
constexpr u32 kPopBlocks = 240;
static bool popcounts_pay(u64 ny, u64 nx, u64 ncol) {
    const u64 blocksY = (ny + kTY - 1) / kTY, blocks = (nx + kTX - 1) / kTX * blocksY;
    return blocksY <= 65535 && (blocks <= kPopBlocks || ny * nx <= kPopcounts / ncol);
}

// Rows r00 .. r00 + m - 1 of n, ncol words each (M: row r00) -> 128-bit chunks,
// uint4 at [c * n + row], and the rows' popcounts and sizes, and the minima's start:
// a block takes 32 rows, a warp four of them at a time.  Clears *err for the kernel
// that follows.
__global__ void __launch_bounds__(256) k_pack_rows(const u32* __restrict__ M, u32 r00, u32 m, u32 n, u32 ncol, u32 ntip,
                                                   uint4* __restrict__ out, u32* __restrict__ pop, u32* __restrict__ size,
                                                   u32* __restrict__ least, int* err) {
    __shared__ u32 t[32][33];
    if (blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = blockIdx.x * 32;
    u32 cnt[4] = {0u, 0u, 0u, 0u};  // rows r0 + warp + 8 i
    for (u32 k0 = 0; k0 < ncol; k0 += 32) {
#pragma unroll
        for (u32 i = 0; i < 4; i++) {
            const u32 r = r0 + warp + 8 * i, k = k0 + lane;
            const u32 v = r < m && k < ncol ? M[(size_t)r * ncol + k] : 0u;
            t[warp + 8 * i][lane] = v;
            cnt[i] += (u32)__popc(v);
        }
        __syncthreads();
        // warp w: chunk w of the eight, lane = row
        const u32 c = k0 / 4 + warp;
        if (4 * c < ncol && r0 + lane < m)
            out[(size_t)c * n + r00 + r0 + lane] =
                make_uint4(t[lane][4 * warp], t[lane][4 * warp + 1], t[lane][4 * warp + 2], t[lane][4 * warp + 3]);
        __syncthreads();
    }
#pragma unroll
    for (u32 i = 0; i < 4; i++) {
        const u32 c = __reduce_add_sync(0xFFFFFFFFu, cnt[i]), r = r0 + warp + 8 * i;
        if (lane == 0 && r < m) {
            pop[r00 + r] = c;
            size[r00 + r] = c > ntip - c ? ntip - c : c;
            least[r00 + r] = 32u * ncol;
        }
    }
}

}  // namespace tdis

// Rows of one side on the device.
struct TransferSide {
    u32 n;
    const u32* host;
    uint4* chunks;
    u32* pop;
    u32 *least, *size;  // minima and sizes
};

// Uploads and packs a side's rows, `per` at a time through `panel`.  The chunks are
// all that is kept: beside the rows themselves they would take twice the memory,
// and 600,000 clades a side (90 GB) would not fit any more.
constexpr size_t kPanelBytes = size_t(64) << 20;
static u32 panel_rows(u32 n, u32 ncol) {
    return std::min(n, (u32)std::max<size_t>(kPanelBytes / (sizeof(u32) * ncol) / 32 * 32, 32));
}
static int pack_side(DeviceScope& ds, const TransferSide& s, u32 ncol, u32 ntip, u32* panel, int* err, cudaStream_t st) {
    const u32 per = panel_rows(s.n, ncol);
    for (u32 r = 0; r < s.n; r += per) {
        const u32 m = std::min(per, s.n - r);
        if (int rc = Staged::to_device(ds, panel, s.host + (size_t)r * ncol, sizeof(u32) * (size_t)m * ncol, st)) return rc;
        tdis::k_pack_rows<<<(m + 31) / 32, 256, 0, st>>>(panel, r, m, s.n, ncol, ntip, s.chunks, s.pop, s.size, s.least, err);
    }
    return CASPHY_OK;
}

static int transfer_tiles(const TransferSide& y, const TransferSide& x, u32 ncol, u32 ntip, int* err, cudaStream_t st) {
    using namespace tdis;
    const u32 full = 32u * ncol, nx = x.n, ny = y.n;
    if (nx && ny) {
        bitdot::Args a{};
        a.A = x.chunks;
        a.B = y.chunks;
        a.ldA = a.rowsA = nx;
        a.ldB = a.rowsB = ny;
        a.chunks = a.negFrom = (ncol + 3) / 4;
        a.tilesN = bitdot::tiles_n(ny);
        a.err = err;
        const u64 nt = bitdot::tiles(nx, ny, false);
        if (nt > 0x7FFFFFFFull) {
            casphy_set_last_error_msg("transfer: too many rows");
            return CASPHY_ERANGE;
        }
        CASPHY_CUDA_TRY(cudaFuncSetAttribute((void*)bitdot::k_bitdot<TransferTile>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bitdot::kSmemBytes));
        bitdot::k_bitdot<TransferTile><<<(u32)nt, bitdot::kThreads, bitdot::kSmemBytes, st>>>(
            a, TransferTile::Params{full, full - ntip, x.pop, y.pop, x.least, y.least});
    }
    CASPHY_CUDA_TRY(cudaGetLastError());
    return CASPHY_OK;
}

// Both sides' rows into `rows`, then sizes and distances by popcounts.
static int transfer_popcounts(DeviceScope& ds, const TransferSide& y, const TransferSide& x, u32 ncol, u32 ntip, u32* rows,
                              cudaStream_t st) {
    using namespace tdis;
    u32* dx = rows + (size_t)y.n * ncol;
    if (y.n)
        if (int rc = Staged::to_device(ds, rows, y.host, sizeof(u32) * (size_t)y.n * ncol, st)) return rc;
    if (x.n)
        if (int rc = Staged::to_device(ds, dx, x.host, sizeof(u32) * (size_t)x.n * ncol, st)) return rc;
    k_sizes<<<(y.n + x.n + 7) / 8, 256, 0, st>>>(rows, y.n, dx, x.n, ncol, ntip, y.size, y.least, x.size, x.least);
    if (x.n && y.n)
        k_cross<<<dim3((x.n + kTX - 1) / kTX, (y.n + kTY - 1) / kTY), 256, 0, st>>>(dx, rows, x.n, y.n, ncol, ntip, x.least,
                                                                                y.least);
    CASPHY_CUDA_TRY(cudaGetLastError());
    return CASPHY_OK;
}

}  // namespace casphy

extern "C" int casphy_transfer_dis(uint32_t nrow_y, uint32_t nrow_x, uint32_t ncol, uint32_t ntip, const uint32_t* y,
                                   const uint32_t* x, uint32_t* ymin, uint32_t* ysize, uint32_t* xmin,
                                   uint32_t* xsize) {
    using namespace casphy;
    int rc = require_device();
    if (rc) return rc;
    if (ncol == 0 || (nrow_y && (!y || !ymin || !ysize)) || (nrow_x && (!x || !xmin || !xsize))) return CASPHY_EINVAL;
    if (!nrow_y && !nrow_x) return CASPHY_OK;
    DeviceScope ds;
    cudaStream_t st = 0;
    const u64 nrow = (u64)nrow_y + nrow_x;
    const bool tiles = nrow > 0xFFFFFFFFull || !tdis::popcounts_pay(nrow_y, nrow_x, ncol);
    const u32 per = std::max(panel_rows(nrow_y, ncol), panel_rows(nrow_x, ncol));
    const size_t chunks = (ncol + 3) / 4;
    TransferSide Y{nrow_y, y, nullptr, nullptr, nullptr, nullptr}, X{nrow_x, x, nullptr, nullptr, nullptr, nullptr};
    u32 *panel, *out;
    auto lay = [&](Carve& c) {
        // minima and sizes of both sides and the error of a device-side wait, read
        // back together
        out = c.take<u32>(2 * (size_t)nrow + 1);
        if (!tiles) {  // both sides' rows
            panel = c.take<u32>((size_t)nrow * ncol);
            return;
        }
        panel = c.take<u32>((size_t)per * ncol);
        for (TransferSide* s : {&Y, &X}) {
            s->chunks = c.take<uint4>(chunks * s->n);
            s->pop = c.take<u32>(s->n);
        }
    };
    Carve cv;
    lay(cv);
    void* base = nullptr;
    rc = ds.reserve(cv.off + 256, &base);
    if (rc) return rc;
    Carve c2;
    c2.base = static_cast<char*>(base);
    lay(c2);
    Y.least = out;
    Y.size = Y.least + nrow_y;
    X.least = Y.size + nrow_y;
    X.size = X.least + nrow_x;
    int* err = reinterpret_cast<int*>(X.size + nrow_x);
    if (tiles) {
        if ((rc = pack_side(ds, Y, ncol, ntip, panel, err, st))) return rc;
        if ((rc = pack_side(ds, X, ncol, ntip, panel, err, st))) return rc;
        if ((rc = transfer_tiles(Y, X, ncol, ntip, err, st))) return rc;
    } else if ((rc = transfer_popcounts(ds, Y, X, ncol, ntip, panel, st))) {
        return rc;
    }
    u32 werr = 0;
    ReadBack back;
    back.add(ymin, nrow_y);
    back.add(ysize, nrow_y);
    back.add(xmin, nrow_x);
    back.add(xsize, nrow_x);
    if (tiles) back.add(&werr, 1);
    if ((rc = back.run(out, st))) return rc;
    if (werr) casphy_set_last_error_msg("transfer: a device-side wait timed out");
    return (int)werr;
}
