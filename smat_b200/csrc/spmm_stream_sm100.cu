// Block-sparse SpMM for NVIDIA B200 (sm_100a), "stream" variant: no panels, no pipeline of roles -- every warp walks the
// blocks of (a piece of) ONE block-row and feeds warp-level MMAs straight from global memory through L2 and L1.  Same
// boundary and layouts as spmm_sm100.cu (replaces mmaCBTKernel, src/cuda_hgemm/src/mma/mmaCBT.cu:13-88).
//
// What it is for.  The tcgen05 kernels pay ~470-550 cycles per step (four block-columns of a group of block-rows)
// whatever the step holds and however narrow C is, and their items are 128 columns wide.  Three kinds of work leave them
// far from their bounds: a narrow C (decoding: the matrix has to stream from HBM, hardly any arithmetic), scattered
// blocks (a step holds one or two), and small products, where set-up and hand-overs are most of the time.  Here a block
// costs its 512 bytes of A, its 16 x N slice of B and N / 8 MMAs, and nothing is needed beforehand, so that a product
// without a plan reads the boundary's arrays as they are.
//
// What bounds it (measured, one B200): A from HBM while C is narrow; then the slices of B that every block fetches through
// L2, 32 N bytes per block.  From the [N][K] array a slice is N sectors of 32 bytes, each in a line of its own, and an SM
// takes one such sector per cycle from L2 or L1 (131 cycles per slice of 128 columns); contiguous slices come at 64 bytes per
// cycle (60 cycles; 33 out of L1).  So where the blocks outnumber the block-columns enough, B is first rewritten as slabs
// [K / 16][N][16], one pass over B.  mma.sync runs at 2.1-2.6 cycles per 16x8x16 MMA and SM (34 cycles per block of 128
// columns) and is not what bounds it; a tcgen05.mma on one block would need its slice in shared memory (39 cycles for the
// operand port alone) and a barrier round trip per hand-over.  Most tiles of more than 32 columns from slabs have a kernel of
// their own below, with the loads in flight in shared memory instead of registers.
//
// Measured against the tcgen05 kernels (theirs -> these, inputs that change from pass to pass): 8192 x 28672 layer, 183 000
// blocks, N = 16: 67.7 -> 24.4 us (3.9 TB/s); power-law matrix of 2.05 million blocks, N = 128: 1706 -> 694 us, N = 8 (1.78
// million): 2076 -> 208 us; band matrix of 2284 blocks, N = 64: 10 -> 4.1 us.  Where blocks share their slices of B (a layer
// or a random matrix at N >= 128: the tall kernel takes 8-10 ns per block, 128 columns and SM, this one 55-60) the tcgen05
// kernels stay.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "ptx_sm100.cuh"
#include "smat_internal.h"
#include "spmm_stream.h"

namespace smat {
namespace {

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint4& a, const uint2& b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a.x), "r"(a.z), "r"(a.y), "r"(a.w), "r"(b.x), "r"(b.y));
}
// Values of A are read once per column tile: not kept in L1, which the slices of B need.
__device__ __forceinline__ uint4 load_a16(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 load_a8(const void* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ uint4 lds16(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ uint2 lds8(uint32_t at) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at) : "memory");
    return v;
}
constexpr int kRingWaitCode = 40;  // status word: a bounded wait of the ring kernel ran out
// late: a wait of this lane ran out, here or before; no wait is waited for after that.
__device__ __forceinline__ void ring_wait(uint32_t bar, uint32_t parity, long long limit, bool& late) {
    if (ptx::mbar_try_wait(bar, parity) || late) return;
    const long long t0 = clock64();
    while (!ptx::mbar_try_wait_suspend(bar, parity, 2000u))
        if (clock64() - t0 > limit) {
            late = true;
            return;
        }
}

// The blocks [b0, b1) of block-row `row` that a warp (or several) multiplies; count > 1: one of `count` pieces of a long block-row.
struct Piece {
    int row = 0, b0 = 0, b1 = 0, count = 1, my_slot = 0, first_slot = 0;
    bool live = false;
};
template <bool PLAN>
__device__ __forceinline__ Piece piece_of(const StreamArgs& p, int piece, int lane) {
    Piece q;
    q.live = piece < p.n_pieces;
    if (!q.live) return q;
    if (PLAN) {
        const uint4 d = __ldg(p.pieces + piece);
        q.row = (int)d.x; q.b0 = (int)d.y; q.b1 = (int)d.z;
        if (d.w) {
            const int2 s = __ldg(p.slots + (d.w - 1));
            q.my_slot = (int)d.w - 1; q.first_slot = s.x; q.count = s.y;
        }
        return q;
    }
    const int n_rows = p.brow_end - p.brow_begin;
    if (piece < n_rows) {
        const int lo = __ldg(p.rowptr + p.brow_begin), hi = __ldg(p.rowptr + p.brow_end);
        // row pointers that would lead past the arrays: an empty product and a status code
        const bool bad = lo < 0 || hi < lo || hi > p.nnzb || (p.long_rows && __ldg(p.long_rows) > p.n_pieces - n_rows);
        if (bad && piece == 0 && lane == 0) atomicCAS(p.status, 0, kStatusBadRowptr);
        q.row = piece;
        q.b0 = bad ? 0 : min(max(__ldg(p.rowptr + p.brow_begin + q.row), lo), hi);
        q.b1 = bad ? 0 : min(max(__ldg(p.rowptr + p.brow_begin + q.row + 1), q.b0), hi);
        if (q.b1 - q.b0 > p.chunk && p.long_rows) {
            q.my_slot = q.first_slot = __ldg(p.row_slot + q.row);
            q.count = (q.b1 - q.b0 + p.chunk - 1) / p.chunk;
            q.b1 = q.b0 + p.chunk;
        }
        return q;
    }
    const int listed = __ldg(p.long_rows);
    q.live = piece - n_rows < listed && listed <= p.n_pieces - n_rows;
    if (q.live) {
        const uint4 d = __ldg(p.pieces + (piece - n_rows));
        q.row = (int)d.x; q.b0 = (int)d.y; q.b1 = (int)d.z; q.my_slot = (int)d.w;
        const int2 s = __ldg(p.slots + q.my_slot);
        q.first_slot = s.x; q.count = s.y;
    }
    return q;
}

// What a warp does with its sums (of all warps of the piece): to C, or to scratch and on to C by the last piece of the row.
template <int T>
__device__ __forceinline__ void finish_piece(const StreamArgs& p, const Piece& q, float (&acc)[T][4], int tile, int n0, int octets, int lane) {
    const int g = lane >> 2, t = lane & 3;
    // ---- a piece of a long block-row: partial sums to scratch; the last piece to arrive adds them up in order ----
    if (q.count > 1) {
        float4* mine = p.partial + ((size_t)q.my_slot * p.n_tiles + tile) * (T * 32) + lane;
#pragma unroll
        for (int j = 0; j < T; j++) __stcg(mine + j * 32, make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]));
        // lane 0's arrival stands for all 32 lanes: their stores and fences come before it only through a warp barrier (a
        // shuffle does not order memory), and what it has seen reaches their loads only through another
        __threadfence();
        __syncwarp();
        int old = 0;
        if (lane == 0) old = atomicAdd(p.counters + (size_t)q.first_slot * p.n_tiles + tile, 1);
        old = __shfl_sync(0xffffffffu, old, 0);
        if (old != q.count - 1) return;
        __threadfence();
        __syncwarp();
        if (lane == 0) p.counters[(size_t)q.first_slot * p.n_tiles + tile] = 0;  // ready for the next launch
#pragma unroll
        for (int j = 0; j < T; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
        for (int i = 0; i < q.count; i++) {
            const float4* src = p.partial + ((size_t)(q.first_slot + i) * p.n_tiles + tile) * (T * 32) + lane;
#pragma unroll
            for (int j = 0; j < T; j++) {
                const float4 v = __ldcg(src + j * 32);
                acc[j][0] += v.x; acc[j][1] += v.y; acc[j][2] += v.z; acc[j][3] += v.w;
            }
        }
    }

    // ---- fp16 rows of C: neighbouring threads exchange halves of two octets, so that a quad stores 32 contiguous bytes ----
    __half* crow = p.C + (size_t)(q.row * 16 + g) * p.ldc + n0;
    if constexpr (T == 1) {
        *reinterpret_cast<__half2*>(crow + 2 * t) = __floats2half2_rn(acc[0][0], acc[0][1]);
        *reinterpret_cast<__half2*>(crow + 8 * p.ldc + 2 * t) = __floats2half2_rn(acc[0][2], acc[0][3]);
    } else {
        const bool odd = t & 1;
#pragma unroll
        for (int j = 0; j < T; j += 2) {
            if (j >= octets) break;
            const __half2 x0 = __floats2half2_rn(acc[j][0], acc[j][1]), y0 = __floats2half2_rn(acc[j][2], acc[j][3]);
            const __half2 x1 = __floats2half2_rn(acc[j + 1][0], acc[j + 1][1]), y1 = __floats2half2_rn(acc[j + 1][2], acc[j + 1][3]);
            const __half2 rx = __shfl_xor_sync(0xffffffffu, odd ? x0 : x1, 1), ry = __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 1);
            const int col = 8 * j + (odd ? 8 + 2 * (t - 1) : 2 * t);
            if (!odd || j + 1 < octets) {
                union { __half2 h[2]; uint2 u; } vx, vy;
                vx.h[0] = odd ? rx : x0; vx.h[1] = odd ? x1 : rx;
                vy.h[0] = odd ? ry : y0; vy.h[1] = odd ? y1 : ry;
                *reinterpret_cast<uint2*>(crow + col) = vx.u;
                *reinterpret_cast<uint2*>(crow + 8 * p.ldc + col) = vy.u;
            }
        }
    }
}

template <int NT, int W, int kWarps, int U, int MINB, bool SLAB, bool PLAN>
__global__ void __launch_bounds__(kWarps * 32, MINB) spmm_bcsr_stream_kernel(const StreamArgs p) {
    constexpr int T = NT / 8;                                       // MMAs (8 columns each) per block
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int tile = (int)(blockIdx.x % (unsigned)p.n_tiles);
    const int piece = (int)(blockIdx.x / (unsigned)p.n_tiles) * (kWarps / W) + warp / W;
    const int n0 = tile * p.tile_cols;
    if (PLAN && p.ahead > 0.0f && lane == 0 && tile == 0 && piece < p.n_pieces) {
        // about where this warp's blocks begin, were they dealt out evenly: on their way to L2 before the kernel before this one
        // has ended (nothing is read here, so it matters neither whether that one writes them nor whether the place is right)
        const int at = min((int)(p.ahead * (float)(piece * W + warp % W)), p.nnzb - 1), n = min(p.nnzb - at, 8);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const uint8_t*>(p.vals) + (size_t)at * 512), "r"(n * 512) : "memory");
    }
    ptx::pdl_wait();
    Piece q = piece_of<PLAN>(p, piece, lane);
    const bool live = q.live;
    const int b0 = q.b0, b1 = q.b1;
    if (W == 1 && !live) return;
    // this warp's share of the piece
    int c0 = b0, c1 = b1;
    if (W > 1) {
        const int per = (b1 - b0 + W - 1) / W, w = warp % W;
        c0 = min(b1, b0 + w * per);
        c1 = min(b1, c0 + per);
        if (!live) c0 = c1 = 0;
    }
    float acc[T][4];
#pragma unroll
    for (int j = 0; j < T; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;

    // k inside a block is permuted the same way for both operands, so that a thread's four values of a row are adjacent
    // in memory: thread t of a quad holds k = 4t .. 4t + 3
    const uint2* __restrict__ b_lane;
    size_t b_step;   // uint2 between neighbouring column octets
    if (SLAB) {
        b_lane = reinterpret_cast<const uint2*>(p.B) + (size_t)(n0 + g) * 4 + t;
        b_step = 32;
    } else {
        b_lane = reinterpret_cast<const uint2*>(p.B) + ((size_t)(n0 + g) * p.K >> 2) + t;
        b_step = (size_t)p.K * 2;
    }
    const size_t slab = SLAB ? (size_t)p.N * 4 : 4;  // uint2 between neighbouring block-columns
    const int octets = min(p.tile_cols, p.N - n0) >> 3;
    const uint8_t* a_lane = reinterpret_cast<const uint8_t*>(p.vals) + (PLAN ? lane * 16 : lane * 8);
    const int Kb = p.K >> 4;

    uint4 a[2][U];
    uint2 b[2][U][T];
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int j = 0; j < T; j++) b[s][u][j] = make_uint2(0u, 0u);
    bool ok[2][U];
    int cols = 0, cols_at = c0;  // 32 column indices at a time, one per lane
    auto load_cols = [&](int at) {
        cols_at = at;
        int c = (at + lane < c1) ? __ldg(p.colidx + at + lane) >> (PLAN ? 0 : 4) : 0;
        if (!PLAN && (c < 0 || c >= Kb)) {
            atomicCAS(p.status, 0, kStatusBadColumns);
            c = -1;
        }
        cols = c;
        // what the warp will read of A after this batch of 32 blocks is on its way to L2 meanwhile
        const int ahead = min(c1 - (at + 32), 32);
        if (lane == 0 && ahead > 0)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const uint8_t*>(p.vals) + (size_t)(at + 32) * 512), "r"(ahead * 512) : "memory");
    };
    load_cols(c0);
    auto fetch = [&](auto S, int at) {
        constexpr int s = decltype(S)::value;
        if (at - cols_at >= 32) load_cols(at);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int cb = __shfl_sync(0xffffffffu, cols, (at + u - cols_at) & 31);
            ok[s][u] = at + u < c1 && cb >= 0;
            if (ok[s][u]) {
                const uint8_t* ap = a_lane + (size_t)(at + u) * 512;
                if (PLAN) {
                    a[s][u] = load_a16(ap);
                } else {
                    const uint2 lo = load_a8(ap), hi = load_a8(ap + 256);
                    a[s][u] = make_uint4(lo.x, lo.y, hi.x, hi.y);
                }
                const uint2* bp = b_lane + (size_t)cb * slab;
#pragma unroll
                for (int j = 0; j < T; j++)
                    if (j < octets) b[s][u][j] = __ldg(bp + j * b_step);
            }
        }
    };
    auto multiply = [&](auto S) {
        constexpr int s = decltype(S)::value;
#pragma unroll
        for (int u = 0; u < U; u++)
            if (ok[s][u]) {
#pragma unroll
                for (int j = 0; j < T; j++) mma_16816(acc[j], a[s][u], b[s][u][j]);
            }
    };
    using I0 = std::integral_constant<int, 0>;
    using I1 = std::integral_constant<int, 1>;
    fetch(I0{}, c0);
    for (int at = c0; at < c1; at += 2 * U) {
        fetch(I1{}, at + U);
        multiply(I0{});
        fetch(I0{}, at + 2 * U);
        multiply(I1{});
    }

    // ---- sum over the W warps of the piece (fixed order) ----
    if constexpr (W > 1) {
        __shared__ float4 red[kWarps / 2][T][32];
        const int w = warp % W, base = (warp / W) * (W / 2);
#pragma unroll
        for (int half = W / 2; half >= 1; half >>= 1) {
            if (w >= half && w < 2 * half) {
#pragma unroll
                for (int j = 0; j < T; j++) red[base + w - half][j][lane] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
            }
            __syncthreads();
            if (w < half) {
#pragma unroll
                for (int j = 0; j < T; j++) {
                    const float4 v = red[base + w][j][lane];
                    acc[j][0] += v.x; acc[j][1] += v.y; acc[j][2] += v.z; acc[j][3] += v.w;
                }
            }
            if (half > 1) __syncthreads();
        }
        if (w != 0 || !live) return;
    }

    finish_piece<T>(p, q, acc, tile, n0, octets, lane);
}

// The same product for wide tiles whose B is slabs: a warp's next S slices and blocks are on their way to a ring in shared memory
// (a bulk copy each) while it multiplies, so that the loads in flight are not bounded by registers: at 128 columns 12 warps of the
// kernel above (166 registers) would have one block of 4.6 KB each on its way.  Power-law matrix of 262144 rows, 128 columns: 826 -> 630 us (58 of
// the 67-72 bytes per cycle and SM that L2 serves to a pure streaming kernel), 96 columns 731 -> 480, 64 columns 515 -> 403;
// 65536 rows without a plan, 128 columns: 266 -> 212.  32 columns stay with the kernel above (179 us against 234): a
// block then costs its two copies, 28 cycles each, more than its bytes.  The blocks of A come as copies too, although a lane
// could load its 16 bytes itself: a wait for one such load waits for all later ones of the warp as well (1100 cycles a block).
template <int NT, int S, int W, int kWarps, int MINB, bool PLAN>
__global__ void __launch_bounds__(kWarps * 32, MINB) spmm_bcsr_ring_kernel(const StreamArgs p) {
    constexpr int T = NT / 8;
    constexpr uint32_t STAGE = NT * 32 + 512;  // bytes: a slice of NT columns, then the block
    extern __shared__ __align__(128) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = (int)(blockIdx.x % (unsigned)p.n_tiles);
    const int piece = (int)(blockIdx.x / (unsigned)p.n_tiles) * (kWarps / W) + warp / W;
    const int n0 = tile * p.tile_cols;
    const uint32_t ring = ptx::smem_u32(smem) + warp * (S * STAGE), bars = ptx::smem_u32(smem) + kWarps * (S * STAGE) + warp * (S * 8);
    if (lane == 0) {
#pragma unroll
        for (int s = 0; s < S; s++) ptx::mbar_init(bars + 8 * s, 1);
        ptx::fence_barrier_init();
    }
    __syncwarp();
    ptx::pdl_wait();
    const Piece q = piece_of<PLAN>(p, piece, lane);
    if (W == 1 && !q.live) return;
    int c0 = q.b0, c1 = q.b1;  // this warp's share of the piece
    if (W > 1) {
        const int per = (q.b1 - q.b0 + W - 1) / W, w = warp % W;
        c0 = min(q.b1, q.b0 + w * per);
        c1 = min(q.b1, c0 + per);
        if (!q.live) c0 = c1 = 0;
    }
    float acc[T][4];
#pragma unroll
    for (int j = 0; j < T; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    const int octets = min(p.tile_cols, p.N - n0) >> 3, Kb = p.K >> 4;
    const uint32_t bytes = (uint32_t)octets * 256u, awaited = bytes + 512u + p.lost_bytes;
    const uint8_t* vals = static_cast<const uint8_t*>(p.vals);
    const uint8_t* slabs = static_cast<const uint8_t*>(p.B) + (size_t)n0 * 32;
    const size_t slab = (size_t)p.N * 32;
    const uint32_t a_lane = ring + NT * 32 + (PLAN ? lane * 16 : lane * 8), b_lane = ring + lane * 8;
    const uint64_t once = ptx::policy_evict_first();  // a block is read once per column tile: it is not to push slabs out of L2
    // 32 block-columns at a time, one per lane, and the 32 that follow
    auto load_cols = [&](int at) {
        int c = (at + lane < c1) ? __ldg(p.colidx + at + lane) >> (PLAN ? 0 : 4) : 0;
        if (!PLAN && (c < 0 || c >= Kb)) {
            atomicCAS(p.status, 0, kStatusBadColumns);
            c = -1;
        }
        return c;
    };
    int cols_at = c0, cols = load_cols(c0), cols_next = load_cols(c0 + 32);
    uint32_t ok = 0, phase = 0;  // bit s: stage s holds a block; parity of its next wait
    // At the limit of a wait one lane may give up where the next still sees the copy arrive.  Giving up changes no branch that all
    // lanes take part in: the lane goes on with what the stage holds, and lane 0 starts no more copies, so that the others' next
    // waits run out too.  (A vote after every wait instead: 2 to 3 % at 64 columns.)
    bool late = false;
    auto fetch = [&](int s, int at) {
        if (at - cols_at >= 32) {
            cols_at += 32;
            cols = cols_next;
            cols_next = load_cols(cols_at + 32);
        }
        const int cb = __shfl_sync(0xffffffffu, cols, at - cols_at);
        ok &= ~(1u << s);
        if (at < c1 && cb >= 0) {
            ok |= 1u << s;
            if (lane == 0 && !late) {
                ptx::mbar_arrive_expect_tx(bars + 8 * s, awaited);
                ptx::bulk_load(ring + s * STAGE, slabs + (size_t)cb * slab, bytes, bars + 8 * s);
                ptx::bulk_load_hint(ring + s * STAGE + NT * 32, vals + (size_t)at * 512, 512u, bars + 8 * s, once);
            }
        }
    };
#pragma unroll
    for (int s = 0; s < S; s++) fetch(s, c0 + s);
    for (int at = c0; at < c1; at += S) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            if (ok & (1u << s)) {
                ring_wait(bars + 8 * s, (phase >> s) & 1u, p.wait_cycles, late);
                __syncwarp();  // for the MMAs
                phase ^= 1u << s;
                // all of the stage: what a narrower tile leaves of it goes to columns that are not stored
                uint4 a;
                uint2 b[T];
                if (PLAN) {
                    a = lds16(a_lane + s * STAGE);
                } else {
                    const uint2 lo = lds8(a_lane + s * STAGE), hi = lds8(a_lane + s * STAGE + 256);
                    a = make_uint4(lo.x, lo.y, hi.x, hi.y);
                }
#pragma unroll
                for (int j = 0; j < T; j++) b[j] = lds8(b_lane + s * STAGE + j * 256);
#pragma unroll
                for (int j = 0; j < T; j++) mma_16816(acc[j], a, b[j]);
            }
            __syncwarp();  // all lanes have read the stage before it is filled again
            fetch(s, at + S + s);
        }
    }
    if (late) {  // a copy did not arrive in time: the host sees a status, copies in flight get time to land
        atomicCAS(p.status, 0, kRingWaitCode);
        for (int i = 0; i < 64; i++) __nanosleep(1000);
    }
    __syncwarp();
    if constexpr (W > 1) {  // sum over the W warps of the piece (fixed order), in the rings
        const int w = warp % W;
#pragma unroll
        for (int half = W / 2; half >= 1; half >>= 1) {
            float4* red = reinterpret_cast<float4*>(smem + (warp - w + (w < half ? w : w - half)) * (S * STAGE)) + lane;
            static_assert(T * 32 * 16 <= S * STAGE, "a warp's sums fit its ring");
            __syncthreads();
            if (w >= half && w < 2 * half) {
#pragma unroll
                for (int j = 0; j < T; j++) red[j * 32] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
            }
            __syncthreads();
            if (w < half) {
#pragma unroll
                for (int j = 0; j < T; j++) {
                    const float4 v = red[j * 32];
                    acc[j][0] += v.x; acc[j][1] += v.y; acc[j][2] += v.z; acc[j][3] += v.w;
                }
            }
        }
        if (w != 0 || !q.live) return;
    }
    // (also after a wait that ran out: a piece of a long block-row that did not arrive would leave the row's counter, which the last
    // one resets, part-way up for the plan's next product)
    finish_piece<T>(p, q, acc, tile, n0, octets, lane);
}

// B ([N][K], k contiguous) -> slabs [K / 16][N][16]: the 16 x N slice of one block-column becomes contiguous.
__global__ void __launch_bounds__(256) slab_kernel(const uint4* __restrict__ B, uint4* __restrict__ out, int N, int K8) {
    ptx::pdl_wait();
    // a warp moves 16 rows x 32 bytes; the eight warps of a CTA take neighbouring block-columns
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * 8 + warp;  // block-column
    if (2 * c >= K8) return;
    for (int n = blockIdx.y * 16 + (lane >> 1); n < N; n += gridDim.y * 16)
        out[((size_t)c * N + n) * 2 + (lane & 1)] = __ldg(B + (size_t)n * K8 + 2 * c + (lane & 1));
}

// Product without a plan: the block-rows of more than `chunk` blocks, cut into pieces.  The first piece stays with the
// row's own warps; the others are listed here, in whatever order the rows arrive (the sums of a row are added up by
// piece number, so the order does not show in the result).  head[0], head[1]: pieces listed, slots taken (zero before).
__global__ void __launch_bounds__(256) long_rows_kernel(const int* __restrict__ rowptr, int brow_begin, int brow_end, int nnzb, int chunk,
                                                       int room, int* head, uint4* __restrict__ pieces, int2* __restrict__ slots,
                                                       int* __restrict__ row_slot) {
    ptx::pdl_wait();
    const int lo = __ldg(rowptr + brow_begin), hi = __ldg(rowptr + brow_end);
    const int row = blockIdx.x * 256 + threadIdx.x;
    if (lo < 0 || hi < lo || hi > nnzb || row >= brow_end - brow_begin) return;
    const int b0 = min(max(__ldg(rowptr + brow_begin + row), lo), hi), b1 = min(max(__ldg(rowptr + brow_begin + row + 1), b0), hi);
    if (b1 - b0 <= chunk) return;
    const int k = (b1 - b0 + chunk - 1) / chunk;
    const int at = atomicAdd(head, k - 1), slot = atomicAdd(head + 1, k);
    if (at + k - 1 > room) return;  // row pointers that overlap: the kernel sees more pieces than there can be and refuses
    row_slot[row] = slot;
    slots[slot] = make_int2(slot, k);
    for (int i = 1; i < k; i++) {
        pieces[at + i - 1] = make_uint4((uint32_t)row, (uint32_t)(b0 + i * chunk), (uint32_t)min(b1, b0 + (i + 1) * chunk), (uint32_t)(slot + i));
        slots[slot + i] = make_int2(slot, k);
    }
}

// Product without a plan of a matrix of several windows of block-columns: what the plan kernels refuse there is refused here as
// well.  (In the kernel that multiplies, the look costs the eight-column shapes registers they do not have: 43 -> 62 us.)
__global__ void __launch_bounds__(256) column_order_kernel(const int* __restrict__ rowptr, const int* __restrict__ colidx, int brow_begin,
                                                          int brow_end, int nnzb, int* status) {
    ptx::pdl_wait();
    constexpr int W = kOrderWindow * 16;  // columns of a window
    const int lo = __ldg(rowptr + brow_begin), hi = __ldg(rowptr + brow_end), lane = threadIdx.x & 31;
    if (lo < 0 || hi < lo || hi > nnzb) return;
    const int warps = (int)((gridDim.x * blockDim.x) >> 5);
    for (int row = brow_begin + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); row < brow_end; row += warps) {
        const int b0 = min(max(__ldg(rowptr + row), lo), hi), b1 = min(max(__ldg(rowptr + row + 1), b0), hi);
        bool bad = false;
        for (int j = b0 + 1 + lane; j < b1; j += 32) bad |= __ldg(colidx + j) / W < __ldg(colidx + j - 1) / W;
        if (bad) atomicCAS(status, 0, kStatusBadColumns);
    }
}

// The plan's copy of the values in the order a warp's lanes read them (lane (g, t): rows g and g + 8, k = 4t .. 4t + 3), and
// of the block columns; a column outside the matrix becomes -1.  Where the plan holds the blocks in the walk order of a
// tcgen05 kernel as well, block i also goes to place pos[i] of that copy, in its swizzled form (16-byte chunk index XOR bit 2
// of the row): read once for both (183 000 blocks: 47 us, 64 with a kernel for each, 33 for one copy alone; 52 with a block at a
// time instead of four).
__global__ void __launch_bounds__(256) stream_pack_kernel(const uint2* __restrict__ vals, const int* __restrict__ colidx,
                                                         uint4* __restrict__ packed, int* __restrict__ cols, int first, int n, int Kb,
                                                         const int* __restrict__ pos, uint2* __restrict__ walk) {
    ptx::pdl_wait();
    const int lane = threadIdx.x & 31;
    const int row = lane >> 2, chunk = 2 * row + ((lane >> 1) & 1), to = 2 * (chunk ^ ((row >> 2) & 1)) + (lane & 1);
    constexpr int U = 4;  // blocks of a warp at a time, all loads before the stores
    const int stride = (int)((gridDim.x * blockDim.x) >> 5) * U;
    for (int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * U; i < n; i += stride) {
        uint2 lo[U], hi[U];
        int p[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u < n) {
                lo[u] = __ldg(vals + (size_t)(first + i + u) * 64 + lane);
                hi[u] = __ldg(vals + (size_t)(first + i + u) * 64 + 32 + lane);
                p[u] = pos ? __ldg(pos + i + u) : -1;
            }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u < n) {
                packed[(size_t)(i + u) * 32 + lane] = make_uint4(lo[u].x, lo[u].y, hi[u].x, hi[u].y);
                if (p[u] >= 0) {
                    walk[(size_t)p[u] * 64 + to] = lo[u];
                    walk[(size_t)p[u] * 64 + 32 + to] = hi[u];
                }
                if (cols && lane == 0) {
                    const int c = __ldg(colidx + first + i + u) >> 4;
                    cols[i + u] = (c >= 0 && c < Kb) ? c : -1;
                }
            }
    }
}

// pos[j] = place of block j in the walk order `blk` (both counted from the range's first block; -1 where it has none).
__global__ void __launch_bounds__(256) walk_place_kernel(const int* __restrict__ blk, int* __restrict__ pos, int first, int n) {
    ptx::pdl_wait();
    for (int p = blockIdx.x * 256 + threadIdx.x; p < n; p += gridDim.x * 256) {
        const int j = __ldg(blk + first + p) - first;
        if (j >= 0 && j < n) pos[j] = p;
    }
}

// warps of a CTA, blocks per load batch (two batches in flight) and CTAs per SM of the kernel for NT columns, W warps per piece
template <int NT, int W>
struct Tune {
    static constexpr int WARPS = W == 8 ? 8 : 4;
    static constexpr int U = NT == 8 ? 4 : NT <= 32 ? 2 : 1;
    static constexpr int MINB = W == 8 ? (NT <= 16 ? 4 : NT <= 64 ? 2 : 1) : (NT <= 16 ? 8 : NT == 32 ? 5 : NT == 64 ? 4 : 3);
};

template <int NT, int W, bool SLAB, bool PLAN>
cudaError_t launch_one(const StreamArgs& a, cudaStream_t stream) {
    using Q = Tune<NT, W>;
    constexpr long long per = Q::WARPS / W;
    const long long grid = (((long long)a.n_pieces + per - 1) / per) * a.n_tiles;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    return launch_pdl(spmm_bcsr_stream_kernel<NT, W, Q::WARPS, Q::U, Q::MINB, SLAB, PLAN>, dim3((unsigned)grid), dim3(Q::WARPS * 32), 0, stream, a);
}

// slabs of more bytes than this are taken not to stay in L2 beside A (126 MB, each half of the SMs by its own half)
constexpr size_t kSlabBytesL2 = (size_t)62 << 20;

// FEWER: CTAs per SM where `fewer` asks for them instead of MINB (0: never).  The limit that is set on the kernel is the most that
// either launch of it wants: it belongs to the kernel, and another thread's launch may come between setting it and launching.
template <int NT, int S, int W, int kWarps, int MINB, bool PLAN, int FEWER = 0>
cudaError_t launch_ring(const StreamArgs& a, cudaStream_t stream, bool fewer = false) {
    const long long grid = (((long long)a.n_pieces + kWarps / W - 1) / (kWarps / W)) * a.n_tiles;
    if (grid > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    constexpr int own = kWarps * S * (NT * 32 + 512 + 8), large = FEWER && FEWER < MINB ? 228 * 1024 / (FEWER + 1) : 0;  // large: one CTA more would not fit
    constexpr int most = own > large ? own : large;
    static_assert((own + 1024) * MINB <= 228 * 1024, "shared memory of the resident CTAs");
    auto kernel = spmm_bcsr_ring_kernel<NT, S, W, kWarps, MINB, PLAN>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
    return launch_pdl(kernel, dim3((unsigned)grid), dim3(kWarps * 32), fewer ? most : own, stream, a);
}

// Whether 33 to 64 columns from slabs stay with the loads in registers: slabs of a few megabytes come fast enough, and a block's two
// copies cost more than its bytes.  us, registers and ring, 64 columns, without a plan: random matrices of 16384 rows 26 and 28, 38
// and 41, of 32768 rows 40 and 42, 103 and 109; power-law 32768 rows 83 and 82; block-rows of very different length 48 and 56, 120 and
// 118; of 65536 rows random 125 and 132, power-law 153 and 144, 131 and 129; 131072 rows 131 and 116, 270 and 229.  With a plan the
// ring is the better from 65 000 blocks on (32768 rows: 68 and 65, 126 and 103) and below 32 000 (11.7 and 11.6), not between (19.8
// and 21.4, 16.2 and 17.8, unequal block-rows 36 and 43).
bool ring_not_for_64(const StreamArgs& a, bool plan) {
    return (size_t)a.N * a.K * 2 <= (size_t)9 << 19 && (!plan || (a.nnzb >= 32768 && a.nnzb < 65536));
}

// Whether 97 to 128 columns take 12 warps an SM instead of 14 (launch_nt): where slabs of more than half of L2 leave it less room for
// A, and, with a plan, where 14 warps would have more than some 170 KB of slices an SM on their way, from 113 columns on.  There they
// fall off, but for products that are one round of 14 warps and for short block-rows.  us, 14 and 12 warps, 128 columns: random
// matrices of 65536 rows with 120 blocks a block-row 224 and 172, 20 blocks 41 and 44, of 131072 rows with 60 blocks 183 and 176, of
// 16384 rows (one round) 29 and 35; power-law in given order, 98304 rows 285 and 274, 160000 rows 383 and 412; sorted by degree, 65536
// rows 206 and 158, 160000 rows 432 and 356.  112 columns: 150 and 171, 264 and 271, 377 and 408, 333 and 346.  Without a plan 14 are
// the better more often: 184 and 194, 430 and 469, 199 and 186.
bool ring_fewer_warps(const StreamArgs& a, int w, bool plan) {
    if ((size_t)a.N * a.K * 2 > kSlabBytesL2) return true;
    const long long warps = (long long)a.n_pieces * a.n_tiles * w;
    if (!plan || a.tile_cols <= 112 || (warps > 12LL * a.sm_count && warps <= 14LL * a.sm_count)) return false;
    return a.nnzb >= 40LL * a.n_pieces;
}

template <bool PLAN, bool SLAB, int W>
cudaError_t launch_nt(int nt, const StreamArgs& a, cudaStream_t stream) {
    if constexpr (SLAB && W < 8) {
        constexpr int kWarps = W == 4 ? 4 : 2;
        // Slices of N columns in flight per SM: 14 warps x 3 (or 12 x 3) of 97 to 128 columns, 16 x 3 of 65 to 96, 20 x 2 of 33 to
        // 64.  Beyond that the kernel falls off: 18 x 3 of 96 columns take 795 us instead of 480 (power-law matrix of 262144 rows), 16
        // x 4 of 64 columns 575 (12 x 4) to 1000.
        if (nt == 128 && a.tile_cols > 96) return launch_ring<128, 3, W, kWarps, 14 / kWarps, PLAN, 12 / kWarps>(a, stream, ring_fewer_warps(a, W, PLAN));
        if (nt == 128) return launch_ring<96, 3, W, kWarps, 16 / kWarps, PLAN>(a, stream);
        if (nt == 64 && ring_not_for_64(a, PLAN)) return launch_one<64, W, SLAB, PLAN>(a, stream);
        if (nt == 64) return launch_ring<64, 2, W, kWarps, 20 / kWarps, PLAN>(a, stream);
    }
    if constexpr (!SLAB && W < 8) {
        if (nt == 128) return launch_one<128, W, SLAB, PLAN>(a, stream);
    }
    if constexpr (!SLAB || W == 8) {
        if (nt == 64) return launch_one<64, W, SLAB, PLAN>(a, stream);
    }
    if (nt == 32) return launch_one<32, W, SLAB, PLAN>(a, stream);
    if constexpr (!SLAB) {
        if (nt == 16) return launch_one<16, W, SLAB, PLAN>(a, stream);
        if (nt == 8) return launch_one<8, W, SLAB, PLAN>(a, stream);
    }
    return cudaErrorInvalidValue;
}

template <bool PLAN, bool SLAB>
cudaError_t launch_w(const StreamShape& s, const StreamArgs& a, cudaStream_t stream) {
    if (s.w == 8 && s.nt < 128) return launch_nt<PLAN, SLAB, 8>(s.nt, a, stream);
    if (s.w >= 4) return launch_nt<PLAN, SLAB, 4>(s.nt, a, stream);
    if (s.w == 2) return launch_nt<PLAN, SLAB, 2>(s.nt, a, stream);
    return launch_nt<PLAN, SLAB, 1>(s.nt, a, stream);
}

template <bool PLAN>
int launch(const StreamShape& s, const StreamArgs& a, cudaStream_t stream) {
    const cudaError_t e = s.slab ? launch_w<PLAN, true>(s, a, stream) : launch_w<PLAN, false>(s, a, stream);
    if (e != cudaSuccess) return fail(SMAT_ERR_CUDA, "launch of the stream kernel failed: %s", cudaGetErrorString(e));
    count_launch();
    return SMAT_OK;
}

int make_slabs(const void* B, void* slabs, size_t N, size_t K, cudaStream_t stream) {
    SMAT_CUDA_TRY(launch_pdl(slab_kernel, dim3((unsigned)((K / 16 + 7) / 8), (unsigned)std::min<size_t>((N + 15) / 16, 65535)), dim3(256), 0, stream,
                             reinterpret_cast<const uint4*>(B), reinterpret_cast<uint4*>(slabs), (int)N, (int)(K / 8)));
    count_launch();
    return SMAT_OK;
}

// Plans of fewer bytes of blocks than this do without the prefetch at the kernel's start.  Without and with it, one plan and four in
// turn, us: 0.8 MB of blocks, N = 16: 3.7 and 3.7, 3.7 and 3.6; 8.4 MB, N = 32: 6.02 and 6.02, 6.25 and 6.07; 13 MB, N = 32: 9.0 and
// 8.9, 10.2 and 9.2; 27 MB: 12.8 and 11.7, 15.6 and 14.4; 94 MB, N = 16: 22.6 and 22.3, 24.4 and 23.7.
constexpr size_t kAheadBytes = (size_t)4 << 20;

// Columns of a tile: N spread evenly over the tiles, in octets.
int tile_cols(size_t N, int tiles) { return (int)((N / 8 + (size_t)tiles - 1) / (size_t)tiles) * 8; }

size_t round256(size_t x) { return (x + 255) / 256 * 256; }

}  // namespace

// Columns per warp, warps per piece, blocks per piece, and whether B is rewritten as slabs.
StreamShape stream_shape(size_t N, size_t rows, size_t nnzb, size_t K, int sm_count, bool plan) {
    StreamShape s;
    const size_t sms = (size_t)sm_count, avg = rows ? nnzb / rows : 0;
    // One tile across C as long as it holds in registers: A is then read once.
    s.nt = N <= 8 ? 8 : N <= 16 ? 16 : N <= 32 ? 32 : N <= 64 ? 64 : 128;
    // Slabs: a slice then costs 0.27 ns less per column and SM; the pass costs its launch and B twice at 5.5 TB/s.
    const double gain = (double)nnzb * (double)N * 0.27e-3 / (double)sms, cost = 2.0 + 4e-6 * (double)N * (double)K / 5.5;
    s.slab = s.nt >= 32 && gain > cost;
    // Enough warps to keep the SMs' load queues full (12 of 128 columns, 16 of 64, 32 of fewer): first several warps per
    // block-row, each with at least four blocks, then narrower tiles.
    auto tiles = [&] { return (N + (size_t)s.nt - 1) / (size_t)s.nt; };
    auto wanted = [&] { return sms * (s.nt == 128 ? 12 : s.nt == 64 ? 16 : 32); };
    while (s.w < (s.nt == 128 ? 4 : 8) && rows * tiles() * (size_t)s.w < wanted() && avg >= 8 * (size_t)s.w) s.w *= 2;
    while (s.nt > (s.slab ? 32 : 16) && rows * tiles() * (size_t)s.w * 2 < wanted()) s.nt /= 2;
    // A piece: a few rounds of work per resident warp, so that long block-rows neither trail nor pay much for their
    // partial tiles.  Measured on power-law matrices of 0.2 to 2.2 million blocks: 96 to 192, flat in between.
    const size_t per_warp = nnzb / (sms * 12) / 2;
    const size_t warp_chunk = std::min<size_t>(std::max<size_t>(per_warp, 96), 192);
    // Without a plan long block-rows have to be listed first (two more operations on the stream, ~4 us): small matrices go
    // without, with enough warps per block-row that even a full one is no longer than their pieces.
    if (!plan && nnzb < 32 * 1024)
        while (s.w < (s.nt == 128 ? 4 : 8) && K / 16 > warp_chunk * (size_t)s.w && K / 16 <= warp_chunk * 8) s.w *= 2;
    s.chunk = (int)(warp_chunk * (size_t)s.w);
    return s;
}

// Microseconds a product takes with this kernel (one B200), within some 20 %: a launch, the slabs, and per block and SM the
// streaming of A (10 ns) and the fetch of the slice of B.  From slabs, fitted to 150 random, power-law, layer, band and clustered
// matrices of 6 000 to 3.8 million blocks, with 40 to 256 columns: 0.46 ns a column, and no less than 40 ns beyond 32 columns;
// without a plan 0.33 ns a column and 12 ns for every tile, no less than 34 ns.
double stream_estimate_us(size_t N, size_t rows, size_t nnzb, size_t K, int sm_count, bool plan) {
    const StreamShape s = stream_shape(N, rows, nnzb, K, sm_count, plan);
    const double n = (double)N, tiles = std::ceil(n / s.nt);
    double per_block = s.slab ? std::max(N <= 32 ? 22.0 : plan ? 40.0 : 34.0, plan ? 0.46 * n : 12.0 * tiles + 0.33 * n) : 10.0 + 0.6 * n;
    const double warps = (double)rows * tiles * s.w, full = (double)sm_count * (s.nt == 128 ? 12 : s.nt == 64 ? 16 : 32);
    if (s.slab && warps < full) per_block *= full / warps;  // block-rows too few and too short to fill the SMs' load queues
    return 4.0 + (s.slab ? 2.0 + 4e-6 * n * (double)K / 5.5 : 0.0) + (double)nnzb / sm_count * per_block * 1e-3 + (double)(rows * 16) * n * 2.0 / 6e6;
}

double stream_passes_us(size_t N, size_t N_hint, size_t rows, size_t nnzb, size_t K, int sm_count) {
    const size_t cap = stream_pass_columns(N_hint), rest = N % cap;
    return (double)(N / cap) * stream_estimate_us(cap, rows, nnzb, K, sm_count, true) +
           (rest ? stream_estimate_us(rest, rows, nnzb, K, sm_count, true) : 0.0);
}

// A product without a plan takes this kernel unless building a plan inside the call and a tcgen05 kernel are estimated to be
// faster: 12 us for the launches and small plan kernels, 0.02 ns per block for the walk order, and the product -- rounds of
// items at 0.26 us a step, or 20 ns per block, tile and SM, whichever is more.
bool stream_for_call(size_t N, size_t rows, size_t nnzb, size_t K, int sm_count) {
    if (g_spmm_variant) return g_spmm_variant == 5;
    const size_t rg = choose_rows_per_group(rows, N, sm_count, true, nnzb, K), groups = (rows + rg - 1) / rg, tiles = (N + 127) / 128;
    const double throughput = (double)nnzb * (double)tiles / sm_count * 20e-3, build = 12.0 + 0.02e-3 * (double)nnzb;
    const double stream = stream_estimate_us(N, rows, nnzb, K, sm_count, false);
    if ((double)nnzb < 0.12 * (double)rows * (double)(K / 16)) {
        // Few of the possible blocks: how they lie is not known here, and no rule on these four sizes suits all.  Clustered
        // blocks and bands suit the other kernel, whose steps they fill, scattered ones this one, and skewed ones more, since
        // it cuts long block-rows.  What sizes tell is the number of blocks of a block-row: bands and clusters have some tens,
        // random matrices and graphs of this fill a hundred and more.  So up to 48 the other kernel is taken at the estimate of
        // its throughput (and this one for what is close), beyond that at three times it.  What that gets wrong are bands of more
        // than 48 blocks a block-row (half bandwidth beyond some 380; none among the products below): this kernel is taken for
        // them and takes up to twice the other's time.
        // Both kernels timed on 216 products (40 to 400 columns), time of the chosen one to the faster one, geometric mean and
        // worst, with this rule and before it (which drew the line at 24 and twice the throughput, with estimates from
        // before slices came through a ring and blocks were gathered): random 1.00, 1.06 and 1.03, 1.82; power-law 1.00, 1.00
        // and 1.45, 3.43; layers 1.01, 1.09 and 1.02, 1.18; bands 1.02, 1.21 and 1.13, 2.41; clusters 1.01, 1.14 and 1.03, 1.20.
        return stream < (nnzb > 48 * rows ? 3.0 : 1.15) * (build + throughput);
    }
    const double quads = std::ceil((double)K / 64.0), steps = quads * (1.0 - std::exp(-(double)nnzb / (double)groups / quads));
    return stream < build + std::max(throughput, rounds_for(groups * tiles, (size_t)sm_count, true, (size_t)steps, false) * steps * 0.26);
}

StreamLayout stream_plan_layout(const int* h_rowptr, size_t rows, size_t K, size_t N_hint, int sm_count, bool beside) {
    StreamLayout l;
    const int first = h_rowptr[0];
    const size_t n = (size_t)(h_rowptr[rows] - first);
    const StreamShape s = stream_shape(N_hint, rows, n, K, sm_count, true);
    l.pieces.reserve(rows + n / (size_t)s.chunk + 1);
    l.row_piece.resize(rows + 1);
    for (size_t r = 0; r < rows; r++) {
        const unsigned b0 = (unsigned)(h_rowptr[r] - first), len = (unsigned)(h_rowptr[r + 1] - h_rowptr[r]);
        const unsigned k = len ? (len + (unsigned)s.chunk - 1) / (unsigned)s.chunk : 1, per = (len + k - 1) / k;
        l.row_piece[r] = (int)l.pieces.size();
        const int slot0 = (int)l.slots.size();
        for (unsigned i = 0; i < k; i++) {
            if (k > 1) l.slots.push_back(make_int2(slot0, (int)k));
            l.pieces.push_back(make_uint4((unsigned)r, b0 + std::min(len, i * per), b0 + std::min(len, (i + 1) * per), k > 1 ? (unsigned)l.slots.size() : 0u));
        }
    }
    l.row_piece[rows] = (int)l.pieces.size();
    l.first = (size_t)first;
    l.n_cap = stream_pass_columns(N_hint);
    l.pieces_bytes = round256(l.pieces.size() * sizeof(uint4));
    l.slots_bytes = round256(l.slots.size() * sizeof(int2));
    l.counter_bytes = round256(l.slots.size() * (l.n_cap / 8) * sizeof(int));
    l.partial_bytes = round256(l.slots.size() * l.n_cap * 64);
    l.cols_bytes = round256(n * sizeof(int));
    l.pos_bytes = beside ? l.cols_bytes : 0;
    l.packed_bytes = n * 512;
    // slabs for the widest pass, whatever the hint: where a narrower one wants them the widest does too
    l.slab_bytes = stream_shape(l.n_cap, rows, n, K, sm_count, true).slab ? round256(l.n_cap * K * 2) : 0;
    return l;
}

int stream_plan_fill(StreamPlan& sp, PlanView& v, StreamLayout& l, void* memory, const void* vals, const int* colidx, int sm_count,
                     const PlanView* walk, cudaStream_t stream) {
    char* b = static_cast<char*>(memory);
    StreamArgs& a = sp.args;
    a = StreamArgs{};
    a.pieces = reinterpret_cast<uint4*>(b); b += l.pieces_bytes;
    a.slots = reinterpret_cast<int2*>(b); b += l.slots_bytes;
    a.counters = reinterpret_cast<int*>(b); b += l.counter_bytes;
    a.partial = reinterpret_cast<float4*>(b); b += l.partial_bytes;
    a.colidx = reinterpret_cast<int*>(b); b += l.cols_bytes;
    if (walk) sp.pos = reinterpret_cast<int*>(b);
    b += l.pos_bytes;
    a.vals = b; b += l.packed_bytes;
    sp.slabs = l.slab_bytes ? b : nullptr;
    sp.first = l.first;
    sp.n_cap = l.n_cap;
    sp.row_piece = std::move(l.row_piece);
    SMAT_CUDA_TRY(cudaMemcpyAsync(const_cast<uint4*>(a.pieces), l.pieces.data(), l.pieces.size() * sizeof(uint4), cudaMemcpyHostToDevice, stream));
    if (!l.slots.empty()) {
        SMAT_CUDA_TRY(cudaMemcpyAsync(const_cast<int2*>(a.slots), l.slots.data(), l.slots.size() * sizeof(int2), cudaMemcpyHostToDevice, stream));
        SMAT_CUDA_TRY(cudaMemsetAsync(a.counters, 0, l.counter_bytes, stream));
    }
    if (walk) {
        sp.walk = const_cast<void*>(walk->packed);
        SMAT_CUDA_TRY(cudaMemsetAsync(sp.pos, 0xff, l.pos_bytes, stream));
        SMAT_CUDA_TRY(launch_pdl(walk_place_kernel, dim3((unsigned)std::min((v.nnzb + 255) / 256, (size_t)sm_count * 8)), dim3(256), 0, stream,
                                 walk->blk, sp.pos, (int)sp.first, (int)v.nnzb));
        count_launch();
    }
    v.stream = &sp;
    v.n_groups = v.brow_end - v.brow_begin;
    v.rg = 1;
    v.total_steps = l.pieces.size();
    return stream_plan_values(v, vals, colidx, sm_count, stream);  // pageable sources: the copies above have left them
}

int stream_plan_values(const PlanView& v, const void* vals, const int* colidx, int sm_count, cudaStream_t stream) {
    if (v.nnzb == 0) return SMAT_OK;
    const StreamArgs& a = v.stream->args;
    const unsigned grid = (unsigned)std::min((v.nnzb + 7) / 8, (size_t)sm_count * 8);
    SMAT_CUDA_TRY(launch_pdl(stream_pack_kernel, dim3(grid), dim3(256), 0, stream,
                             reinterpret_cast<const uint2*>(vals), colidx, reinterpret_cast<uint4*>(const_cast<void*>(a.vals)),
                             colidx ? const_cast<int*>(a.colidx) : nullptr, (int)v.stream->first, (int)v.nnzb, (int)(v.K / 16), v.stream->pos,
                             static_cast<uint2*>(v.stream->walk)));
    count_launch();
    SMAT_CUDA_TRY(cudaGetLastError());
    return SMAT_OK;
}

int launch_stream(const PlanView& v, const void* B, void* C, size_t N, cudaStream_t stream, const DeviceCtx* ctx, size_t ldc,
                  size_t row_begin, size_t row_end) {
    const StreamPlan& sp = *v.stream;
    const size_t rows = v.brow_end - v.brow_begin;
    if (row_end > rows) row_end = rows;
    if (row_begin >= row_end) return SMAT_OK;
    // scratch and slabs were sized for n_cap columns: wider products go in several passes
    for (size_t n0 = 0; n0 < N; n0 += sp.n_cap) {
        const size_t n = std::min(sp.n_cap, N - n0);
        StreamShape s = stream_shape(n, rows, v.nnzb, v.K, ctx->sm_count, true);
        if (!sp.slabs) s.slab = false;
        StreamArgs a = sp.args;
        a.B = static_cast<const char*>(B) + n0 * v.K * 2;
        a.C = static_cast<__half*>(C) + n0 - row_begin * 16 * ldc;  // pieces count block-rows from the plan's first
        a.status = ctx->d_status;
        a.ldc = ldc;
        a.pieces += sp.row_piece[row_begin];
        a.n_pieces = sp.row_piece[row_end] - sp.row_piece[row_begin];
        a.N = (int)n;
        a.K = (int)v.K;
        a.n_tiles = (int)((n + (size_t)s.nt - 1) / (size_t)s.nt);
        a.tile_cols = tile_cols(n, a.n_tiles);
        if (s.slab) {
            if (int rc = make_slabs(a.B, sp.slabs, n, v.K, stream)) return rc;
            a.B = sp.slabs;
        }
        a.wait_cycles = v.selftest ? kSelftestWaitCycles : kWaitCycles;
        a.lost_bytes = v.selftest ? 16 : 0;
        // The kernel's first lines, where they can pay: one round of warps (with more, most begin long after the kernel before this
        // one), and not the smallest products, which are all launch.
        const long long warps = (long long)a.n_pieces * a.n_tiles * s.w;
        a.nnzb = (int)v.nnzb;
        a.sm_count = ctx->sm_count;
        a.ahead = warps <= 40LL * ctx->sm_count && row_begin == 0 && row_end == rows && v.nnzb * 512 > kAheadBytes ? (float)((double)v.nnzb / ((double)a.n_pieces * s.w)) : 0.0f;
        if (int rc = launch<true>(s, a, stream)) return rc;
    }
    return SMAT_OK;
}

// Scratch of a product without a plan: slabs, and where a block-row can be longer than a piece the list of pieces,
// their partial tiles and counters.
size_t stream_call_bytes(const StreamShape& s, size_t N, size_t rows, size_t nnzb, size_t K) {
    const size_t extra = K / 16 > (size_t)s.chunk ? nnzb / (size_t)s.chunk + 1 : 0, n_pad = (N + (size_t)s.nt - 1) / (size_t)s.nt * (size_t)s.nt;
    return (s.slab ? round256(N * K * 2) : 0) +
           (extra ? 256 + round256(2 * extra * (n_pad / (size_t)s.nt) * sizeof(int)) + round256(extra * sizeof(uint4)) + round256(2 * extra * sizeof(int2)) +
                        round256(rows * sizeof(int)) + 2 * extra * n_pad * 64
                  : 0);
}

int stream_call(const StreamShape& s, const void* vals, const int* rowptr, const int* colidx, const void* B, void* C, size_t N, size_t K,
                size_t nnzb, size_t brow_begin, size_t brow_end, void* scratch, const DeviceCtx* ctx, cudaStream_t stream) {
    const size_t rows = brow_end - brow_begin;
    const size_t extra = K / 16 > (size_t)s.chunk ? nnzb / (size_t)s.chunk + 1 : 0, tiles = (N + (size_t)s.nt - 1) / (size_t)s.nt;
    char* b = static_cast<char*>(scratch);
    StreamArgs a = {};
    a.vals = vals;
    a.rowptr = rowptr;
    a.colidx = colidx;
    a.B = B;
    a.C = static_cast<__half*>(C);
    a.status = ctx->d_status;
    a.ldc = N;
    a.n_pieces = (int)(rows + extra);
    a.n_tiles = (int)tiles;
    a.tile_cols = tile_cols(N, a.n_tiles);
    a.N = (int)N;
    a.K = (int)K;
    a.brow_begin = (int)brow_begin;
    a.brow_end = (int)brow_end;
    a.nnzb = (int)nnzb;
    a.chunk = s.chunk;
    a.sm_count = ctx->sm_count;
    a.wait_cycles = kWaitCycles;
    if (extra) {
        int* head = reinterpret_cast<int*>(b); b += 256;
        a.long_rows = head;
        a.counters = reinterpret_cast<int*>(b);
        const size_t counter_bytes = round256(2 * extra * tiles * sizeof(int)); b += counter_bytes;
        uint4* pieces = reinterpret_cast<uint4*>(b); b += round256(extra * sizeof(uint4));
        int2* slots = reinterpret_cast<int2*>(b); b += round256(2 * extra * sizeof(int2));
        int* row_slot = reinterpret_cast<int*>(b); b += round256(rows * sizeof(int));
        a.partial = reinterpret_cast<float4*>(b); b += 2 * extra * tiles * (size_t)s.nt * 64;
        a.pieces = pieces;
        a.slots = slots;
        a.row_slot = row_slot;
        SMAT_CUDA_TRY(cudaMemsetAsync(head, 0, 256 + counter_bytes, stream));
        SMAT_CUDA_TRY(launch_pdl(long_rows_kernel, dim3((unsigned)((rows + 255) / 256)), dim3(256), 0, stream,
                                 rowptr, (int)brow_begin, (int)brow_end, (int)nnzb, s.chunk, (int)extra, head,
                                 pieces, slots, row_slot));
        count_launch();
        SMAT_CUDA_TRY(cudaGetLastError());
    }
    if (K / 16 > (size_t)kOrderWindow) {
        SMAT_CUDA_TRY(launch_pdl(column_order_kernel, dim3((unsigned)std::min((rows + 7) / 8, (size_t)ctx->sm_count * 8)), dim3(256), 0, stream,
                                 rowptr, colidx, (int)brow_begin, (int)brow_end, (int)nnzb, ctx->d_status));
        count_launch();
    }
    if (s.slab) {
        if (int rc = make_slabs(B, b, N, K, stream)) return rc;
        a.B = b;
    }
    return launch<false>(s, a, stream);
}

}  // namespace smat
