// Multiplication plan: the walk order of the SpMM kernel, computed on the device from the BCSR
// structure.
//
// For every group of 16 consecutive block-rows the kernel visits the group's block-columns in
// ascending order, four block-columns ("quad") at a time; per visited quad ("step") it needs the
// quad's column, which (sub-column, row) positions hold a block (a 64-bit mask) and the indices of
// those blocks.  Quads holding more than kPlanBlocksPerStep blocks are cut into several steps.
// The reference kernel has no such structure: it launches one CTA per (block-row, 8 columns of C)
// and walks bcsrColIdx directly (src/cuda_hgemm/src/mma/mmaCBT.cu:38-43), re-fetching the same B
// slab for every block-row that shares a block-column.
//
// Build: one CTA (16 warps) per group, warp w owns block-row w of the group.  Block-columns are
// processed in windows of 16384; inside a window a shared word per block-column collects the row
// mask (atomicOr), block-wide prefix sums number the steps and the blocks, then every block
// scatters its own index into the (group, column, row) order.  The number of steps per group is
// counted first (same pass without the scatter) and scanned; a product without a plan does without the count (`loose`).
#include <cuda_fp16.h>

#include <new>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include <type_traits>
#include <utility>
#include <queue>
#include <algorithm>

#include "host_range.h"
#include "ptx_sm100.cuh"
#include "smat_internal.h"
#include "spmm_stream.h"

namespace smat {
namespace {

constexpr int RG = kPlanRowsPerGroup;
constexpr int kPlanThreads = RG * 32;
// Block-columns per pass, a template parameter WIN: 16384 (64 KB of masks + 64 KB of block prefixes), or as few as the matrix
// has.  Masks are cleared and scanned for the whole window, so a window of 16384 for a matrix of 1024 block-columns left the
// scan to 32 of the 512 threads, each with eight quads one after the other.
constexpr int kWindow = kOrderWindow;

// Fills masks[0..WIN) for block-columns [w0, w0 + WIN) of the group; cursor[] (one per warp,
// kept by lane 0 semantics via registers) walks each row once over all windows.
// A block column below the window start (columns not ascending, or negative) or beyond the matrix is not marked, and a
// batch of 32 in which one of this window follows one of a later window is not consumed whole; the status word then
// tells the host that the structure is inconsistent.
template <int THREADS, int WIN>
__device__ __forceinline__ void mark_window(const int* __restrict__ colidx, int& cur, int end, int w0, int Kb, uint32_t* masks,
                                            int warp, int lane, int* status) {
    for (int i = threadIdx.x; i < WIN; i += THREADS) masks[i] = 0u;
    __syncthreads();
    // every lane keeps the same `cur`; lanes stride over the row until the window ends, four batches of 32 on their way at a time
    // (one after the other they were a chain of loads; products without a plan, random matrix of 16384 rows, 411 blocks a block-row,
    // N = 128: 109 -> 104 us; layer 8192 x 28672 at 20 %: 83 -> 78; bands of three blocks a block-row as before)
    constexpr int U = 4;
    for (bool more = true; more;) {
        int cbs[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = cur + 32 * u + lane;
            cbs[u] = (j < end) ? (__ldg(colidx + j) >> 4) : INT_MAX;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (!more) break;
            int cb = cbs[u];
            if (cur + lane < end && cb >= Kb) {  // beyond the last block-column: consume it without marking
                if (status) atomicCAS(status, 0, kStatusBadColumns);
                cb = w0 - 1;
            }
            const bool in = cb < w0 + WIN;
            if (in && cb >= w0) atomicOr(&masks[cb - w0], 1u << warp);
            else if (in && status) atomicCAS(status, 0, kStatusBadColumns);
            const uint32_t b = __ballot_sync(0xffffffffu, in);
            if (WIN == kOrderWindow && lane == 0 && status && (b & (b + 1u))) atomicCAS(status, 0, kStatusBadColumns);  // smaller ones hold all
            cur += __popc(b);
            more = b == 0xffffffffu;
        }
    }
    __syncthreads();
}

// True when row pointers [brow_begin, brow_end] cannot belong to a matrix of nnzb blocks (checked by every thread on the two
// ends; a dip in between shows up as a block-row whose end lies before its start and contributes nothing).
__device__ __forceinline__ bool range_is_bad(const int* __restrict__ rowptr, int brow_begin, int brow_end, int nnzb) {
    const int first = __ldg(rowptr + brow_begin), last = __ldg(rowptr + brow_end);
    return first < 0 || last < first || last > nnzb;
}

// Block-wide exclusive scan of one int per thread; returns the exclusive prefix, *total gets the sum.
template <int THREADS = kPlanThreads>
__device__ __forceinline__ int block_exclusive_scan(int v, int* total, int* sh) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += t;
    }
    if (lane == 31) sh[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int w = lane < (THREADS >> 5) ? sh[lane] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += t;
        }
        sh[32 + lane] = w;  // inclusive warp totals
    }
    __syncthreads();
    const int before = warp ? sh[32 + warp - 1] : 0;
    *total = sh[32 + (THREADS >> 5) - 1];
    __syncthreads();
    return before + inc - v;
}

template <bool FILL, int WIN>
__global__ void __launch_bounds__(kPlanThreads)
plan_kernel(const int* __restrict__ rowptr, const int* __restrict__ colidx, int brow_begin, int brow_end, int rg, int CAP, int Kb,
            int n_groups, int* __restrict__ gsp, uint4* __restrict__ steps, int* __restrict__ blk, int nnzb, int* status, int* units, bool loose) {
    ptx::pdl_wait();
    extern __shared__ uint32_t sm[];
    uint32_t* masks = sm;                                 // [WIN] row mask per block-column
    int* blk_pre = reinterpret_cast<int*>(sm + WIN);  // [WIN] exclusive block number (FILL only)
    __shared__ int scan_sh[64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The buffers of the plan are sized from the caller's block count: a range of row pointers that is not monotone or
    // holds more blocks than that would be written past their end.  Such a range gets an empty plan and a status code.
    if (range_is_bad(rowptr, brow_begin, brow_end, nnzb)) {
        if (!FILL || loose) {
            for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= n_groups; g += gridDim.x * blockDim.x) gsp[g] = 0;
            if (blockIdx.x == 0 && threadIdx.x == 0 && status) atomicCAS(status, 0, kStatusBadRowptr);
        }
        return;
    }
    for (int g = blockIdx.x; g < n_groups; g += gridDim.x) {
        const int row = brow_begin + g * rg + warp;  // warps >= rg hold no row
        const bool have = warp < rg && row < brow_end;
        const int r_lo = __ldg(rowptr + brow_begin), r_hi = __ldg(rowptr + brow_end);
        const int beg = have ? min(max(__ldg(rowptr + row), r_lo), r_hi) : 0;  // clamped: a dip inside the range reads nothing outside it
        const int end = have ? min(max(__ldg(rowptr + row + 1), beg), r_hi) : 0;
        const int gfirst = min(max(__ldg(rowptr + brow_begin + g * rg), r_lo), r_hi);  // first block of the group
        const int rfirst = __ldg(rowptr + brow_begin);           // first block of the whole range
        int cur = beg;
        int steps_done = 0, blocks_done = 0;
        // loose: nothing was counted, the group's steps (at most one a block) begin where its blocks do
        const int gs = FILL ? (loose ? gfirst - rfirst : __ldg(gsp + g)) : 0;
        const int room = FILL && loose ? min(max(__ldg(rowptr + min(brow_end, brow_begin + (g + 1) * rg)), r_lo), r_hi) - gfirst : INT_MAX;
        for (int w0 = 0; w0 < Kb; w0 += WIN) {
            const int cur_before = cur;
            mark_window<kPlanThreads, WIN>(colidx, cur, end, w0, Kb, masks, warp, lane, status);
            // per-thread chunk of the window: PER consecutive block-columns = PER / 4 quads
            constexpr int PER = WIN / kPlanThreads;
            static_assert(PER % 4 == 0, "a thread owns whole quads");
            const int i0 = threadIdx.x * PER;
            int ns = 0, nb = 0;
#pragma unroll
            for (int qd = 0; qd < PER / 4; qd++) {
                const int c = __popc(masks[i0 + 4 * qd]) + __popc(masks[i0 + 4 * qd + 1]) + __popc(masks[i0 + 4 * qd + 2]) +
                              __popc(masks[i0 + 4 * qd + 3]);
                ns += (c + CAP - 1) / CAP;
                nb += c;
            }
            if (!FILL && units) {  // MMAs of the 16-row kernel: one per block or pair of blocks in rows 2m, 2m + 1
                int nu = 0;
                for (int i = 0; i < PER; i++) nu += __popc((masks[i0 + i] | (masks[i0 + i] >> 1)) & 0x55555555u);
                nu = __reduce_add_sync(0xffffffffu, nu);
                if (lane == 0 && nu) atomicAdd(units, nu);
            }
            int tot_s, tot_b = 0;
            const int pre_s = block_exclusive_scan(ns, &tot_s, scan_sh);
            if (FILL) {
                const int pre_b = block_exclusive_scan(nb, &tot_b, scan_sh);
                if (blocks_done + tot_b > room) {  // row pointers that go down inside the range: more blocks than the group has room for
                    if (threadIdx.x == 0 && status) atomicCAS(status, 0, kStatusBadRowptr);
                    break;
                }
                int s = steps_done + pre_s, b = blocks_done + pre_b;
                for (int qd = 0; qd < PER / 4; qd++) {
                    unsigned long long m64 = 0;
#pragma unroll
                    for (int sub = 0; sub < 4; sub++) {
                        const uint32_t mk = masks[i0 + 4 * qd + sub];
                        blk_pre[i0 + 4 * qd + sub] = b + __popcll(m64);
                        m64 |= (unsigned long long)mk << (16 * sub);
                    }
                    // cut the quad into steps of at most CAP blocks, in (sub-column, row) order
                    while (m64) {
                        unsigned long long part = 0;
                        for (int t = 0; t < CAP && m64; t++) {
                            const unsigned long long low = m64 & (~m64 + 1ull);
                            part |= low;
                            m64 ^= low;
                        }
                        // position of the step's first block in the packed stream, in 256-byte units
                        const uint32_t pos = 2u * (uint32_t)(gfirst - rfirst + b);
                        steps[gs + s] = make_uint4((uint32_t)(w0 + i0 + 4 * qd) << 4, pos, (uint32_t)part, (uint32_t)(part >> 32));
                        s++;
                        b += __popcll(part);
                    }
                }
                __syncthreads();
                // scatter: block j of this warp's row goes to its (column, row) rank inside the group
                for (int j = cur_before + lane; j < cur; j += 32) {
                    const int cbx = __ldg(colidx + j) >> 4;
                    const int cb = cbx - w0;
                    if (cb < 0 || cb >= WIN || cbx >= Kb) continue;  // not marked above (status set there)
                    blk[gfirst + blk_pre[cb] + __popc(masks[cb] & ((1u << warp) - 1u))] = j;
                }
                blocks_done += tot_b;
            }
            steps_done += tot_s;
            __syncthreads();
        }
        if (!FILL && threadIdx.x == 0) gsp[g + 1] = steps_done;
        if (FILL && loose) {
            if (threadIdx.x == 0) gsp[g] = steps_done;
            __syncthreads();  // (after a break: all have left the scans)
        }
    }
    if (!FILL && blockIdx.x == 0 && threadIdx.x == 0) gsp[0] = 0;
}

// In-place inclusive scan of data[0..n) by one CTA.
__global__ void __launch_bounds__(1024) plan_scan_kernel(int* data, int n) {
    ptx::pdl_wait();
    __shared__ int warp_tot[32];
    __shared__ int carry_s, max_s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) { carry_s = 0; max_s = 0; }
    __syncthreads();
    int vmax = 0;  // the largest entry before the scan = the most steps of any group, stored behind the scanned array
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        int v = i < n ? data[i] : 0;
        vmax = max(vmax, v);
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v += t;
        }
        if (lane == 31) warp_tot[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int w = warp_tot[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, d);
                if (lane >= d) w += t;
            }
            warp_tot[lane] = w;
        }
        __syncthreads();
        v += carry_s + (warp ? warp_tot[warp - 1] : 0);
        if (i < n) data[i] = v;
        __syncthreads();
        if (threadIdx.x == 1023) carry_s = v;
        __syncthreads();
    }
    atomicMax(&max_s, vmax);
    __syncthreads();
    if (threadIdx.x == 0) data[n] = max_s;
}

// Copies the value blocks into walk order: position p of the packed stream holds block blk[first block of the range + p].
// A warp moves four blocks at a time, all loads before the stores (a warp per step, which went through the step's record and
// then its blocks one after the other, left most of the memory latency exposed: 8.4 MB of blocks 8.6 -> 3.5 us).  Lane l
// moves the 16-byte chunk l of a block (row l/2, half l%2) to chunk l ^ ((l >> 3) & 1), i.e. the 32-byte swizzle.
// Positions behind the blocks of a group whose columns were found inconsistent hold nothing: skipped by the range check.
__global__ void __launch_bounds__(256) pack_kernel(const uint4* __restrict__ vals, const int* __restrict__ blk, uint4* __restrict__ packed,
                                                  const int* __restrict__ rowptr, int brow_begin, int brow_end, int nnzb) {
    ptx::pdl_wait();
    constexpr int U = 4;
    if (range_is_bad(rowptr, brow_begin, brow_end, nnzb)) return;
    const int first = __ldg(rowptr + brow_begin), n = __ldg(rowptr + brow_end) - first;
    const int lane = threadIdx.x & 31, to = lane ^ ((lane >> 3) & 1);
    const int stride = (int)((gridDim.x * blockDim.x) >> 5) * U;
    for (int p = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * U; p < n; p += stride) {
        const int src_l = lane < U && p + lane < n ? __ldg(blk + first + p + lane) - first : -1;
        uint4 v[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int src = __shfl_sync(0xffffffffu, src_l, u);
            ok[u] = (unsigned)src < (unsigned)n;
            if (ok[u]) v[u] = __ldg(vals + (size_t)(first + src) * 32 + lane);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (ok[u]) packed[(size_t)(p + u) * 32 + to] = v[u];
    }
}


// ---- tall plans: groups of up to kTallRows block-rows (one warp of this kernel per block-row), 16-byte step records,
// ---- 64 bytes of per-warp words per step (the input of tall_pair_kernel below), groups padded to an even step count ----
constexpr int kTallPlanThreads = 1024;  // warp w owns block-row w of the group
static_assert(kTallRows == 24 && kTallBlocksPerStep <= 64, "the per-warp step words below are laid out for 12 warps of two rows and 6-bit block positions");

template <bool FILL, int WIN>
__global__ void __launch_bounds__(kTallPlanThreads)
plan_tall_kernel(const int* __restrict__ rowptr, const int* __restrict__ colidx, int brow_begin, int brow_end, int rg, int CAP, int Kb,
                 int n_groups, int* __restrict__ gsp, uint4* __restrict__ steps, uint4* __restrict__ winfo, int* __restrict__ blk,
                 int nnzb, int* status) {
    ptx::pdl_wait();
    extern __shared__ uint32_t sm[];
    uint32_t* masks = sm;                                 // [WIN] row mask per block-column
    int* blk_pre = reinterpret_cast<int*>(sm + WIN);  // [WIN] exclusive block number (FILL only)
    __shared__ int scan_sh[64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // The buffers of the plan are sized from the caller's block count: a range of row pointers that is not monotone or
    // holds more blocks than that would be written past their end.  Such a range gets an empty plan and a status code.
    if (range_is_bad(rowptr, brow_begin, brow_end, nnzb)) {
        if (!FILL) {
            for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= n_groups; g += gridDim.x * blockDim.x) gsp[g] = 0;
            if (blockIdx.x == 0 && threadIdx.x == 0 && status) atomicCAS(status, 0, kStatusBadRowptr);
        }
        return;
    }
    for (int g = blockIdx.x; g < n_groups; g += gridDim.x) {
        const int row = brow_begin + g * rg + warp;
        const bool have = warp < rg && row < brow_end;
        const int r_lo = __ldg(rowptr + brow_begin), r_hi = __ldg(rowptr + brow_end);
        const int beg = have ? min(max(__ldg(rowptr + row), r_lo), r_hi) : 0;
        const int end = have ? min(max(__ldg(rowptr + row + 1), beg), r_hi) : 0;
        const int gfirst = min(max(__ldg(rowptr + brow_begin + g * rg), r_lo), r_hi);
        const int rfirst = __ldg(rowptr + brow_begin);
        int cur = beg;
        int steps_done = 0, blocks_done = 0;
        const int gs = FILL ? __ldg(gsp + g) : 0;
        for (int w0 = 0; w0 < Kb; w0 += WIN) {
            const int cur_before = cur;
            mark_window<kTallPlanThreads, WIN>(colidx, cur, end, w0, Kb, masks, warp, lane, status);
            constexpr int PER = WIN / kTallPlanThreads;
            static_assert(PER % 4 == 0, "a thread owns whole quads");
            const int i0 = threadIdx.x * PER;
            int ns = 0, nb = 0;
#pragma unroll
            for (int qd = 0; qd < PER / 4; qd++) {
                const int c = __popc(masks[i0 + 4 * qd]) + __popc(masks[i0 + 4 * qd + 1]) + __popc(masks[i0 + 4 * qd + 2]) +
                              __popc(masks[i0 + 4 * qd + 3]);
                ns += (c + CAP - 1) / CAP;
                nb += c;
            }
            int tot_s, tot_b = 0;
            const int pre_s = block_exclusive_scan<kTallPlanThreads>(ns, &tot_s, scan_sh);
            if (FILL) {
                const int pre_b = block_exclusive_scan<kTallPlanThreads>(nb, &tot_b, scan_sh);
                int s = steps_done + pre_s, b = blocks_done + pre_b;
                for (int qd = 0; qd < PER / 4; qd++) {
                    uint32_t m[4];
                    int c = 0;
#pragma unroll
                    for (int sub = 0; sub < 4; sub++) {
                        m[sub] = masks[i0 + 4 * qd + sub];
                        blk_pre[i0 + 4 * qd + sub] = b + c;
                        c += __popc(m[sub]);
                    }
                    // cut the quad into steps of at most CAP blocks, in (sub-column, row) order
                    while (c > 0) {
                        uint32_t part[4] = {0u, 0u, 0u, 0u};
                        int taken = 0;
#pragma unroll
                        for (int sub = 0; sub < 4; sub++) {
                            while (m[sub] && taken < CAP) {
                                const uint32_t low = m[sub] & (~m[sub] + 1u);
                                part[sub] |= low;
                                m[sub] ^= low;
                                taken++;
                            }
                        }
                        const uint32_t pos = 2u * (uint32_t)(gfirst - rfirst + b);
                        steps[gs + s] = make_uint4((uint32_t)(w0 + i0 + 4 * qd) << 4, pos, (uint32_t)taken,
                                                    (part[0] ? 1u : 0u) | (part[1] ? 2u : 0u) | (part[2] ? 4u : 0u) | (part[3] ? 8u : 0u));
                        // what each MMA-issuing warp needs of the step: warp m owns block-rows 2m, 2m + 1
                        const uint32_t pre1 = (uint32_t)__popc(part[0]), pre2 = pre1 + (uint32_t)__popc(part[1]),
                                       pre3 = pre2 + (uint32_t)__popc(part[2]);
                        const uint32_t pre[4] = {0u, pre1, pre2, pre3};
                        uint4* wdst = winfo + 4 * (size_t)(gs + s);
#pragma unroll
                        for (int v = 0; v < 3; v++) {
                            uint32_t wi[4];
#pragma unroll
                            for (int mm = 0; mm < 4; mm++) {
                                const int m = 4 * v + mm;
                                uint32_t word = 0;
#pragma unroll
                                for (int sub = 0; sub < 4; sub++) {
                                    const uint32_t own = (part[sub] >> (2 * m)) & 3u;
                                    const uint32_t q = pre[sub] + (uint32_t)__popc(part[sub] & ((1u << (2 * m)) - 1u));
                                    word |= own << (2 * sub);
                                    word |= (q & 63u) << (8 + 6 * sub);
                                }
                                wi[mm] = word;
                            }
                            wdst[v] = make_uint4(wi[0], wi[1], wi[2], wi[3]);
                        }
                        wdst[3] = make_uint4((uint32_t)taken, 0u, 0u, 0u);
                        s++;
                        b += taken;
                        c -= taken;
                    }
                }
                __syncthreads();
                for (int j = cur_before + lane; j < cur; j += 32) {
                    const int cbx = __ldg(colidx + j) >> 4;
                    const int cb = cbx - w0;
                    if (cb < 0 || cb >= WIN || cbx >= Kb) continue;  // not marked above (status set there)
                    blk[gfirst + blk_pre[cb] + __popc(masks[cb] & ((1u << warp) - 1u))] = j;
                }
                blocks_done += tot_b;
            }
            steps_done += tot_s;
            __syncthreads();
        }
        // The kernel hands steps to its MMA warps two at a time: a group with an odd number of steps gets one more
        // without blocks (no panel is fetched for it).
        if (!FILL && threadIdx.x == 0) gsp[g + 1] = (steps_done + 1) & ~1;
        if (FILL && threadIdx.x == 0 && (steps_done & 1)) {
            steps[gs + steps_done] = make_uint4(0u, 2u * (uint32_t)(gfirst - rfirst + blocks_done), 0u, 0u);
            uint4* wdst = winfo + 4 * (size_t)(gs + steps_done);
            for (int v = 0; v < 4; v++) wdst[v] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    if (!FILL && blockIdx.x == 0 && threadIdx.x == 0) gsp[0] = 0;
}

// Tall plans, last pass: the kernel hands its MMA warps the steps two at a time, so what each warp has to issue for a
// pair is listed here once, ready to use.  One thread per (pair, warp m): from the two steps' words (bits 2s, 2s + 1
// = rows 2m, 2m + 1 have a block in sub-column s; bits [8 + 6s, 14 + 6s) = position of the first of them among the
// step's blocks) to the list described at kTallListBytes, its entries in (step, sub-column, row) order.
__global__ void __launch_bounds__(256) tall_pair_kernel(const uint32_t* __restrict__ wstep, uint4* __restrict__ winfo,
                                                       const int* __restrict__ gsp, int n_groups) {
    ptx::pdl_wait();
    constexpr uint32_t NM = kTallRows / 2;
    const unsigned n_lists = (unsigned)(__ldg(gsp + n_groups) >> 1) * NM;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n_lists; i += gridDim.x * blockDim.x) {
        const unsigned pr = i / NM, m = i - pr * NM;
        const uint32_t word[2] = {__ldg(wstep + ((size_t)(2 * pr)) * 16 + m), __ldg(wstep + ((size_t)(2 * pr) + 1) * 16 + m)};
        const uint32_t first_blocks = __ldg(wstep + ((size_t)(2 * pr)) * 16 + NM);  // of the first step: the second's follow them
        const uint32_t n = (uint32_t)__popc(word[0] & 0xffu) + (uint32_t)__popc(word[1] & 0xffu);
        uint32_t left[2] = {word[0], word[1]};  // bits [0, 8): blocks not listed yet
        auto next = [&]() {                     // entry of the next block
            const uint32_t st = (left[0] & 0xffu) ? 0u : 1u;
            const uint32_t x = word[st], bit = (uint32_t)__ffs((int)(left[st] & 0xffu)) - 1u, sub = bit >> 1, row = bit & 1u;
            left[st] &= left[st] - 1u;
            // position: that of the first block of the warp in this sub-column, one more for the second row behind the first
            const uint32_t q = ((x >> (8 + 6 * sub)) & 63u) + (row & (x >> (2 * sub)) & 1u);
            return ((st * first_blocks + q) * 32u) << 16 | ((4 * st + sub) * 8u) << 8 | row * 16u;
        };
        uint4* out = winfo + (size_t)i * (kTallListBytes / 16);
        uint4 v = make_uint4(0u, 0u, 0u, 0u), z = v, e = v, f = v;
        const uint32_t last = n == 16 ? 1u : 0u, c = n - last;
        v.x = (c & 1u ? kTallList1 : 0u) | (c & 2u ? kTallList2 : 0u) | (c & 4u ? kTallList4 : 0u) | (c & 8u ? kTallList8 : 0u);
        if (c & 1u) v.y = next();
        if (c & 2u) { v.z = next(); v.w = next(); }
        if (c & 4u) { z.x = next(); z.y = next(); z.z = next(); z.w = next(); }
        if (c & 8u) {
            e.x = next(); e.y = next(); e.z = next(); e.w = next();
            f.x = next(); f.y = next(); f.z = next(); f.w = next();
        }
        if (last) v.x |= kTallListLast | next();
        out[0] = v;
        out[1] = z;
        out[2] = e;
        out[3] = f;
    }
}

}  // namespace

int pack_values_async(const int* rowptr, const void* vals, const int* blk, void* packed, size_t brow_begin, size_t brow_end, size_t nnzb,
                      cudaStream_t stream, const DeviceCtx* ctx_in) {
    if (nnzb == 0 || brow_end == brow_begin) return SMAT_OK;
    const DeviceCtx* ctx = ctx_in;
    if (!ctx) {
        DeviceCtx* c = nullptr;
        if (int rc = get_device_ctx(&c)) return rc;
        ctx = c;
    }
    const size_t want = (nnzb + 31) / 32, most = (size_t)ctx->sm_count * 8;  // 32 blocks per CTA and trip
    SMAT_CUDA_TRY(launch_pdl(pack_kernel, dim3((unsigned)(want < most ? want : most)), dim3(256), 0, stream,
                             reinterpret_cast<const uint4*>(vals), blk,
                             reinterpret_cast<uint4*>(packed), rowptr, (int)brow_begin,
                             (int)brow_end, (int)nnzb));
    count_launch();
    SMAT_CUDA_TRY(cudaGetLastError());
    return SMAT_OK;
}

size_t choose_rows_per_group(size_t block_rows, size_t N, int sm_count, bool can_cut, size_t nnzb, size_t K) {
    static const int forced = [] {  // tuning knob: SMAT_ROWS_PER_GROUP=4..16 overrides the choice
        const char* e = std::getenv("SMAT_ROWS_PER_GROUP");
        const int v = e ? std::atoi(e) : 0;
        return (v >= 4 && v <= kPlanRowsPerGroup) ? v : 0;
    }();
    if (forced) return (size_t)forced;
    if (N == 0 || block_rows == 0) return kPlanRowsPerGroup;
    const size_t sms = (size_t)sm_count;
    size_t best = kPlanRowsPerGroup;
    double best_cost = 0.0;
    for (size_t rg = kPlanRowsPerGroup; rg >= 8; rg--) {
        const size_t groups = (block_rows + rg - 1) / rg;
        size_t est_steps = nnzb / groups;  // steps per item: at most one per block and one per 64 columns
        if (K / 64 < est_steps) est_steps = K / 64;
        // the per-item overhead (pipeline fill, epilogue, steps that do not shrink with the height) is worth about
        // four block-rows of work
        double cost = rounds_for(groups * ((N + 127) / 128), sms, can_cut, est_steps, false) * (double)(rg + 4);
        if (N >= 256 && nnzb / groups >= 256 && est_steps >= 64) {
            const double wide = kWideItemCost * rounds_for(groups * ((N + 255) / 256), sms, can_cut, est_steps, true) * (double)(rg + 4);
            if (wide < cost) cost = wide;
        }
        if (rg == kPlanRowsPerGroup || cost < best_cost * 0.97) {  // a smaller group must pay for its lower panel reuse
            best = rg;
            best_cost = cost;
        }
    }
    return best;
}

PlanSizes plan_sizes(size_t nnzb, size_t brow_begin, size_t brow_end, size_t rg, size_t max_steps) {
    PlanSizes s;
    s.n_groups = (brow_end - brow_begin + rg - 1) / rg;
    s.gsp_bytes = ((s.n_groups + 3) * sizeof(int) + 255) / 256 * 256;  // + the largest step count of a group and the MMA count
    // a step holds at least one block, so nnzb bounds the number of steps
    const size_t steps = max_steps ? max_steps : (nnzb ? nnzb : 1);
    s.steps_bytes = (steps * sizeof(uint4) + 255) / 256 * 256;
    s.blk_bytes = ((nnzb ? nnzb : 1) * sizeof(int) + 255) / 256 * 256;
    s.packed_bytes = (nnzb ? nnzb : 1) * 512;
    return s;
}

// Packing costs its launches and a pass over the blocks, gathering a copy for every block of every tile of C: 28 cycles each, which
// hide behind the MMA of a block (39 and more), not behind one MMA for several blocks above one another, and not all of the time
// where many CTAs gather at once.  us, packed and gathered, by columns:
//   4096 block-rows, clusters, 65 536 blocks: 1024: 104 and 98, 1536: 135 and 135, 2048: 165 and 175, 8192: 546 and 603
//   2048, band of 67 000: 1024: 98 and 90, 1536: 139 and 146, 2048: 160 and 170, 8192: 531 and 609; of 164 000: 1024: 192 and 177,
//     2048: 330 and 350, 4096: 609 and 648; of 10 000: 2048: 82 and 76, 4096: 130 and 126, 8192: 229 and 225
//   1024, clusters, 16 384: 1536: 56 and 51, 2560: 72 and 72, 8192: 155 and 170; random, 237 000: 2048: 647 and 624, 4096: 1278 and 1277
//   512, layer, 183 000: 2048: 560 and 534, 3072: 827 and 844, 4096: 1020 and 1055; dense, 262 000: 2048: 523 and 506, 4096: 898 and 951
//   256, layer, 26 000: 4096: 180 and 170, 8192: 303 and 305;  128, dense, 65 536: 4096: 308 and 280, 8192: 603 and 578
bool pack_for_call(size_t N, size_t rows, size_t nnzb) {
    if (g_spmm_variant == 2 || g_spmm_variant == 3) return true;  // these read a packed copy
    const size_t tiles = (N + 127) / 128;
    return rows >= 512 && tiles > (rows >= 2048 ? 12u : 24u) && tiles * nnzb > 350000;
}

double tc_estimate_us(const PlanView& v, size_t N, size_t sms) {
    const size_t items = v.n_groups * ((N + 127) / 128);
    const double per_group = (double)v.total_steps / (double)v.n_groups;
    // the heaviest item is cut into as many segments as the others, or not at all
    const double longest = v.heaviest_cycles / (items < sms ? (double)tail_parts_for(items, sms, true, (size_t)per_group) : 1.0);
    double cycles;
    if (v.tall)
        cycles = std::max(tall_rounds(items, sms, per_group) * per_group * std::max(v.step_cycles, kTallLeastCycles), longest) + kTallExtraCycles;
    // (graphs, whose steps differ as much as their groups: measured 1.5 to 1.6 times the even share of the steps)
    else if (v.balanced || v.sched_list) cycles = 1.55 * (double)items / (double)sms * per_group * v.step_cycles;
    else cycles = std::max(rounds_for(items, sms, true, (size_t)per_group, false) * per_group * v.step_cycles, longest);
    return 8.0 + cycles / 1850.0;
}

// Launches a plan kernel with the smallest window that holds the matrix, with as many CTAs as fit the SMs.
template <int THREADS, class Launch>
static int launch_windowed(size_t Kb, size_t n_groups, int words_per_column, int sm_count, Launch&& launch) {
    auto go = [&](auto win) -> int {
        const size_t smem = (size_t)decltype(win)::value * 4 * (size_t)words_per_column;
        const size_t resident = std::max<size_t>(1, std::min<size_t>(2048 / THREADS, (200 * 1024) / (smem + 1024)));
        return launch(win, (int)std::min(n_groups, (size_t)sm_count * resident), smem);
    };
    if (Kb <= THREADS * 4) return go(std::integral_constant<int, THREADS * 4>{});
    if (THREADS * 8 < kWindow && Kb <= THREADS * 8) return go(std::integral_constant<int, THREADS * 8>{});
    return go(std::integral_constant<int, kWindow>{});
}

static int plan_launch_setup(const DeviceCtx* ctx_in, const DeviceCtx** ctx) {
    *ctx = ctx_in;
    if (!*ctx) {
        DeviceCtx* c = nullptr;
        if (int rc = get_device_ctx(&c)) return rc;
        *ctx = c;
    }
    return SMAT_OK;
}

int plan_count_async(const int* rowptr, const int* colidx, size_t K, size_t nnzb, size_t brow_begin, size_t brow_end,
                     size_t rg, int* gsp, cudaStream_t stream, const DeviceCtx* ctx_in, size_t cap, int* units) {
    const DeviceCtx* ctx = nullptr;
    if (int rc = plan_launch_setup(ctx_in, &ctx)) return rc;
    const size_t n_groups = (brow_end - brow_begin + rg - 1) / rg;
    if (n_groups == 0) return SMAT_OK;
    if (nnzb == 0) {
        SMAT_CUDA_TRY(cudaMemsetAsync(gsp, 0, (n_groups + 1) * sizeof(int), stream));
        return SMAT_OK;
    }
    const int rc = launch_windowed<kPlanThreads>(K / 16, n_groups, 1, ctx->sm_count, [&](auto win, int grid, size_t smem) -> int {
        auto kernel = plan_kernel<false, decltype(win)::value>;
        SMAT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        SMAT_CUDA_TRY(launch_pdl(kernel, dim3(grid), dim3(kPlanThreads), smem, stream,
                                 rowptr, colidx, (int)brow_begin, (int)brow_end, (int)rg, (int)cap, (int)(K / 16),
                                 (int)n_groups, gsp, nullptr, nullptr, (int)nnzb, ctx->d_status, units, false));
        return SMAT_OK;
    });
    if (rc) return rc;
    count_launch();
    SMAT_CUDA_TRY(launch_pdl(plan_scan_kernel, dim3(1), dim3(1024), 0, stream,
                             gsp, (int)n_groups + 1));
    count_launch();
    SMAT_CUDA_TRY(cudaGetLastError());
    return SMAT_OK;
}

static int plan_fill(const int* rowptr, const int* colidx, size_t K, size_t nnzb, size_t brow_begin, size_t brow_end, size_t rg, int* gsp,
                     void* steps, int* blk, cudaStream_t stream, const DeviceCtx* ctx_in, size_t cap, bool loose) {
    const DeviceCtx* ctx = nullptr;
    if (int rc = plan_launch_setup(ctx_in, &ctx)) return rc;
    const size_t n_groups = (brow_end - brow_begin + rg - 1) / rg;
    if (n_groups == 0 || nnzb == 0) return SMAT_OK;
    const int rc = launch_windowed<kPlanThreads>(K / 16, n_groups, 2, ctx->sm_count, [&](auto win, int grid, size_t smem) -> int {
        auto kernel = plan_kernel<true, decltype(win)::value>;
        SMAT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        SMAT_CUDA_TRY(launch_pdl(kernel, dim3(grid), dim3(kPlanThreads), smem, stream,
                                 rowptr, colidx, (int)brow_begin, (int)brow_end, (int)rg, (int)cap, (int)(K / 16),
                                 (int)n_groups, gsp, reinterpret_cast<uint4*>(steps), blk, (int)nnzb,
                                 ctx->d_status, nullptr, loose));
        return SMAT_OK;
    });
    if (rc) return rc;
    count_launch();
    SMAT_CUDA_TRY(cudaGetLastError());
    return SMAT_OK;
}
int plan_fill_async(const int* rowptr, const int* colidx, size_t K, size_t nnzb, size_t brow_begin, size_t brow_end,
                    size_t rg, const int* gsp, void* steps, int* blk, cudaStream_t stream, const DeviceCtx* ctx, size_t cap) {
    return plan_fill(rowptr, colidx, K, nnzb, brow_begin, brow_end, rg, const_cast<int*>(gsp), steps, blk, stream, ctx, cap, false);
}
int plan_fill_loose_async(const int* rowptr, const int* colidx, size_t K, size_t nnzb, size_t brow_begin, size_t brow_end,
                          size_t rg, int* gsp, void* steps, int* blk, cudaStream_t stream, const DeviceCtx* ctx) {
    return plan_fill(rowptr, colidx, K, nnzb, brow_begin, brow_end, rg, gsp, steps, blk, stream, ctx, kPlanBlocksPerStep, true);
}


int plan_count_tall_async(const int* rowptr, const int* colidx, size_t K, size_t nnzb, size_t brow_begin, size_t brow_end,
                          size_t rg, int* gsp, cudaStream_t stream, const DeviceCtx* ctx_in) {
    const DeviceCtx* ctx = nullptr;
    if (int rc = plan_launch_setup(ctx_in, &ctx)) return rc;
    const size_t n_groups = (brow_end - brow_begin + rg - 1) / rg;
    if (n_groups == 0) return SMAT_OK;
    if (nnzb == 0) {
        SMAT_CUDA_TRY(cudaMemsetAsync(gsp, 0, (n_groups + 1) * sizeof(int), stream));
        return SMAT_OK;
    }
    const int rc = launch_windowed<kTallPlanThreads>(K / 16, n_groups, 1, ctx->sm_count, [&](auto win, int grid, size_t smem) -> int {
        auto kernel = plan_tall_kernel<false, decltype(win)::value>;
        SMAT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        SMAT_CUDA_TRY(launch_pdl(kernel, dim3(grid), dim3(kTallPlanThreads), smem, stream,
                                 rowptr, colidx, (int)brow_begin, (int)brow_end, (int)rg, kTallBlocksPerStep,
                                 (int)(K / 16), (int)n_groups, gsp, nullptr, nullptr, nullptr, (int)nnzb,
                                 ctx->d_status));
        return SMAT_OK;
    });
    if (rc) return rc;
    count_launch();
    SMAT_CUDA_TRY(launch_pdl(plan_scan_kernel, dim3(1), dim3(1024), 0, stream,
                             gsp, (int)n_groups + 1));
    count_launch();
    SMAT_CUDA_TRY(cudaGetLastError());
    return SMAT_OK;
}

int plan_fill_tall_async(const int* rowptr, const int* colidx, size_t K, size_t nnzb, size_t brow_begin, size_t brow_end,
                         size_t rg, const int* gsp, void* steps, void* wstep, void* winfo, int* blk, cudaStream_t stream,
                         const DeviceCtx* ctx_in) {
    const DeviceCtx* ctx = nullptr;
    if (int rc = plan_launch_setup(ctx_in, &ctx)) return rc;
    const size_t n_groups = (brow_end - brow_begin + rg - 1) / rg;
    if (n_groups == 0 || nnzb == 0) return SMAT_OK;
    const int rc = launch_windowed<kTallPlanThreads>(K / 16, n_groups, 2, ctx->sm_count, [&](auto win, int grid, size_t smem) -> int {
        auto kernel = plan_tall_kernel<true, decltype(win)::value>;
        SMAT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        SMAT_CUDA_TRY(launch_pdl(kernel, dim3(grid), dim3(kTallPlanThreads), smem, stream,
                                 rowptr, colidx, (int)brow_begin, (int)brow_end, (int)rg, kTallBlocksPerStep,
                                 (int)(K / 16), (int)n_groups, const_cast<int*>(gsp), reinterpret_cast<uint4*>(steps),
                                 reinterpret_cast<uint4*>(wstep), blk, (int)nnzb, ctx->d_status));
        return SMAT_OK;
    });
    if (rc) return rc;
    count_launch();
    SMAT_CUDA_TRY(launch_pdl(tall_pair_kernel, dim3(ctx->sm_count * 4), dim3(256), 0, stream,
                             reinterpret_cast<const uint32_t*>(wstep), reinterpret_cast<uint4*>(winfo), gsp,
                             (int)n_groups));
    count_launch();
    SMAT_CUDA_TRY(cudaGetLastError());
    return SMAT_OK;
}

}  // namespace smat

using namespace smat;

struct smat_plan {
    PlanView v;          // for products about as wide as the hint
    // A stream plan of a matrix on which a tcgen05 kernel is faster for wide products: the plan of that kernel, for products
    // of `wide_from` columns or more (0: no such plan).  smat_plan_set_values keeps both up to date.
    PlanView wide;
    size_t wide_from = 0;
    int sms = 0;
    // everything the plan holds on the device but step counts and schedule: one allocation (each costs 0.3 ms, whatever its size)
    void* buffer = nullptr;
    void* gsp_buffer = nullptr;
    StreamPlan stream;
    void* sched_buffer = nullptr;  // listed schedule: offsets per CTA, then the groups
    int device = -1;
    size_t nnzb = 0;  // blocks of the whole arrays, as given
    // smat_plan_spmm_host: device staging (B and C whole), the copy streams, per-chunk and per-range events
    void* host_B = nullptr;
    void* host_C = nullptr;
    size_t host_B_bytes = 0, host_C_bytes = 0;
    cudaStream_t s_in = nullptr, s_out = nullptr;
    cudaEvent_t ev_start = nullptr;
    std::vector<cudaEvent_t> ev_in, ev_done, ev_out;
};

// One chunk of columns of C, rows x `width16` 16-byte words, from device memory to pinned host memory that the device can
// address, both `pitch16` words from row to row.  A 2-D copy of the copy engine moves rows of 512 bytes at 8 GB/s
// (measured; 50 GB/s in one piece), stores from the SMs at the rate of the link; eight CTAs are enough for that and leave
// the other SMs to the product of the next chunk.
static __global__ void __launch_bounds__(256) copy_out_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, size_t rows, size_t pitch16,
                                                             unsigned width16) {
    const size_t n = rows * width16, stride = (size_t)gridDim.x * 256;
    constexpr int U = 4;
    for (size_t i0 = (size_t)blockIdx.x * 256 + threadIdx.x; i0 < n; i0 += U * stride) {
        uint4 v[U];
        size_t at[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const size_t i = i0 + u * stride, row = i / width16;
            at[u] = row * pitch16 + (i - row * width16);
            if (i < n) v[u] = __ldg(src + at[u]);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * stride < n) dst[at[u]] = v[u];
    }
}

// The device's address of `bytes` of host memory, or null when not all of it is pinned (then only the copy engine can reach it).
static char* device_view_of_host(void* p, size_t bytes) {
    if ((uintptr_t)p & 15) return nullptr;
    typedef CUresult (*AttributeFn)(void*, CUpointer_attribute, CUdeviceptr);
    static const AttributeFn attribute = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            fn = nullptr;
        }
        return (AttributeFn)fn;
    }();
    if (!attribute) return nullptr;
    return device_view_of_range(p, bytes, [](uintptr_t at, HostMapping* m) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, reinterpret_cast<void*>(at)) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        CUdeviceptr base = 0;
        if (a.type != cudaMemoryTypeHost || attribute(&base, CU_POINTER_ATTRIBUTE_MAPPING_BASE_ADDR, at) != CUDA_SUCCESS ||
            attribute(&m->size, CU_POINTER_ATTRIBUTE_MAPPING_SIZE, at) != CUDA_SUCCESS)
            return false;
        m->base = base;
        m->device = static_cast<char*>(a.devicePointer);
        return true;
    });
}

static const PlanView& view_for(const smat_plan* p, size_t N) { return p->wide_from && N >= p->wide_from ? p->wide : p->v; }

// The width from which a matrix planned with the stream kernel for `hint` columns is multiplied by the tcgen05 kernel of `tc`; 0:
// at no width looked at.  The two estimates are off by some 20 %, so the kernel for the hint stays until the other's is lower
// by that: dense clusters of 131072 rows planned for 8 columns and used with 16 take 16.6 us with it, 25.7 with the other
// kernel, whose estimate is the lower one.  From there on it is the other: 8192 x 28672 layer planned for 16 columns,
// 2048 columns in 2560 us by passes of 128, in 484 by it; 256 columns 318 and 73.
static size_t wide_from_width(const PlanView& tc, size_t hint, int sms) {
    const size_t rows = tc.brow_end - tc.brow_begin, cap = stream_pass_columns(hint), last = std::max<size_t>(4096, 2 * cap);
    for (size_t N = (hint + 7) / 8 * 8; N <= last; N += N < 2 * cap ? 8 : 128)
        if (N > hint && stream_passes_us(N, hint, rows, tc.nnzb, tc.K, sms) >= 1.25 * tc_estimate_us(tc, N, (size_t)sms)) return N;
    return 0;
}

static cudaError_t free_plan(smat_plan* p) {
    cudaError_t e = cudaSuccess;
    for (void* b : {p->buffer, p->gsp_buffer, p->sched_buffer}) {
        const cudaError_t eb = cudaFree(b);
        if (e == cudaSuccess) e = eb;
    }
    delete p;
    return e;
}

// A plan's memory and tuning belong to the device it was created on.
static int check_plan_device(const smat_plan* plan) {
    int dev = -1;
    SMAT_CUDA_TRY(cudaGetDevice(&dev));
    if (dev != plan->device)
        return fail(SMAT_ERR_BAD_ARG, "the plan belongs to device %d but device %d is current", plan->device, dev);
    return SMAT_OK;
}

extern "C" {

int smat_plan_create(smat_plan** out, const void* bcsrValuesA, const int* bcsrRowPtrA, const int* bcsrColIdxA, size_t M,
                     size_t K, size_t nnzb, size_t brow_begin, size_t brow_end, size_t N_hint, void* stream) {
    clear_error();
    if (!out || !bcsrRowPtrA || (nnzb && (!bcsrColIdxA || !bcsrValuesA))) return fail(SMAT_ERR_BAD_ARG, "NULL argument");
    if (M % 16 || K % 16) return fail(SMAT_ERR_BAD_ARG, "M (%zu) and K (%zu) must be multiples of 16", M, K);
    if ((uintptr_t)bcsrValuesA & 15) return fail(SMAT_ERR_BAD_ARG, "bcsrValuesA must be 16-byte aligned");
    if (brow_begin > brow_end || brow_end > M / 16)
        return fail(SMAT_ERR_BAD_ARG, "block-row range [%zu, %zu) outside [0, %zu]", brow_begin, brow_end, M / 16);
    if (nnzb * 16 >= ((size_t)1 << 31) || K >= ((size_t)1 << 31)) return fail(SMAT_ERR_RANGE, "size beyond 2^31");
    smat_plan* p = new (std::nothrow) smat_plan();
    if (!p) return fail(SMAT_ERR_NOMEM, "out of host memory");
    DeviceCtx* ctx = nullptr;
    if (int rc0 = get_device_ctx(&ctx)) {
        delete p;
        return rc0;
    }
    const size_t rg = choose_rows_per_group(brow_end - brow_begin, N_hint, ctx->sm_count, true, nnzb, K);
    // phase 1 into a small buffer of its own; the step total then sizes the rest exactly
    PlanSizes sz = plan_sizes(nnzb, brow_begin, brow_end, rg);
    cudaError_t e = cudaGetDevice(&p->device);
    if (e == cudaSuccess) e = cudaMalloc(&p->gsp_buffer, sz.gsp_bytes);
    if (e != cudaSuccess) {
        cudaFree(p->gsp_buffer);
        delete p;
        return fail(SMAT_ERR_CUDA, "plan allocation failed: %s", cudaGetErrorString(e));
    }
    int* gsp = static_cast<int*>(p->gsp_buffer);
    int* units = nnzb && sz.n_groups ? gsp + sz.n_groups + 2 : nullptr;  // behind the scanned counts and their maximum
    int rc = SMAT_OK;
    if (units) {
        e = cudaMemsetAsync(units, 0, sizeof(int), (cudaStream_t)stream);
        if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
    }
    if (rc == SMAT_OK)
        rc = plan_count_async(bcsrRowPtrA, bcsrColIdxA, K, nnzb, brow_begin, brow_end, rg, gsp, (cudaStream_t)stream, nullptr, kPlanBlocksPerStep, units);
    // ... and the blocks of THIS range (nonzeroBlocks counts the whole arrays): what the choices below and at launch go by
    int total_and_max[3] = {0, 0, 0}, ends[2] = {0, 0};
    if (rc == SMAT_OK && sz.n_groups) {
        e = cudaMemcpyAsync(total_and_max, gsp + sz.n_groups, (units ? 3 : 2) * sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
        if (e == cudaSuccess && nnzb)
            e = cudaMemcpyAsync(&ends[0], bcsrRowPtrA + brow_begin, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
        if (e == cudaSuccess && nnzb)
            e = cudaMemcpyAsync(&ends[1], bcsrRowPtrA + brow_end, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
        if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
    }
    const int mmas16 = total_and_max[2];
    size_t range_blocks = nnzb;
    if (rc == SMAT_OK && nnzb && sz.n_groups && ends[1] >= ends[0] && (size_t)(ends[1] - ends[0]) <= nnzb) range_blocks = (size_t)(ends[1] - ends[0]);
    // Densely filled quads (dense clusters: every quad of a cluster holds all 64 blocks) are cut into pieces of at most 24
    // blocks that each fetch the B panel again; when the steps are that full on average, recount with 32 per step.
    size_t cap = kPlanBlocksPerStep;
    if (rc == SMAT_OK && total_and_max[0] > 0 && range_blocks >= 18 * (size_t)total_and_max[0]) {
        cap = kPlanBlocksPerStepDense;
        rc = plan_count_async(bcsrRowPtrA, bcsrColIdxA, K, nnzb, brow_begin, brow_end, rg, gsp, (cudaStream_t)stream, nullptr, cap);
        if (rc == SMAT_OK) {
            e = cudaMemcpyAsync(total_and_max, gsp + sz.n_groups, 2 * sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
            if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
        }
    }
    const int total_steps = total_and_max[0];  // of the 16-row plan
    // Schedule: when the heaviest group holds many times the average number of steps, items dealt out round-robin
    // leave most SMs waiting for the one with the heaviest item; such plans deal out equal step ranges instead.
    bool balanced = (size_t)total_and_max[1] * sz.n_groups > 4 * (size_t)total_steps &&
                    (size_t)total_steps >= 8 * (size_t)ctx->sm_count;
    if (rc == SMAT_OK && balanced && sz.n_groups >= 4 * (size_t)ctx->sm_count) {
        // First choice: whole groups dealt out heaviest first to the least loaded CTA (keeps every item in one piece
        // and the CTAs sweeping the block-columns the way the round-robin schedule does); taken when the heaviest
        // CTA ends up within a quarter of the average load.
        const int G = ctx->sm_count;
        std::vector<int> h_gsp(sz.n_groups + 1);
        e = cudaMemcpy(h_gsp.data(), gsp, (sz.n_groups + 1) * sizeof(int), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
        if (rc == SMAT_OK) {
            std::vector<int> order(sz.n_groups);
            for (size_t g = 0; g < sz.n_groups; g++) order[g] = (int)g;
            std::stable_sort(order.begin(), order.end(),
                             [&](int a, int b) { return h_gsp[a + 1] - h_gsp[a] > h_gsp[b + 1] - h_gsp[b]; });
            std::priority_queue<std::pair<long long, int>, std::vector<std::pair<long long, int>>, std::greater<>> heap;
            for (int c = 0; c < G; c++) heap.push({0, c});
            std::vector<std::vector<int>> lists(G);
            long long heaviest = 0;
            for (int g : order) {
                auto [load, c] = heap.top();
                heap.pop();
                load += h_gsp[g + 1] - h_gsp[g];
                lists[c].push_back(g);
                if (load > heaviest) heaviest = load;
                heap.push({load, c});
            }
            if (heaviest * 4 * G <= 5LL * total_steps) {
                std::vector<int> flat(G + 1 + sz.n_groups);
                int pos = 0;
                for (int c = 0; c < G; c++) {
                    flat[c] = pos;
                    for (int g : lists[c]) flat[G + 1 + pos++] = g;
                }
                flat[G] = pos;
                e = cudaMalloc(&p->sched_buffer, flat.size() * sizeof(int));
                if (e == cudaSuccess) e = cudaMemcpy(p->sched_buffer, flat.data(), flat.size() * sizeof(int), cudaMemcpyHostToDevice);
                if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan allocation failed: %s", cudaGetErrorString(e));
                p->v.sched_off = static_cast<const int*>(p->sched_buffer);
                p->v.sched_list = static_cast<const int*>(p->sched_buffer) + G + 1;
                p->v.sched_ctas = G;
                balanced = false;
            }
        }
    }
    // Tall plan: groups of up to 24 block-rows for the kernel that reads the B panels from tensor memory.  Its steps
    // cost as much as those of the 16-row kernels or more (tall_step_cycles(), at least 500, against ~480 cycles, the latter growing with
    // the MMAs of the step: ~58 cycles each with the hand-overs, the shared-memory operand port; vertical neighbours
    // share one, which is what keeps dense clusters with this kernel), so it pays where taller groups mean
    // fewer steps: matrices whose quads mostly hold a block (a block-sparse layer, a reordered random matrix: three
    // quarters of the steps), not those of a block or less a quad (as many steps as before) and not dense clusters (steps of 32
    // blocks already).  Both plans are counted and the estimates compared; smat_spmm_set_variant(4) forces a tall plan,
    // 1..3 exclude it.
    const double mma_per_step = total_steps > 0 ? (double)mmas16 / (double)total_steps : 0.0;
    // cycles of a 16-row step: an MMA per block or pair of vertical neighbours, or, where whole columns of blocks are there
    // (dense clusters), one per column
    const bool vertical = mmas16 > 0 && (double)range_blocks >= 1.7 * (double)mmas16;
    const double work16 = vertical ? 20.0 * (double)range_blocks / (double)(total_steps > 0 ? total_steps : 1) : 58.0 * mma_per_step;
    const double step16 = work16 > 480.0 ? work16 : 480.0;
    bool tall = false;
    size_t rg_used = rg;
    const size_t rows = brow_end - brow_begin, tiles = ((N_hint ? N_hint : 128) + 127) / 128;
    const bool tall_forced = g_spmm_variant == 4;
    const bool tall_possible = rc == SMAT_OK && !balanced && !p->v.sched_list && total_steps > 0 && rows > 0 &&
                               (tall_forced || (g_spmm_variant == 0 && rows >= 12 && N_hint >= 16 &&
                                                (size_t)total_steps * tiles >= 16 * (size_t)ctx->sm_count));
    if (tall_possible) {
        // Height of the groups: what a launch costs is about (rounds of work items) x (steps of an item) x (cycles of
        // a step, which grow with its blocks).  The quads of an item hardly change with the height as
        // long as most hold a block, but those with more blocks than a step holds are cut into several steps: with the
        // blocks of a quad spread like a binomial count, the share of them is taken from the logistic curve closest to it.
        size_t rg_tall = kTallRows;
        double best = 0.0;
        const double quads = std::max(1.0, std::min((double)total_steps / (double)sz.n_groups, std::ceil((double)K / 64.0)));
        for (size_t r = kTallRows; r >= 12; r -= 2) {
            const size_t groups = (rows + r - 1) / r;
            const double per_quad = (double)range_blocks / (double)rows * (double)(r < rows ? r : rows) / quads;
            double pieces = 1.0;
            for (int k = 1; k <= 3; k++)
                pieces += 1.0 / (1.0 + std::exp(((double)(k * kTallBlocksPerStep) + 0.5 - per_quad) / (0.5 * std::sqrt(per_quad) + 1e-9)));
            const double steps = quads * pieces;
            const double cost = tall_rounds(groups * tiles, (size_t)ctx->sm_count, steps) * steps * tall_step_cycles(per_quad / pieces);
            if (r == (size_t)kTallRows || cost < best * 0.97) {
                best = cost;
                rg_tall = r;
            }
        }
        if (const char* ev = std::getenv("SMAT_TALL_ROWS")) {  // tuning knob
            const int v = std::atoi(ev);
            if (v >= 1 && v <= kTallRows) rg_tall = (size_t)v;
        }
        // the group count changes with the height: count into a buffer of its own, kept if the tall plan is taken
        const PlanSizes sz_tall = plan_sizes(nnzb, brow_begin, brow_end, rg_tall);
        void* gsp_tall = nullptr;
        int tall_total_and_max[2] = {0, 0};
        e = cudaMalloc(&gsp_tall, sz_tall.gsp_bytes);
        if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan allocation failed: %s", cudaGetErrorString(e));
        if (rc == SMAT_OK)
            rc = plan_count_tall_async(bcsrRowPtrA, bcsrColIdxA, K, nnzb, brow_begin, brow_end, rg_tall, static_cast<int*>(gsp_tall),
                                       (cudaStream_t)stream);
        if (rc == SMAT_OK) {
            e = cudaMemcpyAsync(tall_total_and_max, static_cast<int*>(gsp_tall) + sz_tall.n_groups, 2 * sizeof(int), cudaMemcpyDeviceToHost,
                                (cudaStream_t)stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
            if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
        }
        if (rc == SMAT_OK) {
            const double steps_per_group = (double)total_steps / (double)sz.n_groups;
            const double est16 = rounds_for(sz.n_groups * tiles, (size_t)ctx->sm_count, true, (size_t)steps_per_group, false) * steps_per_group * step16;
            const double steps_per_tall = (double)tall_total_and_max[0] / (double)sz_tall.n_groups;
            const double est_tall =
                tall_rounds(sz_tall.n_groups * tiles, (size_t)ctx->sm_count, steps_per_tall) * steps_per_tall *
                    std::max(tall_step_cycles((double)range_blocks / (double)(tall_total_and_max[0] > 0 ? tall_total_and_max[0] : 1)), kTallLeastCycles16) +
                kTallExtraCycles;
            tall = tall_forced || est_tall < est16;
            if (std::getenv("SMAT_PLAN_DEBUG"))
                fprintf(stderr, "[smat plan] estimates: 16-row %.0f cycles, tall (rg %zu, %d steps) %.0f cycles -> %s\n", est16, rg_tall,
                        tall_total_and_max[0], est_tall, tall ? "tall" : "16-row");
        }
        if (rc == SMAT_OK && tall) {
            cudaFree(p->gsp_buffer);
            p->gsp_buffer = gsp_tall;
            gsp = static_cast<int*>(gsp_tall);
            sz = sz_tall;
            rg_used = rg_tall;
            total_and_max[0] = tall_total_and_max[0];
            total_and_max[1] = tall_total_and_max[1];
            cap = kTallBlocksPerStep;
        } else {
            cudaFree(gsp_tall);
        }
    }
    const int steps_final = total_and_max[0];
    PlanView& v = p->v;
    p->sms = ctx->sm_count;
    v.rowptr = bcsrRowPtrA;
    v.gsp = gsp;
    v.K = K;
    v.nnzb = range_blocks;  // blocks of the plan's range
    v.brow_begin = brow_begin;
    v.brow_end = brow_end;
    v.n_groups = sz.n_groups;
    v.rg = rg_used;
    v.total_steps = (size_t)(steps_final > 0 ? steps_final : 0);
    v.balanced = balanced;
    v.cap = cap;
    v.vertical = vertical;
    v.tall = tall;
    v.step_cycles = tall ? tall_step_cycles((double)range_blocks / (double)(steps_final > 0 ? steps_final : 1)) : step16;
    // (a tall group of many more steps than quads holds full steps)
    v.heaviest_cycles = total_and_max[1] * (tall && (double)total_and_max[1] > 1.2 * std::ceil((double)K / 64.0) ? tall_step_cycles(40.0) : v.step_cycles);
    // Stream plan (spmm_stream_sm100.cu): taken where its estimate is below that of the kernel chosen so far.  That one is kept
    // beside it where it is faster for wide products: each pass over the matrix with the stream kernel multiplies 128 columns
    // or as many as the hint names, so a plan made for 16 columns would take 32 passes for 4096.
    bool stream_too = false;
    StreamLayout layout;
    PlanView narrow;  // the stream plan's
    narrow.K = K;
    narrow.nnzb = range_blocks;
    narrow.brow_begin = brow_begin;
    narrow.brow_end = brow_end;
    if (rc == SMAT_OK && total_steps > 0 && (g_spmm_variant == 5 || (g_spmm_variant == 0 && N_hint > 0))) {
        const size_t hint = N_hint ? N_hint : 128;
        const double us = stream_estimate_us(hint, rows, range_blocks, K, ctx->sm_count, true), other = tc_estimate_us(v, hint, (size_t)ctx->sm_count);
        if (std::getenv("SMAT_PLAN_DEBUG"))
            fprintf(stderr, "[smat plan] stream %.1f us, %s %.1f us; the latter from %zu columns\n", us, tall ? "tall" : "16-row", other,
                    wide_from_width(v, hint, ctx->sm_count));
        if (g_spmm_variant == 5 || us < other) {
            std::vector<int> h_rowptr(rows + 1);
            e = cudaMemcpyAsync(h_rowptr.data(), bcsrRowPtrA + brow_begin, (rows + 1) * sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
            if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
            stream_too = rc == SMAT_OK && std::is_sorted(h_rowptr.begin(), h_rowptr.end());
            if (stream_too) {
                if (g_spmm_variant != 5) p->wide_from = wide_from_width(v, hint, ctx->sm_count);
                layout = stream_plan_layout(h_rowptr.data(), rows, K, hint, ctx->sm_count, p->wide_from != 0);
            }
            if (stream_too && p->wide_from == 0) {
                cudaFree(p->gsp_buffer);
                cudaFree(p->sched_buffer);
                p->gsp_buffer = p->sched_buffer = nullptr;
                e = cudaMalloc(&p->buffer, layout.bytes());
                if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan allocation failed: %s", cudaGetErrorString(e));
                if (rc == SMAT_OK)
                    rc = stream_plan_fill(p->stream, narrow, layout, p->buffer, bcsrValuesA, bcsrColIdxA, ctx->sm_count, nullptr, (cudaStream_t)stream);
                if (rc) {
                    free_plan(p);
                    return rc;
                }
                v = narrow;
                *out = p;
                return SMAT_OK;
            }
        }
    }
    if (std::getenv("SMAT_PLAN_DEBUG"))
        fprintf(stderr, "[smat plan] rows %zu blocks %zu: 16-row plan rg %zu steps %d cap %zu balanced %d listed %d; tall %d rg %zu steps %d max/group %d\n",
                brow_end - brow_begin, range_blocks, rg, total_steps, cap, (int)balanced, p->v.sched_list != nullptr, (int)tall, rg_used,
                steps_final, total_and_max[1]);
    // a partial tile per CTA, two for the balanced schedule; then steps, order and blocks; then the stream plan beside them
    const size_t fix_bytes = (balanced ? 2 : 1) * fix_scratch_bytes(ctx->sm_count);
    size_t plan_bytes = 0;
    if (rc == SMAT_OK) {
        // tall: + 64 bytes of per-step words + half a pair's lists
        sz = plan_sizes(nnzb, brow_begin, brow_end, rg_used, (size_t)(steps_final > 0 ? steps_final : 1) * (tall ? 5 + kTallRows / 2 * kTallListBytes / 32 : 1));
        plan_bytes = fix_bytes + sz.steps_bytes + sz.blk_bytes + sz.packed_bytes;
        e = cudaMalloc(&p->buffer, plan_bytes + (stream_too ? layout.bytes() : 0));
        if (e == cudaErrorMemoryAllocation && stream_too) {  // no room for two copies of the blocks: all products with the first
            cudaGetLastError();
            stream_too = false;
            p->wide_from = 0;
            e = cudaMalloc(&p->buffer, plan_bytes);
        }
        if (e != cudaSuccess) rc = fail(SMAT_ERR_CUDA, "plan allocation failed: %s", cudaGetErrorString(e));
    }
    if (rc) {
        free_plan(p);
        return rc;
    }
    char* b = static_cast<char*>(p->buffer);
    p->nnzb = nnzb;
    v.fix_scratch = reinterpret_cast<float*>(b);
    b += fix_bytes;
    v.steps = b;
    v.blk = reinterpret_cast<int*>(b + sz.steps_bytes);
    v.packed = b + sz.steps_bytes + sz.blk_bytes;
    if (stream_too) {  // places without a block stay marked as such (stream_plan_build)
        e = cudaMemsetAsync(const_cast<int*>(v.blk), 0xff, sz.blk_bytes, (cudaStream_t)stream);
        if (e != cudaSuccess) {
            free_plan(p);
            return fail(SMAT_ERR_CUDA, "plan build failed: %s", cudaGetErrorString(e));
        }
    }
    if (tall) {
        // behind the step records, in the same region: the per-step words (only read while the plan is built), then the per-pair lists
        char* wstep = b + (size_t)(steps_final > 0 ? steps_final : 1) * 16;
        v.winfo = wstep + (size_t)(steps_final > 0 ? steps_final : 1) * 64;
        rc = plan_fill_tall_async(bcsrRowPtrA, bcsrColIdxA, K, nnzb, brow_begin, brow_end, rg_used, gsp, const_cast<void*>(v.steps), wstep,
                                  const_cast<void*>(v.winfo), const_cast<int*>(v.blk), (cudaStream_t)stream);
    } else {
        rc = plan_fill_async(bcsrRowPtrA, bcsrColIdxA, K, nnzb, brow_begin, brow_end, rg, gsp, const_cast<void*>(v.steps),
                             const_cast<int*>(v.blk), (cudaStream_t)stream, nullptr, cap);
    }
    if (rc == SMAT_OK && stream_too) {
        rc = stream_plan_fill(p->stream, narrow, layout, static_cast<char*>(p->buffer) + plan_bytes, bcsrValuesA, bcsrColIdxA, ctx->sm_count, &v,
                              (cudaStream_t)stream);
        p->wide = v;
        v = narrow;
    } else if (rc == SMAT_OK) {
        rc = pack_values_async(bcsrRowPtrA, bcsrValuesA, v.blk, const_cast<void*>(v.packed), brow_begin, brow_end, nnzb, (cudaStream_t)stream);
    }
    if (rc) {
        free_plan(p);
        return rc;
    }
    *out = p;
    return SMAT_OK;
}

int smat_plan_set_values(smat_plan* plan, const void* bcsrValuesA, void* stream) {
    clear_error();
    if (!plan || (plan->v.nnzb && !bcsrValuesA)) return fail(SMAT_ERR_BAD_ARG, "NULL argument");
    if ((uintptr_t)bcsrValuesA & 15) return fail(SMAT_ERR_BAD_ARG, "bcsrValuesA must be 16-byte aligned");
    if (int rc = check_plan_device(plan)) return rc;
    if (plan->v.stream) return stream_plan_values(plan->v, bcsrValuesA, nullptr, plan->sms, (cudaStream_t)stream);
    // (the row pointers were checked against the whole arrays' block count, which only bounds what the kernel may read)
    return pack_values_async(plan->v.rowptr, bcsrValuesA, plan->v.blk, const_cast<void*>(plan->v.packed), plan->v.brow_begin,
                             plan->v.brow_end, plan->nnzb, (cudaStream_t)stream);
}

int smat_plan_spmm(const smat_plan* plan, const void* B, void* C, size_t N, void* stream) {
    clear_error();
    if (!plan) return fail(SMAT_ERR_BAD_ARG, "plan is NULL");
    if (N % 8) return fail(SMAT_ERR_BAD_ARG, "N (%zu) must be a multiple of 8", N);
    if (plan->v.brow_end > plan->v.brow_begin && N && (!C || (plan->v.nnzb && !B)))
        return fail(SMAT_ERR_BAD_ARG, "B or C is NULL");
    if (((uintptr_t)B | (uintptr_t)C) & 15) return fail(SMAT_ERR_BAD_ARG, "B and C must be 16-byte aligned");
    if (N >= ((size_t)1 << 31)) return fail(SMAT_ERR_RANGE, "N beyond 2^31");
    if (int rc = check_plan_device(plan)) return rc;
    return launch_spmm(view_for(plan, N), B, C, N, (cudaStream_t)stream);
}

int smat_selftest_plan_wait_timeout(const smat_plan* plan, const void* B, void* C, size_t N, void* stream) {
    clear_error();
    if (!plan || !B || !C) return fail(SMAT_ERR_BAD_ARG, "NULL argument");
    if (N == 0 || N % 8 || N >= ((size_t)1 << 31)) return fail(SMAT_ERR_BAD_ARG, "N (%zu) must be a multiple of 8 below 2^31", N);
    if (((uintptr_t)B | (uintptr_t)C) & 15) return fail(SMAT_ERR_BAD_ARG, "B and C must be 16-byte aligned");
    if (int rc = check_plan_device(plan)) return rc;
    PlanView v = view_for(plan, N);
    if (!v.stream && !v.tall) return fail(SMAT_ERR_BAD_ARG, "this plan's kernel has no such self-test");
    v.selftest = true;
    return launch_spmm(v, B, C, N, (cudaStream_t)stream);
}

int smat_plan_spmm_host(smat_plan* plan, const void* B_host, void* C_host, size_t N, void* stream) {
    clear_error();
    if (!plan) return fail(SMAT_ERR_BAD_ARG, "plan is NULL");
    if (N % 8) return fail(SMAT_ERR_BAD_ARG, "N (%zu) must be a multiple of 8", N);
    if (N >= ((size_t)1 << 31)) return fail(SMAT_ERR_RANGE, "N beyond 2^31");
    const size_t rows = (plan->v.brow_end - plan->v.brow_begin) * 16, K = plan->v.K;
    if (rows == 0 || N == 0) return SMAT_OK;
    if (!B_host || !C_host) return fail(SMAT_ERR_BAD_ARG, "B_host or C_host is NULL");
    if (int rc = check_plan_device(plan)) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    // B comes in by column chunks (rows of the [N][K] array: contiguous), each multiplied for all block-rows as soon as it has
    // arrived.  Where the device can address C_host, the columns of C that a chunk completes go out at once, under the
    // arrival of the next chunks; what is left after the last arrival is one chunk's product and its columns, so the
    // last chunks are half as wide.  Else C has to go out in whole rows: the last chunk is multiplied group range by
    // group range, and the rows that it completes go out under the multiplication of the next range.
    char* const out_view = device_view_of_host(C_host, rows * N * 2);
    const size_t W = N >= 512 ? 256 : (N > 128 ? 128 : N);
    std::vector<size_t> chunk_at;  // first column of every chunk, then N
    for (size_t n0 = 0; n0 < N; n0 += W) {
        chunk_at.push_back(n0);
        const size_t w = N - n0 < W ? N - n0 : W;
        if (out_view && n0 + W >= N && w >= 64) chunk_at.push_back(n0 + (w / 2 + 7) / 8 * 8);
    }
    chunk_at.push_back(N);
    const size_t n_chunks = chunk_at.size() - 1;
    const PlanView& v = view_for(plan, W);
    const size_t n_groups = v.n_groups;
    // ranges of the last chunk: each should still fill the SMs for about one round of work items (shorter launches
    // lose more to partly filled rounds than the overlap of the copy-out wins back); at most 4
    DeviceCtx* ctx = nullptr;
    if (int rc0 = get_device_ctx(&ctx)) return rc0;
    size_t n_ranges = (n_groups * ((W + 127) / 128) + (size_t)ctx->sm_count / 2) / (size_t)ctx->sm_count;
    if (v.stream) n_ranges = n_groups / 16 * ((W + 127) / 128) / (size_t)ctx->sm_count;
    if (v.sched_list || v.balanced) n_ranges = 1;  // such plans balance a launch over all their groups
    if (const char* e = std::getenv("SMAT_HOST_RANGES")) n_ranges = (size_t)std::atoi(e);  // tuning knob
    if (out_view) n_ranges = 1;
    if (n_ranges > 4) n_ranges = 4;
    if (n_ranges > n_groups) n_ranges = n_groups;
    if (n_ranges < 1) n_ranges = 1;
    // staging memory and streams: created on first use and kept with the plan (grown when a later call is wider)
    if (!plan->s_in) {
        SMAT_CUDA_TRY(cudaStreamCreateWithFlags(&plan->s_in, cudaStreamNonBlocking));
        SMAT_CUDA_TRY(cudaStreamCreateWithFlags(&plan->s_out, cudaStreamNonBlocking));
        SMAT_CUDA_TRY(cudaEventCreateWithFlags(&plan->ev_start, cudaEventDisableTiming));
    }
    if (plan->host_B_bytes < N * K * 2 || plan->host_C_bytes < rows * N * 2) {
        SMAT_CUDA_TRY(cudaStreamSynchronize(plan->s_in));
        SMAT_CUDA_TRY(cudaStreamSynchronize(plan->s_out));
        SMAT_CUDA_TRY(cudaStreamSynchronize(s));
        SMAT_CUDA_TRY(cudaFree(plan->host_B));
        SMAT_CUDA_TRY(cudaFree(plan->host_C));
        plan->host_B = plan->host_C = nullptr;
        plan->host_B_bytes = plan->host_C_bytes = 0;
        SMAT_CUDA_TRY(cudaMalloc(&plan->host_B, N * K * 2));
        plan->host_B_bytes = N * K * 2;
        SMAT_CUDA_TRY(cudaMalloc(&plan->host_C, rows * N * 2));
        plan->host_C_bytes = rows * N * 2;
    }
    while (plan->ev_in.size() < n_chunks) {
        cudaEvent_t e = nullptr;
        SMAT_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        plan->ev_in.push_back(e);
    }
    while (plan->ev_done.size() < (out_view ? n_chunks : n_ranges)) {
        cudaEvent_t a = nullptr, b = nullptr;
        SMAT_CUDA_TRY(cudaEventCreateWithFlags(&a, cudaEventDisableTiming));
        plan->ev_done.push_back(a);
        SMAT_CUDA_TRY(cudaEventCreateWithFlags(&b, cudaEventDisableTiming));
        plan->ev_out.push_back(b);
    }
    // the copies start after whatever the caller had put on its stream (e.g. the previous call's use of the buffers)
    SMAT_CUDA_TRY(cudaEventRecord(plan->ev_start, s));
    SMAT_CUDA_TRY(cudaStreamWaitEvent(plan->s_in, plan->ev_start, 0));
    SMAT_CUDA_TRY(cudaStreamWaitEvent(plan->s_out, plan->ev_start, 0));
    const char* Bh = static_cast<const char*>(B_host);
    char* Ch = static_cast<char*>(C_host);
    char* Bd = static_cast<char*>(plan->host_B);
    char* Cd = static_cast<char*>(plan->host_C);
    for (size_t j = 0; j < n_chunks; j++) {
        const size_t n0 = chunk_at[j], w = chunk_at[j + 1] - n0;
        SMAT_CUDA_TRY(cudaMemcpyAsync(Bd + n0 * K * 2, Bh + n0 * K * 2, w * K * 2, cudaMemcpyHostToDevice, plan->s_in));
        SMAT_CUDA_TRY(cudaEventRecord(plan->ev_in[j], plan->s_in));
    }
    for (size_t j = 0; j < n_chunks; j++) {
        const size_t n0 = chunk_at[j], w = chunk_at[j + 1] - n0;
        SMAT_CUDA_TRY(cudaStreamWaitEvent(s, plan->ev_in[j], 0));
        if (out_view) {
            if (int rc = launch_spmm(v, Bd + n0 * K * 2, Cd + n0 * 2, w, s, nullptr, N)) return rc;
            SMAT_CUDA_TRY(cudaEventRecord(plan->ev_done[j], s));
            SMAT_CUDA_TRY(cudaStreamWaitEvent(plan->s_out, plan->ev_done[j], 0));
            const size_t words = rows * w / 8, ctas = (words + 1023) / 1024;
            copy_out_kernel<<<(unsigned)(ctas < 8 ? ctas : 8), 256, 0, plan->s_out>>>(
                reinterpret_cast<const uint4*>(Cd + n0 * 2), reinterpret_cast<uint4*>(out_view + n0 * 2), rows, N / 8, (unsigned)(w / 8));
            count_launch();
            SMAT_CUDA_TRY(cudaGetLastError());
            if (j + 1 == n_chunks) SMAT_CUDA_TRY(cudaEventRecord(plan->ev_out[0], plan->s_out));
            continue;
        }
        if (j + 1 < n_chunks) {
            if (int rc = launch_spmm(v, Bd + n0 * K * 2, Cd + n0 * 2, w, s, nullptr, N)) return rc;
            continue;
        }
        for (size_t r = 0; r < n_ranges; r++) {
            const size_t g0 = n_groups * r / n_ranges, g1 = n_groups * (r + 1) / n_ranges;
            const size_t row0 = g0 * v.rg * 16;
            const size_t row1 = (g1 * v.rg * 16 < rows) ? g1 * v.rg * 16 : rows;
            if (int rc = launch_spmm(v, Bd + n0 * K * 2, Cd + (row0 * N + n0) * 2, w, s, nullptr, N, g0, g1)) return rc;
            SMAT_CUDA_TRY(cudaEventRecord(plan->ev_done[r], s));
            SMAT_CUDA_TRY(cudaStreamWaitEvent(plan->s_out, plan->ev_done[r], 0));
            SMAT_CUDA_TRY(cudaMemcpyAsync(Ch + row0 * N * 2, Cd + row0 * N * 2, (row1 - row0) * N * 2, cudaMemcpyDeviceToHost,
                                          plan->s_out));
            SMAT_CUDA_TRY(cudaEventRecord(plan->ev_out[r], plan->s_out));
        }
    }
    // the caller's stream ends after the last copy out, so that ordering on it covers the whole call
    SMAT_CUDA_TRY(cudaStreamWaitEvent(s, plan->ev_out[out_view ? 0 : n_ranges - 1], 0));
    return SMAT_OK;
}

int smat_plan_info(const smat_plan* plan, int* tall, int* rows_per_item, size_t* steps) {
    clear_error();
    if (!plan) return fail(SMAT_ERR_BAD_ARG, "NULL plan");
    if (tall) *tall = plan->v.tall ? 1 : 0;
    if (rows_per_item) *rows_per_item = (int)plan->v.rg;
    if (steps) *steps = plan->v.total_steps;
    return SMAT_OK;
}

int smat_plan_destroy(smat_plan* plan) {
    clear_error();
    if (!plan) return SMAT_OK;
    if (plan->s_in) {
        cudaStreamSynchronize(plan->s_in);
        cudaStreamSynchronize(plan->s_out);
        cudaStreamDestroy(plan->s_in);
        cudaStreamDestroy(plan->s_out);
        cudaEventDestroy(plan->ev_start);
        for (auto& v : {plan->ev_in, plan->ev_done, plan->ev_out})
            for (cudaEvent_t ev : v) cudaEventDestroy(ev);
        cudaFree(plan->host_B);
        cudaFree(plan->host_C);
    }
    const cudaError_t e = free_plan(plan);
    if (e != cudaSuccess) return fail(SMAT_ERR_CUDA, "cudaFree failed: %s", cudaGetErrorString(e));
    return SMAT_OK;
}

}  // extern "C"
