// The stream kernel (spmm_stream_sm100.cu): arguments of a launch.
#pragma once
#include <cuda_fp16.h>

#include <vector>

#include "smat_internal.h"

namespace smat {

struct StreamArgs {
    const void* vals;      // value blocks: as the boundary stores them, or (plan) in fragment order
    const int* rowptr;     // no plan: row pointers of the whole matrix
    const int* colidx;     // no plan: element columns; plan: block-columns of the plan's blocks, -1 = skip
    // plan: every piece, {block-row, first block, last block + 1, 1 + slot of a piece of a long block-row or 0};
    // no plan: {block-row, first block, last block + 1, slot} of the pieces that follow the first of a long block-row
    const uint4* pieces;
    const int2* slots;     // per slot {first slot of its block-row, pieces of the block-row}
    const int* row_slot;   // no plan: first slot of a long block-row
    const int* long_rows;  // no plan: number of entries of `pieces`; null = no block-row is longer than `chunk`
    const void* B;         // [N][K], or slabs [K / 16][N][16]
    __half* C;
    float4* partial;       // partial tiles of the pieces of long block-rows
    int* counters;         // arrivals per long block-row (first slot) and tile, zero between launches
    int* status;
    size_t ldc;
    int n_pieces, n_tiles, tile_cols, N, K, brow_begin, brow_end, nnzb, chunk, sm_count;
    float ahead;            // plan: blocks of a warp, on average, where its first ones are prefetched early; else 0
    long long wait_cycles;  // limit of a wait
    unsigned lost_bytes;    // bytes that a wait expects beyond those that are copied: 0, but for a self-test
};

struct StreamShape {
    int nt = 128;       // columns of C per warp: 8, 16, 32, 64, 128
    int w = 1;          // warps that share a piece: 1, 2, 4, 8
    int chunk = 128;    // most blocks of a piece
    bool slab = false;  // B rewritten as slabs first
};
StreamShape stream_shape(size_t N, size_t rows, size_t nnzb, size_t K, int sm_count, bool plan);
bool stream_for_call(size_t N, size_t rows, size_t nnzb, size_t K, int sm_count);
double stream_estimate_us(size_t N, size_t rows, size_t nnzb, size_t K, int sm_count, bool plan);
// Columns a plan made for N_hint columns multiplies in one pass, and its estimate for N columns.
inline size_t stream_pass_columns(size_t N_hint) { return (N_hint + 127) / 128 * 128; }
double stream_passes_us(size_t N, size_t N_hint, size_t rows, size_t nnzb, size_t K, int sm_count);

// What a plan for this kernel holds (PlanView::stream): the values in fragment order, the block-columns, the pieces.
struct StreamPlan {
    StreamArgs args = {};         // pieces, slots, counters, partial, colidx, vals
    void* slabs = nullptr;
    size_t n_cap = 0, first = 0;  // columns that scratch and slabs hold; position of the plan's first block in the boundary's arrays
    std::vector<int> row_piece;   // first piece of every block-row
    // beside the plan of a tcgen05 kernel (null: none): its copy of the blocks, and every block's place there
    void* walk = nullptr;
    int* pos = nullptr;
};
// Its pieces, and the device memory that it takes (bytes() of it, 256-byte aligned).  h_rowptr: the plan's row pointers on the
// host (block-rows brow_begin .. brow_end), checked to be monotone.  beside: kept beside the plan of a tcgen05 kernel.
struct StreamLayout {
    std::vector<uint4> pieces;
    std::vector<int2> slots;
    std::vector<int> row_piece;
    size_t n_cap = 0, first = 0;
    size_t pieces_bytes = 0, slots_bytes = 0, counter_bytes = 0, partial_bytes = 0, cols_bytes = 0, pos_bytes = 0, packed_bytes = 0, slab_bytes = 0;
    size_t bytes() const { return pieces_bytes + slots_bytes + counter_bytes + partial_bytes + cols_bytes + pos_bytes + packed_bytes + slab_bytes; }
};
StreamLayout stream_plan_layout(const int* h_rowptr, size_t rows, size_t K, size_t N_hint, int sm_count, bool beside);
// v: the range, K and blocks of the plan; becomes the stream plan's view.  walk: the plan beside it (or null), its walk order
// filled (blk -1 where it holds no block); its copy of the blocks is filled here.
int stream_plan_fill(StreamPlan& sp, PlanView& v, StreamLayout& l, void* memory, const void* vals, const int* colidx, int sm_count,
                     const PlanView* walk, cudaStream_t stream);
// New values into an existing plan (colidx null) or values and columns into a new one; into the plan beside it as well.
int stream_plan_values(const PlanView& v, const void* vals, const int* colidx, int sm_count, cudaStream_t stream);
int launch_stream(const PlanView& v, const void* B, void* C, size_t N, cudaStream_t stream, const DeviceCtx* ctx, size_t ldc,
                  size_t row_begin, size_t row_end);

// One product without a plan, in `scratch` of stream_call_bytes() bytes (256-byte aligned).
size_t stream_call_bytes(const StreamShape& s, size_t N, size_t rows, size_t nnzb, size_t K);
int stream_call(const StreamShape& s, const void* vals, const int* rowptr, const int* colidx, const void* B, void* C, size_t N, size_t K,
                size_t nnzb, size_t brow_begin, size_t brow_end, void* scratch, const DeviceCtx* ctx, cudaStream_t stream);

}  // namespace smat
