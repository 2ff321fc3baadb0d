// Device helpers of the attention kernels: tile rows, index translation and the exact e4m3 -> bf16 conversion.
#pragma once
#include "defs.h"
#include "ptx.cuh"

namespace dsa {

// ------------------------------------------------------------------ tile row -> (query row, head)
// Tile row r of a work item is head head_block * 128 + r of query row q_row, or, for an item that stacks
// the query rows of one sequence that share an index list, head r % H of query row q_row + r / H.
struct RowMap {
    int q_row, head;
    bool live;
};
__device__ __forceinline__ RowMap map_row(const dsa_v32_work_info& w, int row, int H) {
    RowMap m;
    if (w.stacked_rows > 1) {
        const int sub = row / H;
        m.q_row = w.q_row + sub;
        m.head = row - sub * H;
        m.live = sub < w.stacked_rows;
    } else {
        m.q_row = w.q_row;
        m.head = w.head_block * kHeadsPerBlock + row;
        m.live = m.head < H;
    }
    return m;
}

// ------------------------------------------------------------------ index translation
// Top-k slot value -> physical cache row, or -1 when the slot is padding / unusable.  Split in two so
// the loader warps can issue the block-table load of one tile and finish the arithmetic tiles later:
//   block_of(idx)        issues the block-table load (0 when there is nothing to load)
//   row_of(idx, phys)    the physical row from the loaded block number
__device__ __forceinline__ int block_of(int idx, int seq, const AttnParams& p) {
    if (idx < 0 || p.block_table == nullptr) return 0;
    const int blk = p.page_shift >= 0 ? (idx >> p.page_shift) : idx / p.page_block_size;
    if (blk >= p.block_table_stride) return -1;
    return __ldg(p.block_table + (size_t)seq * p.block_table_stride + blk);
}
__device__ __forceinline__ int row_of(int idx, int phys, int seq, const AttnParams& p) {
    if (idx < 0) return -1;
    long long row;
    if (p.block_table != nullptr) {
        if (phys < 0) return -1;
        const int in_page = p.page_shift >= 0 ? (idx & (p.page_block_size - 1)) : idx % p.page_block_size;
        row = (long long)phys * p.page_block_size + in_page;
    } else {
        row = (long long)seq * p.kv_batch_stride_rows + idx;
    }
    if (row < 0 || row >= p.num_kv_rows) return -1;
    return (int)row;
}
__device__ __forceinline__ int translate_row(int idx, int seq, const AttnParams& p) {
    return row_of(idx, block_of(idx, seq, p), seq, p);
}

// ------------------------------------------------------------------ e4m3 -> bf16, exact, two at a time
// Input: the two e4m3 bytes in the high byte of each 16-bit half.  Moving the 7 magnitude bits down
// by 4 puts the 4 exponent bits and 3 mantissa bits where bf16 keeps them; read as bf16 that number
// is the e4m3 value times 2^-120 (normal and subnormal codes alike), so one exact multiply by 2^120
// finishes the conversion without going through the conversion unit.  (The e4m3 NaN, 0x7F or 0xFF, becomes +-480: the caller
// looks for it with nan_codes.)
__device__ __forceinline__ uint32_t nan_codes(uint32_t bytes) { return (bytes & 0x7F7F7F7Fu) + 0x01010101u; }   // bit 7 of each byte that is one
__device__ __forceinline__ uint32_t e4m3x2_to_bf16x2(uint32_t hi_bytes) {
    const uint32_t y = (hi_bytes & 0x80008000u) | ((hi_bytes >> 4) & 0x07F007F0u);
    uint32_t z;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(z) : "r"(y), "r"(0x7B807B80u));
    return z;
}

}  // namespace dsa
