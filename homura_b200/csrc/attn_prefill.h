// Attention of prompt rows over the paged cache (attn_prefill.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace hm {

constexpr int PREFILL_TILE = 64;   // rows of a query tile, and keys of a staged block

// One query tile: rows [row0, row0 + rows) of the pass, consecutive tokens of one sequence from position pos0 on; the sequence's staged
// blocks start at block0.
struct PrefillTile {
    int32_t row0, rows, pos0, block0;
};
// One staged block: tokens [key0, key0 + PREFILL_TILE) of sequence seq, of which the first `valid` exist.
struct PrefillBlock {
    int32_t seq, key0, valid, unused;
};

struct PrefillArgs {
    KvDesc kv;
    int heads;
    float scale;
    const float* q;               // [M][heads * hd]
    unsigned char* staged;        // prefill_staged_bytes of all blocks
    const PrefillTile* tiles;
    const PrefillBlock* blocks;
    int n_tiles, n_blocks;
    unsigned char* xp_out;        // the O projection's activation image (gemm_wide.h)
    size_t xp_block;
    int* err_flag;
};

// Bytes of one staged block: keys and values of every KV head as the MMA operands' bf16 terms (one on bf16 pages, three on f32 pages).
inline size_t prefill_block_bytes(int kv_heads, int hd, bool bf16) { return (size_t)kv_heads * 2 * (bf16 ? 1 : 3) * PREFILL_TILE * hd * 2; }
// Two launches: pages -> staged blocks, then the attention.
cudaError_t launch_attn_prefill(const PrefillArgs& a, cudaStream_t st, bool pdl, int* launches);

}  // namespace hm
