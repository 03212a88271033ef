// Argument block and launchers of the many-row tensor-core GEMM (gemm_wide.cu) of prompt passes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace hm {

constexpr int WIDE_BLOCK = 128;   // rows of an activation block (the MMA's M)
constexpr int WIDE_ROWS = 2048;   // rows of a pass at most: activations and images of the widest models here stay within 300 MB

// Activation image: [row block of 128][64-element k-block][3 bf16 terms][128 rows][64], rows of 128 bytes with the 128-byte swizzle
// (tc_xpack_store8 with mpad 128 on one block).
__host__ __device__ inline size_t wide_block_bytes(int K) { return (size_t)((K + 63) / 64) * 3 * WIDE_BLOCK * 128; }
inline int wide_blocks(int M) { return (M + WIDE_BLOCK - 1) / WIDE_BLOCK; }

struct WideArgs {
    const uint16_t* W;        // weights as the tensor-core tiles of launch_pack_tc, or of launch_wide_pack_quant:
    int w_terms;              // bf16 terms per weight: 1; 2 or 3, the terms of a tile in a row
    int K, N, M;
    const unsigned char* xp;  // activation image
    int epi;                  // EPI_STORE (residual, next image), EPI_SWIGLU (image), EPI_QKV_ROPE
    const float* bias;        // EPI_QKV_ROPE, optional
    const float* resid;       // EPI_STORE, optional: [M][ldy]
    float* y;                 // EPI_STORE: [M][ldy]; EPI_QKV_ROPE: queries
    int ldy;
    unsigned char* xp_out;    // EPI_SWIGLU: image of the activations; EPI_STORE, optional: image of y * next_norm_w
    const float* next_norm_w;
    // Sums of squares, f32 of bf16 models and f64 of quantised ones (w_terms > 1), as either path is specified (src/hf/emitter_quant.rs:713-791):
    void* ss_out;             // EPI_STORE with xp_out: [N / 128][ss_ld] of y
    const void* ss_in;        // optional: [ss_parts][ss_ld] of the rows, whose RMSNorm factor scales the accumulators
    int ss_parts, ss_ld;
    float eps;
    // EPI_QKV_ROPE
    int q_dim, kv_dim, hd, has_qk_norm;
    const float *q_norm_w, *k_norm_w, *rope_cos, *rope_sin;
    const int32_t *row_pos, *row_seq;
    KvDesc kv;
    float* part;              // partial tiles (wide_split)
    int* err_flag;
    // filled in by launch_gemm_wide
    int kblocks, nblocks, tiles, row_blocks, split, kb_per, units;
};

// How a projection over M rows splits its contraction, and the scratch for its partial tiles.
struct WideSplit {
    int split;
    size_t part_floats;
};
WideSplit wide_split(int M, int K, int N, int w_terms, int epi, int sm_count);
// One launch, or two: the product, and what follows it (see gemm_wide.cu).
cudaError_t launch_gemm_wide(const WideArgs& a, int sm_count, cudaStream_t st, bool pdl, int* launches);
// Q8_0 / Q4_0 blocks [n_rows][K / 32] -> tiles [ceil(N / 128)][K / 64][terms][128][64] of bf16 terms whose sum is the weight exactly (f16
// scale times code: 19 bits, three terms; 15 bits, two).  Rows land at n_off + n, or interleaved 64 / 64 per block of 128 when
// interleave_which is 0 (gate) or 1 (up).  K a multiple of 64.
inline int wide_quant_terms(bool q4) { return q4 ? 2 : 3; }
cudaError_t launch_wide_pack_quant(const uint8_t* blocks, int n_rows, int K, bool q4, uint16_t* dst, int n_off, int interleave_which, cudaStream_t st);
// f32 rows -> activation image; folds an RMSNorm (weight norm_w, squares summed in f64 on request) when norm_w is not null.
cudaError_t launch_wide_pack(const float* x, int ldx, int M, int K, const float* norm_w, float eps, bool f64, unsigned char* xp, cudaStream_t st, bool pdl);

}  // namespace hm
