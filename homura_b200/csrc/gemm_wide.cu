// Many-row tensor-core GEMM of prompt passes: y[M,N] = x[M,K] @ W for 65..2048 activation rows, bf16 weights, f32 activations and
// f32 accumulation (src/graph_builder/emit_linalg.rs:1928-2008).
//
// The 64-row GEMM (gemm_tc.cu) is bound by the weights it streams per 64 rows; a prompt pass has rows enough that the
// tensor pipe is the bound, so the roles are the other way round:
//   * one unit = 128 rows (the MMA's M) x 256 output features (its N); an SM keeps one CTA, which walks its units
//     (persistent, static round robin) without draining the pipeline in between.
//   * the f32 activations come as three bf16 terms (x = hi + mid + lo to 2^-24), three MMAs of M128 N256 K16 per k-step, all into
//     one accumulator.  Weights: 32 KB per 64-element k-block, shared by the three terms; activations: 16 KB per term.  Two rings
//     (three weight slots, six term slots: 192 KB) so that a slot is refilled as soon as its own MMAs have read it.
//   * the tensor core truncates when it adds to the accumulator, an error that grows with the length of the chain (2e-8 of the result
//     per addition at the result's magnitude).  Accumulators therefore cover CHUNK k-blocks only, the small terms of all of them first; two of them (256 TMEM columns each) alternate,
//     and eight warps add the finished one to f32 registers (round to nearest) while the other is being filled.  A thread owns
//     one row and 128 consecutive features, so that norms, rotation and gating need no exchange between threads.
//   * Q8_0 and Q4_0 weights (f16 scale times code: 19 and 15 bits) come as three and two bf16 terms, exactly, and take the six and five
//     products that reach 2^-24; a weight tile then serves the activation terms that it meets, the small products first.
//   * the gated activations of a whole contraction leave from the same registers.  Everything else goes as f32 partial tiles to scratch
//     (the L2) and a second launch (wide_finish_kernel) adds the parts of a split contraction in their order and does the epilogue, a
//     warp per row of 128 features: the outputs of a unit that no other unit of its CTA follows would otherwise leave at the pace of
//     eight warps (15 us for 128 x 256 residuals, images and sums of squares; 3 us for the partial tile).
// Measured: gate/up of 2048 rows (K 1536, N 17920) 287 us = 1.18 PFLOP/s of bf16 products, down (K 8960, N 1536) 119 + 14 us, where the
// 64-row launches took 32 x 15.0 and 32 x 13.2 us; a prompt of 1999 tokens on the 0.5 B stack 52.1 -> 9.2 ms,
// 1021 tokens on TinyLlama Q8_0 60.1 -> 12.1 ms and Q4_0 66.8 -> 10.7 ms (64-row launches on digit planes and integer MMAs before).  By the sizes (no counter
// was taken) the traffic between L2 and shared memory bounds it (80 KB per k-block and SM), and the read-back of the accumulators: one per two k-blocks costs
// 12 % against one per four, which leaves 1.8 times the error.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "gemm_wide.h"
#include "launch_attrs.h"
#include "mbarrier.cuh"

namespace hm {
namespace {

constexpr int BK = 64;
constexpr int WB_TILE = 128 * BK * 2;        // one block of 128 features
constexpr int W_SLOT = 2 * WB_TILE;          // 256 features x 64 k
constexpr int X_SLOT = WIDE_BLOCK * BK * 2;  // one term of 128 rows x 64 k
constexpr int W_SLOTS = 3, X_SLOTS = 6;
// k-blocks per accumulator
template <int WT>
constexpr int CHUNK = WT == 1 ? 2 : 1;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr int STAGE = 32 * 32 * 4;           // an epilogue warp's 32 rows x 32 columns on their way to or from global memory
constexpr size_t SMEM = (size_t)W_SLOTS * W_SLOT + (size_t)X_SLOTS * X_SLOT + (size_t)EPI_WARPS * STAGE + 1024;

__device__ __forceinline__ uint64_t desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t (&r)[32], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr));
}
// Names the registers, so that no use of them moves in front of the wait.
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :: "memory");
}

struct WideShared {
    uint64_t wfull[W_SLOTS], wempty[W_SLOTS], xfull[X_SLOTS], xempty[X_SLOTS], afull[2], aempty[2], done;
    uint32_t tmem;
    volatile int abort_flag;
};

// Units that run at the same time should share operands: groups of eight row blocks, within a group rows fastest, then features, then
// the parts of a split contraction (148 units in flight: 8 x 48 KB of rows and 18 x 32 KB of weights per k-block).
constexpr int GROUP = 8;
struct Unit {
    int rb, tile, split, kb0, kb1;
};
__device__ __forceinline__ Unit unit_at(const WideArgs& a, int u) {
    Unit r;
    const int per = GROUP * a.tiles * a.split, g = u / per, rows = min(GROUP, a.row_blocks - g * GROUP);
    u -= g * per;
    r.rb = g * GROUP + u % rows;
    u /= rows;
    r.tile = u % a.tiles;
    r.split = u / a.tiles;
    r.kb0 = r.split * a.kb_per;
    r.kb1 = min(a.kblocks, r.kb0 + a.kb_per);
    return r;
}

// Sums of squares: f32, or f64 for quantised weights (Q).
template <bool Q>
using Sum = typename std::conditional<Q, double, float>::type;
template <typename T>
__device__ __forceinline__ T squares(const float4& v) { return fma((T)v.x, (T)v.x, fma((T)v.y, (T)v.y, fma((T)v.z, (T)v.z, (T)v.w * (T)v.w))); }
template <typename T>
__device__ __forceinline__ T lanes_sum(T v, int lanes) {  // over groups of `lanes` lanes
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        if (o < lanes) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <typename T>
__device__ __forceinline__ float norm_factor(T sum, int n, float eps) { return 1.0f / sqrtf((float)(sum / (T)n) + eps); }
// RMSNorm factor of row m from the sums of squares that the launch in front left.
template <typename T>
__device__ __forceinline__ float row_factor(const WideArgs& a, int m) {
    if (!a.ss_in) return 1.0f;
    T s = 0;
    for (int p = 0; p < a.ss_parts; ++p) s += __ldcg(static_cast<const T*>(a.ss_in) + (size_t)p * a.ss_ld + m);
    return norm_factor(s, a.K, a.eps);
}

// Partial tile of a unit: [32 pieces of four columns][256 threads of the epilogue warps] float4.
__device__ __forceinline__ float4* part_at(const WideArgs& a, int split, int rb, int tile) {
    return reinterpret_cast<float4*>(a.part) + (((size_t)split * a.tiles + tile) * a.row_blocks + rb) * (32 * EPI_WARPS * 32);
}

// A warp's staging tile [32 rows][8 pieces of 4 floats], pieces XOR-swizzled by the row: free of bank conflicts both ways.
__device__ __forceinline__ float4& piece(float* st, int row, int c) { return reinterpret_cast<float4*>(st)[row * 8 + (c ^ (row & 7))]; }
__device__ __forceinline__ void stage_put(float* st, int lane, const float* v) {
#pragma unroll
    for (int c = 0; c < 8; ++c) piece(st, lane, c) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    __syncwarp();
}

// 32 staged columns -> the three-term image, columns k0 .. k0 + 31: lanes cover eight rows of four 16-byte pieces.  Rows [0, n) exist.
__device__ __forceinline__ void stage_to_image(float* st, unsigned char* xp, int row0, int k0, int lane, int n) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = i * 8 + (lane >> 2), c = lane & 3;
        const float4 p = piece(st, r, 2 * c), q = piece(st, r, 2 * c + 1);
        const float v[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
        if (r < n) tc_xpack_store8(xp, WIDE_BLOCK, row0 + r, k0 + 8 * c, v);
    }
    __syncwarp();
}

// block = 64 gate features, then the 64 matching up features
__device__ __forceinline__ void epi_swiglu(const WideArgs& a, float (&acc)[128], float* st, int rb, int row0, int lane, int n, int nblk) {
    unsigned char* xp = a.xp_out + (size_t)rb * wide_block_bytes(a.N / 2);
#pragma unroll
    for (int j = 0; j < 64; j += 32) {
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[j + e] = (acc[j + e] / (1.0f + expf(-acc[j + e]))) * acc[64 + j + e];
        stage_put(st, lane, acc + j);
        stage_to_image(st, xp, row0, nblk * 64 + j, lane, n);
    }
}

// GLU: gated activations of unsplit contractions; else partial tiles.  WT: terms of a weight; term w meets the activation terms 2 - w .. 0.
template <bool GLU, int WT>
__global__ void __launch_bounds__(THREADS, 1) gemm_wide_kernel(const WideArgs a) {
    extern __shared__ __align__(1024) unsigned char dsm[];
    __shared__ WideShared sh;
    unsigned char* wring = dsm + ((1024u - (s32(dsm) & 1023u)) & 1023u);  // swizzle atoms need 1024-byte alignment
    unsigned char* xring = wring + (size_t)W_SLOTS * W_SLOT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < W_SLOTS; ++s) { mb_init(&sh.wfull[s], 1); mb_init(&sh.wempty[s], 1); }
        for (int s = 0; s < X_SLOTS; ++s) { mb_init(&sh.xfull[s], 1); mb_init(&sh.xempty[s], 1); }
        for (int s = 0; s < 2; ++s) { mb_init(&sh.afull[s], 1); mb_init(&sh.aempty[s], EPI_WARPS); }
        mb_init(&sh.done, 1);
        sh.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(s32(&sh.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh.tmem;
    pdl_launch_dependents();
    if (warp != 0) pdl_wait();

    uint32_t w_issued = 0, x_issued = 0;
    if (warp == 0) {
        if (lane == 0) {
            const unsigned char* W = reinterpret_cast<const unsigned char*>(a.W);
            const size_t nb_bytes = (size_t)a.kblocks * WT * WB_TILE, rb_bytes = (size_t)a.kblocks * 3 * X_SLOT;
            uint32_t wi = 0, xi = 0;  // slots used so far
            auto load_w = [&](const Unit& t, int i, uint32_t s) {  // the unit's i-th weight tile, the small terms of a k-block first
                const bool two = 2 * t.tile + 1 < a.nblocks;
                const unsigned char* src = W + (size_t)(2 * t.tile) * nb_bytes + ((size_t)(t.kb0 + i / WT) * WT + (WT - 1 - i % WT)) * WB_TILE;
                unsigned char* dst = wring + (size_t)s * W_SLOT;
                mb_expect_tx(&sh.wfull[s], two ? W_SLOT : WB_TILE);
                bulk_copy(dst, src, WB_TILE, &sh.wfull[s]);
                if (two) bulk_copy(dst + WB_TILE, src + nb_bytes, WB_TILE, &sh.wfull[s]);
            };
            // weights do not depend on the launch in front: the first slots are filled before its end
            const Unit first = unit_at(a, blockIdx.x);
            const uint32_t ahead = min(W_SLOTS, (first.kb1 - first.kb0) * WT);
            for (uint32_t i = 0; i < ahead; ++i) load_w(first, (int)i, i);
            pdl_wait();
            bool ok = true;
            for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
                const Unit t = unit_at(a, u);
                const unsigned char* x0 = a.xp + (size_t)t.rb * rb_bytes;
                auto load_x = [&](int kb, int term) {
                    const uint32_t x = xi % X_SLOTS;
                    if (xi >= X_SLOTS) ok = mb_wait(&sh.xempty[x], ((xi / X_SLOTS) & 1u) ^ 1u, a.err_flag, &sh.abort_flag);
                    if (!ok) return;
                    mb_expect_tx(&sh.xfull[x], X_SLOT);
                    bulk_copy(xring + (size_t)x * X_SLOT, x0 + ((size_t)kb * 3 + term) * X_SLOT, X_SLOT, &sh.xfull[x]);
                    ++xi;
                };
                for (int i = 0; i < (t.kb1 - t.kb0) * WT && ok; ++i, ++wi) {
                    const uint32_t s = wi % W_SLOTS;
                    if (wi >= W_SLOTS) ok = mb_wait(&sh.wempty[s], ((wi / W_SLOTS) & 1u) ^ 1u, a.err_flag, &sh.abort_flag);
                    if (!ok) break;
                    if (wi >= ahead) load_w(t, i, s);
                    const int kb = t.kb0 + i / WT;
                    if (WT == 1) {  // the leading terms of a chunk behind the others of all its k-blocks
                        for (int term = 2; term > 0 && ok; --term) load_x(kb, term);
                        if (i % CHUNK<WT> == CHUNK<WT> - 1 || kb + 1 == t.kb1)
                            for (int k = kb - i % CHUNK<WT>; k <= kb && ok; ++k) load_x(k, 0);
                    } else {  // the activation terms that this weight term is the first to meet
                        const int w = WT - 1 - i % WT;
                        for (int term = 2 - w; term >= (w == WT - 1 ? 0 : 2 - w) && ok; --term) load_x(kb, term);
                    }
                }
            }
            w_issued = max(wi, ahead);
            x_issued = xi;
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);  // D f32, A and B bf16 K-major, M 128, N 256
            uint32_t wi = 0, xi = 0, ci = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
                const Unit t = unit_at(a, u);
                for (int kc = t.kb0; kc < t.kb1 && ok; kc += CHUNK<WT>, ++ci) {
                    const uint32_t buf = ci & 1u, d = tmem + buf * 256u;
                    if (ci >= 2) ok = mb_wait(&sh.aempty[buf], ((ci >> 1) & 1u) ^ 1u, a.err_flag, &sh.abort_flag);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t more = 0;
                    const int ke = min(t.kb1, kc + CHUNK<WT>);
                    if (WT == 1) {
                        auto product = [&](uint32_t s) {  // the next activation term with weight slot s
                            const uint32_t x = xi % X_SLOTS, wa = s32(wring + (size_t)s * W_SLOT), xa = s32(xring + (size_t)x * X_SLOT);
                            ok = ok && mb_wait(&sh.xfull[x], (xi / X_SLOTS) & 1u, a.err_flag, &sh.abort_flag);
                            if (!ok) return;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                            for (int ks = 0; ks < BK / 16; ++ks) {
                                mma_f16(d, desc_sw128(xa + ks * 32), desc_sw128(wa + ks * 32), idesc, more);
                                more = 1;
                            }
                            mma_commit(&sh.xempty[x]);
                            ++xi;
                        };
                        // The small terms of the chunk while the accumulator is small, the leading ones last: only their additions
                        // truncate at the magnitude of the result.
                        for (int k = kc; k < ke && ok; ++k) {
                            const uint32_t s = (wi + (k - kc)) % W_SLOTS;
                            ok = mb_wait(&sh.wfull[s], ((wi + (k - kc)) / W_SLOTS) & 1u, a.err_flag, &sh.abort_flag);
                            product(s);
                            product(s);
                        }
                        for (int k = kc; k < ke && ok; ++k, ++wi) {
                            product(wi % W_SLOTS);
                            if (ok) mma_commit(&sh.wempty[wi % W_SLOTS]);
                        }
                    }
                    for (int kb = kc; WT > 1 && kb < ke && ok; ++kb, xi += 3) {
#pragma unroll
                        for (int w = WT - 1; w >= 0; --w, ++wi) {
                            const uint32_t s = wi % W_SLOTS;
                            ok = ok && mb_wait(&sh.wfull[s], (wi / W_SLOTS) & 1u, a.err_flag, &sh.abort_flag);
                            const uint32_t wa = s32(wring + (size_t)s * W_SLOT);
#pragma unroll
                            for (int term = 2 - w; term >= 0; --term) {  // small products first
                                // place of the term among the three of this k-block: in the order of their first use
                                const uint32_t xn = xi + (WT == 2 ? (term == 2 ? 2 : 1 - term) : term), x = xn % X_SLOTS;
                                if (w == WT - 1 || term == 2 - w) ok = ok && mb_wait(&sh.xfull[x], (xn / X_SLOTS) & 1u, a.err_flag, &sh.abort_flag);
                                if (!ok) break;
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                                const uint32_t xa = s32(xring + (size_t)x * X_SLOT);
#pragma unroll
                                for (int ks = 0; ks < BK / 16; ++ks) {
                                    mma_f16(d, desc_sw128(xa + ks * 32), desc_sw128(wa + ks * 32), idesc, more);
                                    more = 1;
                                }
                                if (w == 0) mma_commit(&sh.xempty[x]);
                            }
                            if (ok) mma_commit(&sh.wempty[s]);
                        }
                    }
                    if (ok) mma_commit(&sh.afull[buf]);
                }
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;  // a warp reads its own quarter of the TMEM lanes
        const int ml = quarter * 32 + lane, et = tid - 64;
        float* st = reinterpret_cast<float*>(xring + (size_t)X_SLOTS * X_SLOT + (size_t)(warp - 2) * STAGE);
        const uint32_t tbase = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 128);
        uint32_t ci = 0;
        float acc[128];
        for (int u = blockIdx.x; u < a.units; u += gridDim.x) {
            const Unit t = unit_at(a, u);
            const int m = t.rb * WIDE_BLOCK + ml, nblk = 2 * t.tile + half;
            float inv = 1.0f;
            if (GLU && m < a.M) inv = row_factor<Sum<(WT > 1)>>(a, m);
#pragma unroll
            for (int j = 0; j < 128; ++j) acc[j] = 0.f;
            bool ok = true;
            for (int kc = t.kb0; kc < t.kb1; kc += CHUNK<WT>, ++ci) {
                const uint32_t buf = ci & 1u;
                ok = __all_sync(0xffffffffu, mb_wait(&sh.afull[buf], (ci >> 1) & 1u, a.err_flag, &sh.abort_flag));
                if (!ok) continue;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 128; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(r, tbase + buf * 256u + c);
                    tmem_wait(r);
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[c + j] += __uint_as_float(r[j]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mb_arrive(&sh.aempty[buf]);
            }
            const int n = min(32, a.M - (t.rb * WIDE_BLOCK + quarter * 32));  // this warp's rows that exist
            if (n <= 0 || nblk >= a.nblocks) continue;
            if (GLU) {
#pragma unroll
                for (int j = 0; j < 128; ++j) acc[j] *= inv;
                epi_swiglu(a, acc, st, t.rb, quarter * 32, lane, n, nblk);
            } else {
                float4* part = part_at(a, t.split, t.rb, t.tile) + et;
#pragma unroll
                for (int j = 0; j < 32; ++j) __stcg(part + j * (EPI_WARPS * 32), make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (sh.abort_flag) {  // a wait ran out: the copies and MMAs in flight end before the CTA does and its accumulators are freed
        if (tid == 0) {
            mb_land_ring(sh.wfull, w_issued, W_SLOTS);
            mb_land_ring(sh.xfull, x_issued, X_SLOTS);
        } else if (tid == 32) {
            mma_commit(&sh.done);
            mb_land(&sh.done, 0);
        }
        __syncthreads();
    }
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Sums the parts of 32 rows x 128 features and finishes them, four rows per warp; grid (blocks of 128 features, blocks of 32 rows).
// Latency is all there is to it: whatever does not depend on the sums is requested with them, for all rows of the warp.
// S: parts at most (what their sum holds in registers decides how many CTAs share an SM).  Q: quantised weights, whose norms sum in f64:
// 256 tokens on TinyLlama Q8_0 3.85 -> 3.92 ms (bf16 models would pay up to 4 %); error of all logits of a prompt, mean of four, with f32 sums,
// f64 sums and on the 64-row kernels: TinyLlama Q8_0 9.72e-7, 9.70e-7, 11.9e-7, Q4_0 9.24, 9.12, 11.8; 0.5 B stack in Q8_0 10.3, 10.2, 10.2.
constexpr int FIN_WARPS = 8, FIN_ROWS = 32 / FIN_WARPS, FIN_LD = 132;
template <int EPI, int HD, int S, bool Q>
__global__ void __launch_bounds__(FIN_WARPS * 32) wide_finish_kernel(const WideArgs a) {
    using T = Sum<Q>;
    __shared__ __align__(16) float tile[32 * FIN_LD];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nblk = blockIdx.x, rb = blockIdx.y >> 2, quarter = blockIdx.y & 3, n0 = nblk * 128, c = lane * 4;  // four columns of a row
    const int row0 = quarter * 32, m0 = rb * WIDE_BLOCK + row0, n = min(32, a.M - m0);
    const int nh = (n0 + c) / HD * HD, d = (n0 + c) - nh;  // QKV: this lane's head and first dim
    const bool ok = nh < a.N, is_q = nh < a.q_dim, is_k = !is_q && nh < a.q_dim + a.kv_dim;
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f), bias = w;
    if (EPI == EPI_STORE && a.xp_out) w = __ldg(reinterpret_cast<const float4*>(a.next_norm_w + n0 + c));
    if (EPI == EPI_QKV_ROPE && a.bias && ok) bias = __ldg(reinterpret_cast<const float4*>(a.bias + n0 + c));
    if (EPI == EPI_QKV_ROPE && a.has_qk_norm && (is_q || is_k)) w = __ldg(reinterpret_cast<const float4*>((is_q ? a.q_norm_w : a.k_norm_w) + d));
    int pos[FIN_ROWS], page[FIN_ROWS];  // (tables of the call: final before its first launch)
    float4 cs[FIN_ROWS], sn[FIN_ROWS];
    if (EPI == EPI_QKV_ROPE) {
#pragma unroll
        for (int i = 0; i < FIN_ROWS; ++i) {
            const int m = min(m0 + warp * FIN_ROWS + i, a.M - 1);
            pos[i] = a.row_pos[m];
            page[i] = a.row_seq[m];
        }
#pragma unroll
        for (int i = 0; i < FIN_ROWS; ++i) {
            page[i] = a.kv.page_table[(size_t)page[i] * a.kv.max_pages + pos[i] / a.kv.page_tokens];
            cs[i] = __ldg(reinterpret_cast<const float4*>(a.rope_cos + (size_t)pos[i] * HD + d));
            sn[i] = __ldg(reinterpret_cast<const float4*>(a.rope_sin + (size_t)pos[i] * HD + d));
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    float4 x[FIN_ROWS];
    float inv[FIN_ROWS];
    T sums[FIN_ROWS];
#pragma unroll
    for (int i = 0; i < FIN_ROWS; ++i) {
        const int m = min(m0 + warp * FIN_ROWS + i, a.M - 1);
        sums[i] = 0;
        if (EPI != EPI_STORE && a.ss_in && lane < a.ss_parts) sums[i] = __ldcg(static_cast<const T*>(a.ss_in) + (size_t)lane * a.ss_ld + m);
        if (EPI == EPI_STORE) x[i] = a.resid ? ld_cg_f32x4(a.resid + (size_t)m * a.ldy + n0 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    {
        // the unit's epilogue warp of this quarter of the rows and half of the features; here a lane per row, 16 columns per warp
        constexpr int NJ = 32 / FIN_WARPS;
        const size_t step = (size_t)a.tiles * a.row_blocks * (32 * EPI_WARPS * 32);
        const float4* src = part_at(a, 0, rb, nblk >> 1) + (size_t)warp * NJ * (EPI_WARPS * 32) + ((nblk & 1) * 4 + ((quarter + 2) & 3)) * 32 + lane;
        float4 v[S][NJ];
#pragma unroll
        for (int p = 0; p < S; ++p)
            if (p < a.split)
#pragma unroll
                for (int j = 0; j < NJ; ++j) v[p][j] = __ldcg(src + p * step + j * (EPI_WARPS * 32));
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            float4 s = v[0][j];
#pragma unroll
            for (int p = 1; p < S; ++p)
                if (p < a.split) { s.x += v[p][j].x; s.y += v[p][j].y; s.z += v[p][j].z; s.w += v[p][j].w; }
            *reinterpret_cast<float4*>(tile + lane * FIN_LD + (warp * NJ + j) * 4) = s;
        }
    }
    if (EPI != EPI_STORE) {
#pragma unroll
        for (int i = 0; i < FIN_ROWS; ++i) {
            for (int p = lane + 32; a.ss_in && p < a.ss_parts; p += 32) sums[i] += __ldcg(static_cast<const T*>(a.ss_in) + (size_t)p * a.ss_ld + min(m0 + warp * FIN_ROWS + i, a.M - 1));
            inv[i] = a.ss_in ? norm_factor(lanes_sum(sums[i], 32), a.K, a.eps) : 1.0f;
        }
    }
    __syncthreads();
    unsigned char* image = a.xp_out ? a.xp_out + (size_t)rb * wide_block_bytes(EPI == EPI_SWIGLU ? a.N / 2 : a.N) : nullptr;
#pragma unroll
    for (int i = 0; i < FIN_ROWS; ++i) {
        const int r = warp * FIN_ROWS + i, m = m0 + r;
        if (r >= n) break;
        float4 v = *reinterpret_cast<const float4*>(tile + r * FIN_LD + c);
        if (EPI == EPI_STORE) {
            v = make_float4(v.x + x[i].x, v.y + x[i].y, v.z + x[i].z, v.w + x[i].w);
            *reinterpret_cast<float4*>(a.y + (size_t)m * a.ldy + n0 + c) = v;
            if (image) {
                const T ss = lanes_sum(squares<T>(v), 32);
                if (lane == 0) static_cast<T*>(a.ss_out)[(size_t)nblk * a.ss_ld + m] = ss;
                uint32_t t[3][2];
                bf16x2_split3(v.x * w.x, v.y * w.y, t[0][0], t[1][0], t[2][0]);
                bf16x2_split3(v.z * w.z, v.w * w.w, t[0][1], t[1][1], t[2][1]);
                unsigned char* dst = image + (size_t)((n0 + c) >> 6) * (3 * X_SLOT) + (row0 + r) * 128 + (((((n0 + c) & 63) >> 3) ^ (r & 7)) << 4) + (lane & 1) * 8;
#pragma unroll
                for (int k = 0; k < 3; ++k) *reinterpret_cast<uint2*>(dst + k * X_SLOT) = make_uint2(t[k][0], t[k][1]);
            }
        } else if (EPI == EPI_SWIGLU) {
            const float2 g = *reinterpret_cast<const float2*>(tile + r * FIN_LD + 2 * lane), u = *reinterpret_cast<const float2*>(tile + r * FIN_LD + 64 + 2 * lane);
            const float g0 = g.x * inv[i], g1 = g.y * inv[i];
            uint32_t t[3];
            bf16x2_split3((g0 / (1.0f + expf(-g0))) * (u.x * inv[i]), (g1 / (1.0f + expf(-g1))) * (u.y * inv[i]), t[0], t[1], t[2]);
            unsigned char* dst = image + (size_t)nblk * (3 * X_SLOT) + (row0 + r) * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4;
#pragma unroll
            for (int k = 0; k < 3; ++k) *reinterpret_cast<uint32_t*>(dst + k * X_SLOT) = t[k];
        } else {  // bias, per-head QK RMSNorm, RoPE half rotation, K/V page write (src/hf/emitter.rs:604-649)
            v = make_float4(fmaf(v.x, inv[i], bias.x), fmaf(v.y, inv[i], bias.y), fmaf(v.z, inv[i], bias.z), fmaf(v.w, inv[i], bias.w));
            if (a.has_qk_norm) {
                const T ss = lanes_sum(squares<T>(v), HD / 4);
                if (is_q || is_k) {
                    const float f = norm_factor(ss, HD, a.eps);
                    v = make_float4((v.x * f) * w.x, (v.y * f) * w.y, (v.z * f) * w.z, (v.w * f) * w.w);
                }
            }
            const float4 o = make_float4(__shfl_xor_sync(0xffffffffu, v.x, HD / 8), __shfl_xor_sync(0xffffffffu, v.y, HD / 8), __shfl_xor_sync(0xffffffffu, v.z, HD / 8), __shfl_xor_sync(0xffffffffu, v.w, HD / 8));
            if (is_q || is_k) {
                const float sg = d < HD / 2 ? -1.0f : 1.0f;
                v = make_float4(fmaf(sg * o.x, sn[i].x, v.x * cs[i].x), fmaf(sg * o.y, sn[i].y, v.y * cs[i].y), fmaf(sg * o.z, sn[i].z, v.z * cs[i].z), fmaf(sg * o.w, sn[i].w, v.w * cs[i].w));
            }
            if (is_q) {
                *reinterpret_cast<float4*>(a.y + (size_t)m * a.ldy + n0 + c) = v;
            } else if (ok) {
                const int kvh = (nh - a.q_dim - (is_k ? 0 : a.kv_dim)) / HD, tok = pos[i] % a.kv.page_tokens;
                const size_t off = ((size_t)page[i] * a.kv.kv_heads + kvh) * a.kv.page_tokens * HD + (is_k ? k_tile_off(tok, d) : v_tile_off(tok, d, HD, a.kv.bf16));
                void* pool = is_k ? a.kv.k_pool : a.kv.v_pool;
                if (a.kv.bf16) *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(pool) + off) = make_uint2(bf16x2_rne(v.x, v.y), bf16x2_rne(v.z, v.w));
                else *reinterpret_cast<float4*>(reinterpret_cast<float*>(pool) + off) = v;
            }
        }
    }
}

// One CTA per row.
template <bool Q>
__global__ void __launch_bounds__(256) wide_pack_kernel(const float* __restrict__ x, int ldx, int K, const float* __restrict__ norm_w, float eps, unsigned char* __restrict__ xp, size_t block_bytes) {
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x, tid = threadIdx.x;
    const float* xr = x + (size_t)m * ldx;
    using T = Sum<Q>;
    __shared__ T sw[8];
    float inv = 1.0f;
    if (norm_w) {
        T s = 0;
        for (int i = tid; i < K; i += 256) s = fma((T)xr[i], (T)xr[i], s);
        s = lanes_sum(s, 32);
        if ((tid & 31) == 0) sw[tid >> 5] = s;
        __syncthreads();
        T t = 0;
        for (int i = 0; i < 8; ++i) t += sw[i];
        inv = norm_factor(t, K, eps);
    }
    unsigned char* out = xp + (size_t)(m / WIDE_BLOCK) * block_bytes;
    for (int k0 = tid * 8; k0 < (K + 63) / 64 * 64; k0 += 256 * 8) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = k0 + e < K ? xr[k0 + e] : 0.f;
            if (norm_w && k0 + e < K) v[e] = (v[e] * inv) * __ldg(norm_w + k0 + e);
        }
        tc_xpack_store8(out, WIDE_BLOCK, m % WIDE_BLOCK, k0, v);
    }
}

// a thread per eight consecutive inputs of a row
__global__ void __launch_bounds__(256) wide_pack_quant_kernel(const uint8_t* __restrict__ blocks, int n_rows, int K, int q4, unsigned char* __restrict__ dst, int n_off, int interleave_which, int terms) {
    const size_t total = (size_t)n_rows * (K / 8);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int n = (int)(i / (K / 8)), k = (int)(i % (K / 8)) * 8, c = (k & 31) >> 3;
        const uint8_t* b = blocks + ((size_t)n * (K / 32) + k / 32) * (q4 ? 18 : 34);
        const float d = f16_bits_to_f32((uint16_t)(b[0] | b[1] << 8));
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (q4) {  // byte j: element j in the low, element j + 16 in the high nibble
                const uint8_t q = b[2 + (c & 1) * 8 + e];
                v[e] = d * (float)((int)(c >= 2 ? q >> 4 : q & 15) - 8);
            } else {
                v[e] = d * (float)(int8_t)b[2 + c * 8 + e];
            }
        }
        uint32_t w[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) bf16x2_split3(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
        const int row = interleave_which >= 0 ? (n / 64) * 128 + interleave_which * 64 + n % 64 : n + n_off;
        unsigned char* tile = dst + (((size_t)(row / 128) * (K / BK) + k / BK) * terms) * WB_TILE + (row % 128) * 128 + ((((k % BK) >> 3) ^ (row & 7)) << 4);
#pragma unroll
        for (int t = 0; t < 3; ++t)
            if (t < terms) *reinterpret_cast<uint4*>(tile + (size_t)t * WB_TILE) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
    }
}

template <typename F>
cudaError_t launch(F* kernel, const WideArgs& a, dim3 grid, int threads, size_t smem, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <bool GLU, int WT>
cudaError_t launch_product(const WideArgs& a, int sm_count, cudaStream_t st, bool pdl) {
    const cudaError_t e = ensure_dyn_smem(gemm_wide_kernel<GLU, WT>, SMEM);
    return e == cudaSuccess ? launch(gemm_wide_kernel<GLU, WT>, a, dim3((unsigned)std::min(a.units, sm_count)), THREADS, SMEM, st, pdl) : e;
}

template <int S, bool Q>
cudaError_t launch_finish(const WideArgs& a, cudaStream_t st, bool pdl) {
    const dim3 grid((unsigned)a.nblocks, (unsigned)((a.M + 31) / 32));
    if (a.epi == EPI_STORE) return launch(wide_finish_kernel<EPI_STORE, 64, S, Q>, a, grid, FIN_WARPS * 32, 0, st, pdl);
    if (a.epi == EPI_SWIGLU) return launch(wide_finish_kernel<EPI_SWIGLU, 64, S, Q>, a, grid, FIN_WARPS * 32, 0, st, pdl);
    return a.hd == 64 ? launch(wide_finish_kernel<EPI_QKV_ROPE, 64, S, Q>, a, grid, FIN_WARPS * 32, 0, st, pdl) : launch(wide_finish_kernel<EPI_QKV_ROPE, 128, S, Q>, a, grid, FIN_WARPS * 32, 0, st, pdl);
}
template <bool Q>
cudaError_t launch_finish_of(const WideArgs& a, cudaStream_t st, bool pdl) {
    return a.split == 1 ? launch_finish<1, Q>(a, st, pdl) : a.split <= 4 ? launch_finish<4, Q>(a, st, pdl) : launch_finish<8, Q>(a, st, pdl);
}

}  // namespace

WideSplit wide_split(int M, int K, int N, int w_terms, int epi, int sm_count) {
    const double per_kb = w_terms == 1 ? 0.82 : w_terms == 2 ? 1.37 : 1.64;  // three, five and six products
    const int kb = (K + BK - 1) / BK, tiles = ((N + 127) / 128 + 1) / 2 * wide_blocks(M);
    // Microseconds: rounds of units (0.82 per k-block of three products, of a CTA's last unit also 3 for its partial tile), and the second launch, which
    // reads the parts and writes ten bytes per output (6 TB/s in the L2, 4 us at least).
    int best = 1;
    double best_cost = 0;
    for (int s = 1; s <= 8 && (s == 1 || kb / s >= 2); ++s) {
        const int per = (kb + s - 1) / s;
        const double rounds = (double)(((long)tiles * s + sm_count - 1) / sm_count);
        const bool parts = epi != EPI_SWIGLU || s > 1;
        const double cost = rounds * (per * per_kb + 0.5) + (parts ? 3.0 + std::max(4.0, (double)tiles * 128 * 256 * (4.0 * s + 10) / 6e6) : 6.0);
        if (s == 1 || cost < best_cost) {
            best_cost = cost;
            best = s;
        }
    }
    return {best, epi != EPI_SWIGLU || best > 1 ? (size_t)tiles * best * 128 * 256 : 0};
}

cudaError_t launch_gemm_wide(const WideArgs& a_in, int sm_count, cudaStream_t st, bool pdl, int* launches) {
    WideArgs a = a_in;
    if (a.M < 1 || a.M > WIDE_ROWS || !a.xp || !a.W) return cudaErrorInvalidValue;
    // whole heads, and whole blocks of 128 outputs elsewhere: vector accesses without a look at the end
    const bool qkv = a.epi == EPI_QKV_ROPE;
    if (qkv ? (a.hd != 64 && a.hd != 128) || a.N % a.hd != 0 : (a.epi != EPI_STORE && a.epi != EPI_SWIGLU) || a.N % 128 != 0) return cudaErrorInvalidValue;
    if (a.epi != EPI_SWIGLU && ((a.ldy & 3) || ((reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.resid)) & 15))) return cudaErrorInvalidValue;
    a.kblocks = (a.K + BK - 1) / BK;
    a.nblocks = (a.N + 127) / 128;
    a.tiles = (a.nblocks + 1) / 2;
    a.row_blocks = wide_blocks(a.M);
    const int split = wide_split(a.M, a.K, a.N, a.w_terms, a.epi, sm_count).split;
    a.kb_per = (a.kblocks + split - 1) / split;
    a.split = (a.kblocks + a.kb_per - 1) / a.kb_per;
    a.units = a.tiles * a.row_blocks * a.split;
    const bool whole = a.epi == EPI_SWIGLU && a.split == 1;
    if (!whole && !a.part) return cudaErrorInvalidValue;
    ++*launches;
    const cudaError_t e = a.w_terms == 1   ? (whole ? launch_product<true, 1>(a, sm_count, st, pdl) : launch_product<false, 1>(a, sm_count, st, pdl))
                          : a.w_terms == 2 ? (whole ? launch_product<true, 2>(a, sm_count, st, pdl) : launch_product<false, 2>(a, sm_count, st, pdl))
                          : a.w_terms == 3 ? (whole ? launch_product<true, 3>(a, sm_count, st, pdl) : launch_product<false, 3>(a, sm_count, st, pdl))
                                           : cudaErrorInvalidValue;
    if (e != cudaSuccess || whole) return e;
    ++*launches;
    return a.w_terms == 1 ? launch_finish_of<false>(a, st, pdl) : launch_finish_of<true>(a, st, pdl);
}

cudaError_t launch_wide_pack_quant(const uint8_t* blocks, int n_rows, int K, bool q4, uint16_t* dst, int n_off, int interleave_which, cudaStream_t st) {
    if (K % BK != 0 || n_rows < 1) return cudaErrorInvalidValue;
    const size_t g = std::min<size_t>(((size_t)n_rows * (K / 8) + 255) / 256, 148 * 32);
    wide_pack_quant_kernel<<<(unsigned)g, 256, 0, st>>>(blocks, n_rows, K, q4 ? 1 : 0, reinterpret_cast<unsigned char*>(dst), n_off, interleave_which, wide_quant_terms(q4));
    return cudaGetLastError();
}

cudaError_t launch_wide_pack(const float* x, int ldx, int M, int K, const float* norm_w, float eps, bool f64, unsigned char* xp, cudaStream_t st, bool pdl) {
    if (M < 1) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)M);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return f64 ? cudaLaunchKernelEx(&cfg, wide_pack_kernel<true>, x, ldx, K, norm_w, eps, xp, wide_block_bytes(K)) : cudaLaunchKernelEx(&cfg, wide_pack_kernel<false>, x, ldx, K, norm_w, eps, xp, wide_block_bytes(K));
}

}  // namespace hm
