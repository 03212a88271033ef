// Causal attention of a prompt's rows over a paged KV cache: many query rows per key, where the decode kernels (attention.cu) read the
// context once per row.
//
// Two launches per layer.  The first turns the pages of the sequences (context and new rows) into dense blocks of 64 keys: the bf16 terms
// of keys and values (one on bf16 pages, three on f32 pages: hi + mid + lo is exact to 2^-24), rows of 64 dims in 128 bytes with the
// 128-byte swizzle, so that the second launch needs one bulk copy per operand and its ldmatrix reads are free of bank conflicts.
// Splitting in the attention itself would repeat for every query tile and head.
//
// The second: one CTA = 64 rows of one query head; four warps own 16 rows each, a fifth feeds a ring of K and V blocks.  Both
// contractions are warp-level MMAs (m16n8k16, f32 accumulate) on terms whose products reach 2^-24: queries and probabilities are f32 (three
// terms each), so bf16 pages take three products and f32 pages six, the leading one in an accumulator of its own.  The sums of a 64-key block start from zero and join the
// running result as one f32 multiply-add (the rescaling that the online softmax does anyway), so that the tensor core's truncating
// additions never form a chain longer than a block.  Masked keys have probability zero: a value that is not finite reaches the rows of its own block of 64
// keys in front of it too (in the decode kernels, those of its page of 16).
// Measured: 2048 rows x 12 heads of 128 on bf16 pages 142 us (272 TFLOP/s of products), 1999 rows x 14 heads of 64 on f32 pages 126 us, bound
// by the warp-level MMAs; the decode kernel took 32 launches of 64 rows for the same, 3500 rows of the 0.6 B geometry 113 -> 14 ms.
#include <algorithm>

#include "attn_prefill.h"
#include "gemm_wide.h"
#include "launch_attrs.h"
#include "mbarrier.cuh"

namespace hm {
namespace {

constexpr int QT = PREFILL_TILE;
constexpr int WARPS = 4;
constexpr int THREADS = (WARPS + 1) * 32;
constexpr int MAX_SLOTS = 8;

template <int HD, bool BF16>
struct Shape {
    static constexpr int KT = BF16 ? 1 : 3;          // terms of a cached element
    static constexpr int PANEL = QT * 128;           // [64 rows][64 dims] bf16
    static constexpr int PANELS = HD / 64;
    static constexpr int SLOT = KT * PANELS * PANEL;  // K or V of one block
    static constexpr int Q_BYTES = 3 * PANELS * PANEL;
    // two CTAs per SM where three slots and the queries fit half of its shared memory, else as deep a ring as one CTA may have
    static constexpr int CTAS = Q_BYTES + 3 * SLOT + 1024 <= 112 * 1024 ? 2 : 1;
    static constexpr int FIT = ((CTAS == 2 ? 112 : 224) * 1024 - 1024 - Q_BYTES) / SLOT;
    static constexpr int SLOTS = FIT < MAX_SLOTS ? FIT : MAX_SLOTS;
    static constexpr size_t SMEM = (size_t)Q_BYTES + (size_t)SLOTS * SLOT + 1024;
    static_assert(SLOTS >= 2, "ring too small");
};

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// eight consecutive dims of one row -> the 16-byte pieces of its terms at `dst` (terms `term_stride` bytes apart)
template <int TERMS>
__device__ __forceinline__ void store_terms(unsigned char* dst, size_t term_stride, const float (&v)[8]) {
    uint32_t w[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (TERMS == 3) bf16x2_split3(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
        else w[0][e] = bf16x2_rne(v[2 * e], v[2 * e + 1]);
    }
#pragma unroll
    for (int t = 0; t < TERMS; ++t) *reinterpret_cast<uint4*>(dst + t * term_stride) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
}

// grid (blocks, kv heads)
template <int HD, bool BF16>
__global__ void __launch_bounds__(256) prefill_stage_kernel(const PrefillArgs a) {
    using S = Shape<HD, BF16>;
    pdl_launch_dependents();
    pdl_wait();
    const PrefillBlock b = a.blocks[blockIdx.x];
    const int kvh = blockIdx.y;
    unsigned char* out = a.staged + ((size_t)blockIdx.x * a.kv.kv_heads + kvh) * (2 * S::SLOT);
    const int32_t* pt = a.kv.page_table + (size_t)b.seq * a.kv.max_pages + b.key0 / 16;
    for (int i = threadIdx.x; i < 2 * QT * (HD / 8); i += 256) {
        // consecutive threads take consecutive tokens: pieces of a page are chunk-major (values of f32 pages are rows)
        const bool is_v = i >= QT * (HD / 8);
        const int j = is_v ? i - QT * (HD / 8) : i;
        const int t = j % QT, c = j / QT;
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (t < b.valid) {  // what lies behind the end must be finite: its probabilities are zero
            const size_t tile = ((size_t)pt[t / 16] * a.kv.kv_heads + kvh) * 16 * HD;
            const int tk = t & 15;
            if (BF16) {
                const uint16_t* p = reinterpret_cast<const uint16_t*>(is_v ? a.kv.v_pool : a.kv.k_pool) + tile;
                uint32_t w[4];
                if (is_v) {
                    const uint4 u = *reinterpret_cast<const uint4*>(p + v_tile_off(tk, c * 8, HD, 1));
                    w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w;
                } else {
                    const uint2 u0 = *reinterpret_cast<const uint2*>(p + k_tile_off(tk, c * 8)), u1 = *reinterpret_cast<const uint2*>(p + k_tile_off(tk, c * 8 + 4));
                    w[0] = u0.x; w[1] = u0.y; w[2] = u1.x; w[3] = u1.y;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) { v[2 * e] = bf16_lo(w[e]); v[2 * e + 1] = bf16_hi(w[e]); }
            } else {
                const float* p = reinterpret_cast<const float*>(is_v ? a.kv.v_pool : a.kv.k_pool) + tile;
                const float4 f0 = *reinterpret_cast<const float4*>(p + (is_v ? v_tile_off(tk, c * 8, HD, 0) : k_tile_off(tk, c * 8)));
                const float4 f1 = *reinterpret_cast<const float4*>(p + (is_v ? v_tile_off(tk, c * 8 + 4, HD, 0) : k_tile_off(tk, c * 8 + 4)));
                v[0] = f0.x; v[1] = f0.y; v[2] = f0.z; v[3] = f0.w; v[4] = f1.x; v[5] = f1.y; v[6] = f1.z; v[7] = f1.w;
            }
        }
        unsigned char* dst = out + (is_v ? S::SLOT : 0) + (c >> 3) * S::PANEL + t * 128 + (((c & 7) ^ (t & 7)) << 4);
        store_terms<S::KT>(dst, (size_t)S::PANELS * S::PANEL, v);
    }
}

// Products of two operands' terms that reach 2^-24 of the result, the small ones first: term i of the f32 operand with term j of the
// cached one, i + j <= 2.
template <int KT>
struct Pairs {
    static constexpr int N = KT == 1 ? 3 : 6;
    __host__ __device__ static constexpr int a(int p) { return KT == 1 ? 2 - p : p == 0 ? 2 : p == 1 || p == 3 ? 1 : 0; }
    __host__ __device__ static constexpr int b(int p) { return KT == 1 ? 0 : p == 2 ? 2 : p == 1 || p == 4 ? 1 : 0; }
};

template <int HD, bool BF16>
__global__ void __launch_bounds__(THREADS, (Shape<HD, BF16>::CTAS)) attn_prefill_kernel(const PrefillArgs a) {
    using S = Shape<HD, BF16>;
    using P = Pairs<S::KT>;
    constexpr int KS = HD / 16, TERM = S::PANELS * S::PANEL;
    extern __shared__ __align__(1024) unsigned char dsm[];
    __shared__ uint64_t full[MAX_SLOTS], empty[MAX_SLOTS];
    __shared__ volatile int s_abort;
    unsigned char* qs = dsm + ((1024u - (s32(dsm) & 1023u)) & 1023u);
    unsigned char* ring = qs + S::Q_BYTES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int head = blockIdx.x % a.heads, kvh = head / (a.heads / a.kv.kv_heads);
    if (tid == 0) {
        for (int s = 0; s < S::SLOTS; ++s) { mb_init(&full[s], 1); mb_init(&empty[s], WARPS); }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_launch_dependents();
    pdl_wait();
    const PrefillTile t = a.tiles[blockIdx.x / a.heads];
    const int nb = (t.pos0 + t.rows - 1) / QT + 1;
    // queries: f32 rows -> three terms in the operand's layout; rows behind the end are zero
    for (int i = tid; i < QT * (HD / 8); i += THREADS) {
        const int r = i / (HD / 8), c = i % (HD / 8);
        float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (r < t.rows) {
            const float* q = a.q + (size_t)(t.row0 + r) * a.heads * HD + (size_t)head * HD + c * 8;
            const float4 f0 = ld_cg_f32x4(q), f1 = ld_cg_f32x4(q + 4);
            v[0] = f0.x; v[1] = f0.y; v[2] = f0.z; v[3] = f0.w; v[4] = f1.x; v[5] = f1.y; v[6] = f1.z; v[7] = f1.w;
        }
        store_terms<3>(qs + (c >> 3) * S::PANEL + r * 128 + (((c & 7) ^ (r & 7)) << 4), TERM, v);
    }
    __syncthreads();
    if (warp == WARPS) {
        if (lane == 0) {
            const unsigned char* src = a.staged + ((size_t)t.block0 * a.kv.kv_heads + kvh) * (2 * S::SLOT);
            const size_t step = (size_t)a.kv.kv_heads * (2 * S::SLOT);
            int i = 0;
            for (; i < 2 * nb; ++i) {  // K and V of a block in turn
                const int s = i % S::SLOTS;
                if (i >= S::SLOTS && !mb_wait(&empty[s], ((i / S::SLOTS) & 1u) ^ 1u, a.err_flag, &s_abort)) break;
                mb_expect_tx(&full[s], S::SLOT);
                bulk_copy(ring + (size_t)s * S::SLOT, src + (i >> 1) * step + (i & 1) * S::SLOT, S::SLOT, &full[s]);
            }
            mb_land_ring(full, (uint32_t)i, S::SLOTS);  // (consumers that gave up leave at once)
        }
        return;
    }
    const int gid = lane >> 2, tig = lane & 3, r0 = warp * 16;
    const uint32_t q32 = s32(qs), ring32 = s32(ring);
    // ldmatrix: the row that this lane addresses within 16 rows, and which of the two 16-byte chunks
    const int arow = r0 + (lane & 15), achunk = lane >> 4;                       // A of Q; also V (keys as rows)
    const int brow = (lane & 7) + ((lane >> 4) << 3), bchunk = (lane >> 3) & 1;  // B of K
    const int vrow = lane & 15;
    float o[HD / 8][4], mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < HD / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    for (int b = 0; b < nb; ++b) {
        const int ik = 2 * b, iv = 2 * b + 1, sk = ik % S::SLOTS, sv = iv % S::SLOTS;
        // the leading products in a chain of their own: the tensor core truncates at the accumulator's magnitude
        float sc[8][4], lo[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = lo[n][0] = lo[n][1] = lo[n][2] = lo[n][3] = 0.f;
        if (!__all_sync(0xffffffffu, mb_wait(&full[sk], (ik / S::SLOTS) & 1u, a.err_flag, &s_abort))) return;
        const uint32_t kbase = ring32 + sk * S::SLOT;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            uint32_t qa[3][4];
            const uint32_t qoff = (ks >> 2) * S::PANEL + arow * 128 + ((((ks & 3) * 2 + achunk) ^ (arow & 7)) << 4);
#pragma unroll
            for (int i = 0; i < 3; ++i) ldsm4(qa[i], q32 + i * TERM + qoff);
#pragma unroll
            for (int np = 0; np < 4; ++np) {  // pairs of 8-key tiles
                uint32_t kf[S::KT][4];
                const int kr = np * 16 + brow;
                const uint32_t koff = (ks >> 2) * S::PANEL + kr * 128 + ((((ks & 3) * 2 + bchunk) ^ (kr & 7)) << 4);
#pragma unroll
                for (int i = 0; i < S::KT; ++i) ldsm4(kf[i], kbase + i * TERM + koff);
#pragma unroll
                for (int p = 0; p < P::N - 1; ++p) {
                    mma16816(lo[2 * np], qa[P::a(p)], kf[P::b(p)][0], kf[P::b(p)][1]);
                    mma16816(lo[2 * np + 1], qa[P::a(p)], kf[P::b(p)][2], kf[P::b(p)][3]);
                }
                mma16816(sc[2 * np], qa[0], kf[0][0], kf[0][1]);
                mma16816(sc[2 * np + 1], qa[0], kf[0][2], kf[0][3]);
            }
        }
        __syncwarp();
        if (lane == 0) mb_arrive(&empty[sk]);
        // online softmax of rows r0 + gid and r0 + gid + 8; a row's keys are spread over four lanes
        float corr[2];
        const bool diagonal = b * QT + QT - 1 > t.pos0 + r0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int pos = t.pos0 + r0 + gid + 8 * h - b * QT;  // last key of this block that the row sees
            float top = -INFINITY;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float s = (lo[n][2 * h + e] + sc[n][2 * h + e]) * a.scale;
                    if (diagonal && n * 8 + tig * 2 + e > pos) s = -INFINITY;
                    sc[n][2 * h + e] = s;
                    top = fmaxf(top, s);
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const float m_new = fmaxf(mx[h], top);  // finite: key 0 is in the first block and every row sees it
            corr[h] = exp2f((mx[h] - m_new) * 1.4426950408889634f);
            mx[h] = m_new;
            float l = 0.f;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float p = exp2f((sc[n][2 * h + e] - m_new) * 1.4426950408889634f);
                    sc[n][2 * h + e] = p;
                    l += p;
                }
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            sum[h] = fmaf(sum[h], corr[h], l);
        }
        // probabilities as A operands: the accumulator's layout is the operand's
        uint32_t pa[4][3][4];
#pragma unroll
        for (int kt = 0; kt < 4; ++kt)
#pragma unroll
            for (int q = 0; q < 4; ++q) bf16x2_split3(sc[2 * kt + (q >> 1)][2 * (q & 1)], sc[2 * kt + (q >> 1)][2 * (q & 1) + 1], pa[kt][0][q], pa[kt][1][q], pa[kt][2][q]);
        if (!__all_sync(0xffffffffu, mb_wait(&full[sv], (iv / S::SLOTS) & 1u, a.err_flag, &s_abort))) return;
        const uint32_t vbase = ring32 + sv * S::SLOT;
#pragma unroll
        for (int np = 0; np < HD / 16; ++np) {  // 16 dims at a time
            float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f}, d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                uint32_t vf[S::KT][4];
                const int vr = kt * 16 + vrow;
                const uint32_t voff = (np >> 2) * S::PANEL + vr * 128 + ((((np & 3) * 2 + achunk) ^ (vr & 7)) << 4);
#pragma unroll
                for (int i = 0; i < S::KT; ++i) ldsm4t(vf[i], vbase + i * TERM + voff);
#pragma unroll
                for (int p = 0; p < P::N - 1; ++p) {
                    mma16816(d0, pa[kt][P::a(p)], vf[P::b(p)][0], vf[P::b(p)][1]);
                    mma16816(d1, pa[kt][P::a(p)], vf[P::b(p)][2], vf[P::b(p)][3]);
                }
                mma16816(c0, pa[kt][0], vf[0][0], vf[0][1]);
                mma16816(c1, pa[kt][0], vf[0][2], vf[0][3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[2 * np][e] = fmaf(o[2 * np][e], corr[e >> 1], d0[e] + c0[e]);
                o[2 * np + 1][e] = fmaf(o[2 * np + 1][e], corr[e >> 1], d1[e] + c1[e]);
            }
        }
        __syncwarp();
        if (lane == 0) mb_arrive(&empty[sv]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = r0 + gid + 8 * h, m = t.row0 + r;
        if (r >= t.rows) continue;
        const float inv = 1.0f / sum[h];
        unsigned char* row = a.xp_out + (size_t)(m / WIDE_BLOCK) * a.xp_block + (size_t)(m % WIDE_BLOCK) * 128;
#pragma unroll
        for (int n = 0; n < HD / 8; ++n) {
            const int k = head * HD + n * 8;
            uint32_t w[3];
            bf16x2_split3(o[n][2 * h] * inv, o[n][2 * h + 1] * inv, w[0], w[1], w[2]);
            unsigned char* dst = row + (size_t)(k >> 6) * (3 * WIDE_BLOCK * 128) + ((((k & 63) >> 3) ^ (m & 7)) << 4) + tig * 4;
#pragma unroll
            for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(dst + (size_t)i * WIDE_BLOCK * 128) = w[i];
        }
    }
}

template <int HD, bool BF16>
cudaError_t launch_t(const PrefillArgs& a, cudaStream_t st, bool pdl, int* launches) {
    using S = Shape<HD, BF16>;
    cudaError_t e = ensure_dyn_smem(attn_prefill_kernel<HD, BF16>, S::SMEM);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    cfg.stream = st;
    cfg.gridDim = dim3((unsigned)a.n_blocks, (unsigned)a.kv.kv_heads);
    cfg.blockDim = dim3(256);
    e = cudaLaunchKernelEx(&cfg, prefill_stage_kernel<HD, BF16>, a);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3((unsigned)(a.n_tiles * a.heads));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    *launches += 2;
    return cudaLaunchKernelEx(&cfg, attn_prefill_kernel<HD, BF16>, a);
}

}  // namespace

cudaError_t launch_attn_prefill(const PrefillArgs& a, cudaStream_t st, bool pdl, int* launches) {
    if (a.n_tiles < 1 || a.n_blocks < 1 || a.kv.page_tokens != 16 || a.heads % a.kv.kv_heads != 0) return cudaErrorInvalidValue;
    if (a.kv.hd == 64) return a.kv.bf16 ? launch_t<64, true>(a, st, pdl, launches) : launch_t<64, false>(a, st, pdl, launches);
    if (a.kv.hd == 128) return a.kv.bf16 ? launch_t<128, true>(a, st, pdl, launches) : launch_t<128, false>(a, st, pdl, launches);
    return cudaErrorInvalidValue;
}

}  // namespace hm
