// Passes over many rows of prompts (65 to 2048) on the uniform stacks (bf16, Q8_0 and Q4_0 weights): every weight is read once per pass instead of once per 64
// rows, projections run on the many-row GEMM (gemm_wide.cu) and runs of a sequence's rows on the prompt attention (attn_prefill.cu).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "engine.h"
#include "engine_util.h"
#include "gemm_tc.h"
#include "gemm_wide.h"

namespace hm {

// Runs shorter than this go to the decode attention, row by row: a tile of the prompt attention costs as much for one row as for 64,
// and its context is staged first.
constexpr int WIDE_MIN_RUN = 8;

// Sizes that the wide passes take.
bool Engine::wide_sizes() const { return !spec_.listed() && use_tc_ && H_ % 128 == 0 && I_ % 64 == 0; }

bool Engine::wide_fits() const {
    if (!wide_sizes() || page_tokens_ != 16) return false;
    for (const LayerW& l : layers_)
        for (const LinearW* w : {&l.qkv, &l.o, &l.gu, &l.down})
            if (!w->tc && !w->wide) return false;
    return true;
}

// Whether the projections of a quantised model are held as bf16 terms as well.  Decided once, when the first of them is loaded, so that a model
// has all copies or none: where the wide passes take its sizes, and the copies take an eighth of the free memory at most (of a GPU of its
// own 22 GB: models of up to 3.8 B weights in Q8_0).  The rest of the weights, a fifth of the copies at most, and the caches find room beside them.
bool Engine::wide_copies(int terms) {
    if (wide_copies_ < 0) {
        size_t free_bytes = 0, total = 0;
        const double weights = (double)L_ * ((double)H_ * (2.0 * qdim_ + 2.0 * kvdim_) + 3.0 * H_ * I_);
        const bool known = cudaMemGetInfo(&free_bytes, &total) == cudaSuccess;
        if (!known) cudaGetLastError();
        wide_copies_ = known && wide_sizes() && weights * 2 * terms <= (double)free_bytes / 8;
    }
    return wide_copies_ > 0;
}

// Frees what the engine can do without: the wide passes' scratch and a quantised model's copies (its prompts then run in passes of 64 rows).
// The calls that allocate do so before they plan a pass.  False: there was nothing.
bool Engine::give_back() {
    bool any = wide_.cap > 0 || wide_copies_ > 0;
    if (stream_) cudaStreamSynchronize(stream_);
    free_wide();
    each_linear([&](LinearW& w) {
        if (w.wide) cudaFree(w.wide);
        w.wide = nullptr;
    });
    if (wide_copies_ > 0) wide_copies_ = 0;
    return any;
}

void Engine::free_wide() {
    for (void* p : {(void*)wide_.base, (void*)wide_.own_staged, (void*)wide_.own_tables})
        if (p) cudaFree(p);
    wide_ = Wide();
}

// Scratch of the passes that a call on this cache can ask for, in one allocation (the stream is idle).  Taken with the cache and kept for the
// next one: an allocation takes 0.35 ms whatever its size, and eleven of them, with pinned memory for the tables, in a prompt's first
// pass took longer than the pass saves up to 200 tokens (the first 100 tokens of a cache, 0.5 B stack: 2.33 ms in passes of 64 rows, 2.06 here, 4.9 with them).
// False without memory for it: the caller then takes passes of 64 rows.
bool Engine::ensure_wide() {
    const long all = (long)batch_ * max_seq_;
    if (all <= TC_ROWS || !wide_fits()) return false;
    const int rows = (int)std::min<long>(WIDE_ROWS, (all + WIDE_BLOCK - 1) / WIDE_BLOCK * WIDE_BLOCK), blocks = wide_blocks(rows);
    const size_t staged = std::min(staged_kept_, (size_t)batch_ * ((max_seq_ + PREFILL_TILE - 1) / PREFILL_TILE) * prefill_block_bytes(kvh_, hd_, kv_bf16_));
    if (rows <= wide_.cap && staged <= wide_.kept_bytes) return true;
    free_wide();
    size_t part = 1, bytes = 0;
    for (int b = 1; b <= blocks; ++b)
        for (const LinearW* w : {&layers_[0].qkv, &layers_[0].o, &layers_[0].gu, &layers_[0].down})
            part = std::max(part, wide_split(b * WIDE_BLOCK, w->K, w->N, w->tc ? 1 : w->wide_terms, w == &layers_[0].gu ? EPI_SWIGLU : EPI_STORE, sm_count_).part_floats);
    auto place = [&](auto** p, size_t count) {  // without a base: sizes only
        *p = wide_.base ? reinterpret_cast<std::remove_reference_t<decltype(*p)>>(wide_.base + bytes) : nullptr;
        bytes += (count * sizeof(**p) + 65535) / 65536 * 65536;  // (parts on multiples of 1 KB: 66 tokens on the 0.5 B stack 1.83 -> 1.87 ms)
    };
    auto lay = [&]() {
        bytes = 0;
        place(&wide_.h, (size_t)rows * H_);
        place(&wide_.q, (size_t)rows * qdim_);
        place(&wide_.ss, (size_t)(H_ / 128) * rows);
        place(&wide_.ss2, (size_t)(H_ / 128) * rows);
        place(&wide_.x, blocks * wide_block_bytes(H_));
        place(&wide_.x2, blocks * wide_block_bytes(H_));
        place(&wide_.att, blocks * wide_block_bytes(qdim_));
        place(&wide_.act, blocks * wide_block_bytes(I_));
        place(&wide_.part, part);
        place(&wide_.kept_staged, staged);
        place(&wide_.kept_tables, WIDE_TABLE);
    };
    lay();
    if (cudaMalloc((void**)&wide_.base, bytes) != cudaSuccess) {
        cudaGetLastError();
        wide_ = Wide();
        return false;
    }
    lay();
    wide_.cap = rows;
    wide_.kept_bytes = staged;
    return true;
}

// Rows from which a call takes wide passes: more than one 64-row pass.  One prompt, ms in passes of the 64-row kernels and here: of 100 rows
// 0.5 B 2.30 and 2.00, 1.5 B 3.51 and 3.27, TinyLlama Q8_0 6.77 and 2.95; of 65 rows 1.86 and 1.87, 3.0 to 3.8 (by the cache's capacity) and 3.07 to
// 3.20, 4.03 and 2.94.  Single tokens of as many sequences, row by row in the attention: 65 of 1.5 B 6.5 and 3.5, of 0.5 B 3.0 and 2.3, of TinyLlama Q8_0 4.6 and
// 3.3; 64 of them and a prompt of 20: 4.15 and 4.24, 2.88 and 2.74, 7.3 and 3.8.
// Cuts the n rows of a call (host arrays: position and sequence of each; a sequence's rows are consecutive) into wide passes and sends
// the tables of their attention to the device.  No passes where the rows are few or the model has no wide path.
int Engine::plan_wide(const uint32_t* pos, const uint32_t* seq, int n, WidePlan* plan) {
    plan->passes.clear();
    plan->rows = 0;
    if (n <= TC_ROWS || !ensure_wide()) return HM_OK;
    const int n_pass = (n + WIDE_ROWS - 1) / WIDE_ROWS;
    const int per = std::min(WIDE_ROWS, ((n + n_pass - 1) / n_pass + WIDE_BLOCK - 1) / WIDE_BLOCK * WIDE_BLOCK);
    const size_t block_bytes = prefill_block_bytes(kvh_, hd_, kv_bf16_);
    const int budget = (int)std::max<size_t>(1, staged_most_ / block_bytes);
    std::vector<PrefillTile> tiles;
    std::vector<PrefillBlock> blocks;
    int most = 0;
    while (n - plan->rows > TC_ROWS) {
        WidePass p;
        p.row0 = plan->rows;
        p.rows = std::min(per, n - p.row0);
        auto close = [&]() {  // the longest tiles first, so that the last CTAs of the launch are short
            WidePass::Group& g = p.groups.back();
            g.tiles = (int)tiles.size() - g.tile0;
            g.blocks = (int)blocks.size() - g.block0;
            most = std::max(most, g.blocks);
            std::stable_sort(tiles.begin() + g.tile0, tiles.end(), [](const PrefillTile& a, const PrefillTile& b) { return a.pos0 + a.rows > b.pos0 + b.rows; });
        };
        for (int r = 0; r < p.rows;) {
            const uint32_t *ps = pos + p.row0 + r, *sq = seq + p.row0 + r;
            int run = 1;
            while (r + run < p.rows && sq[run] == sq[0]) ++run;
            if (run < WIDE_MIN_RUN) {
                if (!p.singles.empty() && p.singles.back().row0 + p.singles.back().rows == r) p.singles.back().rows += run;
                else p.singles.push_back({r, run});
            } else {
                const int len = (int)ps[0] + run, nb = (len + PREFILL_TILE - 1) / PREFILL_TILE;
                if (p.groups.empty() || (int)blocks.size() - p.groups.back().block0 + nb > budget) {
                    if (!p.groups.empty()) close();
                    p.groups.push_back({(int)tiles.size(), 0, (int)blocks.size(), 0});
                }
                const int b0 = (int)blocks.size() - p.groups.back().block0;
                for (int b = 0; b < nb; ++b) blocks.push_back({(int32_t)sq[0], b * PREFILL_TILE, std::min(PREFILL_TILE, len - b * PREFILL_TILE), 0});
                for (int t = 0; t < run; t += PREFILL_TILE) tiles.push_back({r + t, std::min(PREFILL_TILE, run - t), (int32_t)ps[0] + t, b0});
            }
            r += run;
        }
        if (!p.groups.empty()) close();
        plan->rows += p.rows;
        plan->passes.push_back(std::move(p));
    }
    static_assert(sizeof(PrefillTile) == 16 && sizeof(PrefillBlock) == 16, "table entries are four words");
    const size_t words = 4 * (tiles.size() + blocks.size());
    auto give_up = [&]() {  // without memory: passes of 64 rows
        cudaGetLastError();
        plan->passes.clear();
        plan->rows = 0;
        return HM_OK;
    };
    // what the kept parts do not hold (passes of many thousand tokens) is allocated once and grows
    if (words > WIDE_TABLE && words > wide_.own_words) {
        if (wide_.own_tables) cudaFree(wide_.own_tables);
        wide_.own_tables = nullptr;
        wide_.own_words = 0;
        const size_t cap = words + words / 2;
        if (cudaMalloc((void**)&wide_.own_tables, cap * 4) != cudaSuccess) return give_up();
        wide_.own_words = cap;
    }
    if (most * block_bytes > std::max(wide_.kept_bytes, wide_.own_bytes)) {
        if (wide_.own_staged) cudaFree(wide_.own_staged);
        wide_.own_staged = nullptr;
        wide_.own_bytes = 0;
        const size_t bytes = std::max<size_t>(most * block_bytes, std::min<size_t>(staged_most_, 2 * most * block_bytes));
        if (cudaMalloc((void**)&wide_.own_staged, bytes) != cudaSuccess) return give_up();
        wide_.own_bytes = bytes;
    }
    plan->staged = most * block_bytes > wide_.kept_bytes ? wide_.own_staged : wide_.kept_staged;
    int32_t* tables = words > WIDE_TABLE ? wide_.own_tables : wide_.kept_tables;
    plan->tiles = reinterpret_cast<PrefillTile*>(tables);
    plan->blocks = reinterpret_cast<PrefillBlock*>(plan->tiles + tiles.size());
    const size_t tile_bytes = tiles.size() * sizeof(PrefillTile), block_table = blocks.size() * sizeof(PrefillBlock);
    if (words && words <= WIDE_TABLE) {  // through pinned memory, as one copy
        unsigned char* pin = reinterpret_cast<unsigned char*>(pin_u32_ + pin_u32_cap_);
        std::memcpy(pin, tiles.data(), tile_bytes);
        std::memcpy(pin + tile_bytes, blocks.data(), block_table);
        HM_CUDA(cudaMemcpyAsync(plan->tiles, pin, tile_bytes + block_table, cudaMemcpyHostToDevice, stream_));
    } else if (words) {  // a copy from pageable memory has read it when it returns
        HM_CUDA(cudaMemcpyAsync(plan->tiles, tiles.data(), tile_bytes, cudaMemcpyHostToDevice, stream_));
        HM_CUDA(cudaMemcpyAsync(plan->blocks, blocks.data(), block_table, cudaMemcpyHostToDevice, stream_));
    }
    return HM_OK;
}

// All layers of one pass; the residual stream is left in wide_.h.
int Engine::enqueue_wide(const WidePlan& plan, const WidePass& p, const uint32_t* tokens, const int32_t* row_pos, const int32_t* row_seq, int* launches) {
    const int M = p.rows;
    const float eps = (float)cfg_.rms_norm_eps;
    cudaError_t ce = launch_embed_gather(embed_, embed_dtype_ == HM_BF16 ? 1 : 0, tokens, M, H_, V_, wide_.h, err_flag_, stream_, pdl_);
    if (ce != cudaSuccess) return cuda_fail(ce, "embed_gather");
    ce = launch_wide_pack(wide_.h, H_, M, H_, layers_[0].in_ln, eps, quant_, wide_.x, stream_, pdl_);
    if (ce != cudaSuccess) return cuda_fail(ce, "activation pack");
    *launches += 2;
    for (int l = 0; l < L_; ++l) {
        const LayerW& w = layers_[l];
        const KvDesc kv{k_pool_[l], v_pool_[l], page_table_, max_pages_, page_tokens_, kvh_, hd_, kv_bf16_ ? 1 : 0};
        auto project = [&](const LinearW& L, const unsigned char* xp, int epi, WideArgs a) {
            a.W = L.tc ? L.tc : L.wide;
            a.w_terms = L.tc ? 1 : L.wide_terms;
            a.K = L.K;
            a.N = L.N;
            a.M = M;
            a.xp = xp;
            a.epi = epi;
            a.eps = eps;
            a.ss_parts = H_ / 128;
            a.ss_ld = wide_.cap;
            a.part = wide_.part;
            a.err_flag = err_flag_;
            return launch_gemm_wide(a, sm_count_, stream_, pdl_, launches);
        };
        WideArgs qkv{};
        qkv.bias = w.qkv_bias;
        qkv.y = wide_.q;
        qkv.ldy = qdim_;
        qkv.ss_in = l > 0 ? wide_.ss : nullptr;  // the first layer's rows were normalised when they were packed
        qkv.q_dim = qdim_;
        qkv.kv_dim = kvdim_;
        qkv.hd = hd_;
        qkv.has_qk_norm = cfg_.has_qk_norm;
        qkv.q_norm_w = w.q_norm;
        qkv.k_norm_w = w.k_norm;
        qkv.rope_cos = rope_cos_;
        qkv.rope_sin = rope_sin_;
        qkv.row_pos = row_pos;
        qkv.row_seq = row_seq;
        qkv.kv = kv;
        ce = project(w.qkv, wide_.x, EPI_QKV_ROPE, qkv);
        if (ce != cudaSuccess) return cuda_fail(ce, "wide QKV projection");
        for (const WidePass::Group& g : p.groups) {
            PrefillArgs a{};
            a.kv = kv;
            a.heads = heads_;
            a.scale = (float)(1.0 / std::sqrt((double)hd_));
            a.q = wide_.q;
            a.staged = plan.staged;
            a.tiles = plan.tiles + g.tile0;
            a.blocks = plan.blocks + g.block0;
            a.n_tiles = g.tiles;
            a.n_blocks = g.blocks;
            a.xp_out = wide_.att;
            a.xp_block = wide_block_bytes(qdim_);
            a.err_flag = err_flag_;
            ce = launch_attn_prefill(a, stream_, pdl_, launches);
            if (ce != cudaSuccess) return cuda_fail(ce, "prompt attention");
        }
        // A launch writes the image from its own row 0 on: it stays within a block of 128 rows and starts on a multiple of eight, with which
        // the image's swizzle repeats (the up to seven rows in front, of the prompt attention above, are done again).  An offset within the
        // image as arguments of the decode kernel cost it four registers, and the steps of the 1.5 B stack 8 us per layer (f32 pages: 1.25 -> 1.49 ms).
        for (const WidePass::Range& r : p.singles)
            for (int r0 = r.row0 & ~7, end = r.row0 + r.rows; r0 < end;) {
                const int in_block = r0 % WIDE_BLOCK, n = std::min(std::min(scratch_rows_, end - r0), WIDE_BLOCK - in_block);
                AttnArgs at = attn_args(l, n, wide_.q + (size_t)r0 * qdim_, row_pos + r0, row_seq + r0);
                at.xp_out = wide_.att + (size_t)(r0 / WIDE_BLOCK) * wide_block_bytes(qdim_) + (size_t)in_block * 128;
                at.xp_mpad = WIDE_BLOCK;
                ce = launch_attn_decode(at, n, kv_bf16_, stream_, pdl_);
                if (ce != cudaSuccess) return cuda_fail(ce, "attention launch");
                ++*launches;
                r0 += n;
            }
        WideArgs o{};
        o.resid = wide_.h;
        o.y = wide_.h;
        o.ldy = H_;
        o.xp_out = wide_.x2;
        o.next_norm_w = w.post_ln;
        o.ss_out = wide_.ss2;
        ce = project(w.o, wide_.att, EPI_STORE, o);
        if (ce != cudaSuccess) return cuda_fail(ce, "wide output projection");
        WideArgs gu{};
        gu.ss_in = wide_.ss2;
        gu.xp_out = wide_.act;
        ce = project(w.gu, wide_.x2, EPI_SWIGLU, gu);
        if (ce != cudaSuccess) return cuda_fail(ce, "wide gate/up projection");
        WideArgs dn{};
        dn.resid = wide_.h;
        dn.y = wide_.h;
        dn.ldy = H_;
        if (l + 1 < L_) {
            dn.xp_out = wide_.x;
            dn.next_norm_w = layers_[l + 1].in_ln;
            dn.ss_out = wide_.ss;
        }
        ce = project(w.down, wide_.act, EPI_STORE, dn);
        if (ce != cudaSuccess) return cuda_fail(ce, "wide down projection");
        if (tap_) HM_CUDA(cudaMemcpyAsync(tap_ + ((size_t)l * tap_rows_ + tap_row0_) * H_, wide_.h, (size_t)M * H_ * 4, cudaMemcpyDeviceToHost, stream_));
    }
    return HM_OK;
}

}  // namespace hm
