// Pages shared by the sequences of an engine, and the step over portions of several sequences (every design).
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

#include "engine.h"
#include "engine_util.h"
#include "gemm_tc.h"

namespace hm {

// The logits of a large batch (39 MB for 64 rows of 151,936) land in memory that the caller has just been given: one thread is bound by
// the page faults of its first touch (12 ms), eight take 2 ms.  Up to 4 MB one thread is as fast.
void copy_out(void* dst, const void* src, size_t bytes) {
    constexpr size_t SMALL = 4u << 20, MOST = 8;
    const size_t n = bytes <= SMALL ? 1 : std::min<size_t>(MOST, std::max(1u, std::thread::hardware_concurrency()));
    const size_t per = ((bytes + n - 1) / n + 4095) / 4096 * 4096;
    auto part = [=](size_t i) {
        const size_t lo = std::min(bytes, i * per), hi = std::min(bytes, lo + per);
        std::memcpy((char*)dst + lo, (const char*)src + lo, hi - lo);
    };
    std::thread helpers[MOST - 1];
    size_t started = 0;
    try {
        for (; started + 1 < n; ++started) helpers[started] = std::thread(part, started + 1);
    } catch (...) {  // no more threads to be had: the rest is copied here
    }
    part(0);
    for (size_t i = started + 1; i < n; ++i) part(i);
    for (size_t i = 0; i < started; ++i) helpers[i].join();
}

// A caller's fresh array of logits is 149 pages per row of 151,936, each a fault when it is first written: 0.1 ms of a 0.68 ms step of one
// sequence.  In pieces, so that it ends when the stream does; a kernel without MADV_POPULATE_WRITE leaves them to the copy.
void touch_out(void* dst, size_t bytes, cudaStream_t stream) {
#ifdef MADV_POPULATE_WRITE
    constexpr int POPULATE = MADV_POPULATE_WRITE;
#else
    constexpr int POPULATE = 23;
#endif
    constexpr size_t PIECE = 1u << 20;
    const uintptr_t page = 4095, end = ((uintptr_t)dst + bytes + page) & ~page;
    for (uintptr_t at = (uintptr_t)dst & ~page; at < end; at += PIECE) {
        if (madvise((void*)at, std::min<size_t>(PIECE, end - at), POPULATE) != 0 || cudaStreamQuery(stream) != cudaErrorNotReady) break;
        cudaGetLastError();  // "not ready" is not an error of the next launch
    }
}

// ---- pages ------------------------------------------------------------------------------------------

// Gives every listed sequence the pages for the tokens it will hold.  All or nothing: HM_ERR_KV_FULL when the pool is short.
int Engine::ensure_pages(const std::vector<std::pair<int, long>>& need) {
    if (!pooled_) return HM_OK;
    size_t missing = 0;
    for (auto& n : need) {
        const size_t pages = (size_t)(n.second + page_tokens_ - 1) / page_tokens_, have = seq_pages_[n.first].size();
        if (pages > (size_t)max_pages_) return fail(HM_ERR_KV_FULL, "KV cache full (sequence longer than max_seq_len)");
        if (pages > have) missing += pages - have;
    }
    if (missing > free_pages_.size())
        return fail(HM_ERR_KV_FULL, "KV cache full (" + std::to_string(missing) + " more pages wanted, " + std::to_string(free_pages_.size()) + " free in the pool)");
    for (auto& n : need) {
        std::vector<int32_t>& own = seq_pages_[n.first];
        const size_t pages = (size_t)(n.second + page_tokens_ - 1) / page_tokens_, first = own.size();
        if (pages <= first) continue;
        for (size_t i = first; i < pages; ++i) {
            own.push_back(free_pages_.back());
            free_pages_.pop_back();
        }
        HM_CUDA(cudaMemcpyAsync(page_table_ + (size_t)n.first * max_pages_ + first, own.data() + first, (pages - first) * 4, cudaMemcpyHostToDevice, stream_));
    }
    return HM_OK;
}

int Engine::ensure_pages_all(int more) {
    if (!pooled_) return HM_OK;
    std::vector<std::pair<int, long>> need;
    for (int b = 0; b < batch_; ++b) need.push_back({b, (long)len_[b] + more});
    return ensure_pages(need);
}

void Engine::release_pages(int seq) {
    if (!pooled_) return;
    std::vector<int32_t>& own = seq_pages_[seq];
    while (!own.empty()) {
        free_pages_.push_back(own.back());
        own.pop_back();
    }
}

int Engine::kv_free_tokens(long* out) {
    if (!out) return fail(HM_ERR_INVALID, "kv_free_tokens: null output");
    if (batch_ == 0 || !pooled_) return fail(HM_ERR_STATE, "kv_free_tokens: the cache has no shared pool");
    *out = (long)free_pages_.size() * page_tokens_;
    return HM_OK;
}

// ---- step ---------------------------------------------------------------------------------------------

int Engine::tap(int layer, int M) {
    if (!tap_ || only_class_ >= 0) return HM_OK;
    HM_CUDA(cudaMemcpyAsync(tap_ + ((size_t)layer * tap_rows_ + tap_row0_) * H_, h_, (size_t)M * H_ * 4, cudaMemcpyDeviceToHost, stream_));
    return HM_OK;
}

int Engine::step(const hm_step_entry* entries, int n, float* logits, uint32_t* greedy, float* hidden) {
    if (!set_device()) return fail(HM_ERR_CUDA, "cudaSetDevice failed");
    if (batch_ == 0) return fail(HM_ERR_STATE, "step before kv_alloc");
    if (!entries || n < 1) return fail(HM_ERR_INVALID, "step: bad arguments");
    size_t rows = 0, wants = 0;
    std::vector<char> seen(batch_, 0);
    std::vector<std::pair<int, long>> need;
    for (int i = 0; i < n; ++i) {
        const hm_step_entry& e = entries[i];
        if (e.seq < 0 || e.seq >= batch_ || seen[e.seq]) return fail(HM_ERR_INVALID, "step: sequence index out of range or named twice");
        seen[e.seq] = 1;
        if (e.n_tokens < 1 || !e.tokens || e.n_want < 0 || (e.n_want > 0 && !e.want)) return fail(HM_ERR_INVALID, "step: bad entry");
        for (int k = 0; k < e.n_tokens; ++k)
            if (e.tokens[k] >= (uint32_t)V_) return fail(HM_ERR_INVALID, "step: token id out of range");
        for (int k = 0; k < e.n_want; ++k)
            if (e.want[k] < 0 || e.want[k] >= e.n_tokens || (k > 0 && e.want[k] <= e.want[k - 1])) return fail(HM_ERR_INVALID, "step: wanted places must ascend within the portion");
        if ((long)len_[e.seq] + e.n_tokens > max_seq_)
            return fail(HM_ERR_KV_FULL, "KV cache full (" + std::to_string(len_[e.seq]) + " + " + std::to_string(e.n_tokens) + " > " + std::to_string(max_seq_) + ")");
        need.push_back({e.seq, (long)len_[e.seq] + e.n_tokens});
        rows += e.n_tokens;
        wants += e.n_want;
    }
    const int prc = ensure_pages(need);
    if (prc) return prc;
    HM_CUDA(cudaStreamSynchronize(stream_));
    // staging: tokens, positions, sequences [rows]; wanted rows (index within their pass) and greedy results [rows]; new lengths [batch]
    if (rows > st_rows_) {
        const size_t cap = std::max<size_t>(rows, 256);
        auto re = [&](auto** p) -> cudaError_t {
            if (*p) cudaFree(*p);
            *p = nullptr;
            return dev_alloc((void**)p, cap * 4);
        };
        st_rows_ = 0;
        HM_CUDA(re(&st_tokens_));
        HM_CUDA(re(&st_pos_));
        HM_CUDA(re(&st_seq_));
        HM_CUDA(re(&st_want_));
        HM_CUDA(re(&st_next_));
        if (st_pin_) cudaFreeHost(st_pin_);
        st_pin_ = nullptr;
        HM_CUDA(cudaMallocHost(&st_pin_, (5 * cap + 2 * (size_t)batch_) * 4));
        st_rows_ = cap;
    }
    uint32_t *p_tok = st_pin_, *p_pos = p_tok + st_rows_, *p_seq = p_pos + st_rows_, *p_want = p_seq + st_rows_, *p_next = p_want + st_rows_, *p_len = p_next + st_rows_;
    const int chunk = std::min(TC_ROWS, scratch_rows_);
    size_t r = 0, q = 0;
    for (int i = 0; i < n; ++i) {
        const hm_step_entry& e = entries[i];
        for (int k = 0; k < e.n_tokens; ++k, ++r) {
            p_tok[r] = e.tokens[k];
            p_pos[r] = (uint32_t)(len_[e.seq] + k);
            p_seq[r] = (uint32_t)e.seq;
        }
        p_len[2 * i] = (uint32_t)(len_[e.seq] + e.n_tokens);
    }
    WidePlan plan;
    if (const int wrc = plan_wide(p_pos, p_seq, (int)rows, &plan)) return wrc;
    wide_rows_ = plan.rows;
    // passes: the wide ones, then chunks; wanted rows as indices within their pass
    struct Pass { size_t row0; int rows, wants, longest; };
    std::vector<Pass> passes;
    for (const WidePass& w : plan.passes) passes.push_back({(size_t)w.row0, w.rows, 0, 0});
    for (size_t c0 = plan.rows; c0 < rows; c0 += chunk) passes.push_back({c0, (int)std::min<size_t>(chunk, rows - c0), 0, 0});
    r = 0;
    size_t at = 0;
    for (int i = 0; i < n; ++i) {
        const hm_step_entry& e = entries[i];
        int w = 0;
        for (int k = 0; k < e.n_tokens; ++k, ++r) {
            while (r >= passes[at].row0 + passes[at].rows) ++at;
            Pass& p = passes[at];
            p.longest = std::max(p.longest, len_[e.seq] + k + 1);
            if (w < e.n_want && e.want[w] == k) {
                p_want[q++] = (uint32_t)(r - p.row0);
                p.wants++;
                ++w;
            }
        }
    }
    HM_CUDA(cudaMemcpyAsync(st_tokens_, p_tok, rows * 4, cudaMemcpyHostToDevice, stream_));
    HM_CUDA(cudaMemcpyAsync(st_pos_, p_pos, rows * 4, cudaMemcpyHostToDevice, stream_));
    HM_CUDA(cudaMemcpyAsync(st_seq_, p_seq, rows * 4, cudaMemcpyHostToDevice, stream_));
    if (wants) HM_CUDA(cudaMemcpyAsync(st_want_, p_want, wants * 4, cudaMemcpyHostToDevice, stream_));
    float* land = logits && wants ? logits_landing(logits, wants * V_ * 4) : nullptr;
    int launches = 0, rc = HM_OK;
    size_t done = 0;
    tap_ = hidden;
    tap_rows_ = rows;
    auto logits_out = [&](int nw) -> int {  // the wanted rows that the pass enqueued last left in logits_
        if (!logits || !nw) return HM_OK;
        const cudaError_t ce = cudaMemcpyAsync(land + done * V_, logits_, (size_t)nw * V_ * 4, cudaMemcpyDeviceToHost, stream_);
        return ce == cudaSuccess ? HM_OK : cuda_fail(ce, "logits copy");
    };
    for (size_t i = 0; i < passes.size() && rc == HM_OK; ++i) {
        const size_t c0 = passes[i].row0;
        const int mc = passes[i].rows, nw = logits || greedy ? passes[i].wants : 0;
        tap_row0_ = c0;
        if (i < plan.passes.size()) {
            rc = enqueue_wide(plan, plan.passes[i], st_tokens_ + c0, st_pos_ + c0, st_seq_ + c0, &launches);
            for (int w = 0; w < nw && rc == HM_OK; w += chunk) {
                const int g = std::min(chunk, nw - w);
                const cudaError_t ce = launch_gather_rows(wide_.h, st_want_ + done, g, H_, hsel_, stream_, pdl_);
                rc = ce == cudaSuccess ? enqueue_logits(hsel_, g, false, false, st_next_ + done, nullptr, nullptr, nullptr, &launches) : cuda_fail(ce, "gather_rows");
                if (rc == HM_OK) rc = logits_out(g);
                done += g;
            }
            continue;
        }
        pass_longest_ = passes[i].longest;
        pass_runs_.clear();
        for (int m = 0; m < mc; ++m) {  // a sequence's tokens are consecutive, so its rows within the pass are one run
            if (m > 0 && p_seq[c0 + m] == p_seq[c0 + m - 1]) pass_runs_.back().second++;
            else pass_runs_.push_back({m, 1});
        }
        lm_pick_ = nw ? st_want_ + done : nullptr;
        rc = enqueue_pass(mc, st_tokens_ + c0, st_pos_ + c0, st_seq_ + c0, 0, nw, false, st_next_ + done, nullptr, nullptr, nullptr, &launches);
        if (rc == HM_OK) rc = logits_out(nw);
        done += nw;
    }
    pass_runs_.clear();
    tap_ = nullptr;
    lm_pick_ = nullptr;
    if (rc) return rc;
    for (int i = 0; i < n; ++i) {
        const int seq = entries[i].seq;
        HM_CUDA(cudaMemcpyAsync(pos_dev_ + seq, p_len + 2 * i, 4, cudaMemcpyHostToDevice, stream_));
        // what follows a prompt's portion counts as generated for the sampler's penalties
        if (entries[i].n_tokens > 1 || len_[seq] == 0) HM_CUDA(cudaMemcpyAsync(smp_gen_start_ + seq, p_len + 2 * i, 4, cudaMemcpyHostToDevice, stream_));
    }
    if (greedy && wants) HM_CUDA(cudaMemcpyAsync(p_next, st_next_, wants * 4, cudaMemcpyDeviceToHost, stream_));
    if (int qrc = queue_error_copy()) return qrc;
    if (land && land != logits) touch_out(logits, wants * V_ * 4, stream_);
    HM_CUDA(cudaStreamSynchronize(stream_));
    rc = check_device_error();
    if (rc) return rc;
    if (land && land != logits) copy_out(logits, land, wants * V_ * 4);
    if (greedy && wants) std::memcpy(greedy, p_next, wants * 4);
    for (int i = 0; i < n; ++i) {
        const int seq = entries[i].seq;
        if (entries[i].n_tokens > 1 || len_[seq] == 0) gen_start_[seq] = len_[seq] + entries[i].n_tokens;
        len_[seq] += entries[i].n_tokens;
    }
    return HM_OK;
}

}  // namespace hm
