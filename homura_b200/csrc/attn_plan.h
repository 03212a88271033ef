// How the attention launches of steps and small passes over the paged cache are cut (attention.cu).  Host only and free of CUDA.
#pragma once
#include <algorithm>

namespace hm {

constexpr int ATT_ST_MIN_PAGES = 16;  // pages per CTA from which the streaming variant is used (in clusters: attn_stream_from)

// Splits per (row, KV head) through global scratch: minimise waves x (fixed cost per CTA + pages per CTA) + merge cost.
// Units are "pages streamed by one CTA": the fixed cost (launch, query and page-table loads) is
// worth about eight pages, merging one more partial about half a page.  The streaming variant
// (>= ATT_ST_MIN_PAGES pages per CTA) keeps two CTAs per SM resident, the short-context kernel four.
// max_pages is the capacity the launch is sized for (a captured graph cannot follow the length).
inline int attn_pick_nsplit(int M, int kv_heads, int max_pages, int sm_count, bool bf16_pages) {
    const long pairs = (long)M * kv_heads;
    int cap = (max_pages + 1) / 2;  // at least two pages per split
    if (cap > sm_count) cap = sm_count;
    if (cap < 1) cap = 1;
    int best = 1;
    long best_cost = -1;
    for (int n = 1; n <= cap; ++n) {
        const int ppc = (max_pages + n - 1) / n;
        const bool streaming = ppc >= ATT_ST_MIN_PAGES;
        const long slots = (streaming ? 2L : 4L) * sm_count;
        const long waves = (pairs * n + slots - 1) / slots;
        // doubled so that the half page per partial stays an integer; a page costs the short-context
        // kernel about twice what it costs the streaming one (every query head re-reads the tile)
        // having any split at all costs a round trip of the partial triples through global memory, a ticket and a
        // second merge by the last CTA: about twenty pages' worth (64 sequences at 36 pages: one split 15.4 us, two 17.1)
        // a streaming launch that leaves every CTA an SM to itself gets the deep page ring (launch_tc), which about
        // halves what a page costs its CTA while the cache is short (measured on bf16 pages: 64 x 2 CTAs at 43 pages, one
        // split 11.9 us, two 18.7); on long caches two CTAs per SM stream faster than one with a deep ring, and on f32
        // pages fewer splits lost at every length
        const bool deep = streaming && bf16_pages && max_pages <= 64 && pairs * n <= sm_count;
        const long cost = 2 * waves * (8 + (streaming ? ppc : 2 * ppc)) / (deep ? 2 : 1) + (deep ? 8 : 0) + n + (n > 1 ? 40 : 0);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = n;
        }
    }
    return best;
}

// Pages per CTA from which the streaming kernel takes a launch in clusters: its warps take whole pages for all query heads, the short kernel's a head each.
// two_fit: its shared memory leaves room for two CTAs per SM.  early: a row per sequence, pages are read ahead of the wait.  Short and streaming kernel:
// - Up to a CTA per SM, from three pages on.  ms per step: 1.5 B with 1000 tokens (four pages) 1.29 and 1.22, bf16 pages 1.30 and 1.16; TinyLlama Q8_0 0.67 and 0.65;
//   two sequences of the 0.5 B stack with 900 0.66 and 0.61; one of bf16 pages with 1000 0.56 and 0.535.  One sequence on f32 pages of more than four
//   64-wide heads (32 CTAs) from five on: 0.5 B, four pages 0.555 and 0.563, five 0.583 and 0.572.  CTAs that cannot share an SM (f32 pages of 128-wide heads)
//   from five on where there are more than 64: 0.6 B, three pages 0.71 and 0.75, five 0.77 and 0.76; four sequences of 1.5 B on bf16 pages, four 1.71 and 1.77.
// - More CTAs than SMs, 64-wide heads, up to four rows: the next launch streams its weights into the shared memory that a ring would take.  us per layer, four
//   sequences of 1000 on four KV heads of three 31.1 and 34.4 (f32 pages), of eight 37.6 and 43.0; seven pages 32.6 and 33.6.
// - More, and more rows, steps: eight sequences, us per layer, four pages of one head 39.7 and 37.3, of eight 44.6 and 46.4, five of eight 49.0 and 47.8; bf16 pages,
//   four of eight 45.4 and 43.6.
// - More, rows that may not read ahead (prompt chunks, mixed batches): f32 pages, chunks of 40 rows on 128-wide heads, five pages 67.8 and 70.9, eight 77.9 and 74.4; on
//   64-wide ones eight 64.0 and 65.0, thirteen 71.4 and 69.3; eight sequences, five 60.0 and 61.2, seven 64.4 and 62.7.  bf16 pages, 64-wide, chunks,
//   four 55.6 and 59.1, five 59.1 and 58.9.
inline int attn_stream_from(int hd, bool bf16, int group, int M, long ctas, bool early, bool two_fit, int sms) {
    if (ctas > sms) {
        if (hd == 64 && M <= 4) return ATT_ST_MIN_PAGES;
        if (!bf16 && !early) return hd == 128 ? 8 : M <= 16 ? 7 : 10;
        if (hd == 64) return early && (bf16 || group <= 2) ? 3 : 5;
    }
    if (hd == 64) return !bf16 && group > 4 && ctas <= 32 ? 5 : 3;
    return ctas > 64 && !two_fit ? 5 : 3;
}

// One launch: splits of a (row, KV head), and whether they are a cluster.
struct AttnCut {
    int nsplit;
    bool cluster;
    int early_pages;  // AttnArgs::early_pages
};

// What a cache's shape decides (made with the cache), and what a launch of M rows adds to it.
struct AttnPlan {
    int kvh = 1, group = 1, hd = 64, max_pages = 1, sms = 148;
    bool bf16 = false;
    int by_pages = 1;             // splits of a cluster: a page each while the cache is short
    int batch_splits = 1;         // of a pass of as many rows as there are sequences through global scratch
    bool cluster = false;         // passes with several rows of a sequence (prompt chunks, mixed batches)
    bool decode_cluster = false;  // steps: a row per sequence

    AttnPlan() = default;
    AttnPlan(int batch, int heads, int kvh_, int hd_, bool bf16_, int pages, int sm_count, bool use_clusters, int max_cluster) : kvh(kvh_), group(heads / kvh_), hd(hd_), max_pages(pages), sms(sm_count), bf16(bf16_) {
        const long pairs = (long)batch * kvh;
        by_pages = std::max(1, std::min(pages, std::min(max_cluster, 16)));
        batch_splits = attn_pick_nsplit(batch, kvh, pages, sms, bf16);
        // up to 1024 tokens of capacity the splits of a (row, KV head) are one cluster of at most 16 CTAs, one page
        // per split while the context allows (a page is about 0.65 us of dependent instructions, so pages of a
        // split cost more than the wider merge); longer caches need more CTAs than a cluster holds and merge
        // through global scratch + ticket
        // ... and only while the (row, KV head) pairs alone do not fill the GPU: with half an SM's worth of pairs or more
        // the launch is a throughput problem (64 sequences stream 39 MB of pages per layer), which the cost model
        // of attn_pick_nsplit answers with few splits of many pages each, i.e. the bulk-copy ring kernel
        cluster = use_clusters && pages <= 64 && pairs < sms / 2;
        // Decode passes of few (row, KV head) pairs stay clusters of sixteen CTAs on longer caches too (the streaming kernel from a few pages per CTA on, launch_tc): ms per
        // step with splits through global scratch and so, 1.5 B with 1200 tokens 1.62 and 1.23, 2000 1.63 and 1.25 (bf16 pages 1.48 and 1.17), 4000 1.53 and
        // 1.38; 0.5 B 1200 0.79 and 0.59, 4000 0.71 and 0.63; TinyLlama Q8_0 2000 0.76 and 0.67; two sequences of 1.5 B, 1500 1.70 and 1.29.  Eight pairs are 128 CTAs,
        // which must share SMs to be eight clusters at once: f32 pages of 128-wide heads do not fit twice (0.6 B with 1200 0.85 and 0.78, 2000 0.76 and 0.79, 4000 0.81 and
        // 0.96).  On bf16 pages they do, but rank 0 of a cluster takes 16 results per query head and dimension: with six or eight heads of 128 per KV head
        // longer caches are slower (1.5 B, four sequences of 4000 1.81 and 1.95 ms; us per layer at 2500 43.2 and 44.4, of eight heads, two sequences 42.3 and 40.6).
        const int reach = pairs <= 4 ? 256 : pairs <= 8 ? (hd == 64 || (bf16 && group <= 4) ? 256 : bf16 ? 160 : 80) : 64;
        decode_cluster = use_clusters && pages <= reach && pairs < sms / 2;
    }

    // Splits that the scratch of a row must hold: of every launch that goes through it.
    int scratch_splits() const { return cluster || decode_cluster ? std::max(by_pages, batch_splits) : batch_splits; }

    // AttnArgs::early_pages of a decode pass: one row per sequence (prefill chunks write several positions of one sequence).  Launches of at most two CTAs
    // per SM may keep the pages of a split (eight at most) in slots of their own, which takes the loads in front of the wait; but shared memory keeps the next
    // projection's CTAs, whose weights arrive meanwhile, off those SMs, and a page of 128-wide heads is 16 KB of it.  One slot per split and up to eight:
    // - 64-wide heads: 0.5 B stack, one sequence, two pages per CTA 0.506 and 0.490 ms per step, four of them (32 CTAs) 0.555 and 0.576; four sequences of 1000 0.82 and 0.80.
    // - 128-wide heads in clusters, launches of 32 CTAs: us per layer of eight heads and 300 tokens 22.2 and 23.4; of up to 64: 1.5 B, two sequences of 800
    //   1.43 and 1.36 ms; of more: four of 1000 1.69 and 2.00 ms, but with two pages per CTA 35.3 and 33.5 us per layer of four of 300 (bf16 pages).
    // - 128-wide heads through global scratch, us per layer: eight sequences of 1100 on two KV heads of eight 69 and 64, two of 1100 on eight of three 44 and 39;
    //   where the CTA works on four pages at a time anyway (one or two heads per KV head) 36.8 and 39.2.
    int early(long ctas, int pages_per_cta, bool in_cluster) const {
        if (ctas > 2L * sms) return 1;
        if (hd == 64) return in_cluster && ctas <= 32 && pages_per_cta > 2 ? 2 : 9;
        if (!in_cluster) return group > 2 || ctas <= 64 ? 9 : 2;
        return ctas <= 32 || (ctas > 64 && pages_per_cta > 2) ? 2 : 9;
    }

    AttnCut cut(int M, bool decode) const {
        AttnCut c;
        c.cluster = decode ? decode_cluster : cluster;
        // Fewer splits where the rows alone fill the SMs: about two CTAs per SM in clusters, the kernel's cost model otherwise.  The model knows neither
        // that the rows of a prompt share their pages nor what the merge of so many partials costs: it is held to the splits of a step (a 40-row chunk
        // behind 1500 tokens of the 1.5 B shapes, bf16 pages: 77 us per layer with the step's 7 splits at most, 143 with the 16 of its clusters).
        c.nsplit = c.cluster ? std::min(by_pages, std::max(1, (2 * sms + M * kvh - 1) / (M * kvh))) : std::min(batch_splits, attn_pick_nsplit(M, kvh, max_pages, sms, bf16));
        c.early_pages = !decode ? 0 : early((long)M * kvh * c.nsplit, (max_pages + c.nsplit - 1) / c.nsplit, c.cluster);
        return c;
    }
};

// A cluster wants that many SMs of one GPC at once, with the shared memory of its CTAs free: where the device has no room for a launch that a plan holds (fits) its
// clusters are eight CTAs, and there are none where these do not fit either.
template <class Fits>
AttnPlan attn_plan_that_fits(int batch, int heads, int kvh, int hd, bool bf16, int pages, int sm_count, bool use_clusters, int max_cluster, Fits fits) {
    for (int most : {max_cluster, 8}) {
        const AttnPlan p(batch, heads, kvh, hd, bf16, pages, sm_count, use_clusters, most);
        if ((!p.cluster && !p.decode_cluster) || fits(p)) return p;
    }
    return AttnPlan(batch, heads, kvh, hd, bf16, pages, sm_count, false, 8);
}

}  // namespace hm
