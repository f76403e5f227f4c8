// Launch shapes of decode steps and prompt chunks that follow from sizes alone: plain C++, so that their rules can be held to on the CPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <numeric>
#include <vector>

namespace mlb {

// Sequences that a CTA of the streamed GEMV takes its slab of rows for, one to three. A CTA has an SM to itself, so taking more sequences pays
// where it saves a wave of CTAs, and only there: the fewest waves that groups of three allow, with the sequences shared out evenly over
// them (a CTA computes its whole group, present or not), and smaller groups where their CTAs fit the SMs side by side. Steps on the fp32
// model of 512 x 8 (QKV cut by heads: 32 slabs; gate/up 141, LM head 148), at 2 / 3 / 4 sequences: min(batch, 3) to a CTA everywhere
// 282 / 319 / 419 us, one 258 / 293 / 365, this rule 254 / 262 / 336.
inline int sg_sequences(int batch, int slabs, int sm_count) {
    const int rows = std::max((batch + 2) / 3, std::min(batch, sm_count / std::max(1, slabs)));
    return (batch + rows - 1) / rows;
}

// Decode attention: one CTA takes all splits of a sequence and group of query heads, in turn, where the sequences and groups alone fill the
// SMs; else every split has a CTA. (Figures at attn_grid.)
constexpr int kAttnLoopSplits = 4;                 // most splits that one CTA takes in turn
inline bool attn_splits_in_turn(int splits, long sequence_groups, int sm_count) { return splits <= kAttnLoopSplits && sequence_groups >= sm_count; }

// Shared memory of decode attention: a ring of two stages of K and V rows for each of four streams of pages, the streams' and the splits' results.
// A stage is a page of 16 rows, or fewer rows where that lets the CTAs which registers leave room for stand side by side on an SM: with pages
// alone fp32 rows of 128 took 132 KB, one CTA per SM (64 sequences of 300 positions, 8 heads: 48.4 us in one split, 143 in eight; 35.0 and
// 49.6 with stages of 4 rows), of 64 with one head per CTA 68 KB, three for five (24.2, 50.0 -> 19.8, 37.4 with 8). Where the launch has too few
// CTAs for that, pages stay: a stage costs a wait and a hand-back (one sequence of 1000 positions, rows of 128: 28.1 us with pages, 33.5 with 4 rows).
constexpr int kAttnStreams = 4, kAttnStages = 2, kAttnPageRows = 16;
constexpr int attn_resident(int heads) { return heads == 1 ? 5 : (heads == 2 ? 3 : (heads == 4 ? 2 : 1)); }      // CTAs per SM, by registers
constexpr long attn_smem(int kv_bytes, int head_dim, int heads, int rows) {
    return (long)kAttnStreams * kAttnStages * 2 * rows * head_dim * kv_bytes + (long)(kAttnStreams + kAttnLoopSplits) * heads * (head_dim + 2) * 4;
}
// rows per stage where pages leave too little room; bf16 pages leave it, or gain nothing from less (rows of 128, one head: 139 us with pages, 149 with 8)
constexpr int attn_few_rows(int kv_bytes, int head_dim, int heads) {
    return kv_bytes == 2 || heads == 8 || (head_dim == 64 && heads > 1) ? kAttnPageRows : (head_dim == 128 && heads == 1 ? 4 : 8);
}
// CTAs with work where contexts fill half of the page table: a split with fewer than min_pages has none (8 sequences of 200 of 1024 positions, 8 heads:
// 64 of 640 CTAs, which pages serve better: 601 us a step, 613 with 8 rows).
inline long attn_ctas_with_work(long sequence_groups, int grid_splits, int table_pages, int min_pages) {
    return sequence_groups * std::min(grid_splits, std::max(1, table_pages / 2 / std::max(1, min_pages)));
}
inline bool attn_whole_pages(int kv_bytes, int head_dim, int heads, long ctas, int sm_count) {
    const long per_sm = std::min<long>(attn_resident(heads), (ctas + sm_count - 1) / sm_count);
    return attn_few_rows(kv_bytes, head_dim, heads) == kAttnPageRows ||
           attn_smem(kv_bytes, head_dim, heads, kAttnPageRows) <= 227 * 1024 / per_sm - 2048;      // (static shared memory, the system's share)
}

// Ring of a decode GEMM CTA. Two CTAs per SM share its shared memory, so that the next launch's weights arrive under this one. Where there are
// more CTAs than two per SM, a CTA's own chain of barriers, operands and epilogue bounds the launch, and more of them side by side hide
// it: a quarter or half of the ring, the least that holds two stages. LM heads of 256 sequences: 8192 x 512, stages of 12 KB, 35.5 us with
// whole rings, 15.3 with quarters; step of four layers with 384 or 304 CTAs in one projection, whole / half / quarter (two, two, one
// stage of 24 KB): QKV of 3072 x 1024 357 / 332 / 344 us, residual of 2432 x 896 616 / 584 / 606; QKV of 3072 x 2432 (48 KB: 2, 1, 1)
// 560 / 605 / 605. Gate/up keeps the whole ring: its CTAs have twice the warps and operands (3584 x 512, 448 CTAs: 241 / 249 / 249 us, e4m3
// 277 / 293 / 307).
inline size_t gd_ring(size_t whole, long ctas, int sm_count, bool gate_up, size_t two_stages) {
    if (ctas <= 2L * sm_count || gate_up) return whole;
    return two_stages <= whole / 4 ? whole / 4 : (two_stages <= whole / 2 ? whole / 2 : whole);
}

// What a prompt chunk of `want` columns takes of each sequence: rest[b] tokens wait, cursor[b] were taken before. The largest equal share that
// fits; what is left over goes to the first sequences, one token each. With attention tiles of `tile` > 0 queries a share that ends inside one
// leaves the tile's other rows idle (256 sequences: 16 of 32 rows of every tile). It is rounded up to whole tiles, for as many of the sequences
// furthest behind as then fit, the last of them with what room there is: the chunk is full either way, so that a prompt takes no more
// chunks (request of 256 prompts of 256 tokens, 8 heads of 64: 104.7 -> 95.5 ms).
inline void cols_shares(const std::vector<int>& rest, const std::vector<int>& cursor, int want, int tile, std::vector<int>& take) {
    const int B = (int)rest.size();
    take.assign(B, 0);
    auto filled = [&](int share) {
        long n = 0;
        for (int r : rest) n += std::min(share, r);
        return n;
    };
    int lo = 0, hi = want;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (filled(mid) <= want) lo = mid; else hi = mid - 1;
    }
    int extra = want - (int)filled(lo);
    const bool all = std::all_of(rest.begin(), rest.end(), [&](int r) { return r <= lo; });
    if (tile > 0 && !all && lo > 0 && (lo % tile || extra > 0)) {
        const int share = (lo / tile + 1) * tile;      // (more than fits for all)
        std::vector<int> order(B);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cursor[x] < cursor[y]; });
        int room = want;
        for (const int b : order) {
            take[b] = std::min(std::min(rest[b], share), room);
            room -= take[b];
        }
    } else {
        for (int b = 0; b < B; ++b) {
            take[b] = std::min(rest[b], lo);
            if (extra > 0 && take[b] < rest[b]) { ++take[b]; --extra; }
        }
    }
}

}  // namespace mlb
