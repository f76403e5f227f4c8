// Launch shapes of a decode step that follow from sizes alone: plain C++, so that their rules can be held to on the CPU.
#pragma once
#include <algorithm>

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

}  // namespace mlb
