// ------------------------------------------------------------------------------------
// Split-K flash-decode over the paged KV cache, with the split combine and the query
// gating in the same kernel.
//
// Reference ops replaced: K^T Q GEMM, getHeadDimScaledMaskedAttn, the max / sum / apply
// softmax kernels, V P GEMM, applyGatingToValueScaledAttnPostSoftmax
// (inference.cu:510-579, kernels :136-250). Scores are divided by sqrtf(head_dim) as there.
// grid = (splits or 1, kv_heads, B), block = 4 streams x the head groups of a kv head.
//
// A stream takes the pages w, w + 4, .. of a split (w = 0 .. 3). The 16 rows of a head in a page are one contiguous block, so
// one lane copies a page's K and V rows (or a half or a quarter of them: attn_few_rows) with two bulk copies into the stream's own ring of
// shared-memory stages: no registers hold loads in flight. With four query heads or more per kv head a stream has a warp per two of
// them, which share its ring.
// In a decode session the K/V rows of earlier tokens were written by earlier steps, which are complete when a step's first
// kernel starts (it is launched without overlap): only the page of the current position and the queries wait for the predecessor.
// The scores of four positions per lane group and GW heads are summed over the lanes by a butterfly that leaves every lane
// its share of them, so that a score is divided and its exponential taken once and not by every lane of the group. Sums,
// maxima and products are those of a butterfly over every score, in its order.
// What bounds it: with one head per kv head HBM and the start and end of each CTA (256 sequences of 320 positions, 8 heads of 64: 32.9 us,
// 5.1 TB/s; 36.8 with per-thread loads); with four the chain of a chunk (scores, butterfly, exponentials, products: 550 cycles) under
// few warps (64 sequences of 528, 16 heads over 4 of 128, three splits: 57.5 -> 27.7 us, 2.5 TB/s).
// ------------------------------------------------------------------------------------
#pragma once
#include <type_traits>

#include "ring.cuh"
#include "step_shapes.h"

namespace mlb {

struct AttnParams {
    const void* kpool; const void* vpool;     // [page][kv_heads][16][hd]
    const int* page_table; int pt_stride;
    const float* qbuf;      // [B][heads*hd]
    const float* gbuf;      // [B][heads*hd] sigmoid gates or null
    float* abuf;            // [B][heads*hd]
    bf16_t* abuf16;         // same values as the bf16 operand of a tensor-core O projection, or null
    int perm;               // features of abuf16 in perm16 order
    float* part;            // [B][heads][splits][hd+2]
    int* ticket;            // [B * gridDim.y]
    int heads, kv_heads;
    int hg;                 // CTAs per kv head along grid.y: each takes G of the kv head's query heads
    // A caller-owned page table (the operator entry points) is not trusted: with num_pages > 0 a sequence
    // whose position needs more than pt_stride pages is skipped (code 4 in *err) and a page id outside
    // [0, num_pages) is replaced by page 0 (code 5), so that nothing outside the caller's buffers is read.
    // The session passes 0: its own allocator filled the table.
    int num_pages;
    int* err;               // also the code of a wait that ran out
    // A split is worth its partials and the combine only with enough positions in it: a sequence uses
    // min(grid splits, pages / min_pages_per_split) of them. 1 = every page may be a split.
    int min_pages_per_split;
    int early;              // the K/V rows before the current position may be read before the predecessor kernel has ended
    int splits;             // most splits of a sequence: grid.x CTAs of one each, or (grid.x = 1) one CTA that takes them in turn
};

template <int G> constexpr int attn_heads_per_warp() { return G < 2 ? 1 : 2; }
template <int G> constexpr int attn_threads() { return 32 * (kAttnStreams * (G / attn_heads_per_warp<G>()) + 1); }      // and the producer warp

// Launch grid. One CTA for all splits of a sequence where there are CTAs enough without them: no partial results in global memory, no
// CTA that waits for others' tickets (64 sequences of 528 positions, 16 heads over 4 of 128, three splits: 26.7 us, 32 with a CTA each).
inline dim3 attn_grid(const AttnParams& p, int B, int sm_count) {
    const int groups = p.kv_heads * p.hg;
    return dim3(attn_splits_in_turn(p.splits, (long)groups * B, sm_count) ? 1 : p.splits, groups, B);
}

static_assert(kAttnPageRows == kKvBlock, "rows of a page");
// SR: rows of a page per stage (attn_few_rows)
template <typename KVT, int HD, int G, int SR>
__global__ void __launch_bounds__(attn_threads<G>(), attn_resident(G))
    attn_decode_kernel(const __grid_constant__ StepCtl c, const __grid_constant__ AttnParams p) {
    constexpr int EPL = 16 / sizeof(KVT);          // elements per lane per row
    constexpr int LPR = HD / EPL;                  // lanes per row
    constexpr int PPI = 32 / LPR;                  // positions per warp iteration
    constexpr int NW = kAttnStreams;
    constexpr int GW = attn_heads_per_warp<G>();   // heads of a warp
    constexpr int HG = G / GW;                     // warps of a stream
    constexpr int CH = 4;                          // positions per lane group handled together
    constexpr int RB = HD * (int)sizeof(KVT);      // bytes per row
    constexpr int N = GW * CH;                     // scores of a lane group,
    constexpr int D = LPR / N;                     // each kept by D lanes
    constexpr int GL = D * CH;                     // lanes that hold a head's scores
    constexpr int NST = kAttnStages;
    constexpr int SB = SR * RB;                    // bytes of K, and of V, per stage (SR rows of a page)
    constexpr int CPS = SR / PPI / CH;             // chunks per stage
    constexpr int W = HD + 2;
    static_assert(LPR <= 32 && PPI >= 1 && CPS >= 1 && kKvBlock % SR == 0 && D >= 1, "head_dim does not fit one warp row");
    extern __shared__ __align__(128) unsigned char attn_sm[];
    float* sred = reinterpret_cast<float*>(attn_sm + (size_t)NW * NST * 2 * SB);      // [stream][G][HD + 2] of a split
    float* spart = sred + NW * G * W;              // [split][G][HD + 2] where one CTA takes all splits
    __shared__ __align__(8) uint64_t bars[2 * NW * NST];
    __shared__ int is_last;
    const int b = blockIdx.z;
    pdl_launch_dependents();
    const bool early = p.early != 0 && c.seq_of == nullptr;
    if (!early) pdl_wait();                        // q and this step's K/V row come from the projection kernel
    // (the kernel behind this one counts on the projection to be complete as well: no CTA leaves before the wait)
    if (!seq_active(c, b)) {                       // uniform for all CTAs of this sequence
        pdl_wait();
        return;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w = warp / HG, hgrp = warp % HG;
    const int lr = lane % LPR, grp = lane / LPR;
    // An operator's caller may mark an idle sequence with a negative position: it has no pages, and nothing of its row of the table is read
    // (the producer copies nothing, the sums stay empty, the row becomes 0 / 0).
    const int ctx = c.pos[b] + 1;
    const int npages = c.pos[b] < 0 ? 0 : c.pos[b] / kKvBlock + 1;
    // The splits are sized for the longest context; a split needs at least one page, and the CTAs
    // beyond the page count leave at once (fewer partials for the combine to read). Every CTA of a
    // (sequence, kv head) computes the same S.
    if (p.num_pages > 0 && npages > p.pt_stride) {   // uniform for all CTAs of this sequence
        if (threadIdx.x == 0) atomicExch(p.err, 4);
        return;
    }
    const int S = max(1, min(p.splits, npages / max(1, p.min_pages_per_split)));
    const int SG = p.splits;                       // stride of the partial buffer, whatever S
    const bool loop = gridDim.x == 1 && p.splits > 1;      // one CTA takes all S splits
    if ((int)blockIdx.x >= S) {
        pdl_wait();
        return;
    }
    const int s_first = loop ? 0 : (int)blockIdx.x, s_end = loop ? S : s_first + 1;
    const int pps = (npages + S - 1) / S;
    // With many query heads per kv head and few CTAs, hg CTAs share a kv head, G heads each; the K/V rows they re-read come from L2.
    const int kvh = (int)blockIdx.y / p.hg, h0 = (kvh * p.hg + (int)blockIdx.y % p.hg) * G;
    // pages of stream w in split s: s * pps + w + NW * i
    auto pages_of = [&](int s) {
        const int span = min(npages, (s + 1) * pps) - s * pps - w;
        return span > 0 ? (span + NW - 1) / NW : 0;
    };

    // ---- producer: lane w asks for the pages of stream w, for all its splits, in order ----------------------------------------
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8u * NW * NST;      // [stream][stage]
    if (tid < NW * NST) {
        mbar_init(full0 + 8u * tid, 1);
        mbar_init(empty0 + 8u * tid, HG);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == NW * HG) {
        if (lane < NW) {
            const int* pt = p.page_table + kv_seq(c, b) * p.pt_stride;
            auto pool_index = [&](int pg) {
                int page = pt[pg];
                if (p.num_pages > 0 && (unsigned)page >= (unsigned)p.num_pages) {
                    atomicExch(p.err, 5);
                    page = 0;
                }
                return page;
            };
            const uint32_t ring0 = smem_u32(attn_sm) + (uint32_t)(lane * NST * 2 * SB), f0 = full0 + 8u * lane * NST, e0 = empty0 + 8u * lane * NST;
            bool waited = !early;
            int st = 0;
            uint32_t ph = 1;
            bool good = true;
            for (int s = s_first; s < s_end && good; ++s) {
                const int end = min(npages, (s + 1) * pps);
                int pg = s * pps + lane, page = pg < end ? pool_index(pg) : 0;
                for (; pg < end && good; pg += NW) {
                    const int next = pg + NW < end ? pool_index(pg + NW) : 0;      // on its way while this page waits for its stage
                    if (!waited && pg == npages - 1) {
                        pdl_wait();
                        waited = true;
                    }
                    const int rows = min(kKvBlock, ctx - pg * kKvBlock);
                    for (int r0 = 0; r0 < rows && good; r0 += SR) {
                        good = mbar_wait_bounded(e0 + 8u * st, ph, kRingSpinLimit, 0);
                        if (!good) break;          // (the consumers' waits run out and report it)
                        const uint32_t bytes = (uint32_t)(min(SR, rows - r0) * RB), bar = f0 + 8u * st;
                        const size_t at = (((size_t)page * p.kv_heads + kvh) * kKvBlock + r0) * RB;
                        mbar_expect_tx(bar, 2 * bytes);
                        bulk_g2s(ring0 + (uint32_t)(st * 2 * SB), static_cast<const unsigned char*>(p.kpool) + at, bytes, bar);
                        bulk_g2s(ring0 + (uint32_t)(st * 2 * SB + SB), static_cast<const unsigned char*>(p.vpool) + at, bytes, bar);
                        if (++st == NST) { st = 0; ph ^= 1u; }
                    }
                    page = next;
                }
            }
            if (!waited) pdl_wait();
        }
        return;
    }
    // the other warps; the producer takes no part in their barriers: it is pages ahead of them, or behind a full ring
    auto sync = []() { asm volatile("bar.sync 1, %0;" ::"n"(32 * NW * HG) : "memory"); };
    if (early) pdl_wait();
    unsigned char* ring = attn_sm + (size_t)w * NST * 2 * SB;
    const uint32_t my_full = full0 + 8u * w * NST, my_empty = empty0 + 8u * w * NST;
    bool ok = true;

    f32x2 q[GW][EPL];                              // every element twice: two positions at a time
#pragma unroll
    for (int g = 0; g < GW; ++g) {
        const float* qp = p.qbuf + ((size_t)b * p.heads + h0 + hgrp * GW + g) * HD + lr * EPL;
        float t[EPL];
        if ((reinterpret_cast<uintptr_t>(p.qbuf) & 15) == 0) {
#pragma unroll
            for (int e = 0; e < EPL; e += 4) {
                const float4 x = __ldcg(reinterpret_cast<const float4*>(qp + e));
                t[e] = x.x; t[e + 1] = x.y; t[e + 2] = x.z; t[e + 3] = x.w;
            }
        } else {                                   // an operator's caller may hand in any float pointer
#pragma unroll
            for (int e = 0; e < EPL; ++e) t[e] = __ldcg(qp + e);
        }
#pragma unroll
        for (int e = 0; e < EPL; ++e) q[g][e] = pack2(t[e], t[e]);
    }
    float m, l[GW];                                // m: of the head whose score this lane keeps
    f32x2 acc[GW][EPL / 2];
    const int src0 = lane - lr, own_u = (lr / D) % CH;
    // CH positions of every lane group; cnt: rows of the stage that hold a position (what lies behind them may be no number)
    auto use_chunk = [&](const unsigned char* kt, int cnt, int c0) {
        float s[N];
#pragma unroll
        for (int u = 0; u < CH; u += 2) {
            const unsigned char* row = kt + ((c0 + u) * PPI + grp) * RB + lr * 16;
            float k0[EPL], k1[EPL];
            Elem<KVT>::unpack(*reinterpret_cast<const uint4*>(row), k0);
            Elem<KVT>::unpack(*reinterpret_cast<const uint4*>(row + PPI * RB), k1);
#pragma unroll
            for (int g = 0; g < GW; ++g) {
                f32x2 d = 0ull;
#pragma unroll
                for (int e = 0; e < EPL; ++e) d = fma2(q[g][e], pack2(k0[e], k1[e]), d);
                unpack2(d, s[g * CH + u], s[g * CH + u + 1]);
            }
        }
#pragma unroll
        for (int o = LPR / 2, n = N / 2; o > 0; o >>= 1, n >>= 1) {
            if (n > 0) {
                const bool up = (lr & o) != 0;
#pragma unroll
                for (int j = 0; j < n; ++j) {
                    const float send = up ? s[j] : s[j + n], keep = up ? s[j + n] : s[j];
                    s[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            } else {
                s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
            }
        }
        const bool valid = (c0 + own_u) * PPI + grp < cnt;
        float x = valid ? (HD == 64 ? s[0] * 0.125f : s[0] / sqrtf((float)HD)) : kNegBig;
        float mn = fmaxf(m, x);
#pragma unroll
        for (int o = D; o < GL; o <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        const float sc = expf(m - mn);
        x = valid ? expf(x - mn) : 0.f;
        m = mn;
        if (__any_sync(0xffffffffu, sc != 1.0f)) {
#pragma unroll
            for (int g = 0; g < GW; ++g) {
                const float y = __shfl_sync(0xffffffffu, sc, src0 + g * GL);
                const f32x2 yy = pack2(y, y);
                l[g] = __fmul_rn(l[g], y);
#pragma unroll
                for (int e = 0; e < EPL / 2; ++e) acc[g][e] = mul2(acc[g][e], yy);
            }
        }
#pragma unroll
        for (int u = 0; u < CH; ++u) {
            uint4 raw = *reinterpret_cast<const uint4*>(kt + SB + ((c0 + u) * PPI + grp) * RB + lr * 16);
            if (cnt < SR && (c0 + u) * PPI + grp >= cnt) raw = make_uint4(0, 0, 0, 0);
            float vv[EPL];
            Elem<KVT>::unpack(raw, vv);
#pragma unroll
            for (int g = 0; g < GW; ++g) {
                const float y = __shfl_sync(0xffffffffu, x, src0 + (g * CH + u) * D);
                const f32x2 yy = pack2(y, y);
                l[g] = __fadd_rn(l[g], y);
#pragma unroll
                for (int e = 0; e < EPL / 2; ++e) acc[g][e] = fma2(yy, pack2(vv[2 * e], vv[2 * e + 1]), acc[g][e]);
            }
        }
    };
    int st = 0;
    uint32_t ph = 0;
#pragma unroll 1
    for (int s = s_first; s < s_end; ++s) {
        m = kNegBig;
#pragma unroll
        for (int g = 0; g < GW; ++g) {
            l[g] = 0.f;
#pragma unroll
            for (int e = 0; e < EPL / 2; ++e) acc[g][e] = 0ull;
        }
        const int n = pages_of(s);
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
            const int left = ctx - (s * pps + w + NW * i) * kKvBlock;      // rows from the page's first on that hold a position
#pragma unroll 1
            for (int r0 = 0; r0 < kKvBlock && (r0 == 0 || r0 < left); r0 += SR) {
                // a copy that never came: no further ones, nothing is handed back, the host reports the code
                if (ok) ok = __all_sync(0xffffffffu, mbar_wait_bounded(my_full + 8u * st, ph, kRingSpinLimit, 0));
                if (!ok) break;
                const unsigned char* kt = ring + st * 2 * SB;
#pragma unroll 1
                for (int cc = 0; cc < CPS; ++cc) use_chunk(kt, left - r0, cc * CH);
                __syncwarp();
                if (lane == 0) mbar_arrive(my_empty + 8u * st);
                if (++st == NST) { st = 0; ph ^= 1u; }
            }
            if (!ok) {
                if (lane == 0 && p.err != nullptr) atomicExch(p.err, 6);
                break;
            }
        }
        // merge the PPI lane groups of the warp
#pragma unroll
        for (int g = 0; g < GW; ++g) {
            float mg = __shfl_sync(0xffffffffu, m, src0 + g * GL), a[EPL];
#pragma unroll
            for (int e = 0; e < EPL / 2; ++e) unpack2(acc[g][e], a[2 * e], a[2 * e + 1]);
#pragma unroll
            for (int o = LPR; o < 32; o <<= 1) {
                const float mo = __shfl_xor_sync(0xffffffffu, mg, o), lo = __shfl_xor_sync(0xffffffffu, l[g], o);
                const float mn = fmaxf(mg, mo), sa = expf(mg - mn), sb = expf(mo - mn);
                l[g] = fmaf(l[g], sa, __fmul_rn(lo, sb));
#pragma unroll
                for (int e = 0; e < EPL; ++e) {
                    const float ao = __shfl_xor_sync(0xffffffffu, a[e], o);
                    a[e] = fmaf(a[e], sa, __fmul_rn(ao, sb));
                }
                mg = mn;
            }
            if (grp == 0) {
                float* d = sred + (w * G + hgrp * GW + g) * W;
#pragma unroll
                for (int e = 0; e < EPL; ++e) d[lr * EPL + e] = a[e];
                if (lr == 0) { d[HD] = mg; d[HD + 1] = l[g]; }
            }
        }
        sync();
        // merge the streams: one thread per output dim
        for (int i = tid; i < G * HD; i += 32 * NW * HG) {
            const int g = i / HD, e = i % HD, h = h0 + g;
            const float* r = sred + g * W;
            float mn = kNegBig;
#pragma unroll
            for (int v = 0; v < NW; ++v) mn = fmaxf(mn, r[v * G * W + HD]);
            float lt = 0.f, at = 0.f;
#pragma unroll
            for (int v = 0; v < NW; ++v) {
                const float sc = expf(r[v * G * W + HD] - mn);
                lt = fmaf(r[v * G * W + HD + 1], sc, lt);
                at = fmaf(r[v * G * W + e], sc, at);
            }
            if (S == 1) {
                float o = at / lt;
                if (p.gbuf) o *= p.gbuf[((size_t)b * p.heads + h) * HD + e];
                p.abuf[((size_t)b * p.heads + h) * HD + e] = o;
                if (p.abuf16) p.abuf16[((size_t)b * p.heads + h) * HD + (p.perm ? perm16(e) : e)] = __float2bfloat16_rn(p.perm ? o * kOperandScale : o);
            } else {
                float* pp = loop ? spart + (s * G + g) * W : p.part + (((size_t)b * p.heads + h) * SG + s) * W;
                pp[e] = at;
                if (e == 0) { pp[HD] = mn; pp[HD + 1] = lt; }
            }
        }
        sync();                       // the next split's results go to the same place
    }
    if (S == 1) return;
    if (!loop) {
        const int tslot = b * (int)gridDim.y + (int)blockIdx.y;
        __threadfence();
        sync();
        if (tid == 0) is_last = atomicAdd(&p.ticket[tslot], 1) == S - 1;
        sync();
        if (!is_last) return;
        __threadfence();
        if (tid == 0) p.ticket[tslot] = 0;
    }
    // Combine: a warp takes 32 or 64 output elements of a head. Its lanes turn the splits' (max, sum) pairs into normalised weights, which it
    // hands round; the splits' values are asked for eight at a time, the first with the pairs. (One warp of the CTA doing the weights for
    // all, alone between two barriers, took 2.1 us of the 4.8 behind the last split at one head per CTA.) One code for results in shared
    // and in global memory: a copy for each cost launches with one split, which run neither, 0.2 us (step of 3 sequences 213.6 -> 214.8 us).
    constexpr int AHEAD = 8;                       // (of 32: a group's weights are in one register)
    constexpr int PER = G * HD > 32 * NW * HG ? G * HD / (32 * NW * HG) : 1;      // outputs per lane
    static_assert(HD % (32 * PER) == 0, "a warp's outputs are of one head");
    const int first = warp * PER * 32;
    if (first >= G * HD) return;
    auto ld = [](const float* a) {
        float x;
        asm volatile("ld.relaxed.gpu.f32 %0, [%1];" : "=f"(x) : "l"(a) : "memory");
        return x;
    };
    const int g = first / HD, e = first % HD + lane, of_split = loop ? G * W : W;
    const float* part = loop ? spart + g * W : p.part + ((size_t)b * p.heads + h0 + g) * SG * W;
    float m0 = kNegBig, l0 = 0.f, m1 = kNegBig, l1 = 0.f, w0 = 0.f, w1 = 0.f, o[PER];
    if (lane < S) { m0 = ld(part + lane * of_split + HD); l0 = ld(part + lane * of_split + HD + 1); }
    if (lane + 32 < S) { m1 = ld(part + (lane + 32) * of_split + HD); l1 = ld(part + (lane + 32) * of_split + HD + 1); }
#pragma unroll
    for (int j = 0; j < PER; ++j) o[j] = 0.f;
#pragma unroll 1
    for (int s0 = 0; s0 < S; s0 += AHEAD) {
        float v[AHEAD][PER];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
#pragma unroll
            for (int j = 0; j < PER; ++j) v[u][j] = s0 + u < S ? ld(part + (s0 + u) * of_split + e + 32 * j) : 0.f;
        if (s0 == 0) {
            float mx = fmaxf(m0, m1);
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, q));
            w0 = expf(m0 - mx);
            w1 = expf(m1 - mx);
            const float lt = warp_sum(l0 * w0 + l1 * w1);
            w0 /= lt;
            w1 /= lt;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const float y = __shfl_sync(0xffffffffu, s0 < 32 ? w0 : w1, (s0 + u) & 31);
            if (s0 + u < S) {
#pragma unroll
                for (int j = 0; j < PER; ++j) o[j] = fmaf(y, v[u][j], o[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        const int ej = e + 32 * j;
        const size_t at = ((size_t)b * p.heads + h0 + g) * HD;
        if (p.gbuf) o[j] *= p.gbuf[at + ej];
        p.abuf[at + ej] = o[j];
        if (p.abuf16) p.abuf16[at + (p.perm ? perm16(ej) : ej)] = __float2bfloat16_rn(p.perm ? o[j] * kOperandScale : o[j]);
    }
}

// The kernel for G query heads per CTA: launch(kernel, threads, shared memory), its shared-memory limit raised before.
template <typename KVT, int HD, int G, typename Launch>
inline cudaError_t attn_with_kernel(const AttnParams& p, const dim3& grid, int sm_count, Launch launch) {
    auto run = [&](auto kernel, int rows) {
        const size_t smem = attn_smem(sizeof(KVT), HD, G, rows);
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return e == cudaSuccess ? launch(kernel, attn_threads<G>(), smem) : e;
    };
    constexpr int FEW = attn_few_rows(sizeof(KVT), HD, G);
    const long ctas = attn_ctas_with_work((long)grid.y * grid.z, (int)grid.x, p.pt_stride, p.min_pages_per_split);
    if (attn_whole_pages(sizeof(KVT), HD, G, ctas, sm_count)) return run(attn_decode_kernel<KVT, HD, G, kKvBlock>, kKvBlock);
    return run(attn_decode_kernel<KVT, HD, G, FEW>, FEW);
}

}  // namespace mlb
