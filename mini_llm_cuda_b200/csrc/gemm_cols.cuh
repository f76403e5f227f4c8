// Projections of many prompt columns on the 5th-generation tensor cores: Y[c][n] = sum_k X[c][k] W[n][k], bf16 operands,
// fp32 accumulation in tensor memory, persistent CTAs.
//
// A decode batch is at most a few tiles wide and gemm_tc.cuh gives its MMA rows to the weights. A prompt chunk has up to
// 4096 columns, so here the columns are the MMA's M = 128 and BN weight rows its N: a thread of the epilogue then owns
// one column (token), and what the step does per token - the 1/rms scale, QK norm over a head, RoPE pairs, the K/V row,
// the sum of squares for the next norm - stays in its registers; every thread reads and writes whole 32- or 64-byte
// pieces of its token's row.
//   warp 0     TMA loader: [128 x 64] activation tile and [BN x 64] weight tile (gate and up halves for SwiGLU) per stage
//   warp 1     MMA issuer: tcgen05.mma M128 x BN x K16, four per stage, into one of two accumulators
//   warps 2, 3 nothing: they complete the warpgroup that gives its registers to the epilogue's
//   warps 4-11 epilogue of the other accumulator: two warps per TMEM lane quarter, half of the columns each
// PAIR: two CTAs (the SMs of a TPC) share a tile of 256 columns x 256 features (tcgen05 cta_group::2): each loads its own 128 columns and half of
// the weight rows. What bounds the k-loop: the tensor pipe at 256 features (128 x 256 x 64 in 0.43 us on every SM, 1.44 PFLOP/s; a pair's 256 x 256
// 0.42, 1.48), below that the operands (32 KB in 0.36 us at 128 features, 24 KB in 0.26 at 64: about 90 GB/s an SM). A lone CTA whose epilogue adds up
// ranges has registers for 128 features, a pair for 256: that is what pairs give. 4096 columns, 2048 features: O 94 -> 61 us, down
// (K 5632) 177 -> 105, QKV (3072) 88 -> 77, delta-net projections (6176) 142 -> 94 with pairs, the register shares below and staged residuals;
// gate/up (11264), which has no ranges to add up, 144 -> 140.
// One CTA per SM walks tiles of the output; the epilogue of a tile runs under the k-loop of the next one where tensor
// memory holds the accumulators twice.
// FP8 weights come as an exact bf16 copy of their codes; their row scales are applied to the accumulator, and the bf16
// per-layer-embedding operand that rides behind the down projection has an accumulator of its own.
//
// The results are gemm_tc_kernel's to the last bit: behind every layer the activations are rounded to bf16, so sums taken
// in another order end, some layers later, in other roundings and now and then in another token. That kernel splits the
// k-blocks of a tile over the CTAs of a cluster and adds their partial accumulators in order; here the same ranges of
// k-blocks go to accumulators of their own (`split`), and the sums of squares are taken over 32 features at a time in the
// order of its warp shuffles. SUMS: the ranges take turns with four accumulators of 128 columns (PAIR: two of 256), and the epilogue's threads
// add each finished one to sums in registers (64 per thread, 128), so the MMAs go on whatever the number of ranges. Holding all
// of a tile's accumulators in tensor memory until its epilogue left five of them BN = 64 and no second set: cfg4's O and
// down projections at 32768 prompt tokens took 75 ms.
// Every mbarrier wait is bounded; one that runs out records a code and the CTA drains without waiting further.
#pragma once
#include "gemm_tc.cuh"

namespace mlb {

constexpr int kGcM = 128;
constexpr int kGcEpiWarps = 8;
constexpr int kGcThreads = 128 + 32 * kGcEpiWarps;
// Registers of a thread of a kernel with sums (SUMS), at launch (what 384 threads leave each), then of warps 0 - 3 and of the epilogue's:
// 128 sums and an epilogue's values do not fit 168. The shares add up to what the block was launched with (checked where a column set is made,
// gemm_cols_can_sum: a share that the block does not own would be waited for without end).
constexpr int kGcRegsLaunch = 168, kGcRegsFew = 40, kGcRegsMany = 232;
static_assert(128 * kGcRegsFew + 32 * kGcEpiWarps * kGcRegsMany <= kGcThreads * kGcRegsLaunch, "register shares");
constexpr int kGcMaxStages = 8;
constexpr int kGcMaxBufs = 4;
constexpr int kGcStgRow = 36;                  // floats from one token's staging row to the next: 16-byte accesses by rows and by columns without conflicts
constexpr size_t gc_staging(int mode) { return mode == TC_RESID ? (size_t)kGcEpiWarps * 32 * kGcStgRow * 4 : 0; }
constexpr size_t kGcSmem = 216 * 1024;         // of 227 KB; the factors and barriers take 8.5

struct GemmColsParams {
    int N, K, BN;                  // output features (SWIGLU: of h), width of the main operands, MMA N
    int stages, nkb_x;             // ring depth; k-blocks taken from the second operand pair
    int split, mains, exts;        // ranges of k-blocks; of them, how many hold k-blocks of the main pair / of a second pair that
                                   // accumulates separately (scaled weights; 0: it shares the main accumulators)
    int nbuf;                      // sets of accumulators in tensor memory: 2 = epilogue under the next k-loop; SUMS: accumulators, used in turn
    uint32_t tmem_cols;
    float* y;                      // RAW: fp32 [c][N]; RESID: residual stream, updated in place
    bf16_t* h16;                   // SWIGLU: bf16 [c][N]
    const float* ssq_in; int ssq_parts; float eps;      // deferred RMS norm, as in GemmTcParams
    bf16_t* xg16; const float* gain_next; float* ssq_out;      // sums of squares of 32 features each: [c][ssq_parts], a multiple of 4
    const float *s1, *s2;          // row scales of FP8 weights (SWIGLU: gate, up), or null
    int* err;
};

// 32 bytes per thread: one whole sector, so that rows of different tokens do not cost partial sectors
__device__ __forceinline__ void st_f32x8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
                 "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void gc_cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t gc_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void st_bf16x16(bf16_t* p, const float* v) {
    uint4 a, b;
    a.x = gc_pack(v[0], v[1]); a.y = gc_pack(v[2], v[3]); a.z = gc_pack(v[4], v[5]); a.w = gc_pack(v[6], v[7]);
    b.x = gc_pack(v[8], v[9]); b.y = gc_pack(v[10], v[11]); b.z = gc_pack(v[12], v[13]); b.w = gc_pack(v[14], v[15]);
    reinterpret_cast<uint4*>(p)[0] = a;
    reinterpret_cast<uint4*>(p)[1] = b;
}
__device__ __forceinline__ void put16(float* p, const float* v) { st_f32x8(p, v); st_f32x8(p + 8, v + 8); }
__device__ __forceinline__ void put16(bf16_t* p, const float* v) { st_bf16x16(p, v); }
// 16 per-feature values, the same for every lane
__device__ __forceinline__ void ld_feat16(const float* p, float* v) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p) + i);
        v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
    }
}

// ---- two CTAs on one tile (cta_group::2): rank 0 issues the MMAs and owns the barriers of operands and free accumulators -----------
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs
__device__ __forceinline__ void umma_commit_pair(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(mbar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

template <int MODE, typename KVT, bool SUMS, bool PAIR>
__global__ void __launch_bounds__(kGcThreads, 1) gemm_cols_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                                                                  const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmXx,
                                                                  const __grid_constant__ CUtensorMap tmWx, const __grid_constant__ GemmColsParams p,
                                                                  const __grid_constant__ StepCtl c, const __grid_constant__ QkvPostParams q) {
    extern __shared__ unsigned char smem_raw[];
    const int n_cols = *c.n_cols;                                  // in place before the step's first kernel starts
    const int bn_out = MODE == TC_SWIGLU ? p.BN / 2 : p.BN;
    constexpr int TM = PAIR ? 2 * kGcM : kGcM;                     // columns of a tile
    const int rank = PAIR ? (int)cluster_rank() : 0, team = PAIR ? blockIdx.x / 2 : blockIdx.x, n_teams = PAIR ? gridDim.x / 2 : gridDim.x;
    const int n_m = (n_cols + TM - 1) / TM, n_n = (p.N + bn_out - 1) / bn_out;
    const int n_tiles = n_m * n_n;
    if (team >= n_tiles) return;                                   // (the CTAs of a pair alike)
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * kGcMaxStages + 2 * kGcMaxBufs];
    __shared__ uint32_t tmem_slot;
    __shared__ float feat[kGcEpiWarps][2][128];                    // per-feature factors of a warp's part of the tile
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8u * kGcMaxStages;
    const uint32_t tfull0 = empty0 + 8u * kGcMaxStages, tempty0 = tfull0 + 8u * kGcMaxBufs;
    const int b_rows = PAIR ? p.BN / 2 : p.BN;                      // of the weight tile, in this CTA
    const int a_bytes = kGcM * 128, stage_bytes = a_bytes + b_rows * 128;
    const int nkb1 = (p.K + kTcKB - 1) / kTcKB, nkb = nkb1 + p.nkb_x;
    const uint32_t acc_cols = (uint32_t)((SUMS ? 1 : p.mains + p.exts) * p.BN);
    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(full0 + 8u * i, 1);
            mbar_init(empty0 + 8u * i, 1);
        }
        for (int i = 0; i < kGcMaxBufs; ++i) {
            mbar_init(tfull0 + 8u * i, 1);
            mbar_init(tempty0 + 8u * i, PAIR ? 2 * kGcEpiWarps : kGcEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(p.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(p.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();                                  // the other CTA's barriers are set up
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();

    if (warp < 4) {
        if (SUMS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kGcRegsFew));
        if (warp == 0) {
            if (lane == 0) {
                // of a pair, rank r loads columns 128 r .. of the tile and weight rows BN / 2 r .. (SWIGLU: gate | up); all bytes of a
                // stage count on rank 0's barrier, which rank 0 arms for both
                const uint32_t bytes = (uint32_t)(PAIR ? 2 * stage_bytes : stage_bytes);
                const uint32_t lfull0 = PAIR ? cluster_map(full0, 0) : full0;
                auto tma = [&](uint32_t dst, const CUtensorMap* map, int k, int row, uint32_t bar) {
                    if (PAIR) tma_load_2d_pair(dst, map, k, row, bar);
                    else tma_load_2d(dst, map, k, row, bar);
                };
                auto load_w = [&](int kb, int n0, uint32_t base, uint32_t bar) {
                    if (kb < nkb1) {
                        if (PAIR && MODE == TC_SWIGLU) {
                            tma(base + a_bytes, rank ? &tmW2 : &tmW, kb * kTcKB, n0, bar);
                        } else {
                            tma(base + a_bytes, &tmW, kb * kTcKB, n0 + rank * b_rows, bar);
                            if (MODE == TC_SWIGLU) tma(base + a_bytes + bn_out * 128, &tmW2, kb * kTcKB, n0, bar);
                        }
                    } else {
                        tma(base + a_bytes, &tmWx, (kb - nkb1) * kTcKB, n0 + rank * b_rows, bar);
                    }
                };
                auto load_x = [&](int kb, int m0, uint32_t base, uint32_t bar) {
                    if (kb < nkb1) tma(base, &tmX, kb * kTcKB, m0, bar);
                    else tma(base, &tmXx, (kb - nkb1) * kTcKB, m0, bar);
                };
                auto arm = [&](int st) { if (rank == 0) mbar_expect_tx(full0 + 8u * st, bytes); };
                const uint32_t ring = smem_u32(smem);
                // the first tile's first weight tiles depend on nothing: on their way before the predecessor is waited for
                const int first = team;
                const int pre = min(p.stages, nkb);
                for (int kb = 0; kb < pre; ++kb) {
                    arm(kb);
                    load_w(kb, first / n_m * bn_out, ring + (uint32_t)(kb * stage_bytes), lfull0 + 8u * kb);
                }
                pdl_wait();
                int s = 0;
                uint32_t ph = 1;
                bool ok = true;
                for (int t = first; t < n_tiles && ok; t += n_teams) {
                    const int m0 = t % n_m * TM + rank * kGcM, n0 = t / n_m * bn_out;
                    for (int kb = 0; kb < nkb; ++kb) {
                        const uint32_t bar = lfull0 + 8u * s, base = ring + (uint32_t)(s * stage_bytes);
                        if (t != first || kb >= pre) {
                            if (!tc_wait(empty0 + 8u * s, ph, p.err, 21)) { ok = false; break; }
                            arm(s);
                            load_w(kb, n0, base, bar);
                        }
                        load_x(kb, m0, base, bar);
                        if (++s == p.stages) { s = 0; ph ^= 1u; }
                    }
                }
            }
        } else if (warp == 1) {
            if (lane == 0 && rank == 0) {
                auto commit = [](uint32_t bar) {
                    if (PAIR) umma_commit_pair(bar);
                    else umma_commit(bar);
                };
                const uint32_t idesc = umma_idesc_bf16(TM, p.BN);
                const uint32_t ring = smem_u32(smem);
                int s = 0, i = 0, buf = 0, use = 0;        // use: how often this buffer has been filled before
                uint32_t ph = 0;
                bool ok = true;
                for (int t = team; t < n_tiles && ok; t += n_teams, ++i) {
                    if (!SUMS) {
                        if (i >= p.nbuf && !tc_wait(tempty0 + 8u * buf, (uint32_t)(use - 1) & 1u, p.err, 22)) { ok = false; break; }
                        tc_fence_after();
                    }
                    const uint32_t acc = tmem + buf * acc_cols;
                    int r = 0, hi = nkb / p.split;           // range of k-blocks: [nkb r / split, nkb (r + 1) / split)
                    bool fresh = true, xfresh = true;        // the next MMA starts its accumulator
                    for (int kb = 0; kb < nkb; ++kb) {
                        while (kb >= hi) {
                            ++r;
                            hi = (int)((long)nkb * (r + 1) / p.split);
                            fresh = xfresh = true;
                        }
                        if (!tc_wait(full0 + 8u * s, ph, p.err, 23)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t base = ring + (uint32_t)(s * stage_bytes);
                        const uint64_t ad = umma_desc_sw128(base), bd = umma_desc_sw128(base + a_bytes);
                        const bool ext = p.exts > 0 && kb >= nkb1;
                        if (SUMS && (ext ? xfresh : fresh)) {
                            // the next accumulator in turn; the one before it is complete
                            if (kb > 0) {
                                commit(tfull0 + 8u * buf);
                                if (++buf == p.nbuf) { buf = 0; ++use; }
                            }
                            if (use > 0 && !tc_wait(tempty0 + 8u * buf, (uint32_t)(use - 1) & 1u, p.err, 22)) { ok = false; break; }
                            tc_fence_after();
                        }
                        // the separate accumulators of the second pair lie behind the main ones, its ranges are the last ones
                        const uint32_t dst = SUMS ? tmem + (uint32_t)(buf * p.BN) : acc + (uint32_t)((ext ? p.mains + r - (p.split - p.exts) : r) * p.BN);
                        const bool first = ext ? xfresh : fresh;
#pragma unroll
                        for (int j = 0; j < kTcKB / 16; ++j) {
                            if (PAIR) umma_bf16_pair(dst, ad + 2u * j, bd + 2u * j, idesc, (first && j == 0) ? 0u : 1u);
                            else umma_bf16(dst, ad + 2u * j, bd + 2u * j, idesc, (first && j == 0) ? 0u : 1u);
                        }
                        if (ext) xfresh = false; else fresh = false;
                        commit(empty0 + 8u * s);
                        if (++s == p.stages) { s = 0; ph ^= 1u; }
                    }
                    commit(tfull0 + 8u * buf);      // also after a wait that ran out: the epilogue must not hang on it
                    if (++buf == p.nbuf) { buf = 0; ++use; }
                }
            }
        }
    } else {
        if (SUMS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kGcRegsMany));
        // ---- epilogue: one token per thread, half of the tile's columns per warp ---------------------------------
        const int quarter = warp & 3, half = (warp - 4) >> 2;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        // features of this thread per tile, in chunks of 16 (a pair's tile has BN = 256)
        const int span = !PAIR ? bn_out / 2 : (MODE == TC_SWIGLU ? 64 : 128);
        // a pair's sums leave registers for the rest only if those of finished chunks are given up: no rolled loop there
        constexpr int UNROLL = PAIR && SUMS && MODE == TC_RESID ? 4 : 1;
        pdl_wait();
        int buf = 0, use = 0;
        bool ok = true;
        // (tcgen05.ld is a warp-wide instruction: the lanes go on or give up together)
        // an accumulator is free once the warps of both CTAs have read it
        const uint32_t lempty0 = PAIR ? cluster_map(tempty0, 0) : tempty0;
        auto release = [&](int b) {
            if (lane != 0) return;
            if (PAIR) mbar_arrive_cluster(lempty0 + 8u * b);
            else mbar_arrive(tempty0 + 8u * b);
        };
        float (&fw)[2][128] = feat[warp - 4];
        // RESID: staging rows of the warp, [32 tokens][32 features]. A thread computes its token's features; the residual stream, which is read and
        // written, crosses four tokens at a time, eight lanes to 32 consecutive features, and without a register (sums and 16 prefetched
        // residual values spilled: O / down projections of 4096 columns, 2048 features: 75 / 119 us with the spills, 67 / 109 with a lane per
        // token and no prefetch, 61 / 105 staged. The other modes only write, and lose: QKV 77 -> 88 - 99 us.)
        float* stg = reinterpret_cast<float*>(smem + (size_t)p.stages * stage_bytes) + (warp - 4) * 32 * kGcStgRow;
        const int piece = lane & 7, trow = lane >> 3;
        auto arrived = [&](int b, int u) { return (bool)__all_sync(0xffffffffu, tc_wait(tfull0 + 8u * b, (uint32_t)u & 1u, p.err, 24)); };
        for (int t = team; t < n_tiles && ok; t += n_teams) {
            const int m0 = t % n_m * TM + rank * kGcM, n0 = t / n_m * bn_out;
            const int tok0 = m0 + quarter * 32, tok = tok0 + lane;
            const bool live = tok < n_cols;
            const int f_begin = n0 + half * span;
            // the warp's per-feature factors, asked for before the accumulator is waited for: row scales; gains, or scales of the second matrix
            float ff[2][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int f = min(f_begin + lane + 32 * i, p.N - 1);
                ff[0][i] = p.s1 != nullptr ? __ldg(p.s1 + f) : 1.0f;
                if (MODE == TC_RESID) ff[1][i] = __ldg(p.gain_next + f);
                if (MODE == TC_SWIGLU) ff[1][i] = p.s2 != nullptr ? __ldg(p.s2 + f) : 1.0f;
            }
            float rinv = 1.0f;
            if (p.ssq_in != nullptr && live) {
                float tot = 0.f;
                const float4* sp = reinterpret_cast<const float4*>(p.ssq_in + (size_t)tok * p.ssq_parts);
                for (int j = 0; j < p.ssq_parts / 4; ++j) {
                    const float4 x = __ldcg(sp + j);
                    tot += (x.x + x.y) + (x.z + x.w);
                }
                rinv = 1.0f / sqrtf(tot / (float)p.K + p.eps);
            }
            int pos = 0;
            size_t kv_row = 0;                        // row of the token in this layer's pools, for kv head 0
            if (MODE == TC_QKV && live) {
                pos = c.pos[tok];
                const int page = q.page_table[kv_seq(c, tok) * q.pt_stride + pos / kKvBlock];
                kv_row = (size_t)page * q.kv_heads * kKvBlock + (pos % kKvBlock);
            }
            // residual values of 32 features into the warp's staging rows
            auto fetch_resid = [&](int fg) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int row = trow + 4 * i, f = fg + 4 * piece;
                    const bool in = tok0 + row < n_cols && f < p.N;
                    gc_cp_async16(smem_u32(stg + row * kGcStgRow + 4 * piece), in ? p.y + (size_t)(tok0 + row) * p.N + f : p.y, in);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            if (MODE == TC_RESID) fetch_resid(f_begin);
            __syncwarp();                             // the last tile's factors have been read
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                fw[0][lane + 32 * i] = ff[0][i];
                if (MODE == TC_RESID || MODE == TC_SWIGLU) fw[1][lane + 32 * i] = ff[1][i];
            }
            __syncwarp();
            // SUMS: the ranges' accumulators arrive one after another and are added up here, in their order, each given back at once.
            // A sum per thread for half of the tile's BN <= 16 CH features (SWIGLU: the first half of them of gate, the second of up)
            constexpr int CH = PAIR ? 8 : 4;
            float sums[SUMS ? 16 * CH : 1];
            if (SUMS) {
                for (int r = 0; r < p.mains && ok; ++r) {
                    ok = arrived(buf, use);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a = tmem + (uint32_t)(buf * p.BN) + lane_base;
#pragma unroll
                    for (int h = 0; h < CH / 2; ++h) {
                        uint32_t ta[2][16];
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int ch = MODE == TC_SWIGLU ? (2 * h + k) % (CH / 2) : 2 * h + k, up = MODE == TC_SWIGLU ? (2 * h + k) / (CH / 2) : 0;
                            if (16 * ch < span) tmem_ld16_issue(a + (uint32_t)(up * bn_out + half * span + 16 * ch), ta[k]);
                        }
                        tmem_ld_wait();
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                float& o = sums[SUMS ? 16 * (2 * h + k) + j : 0];
                                o = r == 0 ? __uint_as_float(ta[k][j]) : __fadd_rn(o, __uint_as_float(ta[k][j]));
                            }
                    }
                    tc_fence_before();
                    __syncwarp();
                    release(buf);
                    if (++buf == p.nbuf) { buf = 0; ++use; }
                }
                // accumulators of the second pair stay where they are until the element-wise work below has read them
                for (int r = 0, b = buf, u = use; r < p.exts && ok; ++r) {
                    ok = arrived(b, u);
                    if (++b == p.nbuf) { b = 0; ++u; }
                }
                if (!ok) break;
            } else if (!(ok = arrived(buf, use))) {
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + buf * acc_cols + lane_base;
            float head_sc = 1.0f, sqp[16];
            // 16 columns of the sum of `n` accumulators, in their order
            auto load_acc = [&](uint32_t col, int n, float* o) {
                uint32_t ta[16];
                tmem_ld16_issue(col, ta);
                if (n == 1) {
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) o[j] = __uint_as_float(ta[j]);
                    return;
                }
                uint32_t tb[16];
                tmem_ld16_issue(col + (uint32_t)p.BN, tb);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) o[j] = __uint_as_float(ta[j]) + __uint_as_float(tb[j]);
                for (int r = 2; r < n; ++r) {
                    tmem_ld16_issue(col + (uint32_t)(r * p.BN), ta);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) o[j] += __uint_as_float(ta[j]);
                }
            };
            // sum of 16 + 16 values in the order of warp_colsum16
            auto sum32 = [](const float* x, const float* y) {
                float t[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) t[j] = x[j] + y[j];
#pragma unroll
                for (int w = 8; w >= 1; w >>= 1)
#pragma unroll
                    for (int j = 0; j < w; ++j) t[j] += t[j + w];
                return t[0];
            };
#pragma unroll UNROLL
            for (int cg = 0; cg < span; cg += 32) {
                const int fg = f_begin + cg;
                if (fg >= p.N) {                       // uniform for the warp; the sums of squares behind the last feature are zero
                    if (MODE == TC_RESID && live)
                        for (int g = fg / 32; g < (f_begin + span) / 32 && g < p.ssq_parts; ++g) p.ssq_out[(size_t)tok * p.ssq_parts + g] = 0.f;
                    break;
                }
                // q | k | v | gate: whole heads of 64 or 128 features each
                const int seg_k = q.nq, seg_v = q.nq + q.nk, seg_g = seg_v + q.nv;
                const int seg = MODE != TC_QKV ? 0 : (fg < seg_k ? 0 : (fg < seg_v ? 1 : (fg < seg_g ? 2 : 3)));
                const int fs = fg - (seg == 0 ? 0 : (seg == 1 ? seg_k : (seg == 2 ? seg_v : seg_g)));     // feature inside its segment
                const int e0 = MODE == TC_QKV ? fs % q.hd : 0, head = MODE == TC_QKV ? fs / q.hd : 0;
                if (MODE == TC_RESID) {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    __syncwarp();
                }
                // ---- a thread's token: two chunks of 16 features -> memory, or (RESID) staging row
                float4* own = reinterpret_cast<float4*>(stg + lane * kGcStgRow);
#pragma unroll (UNROLL > 1 ? 2 : 1)
                for (int h = 0; h < 2; ++h) {
                    const int cc = cg + 16 * h, f0 = f_begin + cc, col = half * span + cc;
                    if (cc >= span || (MODE != TC_RESID && f0 >= p.N)) break;             // (a group of 16: SWIGLU with BN = 64)
                    const bool whole = f0 + 16 <= p.N;
                    __syncwarp();                      // tcgen05.ld is a warp-wide instruction
                    float v[16], w2[16];
                    if constexpr (SUMS) {
                        // the front 16 of the sums; the others move up, so that a rolled loop names registers
                        constexpr int HALF = MODE == TC_SWIGLU ? CH / 2 : CH;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            v[j] = sums[UNROLL > 1 ? cc + j : j];
                            if (MODE == TC_SWIGLU) w2[j] = sums[16 * (CH / 2) + j];
#pragma unroll
                            for (int g = 0; g < (UNROLL > 1 ? 0 : CH - 1); ++g)
                                if (g != HALF - 1) sums[16 * g + j] = sums[16 * (g + 1) + j];
                        }
                        if (MODE == TC_RESID && p.exts > 0) {
                            load_acc(acc + (uint32_t)col, 1, w2);
                            for (int r = 1, b = buf; !PAIR && r < p.exts; ++r) {          // (a pair's two accumulators leave room for one)
                                if (++b == p.nbuf) b = 0;
                                float e[16];
                                load_acc(tmem + (uint32_t)(b * p.BN + col) + lane_base, 1, e);
#pragma unroll
                                for (int j = 0; j < 16; ++j) w2[j] = __fadd_rn(w2[j], e[j]);
                            }
                        }
                    } else {
                        load_acc(acc + (uint32_t)col, p.mains, v);
                        if (MODE == TC_SWIGLU) load_acc(acc + (uint32_t)(bn_out + col), p.mains, w2);
                        if (MODE == TC_RESID && p.exts > 0) load_acc(acc + (uint32_t)(p.mains * p.BN + col), p.exts, w2);
                    }
                    if (MODE == TC_SWIGLU) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float g = v[j] * fw[0][cc + j] * rinv, u = w2[j] * fw[1][cc + j] * rinv;
                            v[j] = __fdividef(g, 1.0f + __expf(-g)) * u;            // inference.cu:262-281
                        }
                    } else if (MODE == TC_RESID) {
                        // (roundings as in gemm_tc_kernel: scale and second pair in one fma, then the residual)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float4 r = own[4 * h + i];
                            const float rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int j = 4 * i + k;
                                if (p.s1 != nullptr) v[j] = fmaf(v[j], fw[0][cc + j], p.exts > 0 ? w2[j] : 0.f);
                                v[j] = __fadd_rn(v[j], rr[k]);                      // inference.cu:252-260, :283-291
                            }
                        }
                        float sq[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) sq[j] = (whole || f0 + j < p.N) ? __fmul_rn(v[j], v[j]) : 0.f;
                        if (h == 1) {
                            if (live) p.ssq_out[(size_t)tok * p.ssq_parts + f0 / 32] = sum32(sqp, sq);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j) sqp[j] = sq[j];
                        }
                    } else {
                        if (p.s1 != nullptr) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[j] *= fw[0][cc + j];
                        }
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] *= rinv;
                    }
                    if (MODE == TC_QKV && !SUMS && seg < 2 && q.qk_norm) {
                        // per-head RMS norm (inference.cu:52-81, :97-111): the head's other features come from tensor memory
                        const int e1 = e0 + 16 * h;
                        if (e1 == 0 || cc == 0) {
                            float ss = 0.f;
                            for (int e = 0; e < q.hd; e += 32) {
                                float x[2][16];
#pragma unroll
                                for (int b = 0; b < 2; ++b) {
                                    load_acc(acc + (uint32_t)(col - e1 + e + 16 * b), p.mains, x[b]);
#pragma unroll
                                    for (int j = 0; j < 16; ++j) {
                                        if (p.s1 != nullptr) x[b][j] *= __ldg(p.s1 + f0 - e1 + e + 16 * b + j);
                                        x[b][j] *= rinv;
                                        x[b][j] = __fmul_rn(x[b][j], x[b][j]);
                                    }
                                }
                                ss += sum32(x[0], x[1]);
                            }
                            head_sc = rsqrtf(ss * (1.0f / (float)q.hd) + q.eps);
                        }
                        float g[16];
                        ld_feat16((seg == 0 ? q.gq : q.gk) + fs + 16 * h, g);
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] *= head_sc * g[j];
                    }
                    if (MODE == TC_RESID) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) own[4 * h + i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    } else if (MODE == TC_SWIGLU) {
                        if (live) {
                            bf16_t* o = p.h16 + (size_t)tok * p.N + f0;
                            if (whole) {
                                st_bf16x16(o, v);
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    if (f0 + j < p.N) o[j] = __float2bfloat16_rn(v[j]);
                            }
                        }
                    } else if (MODE == TC_RAW) {
                        if (live) {
                            float* o = p.y + (size_t)tok * p.N + f0;
                            if (whole && (p.N & 7) == 0) {
                                put16(o, v);
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    if (f0 + j < p.N) o[j] = v[j];
                            }
                        }
                    } else if (live) {
                        const int e1 = e0 + 16 * h;
                        if (seg < 2) {
                            // RoPE on adjacent pairs (inference.cu:113-134)
                            float r[16];
                            ld_feat16(q.rope + (size_t)pos * q.hd + e1, r);
#pragma unroll
                            for (int j = 0; j < 16; j += 2) {
                                const float a = v[j], b = v[j + 1];
                                v[j] = fmaf(r[j], a, -(r[j + 1] * b));
                                v[j + 1] = fmaf(r[j + 1], a, r[j] * b);
                            }
                        }
                        if (seg == 0) put16(q.qbuf + (size_t)tok * q.nq + fs + 16 * h, v);
                        else if (seg == 1) put16(reinterpret_cast<KVT*>(q.kpool) + (kv_row + (size_t)head * kKvBlock) * q.hd + e1, v);
                        else if (seg == 2) put16(reinterpret_cast<KVT*>(q.vpool) + (kv_row + (size_t)head * kKvBlock) * q.hd + e1, v);
                        else {
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[j] = __fdividef(1.0f, 1.0f + __expf(-v[j]));      // inference.cu:248
                            put16(q.gbuf + (size_t)tok * q.ng + fs + 16 * h, v);
                        }
                    }
                }
                if (MODE != TC_RESID) continue;
                __syncwarp();
                // ---- staging rows -> residual stream and next operand
                const int f = fg + 4 * piece;
                const float* g = fw[1] + cg + 4 * piece;
#pragma unroll 4
                for (int i = 0; i < 8; ++i) {
                    const int row = trow + 4 * i;
                    if (tok0 + row >= n_cols || f >= p.N) continue;              // N is a multiple of 8
                    const float4 x = *reinterpret_cast<const float4*>(stg + row * kGcStgRow + 4 * piece);
                    const size_t at = (size_t)(tok0 + row) * p.N + f;
                    *reinterpret_cast<float4*>(p.y + at) = x;
                    *reinterpret_cast<uint2*>(p.xg16 + at) = make_uint2(gc_pack(x.x * g[0], x.y * g[1]), gc_pack(x.z * g[2], x.w * g[3]));
                }
                __syncwarp();                          // the staging rows have been read
                if (cg + 32 < span) fetch_resid(fg + 32);
            }
            if (MODE == TC_RESID) asm volatile("cp.async.wait_group 0;" ::: "memory");      // (a fetch behind the last feature is not used)
            tc_fence_before();
            __syncwarp();
            for (int r = 0; r < (SUMS ? p.exts : 1); ++r) {
                release(buf);
                if (++buf == p.nbuf) { buf = 0; ++use; }
            }
        }
        if (MODE == TC_RESID) asm volatile("cp.async.wait_group 0;" ::: "memory");      // also of a tile that was given up
    }
    __syncthreads();
    if (PAIR) cluster_sync_all();                     // nothing of the other CTA's reads, writes or arrives here any more
    if (warp == 1) {
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
    }
}

}  // namespace mlb
