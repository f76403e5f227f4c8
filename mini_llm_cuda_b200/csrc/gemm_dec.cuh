// Projections of one decode step for a batch of sequences (4 .. 256) on mma.sync: Y[b][n] = sum_k W[n][k] X[b][k], bf16 (or
// e4m3) weights, bf16 activations, fp32 accumulators, the element-wise work of the step in the epilogue.
//
// A decode GEMM here is not bound by the tensor pipe (15 GFLOP a step) nor by HBM but by the chain wait for the
// predecessor -> operands -> products -> epilogue of every launch. gemm_tc_kernel (tcgen05) spends 8 us on it at 4 to 37
// sequences: its 128-row tiles occupy 4 to 24 SMs, the k-ranges of a tile meet over a thread-block cluster, and its
// epilogue, unrolled over accumulator registers, is fetched cold by every CTA (3.5 - 5.6 us). Here a CTA takes 32
// features and 16, 32 or 64 sequences: five to ten times the CTAs, the k-ranges are warps of one CTA and meet in shared
// memory, and the epilogue is a rolled loop over sequences with a feature per lane. mma.sync m16n8k16 and
// tcgen05.mma kind::f16 return the same bits for the same sixteen products and accumulator, whatever the order inside the sixteen (an
// observation, not documented: the tests compare whole steps on both tiles bit for bit), and k-ranges, their sum and the epilogue's
// operations are gemm_tc_kernel's, so the results are too.
//   producer warp   TMA: per stage G 64-wide k-blocks of every range, weights [G][32 x 64] (two for gate/up) and activations
//                   [G][CT x 64], each one copy of a three-dimensional map (k-block, row, 64 elements): a copy costs the
//                   TMA unit about 300 cycles however small it is, which bound the kernel at one k-block per copy. The weights of
//                   the first stages are requested before the predecessor is waited for.
//   other warps     one per 16 rows and range: ldmatrix, mma; partial sums to shared memory; epilogue
// e4m3 weights: ldmatrix on codes hands lane q of a row the codes 4q .. 4q + 3 of sixteen, so the activation operand of such
// models is written with its features permuted to match inside every sixteen (perm16), and times 2^64 (gd_widen).
// Every mbarrier wait is bounded. A consumer whose wait ran out hands no stage back, so no copy starts behind the last wait of the
// CTA's last consumer, and those under way have had that wait's time to land when the CTA ends. (Stages handed back by a consumer that
// no longer waits were refilled into a block about to end.)
#pragma once
#include "gemm_tc.cuh"

namespace mlb {

constexpr int kGdF = 32;               // output features per CTA
constexpr int kGdMaxStages = 16;
constexpr int kGdMaxSplit = 4;         // k-ranges of a tile, a warp per range and 16 rows
constexpr size_t kGdRing = 108 * 1024; // two CTAs per SM: the next launch's weights arrive under this one (part of it: gd_ring)

struct GemmDecParams {
    int N, K, B;
    int split, nkb_x;              // ranges of k-blocks; k-blocks of the second operand pair (behind the first's)
    int G;                         // k-blocks per copy
    int stages, w_bytes;           // ring depth; bytes of a weight tile's k-block in a stage
    float* y;                      // RAW: fp32 [b][N]; RESID: residual stream, updated in place
    bf16_t* h16;                   // SWIGLU: bf16 [b][N]
    const float* ssq_in; int ssq_parts; float eps;
    bf16_t* xg16; const float* gain_next; float* ssq_out;
    const float *s1, *s2;          // row scales of FP8 weights (SWIGLU: gate, up)
    int* err;
    unsigned long long* trace;     // diagnostics: five %globaltimer stamps of CTA (0, 0), or null
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(mbar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void gd_ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void gd_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Four codes -> two bf16 pairs of value * 2^-120: sign and the seven lower bits of a code moved to the places of bf16's sign, low
// exponent and mantissa bits. Exact, zeros and subnormal codes (-> subnormal bf16) included, in four instructions a pair; rebiasing the
// exponent took twice as many and a branch for exponent field 0, more issue slots than the products of 64 sequences.
// The activation operand is written times 2^64 and the row scales are taken times 2^56: products and sums keep their bits.
__device__ __forceinline__ void gd_widen(uint32_t w, uint32_t& lo, uint32_t& hi) {
    const uint32_t x0 = __byte_perm(w, 0u, 0x1404u), x1 = __byte_perm(w, 0u, 0x3424u);      // codes 0, 1 and 2, 3 in the high bytes of halves
    lo = (x0 & 0x80008000u) | ((x0 >> 4) & 0x07f007f0u);
    hi = (x1 & 0x80008000u) | ((x1 >> 4) & 0x07f007f0u);
}
constexpr float kGdScaleBack = 72057594037927936.0f;       // 2^56

// grid = (ceil(N / 32), ceil(B / (16 NP))), block = 32 (RT split + 1) with RT = 2 (4 for SWIGLU) row tiles of 16.
// Three CTAs an SM asked for where the compiler would otherwise take 56 registers for a fourth (cfg1 at 4 sequences: 186 us a step with
// 56, 178 with 72).
template <int MODE, typename KVT, typename WT, int NP>
__global__ void __launch_bounds__(32 * ((MODE == TC_SWIGLU ? 4 : 2) * kGdMaxSplit + 1), MODE == TC_QKV && sizeof(WT) == 2 && NP == 1 ? 3 : 0) gemm_dec_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2,
                                                                                  const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmWx,
                                                                                  const __grid_constant__ CUtensorMap tmXx, const __grid_constant__ GemmDecParams p,
                                                                                  const __grid_constant__ StepCtl c, const __grid_constant__ QkvPostParams q) {
    constexpr bool W8 = sizeof(WT) == 1;
    constexpr int NA = MODE == TC_SWIGLU ? 2 : 1;
    constexpr bool EXT2 = W8 && MODE == TC_RESID;     // the second pair accumulates separately: it must not be scaled
    constexpr int RT = 2 * NA;
    constexpr int CT = 16 * NP;
    constexpr int FRP = 32 * NA + 4;                  // floats from one column's partial sums to the next
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * kGdMaxStages];
    __shared__ float rinv_s[CT];
    __shared__ int pos_s[CT];
    __shared__ long long kvrow_s[CT];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool tracing = p.trace != nullptr && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0;
    if (tracing) p.trace[0] = globaltimer_ns();          // entry
    const int S = p.split, nw = RT * S;               // consumer warps; the producer is warp nw
    const int f0 = blockIdx.x * kGdF, b0 = blockIdx.y * CT;
    const int nkb1 = (p.K + kTcKB - 1) / kTcKB, nkb = nkb1 + p.nkb_x;
    const int G = p.G, seg_bytes = G * (NA * p.w_bytes + CT * 128), stage_bytes = S * seg_bytes;
    auto seg_lo = [&](int s) { return (int)((unsigned)(nkb * s) / (unsigned)S); };
    // range s holds k-blocks [seg_lo(s), seg_lo(s + 1)): stages of G of the main pair, then stages of G of the second pair
    auto main_len = [&](int s) { return max(0, min(seg_lo(s + 1), nkb1) - seg_lo(s)); };
    auto ext_len = [&](int s) { return seg_lo(s + 1) - seg_lo(s) - main_len(s); };
    auto up = [&](int n) { return (int)((unsigned)(n + G - 1) / (unsigned)G); };
    int n_iter = 0;
    for (int s = 0; s < S; ++s) n_iter = max(n_iter, up(main_len(s)) + up(ext_len(s)));
    const int n_load = S * (NA + 1);                   // producer lanes
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8u * kGdMaxStages;
    if (tid == 0) {
        for (int i = 0; i < p.stages; ++i) {
            mbar_init(full0 + 8u * i, n_load);
            mbar_init(empty0 + 8u * i, nw);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tracing) p.trace[1] = globaltimer_ns();          // barriers set up
    pdl_launch_dependents();

    if (warp == nw) {
        // ---- producer: lane s loads the activations of range s, lanes S + s and 2 S + s its weights; each arms its own bytes --
        const int s = lane % S, what = lane / S;       // what: 0 = X, 1 = W, 2 = W2
        const int lo = seg_lo(s), n_main = up(main_len(s)), len = what <= NA ? n_main + up(ext_len(s)) : 0;
        const int k_ext = max(lo, nkb1) - nkb1;         // first k-block of the second pair in this range
        const uint32_t base0 = smem_u32(ring) + (uint32_t)(s * seg_bytes) + (uint32_t)(G * (what == 0 ? NA * p.w_bytes : (what - 1) * p.w_bytes));
        const CUtensorMap* map = what == 0 ? &tmX : (what == 1 ? &tmW : &tmW2);
        const CUtensorMap* mapx = what == 0 ? &tmXx : &tmWx;
        if (lane < 3) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(lane == 0 ? &tmX : (lane == 1 ? &tmW : &tmW2))) : "memory");
        const int row = what == 0 ? b0 : f0;
        const uint32_t tile = G * (what == 0 ? CT * 128 : kGdF * (W8 ? 64 : 128)), tilex = G * (what == 0 ? CT * 128 : (what == 1 ? kGdF * 128 : 0));
        auto load = [&](int i, int st) {
            if (i >= len) return;
            const uint32_t dst = base0 + (uint32_t)(st * stage_bytes), bar = full0 + 8u * st;
            if (i < n_main) {
                mbar_expect_tx(bar, tile);
                tma_load_3d(dst, map, 0, row, lo + i * G, bar);
            } else {
                mbar_expect_tx(bar, tilex);
                if (tilex) tma_load_3d(dst, mapx, 0, row, k_ext + (i - n_main) * G, bar);
            }
        };
        auto pad = [&](int i, int st) {                // a lane without a tile in this stage arrives all the same
            if (lane < n_load && i >= len) mbar_arrive(full0 + 8u * st);
        };
        const int pre = min(p.stages, n_iter);
        if (what != 0)
            for (int i = 0; i < pre; ++i) {
                load(i, i);
                pad(i, i);
            }
        pdl_wait();                                    // the activation operand comes from the predecessor kernel
        if (what == 0)
            for (int i = 0; i < pre; ++i) {
                load(i, i);
                pad(i, i);
            }
        bool ok = true;
        int st = 0;
        uint32_t ph = 0;
        if (pre == p.stages && pre < n_iter) {
            for (int i = pre; i < n_iter && ok; ++i) {
                ok = tc_wait(empty0 + 8u * st, ph, p.err, 31);
                ok = __all_sync(0xffffffffu, ok);
                if (ok) {
                    load(i, st);
                    pad(i, st);
                }
                if (++st == p.stages) { st = 0; ph ^= 1u; }
            }
        }
        return;
    }
    pdl_wait();
    if (tracing) p.trace[2] = globaltimer_ns();          // predecessor complete
    auto sync_consumers = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(nw * 32) : "memory"); };
    const int f = f0 + lane;                           // epilogue: lane = feature, a warp takes every nw-th sequence
    const bool f_ok = f < p.N;
    const int seg_k = q.nq, seg_v = q.nq + q.nk, seg_g = seg_v + q.nv;
    const int part_of = MODE != TC_QKV ? 0 : (f0 < seg_k ? 0 : (f0 < seg_v ? 1 : (f0 < seg_g ? 2 : 3)));      // q | k | v | gate: whole heads
    const int fs = f - (part_of == 0 ? 0 : (part_of == 1 ? seg_k : (part_of == 2 ? seg_v : seg_g)));
    const int e0 = MODE == TC_QKV ? fs % q.hd : 0, head = MODE == TC_QKV ? fs / q.hd : 0;
    // what the epilogue needs from memory per sequence: residual value or RoPE factor. Those of the first four sequences are
    // requested here, the next four's while four are worked on.
    auto fetch4 = [&](int j0, float (&o)[4]) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = j0 + u * nw, b = b0 + j;
            o[u] = 0.f;
            if (j >= CT || b >= p.B || !f_ok) continue;
            if (MODE == TC_RESID) o[u] = ld_cg_f32_now(p.y + (size_t)b * p.N + f);
            if (MODE == TC_QKV && part_of < 2) o[u] = __ldg(q.rope + (size_t)c.pos[b] * q.hd + e0);
        }
    };
    float got4[4];
    if (MODE == TC_RESID || MODE == TC_QKV) fetch4(warp, got4);
    float sa = 1.0f, sa2 = 1.0f, gain = 0.f;
    if (W8 && f_ok) {
        sa = p.s1[f] * kGdScaleBack;
        if (MODE == TC_SWIGLU) sa2 = p.s2[f] * kGdScaleBack;
    }
    if (MODE == TC_RESID && f_ok) gain = p.gain_next[f];
    // per-sequence words of the epilogue, one sequence per thread: requested here, put into shared memory behind the products
    float tot = 0.f;
    int pos = -1;
    long long kvrow = 0;
    const bool word = tid < CT && b0 + tid < p.B;
    if (word) {
        if (p.ssq_in != nullptr) {
            const float4* sp = reinterpret_cast<const float4*>(p.ssq_in + (size_t)(b0 + tid) * p.ssq_parts);
#pragma unroll 4
            for (int t = 0; t < p.ssq_parts / 4; ++t) {
                const float4 x = __ldcg(sp + t);
                tot += (x.x + x.y) + (x.z + x.w);
            }
        }
        if (MODE == TC_QKV && seq_active(c, b0 + tid)) {
            pos = c.pos[b0 + tid];
            kvrow = (long long)q.page_table[kv_seq(c, b0 + tid) * q.pt_stride + pos / kKvBlock] * q.kv_heads * kKvBlock + (pos % kKvBlock);
        }
    }
    const int rt = warp % RT, seg = warp / RT;
    const int mlen = main_len(seg), n_main = up(mlen), xlen = ext_len(seg), n_all = n_main + up(xlen);
    float acc[2 * NP][4], ext[EXT2 ? 2 * NP : 1][4];
#pragma unroll
    for (int n = 0; n < 2 * NP; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
    if (EXT2) {
#pragma unroll
        for (int n = 0; n < 2 * NP; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) ext[EXT2 ? n : 0][j] = 0.f;
    }
    // shared-memory addresses of this lane's ldmatrix rows inside a stage (matrix mi, row mr): weight rows of 128 bytes (bf16) or 64
    // (codes, 64-byte swizzle), activation rows of 128
    const int mi = lane >> 3, mr = lane & 7, wrow = (rt & 1) * 16 + (mi & 1) * 8 + mr;
    const uint32_t ring0 = smem_u32(ring), wofs = (uint32_t)(seg * seg_bytes + G * (rt >> 1) * p.w_bytes), xofs = (uint32_t)(seg * seg_bytes + G * NA * p.w_bytes);
    uint32_t aofs[4], bofs[4], cofs[2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        aofs[j] = (uint32_t)(wrow * 128 + (((j * 2 + (mi >> 1)) ^ (wrow & 7)) << 4));
        bofs[j] = (uint32_t)(((mi >> 1) * 8 + mr) * 128 + (((j * 2 + (mi & 1)) ^ mr) << 4));
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) cofs[j] = (uint32_t)(wrow * 64 + (((2 * j + (mi >> 1)) ^ ((wrow >> 1) & 3)) << 4));
    bool ok = true;
    int st = 0;
    uint32_t ph = 0;
    for (int i = 0; i < n_iter; ++i) {
        if (ok && !tc_wait(full0 + 8u * st, ph, p.err, 32)) ok = false;
        const bool is_ext = i >= n_main;
        const bool codes = W8 && !is_ext;
        const int n_kb = i >= n_all ? 0 : (is_ext ? min(G, xlen - (i - n_main) * G) : min(G, mlen - i * G));
#pragma unroll 1
        for (int kb = 0; kb < n_kb; ++kb) {
            const uint32_t wb = ring0 + (uint32_t)(st * stage_bytes) + wofs + (uint32_t)(kb * (codes ? kGdF * 64 : kGdF * 128));
            const uint32_t xb = ring0 + (uint32_t)(st * stage_bytes) + xofs + (uint32_t)(kb * CT * 128);
            // operands of a k16 step are requested one step ahead of its products (ldmatrix is kept in program order)
            uint32_t cw[2][4], a[2][4], bf[2][NP][4];
            auto load = [&](int j, int o) {
                if (!codes) gd_ldsm4(wb + aofs[j], a[o]);
#pragma unroll
                for (int np = 0; np < NP; ++np) gd_ldsm4(xb + bofs[j] + np * 2048, bf[o][np]);
            };
            if (codes) {                               // two k16 steps each: rows r, r + 8 of the first, then of the second
                gd_ldsm4(wb + cofs[0], cw[0]);
                gd_ldsm4(wb + cofs[1], cw[1]);
            }
            load(0, 0);
#pragma unroll
            for (int j = 0; j < kTcKB / 16; ++j) {
                const int o = j & 1;
                if (j + 1 < kTcKB / 16) load(j + 1, o ^ 1);
                if (codes) {
                    gd_widen(cw[j >> 1][(j & 1) * 2], a[o][0], a[o][2]);
                    gd_widen(cw[j >> 1][(j & 1) * 2 + 1], a[o][1], a[o][3]);
                }
#pragma unroll
                for (int np = 0; np < NP; ++np) {
                    if (EXT2 && is_ext) {
                        gd_mma(ext[EXT2 ? 2 * np : 0], a[o], bf[o][np][0], bf[o][np][1]);
                        gd_mma(ext[EXT2 ? 2 * np + 1 : 0], a[o], bf[o][np][2], bf[o][np][3]);
                    } else {
                        gd_mma(acc[2 * np], a[o], bf[o][np][0], bf[o][np][1]);
                        gd_mma(acc[2 * np + 1], a[o], bf[o][np][2], bf[o][np][3]);
                    }
                }
            }
        }
        if (i + p.stages < n_iter) {
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive(empty0 + 8u * st);
        }
        if (++st == p.stages) { st = 0; ph ^= 1u; }
    }
    if (tid < CT) {
        rinv_s[tid] = p.ssq_in != nullptr ? 1.0f / sqrtf(tot / (float)p.K + p.eps) : 1.0f;
        if (MODE == TC_QKV) {
            pos_s[tid] = pos;
            kvrow_s[tid] = kvrow;
        }
    }
    // partial sums -> shared memory, over the ring (every stage has been read): [range][column][feature], then the second pair's
    sync_consumers();
    if (tracing) p.trace[3] = globaltimer_ns();          // products complete
    float* part = reinterpret_cast<float*>(ring);
    {
        const int r = lane >> 2, cq = (lane & 3) * 2;
        float* d = part + (size_t)seg * CT * FRP + rt * 16 + r;
#pragma unroll
        for (int n = 0; n < 2 * NP; ++n) {
            d[(n * 8 + cq) * FRP] = acc[n][0];
            d[(n * 8 + cq + 1) * FRP] = acc[n][1];
            d[(n * 8 + cq) * FRP + 8] = acc[n][2];
            d[(n * 8 + cq + 1) * FRP + 8] = acc[n][3];
        }
        if (EXT2) {
            float* e = d + (size_t)S * CT * FRP;
#pragma unroll
            for (int n = 0; n < 2 * NP; ++n) {
                e[(n * 8 + cq) * FRP] = ext[EXT2 ? n : 0][0];
                e[(n * 8 + cq + 1) * FRP] = ext[EXT2 ? n : 0][1];
                e[(n * 8 + cq) * FRP + 8] = ext[EXT2 ? n : 0][2];
                e[(n * 8 + cq + 1) * FRP + 8] = ext[EXT2 ? n : 0][3];
            }
        }
    }
    sync_consumers();
    // ---- epilogue ----------------------------------------------------------------------------------------------
    const int fo = W8 ? perm16(f) : f;                 // where the feature goes in a bf16 operand
    constexpr float opscale = W8 ? kOperandScale : 1.0f;
    auto finish = [&](int j, float got) {
        const int b = b0 + j;
        const float* pp = part + (size_t)j * FRP + lane;
        auto sum = [&](const float* a) {               // over the ranges, in their order
            float x = a[0];
            if (S > 1) x += a[CT * FRP];
            for (int s = 2; s < S; ++s) x += a[s * CT * FRP];
            return x;
        };
        float v = sum(pp);
        const float rinv = rinv_s[j];
        if (MODE == TC_RAW) {
            if (W8) v *= sa;
            if (f_ok) p.y[(size_t)b * p.N + f] = v * rinv;
        } else if (MODE == TC_SWIGLU) {
            float u = sum(pp + 32);
            if (W8) {
                v *= sa;
                u *= sa2;
            }
            const float g = v * rinv, up = u * rinv;
            if (f_ok) p.h16[(size_t)b * p.N + fo] = __float2bfloat16_rn(__fdividef(g, 1.0f + __expf(-g)) * up * opscale);       // inference.cu:262-281
        } else if (MODE == TC_RESID) {
            if (W8) {
                const float u = sum(pp + S * CT * FRP);
                v = fmaf(v, sa, u);                    // gemm_tc_kernel's rounding: one fma, then the residual
            }
            const float xn = __fadd_rn(v, got);        // inference.cu:252-260, :283-291
            if (f_ok) {
                p.y[(size_t)b * p.N + f] = xn;
                p.xg16[(size_t)b * p.N + fo] = __float2bfloat16_rn(xn * gain * opscale);
            }
            const float ss = warp_sum(f_ok ? __fmul_rn(xn, xn) : 0.f);
            if (lane == 0) p.ssq_out[(size_t)b * p.ssq_parts + blockIdx.x] = ss;
        } else {
            if (W8) v *= sa;
            v *= rinv;
            // RoPE on adjacent pairs (inference.cu:113-134): the even lane holds the cosine, the odd one the sine
            const float oth = __shfl_xor_sync(0xffffffffu, v, 1), gth = __shfl_xor_sync(0xffffffffu, got, 1);
            const int pos = pos_s[j];
            if (pos < 0) return;                       // uniform
            if (part_of < 2) {
                const float cs = (lane & 1) ? gth : got, sn = (lane & 1) ? got : gth;
                const float rot = (lane & 1) ? fmaf(sn, oth, cs * v) : fmaf(cs, v, -(sn * oth));
                if (part_of == 0) q.qbuf[(size_t)b * q.nq + fs] = rot;
                else Elem<KVT>::put(reinterpret_cast<KVT*>(q.kpool), ((size_t)kvrow_s[j] + (size_t)head * kKvBlock) * q.hd + e0, rot);
            } else if (part_of == 2) {
                Elem<KVT>::put(reinterpret_cast<KVT*>(q.vpool), ((size_t)kvrow_s[j] + (size_t)head * kKvBlock) * q.hd + e0, v);
            } else {
                q.gbuf[(size_t)b * q.ng + fs] = __fdividef(1.0f, 1.0f + __expf(-v));      // inference.cu:248
            }
        }
    };
#pragma unroll 1
    for (int j0 = warp; j0 < CT; j0 += 4 * nw) {
        float cur[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) cur[u] = got4[u];
        if (MODE == TC_RESID || MODE == TC_QKV) fetch4(j0 + 4 * nw, got4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = j0 + u * nw;
            if (j < CT && b0 + j < p.B) finish(j, cur[u]);      // uniform
        }
    }
    if (tracing) p.trace[4] = globaltimer_ns();          // epilogue done
}

}  // namespace mlb
