// One step as a chain of launches on the session's stream: GEMV chain, tensor-core chain, or the whole-GPU kernels.
#pragma once
#include <algorithm>
#include <type_traits>

#include "session.h"
#include "step_shapes.h"
#include "grid_host.h"
#include "lean_host.h"
#include "sgemv.cuh"
#include "attn_decode.cuh"

namespace mlb {

static int pick_bt(int B, size_t per_seq_floats) {
    int bt = B >= 8 ? 8 : (B >= 4 ? 4 : (B >= 2 ? 2 : 1));
    while (bt > 1 && (size_t)bt * per_seq_floats * 4 > 200 * 1024) bt >>= 1;
    return bt;
}

// Launch with the programmatic-dependent-launch attribute: the kernel may start while its
// predecessor in the stream still runs and orders itself with griddepcontrol.wait.
template <typename... KArgs, typename... Args>
static cudaError_t launch_chain(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                Args... args) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// launch_chain for a grid whose z extent is one thread-block cluster (cluster_z CTAs share an output tile).
template <typename... KArgs, typename... Args>
static cudaError_t launch_cluster(bool pdl, int cluster_z, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                  Args... args) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    if (cluster_z > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = (unsigned)cluster_z;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

template <typename T, typename T2, typename KVT>
struct Chain {
    // TMA-streamed variant: one contiguous slab of rows per CTA (one head per CTA for QKV).
    template <int MODE>
    static int sgemv(mlb_session* s, const StepCtl& c, GemvParams p, Recorder* rec, const char* name, bool* done) {
        *done = false;
        // Worth it only when the matrix is large: below a few MB the per-thread-load kernel's
        // shorter latency chain wins (measured on the 1-GPU latency configuration).
        const size_t mat_bytes = (size_t)p.N * p.K * sizeof(T) * (MODE == GEMV_SWIGLU ? 2 : 1);
        if (!s->force_sgemv && mat_bytes < (4u << 20)) return MLB_OK;
        SgemvGeom g;
        g.stage_bytes = s->sg_stage_kb * 1024;
        if ((size_t)p.K * sizeof(T) > (size_t)g.stage_bytes || (size_t)p.Kp * sizeof(T2) > (size_t)g.stage_bytes) return MLB_OK;
        int grid_x;
        if (MODE == GEMV_QKV) {
            // whole heads when the per-head norm needs them, else 32-row groups (RoPE pairs stay together)
            g.rows_per_cta = p.qk_norm ? p.hd : 32;
            grid_x = p.N / g.rows_per_cta;
        } else {
            const int n_ctas = std::max(1, std::min(s->sm_count, (p.N + 3) / 4));
            g.rows_per_cta = (p.N + n_ctas - 1) / n_ctas;
            grid_x = (p.N + g.rows_per_cta - 1) / g.rows_per_cta;
        }
        auto up4 = [](int v) { return (v + 3) / 4 * 4; };
        g.xs_stride = up4(p.K); g.xs2_stride = up4(std::max(p.Kp, 4)); g.outs_stride = up4(std::max(p.hd, 64)); g.pacc_stride = up4(g.rows_per_cta + 4);
        // no more sequences per CTA than leave three stages; without room for one the other GEMV serves
        int bt = sg_sequences(s->B, grid_x, s->sm_count);
        size_t fixed = 0;
        for (;; --bt) {
            if (bt == 0) return MLB_OK;
            int off = 0;
            g.off_xs = off; off += bt * g.xs_stride;
            g.off_xs2 = off; off += bt * g.xs2_stride;
            g.off_outs = off; off += bt * g.outs_stride;
            g.off_pacc = off; off += bt * g.pacc_stride;
            g.off_red = off; off += 64;
            off = (off + 31) / 32 * 32;
            g.off_bar = off; off += 8 * 4;
            off = (off + 31) / 32 * 32;
            g.off_ring = off;
            fixed = (size_t)off * 4;
            if (fixed + 3 * (size_t)g.stage_bytes <= 210 * 1024) break;
        }
        g.n_stages = (int)std::min<size_t>(s->sg_max_stages, (210 * 1024 - fixed) / g.stage_bytes);
        g.err = s->dev_err;
        const size_t smem = fixed + (size_t)g.n_stages * g.stage_bytes;
        if (rec) {
            const uint64_t wbytes = (uint64_t)p.N * p.K * sizeof(T) * (MODE == GEMV_SWIGLU ? 2 : 1) +
                                    (uint64_t)p.N * p.Kp * sizeof(T2) + (p.wscale ? (uint64_t)p.N * 4 : 0);
            const uint64_t abytes = (uint64_t)s->B * ((uint64_t)p.K + p.N) * 4;
            int rc = rec->begin(name, wbytes + abytes, 2ull * p.N * (p.K + p.Kp) * s->B * (MODE == GEMV_SWIGLU ? 2 : 1));
            if (rc) return rc;
        }
        const dim3 grid(grid_x, (s->B + bt - 1) / bt), block(kSgThreads);
        cudaError_t e;
        switch (bt) {
            case 1: e = launch_chain(s->use_pdl, sgemv_kernel<T, T2, KVT, 1, MODE>, grid, block, smem, s->stream, c, p, g); break;
            case 2: e = launch_chain(s->use_pdl, sgemv_kernel<T, T2, KVT, 2, MODE>, grid, block, smem, s->stream, c, p, g); break;
            default: e = launch_chain(s->use_pdl, sgemv_kernel<T, T2, KVT, 3, MODE>, grid, block, smem, s->stream, c, p, g); break;
        }
        if (e != cudaSuccess) return fail(MLB_E_CUDA, "launch of %s (streamed) failed: %s", name, cudaGetErrorString(e));
        *done = true;
        if (rec) return rec->end();
        return MLB_OK;
    }

    template <int MODE>
    static int gemv(mlb_session* s, const StepCtl& c, GemvParams p, int R, Recorder* rec, const char* name) {
        if (s->use_sgemv) {
            bool done = false;
            int rc = sgemv<MODE>(s, c, p, rec, name, &done);
            if (rc || done) return rc;
        }
        p.R = R;
        const size_t per_seq = (size_t)p.K + p.Kp + R + 1 + 8;
        const int BT = pick_bt(s->B, per_seq);
        if (per_seq * 4 > 200 * 1024) return fail(MLB_E_UNSUPPORTED, "projection input of %d floats does not fit shared memory", p.K);
        const int rwf = BT == 1 ? 2 : 4;                                  // GemvShape<BT>::RW
        const int rw = MODE == GEMV_SWIGLU ? rwf / 2 : rwf;
        const int warps = std::max(1, std::min(8, (R + rw - 1) / rw));
        dim3 grid((p.N + R - 1) / R, (s->B + BT - 1) / BT);
        const size_t smem = (size_t)BT * per_seq * 4;
        if (rec) {
            const uint64_t wbytes = (uint64_t)p.N * p.K * sizeof(T) * (MODE == GEMV_SWIGLU ? 2 : 1) +
                                    (uint64_t)p.N * p.Kp * sizeof(T2) + (p.wscale ? (uint64_t)p.N * 4 : 0);
            const uint64_t abytes = (uint64_t)s->B * ((uint64_t)p.K + p.N) * 4;
            int rc = rec->begin(name, wbytes + abytes, 2ull * p.N * (p.K + p.Kp) * s->B * (MODE == GEMV_SWIGLU ? 2 : 1));
            if (rc) return rc;
        }
        cudaError_t e;
        switch (BT) {
            case 1: e = launch_chain(s->use_pdl, gemv_kernel<T, T2, KVT, 1, MODE>, grid, dim3(warps * 32), smem, s->stream, c, p); break;
            case 2: e = launch_chain(s->use_pdl, gemv_kernel<T, T2, KVT, 2, MODE>, grid, dim3(warps * 32), smem, s->stream, c, p); break;
            case 4: e = launch_chain(s->use_pdl, gemv_kernel<T, T2, KVT, 4, MODE>, grid, dim3(warps * 32), smem, s->stream, c, p); break;
            default: e = launch_chain(s->use_pdl, gemv_kernel<T, T2, KVT, 8, MODE>, grid, dim3(warps * 32), smem, s->stream, c, p); break;
        }
        if (e != cudaSuccess) return fail(MLB_E_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e));
        if (rec) return rec->end();
        return MLB_OK;
    }

    template <int MODE>
    static int configure_mode() {
        const int big = 200 * 1024;
        CU(cudaFuncSetAttribute(sgemv_kernel<T, T2, KVT, 1, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 212 * 1024));
        CU(cudaFuncSetAttribute(sgemv_kernel<T, T2, KVT, 2, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 212 * 1024));
        CU(cudaFuncSetAttribute(sgemv_kernel<T, T2, KVT, 3, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 212 * 1024));
        CU(cudaFuncSetAttribute(gemv_kernel<T, T2, KVT, 1, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CU(cudaFuncSetAttribute(gemv_kernel<T, T2, KVT, 2, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CU(cudaFuncSetAttribute(gemv_kernel<T, T2, KVT, 4, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CU(cudaFuncSetAttribute(gemv_kernel<T, T2, KVT, 8, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        return MLB_OK;
    }
    static int configure() {
        int rc;
        if ((rc = configure_mode<GEMV_RAW>())) return rc;
        if ((rc = configure_mode<GEMV_RESID>())) return rc;
        if ((rc = configure_mode<GEMV_SWIGLU>())) return rc;
        if ((rc = configure_mode<GEMV_QKV>())) return rc;
        if ((rc = configure_mode<GEMV_LMHEAD>())) return rc;
        return MLB_OK;
    }

    template <int HD>
    static int attn_g(mlb_session* s, const StepCtl& c, const AttnParams& p0, int G) {
        AttnParams p = p0;
        p.hg = 1;
        // few CTAs (small batch): two query heads per CTA, G/2 CTAs per kv head (cfg4 at batch 1: 1.28 -> 1.14 ms
        // per step); with the GPU already full the extra CTAs only re-read K/V (62 -> 69 us at 64 sequences)
        if (G >= 4 && G % 2 == 0 && s->splits * p.kv_heads * s->B < 2 * s->sm_count) { p.hg = G / 2; G = 2; }
        p.splits = s->splits;
        const dim3 grid = attn_grid(p, s->B, s->sm_count);
        auto launch = [&](auto kernel, int threads, size_t smem) { return launch_chain(s->use_pdl, kernel, grid, dim3(threads), smem, s->stream, c, p); };
        cudaError_t e;
        switch (G) {
            case 1: e = attn_with_kernel<KVT, HD, 1>(p, grid, s->sm_count, launch); break;
            case 2: e = attn_with_kernel<KVT, HD, 2>(p, grid, s->sm_count, launch); break;
            case 4: e = attn_with_kernel<KVT, HD, 4>(p, grid, s->sm_count, launch); break;
            default: e = attn_with_kernel<KVT, HD, 8>(p, grid, s->sm_count, launch); break;
        }
        if (e != cudaSuccess) return fail(MLB_E_CUDA, "attention launch failed: %s", cudaGetErrorString(e));
        return MLB_OK;
    }

    // Launch shape of the embedding kernel: with per-layer embeddings and a small batch, the rows
    // of a sequence are spread over several CTAs of 64 threads (one projection row per thread).
    static int embed_split(int B, int d, int ple) {
        if (ple <= 0) return 1;
        return std::max(1, std::min((d + 63) / 64, 1024 / std::max(1, B)));
    }
    static dim3 embed_grid(int B, int d, int ple) { return dim3(B, embed_split(B, d, ple)); }
    static dim3 embed_block(int B, int d, int ple) { return dim3(embed_split(B, d, ple) > 1 ? 64 : 256); }

    // One decode (or prefill) step of a batch-1 session as a single cooperative kernel over all
    // SMs (plus the sampler for top-k).
    static int run_grid(mlb_session* s, int kind, const StepCtl& c, Recorder* rec, int* n_launches) {
        int rc, launches = 0;
        if (rec) {
            uint64_t w, kv, st, rows;
            mlb_session_step_bytes(s, &w, &kv, &st, &rows);
            if ((rc = rec->begin(s->use_lean ? "lean_decode_step" : "grid_decode_step", w + kv + st + rows, 0))) return rc;
        }
        if (s->use_lean) {
            LeanParams lp = s->lean;
            lp.tok_arg = s->tok_arg;
            lp.with_lm_head = kind == CHAIN_PREFILL ? 0 : 1;
            lp.do_pick = kind == CHAIN_GREEDY ? 1 : 0;
            CU(lean_kernel_launch(s->lean_idx, s->m->cfg.kv_dtype, s->lean_smem, s->stream, c, lp));
        } else {
            GridParams gp = s->grid;
            gp.tok_arg = s->tok_arg;
            gp.with_lm_head = kind == CHAIN_PREFILL ? 0 : 1;
            gp.do_pick = kind == CHAIN_GREEDY ? 1 : 0;
            CU(grid_kernel_launch(s->m->cfg.weight_dtype, s->m->cfg.kv_dtype, s->grid_ctas, s->grid_smem, s->stream, c, gp));
        }
        if (rec && (rc = rec->end())) return rc;
        ++launches;
        if (kind == CHAIN_TOPK) {
            SampleParams sp;
            sp.logits = s->logits; sp.V = s->m->cfg.vocab; sp.top_k = s->cur_topk; sp.temperature = s->cur_temp; sp.seeds = s->seeds;
            if (rec && (rc = rec->begin("sample_topk_philox", (uint64_t)s->B * s->m->cfg.vocab * 4 * 5, 0))) return rc;
            CU(launch_chain(false, sample_topk_kernel, dim3(s->B), dim3(kPickThreads), 0, s->stream, c, sp));
            if (rec && (rc = rec->end())) return rc;
            ++launches;
        }
        if (n_launches) *n_launches = launches;
        return MLB_OK;
    }

    // The same on mma.sync tiles (gemm_dec.cuh), for decode batches.
    template <int MODE>
    static int gemm_dec(mlb_session* s, const StepCtl& c, const CUtensorMap& A, const CUtensorMap& A2, const CUtensorMap* Bmaps, int N, int K,
                        float* y, bf16_t* h16, bool normed, const float* next_gain, const mlb_session::TcLayerMaps* ext,
                        const QkvPostParams* q, const float* sA, const float* sA2, Recorder* rec, const char* name) {
        const int ple = s->m->cfg.ple_dim, na = MODE == TC_SWIGLU ? 2 : 1;
        constexpr bool w8 = sizeof(T) == 1;
        using KVQ = typename std::conditional<MODE == TC_QKV, KVT, float>::type;      // only the projection of q, k, v writes the cache
        GemmDecParams p;
        p.nkb_x = ext ? (ple + kTcKB - 1) / kTcKB : 0;
        const GdShape g = gd_pick(s, N, (K + kTcKB - 1) / kTcKB + p.nkb_x, MODE, w8, ext != nullptr);
        p.N = N; p.K = K; p.B = s->B; p.split = g.split; p.G = g.g; p.stages = g.stages; p.w_bytes = g.w_bytes;
        p.y = y; p.h16 = h16; p.ssq_in = normed ? s->tc_ssq : nullptr; p.ssq_parts = (s->m->cfg.dim + kTcM - 1) / kTcM * 4; p.eps = s->m->cfg.rms_eps;
        p.xg16 = s->xn16; p.gain_next = next_gain; p.ssq_out = s->tc_ssq; p.s1 = sA; p.s2 = sA2; p.err = s->dev_err;
        p.trace = s->tc_trace ? s->tc_trace + 8 * (size_t)(s->tc_trace_n++ % 64) : nullptr;
        int rc;
        if (rec && (rc = rec->begin(name, ((uint64_t)N * K * sizeof(T) + (uint64_t)N * (ext ? ple : 0) * 2) * na + (uint64_t)s->B * K * 2 + (uint64_t)s->B * N * 4,
                                    2ull * N * (K + (ext ? ple : 0)) * s->B * na)))
            return rc;
        const dim3 grid((N + kGdF - 1) / kGdF, (s->B + 16 * g.np - 1) / (16 * g.np)), block(32 * (2 * na * g.split + 1));
        const CUtensorMap &X = Bmaps[gd_index(g.np, g.g)], &Ax = ext ? ext->pleP : A, &Bx = ext ? ext->pleT : A;
        const QkvPostParams q0{};
        cudaError_t e;
        switch (g.np) {
            case 1: e = launch_chain(s->use_pdl, gemm_dec_kernel<MODE, KVQ, T, 1>, grid, block, g.smem, s->stream, A, A2, X, Ax, Bx, p, c, q ? *q : q0); break;
            case 2: e = launch_chain(s->use_pdl, gemm_dec_kernel<MODE, KVQ, T, 2>, grid, block, g.smem, s->stream, A, A2, X, Ax, Bx, p, c, q ? *q : q0); break;
            default: e = launch_chain(s->use_pdl, gemm_dec_kernel<MODE, KVQ, T, 4>, grid, block, g.smem, s->stream, A, A2, X, Ax, Bx, p, c, q ? *q : q0); break;
        }
        if (e != cudaSuccess) return fail(MLB_E_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e));
        if (rec) return rec->end();
        return MLB_OK;
    }

    // One tensor-core projection. `normed`: the activation operand is bf16(x * gain) and the accumulator
    // columns are scaled by 1 / rms(x) from the partial sums its producer left. `next_gain` (RESID): also
    // write the operand and the partial sums for the next norm. `ext`: the per-layer embedding pair whose
    // k-blocks follow the main operands' (RESID of the down projection).
    template <int MODE>
    static int gemm_tc(mlb_session* s, const StepCtl& c, const CUtensorMap& A, const CUtensorMap& A2, const CUtensorMap* Bmaps, int N, int K,
                       float* y, bf16_t* h16, bool normed, const float* next_gain, const mlb_session::TcLayerMaps* ext,
                       const QkvPostParams* q, const float* sA, const float* sA2, Recorder* rec, const char* name) {
        if (s->use_dec) return gemm_dec<MODE>(s, c, A, A2, Bmaps, N, K, y, h16, normed, next_gain, ext, q, sA, sA2, rec, name);
        GemmTcParams p;
        const int ple = s->m->cfg.ple_dim;
        const int na = MODE == TC_SWIGLU ? 2 : 1;
        p.nkb_x = ext ? (ple + kTcKB - 1) / kTcKB : 0;
        constexpr bool w8 = sizeof(T) == 1;
        const int nacc = (MODE == TC_SWIGLU || (w8 && MODE == TC_RESID)) ? 2 : 1;
        const TcShape sh = ext ? s->tc_shape_down : tc_pick_shape(s, s->B, N, (K + kTcKB - 1) / kTcKB, na, w8, nacc);
        if (sh.nb == 0) return fail(MLB_E_UNSUPPORTED, "%s: no launch shape fits", name);
        const int nb = sh.nb;
        p.N = N; p.K = K; p.B = s->B; p.Nb = nb;
        p.stages = sh.stages; p.group = sh.group; p.tmem_cols = sh.tmem_cols;
        p.y = y; p.resid = MODE == TC_RESID ? y : nullptr; p.h16 = h16; p.err = s->dev_err;
        p.sA = sA; p.sA2 = sA2;
        p.trace = s->tc_trace ? s->tc_trace + 8 * (size_t)(s->tc_trace_n++ % 64) : nullptr;
        p.ssq_in = normed ? s->tc_ssq : nullptr; p.ssq_parts = (s->m->cfg.dim + kTcM - 1) / kTcM * 4; p.eps = s->m->cfg.rms_eps;
        p.xg16 = next_gain ? s->xn16 : nullptr; p.gain_next = next_gain; p.ssq_out = next_gain ? s->tc_ssq : nullptr;
        const size_t smem = sh.smem;
        dim3 grid((N + kTcM - 1) / kTcM, (s->B + nb - 1) / nb, sh.split);
        int rc;
        if (rec && (rc = rec->begin(name, ((uint64_t)N * K * sizeof(T) + (uint64_t)N * (ext ? ple : 0) * 2) * na + (uint64_t)s->B * K * 2 + (uint64_t)s->B * N * 4,
                                    2ull * N * (K + (ext ? ple : 0)) * s->B * na)))
            return rc;
        QkvPostParams q0{};
        const CUtensorMap& Ax = ext ? ext->pleP : A;
        const CUtensorMap& Bx = ext ? ext->pleT : A;
        cudaError_t e = launch_cluster(s->use_pdl, sh.split, gemm_tc_kernel<MODE, KVT, T>, grid, dim3(kTcThreads), smem, s->stream, A, A2, Bmaps[nb_index(nb)], Ax, Bx, p,
                                       c, q ? *q : q0);
        if (e != cudaSuccess) return fail(MLB_E_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e));
        if (rec) return rec->end();
        return MLB_OK;
    }

    // Large-batch step: projections as tcgen05 GEMMs on bf16 operands with the element-wise work in their
    // epilogues; per layer: projection, attention / delta-net, o-projection, gate-up, down.
    static int run_tc(mlb_session* s, int kind, const StepCtl& c, Recorder* rec, int* n_launches) {
        if (std::is_same<T, float>::value) return fail(MLB_E_UNSUPPORTED, "tensor-core projections need bf16 or FP8 weights");
        const mlb_model* m = s->m;
        const mlb_config& cfg = m->cfg;
        const int d = cfg.dim, F = cfg.ffn_dim, B = s->B, ple = cfg.ple_dim;
        const int perm = s->use_dec && sizeof(T) == 1 ? 1 : 0;       // operand order of the FP8 decode GEMMs
        int launches = 0, rc;
        if (rec && (rc = rec->begin("embed_ple_gather_norm", (uint64_t)B * d * 8 + (uint64_t)B * ple * 2 * cfg.layers, 0))) return rc;
        // (without overlap: what the step's kernels read before they wait for their predecessor was written by earlier steps)
        CU(launch_chain(false, embed_tc_kernel<T>, dim3(B, (d + kTcM - 1) / kTcM), dim3(128), (size_t)ple * 4, s->stream, c,
                        static_cast<const T*>(m->E), static_cast<const float*>(m->Es), d, static_cast<const StepLayer*>(s->step_layers), cfg.layers, ple,
                        static_cast<const float*>(m->layers[0].g1), s->x, s->xn16, s->tc_ssq, s->tple16, perm));
        if (rec && (rc = rec->end())) return rc;
        ++launches;
        for (int i = 0; i < cfg.layers; ++i) {
            const DevLayer& L = m->layers[i];
            const mlb_session::TcLayerMaps& M = s->tc_maps[i];
            if (L.type == MLB_LAYER_ATTENTION) {
                QkvPostParams q;
                q.nq = L.nq; q.nk = L.nk; q.nv = L.nv; q.ng = L.ng; q.hd = cfg.head_dim;
                q.kv_heads = cfg.kv_heads; q.qk_norm = cfg.qk_norm; q.eps = cfg.rms_eps; q.gq = L.gq; q.gk = L.gk; q.rope = m->rope;
                q.kpool = s->kpool[i]; q.vpool = s->vpool[i]; q.page_table = s->page_table; q.pt_stride = s->max_pages;
                q.qbuf = s->qbuf; q.gbuf = s->gbuf;
                if ((rc = gemm_tc<TC_QKV>(s, c, M.qkv, M.qkv, s->tc_g.xn, L.n_qkv, d, nullptr, nullptr, true, nullptr, nullptr, &q, L.Sqkv, nullptr, rec,
                                          s->use_dec ? "qkv_gemm_mma_norm_rope_kvappend" : "qkv_gemm_tcgen05_norm_rope_kvappend")))
                    return rc;
                ++launches;
                AttnParams a;
                a.kpool = s->kpool[i]; a.vpool = s->vpool[i];
                a.page_table = s->page_table; a.pt_stride = s->max_pages;
                a.qbuf = s->qbuf; a.gbuf = L.ng ? s->gbuf : nullptr; a.abuf = s->abuf; a.abuf16 = s->a16; a.perm = perm;
                a.part = s->part; a.ticket = s->attn_ticket;
                a.heads = cfg.heads; a.kv_heads = cfg.kv_heads; a.num_pages = 0; a.err = s->dev_err; a.min_pages_per_split = s->attn_min_pps; a.early = 1;
                if (rec) {
                    uint64_t kvb = 0, fl = 0;
                    for (int b = 0; b < B; ++b) {
                        if (!seq_live(s, b)) continue;
                        kvb += 2ull * cfg.kv_heads * cfg.head_dim * sizeof(KVT) * (s->h_pos[b] + 1);
                        fl += 4ull * cfg.heads * cfg.head_dim * (s->h_pos[b] + 1);
                    }
                    if ((rc = rec->begin("attn_flash_decode_paged", kvb, fl))) return rc;
                }
                const int G = cfg.heads / cfg.kv_heads;
                if (s->parent && !s->as_steps && std::is_same<KVT, bf16_t>::value) {
                    AttnColsParams ac;
                    ac.kpool = static_cast<const bf16_t*>(s->kpool[i]); ac.vpool = static_cast<const bf16_t*>(s->vpool[i]);
                    ac.page_table = s->page_table; ac.pt_stride = s->max_pages;
                    ac.qbuf = s->qbuf; ac.gbuf = L.ng ? s->gbuf : nullptr; ac.out16 = s->a16;
                    ac.heads = cfg.heads; ac.kv_heads = cfg.kv_heads;
                    ac.hdr = s->plan.hdr; ac.tiles = reinterpret_cast<const int4*>(s->plan.tiles);
                    CU(attn_cols_launch(cfg.head_dim, G, s->use_pdl, s->plan.max_tiles, s->stream, ac));
                } else {
                    if (cfg.head_dim == 64) rc = attn_g<64>(s, c, a, G); else rc = attn_g<128>(s, c, a, G);
                    if (rc) return rc;
                }
                if (rec && (rc = rec->end())) return rc;
                ++launches;
            } else {
                if ((rc = gemm_tc<TC_RAW>(s, c, M.qkv, M.qkv, s->tc_g.xn, L.n_qkv, d, s->raw, nullptr, true, nullptr, nullptr, nullptr, L.Sqkv, nullptr, rec,
                                          s->use_dec ? "deltanet_proj_gemm_mma" : "deltanet_proj_gemm_tcgen05")))
                    return rc;
                ++launches;
                const int dk = cfg.dn_key_dim, dv = cfg.dn_value_dim, H = cfg.heads;
                if (rec && (rc = rec->begin("deltanet_state_update", (uint64_t)B * 2ull * H * dk * dv * 4, (uint64_t)B * 6ull * H * dk * dv))) return rc;
                if (s->parent) {
                    // prompt columns: the recurrence runs over the columns of a sequence in order
                    CU(delta_cols(s, i, nullptr, s->a16));
                } else {
                    dim3 grid((dv + 31) / 32, H, B);
                    if (dk == 64) CU(launch_chain(s->use_pdl, delta_net_kernel<64>, grid, dim3(256), 0, s->stream, c, static_cast<const float*>(s->raw), s->raw_stride, s->state[i], H, dv, s->abuf, s->a16, perm, 1e-6f));
                    else CU(launch_chain(s->use_pdl, delta_net_kernel<128>, grid, dim3(256), 0, s->stream, c, static_cast<const float*>(s->raw), s->raw_stride, s->state[i], H, dv, s->abuf, s->a16, perm, 1e-6f));
                }
                if (rec && (rc = rec->end())) return rc;
                ++launches;
            }
            const CUtensorMap* amap = L.type == MLB_LAYER_ATTENTION ? s->tc_g.a_attn : s->tc_g.a_dn;
            if ((rc = gemm_tc<TC_RESID>(s, c, M.o, M.o, amap, d, L.o_in, s->x, nullptr, false, L.g2, nullptr, nullptr, L.So, nullptr, rec,
                                        s->use_dec ? "oproj_gemm_mma_residual_norm" : "oproj_gemm_tcgen05_residual_norm")))
                return rc;
            ++launches;
            if ((rc = gemm_tc<TC_SWIGLU>(s, c, M.w1a, M.w1b, s->tc_g.xn, F, d, nullptr, s->h16, true, nullptr, nullptr, nullptr, L.S1a, L.S1b, rec,
                                         s->use_dec ? "ffn_gateup_gemm_mma_swiglu" : "ffn_gateup_gemm_tcgen05_swiglu")))
                return rc;
            ++launches;
            const bool last = i + 1 == cfg.layers;
            const float* g_next = last ? m->g_final : m->layers[i + 1].g1;
            if ((rc = gemm_tc<TC_RESID>(s, c, M.w2, M.w2, s->tc_g.h, d, F, s->x, nullptr, false, g_next,
                                        (!last && ple > 0) ? &s->tc_maps[i + 1] : nullptr, nullptr, L.S2, nullptr, rec, s->use_dec ? "ffn_down_gemm_mma_residual_ple_norm" : "ffn_down_gemm_tcgen05_residual_ple_norm")))
                return rc;
            ++launches;
        }
        if (kind == CHAIN_PREFILL && s->parent) {
            // prompt columns: positions and tokens of the next chunk come from the host
        } else if (kind == CHAIN_PREFILL) {
            if (rec && (rc = rec->begin("advance_prompt", (uint64_t)B * 12, 0))) return rc;
            CU(launch_chain(s->use_pdl, advance_kernel, dim3((B + 127) / 128), dim3(128), 0, s->stream, c));
            if (rec && (rc = rec->end())) return rc;
            ++launches;
        } else {
            if ((rc = gemm_tc<TC_RAW>(s, c, s->tc_g.E, s->tc_g.E, s->tc_g.xn, cfg.vocab, d, s->logits, nullptr, true, nullptr, nullptr, nullptr, static_cast<const float*>(m->Es), nullptr, rec,
                                      s->use_dec ? "lmhead_gemm_mma" : "lmhead_gemm_tcgen05")))
                return rc;
            ++launches;
            if (s->parent) {
                // columns that are scored: their logits are the result
            } else if (kind == CHAIN_GREEDY) {
                if (rec && (rc = rec->begin("argmax_pick", (uint64_t)B * cfg.vocab * 4, 0))) return rc;
                CU(launch_chain(s->use_pdl, argmax_advance_kernel, dim3(B), dim3(kPickThreads), 0, s->stream, c, static_cast<const float*>(s->logits), cfg.vocab));
                if (rec && (rc = rec->end())) return rc;
            } else {
                SampleParams sp;
                sp.logits = s->logits; sp.V = cfg.vocab; sp.top_k = s->cur_topk; sp.temperature = s->cur_temp; sp.seeds = s->seeds;
                if (rec && (rc = rec->begin("sample_topk_philox", (uint64_t)B * cfg.vocab * 4 * 5, 0))) return rc;
                CU(launch_chain(s->use_pdl, sample_topk_kernel, dim3(B), dim3(kPickThreads), 0, s->stream, c, sp));
                if (rec && (rc = rec->end())) return rc;
            }
            ++launches;
        }
        if (n_launches) *n_launches = launches;
        return MLB_OK;
    }

    // One decode (or prefill) step as a chain of launches on the session's stream.
    static int run(mlb_session* s, int kind, Recorder* rec, int* n_launches) {
        const mlb_model* m = s->m;
        const mlb_config& cfg = m->cfg;
        const StepCtl c = make_ctl(s, kind);
        const int d = cfg.dim, F = cfg.ffn_dim, B = s->B, p = cfg.ple_dim;
        int launches = 0, rc;
        if (s->use_lean || s->use_grid) return run_grid(s, kind, c, rec, n_launches);
        if (s->use_tc) return run_tc(s, kind, c, rec, n_launches);

        if (rec && (rc = rec->begin("embed_ple_gather", (uint64_t)B * (d * sizeof(T) + (uint64_t)p * sizeof(T2) + (uint64_t)d * 4) + (uint64_t)d * p * sizeof(T2), 0))) return rc;
        // (without overlap: what the step's kernels read before they wait for their predecessor was written by earlier steps)
        CU(launch_chain(false, embed_kernel<T, T2>, embed_grid(B, d, p), embed_block(B, d, p), (size_t)p * 4, s->stream, c,
                        static_cast<const T*>(m->E), static_cast<const float*>(m->Es), d, static_cast<const T2*>(m->layers[0].pleT),
                        static_cast<const T2*>(m->layers[0].pleP), p, s->x));
        if (rec && (rc = rec->end())) return rc;
        ++launches;

        for (int i = 0; i < cfg.layers; ++i) {
            const DevLayer& L = m->layers[i];
            GemvParams g;
            std::memset(&g, 0, sizeof g);
            g.W = L.Wqkv; g.wscale = L.Sqkv; g.N = L.n_qkv; g.K = d;
            g.xin = s->x; g.gain = L.g1; g.eps = cfg.rms_eps; g.do_norm = 1;
            if (L.type == MLB_LAYER_ATTENTION) {
                g.nq = L.nq; g.nk = L.nk; g.nv = L.nv; g.ng = L.ng;
                g.hd = cfg.head_dim; g.kv_heads = cfg.kv_heads; g.qk_norm = cfg.qk_norm;
                g.gq = L.gq; g.gk = L.gk; g.rope = m->rope;
                g.kpool = s->kpool[i]; g.vpool = s->vpool[i];
                g.page_table = s->page_table; g.pt_stride = s->max_pages;
                g.qbuf = s->qbuf; g.gbuf = s->gbuf;
                const int R = cfg.qk_norm ? cfg.head_dim : 16;
                if ((rc = gemv<GEMV_QKV>(s, c, g, R, rec, "qkv_gemv_norm_rope_kvappend"))) return rc;
                ++launches;
                AttnParams a;
                a.kpool = s->kpool[i]; a.vpool = s->vpool[i];
                a.page_table = s->page_table; a.pt_stride = s->max_pages;
                a.qbuf = s->qbuf; a.gbuf = L.ng ? s->gbuf : nullptr; a.abuf = s->abuf; a.abuf16 = nullptr; a.perm = 0;
                a.part = s->part; a.ticket = s->attn_ticket;
                a.heads = cfg.heads; a.kv_heads = cfg.kv_heads; a.num_pages = 0; a.err = s->dev_err; a.min_pages_per_split = s->attn_min_pps; a.early = 1;
                if (rec) {
                    uint64_t kvb = 0, fl = 0;
                    for (int b = 0; b < B; ++b) {
                        if (!seq_live(s, b)) continue;
                        kvb += 2ull * cfg.kv_heads * cfg.head_dim * sizeof(KVT) * (s->h_pos[b] + 1);
                        fl += 4ull * cfg.heads * cfg.head_dim * (s->h_pos[b] + 1);
                    }
                    if ((rc = rec->begin("attn_flash_decode_paged", kvb, fl))) return rc;
                }
                const int G = cfg.heads / cfg.kv_heads;
                if (cfg.head_dim == 64) rc = attn_g<64>(s, c, a, G); else rc = attn_g<128>(s, c, a, G);
                if (rc) return rc;
                if (rec && (rc = rec->end())) return rc;
                ++launches;
            } else {
                g.y = s->raw;
                if ((rc = gemv<GEMV_RAW>(s, c, g, 16, rec, "deltanet_proj_gemv_norm"))) return rc;
                ++launches;
                const int dk = cfg.dn_key_dim, dv = cfg.dn_value_dim, H = cfg.heads;
                if (rec && (rc = rec->begin("deltanet_state_update", (uint64_t)B * 2ull * H * dk * dv * 4, (uint64_t)B * 6ull * H * dk * dv))) return rc;
                dim3 grid((dv + 31) / 32, H, B);
                if (s->parent) CU(delta_cols(s, i, s->abuf, nullptr));
                else if (dk == 64) CU(launch_chain(s->use_pdl, delta_net_kernel<64>, grid, dim3(256), 0, s->stream, c, static_cast<const float*>(s->raw), s->raw_stride, s->state[i], H, dv, s->abuf, static_cast<bf16_t*>(nullptr), 0, 1e-6f));
                else CU(launch_chain(s->use_pdl, delta_net_kernel<128>, grid, dim3(256), 0, s->stream, c, static_cast<const float*>(s->raw), s->raw_stride, s->state[i], H, dv, s->abuf, static_cast<bf16_t*>(nullptr), 0, 1e-6f));
                if (rec && (rc = rec->end())) return rc;
                ++launches;
            }
            // output projection + residual (in place on the residual stream)
            std::memset(&g, 0, sizeof g);
            g.W = L.Wo; g.wscale = L.So; g.N = d; g.K = L.o_in;
            g.xin = s->abuf; g.y = s->x; g.resid = s->x;
            if ((rc = gemv<GEMV_RESID>(s, c, g, d <= 1024 ? 8 : 16, rec, "oproj_gemv_residual"))) return rc;
            ++launches;
            // FFN gate/up with RMS norm prologue and SwiGLU epilogue
            std::memset(&g, 0, sizeof g);
            g.W = L.W1a; g.Wb = L.W1b; g.wscale = L.S1a; g.wscale_b = L.S1b; g.N = F; g.K = d;
            g.xin = s->x; g.gain = L.g2; g.eps = cfg.rms_eps; g.do_norm = 1; g.y = s->hbuf;
            if ((rc = gemv<GEMV_SWIGLU>(s, c, g, 8, rec, "ffn_gateup_gemv_norm_swiglu"))) return rc;
            ++launches;
            // FFN down + residual (+ the next layer's per-layer embedding)
            std::memset(&g, 0, sizeof g);
            g.W = L.W2; g.wscale = L.S2; g.N = d; g.K = F;
            g.xin = s->hbuf; g.y = s->x; g.resid = s->x;
            if (p > 0 && i + 1 < cfg.layers) { g.P = m->layers[i + 1].pleP; g.Ptab = m->layers[i + 1].pleT; g.Kp = p; }
            if ((rc = gemv<GEMV_RESID>(s, c, g, d <= 1024 ? 8 : 16, rec, "ffn_down_gemv_residual_ple"))) return rc;
            ++launches;
        }
        if (kind == CHAIN_PREFILL && s->parent) {
            // prompt columns: positions and tokens of the next chunk come from the host
        } else if (kind == CHAIN_PREFILL) {
            if (rec && (rc = rec->begin("advance_prompt", (uint64_t)B * 12, 0))) return rc;
            CU(launch_chain(s->use_pdl, advance_kernel, dim3((B + 127) / 128), dim3(128), 0, s->stream, c));
            if (rec && (rc = rec->end())) return rc;
            ++launches;
        } else {
            GemvParams g;
            std::memset(&g, 0, sizeof g);
            g.W = m->E; g.wscale = m->Es; g.N = cfg.vocab; g.K = d;
            g.xin = s->x; g.gain = m->g_final; g.eps = cfg.rms_eps; g.do_norm = 1; g.y = s->logits;
            g.part_val = s->part_val; g.part_idx = s->part_idx; g.ticket = s->lm_ticket;
            g.do_pick = kind == CHAIN_GREEDY ? 1 : 0;
            if ((rc = gemv<GEMV_LMHEAD>(s, c, g, s->lm_rows, rec, "lmhead_gemv_norm_argmax"))) return rc;
            ++launches;
            if (kind == CHAIN_TOPK) {
                SampleParams sp;
                sp.logits = s->logits; sp.V = cfg.vocab; sp.top_k = s->cur_topk; sp.temperature = s->cur_temp; sp.seeds = s->seeds;
                if (rec && (rc = rec->begin("sample_topk_philox", (uint64_t)B * cfg.vocab * 4 * 5, 0))) return rc;
                CU(launch_chain(s->use_pdl, sample_topk_kernel, dim3(B), dim3(kPickThreads), 0, s->stream, c, sp));
                if (rec && (rc = rec->end())) return rc;
                ++launches;
            }
        }
        if (n_launches) *n_launches = launches;
        return MLB_OK;
    }
};

template <int MODE, typename KVT, typename WT>
static int dec_allow_big_smem() {
    const int big = 200 * 1024;
    using KVQ = typename std::conditional<MODE == TC_QKV, KVT, float>::type;
    CU(cudaFuncSetAttribute(gemm_dec_kernel<MODE, KVQ, WT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    CU(cudaFuncSetAttribute(gemm_dec_kernel<MODE, KVQ, WT, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    CU(cudaFuncSetAttribute(gemm_dec_kernel<MODE, KVQ, WT, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    return MLB_OK;
}
template <typename KVT, typename WT>
static int tc_allow_big_smem_t() {
    const int big = 227 * 1024;
    CU(cudaFuncSetAttribute(gemm_tc_kernel<TC_RAW, KVT, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    CU(cudaFuncSetAttribute(gemm_tc_kernel<TC_RESID, KVT, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    CU(cudaFuncSetAttribute(gemm_tc_kernel<TC_SWIGLU, KVT, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    CU(cudaFuncSetAttribute(gemm_tc_kernel<TC_QKV, KVT, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    int rc;
    if ((rc = dec_allow_big_smem<TC_RAW, KVT, WT>()) || (rc = dec_allow_big_smem<TC_RESID, KVT, WT>()) || (rc = dec_allow_big_smem<TC_SWIGLU, KVT, WT>()) ||
        (rc = dec_allow_big_smem<TC_QKV, KVT, WT>()))
        return rc;
    return MLB_OK;
}

}  // namespace mlb
