// Host side of the decode path: model upload, session state (paged KV cache, delta-net
// state, step scratch), the launch chain of one decode step, CUDA-graph replay, and the C ABI
// declared in include/mlb.h.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>

#include "session.h"
#include "cols_host.h"
#include "gemm_cols.cuh"
#include "grid_host.h"
#include "lean_host.h"
#include "model_file.h"

namespace mlb {

// --------------------------------------------------------------------------------------
// errors
// --------------------------------------------------------------------------------------
static thread_local std::string g_err;

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    // The runtime keeps a failed call's code for this thread's next cudaGetLastError, which a later, healthy launch would report as its own.
    if (code == MLB_E_CUDA || code == MLB_E_NOMEM) cudaGetLastError();
    return code;
}

// --------------------------------------------------------------------------------------
// KV page allocator (host only)
// --------------------------------------------------------------------------------------
static int kv_ensure(mlb_kv_alloc* a, int seq, int n_positions, int block) {
    if (!a || seq < 0 || seq >= (int)a->seq_pages.size() || block <= 0 || n_positions < 0)
        return fail(MLB_E_INVALID, "kv allocator: bad argument");
    int need = (n_positions + block - 1) / block;
    if (need > a->max_pages_per_seq)
        return fail(MLB_E_CONTEXT_FULL, "sequence %d needs %d pages, the page table holds %d", seq, need, a->max_pages_per_seq);
    auto& pages = a->seq_pages[seq];
    while ((int)pages.size() < need) {
        if (a->free_list.empty())
            return fail(MLB_E_KV_FULL, "KV page pool exhausted (%d pages) while growing sequence %d", a->num_pages, seq);
        pages.push_back(a->free_list.back());
        a->free_list.pop_back();
    }
    return MLB_OK;
}

// --------------------------------------------------------------------------------------
// model
// --------------------------------------------------------------------------------------
struct Uploader {
    mlb_model* m;
    const std::vector<unsigned char>* file;
    std::vector<float> hbuf;
    float* dstage = nullptr;
    size_t dstage_elems = 0;

    int dev_alloc(void** p, size_t bytes) {
        cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
        if (e != cudaSuccess) return fail(MLB_E_NOMEM, "cudaMalloc of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
        m->allocs.push_back(*p);
        return MLB_OK;
    }
    // file tensor -> float32 on the device staging buffer
    int stage(const TensorDesc& t) {
        size_t n = (size_t)t.rows * t.cols;
        const unsigned char* src = file->data() + t.offset;
        const float* hsrc;
        if (t.dtype == FD_F32) {
            hsrc = reinterpret_cast<const float*>(src);
        } else {
            hbuf.resize(n);
            convert_to_f32(src, t.dtype, n, hbuf.data(), (uint64_t)t.cols);
            hsrc = hbuf.data();
        }
        CU(cudaMemcpy(dstage, hsrc, n * 4, cudaMemcpyHostToDevice));
        return MLB_OK;
    }
    // staged float32 [rows][cols] -> typed matrix rows [row_off, row_off+rows) of dst
    int emit(const TensorDesc& t, int dt, void* dst, size_t row_off, float* scale) {
        size_t n = (size_t)t.rows * t.cols;
        size_t off = row_off * (size_t)t.cols;
        if (dt == MLB_DT_F32) {
            CU(cudaMemcpy(static_cast<float*>(dst) + off, dstage, n * 4, cudaMemcpyDeviceToDevice));
        } else if (dt == MLB_DT_BF16) {
            cvt_f32_to_bf16_kernel<<<1024, 256>>>(dstage, static_cast<bf16_t*>(dst) + off, n);
            CU(cudaGetLastError());
        } else {
            int warps = 8;
            quant_fp8_rows_kernel<<<(t.rows + warps - 1) / warps, warps * 32>>>(dstage, static_cast<fp8_t*>(dst) + off,
                                                                              scale + row_off, t.rows, t.cols);
            CU(cudaGetLastError());
        }
        CU(cudaDeviceSynchronize());
        return MLB_OK;
    }
    int vec(const TensorDesc* t, float** out) {
        int rc = dev_alloc(reinterpret_cast<void**>(out), (size_t)t->rows * 4);
        if (rc) return rc;
        if ((rc = stage(*t))) return rc;
        CU(cudaMemcpy(*out, dstage, (size_t)t->rows * 4, cudaMemcpyDeviceToDevice));
        m->weight_bytes += (uint64_t)t->rows * 4;
        return MLB_OK;
    }
    // a matrix made of several file tensors stacked by rows
    int stacked(const std::vector<const TensorDesc*>& parts, int dt, void** W, float** S, int* total_rows) {
        int rows = 0, cols = parts[0]->cols;
        for (auto* t : parts) rows += t->rows;
        int rc = dev_alloc(W, (size_t)rows * cols * elt_size(dt));
        if (rc) return rc;
        *S = nullptr;
        if (dt == MLB_DT_FP8_E4M3 && (rc = dev_alloc(reinterpret_cast<void**>(S), (size_t)rows * 4))) return rc;
        size_t off = 0;
        for (auto* t : parts) {
            if (t->dtype == FD_FP8 && dt == MLB_DT_FP8_E4M3) {
                // quantised offline: the file's codes and per-row scales are the device's
                const unsigned char* src = file->data() + t->offset;
                const size_t n = (size_t)t->rows * t->cols;
                CU(cudaMemcpy(static_cast<fp8_t*>(*W) + off * (size_t)cols, src, n, cudaMemcpyHostToDevice));
                CU(cudaMemcpy(*S + off, src + n, (size_t)t->rows * 4, cudaMemcpyHostToDevice));
            } else {
                if ((rc = stage(*t))) return rc;
                if ((rc = emit(*t, dt, *W, off, *S))) return rc;
            }
            off += t->rows;
        }
        if (total_rows) *total_rows = rows;
        m->weight_bytes += (uint64_t)rows * cols * elt_size(dt) + (dt == MLB_DT_FP8_E4M3 ? (uint64_t)rows * 4 : 0);
        return MLB_OK;
    }
};

static int validate_for_kernels(const mlb_config& c) {
    const int gran = c.weight_dtype == MLB_DT_FP8_E4M3 ? 16 : (c.weight_dtype == MLB_DT_BF16 ? 8 : 4);
    if (c.dim % gran || c.ffn_dim % gran) return fail(MLB_E_UNSUPPORTED, "dim and ffn_dim must be multiples of %d for this weight type", gran);
    if (c.ple_dim % 8) return fail(MLB_E_UNSUPPORTED, "ple_dim must be a multiple of 8");
    bool has_attn = false, has_dn = false;
    for (int i = 0; i < c.layers; ++i) (c.layer_types[i] == MLB_LAYER_ATTENTION ? has_attn : has_dn) = true;
    if (has_attn) {
        if (c.head_dim != 64 && c.head_dim != 128) return fail(MLB_E_UNSUPPORTED, "attention head_dim must be 64 or 128 (got %d)", c.head_dim);
        int g = c.heads / c.kv_heads;
        if (g != 1 && g != 2 && g != 4 && g != 8) return fail(MLB_E_UNSUPPORTED, "heads/kv_heads must be 1, 2, 4 or 8 (got %d)", g);
        if ((c.heads * c.head_dim) % gran) return fail(MLB_E_UNSUPPORTED, "heads*head_dim must be a multiple of %d", gran);
    }
    if (has_dn) {
        if (c.dn_key_dim != 64 && c.dn_key_dim != 128) return fail(MLB_E_UNSUPPORTED, "delta-net key dim must be 64 or 128 (got %d)", c.dn_key_dim);
        if ((c.heads * c.dn_value_dim) % gran) return fail(MLB_E_UNSUPPORTED, "heads*dn_value_dim must be a multiple of %d", gran);
    }
    if (c.vocab < 2) return fail(MLB_E_INVALID, "vocabulary too small");
    return MLB_OK;
}

static void free_model(mlb_model* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    for (void* p : m->allocs) cudaFree(p);
    delete m;
}


}  // namespace mlb

using namespace mlb;

extern "C" void mlb_rope_table(float* table, int max_len, int head_dim, float base) {
    // Same host arithmetic as getPreComputedRopeTheta (inference.cu:364-374): float powf,
    // integer position times the float frequency, cosf / sinf.
    const int pairs = head_dim / 2;
    for (int pos = 0; pos < max_len; ++pos) {
        for (int i = 0; i < pairs; ++i) {
            float theta = pos * powf(base, (-2.0f * i / head_dim));
            table[(size_t)pos * head_dim + 2 * i] = cosf(theta);
            table[(size_t)pos * head_dim + 2 * i + 1] = sinf(theta);
        }
    }
}

extern "C" int mlb_file_inspect(const char* path, const mlb_config* ov, mlb_config* out, uint64_t* n_params) {
    if (!path || !out) return fail(MLB_E_INVALID, "null argument");
    std::vector<unsigned char> buf;
    std::string err;
    int rc = read_file(path, &buf, &err);
    if (rc) return fail(rc, "%s", err.c_str());
    ParsedModel pm;
    rc = parse_model_header(buf.data(), buf.size(), buf.size(), ov, &pm, &err);
    if (rc) return fail(rc, "%s", err.c_str());
    *out = pm.cfg;
    if (n_params) *n_params = pm.n_params;
    return MLB_OK;
}

extern "C" int mlb_model_load(const char* path, int device, const mlb_config* ov, mlb_model** out) {
    if (!path || !out) return fail(MLB_E_INVALID, "null argument");
    *out = nullptr;
    std::vector<unsigned char> buf;
    std::string err;
    int rc = read_file(path, &buf, &err);
    if (rc) return fail(rc, "%s", err.c_str());
    ParsedModel pm;
    rc = parse_model_header(buf.data(), buf.size(), buf.size(), ov, &pm, &err);
    if (rc) return fail(rc, "%s", err.c_str());
    if ((rc = validate_for_kernels(pm.cfg))) return rc;
    int ndev = 0;
    cudaError_t ce = cudaGetDeviceCount(&ndev);
    if (ce != cudaSuccess || ndev == 0)
        return fail(MLB_E_CUDA, "no CUDA device available (%s); this library has no CPU path", cudaGetErrorString(ce));
    if (device < 0 || device >= ndev) return fail(MLB_E_INVALID, "device %d out of range (0..%d)", device, ndev - 1);
    CU(cudaSetDevice(device));

    mlb_model* m = new mlb_model();
    m->cfg = pm.cfg;
    m->device = device;
    const mlb_config& c = m->cfg;
    const int wdt = c.weight_dtype, pdt = ple_dtype(wdt);
    Uploader up;
    up.m = m;
    up.file = &buf;
    size_t max_elems = 0;
    for (auto& t : pm.tensors) max_elems = std::max(max_elems, (size_t)t.rows * t.cols);
    up.dstage_elems = max_elems;
    if (cudaMalloc(reinterpret_cast<void**>(&up.dstage), max_elems * 4) != cudaSuccess) {
        free_model(m);
        return fail(MLB_E_NOMEM, "cudaMalloc of the %zu-byte staging buffer failed", max_elems * 4);
    }
#define UP(expr) do { int r__ = (expr); if (r__) { cudaFree(up.dstage); free_model(m); return r__; } } while (0)
    UP(up.stacked({pm.find(-1, "tokenEmbeddings")}, wdt, &m->E, &m->Es, nullptr));
    UP(up.vec(pm.find(-1, "finalRMSNormGamma"), &m->g_final));
    m->layers.resize(c.layers);
    for (int i = 0; i < c.layers; ++i) {
        const int blk = c.layers - 1 - i;               // block N-1 runs first (inference.cu:384-385)
        DevLayer& L = m->layers[i];
        L.type = c.layer_types[i];
        UP(up.vec(pm.find(blk, "rmsGamma"), &L.g1));
        UP(up.vec(pm.find(blk, "rmsGamma2"), &L.g2));
        std::vector<const TensorDesc*> parts = {pm.find(blk, "queryWeights"), pm.find(blk, "keyWeights"), pm.find(blk, "valueWeights")};
        L.nq = parts[0]->rows; L.nk = parts[1]->rows; L.nv = parts[2]->rows; L.ng = 0;
        if (L.type == MLB_LAYER_ATTENTION) {
            if (c.query_gating) { parts.push_back(pm.find(blk, "gatedQueryWeights")); L.ng = parts.back()->rows; }
            if (c.qk_norm) {
                UP(up.vec(pm.find(blk, "queryRMSGamma"), &L.gq));
                UP(up.vec(pm.find(blk, "keyRMSGamma"), &L.gk));
            }
        } else {
            parts.push_back(pm.find(blk, "betaWeights"));
            parts.push_back(pm.find(blk, "decayWeights"));
        }
        UP(up.stacked(parts, wdt, &L.Wqkv, &L.Sqkv, &L.n_qkv));
        const TensorDesc* wo = pm.find(blk, "outputProjectionWeights");
        L.o_in = wo->cols;
        UP(up.stacked({wo}, wdt, &L.Wo, &L.So, nullptr));
        UP(up.stacked({pm.find(blk, "feedForwardWeights1A")}, wdt, &L.W1a, &L.S1a, nullptr));
        UP(up.stacked({pm.find(blk, "feedForwardWeights1B")}, wdt, &L.W1b, &L.S1b, nullptr));
        UP(up.stacked({pm.find(blk, "feedForwardWeights2")}, wdt, &L.W2, &L.S2, nullptr));
        if (c.ple_dim > 0) {
            float* unused = nullptr;
            UP(up.stacked({pm.find(blk, "pleTable")}, pdt, &L.pleT, &unused, nullptr));
            UP(up.stacked({pm.find(blk, "pleProjection")}, pdt, &L.pleP, &unused, nullptr));
            // only one table row per sequence is read per step, not the whole table
            m->weight_bytes -= (uint64_t)c.vocab * c.ple_dim * elt_size(pdt);
        }
    }
    {
        std::vector<float> tab((size_t)c.max_context * c.head_dim);
        mlb_rope_table(tab.data(), c.max_context, c.head_dim, c.rope_theta);
        UP(up.dev_alloc(reinterpret_cast<void**>(&m->rope), tab.size() * 4));
        cudaError_t e = cudaMemcpy(m->rope, tab.data(), tab.size() * 4, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) { cudaFree(up.dstage); free_model(m); return fail(MLB_E_CUDA, "rope table upload: %s", cudaGetErrorString(e)); }
    }
#undef UP
    cudaFree(up.dstage);
    *out = m;
    return MLB_OK;
}

extern "C" int mlb_model_get_config(const mlb_model* m, mlb_config* out) {
    if (!m || !out) return fail(MLB_E_INVALID, "null argument");
    *out = m->cfg;
    return MLB_OK;
}
extern "C" uint64_t mlb_model_weight_bytes(const mlb_model* m) { return m ? m->weight_bytes : 0; }
extern "C" void mlb_model_free(mlb_model* m) { free_model(m); }

// --------------------------------------------------------------------------------------
// session
// --------------------------------------------------------------------------------------
namespace mlb {

// The most device memory that the column sets of a session may hold together, in bytes (MLB_COLUMNS_MB).
static size_t cols_limit() {
    const char* v = std::getenv("MLB_COLUMNS_MB");
    return v ? (size_t)std::max(0, std::atoi(v)) << 20 : SIZE_MAX;
}

static int sess_alloc(mlb_session* s, void** p, size_t bytes, bool zero) {
    if (s->parent && s->parent->cols_bytes + bytes > cols_limit())
        return fail(MLB_E_NOMEM, "%zu bytes more for prompt columns exceed MLB_COLUMNS_MB (%zu bytes held)", bytes, s->parent->cols_bytes);
    cudaError_t e = cudaMalloc(p, bytes ? bytes : 16);
    if (e != cudaSuccess) return fail(MLB_E_NOMEM, "cudaMalloc of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
    s->allocs.push_back(*p);
    if (s->parent) {
        s->own_bytes += bytes;
        s->parent->cols_bytes += bytes;
    }
    if (zero) CU(cudaMemset(*p, 0, bytes ? bytes : 16));
    return MLB_OK;
}

// Queue the read-back of the device error word; call before the stream synchronisation.
static int queue_err_readback(mlb_session* s) {
    CU(cudaMemcpyAsync(s->pinned_err, s->dev_err, 4, cudaMemcpyDeviceToHost, s->stream));
    return MLB_OK;
}
// What a code that a kernel left in the error word stands for.
static const char* wait_text(int code) {
    switch (code) {
        case 1: return "producer waiting for a free ring stage";
        case 2: return "consumer waiting for a weight chunk";
        case 6: return "attention waiting for K/V pages";
        case 11: return "tcgen05 GEMM, loader waiting for a free stage";
        case 12: return "tcgen05 GEMM, MMA issuer waiting for operands";
        case 13: return "tcgen05 GEMM, epilogue waiting for the accumulators";
        case 14: return "tcgen05 GEMM, widening warps waiting for codes";
        case 21: return "column GEMM, loader waiting for a free stage";
        case 22: return "column GEMM, MMA issuer waiting for a free accumulator";
        case 23: return "column GEMM, MMA issuer waiting for operands";
        case 24: return "column GEMM, epilogue waiting for an accumulator";
        case 31: return "decode GEMM, producer waiting for a free stage";
        case 32: return "decode GEMM, consumer waiting for operands";
        default: return "consumer waiting for another CTA's results";
    }
}
// After the synchronisation: a bounded device-side wait ran out somewhere in the step.
static int check_err_readback(mlb_session* s) {
    if (*s->pinned_err == 0) return MLB_OK;
    const int code = *s->pinned_err;
    *s->pinned_err = 0;
    cudaMemsetAsync(s->dev_err, 0, 4, s->stream);
    cudaStreamSynchronize(s->stream);
    return fail(MLB_E_TIMEOUT, "a bounded device-side wait ran out (code %d: %s); the results of this call are invalid", code, wait_text(code));
}

static void free_session(mlb_session* s) {
    if (!s) return;
    cudaSetDevice(s->m->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (auto* cs : s->cols) free_session(cs);
    free_session(s->cols_gemv);
    for (auto& e : s->plan_free) if (e) cudaEventDestroy(e);
    if (s->plan_host) cudaFreeHost(s->plan_host);
    for (auto& g : s->graphs) if (g) cudaGraphExecDestroy(g);
    for (auto& g : s->other_graphs) if (g) cudaGraphExecDestroy(g);
    for (auto& g : s->tgraphs) if (g) cudaGraphExecDestroy(g);
    for (void* p : s->allocs) cudaFree(p);
    if (s->parent) s->parent->cols_bytes -= s->own_bytes;
    if (s->pinned_tok) cudaFreeHost(s->pinned_tok);
    if (s->pinned_out) cudaFreeHost(s->pinned_out);
    if (s->pinned_err) cudaFreeHost(s->pinned_err);
    if (s->stream && !s->parent) cudaStreamDestroy(s->stream);      // a column set runs on its parent's stream
    delete s;
}

// After a decode call returned `n` ids of sequence b (ring order): advance the mirror, stop at the stop token,
// blank what lies behind it.
static void note_outputs(mlb_session* s, int b, int32_t* out, int n) {
    int room = seq_live(s, b) ? std::min(n, s->max_ctx - s->h_pos[b]) : 0;
    for (int i = 0; i < room; ++i) {
        if (s->stop_token >= 0 && out[i] == s->stop_token) {
            room = i + 1;
            s->h_stopped[b] = 1;
            break;
        }
    }
    for (int i = room; i < n; ++i) out[i] = -1;
    s->h_pos[b] += room;
}

// A chunk of prompt columns: embedding, then per layer projection, attention or recurrence, o-projection, gate/up and
// down projection, as persistent column GEMMs with the element-wise work in their epilogues; the LM head if the columns
// are scored.
static int run_cols(mlb_session* s, int kind, int* n_launches) {
    const mlb_model* m = s->m;
    const mlb_config& cfg = m->cfg;
    const int d = cfg.dim, F = cfg.ffn_dim, ple = cfg.ple_dim;
    const bool w8 = cfg.weight_dtype == MLB_DT_FP8_E4M3;
    const StepCtl c = make_ctl(s, kind);
    int launches = 0, rc;
    EmbedColsParams e;
    e.E = m->E; e.escale = m->Es; e.d = d; e.layers = s->step_layers; e.n_layers = cfg.layers; e.ple = ple; e.gain = m->layers[0].g1;
    const int parts = (d + 127) / 128 * 4;
    e.x = s->x; e.xg16 = s->xn16; e.ssq = s->tc_ssq; e.parts = parts; e.tple16 = s->tple16; e.T = s->B;
    CU(embed_cols_launch(w8, false, s->stream, c, e));
    ++launches;
    const QkvPostParams q0{};
    auto gemm = [&](int mode, const ColsGemm& g, const CUtensorMap& X, const CUtensorMap& W, const CUtensorMap& W2, int N, int K, float* y, bf16_t* h16,
                    bool normed, const float* next_gain, const mlb_session::TcLayerMaps* ext, const QkvPostParams* q, const float* s1, const float* s2) -> int {
        GemmColsParams p;
        p.N = N; p.K = K; p.BN = g.bn; p.stages = g.stages; p.nkb_x = ext ? (ple + kTcKB - 1) / kTcKB : 0;
        p.split = g.split; p.mains = g.mains; p.exts = g.exts; p.nbuf = g.nbuf; p.tmem_cols = g.tmem_cols;
        p.y = y; p.h16 = h16; p.ssq_in = normed ? s->tc_ssq : nullptr; p.ssq_parts = parts; p.eps = cfg.rms_eps;
        p.xg16 = s->xn16; p.gain_next = next_gain; p.ssq_out = s->tc_ssq;
        p.s1 = s1; p.s2 = s2; p.err = s->dev_err;
        CU(gemm_cols_launch(mode, cfg.kv_dtype, g.sums, g.pair, s->use_pdl, g.ctas, s->stream, X, W, W2, ext ? ext->pleT : X, ext ? ext->pleP : W, p, c, q ? *q : q0));
        ++launches;
        return MLB_OK;
    };
    for (int i = 0; i < cfg.layers; ++i) {
        const DevLayer& L = m->layers[i];
        const mlb_session::TcLayerMaps& M = s->tc_maps[i];
        const bool attn = L.type == MLB_LAYER_ATTENTION;
        if (attn) {
            QkvPostParams q;
            q.nq = L.nq; q.nk = L.nk; q.nv = L.nv; q.ng = L.ng; q.hd = cfg.head_dim;
            q.kv_heads = cfg.kv_heads; q.qk_norm = cfg.qk_norm; q.eps = cfg.rms_eps; q.gq = L.gq; q.gk = L.gk; q.rope = m->rope;
            q.kpool = s->kpool[i]; q.vpool = s->vpool[i]; q.page_table = s->page_table; q.pt_stride = s->max_pages;
            q.qbuf = s->qbuf; q.gbuf = s->gbuf;
            if ((rc = gemm(TC_QKV, s->cg_qkv, s->tc_g.xn[0], M.qkv, M.qkv, L.n_qkv, d, nullptr, nullptr, true, nullptr, nullptr, &q, L.Sqkv, nullptr))) return rc;
            if (cfg.kv_dtype == MLB_DT_BF16) {
                AttnColsParams ac;
                ac.kpool = static_cast<const bf16_t*>(s->kpool[i]); ac.vpool = static_cast<const bf16_t*>(s->vpool[i]);
                ac.page_table = s->page_table; ac.pt_stride = s->max_pages;
                ac.qbuf = s->qbuf; ac.gbuf = L.ng ? s->gbuf : nullptr; ac.out16 = s->a16;
                ac.heads = cfg.heads; ac.kv_heads = cfg.kv_heads;
                ac.hdr = s->plan.hdr; ac.tiles = reinterpret_cast<const int4*>(s->plan.tiles);
                CU(attn_cols_launch(cfg.head_dim, cfg.heads / cfg.kv_heads, s->use_pdl, s->plan.max_tiles, s->stream, ac));
            } else {
                // fp32 K/V: the decode kernel, one column at a time
                AttnParams a;
                a.kpool = s->kpool[i]; a.vpool = s->vpool[i]; a.page_table = s->page_table; a.pt_stride = s->max_pages;
                a.qbuf = s->qbuf; a.gbuf = L.ng ? s->gbuf : nullptr; a.abuf = s->abuf; a.abuf16 = s->a16; a.perm = 0; a.part = s->part; a.ticket = s->attn_ticket;
                a.heads = cfg.heads; a.kv_heads = cfg.kv_heads; a.num_pages = 0; a.err = s->dev_err; a.min_pages_per_split = s->attn_min_pps; a.early = 0;
                rc = chain_attn_f32kv(s, c, a);
                if (rc) return rc;
            }
        } else {
            if ((rc = gemm(TC_RAW, s->cg_dn, s->tc_g.xn[0], M.qkv, M.qkv, L.n_qkv, d, s->raw, nullptr, true, nullptr, nullptr, nullptr, L.Sqkv, nullptr))) return rc;
            CU(delta_cols(s, i, nullptr, s->a16));
        }
        ++launches;
        if ((rc = gemm(TC_RESID, attn ? s->cg_o_attn : s->cg_o_dn, attn ? s->tc_g.a_attn[0] : s->tc_g.a_dn[0], M.o, M.o, d, L.o_in, s->x, nullptr, false, L.g2, nullptr, nullptr, L.So, nullptr)))
            return rc;
        if ((rc = gemm(TC_SWIGLU, s->cg_up, s->tc_g.xn[0], M.w1a, M.w1b, F, d, nullptr, s->h16, true, nullptr, nullptr, nullptr, L.S1a, L.S1b))) return rc;
        const bool last = i + 1 == cfg.layers;
        const bool ext = !last && ple > 0;
        if ((rc = gemm(TC_RESID, ext ? s->cg_down : s->cg_last, s->tc_g.h[0], M.w2, M.w2, d, F, s->x, nullptr, false, last ? m->g_final : m->layers[i + 1].g1,
                       ext ? &s->tc_maps[i + 1] : nullptr, nullptr, L.S2, nullptr)))
            return rc;
    }
    if (kind != CHAIN_PREFILL && (rc = gemm(TC_RAW, s->cg_head, s->tc_g.xn[0], s->tc_g.E, s->tc_g.E, cfg.vocab, d, s->logits, nullptr, true, nullptr, nullptr, nullptr,
                                            static_cast<const float*>(m->Es), nullptr)))
        return rc;
    if (n_launches) *n_launches = launches;
    return MLB_OK;
}

static int chain_run(mlb_session* s, int kind, Recorder* rec, int* n_launches) {
    if (s->use_cols) return run_cols(s, kind, n_launches);
    switch (s->m->cfg.weight_dtype) {
        case MLB_DT_F32: return chain_run_f32(s, kind, rec, n_launches);
        case MLB_DT_BF16: return chain_run_bf16(s, kind, rec, n_launches);
        default: return chain_run_fp8(s, kind, rec, n_launches);
    }
}
static int chain_configure(mlb_session* s) {
    switch (s->m->cfg.weight_dtype) {
        case MLB_DT_F32: return chain_configure_f32(s);
        case MLB_DT_BF16: return chain_configure_bf16(s);
        default: return chain_configure_fp8(s);
    }
}

// Device copy of the per-layer pointer table of the single-kernel steps.
static int build_step_layers(mlb_session* s) {
    if (s->step_layers) return MLB_OK;
    const mlb_config& c = s->m->cfg;
    std::vector<StepLayer> hl(c.layers);
    for (int i = 0; i < c.layers; ++i) {
        const DevLayer& L = s->m->layers[i];
        StepLayer& M = hl[i];
        std::memset(&M, 0, sizeof M);
        M.type = L.type; M.n_qkv = L.n_qkv; M.nq = L.nq; M.nk = L.nk; M.nv = L.nv; M.ng = L.ng; M.o_in = L.o_in;
        M.Wqkv = L.Wqkv; M.Sqkv = L.Sqkv; M.g1 = L.g1; M.g2 = L.g2; M.gq = L.gq; M.gk = L.gk;
        M.Wo = L.Wo; M.So = L.So; M.W1a = L.W1a; M.W1b = L.W1b; M.W2 = L.W2; M.S1a = L.S1a; M.S1b = L.S1b; M.S2 = L.S2;
        M.pleT = L.pleT; M.pleP = L.pleP; M.kpool = s->kpool[i]; M.vpool = s->vpool[i]; M.state = s->state[i];
    }
    int rc = sess_alloc(s, (void**)&s->step_layers, hl.size() * sizeof(StepLayer), false);
    if (rc) return rc;
    CU(cudaMemcpy(s->step_layers, hl.data(), hl.size() * sizeof(StepLayer), cudaMemcpyHostToDevice));
    return MLB_OK;
}

// The whole-GPU step with compile-time shapes (lean.cuh), for batch-1 sessions of the models it is built
// for. MLB_DECODE_PATH = auto (this kernel where it fits, else the generic one) | lean | grid | chain.
static int setup_lean_path(mlb_session* s) {
    const mlb_config& c = s->m->cfg;
    const char* env = std::getenv("MLB_DECODE_PATH");
    const std::string mode = env ? env : "auto";
    s->use_lean = false;
    if (mode != "lean" && mode != "auto") return MLB_OK;
    auto no = [&](const char* why) {
        if (mode == "lean") return fail(MLB_E_UNSUPPORTED, "MLB_DECODE_PATH=lean: %s", why);
        return (int)MLB_OK;
    };
    if (s->B != 1) return no("the whole-GPU step serves batch 1 only");
    const int idx = lean_find_shape(c);
    if (idx < 0) return no("no specialised kernel is built for this model's shape");
    const LeanShapeInfo& si = lean_shape_info(idx);
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->m->device);
    if (!coop || s->sm_count < si.C) return no("the device cannot keep the kernel's CTAs resident");
    for (const DevLayer& L : s->m->layers)
        if (L.o_in != si.H * si.HD) return no("a layer's output projection has another input width");
    auto up4 = [](int v) { return (v + 3) / 4 * 4; };
    LeanParams lp;
    std::memset(&lp, 0, sizeof lp);
    int off = 0;
    lp.xs_stride = up4(si.xs_floats);
    lp.off_xs = off; off += 2 * lp.xs_stride;
    lp.off_xa = off; off += up4(si.D);
    lp.off_xb = off; off += up4(si.D);
    lp.off_parts = off; off += up4(si.parts_floats);
    lp.off_mix = off; off += up4(si.mix_floats);
    lp.off_pacc = off; off += up4(std::max(1, c.layers * si.rx));
    lp.off_red = off; off += 2 * kLeanWarps + 4 + 128;      // + the dead flag, the finished-row counter, the finished rows
    off = (off + 1) / 2 * 2;
    lp.off_layers = off; off += up4((int)(c.layers * sizeof(StepLayer) / 4));
    lp.off_timers = off; off += 2 * kGridTimerSlots;
    lp.off_plan = off; off += 12;
    off = (off + 31) / 32 * 32;
    const int max_stages = 12;
    lp.off_bar = off; off += max_stages * 2 * 2;
    off = (off + 31) / 32 * 32;
    lp.off_ring = off;
    const size_t fixed = (size_t)off * 4;
    if (fixed + 4 * (size_t)kLeanStage > 208 * 1024) return no("too little shared memory is left for the weight ring");
    lp.n_stages = (int)std::min<size_t>(max_stages, (208 * 1024 - fixed) / kLeanStage);
    const size_t smem = fixed + (size_t)lp.n_stages * kLeanStage;
    int per_sm = 0, rc;
    if ((rc = lean_kernel_probe(idx, c.kv_dtype, smem, &per_sm))) return rc;
    if (per_sm < 1) return no("the kernel does not fit an SM");
    if ((rc = build_step_layers(s))) return rc;
    // exchange buffers (zeroed: epoch 0 is never produced)
    const size_t C = (size_t)si.C;
    const size_t n_ll = C * (2 * (size_t)si.slot_x + si.slot_qa + si.slot_qd + si.slot_parts + si.slot_a + si.slot_ah + si.slot_h + 16) + 64;
    unsigned long long* ll = nullptr;
    if ((rc = sess_alloc(s, (void**)&ll, n_ll * 8, true))) return rc;
    lp.x = ll; ll += C * si.slot_x;
    lp.xb = ll; ll += C * si.slot_x;
    lp.pj = ll; ll += C * std::max(si.slot_qa, si.slot_qd);
    ll += C * std::min(si.slot_qa, si.slot_qd);
    lp.parts = ll; ll += C * si.slot_parts;
    lp.a = ll; ll += C * si.slot_a;
    lp.ah = ll; ll += C * si.slot_ah;
    lp.h = ll; ll += C * si.slot_h;
    lp.lm = ll; ll += C * 16;
    if ((rc = sess_alloc(s, (void**)&lp.epoch, 16, true))) return rc;
    if (const char* t = std::getenv("MLB_GRID_TIMERS"))
        if (t[0] == '1' && (rc = sess_alloc(s, (void**)&lp.timers, C * kGridTimerSlots * 8, true))) return rc;
    if (lp.timers && (rc = sess_alloc(s, (void**)&lp.trace, C * kLeanTraceLen * 8, true))) return rc;
    lp.layers = s->step_layers; lp.n_layers = c.layers;
    lp.E = s->m->E; lp.g_final = s->m->g_final; lp.rope = s->m->rope; lp.page_table = s->page_table;
    lp.logits = s->logits; lp.err = s->dev_err;
    lp.tok_arg = -1;
    lp.eps = c.rms_eps; lp.l2_eps = 1e-6f;
    lp.pages_per_split = 4;       // 64 positions per attention item: one round of the 16 warps (measured: 4 beats 16 by 4 us per step at a context of 150)
    if (const char* v = std::getenv("MLB_GRID_PAGES_PER_SPLIT")) lp.pages_per_split = std::max(1, std::min(256, std::atoi(v)));
    s->lean = lp;
    s->lean_idx = idx;
    s->lean_smem = smem;
    s->grid_ctas = si.C;
    s->use_lean = true;
    return MLB_OK;
}

// Geometry of one exchanged vector of the whole-GPU step: N values from P producers, a slot of whole
// 128-byte lines per producer (grid_params.h). `tab` is the shared-memory offset of its row table, -1
// when every producer owns exactly N / P rows.
static GridVec grid_vec(int N, int P, int tab) {
    GridVec v;
    std::memset(&v, 0, sizeof v);
    v.N = N;
    v.P = P;
    v.rpc = (N + P - 1) / P;
    v.slotw = (v.rpc + 15) / 16 * 16;
    v.tab = tab;
    v.inv_n = 1.0f / (float)N;
    v.wpp = (v.rpc + 2) / 3;
    // q / d as one multiply-high, exact over the range the kernel uses (q < P * d < 2^16 * d)
    auto magic = [&](int d) {
        if (d == 1) return 0u;
        const unsigned m = (unsigned)(((1ull << 32) + (unsigned)d - 1) / (unsigned)d);
        for (unsigned q = 0; q < (unsigned)(P * d); ++q)
            if ((unsigned)(((unsigned long long)q * m) >> 32) != q / (unsigned)d) { v.N = -1; break; }     // never seen; the caller refuses
        return m;
    };
    v.magic = magic(v.rpc);
    v.magic3 = magic(v.wpp);
    return v;
}

// Decides whether the whole-GPU single-kernel step serves this session (batch 1) and lays out
// its shared memory and exchange buffers. MLB_DECODE_PATH = chain | grid | auto; auto takes it
// whenever the model fits its constraints.
static int setup_grid_path(mlb_session* s) {
    const mlb_config& c = s->m->cfg;
    const char* env = std::getenv("MLB_DECODE_PATH");
    const std::string mode = env ? env : "auto";
    s->use_grid = false;
    if (mode != "grid" && mode != "auto") return MLB_OK;
    auto no = [&](const char* why) {
        if (mode == "grid") return fail(MLB_E_UNSUPPORTED, "MLB_DECODE_PATH=grid: %s", why);
        return (int)MLB_OK;
    };
    if (s->B != 1) return no("the whole-GPU step serves batch 1 only");
    int coop = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, s->m->device);
    if (!coop) return no("the device has no cooperative launch");
    const int epv = 16 / (int)elt_size(c.weight_dtype);
    bool has_attn = false, has_dn = false;
    int nqkv_attn = 0, nqkv_dn = 0, min_rows = std::min(c.dim, c.ffn_dim), a_dim = 16;
    for (const DevLayer& L : s->m->layers) {
        min_rows = std::min(min_rows, L.n_qkv);
        a_dim = std::max(a_dim, L.o_in);
        if (L.type == MLB_LAYER_ATTENTION) { has_attn = true; nqkv_attn = L.n_qkv; }
        else { has_dn = true; nqkv_dn = L.n_qkv; }
        if (L.o_in % epv) return no("a projection width is not a multiple of the weight vector");
    }
    if (c.dim % epv || c.ffn_dim % epv) return no("a projection width is not a multiple of the weight vector");
    if (has_attn && c.head_dim != 64 && c.head_dim != 128) return no("head_dim must be 64 or 128");
    if (has_attn && (c.heads % c.kv_heads || c.heads / c.kv_heads > 8)) return no("more than 8 query heads per kv head");
    if (has_dn && c.dn_key_dim > 128) return no("delta-net key dim above 128");
    if (has_dn) min_rows = std::min(min_rows, c.heads * c.dn_value_dim);
    min_rows = std::min(min_rows, c.vocab);
    // Every CTA must own rows in every projection phase (the reuse rule of the exchange buffers)
    int C = std::min(s->sm_count, min_rows);
    if (const char* v = std::getenv("MLB_GRID_CTAS")) C = std::max(8, std::min(C, std::atoi(v)));
    if (C < 8) return no("the model is too small to split over the SMs");
    if (has_attn && c.heads > C) return no("more heads than CTAs");
    const int G = has_attn ? c.heads / c.kv_heads : 1;
    auto up4 = [](int v) { return (v + 3) / 4 * 4; };
    GridParams gp;
    std::memset(&gp, 0, sizeof gp);
    // context splits per kv head: at most one item per CTA; a head's partials fit 32 KB of shared memory
    gp.s_max = has_attn ? std::max(1, std::min(C / c.kv_heads, 8192 / (c.head_dim + 2))) : 1;
    gp.s_direct = has_attn ? std::max(1, std::min(gp.s_max, kGridDirectWords / (c.heads * (c.head_dim + 2)))) : 1;
    gp.pages_per_split = 4;        // 64 positions per attention item (measured: the large GQA model 1.07 -> 0.99 ms per token against 16, the reference-shaped fp32 model 207 -> 198 us)
    if (const char* v = std::getenv("MLB_GRID_PAGES_PER_SPLIT")) gp.pages_per_split = std::max(1, std::min(256, std::atoi(v)));
    const int rpc_d = (c.dim + C - 1) / C;
    const int rpc_a = has_dn ? (c.heads * c.dn_value_dim + C - 1) / C : 0;
    int off = 0;
    // row tables (ints) of the vectors whose rows do not divide evenly
    const int tab_d = off; off += up4(C + 1);
    const int tab_f = off; off += up4(C + 1);
    const int tab_qa = off; off += up4(C + 1);
    const int tab_qd = off; off += up4(C + 1);
    const int tab_a = off; off += up4(C + 1);
    const int tab_ah = off; off += up4(C + 1);
    const int tab_lm = off; off += up4(C + 1);
    gp.vocab_tab = off; off += up4(C + 1);
    gp.off_tabs = 0;
    // two input buffers in turn: phases whose input is the residual stream, and the others (output and down projection)
    gp.xs_stride = up4(c.dim);
    gp.off_xs = off; off += gp.xs_stride + up4(std::max(c.ffn_dim, a_dim));
    gp.off_xa = off; off += up4(rpc_d);
    gp.off_xb = off; off += up4(rpc_d);
    gp.off_parts = off; off += up4(std::max(has_attn ? std::max(gp.s_max * (c.head_dim + 2), kGridDirectWords) : 0, 2 * C));
    gp.off_gate = off; off += up4(has_attn && c.query_gating ? c.heads * c.head_dim : 4);
    {
        const int attn_n = has_attn ? G * c.head_dim + 2 * c.head_dim + kRingWarps * (c.head_dim + 2) : 0;
        const int comb_n = has_attn ? std::max(c.heads * gp.s_direct, gp.s_max) : 0;
        const int dn_n = has_dn ? 2 * c.heads * c.dn_key_dim + up4(rpc_a) + 2 * c.heads + 8 : 0;
        gp.off_mix = off; off += up4(std::max(std::max(attn_n, comb_n), std::max(dn_n, 64)));
    }
    gp.off_pacc = off; off += up4(std::max(1, c.layers * rpc_d));
    gp.off_red = off; off += 2 * kRingConsumers + 8;      // + the dead flag and the finished-row counter
    gp.off_obuf = off; off += up4(std::max(std::max((nqkv_attn + C - 1) / C, (nqkv_dn + C - 1) / C), std::max((c.ffn_dim + C - 1) / C, std::max(rpc_d, rpc_a))) + 4);
    off = (off + 1) / 2 * 2;
    gp.off_layers = off; off += up4((int)(c.layers * sizeof(StepLayer) / 4));
    gp.off_timers = off; off += 2 * kGridTimerSlots;
    gp.off_plan = off; off += 12;
    off = (off + 31) / 32 * 32;
    const int max_stages = 12;
    gp.off_bar = off; off += max_stages * 2 * 2;              // 8-byte barriers: full[] then empty[]
    off = (off + 31) / 32 * 32;
    gp.off_ring = off;
    // ring: stages of whole rows (and whole KV pages), 16 KB unless a row is longer, as many as fit below 226 KB
    size_t widest = (size_t)std::max(std::max(c.dim, c.ffn_dim), a_dim) * elt_size(c.weight_dtype);
    if (has_attn) widest = std::max(widest, (size_t)kKvBlock * c.head_dim * elt_size(c.kv_dtype));
    if (has_dn) widest = std::max(widest, (size_t)c.dn_key_dim * 4);
    gp.stage_bytes = (int)std::max<size_t>(16 * 1024, (widest + 1023) / 1024 * 1024);
    if (const char* v = std::getenv("MLB_GRID_STAGE_KB")) gp.stage_bytes = std::max(gp.stage_bytes, std::min(64, std::atoi(v)) * 1024);
    const size_t fixed = (size_t)off * 4;
    if (fixed + 3 * (size_t)gp.stage_bytes > 226 * 1024) return no("the activations leave too little shared memory for the weight ring");
    gp.n_stages = (int)std::min<size_t>(max_stages, (226 * 1024 - fixed) / gp.stage_bytes);
    const size_t smem = fixed + (size_t)gp.n_stages * gp.stage_bytes;
    int per_sm = 0, rc;
    if ((rc = grid_kernel_probe(c.weight_dtype, c.kv_dtype, smem, &per_sm))) return rc;
    if (per_sm < 1) return no("the kernel does not fit an SM");
    if ((rc = build_step_layers(s))) return rc;
    // exchanged vectors and their buffers (zeroed: epoch 0 is never produced)
    gp.vx = grid_vec(c.dim, C, tab_d);
    gp.vxb = grid_vec(c.dim, C, tab_d);
    gp.vproj_attn = grid_vec(std::max(nqkv_attn, C), C, tab_qa);
    gp.vproj_dn = grid_vec(std::max(nqkv_dn, C), C, tab_qd);
    gp.vh = grid_vec(c.ffn_dim, C, tab_f);
    gp.va_dn = grid_vec(has_dn ? c.heads * c.dn_value_dim : C, C, tab_a);
    gp.va_head = grid_vec(has_attn ? c.heads * c.head_dim : 16, has_attn ? c.heads : 1, tab_ah);
    gp.vlm = grid_vec(2 * C, C, tab_lm);
    gp.parts_slotw = (G * (c.head_dim + 2) + 15) / 16 * 16;
    GridVec* vecs[] = {&gp.vx, &gp.vxb, &gp.vproj_attn, &gp.vproj_dn, &gp.vh, &gp.va_dn, &gp.va_head, &gp.vlm};
    size_t n_ll = (size_t)C * gp.parts_slotw + 64;
    for (GridVec* v : vecs) {
        if (v->N < 0) return no("a row split has no exact multiply-high divisor");
        n_ll += (size_t)v->P * v->slotw;
    }
    unsigned long long* ll = nullptr;
    if ((rc = sess_alloc(s, (void**)&ll, n_ll * 8, true))) return rc;
    for (GridVec* v : vecs) { v->buf = ll; ll += (size_t)v->P * v->slotw; }
    gp.parts = ll;
    if ((rc = sess_alloc(s, (void**)&gp.epoch, 16, true))) return rc;
    if (const char* t = std::getenv("MLB_GRID_TIMERS"))
        if (t[0] == '1' && (rc = sess_alloc(s, (void**)&gp.timers, (size_t)C * kGridTimerSlots * 8, true))) return rc;
    gp.layers = s->step_layers; gp.n_layers = c.layers;
    gp.d = c.dim; gp.F = c.ffn_dim; gp.V = c.vocab; gp.heads = c.heads; gp.kv_heads = c.kv_heads; gp.hd = c.head_dim;
    gp.dk = c.dn_key_dim; gp.dv = c.dn_value_dim; gp.ple = c.ple_dim; gp.qk_norm = c.qk_norm;
    gp.eps = c.rms_eps; gp.l2_eps = 1e-6f;
    gp.E = s->m->E; gp.Es = s->m->Es; gp.g_final = s->m->g_final; gp.rope = s->m->rope;
    gp.page_table = s->page_table; gp.logits = s->logits;
    gp.err = s->dev_err;
    gp.tok_arg = -1;
    gp.backoff_ns = 100;
    if (const char* v = std::getenv("MLB_GRID_BACKOFF_NS")) gp.backoff_ns = std::max(0, std::min(10000, std::atoi(v)));
    s->grid = gp;
    s->grid_ctas = C;
    s->grid_smem = smem;
    s->use_grid = true;
    return MLB_OK;
}

// How far a cluster may split the k-blocks of a GEMM tile here.
static int tc_probe_clusters(mlb_session* s) {
    s->tc_max_split = 8;
    if (const char* v = std::getenv("MLB_TC_SPLIT")) {
        s->tc_max_split = std::max(1, std::min(8, std::atoi(v)));
        s->tc_split_forced = true;
    }
    {
        // how many clusters of GEMM CTAs fit on the GPU at once (a 100 KB CTA, typical of a split launch)
        s->tc_cluster_cap[0] = s->sm_count;
        for (int li = 1; li < 4; ++li) {
            int n = 0, rc;
            if ((rc = tc_max_clusters(1 << li, 100 * 1024, &n))) return rc;
            s->tc_cluster_cap[li] = n;
        }
    }
    return MLB_OK;
}

// MLB_GEMM=tcgen05: every tensor-core projection on gemm_tc.cuh, and prompt columns as steps of the decode kernels, whose results those of
// gemm_dec.cuh, gemm_cols.cuh and attn_cols_kernel have to equal bit for bit.
static bool gemm_tcgen05_only() {
    const char* v = std::getenv("MLB_GEMM");
    return v && std::string(v) == "tcgen05";
}

// Tensor-core projections for batches of 4 sequences or more with bf16 or FP8 weights (MLB_GEMM=simt turns them off).
static int setup_tc_path(mlb_session* s) {
    const mlb_config& c = s->m->cfg;
    s->use_tc = false;
    const char* env = std::getenv("MLB_GEMM");
    const std::string mode = env ? env : "auto";
    if (!s->parent && (mode == "simt" || s->use_grid || s->use_lean)) return MLB_OK;
    if (c.weight_dtype != MLB_DT_BF16 && c.weight_dtype != MLB_DT_FP8_E4M3) {
        if (mode != "auto") return fail(MLB_E_UNSUPPORTED, "MLB_GEMM=%s needs bf16 or FP8 weights", mode.c_str());
        return MLB_OK;
    }
    const bool w8 = c.weight_dtype == MLB_DT_FP8_E4M3;
    // auto: from 4 sequences on. The GEMV kernels re-read nothing, but their time grows with the batch
    // (cfg1: 169 us at 1 sequence, 369 at 4, 537 at 8, 635 at 12), while the tensor-core step costs
    // 360-390 us for any batch up to 16 (its floor is its 60 launches).
    if (!s->parent && mode == "auto" && s->B < 4) return MLB_OK;
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) {
        if (mode != "auto") return fail(MLB_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
        return MLB_OK;
    }
    const int B = s->B;
    s->tc_nb = std::min(256, (B + 15) / 16 * 16);
    const size_t budget = 200 * 1024;
    s->tc_stages = (int)std::max<size_t>(2, std::min<size_t>(6, budget / ((size_t)kTcM * 128 + (size_t)s->tc_nb * 128)));
    s->tc_stages_swiglu = (int)std::max<size_t>(2, std::min<size_t>(6, budget / ((size_t)2 * kTcM * 128 + (size_t)s->tc_nb * 128)));
    const int nq = c.heads * c.head_dim, a_dn = c.heads * c.dn_value_dim;
    int rc;
    if (c.ple_dim > 0 && ple_dtype(c.weight_dtype) != MLB_DT_BF16) return MLB_OK;
    if ((rc = build_step_layers(s))) return rc;
    if (const char* v = std::getenv("MLB_TC_TRACE"))
        if (v[0] == '1' && (rc = sess_alloc(s, (void**)&s->tc_trace, 64 * 8 * 8, true))) return rc;
    if ((rc = tc_probe_clusters(s))) return rc;
    const auto kb = [](int k) { return (k + kTcKB - 1) / kTcKB; };
    // mma.sync tiles for the projections, or tcgen05 ones: gd_small_enough. The QK norm needs whole heads in a tile, the k-block maps
    // whole k-blocks, the ranges of a tile a warp each: other models stay on gemm_tc.cuh (cfg1 with QK norm 361 / 380 / 532 us a step at
    // 4 / 37 / 256 sequences, 178 / 224 / 424 without).
    s->use_dec = !s->parent && mode != "tcgen05" && !c.qk_norm && (mode == "mma" ? B <= 256 : gd_small_enough(s)) && c.dim % kTcKB == 0 && c.ffn_dim % kTcKB == 0 && c.ple_dim % kTcKB == 0 &&
                 nq % kTcKB == 0 && a_dn % kTcKB == 0;
    const auto ranges_fit = [&](int n, int nkb, int mode, bool ext) { return gd_pick(s, n, nkb, mode, w8, ext).split <= kGdMaxSplit; };
    for (int i = 0; i < c.layers && s->use_dec; ++i)
        s->use_dec = ranges_fit(s->m->layers[i].n_qkv, kb(c.dim), TC_QKV, false) && ranges_fit(c.dim, kb(s->m->layers[i].o_in), TC_RESID, false);
    s->use_dec = s->use_dec && ranges_fit(c.ffn_dim, kb(c.dim), TC_SWIGLU, false) && ranges_fit(c.vocab, kb(c.dim), TC_RAW, false) &&
                 ranges_fit(c.dim, kb(c.ffn_dim) + kb(c.ple_dim), TC_RESID, c.ple_dim > 0) && ranges_fit(c.dim, kb(c.ffn_dim), TC_RESID, false);
    if (mode == "mma" && !s->use_dec && !s->parent) return fail(MLB_E_UNSUPPORTED, "MLB_GEMM=mma: a QK norm, a width or the batch rules its tiles out");
    s->tc_shape_down = tc_pick_shape(s, B, c.dim, (c.ffn_dim + kTcKB - 1) / kTcKB + (c.ple_dim + kTcKB - 1) / kTcKB, 1, w8, w8 ? 2 : 1);
    const int parts = (c.dim + kTcM - 1) / kTcM * 4;
    if ((rc = sess_alloc(s, (void**)&s->xn16, (size_t)B * c.dim * 2, true))) return rc;
    if ((rc = sess_alloc(s, (void**)&s->a16, (size_t)B * std::max(nq, a_dn) * 2, true))) return rc;
    if ((rc = sess_alloc(s, (void**)&s->h16, (size_t)B * c.ffn_dim * 2, true))) return rc;
    if ((rc = sess_alloc(s, (void**)&s->tc_ssq, (size_t)B * parts * 4, true))) return rc;
    if (c.ple_dim > 0 && (rc = sess_alloc(s, (void**)&s->tple16, (size_t)c.layers * B * c.ple_dim * 2, true))) return rc;
    s->tc_maps.resize(c.layers);
    // weight maps of a projection, by the launch shape it has
    auto wmap = [&](CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, int mode, int kb_ext) {
        if (s->use_dec) return make_kblock_map(enc, out, base, rows, cols, kGdF, gd_pick(s, (int)rows, kb((int)cols) + kb_ext, mode, w8, kb_ext > 0).g, w8);
        return w8 ? make_u8_map(enc, out, base, rows, cols, kTcM) : make_bf16_map(enc, out, base, rows, cols, kTcM);      // codes are widened in the kernel
    };
    for (int i = 0; i < c.layers; ++i) {
        const DevLayer& L = s->m->layers[i];
        auto& M = s->tc_maps[i];
        const int kb_ext = i + 1 < c.layers ? kb(c.ple_dim) : 0;      // k-blocks of the next layer's embedding behind the down projection
        if ((rc = wmap(&M.qkv, L.Wqkv, L.n_qkv, c.dim, L.type == MLB_LAYER_ATTENTION ? TC_QKV : TC_RAW, 0))) return rc;
        if ((rc = wmap(&M.o, L.Wo, c.dim, L.o_in, TC_RESID, 0))) return rc;
        if ((rc = wmap(&M.w1a, L.W1a, c.ffn_dim, c.dim, TC_SWIGLU, 0))) return rc;
        if ((rc = wmap(&M.w1b, L.W1b, c.ffn_dim, c.dim, TC_SWIGLU, 0))) return rc;
        if ((rc = wmap(&M.w2, L.W2, c.dim, c.ffn_dim, TC_RESID, kb_ext))) return rc;
        if (c.ple_dim > 0) {
            // operands of the per-layer embedding folded into the previous layer's down projection
            const bf16_t* rows = s->tple16 + (size_t)i * B * c.ple_dim;
            if (s->use_dec) {
                const GdShape g = gd_pick(s, c.dim, kb(c.ffn_dim) + kb(c.ple_dim), TC_RESID, w8, true);
                if ((rc = make_kblock_map(enc, &M.pleP, L.pleP, c.dim, c.ple_dim, kGdF, g.g, false))) return rc;
                if ((rc = make_kblock_map(enc, &M.pleT, rows, B, c.ple_dim, 16 * g.np, g.g, false))) return rc;
            } else {
                if ((rc = make_bf16_map(enc, &M.pleP, L.pleP, c.dim, c.ple_dim, kTcM))) return rc;
                if ((rc = make_bf16_map(enc, &M.pleT, rows, B, c.ple_dim, s->tc_shape_down.nb))) return rc;
            }
        }
    }
    if ((rc = wmap(&s->tc_g.E, s->m->E, c.vocab, c.dim, TC_RAW, 0))) return rc;
    for (int i = 0; i < (s->use_dec ? 9 : 5); ++i) {
        auto xmap = [&](CUtensorMap* out, const void* base, uint64_t cols) {
            if (s->use_dec) return make_kblock_map(enc, out, base, B, cols, 16u << (i / 3), 1u << (i % 3), false);
            return make_bf16_map(enc, out, base, B, cols, 16u << i);
        };
        if ((rc = xmap(&s->tc_g.xn[i], s->xn16, c.dim))) return rc;
        if ((rc = xmap(&s->tc_g.a_attn[i], s->a16, nq))) return rc;
        if ((rc = xmap(&s->tc_g.a_dn[i], s->a16, a_dn))) return rc;
        if ((rc = xmap(&s->tc_g.h[i], s->h16, c.ffn_dim))) return rc;
    }
    if ((rc = w8 ? tc_allow_big_smem_fp8(c.kv_dtype) : tc_allow_big_smem_bf16(c.kv_dtype))) return rc;
    s->use_tc = true;
    return MLB_OK;
}

// The FP8 codes of a model as bf16, made on first use; false where there is no memory for them (asked for again by the next caller) or
// MLB_FP8_COPY=0 refuses them.
static int model_widen(mlb_model* m, cudaStream_t st, bool* have) {
    std::lock_guard<std::mutex> hold(m->wide_mutex);
    const char* env = std::getenv("MLB_FP8_COPY");
    *have = false;
    if (env && env[0] == '0') return MLB_OK;
    *have = !m->wide.empty();
    if (*have) return MLB_OK;
    const mlb_config& c = m->cfg;
    size_t need = (size_t)c.vocab * c.dim * 2, free_bytes = 0, all = 0;
    for (const DevLayer& L : m->layers) need += ((size_t)L.n_qkv * c.dim + (size_t)c.dim * L.o_in + 3 * (size_t)c.ffn_dim * c.dim) * 2;
    CU(cudaMemGetInfo(&free_bytes, &all));
    if (free_bytes < need) return MLB_OK;
    std::vector<void*> made;
    int rc = MLB_OK;
    auto widen = [&](const void* codes, size_t n) -> void* {
        void* p = nullptr;
        if (rc) return p;
        if (cudaMalloc(&p, n * 2) != cudaSuccess) {
            cudaGetLastError();
            rc = MLB_E_NOMEM;
            return nullptr;
        }
        made.push_back(p);
        if (widen_e4m3_launch(codes, static_cast<bf16_t*>(p), n, st) != cudaSuccess) rc = MLB_E_CUDA;
        return p;
    };
    std::vector<mlb_model::Wide> w(c.layers);
    for (int i = 0; i < c.layers; ++i) {
        const DevLayer& L = m->layers[i];
        w[i].Wqkv = widen(L.Wqkv, (size_t)L.n_qkv * c.dim);
        w[i].Wo = widen(L.Wo, (size_t)c.dim * L.o_in);
        w[i].W1a = widen(L.W1a, (size_t)c.ffn_dim * c.dim);
        w[i].W1b = widen(L.W1b, (size_t)c.ffn_dim * c.dim);
        w[i].W2 = widen(L.W2, (size_t)c.dim * c.ffn_dim);
    }
    void* we = widen(m->E, (size_t)c.vocab * c.dim);
    const cudaError_t e = cudaStreamSynchronize(st);      // sessions on other streams read them from here on
    if (rc || e != cudaSuccess) {
        for (void* p : made) cudaFree(p);
        if (rc == MLB_E_NOMEM && e == cudaSuccess) return MLB_OK;
        return fail(MLB_E_CUDA, "widening of the FP8 weights failed: %s", cudaGetErrorString(e));
    }
    m->allocs.insert(m->allocs.end(), made.begin(), made.end());
    m->wide_E = we;
    m->wide.swap(w);
    *have = true;
    return MLB_OK;
}

// Launch shape of a column GEMM: `T` columns, `N` output features, `nkb` k-blocks of 64, the last `nkb_x` of a second
// operand pair (`exts_apart`: with accumulators of its own), in `split` ranges. Tensor memory (512 columns) bounds BN x
// accumulators x buffers. A 128 x BN x 64 k-block takes about 0.43 / 0.36 / 0.26 us at BN = 256 / 128 / 64 with every SM at it: the tensor
// pipe's rate at 256 (1.44 PFLOP/s), its operands below (32, 24 KB at about 90 GB/s an SM). A pair of CTAs has one of 256 x 256 in 0.42. An epilogue takes 3 us
// at 256, hidden under the next tile's k-loop where there are two buffers; the cheapest in the sum over a CTA's tiles wins. More ranges than
// one: sums in registers (64 a thread, 128 in a pair) over accumulators in turn, except under a QK norm, which looks a head's features up in
// tensor memory. A pair's two accumulators leave room for one range of a second pair. MLB_COLS_PAIR=0|1: never | wherever it can run.
// Without sums (gemm_cols_can_sum, MLB_COLS_SUMS=0) every range has its accumulators until the tile's epilogue.
static ColsGemm gc_pick(int sm_count, int T, int N, int nkb, int nkb_x, int mode, bool exts_apart, int split, int min_bn, bool qk_norm, bool can_sum) {
    ColsGemm best{};
    double best_cost = -1.0;
    static const int bns[3] = {256, 128, 64};
    static const double t_kb[3] = {0.43, 0.36, 0.26};
    int mains = 0, exts = 0;
    for (int r = 0; r < split; ++r) {
        const int lo = (int)((long)nkb * r / split), hi = (int)((long)nkb * (r + 1) / split);
        if (exts_apart ? lo < nkb - nkb_x : hi > lo) ++mains;
        if (exts_apart && hi > nkb - nkb_x) ++exts;
    }
    const bool sums = can_sum && mains + exts > 1 && !(mode == TC_QKV && qk_norm) && exts < kGcMaxBufs;
    auto consider = [&](int bn, bool pair, int nbuf, double t_kb) {
        const int bn_out = mode == TC_SWIGLU ? bn / 2 : bn, rows = pair ? 2 * kGcM : kGcM, teams = pair ? sm_count / 2 : sm_count;
        const long tiles = (long)((T + rows - 1) / rows) * ((N + bn_out - 1) / bn_out);
        const long waves = (tiles + teams - 1) / teams;
        const double loop = nkb * t_kb, epi = 3.0 * bn / 256 + 0.5;
        const double cost = 1.5 + loop + epi + (waves - 1) * (nbuf >= 2 ? std::max(loop, epi) : loop + epi);
        if (best_cost >= 0 && cost >= best_cost) return;
        best_cost = cost;
        const int fit = (int)((kGcSmem - 1024 - gc_staging(mode)) / ((size_t)(kGcM + (pair ? bn / 2 : bn)) * 128));
        best.bn = bn; best.pair = pair;
        best.w_rows = mode == TC_SWIGLU || pair ? bn / 2 : bn;
        best.stages = (int)std::min<long>(std::min(fit, kGcMaxStages), std::max<long>(2, nkb * waves));
        best.ctas = (int)std::min<long>(tiles, teams) * (pair ? 2 : 1);
        best.split = split; best.mains = mains; best.exts = exts; best.sums = sums;
        best.nbuf = nbuf;
        best.tmem_cols = 32;
        while (best.tmem_cols < (uint32_t)(bn * nbuf * (sums ? 1 : mains + exts))) best.tmem_cols <<= 1;
    };
    for (int i = sums ? 1 : 0; i < 3; ++i) {
        if (bns[i] < min_bn) continue;
        if (sums) {
            consider(bns[i], false, kGcMaxBufs, t_kb[i]);
        } else {
            const int acc = bns[i] * (mains + exts);
            if (acc <= 512) consider(bns[i], false, 2 * acc <= 512 ? 2 : 1, t_kb[i]);
        }
    }
    const char* env = std::getenv("MLB_COLS_PAIR");
    if (T >= 2 * kGcM && (sums ? exts < 2 : mains + exts == 1) && !(env && env[0] == '0')) {
        if (env) best_cost = -1.0;
        consider(256, true, 2, 0.42);
    }
    return best;
}

// Buffers, tensor maps and launch shapes of a column set.
static int setup_cols_path(mlb_session* s) {
    const mlb_model* m = s->m;
    const mlb_config& c = m->cfg;
    s->use_cols = false;
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return MLB_OK;
    const bool w8 = c.weight_dtype == MLB_DT_FP8_E4M3;
    int rc;
    if (w8) {
        bool have = false;
        if ((rc = model_widen(s->m, s->stream, &have))) return rc;
        if ((s->no_copy = !have)) return MLB_OK;
    }
    if ((rc = build_step_layers(s))) return rc;
    const int T = s->B, nq = c.heads * c.head_dim, a_dn = c.heads * c.dn_value_dim;
    auto kb = [](int k) { return (k + kTcKB - 1) / kTcKB; };
    const bool ext2 = w8 && c.ple_dim > 0;
    int n_qkv = 0, n_dn = 0;
    for (const DevLayer& L : m->layers) (L.type == MLB_LAYER_ATTENTION ? n_qkv : n_dn) = L.n_qkv;
    // The ranges of k-blocks are those of gemm_tc_kernel's launches with kTcRefCols columns, whatever the width of this set, so
    // that a prompt's cache does not depend on how it is cut into chunks.
    if ((rc = tc_probe_clusters(s))) return rc;
    bool fits = true, can_sum = true;
    CU(gemm_cols_can_sum(&can_sum));
    if (const char* v = std::getenv("MLB_COLS_SUMS")) can_sum = can_sum && v[0] != '0';
    auto pick = [&](int N, int nkb, int nkb_x, int mode, bool apart) {
        const bool resid8 = w8 && mode == TC_RESID;
        const TcShape ref = tc_pick_shape(s, kTcRefCols, N, nkb, mode == TC_SWIGLU ? 2 : 1, w8, mode == TC_SWIGLU || resid8 ? 2 : 1);
        const ColsGemm g = gc_pick(s->sm_count, T, N, nkb, nkb_x, mode, apart, std::max(1, ref.split),
                                    mode == TC_QKV && c.qk_norm ? c.head_dim : 64, c.qk_norm != 0, can_sum);       // a tile holds whole heads for their norm
        fits = fits && g.bn > 0;
        return g;
    };
    if (n_qkv) s->cg_qkv = pick(n_qkv, kb(c.dim), 0, TC_QKV, false);
    if (n_dn) s->cg_dn = pick(n_dn, kb(c.dim), 0, TC_RAW, false);
    if (n_qkv) s->cg_o_attn = pick(c.dim, kb(nq), 0, TC_RESID, false);
    if (n_dn) s->cg_o_dn = pick(c.dim, kb(a_dn), 0, TC_RESID, false);
    s->cg_up = pick(c.ffn_dim, kb(c.dim), 0, TC_SWIGLU, false);
    s->cg_down = pick(c.dim, kb(c.ffn_dim) + kb(c.ple_dim), kb(c.ple_dim), TC_RESID, ext2);
    s->cg_last = pick(c.dim, kb(c.ffn_dim), 0, TC_RESID, false);
    s->cg_head = pick(c.vocab, kb(c.dim), 0, TC_RAW, false);
    if (!fits) return MLB_OK;      // ranges that tensor memory does not hold (a forced split, no sums)
    if ((rc = sess_alloc(s, (void**)&s->xn16, (size_t)T * c.dim * 2, true))) return rc;
    if ((rc = sess_alloc(s, (void**)&s->a16, (size_t)T * std::max(nq, a_dn) * 2, true))) return rc;
    if ((rc = sess_alloc(s, (void**)&s->h16, (size_t)T * c.ffn_dim * 2, true))) return rc;
    if ((rc = sess_alloc(s, (void**)&s->tc_ssq, (size_t)T * ((c.dim + 127) / 128) * 4 * 4, true))) return rc;
    if (c.ple_dim > 0 && (rc = sess_alloc(s, (void**)&s->tple16, (size_t)c.layers * T * c.ple_dim * 2, true))) return rc;
    s->tc_maps.resize(c.layers);
    for (int i = 0; i < c.layers; ++i) {
        const DevLayer& L = m->layers[i];
        auto& M = s->tc_maps[i];
        const void *wqkv = L.Wqkv, *wo = L.Wo, *w1a = L.W1a, *w1b = L.W1b, *w2 = L.W2;
        if (w8) { const auto& w = m->wide[i]; wqkv = w.Wqkv; wo = w.Wo; w1a = w.W1a; w1b = w.W1b; w2 = w.W2; }
        const int rows_qkv = L.type == MLB_LAYER_ATTENTION ? s->cg_qkv.w_rows : s->cg_dn.w_rows;
        if ((rc = make_bf16_map(enc, &M.qkv, wqkv, L.n_qkv, c.dim, rows_qkv))) return rc;
        if ((rc = make_bf16_map(enc, &M.o, wo, c.dim, L.o_in, L.type == MLB_LAYER_ATTENTION ? s->cg_o_attn.w_rows : s->cg_o_dn.w_rows))) return rc;
        if ((rc = make_bf16_map(enc, &M.w1a, w1a, c.ffn_dim, c.dim, s->cg_up.w_rows))) return rc;
        if ((rc = make_bf16_map(enc, &M.w1b, w1b, c.ffn_dim, c.dim, s->cg_up.w_rows))) return rc;
        if ((rc = make_bf16_map(enc, &M.w2, w2, c.dim, c.ffn_dim, (i + 1 < c.layers && c.ple_dim > 0) ? s->cg_down.w_rows : s->cg_last.w_rows))) return rc;
        if (c.ple_dim > 0) {
            if ((rc = make_bf16_map(enc, &M.pleP, L.pleP, c.dim, c.ple_dim, s->cg_down.w_rows))) return rc;
            if ((rc = make_bf16_map(enc, &M.pleT, s->tple16 + (size_t)i * T * c.ple_dim, T, c.ple_dim, kGcM))) return rc;
        }
    }
    if ((rc = make_bf16_map(enc, &s->tc_g.E, w8 ? m->wide_E : m->E, c.vocab, c.dim, s->cg_head.w_rows))) return rc;
    if ((rc = make_bf16_map(enc, &s->tc_g.xn[0], s->xn16, T, c.dim, kGcM))) return rc;
    if ((rc = make_bf16_map(enc, &s->tc_g.a_attn[0], s->a16, T, nq, kGcM))) return rc;
    if ((rc = make_bf16_map(enc, &s->tc_g.a_dn[0], s->a16, T, a_dn, kGcM))) return rc;
    if ((rc = make_bf16_map(enc, &s->tc_g.h[0], s->h16, T, c.ffn_dim, kGcM))) return rc;
    s->use_cols = true;
    return MLB_OK;
}

// Capture the chain once per kind; sampling parameters are baked into the top-k graph.
static int ensure_graph(mlb_session* s, int kind) {
    if (kind == CHAIN_TOPK && s->graphs[kind] && (s->g_topk != s->cur_topk || s->g_temp != s->cur_temp)) {
        cudaGraphExecDestroy(s->graphs[kind]);
        s->graphs[kind] = nullptr;
    }
    if (s->graphs[kind]) return MLB_OK;
    if (s->use_grid || s->use_lean) {
        // one cooperative launch per step (plus the sampler): launched directly, nothing to capture
        s->launches_per_step[kind] = kind == CHAIN_TOPK ? 2 : 1;
        if (kind == CHAIN_TOPK) { s->g_topk = s->cur_topk; s->g_temp = s->cur_temp; }
        return MLB_OK;
    }
    cudaGraph_t graph = nullptr;
    CU(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    int n = 0;
    int rc = chain_run(s, kind, nullptr, &n);
    cudaError_t e = cudaStreamEndCapture(s->stream, &graph);
    if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
    if (e != cudaSuccess) return fail(MLB_E_CUDA, "cudaStreamEndCapture failed: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(&s->graphs[kind], graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return fail(MLB_E_CUDA, "cudaGraphInstantiate failed: %s", cudaGetErrorString(e));
    s->launches_per_step[kind] = n;
    if (kind == CHAIN_TOPK) { s->g_topk = s->cur_topk; s->g_temp = s->cur_temp; }
    return MLB_OK;
}

// The one-token call (mlb_decode_step) as a single graph of the step's own kernels: the embedding
// kernel reads the pending ids from pinned host memory, the kernel that advances a sequence writes
// the picked id and the error word there. One launch and one synchronisation per token, no copy
// queued around the step (as graph nodes such copies cost more than the enqueues they replaced:
// 199 vs 188 us per token). The error word is copied when sequence 0 advances: a wait that runs out
// in the very last kernel of a step may be reported one call late.
static int ensure_token_graph(mlb_session* s, int kind, bool with_input) {
    const int idx = kind * 2 + (with_input ? 1 : 0);
    if (kind == CHAIN_TOPK && s->tgraphs[idx] && (s->tg_topk[with_input] != s->cur_topk || s->tg_temp[with_input] != s->cur_temp)) {
        cudaGraphExecDestroy(s->tgraphs[idx]);
        s->tgraphs[idx] = nullptr;
    }
    if (s->tgraphs[idx]) return MLB_OK;
    cudaGraph_t graph = nullptr;
    CU(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    int n = 0;
    s->ctl_host_io = with_input ? 2 : 1;
    int rc = chain_run(s, kind, nullptr, &n);
    s->ctl_host_io = 0;
    cudaError_t e = cudaStreamEndCapture(s->stream, &graph);
    if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
    if (e != cudaSuccess) return fail(MLB_E_CUDA, "capture of the one-token graph failed: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(&s->tgraphs[idx], graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return fail(MLB_E_CUDA, "cudaGraphInstantiate failed: %s", cudaGetErrorString(e));
    s->launches_per_step[kind] = n;
    if (kind == CHAIN_TOPK) { s->tg_topk[with_input] = s->cur_topk; s->tg_temp[with_input] = s->cur_temp; }
    return MLB_OK;
}

// One step on the session's stream: the captured chain, or the single cooperative kernel.
static int launch_step(mlb_session* s, int kind) {
    if (s->use_grid || s->use_lean) return chain_run(s, kind, nullptr, nullptr);
    CU(cudaGraphLaunch(s->graphs[kind], s->stream));
    return MLB_OK;
}

static int sync_page_table(mlb_session* s) {
    if (!s->table_dirty) return MLB_OK;
    for (int b = 0; b < s->B; ++b) {
        const auto& pg = s->alloc.seq_pages[b];
        for (size_t i = 0; i < pg.size(); ++i) s->h_table[(size_t)b * s->max_pages + i] = pg[i];
    }
    CU(cudaMemcpyAsync(s->page_table, s->h_table.data(), s->h_table.size() * 4, cudaMemcpyHostToDevice, s->stream));
    CU(cudaStreamSynchronize(s->stream));      // h_table may be rewritten by the next call
    s->table_dirty = false;
    return MLB_OK;
}

static int grow_pages(mlb_session* s, int extra_steps) {
    bool has_attn = false;
    for (auto* p : s->kpool) if (p) has_attn = true;
    if (!has_attn) return MLB_OK;
    for (int b = 0; b < s->B; ++b) {
        int want = s->h_stopped[b] ? s->h_pos[b] : std::min(s->h_pos[b] + extra_steps, s->max_ctx);
        size_t before = s->alloc.seq_pages[b].size();
        int rc = kv_ensure(&s->alloc, b, want, kKvBlock);
        if (s->alloc.seq_pages[b].size() != before) s->table_dirty = true;
        if (rc) return rc;
    }
    return sync_page_table(s);
}

// Where the parts of a column plan lie, for `T` columns of a session of `B` sequences.
struct ColsLayout {
    size_t tok, pos, lim, seq, runs, tiles, ints;
    int max_runs, max_tiles;
};
static ColsLayout cols_layout(const mlb_config& c, int B, int T) {
    ColsLayout l;
    l.max_runs = std::min(B, T);
    l.max_tiles = T / attn_cols_queries(c.heads / c.kv_heads) + l.max_runs;      // every run may end in a partial tile
    l.tok = 4; l.pos = l.tok + T; l.lim = l.pos + T; l.seq = l.lim + T;
    l.runs = l.seq + T; l.tiles = l.runs + 4 * (size_t)l.max_runs;
    l.ints = l.tiles + 4 * (size_t)l.max_tiles;
    return l;
}

static int apply_sampling(mlb_session* s, const mlb_sampling* sp, int* kind) {
    *kind = CHAIN_GREEDY;
    if (!sp || sp->mode == 0) return MLB_OK;
    if (sp->mode != 1) return fail(MLB_E_INVALID, "unknown sampling mode %d", sp->mode);
    if (sp->top_k < 1 || sp->top_k > kSampleCap) return fail(MLB_E_INVALID, "top_k must be in 1..%d", kSampleCap);
    if (!(sp->temperature > 0.f)) return fail(MLB_E_INVALID, "temperature must be > 0");
    s->cur_topk = sp->top_k;
    s->cur_temp = sp->temperature;
    *kind = CHAIN_TOPK;
    // The keys lie on the device from call to call; only other ones are sent (a copy and a synchronisation per token took 15 us of a
    // step of 256 sequences).
    bool same = (int)s->h_seeds.size() == s->B;
    for (int b = 0; b < s->B && same; ++b) same = s->h_seeds[b] == (sp->seeds ? sp->seeds[b] : (unsigned long long)b);
    if (same) return MLB_OK;
    s->h_seeds.clear();
    std::vector<unsigned long long> seeds(s->B);
    for (int b = 0; b < s->B; ++b) seeds[b] = sp->seeds ? sp->seeds[b] : (unsigned long long)b;
    CU(cudaMemcpyAsync(s->seeds, seeds.data(), (size_t)s->B * 8, cudaMemcpyHostToDevice, s->stream));
    CU(cudaStreamSynchronize(s->stream));
    s->h_seeds = std::move(seeds);
    return MLB_OK;
}

}  // namespace mlb

// A session, or (parent != null) the column set of one: `batch` columns of step buffers on the
// parent's KV pool, delta-net state and stream, always on the tensor-core step.
static int session_create(mlb_model* m, int batch, int max_context, int kv_block, int kv_pages, mlb_session* parent, mlb_session** out, bool gemv_cols = false) {
    if (!m || !out) return fail(MLB_E_INVALID, "null argument");
    *out = nullptr;
    if (batch < 1) return fail(MLB_E_INVALID, "batch must be >= 1");
    if (kv_block != 0 && kv_block != kKvBlock) return fail(MLB_E_UNSUPPORTED, "kv_block must be %d", kKvBlock);
    if (max_context <= 0) max_context = m->cfg.max_context;
    if (max_context > m->cfg.max_context) return fail(MLB_E_INVALID, "max_context %d exceeds the model's %d (RoPE table size)", max_context, m->cfg.max_context);
    CU(cudaSetDevice(m->device));
    const mlb_config& c = m->cfg;
    mlb_session* s = new mlb_session();
    s->m = m;
    s->B = batch;
    s->max_ctx = max_context;
    s->max_pages = (max_context + kKvBlock - 1) / kKvBlock;
    s->kv_pages = kv_pages > 0 ? kv_pages : batch * s->max_pages;
    s->parent = parent;
    if (parent) s->kv_pages = parent->kv_pages;
#define SA(expr) do { int r__ = (expr); if (r__) { free_session(s); return r__; } } while (0)
#define SCU(expr) do { cudaError_t e__ = (expr); if (e__ != cudaSuccess) { free_session(s); return fail(e__ == cudaErrorMemoryAllocation ? MLB_E_NOMEM : MLB_E_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__)); } } while (0)
    if (parent) s->stream = parent->stream;
    else SCU(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    const size_t B = batch;
    if (parent) {
        // positions, tokens, limits and sequences of the columns are one array, so that a chunk is one copy; no prompt
        // or output ring, no page table of its own
        const ColsLayout lay = cols_layout(c, parent->B, batch);
        SA(sess_alloc(s, (void**)&s->plan_dev, lay.ints * 4, true));
        s->tok = s->plan_dev + lay.tok; s->pos = s->plan_dev + lay.pos; s->seq_of = s->plan_dev + lay.seq;
        s->limit_prefill = s->limit_decode = s->plan_dev + lay.lim;
        s->plan.hdr = s->plan_dev;
        s->plan.runs = s->plan_dev + lay.runs; s->plan.max_runs = lay.max_runs;
        s->plan.tiles = s->plan_dev + lay.tiles; s->plan.max_tiles = lay.max_tiles;
        s->page_table = parent->page_table;
    } else {
        SA(sess_alloc(s, (void**)&s->pos, B * 4, true));
        SA(sess_alloc(s, (void**)&s->tok, B * 4, true));
        SA(sess_alloc(s, (void**)&s->limit_prefill, B * 4, true));
        SA(sess_alloc(s, (void**)&s->limit_decode, B * 4, true));
        SA(sess_alloc(s, (void**)&s->prompt, B * max_context * 4, true));
        SA(sess_alloc(s, (void**)&s->out_ring, B * max_context * 4, true));
        SA(sess_alloc(s, (void**)&s->out_idx, B * 4, true));
        SA(sess_alloc(s, (void**)&s->page_table, B * s->max_pages * 4, true));
        SA(sess_alloc(s, (void**)&s->seeds, B * 8, true));
    }
    const int nq = c.heads * c.head_dim;
    const int a_dim = std::max(nq, c.heads * c.dn_value_dim);
    bool has_dn = false, has_attn = false;
    for (int i = 0; i < c.layers; ++i) (c.layer_types[i] == MLB_LAYER_DELTA_NET ? has_dn : has_attn) = true;
    // a column set's attention over a bf16 cache (attn_cols_kernel) has no splits and writes the next operand only
    s->as_steps = parent && !gemv_cols && gemm_tcgen05_only();
    const bool split_attn = !parent || gemv_cols || s->as_steps || c.kv_dtype == MLB_DT_F32;
    s->max_q = nq;
    s->raw_stride = 2 * c.heads * c.dn_key_dim + c.heads * c.dn_value_dim + 2 * c.heads;
    SA(sess_alloc(s, (void**)&s->x, B * c.dim * 4, true));
    if (has_attn || !parent) SA(sess_alloc(s, (void**)&s->qbuf, B * nq * 4, true));
    if ((c.query_gating && has_attn) || !parent) SA(sess_alloc(s, (void**)&s->gbuf, B * nq * 4, true));
    if (split_attn) SA(sess_alloc(s, (void**)&s->abuf, B * a_dim * 4, true));
    if (has_dn || !parent) SA(sess_alloc(s, (void**)&s->raw, B * s->raw_stride * 4, true));
    if (!parent || gemv_cols) SA(sess_alloc(s, (void**)&s->hbuf, B * c.ffn_dim * 4, true));
    if (!parent) {
        SA(sess_alloc(s, (void**)&s->logits, B * c.vocab * 4, true));        // a column set's are made when a text is scored
        SA(sess_alloc(s, (void**)&s->probe, (size_t)c.vocab * 4, true));
    }
    // split count of the flash-decode: enough CTAs to cover the GPU at small batch, at least
    // four pages of work per split at full context
    int sm_count = 148;
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, m->device);
    int want = (4 * sm_count + c.kv_heads * batch - 1) / (c.kv_heads * batch);
    s->splits = std::max(1, std::min(std::min(want, 32), std::max(1, s->max_pages / 4)));
    if (const char* v = std::getenv("MLB_ATTN_SPLITS")) s->splits = std::max(1, std::min(32, std::atoi(v)));
    // pages a split must hold before a sequence uses it (the grid above already caps the splits at about four
    // CTAs per SM). Measured: cfg1 at 32 / 64 sequences and a context of 260, one split beats two (12.6 vs 15.5,
    // 16.3 vs 22.8 us per launch); the GQA model at 64 sequences and a context of 576, three splits of 11 pages
    // beat two of 18 and four of 9 (63 vs 78 and 74 us).
    s->attn_min_pps = 11;
    if (const char* v = std::getenv("MLB_ATTN_MIN_PAGES")) s->attn_min_pps = std::max(1, std::atoi(v));
    if (split_attn) {
        SA(sess_alloc(s, (void**)&s->part, B * c.heads * s->splits * (c.head_dim + 2) * 4, true));
        SA(sess_alloc(s, (void**)&s->attn_ticket, B * c.heads * 4, true));
    }
    s->lm_rows = 16;
    // argmax partials per sequence: one per LM-head CTA of either GEMV form (the streamed form
    // launches up to one CTA per SM, whatever the vocabulary size)
    s->lm_parts = std::max((c.vocab + s->lm_rows - 1) / s->lm_rows, 2 * sm_count);
    if (!parent) {         // columns pick nothing
        SA(sess_alloc(s, (void**)&s->part_val, B * s->lm_parts * 4, true));
        SA(sess_alloc(s, (void**)&s->part_idx, B * s->lm_parts * 4, true));
        SA(sess_alloc(s, (void**)&s->lm_ticket, (B + 7) / 1 * 4, true));
    }
    s->kpool.assign(c.layers, nullptr);
    s->vpool.assign(c.layers, nullptr);
    s->state.assign(c.layers, nullptr);
    const size_t kv_elt = elt_size(c.kv_dtype);
    for (int i = 0; i < c.layers; ++i) {
        if (parent) {
            s->kpool[i] = parent->kpool[i];
            s->vpool[i] = parent->vpool[i];
            s->state[i] = parent->state[i];
        } else if (c.layer_types[i] == MLB_LAYER_ATTENTION) {
            size_t bytes = (size_t)s->kv_pages * c.kv_heads * kKvBlock * c.head_dim * kv_elt;
            SA(sess_alloc(s, &s->kpool[i], bytes, true));
            SA(sess_alloc(s, &s->vpool[i], bytes, true));
        } else {
            SA(sess_alloc(s, (void**)&s->state[i], B * c.heads * c.dn_value_dim * c.dn_key_dim * 4, true));
        }
    }
    if (!parent) {
        s->flush_n = (192ull << 20) / 16;
        SA(sess_alloc(s, (void**)&s->flush_buf, s->flush_n * 16, false));
    }
    SCU(cudaMallocHost((void**)&s->pinned_err, 4));
    if (!parent) {
        SCU(cudaMallocHost((void**)&s->pinned_tok, B * 4));
        SCU(cudaMallocHost((void**)&s->pinned_out, B * 4));
    }
    *s->pinned_err = 0;
    if (!parent) {
        s->alloc.num_pages = s->kv_pages;
        s->alloc.max_pages_per_seq = s->max_pages;
        s->alloc.seq_pages.assign(batch, {});
        for (int p = s->kv_pages - 1; p >= 0; --p) s->alloc.free_list.push_back(p);
    }
    s->h_pos.assign(batch, 0);
    s->h_stopped.assign(batch, 0);
    if (!parent) {
        s->h_table.assign(B * s->max_pages, 0);
        std::vector<int> lim(batch, max_context);
        SCU(cudaMemcpy(s->limit_decode, lim.data(), B * 4, cudaMemcpyHostToDevice));
    }
    {
        const char* e = std::getenv("MLB_NO_PDL");     // measurement switch: plain stream-ordered launches
        s->use_pdl = !(e && e[0] == '1');
        const char* gv = std::getenv("MLB_GEMV");      // stream | thread | auto (stream for batch <= 4)
        const std::string gmode = gv ? gv : "auto";
        s->use_sgemv = !parent && (gmode == "stream" || (gmode == "auto" && batch <= 4));
        s->force_sgemv = gmode == "stream";
        if (const char* v = std::getenv("MLB_SG_STAGE_KB")) s->sg_stage_kb = std::max(8, std::min(96, std::atoi(v)));
        if (const char* v = std::getenv("MLB_SG_STAGES")) s->sg_max_stages = std::max(2, std::min(8, std::atoi(v)));
        cudaDeviceGetAttribute(&s->sm_count, cudaDevAttrMultiProcessorCount, m->device);
    }
    SA(sess_alloc(s, (void**)&s->dev_err, 4, true));
    if (!parent) {
        SA(chain_configure(s));
        SA(setup_lean_path(s));
        if (!s->use_lean) SA(setup_grid_path(s));
    }
    if (parent && !gemv_cols) {        // columns in fp32 run the GEMV chain
        if (!s->as_steps) SA(setup_cols_path(s));
        if (!s->use_cols) SA(setup_tc_path(s));
        if (!s->use_cols && !s->use_tc) {
            free_session(s);
            return fail(MLB_E_UNSUPPORTED, "prompt columns need tensor maps from the driver");
        }
    } else if (!parent) {
        SA(setup_tc_path(s));
    }
#undef SA
#undef SCU
    *out = s;
    return MLB_OK;
}

extern "C" int mlb_session_new(mlb_model* m, int batch, int max_context, int kv_block, int kv_pages, mlb_session** out) {
    if (!m || !out) return fail(MLB_E_INVALID, "null argument");
    return session_create(m, batch, max_context, kv_block, kv_pages, nullptr, out);
}

// Queues the reset of the device state and resets the host's.
static int reset_queued(mlb_session* s) {
    const size_t B = s->B;
    session_reset_kernel<<<(s->B + 127) / 128, 128, 0, s->stream>>>(s->B, s->max_ctx, s->pos, s->tok, s->limit_prefill, s->limit_decode, s->out_idx);
    CU(cudaGetLastError());
    const mlb_config& c = s->m->cfg;
    for (int i = 0; i < c.layers; ++i)
        if (s->state[i]) CU(cudaMemsetAsync(s->state[i], 0, B * c.heads * c.dn_value_dim * c.dn_key_dim * 4, s->stream));
    for (int b = 0; b < s->B; ++b) {
        for (int pg : s->alloc.seq_pages[b]) s->alloc.free_list.push_back(pg);
        s->alloc.seq_pages[b].clear();
        s->h_pos[b] = 0;
        s->h_stopped[b] = 0;
    }
    s->table_dirty = true;
    s->have_logits = false;
    return MLB_OK;
}

extern "C" int mlb_session_reset(mlb_session* s) {
    if (!s) return fail(MLB_E_INVALID, "null session");
    CU(cudaSetDevice(s->m->device));
    int rc = reset_queued(s);
    if (rc) return rc;
    CU(cudaStreamSynchronize(s->stream));
    return MLB_OK;
}

extern "C" void mlb_session_free(mlb_session* s) { free_session(s); }

// Prompt by columns. The token loop consumes a prompt one token per step and sequence: a
// 512-token prompt costs 511 steps. Here the prompt tokens of all sequences become the columns of
// tensor-core steps (bf16 or FP8 weights): the projections of up to kColMax tokens are one GEMM each,
// every column appends its K/V row and attends to the rows before it, and the delta-net recurrence walks the
// columns of a sequence in order (cols.cu). All tokens but the last of each prompt
// are consumed; the last one stays pending, as after the token loop. MLB_PREFILL = auto | step |
// chunk: auto takes this path from 64 prompt tokens on (its activations are bf16, so the cache
// differs from the token loop's within the low-precision tolerance); `*done` tells whether it ran.
// Models with fp32 weights run their columns through the GEMV chain instead, eight to a CTA, in fp32 like the token loop,
// wherever that loop would take kF32ColSteps steps or more. So do shorter prompts of the other models where the token loop
// has fp32 activations (one to three sequences, which have no tensor-core step), from kGemvColumns columns on.
//
// Width of a step: a column set of 256 leaves most SMs without a tile (d = 512: 4 row tiles of 128) and pays the
// step's ~45 launches once per 256 tokens; at 4096 columns the same launches carry 16 times the work.

// A step of columns costs 3.3 token steps of one sequence (0.27 and 0.59 ms on the two fp32 configurations, 8 or 12 columns), fewer
// of several sequences.
constexpr int kF32ColSteps = 4;
// bf16 / FP8 models, in columns: token loop -> columns, cfg1 553 -> 546 us at 6, 719 -> 537 at 8, 1394 -> 620 at 16, 5180 -> 1097 at 61;
// cfg3 2037 -> 1430 at 8; cfg4 5.0 -> 5.3 ms at 6, 6.6 -> 4.9 at 8, 51 -> 24 at 61. Several sequences share the loop's steps: three
// of 8 tokens 1427 -> 635 us on cfg1, so there a column set also has to replace kF32ColSteps of them.
constexpr int kGemvColumns = 8;

// The column set of kColMin << i columns, with room for their logits if they are `scored`. A set whose logits are refused is given back:
// a narrower one may fit in its place.
static int cols_make(mlb_session* s, int i, bool scored) {
    mlb_session*& cs = s->cols[i];
    int rc = MLB_OK;
    if (cs && cs->no_copy) {
        // made without the bf16 codes of an FP8 model: made again where they can be had by now
        bool have = false;
        if ((rc = model_widen(s->m, s->stream, &have))) return rc;
        if (have) {
            free_session(cs);
            cs = nullptr;
        }
    }
    if (!cs) rc = session_create(s->m, kColMin << i, s->max_ctx, 0, 0, s, &cs, s->m->cfg.weight_dtype == MLB_DT_F32);
    if (rc) cs = nullptr;
    else if (scored && !cs->logits && (rc = sess_alloc(cs, (void**)&cs->logits, (size_t)cs->B * s->m->cfg.vocab * 4, false))) {
        free_session(cs);
        cs = nullptr;
    }
    return rc;
}

// A column set for the next `n` columns: the narrowest that holds them, or, without memory for it, a wider one that exists or a
// narrower one, which takes fewer of them. `cap`: the widest that this call still asks for.
static int cols_get(mlb_session* s, long n, bool scored, int* cap, mlb_session** out) {
    for (;;) {
        int i = 0;
        while ((kColMin << i) < std::min<long>(n, *cap)) ++i;
        const int rc = cols_make(s, i, scored);
        *out = s->cols[i];
        if (rc != MLB_E_NOMEM) return rc;
        for (int j = i + 1; j < kColSets; ++j) {
            *out = s->cols[j];
            if (*out && (!scored || (*out)->logits)) return MLB_OK;
        }
        if (i == 0) return rc;
        *cap = kColMin << (i - 1);
    }
}

// Pinned ring of the chunks' plans.
static int plan_ring(mlb_session* s) {
    if (s->plan_host) return MLB_OK;
    for (auto& e : s->plan_free)
        if (!e) CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    s->plan_host_ints = cols_layout(s->m->cfg, s->B, kColMax).ints;
    CU(cudaMallocHost((void**)&s->plan_host, kPlanSlots * s->plan_host_ints * 4));
    return MLB_OK;
}

// score_out != null: the scoring forward instead (mlb_score_tokens): every token of sequence 0 is a
// column, the LM head runs on the columns too, and the logits of each chunk go to score_out.
static int prefill_columns(mlb_session* s, const int32_t* tokens, const int32_t* lens, int stride, bool* done, float* score_out = nullptr) {
    *done = false;
    const char* env = std::getenv("MLB_PREFILL");
    const std::string mode = score_out ? "chunk" : (env ? env : "auto");
    if (mode == "step") return MLB_OK;
    const int B = score_out ? 1 : s->B;
    const int keep = score_out ? 0 : 1;            // tokens per prompt that stay pending
    const int kind = score_out ? CHAIN_GREEDY : CHAIN_PREFILL;
    long total = 0;
    for (int b = 0; b < B; ++b) total += lens[b] - keep;
    const mlb_config& cfg = s->m->cfg;
    const bool f32 = cfg.weight_dtype == MLB_DT_F32;
    if (f32 && mode == "chunk") return fail(MLB_E_UNSUPPORTED, "MLB_PREFILL=chunk needs bf16 or FP8 weights");
    int longest = 0;
    for (int b = 0; b < B; ++b) longest = std::max(longest, lens[b] - keep);
    const bool gemv = !f32 && mode == "auto" && !s->use_tc && total < kColMin;      // fewer columns than the narrowest set holds
    if (total < 1 || (mode == "auto" && (f32 ? longest < kF32ColSteps : gemv ? (total < kGemvColumns || longest < kF32ColSteps) : total < kColMin))) return MLB_OK;
    int rc, cap = kColMax;
    mlb_session* cs = nullptr;
    if (s->cols_failed && mode != "chunk") return MLB_OK;
    auto get = [&](long n) {
        if (!gemv) return cols_get(s, n, score_out != nullptr, &cap, &cs);
        if (!s->cols_gemv) {
            const int r = session_create(s->m, kColMin, s->max_ctx, 0, 0, s, &s->cols_gemv, true);
            if (r) { s->cols_gemv = nullptr; return r; }
        }
        cs = s->cols_gemv;
        return (int)MLB_OK;
    };
    if ((rc = get(total)) || (rc = plan_ring(s))) {
        s->cols_failed = rc != MLB_E_NOMEM;        // memory may come back: asked for again by the next prompt
        return mode == "chunk" ? rc : (int)MLB_OK;
    }
    bool has_dn = false, has_attn = false;
    for (int i = 0; i < cfg.layers; ++i) (cfg.layer_types[i] == MLB_LAYER_DELTA_NET ? has_dn : has_attn) = true;
    const size_t V = (size_t)cfg.vocab;
    const int qt = attn_cols_queries(cfg.heads / cfg.kv_heads);
    size_t scored = 0;
    // A chunk takes the next tokens of as many sequences as it can, an equal share each: the
    // delta-net recurrence is serial along a sequence and parallel across sequences. Columns stay grouped by
    // sequence, positions ascending.
    std::vector<int> cursor(B, 0), rest(B), take(B);
    long left = total;
    for (int slot = 0; left > 0; slot = (slot + 1) % kPlanSlots) {
        if ((rc = get(left))) return rc;
        const int want = (int)std::min<long>(left, cs->B);
        for (int b = 0; b < B; ++b) rest[b] = lens[b] - keep - cursor[b];
        cols_shares(rest, cursor, want, has_attn && !f32 ? qt : 0, take);
        const ColsLayout lay = cols_layout(cfg, s->B, cs->B);
        int* pl = s->plan_host + slot * s->plan_host_ints;
        CU(cudaEventSynchronize(s->plan_free[slot]));      // the slot's last plan has left it, also one of a call that failed half-way
        int n = 0, runs = 0, tiles = 0, longest = 0;
        for (int b = 0; b < B; ++b) {
            if (take[b] <= 0) continue;
            longest = std::max(longest, take[b]);
            int* r = pl + lay.runs + 4 * (size_t)runs++;
            r[0] = n; r[1] = take[b]; r[2] = b; r[3] = cursor[b];
            for (int q = 0; q < take[b]; q += qt) {
                int* t = pl + lay.tiles + 4 * (size_t)tiles++;
                t[0] = n + q; t[1] = std::min(qt, take[b] - q); t[2] = b; t[3] = cursor[b] + q;
            }
            for (int i = 0; i < take[b]; ++i, ++n) {
                const int t = cursor[b] + i;
                pl[lay.tok + n] = tokens[(size_t)b * stride + t];
                pl[lay.pos + n] = t;
                pl[lay.lim + n] = t + 1;        // active: pos < limit
                pl[lay.seq + n] = b;
            }
            cursor[b] += take[b];
        }
        for (int i = n; i < cs->B; ++i) pl[lay.tok + i] = pl[lay.pos + i] = pl[lay.lim + i] = pl[lay.seq + i] = 0;      // idle columns
        pl[0] = n; pl[1] = runs; pl[2] = tiles; pl[3] = 0;
        left -= n;
        const bool few = has_dn && delta_cols_serial(s->sm_count, cfg.heads, cfg.dn_value_dim, n, longest);
        if (cs->few_runs != few) {
            std::swap(cs->graphs, cs->other_graphs);
            cs->few_runs = few;
        }
        if ((rc = ensure_graph(cs, kind))) return rc;
        CU(cudaMemcpyAsync(cs->plan_dev, pl, lay.ints * 4, cudaMemcpyHostToDevice, s->stream));
        CU(cudaEventRecord(s->plan_free[slot], s->stream));
        CU(cudaGraphLaunch(cs->graphs[kind], s->stream));
        if (score_out) {
            // one sequence: the columns of a chunk are its next n positions, in order
            CU(cudaMemcpyAsync(score_out + scored * V, cs->logits, (size_t)n * V * 4, cudaMemcpyDeviceToHost, s->stream));
            scored += (size_t)n;
        }
        if ((rc = queue_err_readback(cs))) return rc;
    }
    if (!score_out) {
        // what the token loop would have left: position len-1 with the last prompt token pending
        for (int i = 0; i < B; ++i) { s->pinned_out[i] = lens[i] - 1; s->pinned_tok[i] = tokens[(size_t)i * stride + lens[i] - 1]; }
        CU(cudaMemcpyAsync(s->pos, s->pinned_out, (size_t)B * 4, cudaMemcpyHostToDevice, s->stream));
        CU(cudaMemcpyAsync(s->tok, s->pinned_tok, (size_t)B * 4, cudaMemcpyHostToDevice, s->stream));
    }
    CU(cudaStreamSynchronize(s->stream));
    *done = true;
    rc = s->cols_gemv ? check_err_readback(s->cols_gemv) : (int)MLB_OK;
    for (auto* c2 : s->cols)
        if (const int r = c2 ? check_err_readback(c2) : (int)MLB_OK) rc = r;
    return rc;
}

extern "C" int mlb_prefill(mlb_session* s, const int32_t* tokens, const int32_t* lens, int stride) {
    if (!s || !tokens || !lens) return fail(MLB_E_INVALID, "null argument");
    CU(cudaSetDevice(s->m->device));
    const int B = s->B, V = s->m->cfg.vocab;
    int max_len = 0;
    for (int b = 0; b < B; ++b) {
        if (lens[b] < 1) return fail(MLB_E_INVALID, "sequence %d: prompt length must be >= 1 (got %d)", b, lens[b]);
        if (lens[b] > s->max_ctx) return fail(MLB_E_CONTEXT_FULL, "sequence %d: prompt of %d tokens exceeds max_context %d", b, lens[b], s->max_ctx);
        if (lens[b] > stride) return fail(MLB_E_INVALID, "sequence %d: length %d exceeds stride %d", b, lens[b], stride);
        for (int i = 0; i < lens[b]; ++i) {
            int t = tokens[(size_t)b * stride + i];
            if (t < 0 || t >= V) return fail(MLB_E_INVALID, "sequence %d: token %d at position %d is outside the vocabulary (%d)", b, t, i, V);
        }
        max_len = std::max(max_len, lens[b]);
    }
    int rc = reset_queued(s);
    if (rc) return rc;
    // pages for the whole prompt before any launch
    bool has_attn = false;
    for (auto* p : s->kpool) if (p) has_attn = true;
    if (has_attn) {
        for (int b = 0; b < B; ++b) {
            if ((rc = kv_ensure(&s->alloc, b, lens[b], kKvBlock))) return rc;
        }
        s->table_dirty = true;
        if ((rc = sync_page_table(s))) return rc;
    }
    bool by_columns = false;
    if ((rc = prefill_columns(s, tokens, lens, stride, &by_columns))) {
        cudaStreamSynchronize(s->stream);          // chunks may be under way
        return rc;
    }
    if (!by_columns) {
        std::vector<int> hp((size_t)B * s->max_ctx, 0), first(B), lim(B);
        for (int b = 0; b < B; ++b) {
            std::memcpy(&hp[(size_t)b * s->max_ctx], &tokens[(size_t)b * stride], (size_t)lens[b] * 4);
            first[b] = tokens[(size_t)b * stride];
            lim[b] = lens[b] - 1;
        }
        CU(cudaMemcpyAsync(s->prompt, hp.data(), hp.size() * 4, cudaMemcpyHostToDevice, s->stream));
        CU(cudaMemcpyAsync(s->tok, first.data(), (size_t)B * 4, cudaMemcpyHostToDevice, s->stream));
        CU(cudaMemcpyAsync(s->limit_prefill, lim.data(), (size_t)B * 4, cudaMemcpyHostToDevice, s->stream));
        if (max_len > 1) {
            if ((rc = ensure_graph(s, CHAIN_PREFILL))) { cudaStreamSynchronize(s->stream); return rc; }
            for (int t = 0; t < max_len - 1; ++t)
                if ((rc = launch_step(s, CHAIN_PREFILL))) { cudaStreamSynchronize(s->stream); return rc; }
        }
        if ((rc = queue_err_readback(s))) { cudaStreamSynchronize(s->stream); return rc; }
        CU(cudaStreamSynchronize(s->stream));
    }
    for (int b = 0; b < B; ++b) s->h_pos[b] = lens[b] - 1;
    return by_columns ? (int)MLB_OK : check_err_readback(s);
}

extern "C" int mlb_score_tokens(mlb_session* s, const int32_t* tokens, int len, float* logits_out) {
    if (!s || !tokens || !logits_out) return fail(MLB_E_INVALID, "null argument");
    if (len < 1) return fail(MLB_E_INVALID, "len must be >= 1");
    if (len > s->max_ctx) return fail(MLB_E_CONTEXT_FULL, "%d tokens exceed max_context %d", len, s->max_ctx);
    CU(cudaSetDevice(s->m->device));
    const int V = s->m->cfg.vocab;
    for (int i = 0; i < len; ++i)
        if (tokens[i] < 0 || tokens[i] >= V) return fail(MLB_E_INVALID, "token %d at position %d is outside the vocabulary (%d)", tokens[i], i, V);
    const char* mode = std::getenv("MLB_SCORE");
    const bool by_steps = (mode && std::string(mode) == "step") ||
                          (s->m->cfg.weight_dtype != MLB_DT_BF16 && s->m->cfg.weight_dtype != MLB_DT_FP8_E4M3);
    if (by_steps) {
        // fp32 weights (or MLB_SCORE=step): the token loop with the given ids forced in, fp32 activations, the
        // logits of every step copied out - what the reference's trainer reads after runInference(L)
        // (training_orchestrator.cu:308), within the fp32 bound of the decode path
        std::vector<int32_t> first(s->B, 0), lens(s->B, 1), in(s->B, 0), out(s->B, 0);
        first[0] = tokens[0];
        int rc = mlb_prefill(s, first.data(), lens.data(), 1);
        if (rc) return rc;
        std::vector<float> row((size_t)s->B * V);
        for (int t = 0; t < len; ++t) {
            in[0] = tokens[t];
            if ((rc = mlb_decode_step(s, nullptr, in.data(), out.data()))) return rc;
            if ((rc = mlb_get_logits(s, row.data()))) return rc;
            std::memcpy(logits_out + (size_t)t * V, row.data(), (size_t)V * 4);
        }
        return mlb_session_reset(s);
    }
    int rc = mlb_session_reset(s);
    if (rc) return rc;
    bool has_attn = false;
    for (auto* p : s->kpool) if (p) has_attn = true;
    if (has_attn) {
        if ((rc = kv_ensure(&s->alloc, 0, len, kKvBlock))) return rc;
        s->table_dirty = true;
        if ((rc = sync_page_table(s))) return rc;
    }
    bool done = false;
    const int32_t lens[1] = {len};
    rc = prefill_columns(s, tokens, lens, len, &done, logits_out);
    const int rc2 = mlb_session_reset(s);          // the cache holds the scored sequence: not a state to decode from
    if (rc) return rc;
    if (!done) return fail(MLB_E_UNSUPPORTED, "the scoring forward could not set up its tensor-core columns");
    return rc2;
}

extern "C" int mlb_session_set_stop_token(mlb_session* s, int token_id) {
    if (!s) return fail(MLB_E_INVALID, "null session");
    if (token_id >= s->m->cfg.vocab) return fail(MLB_E_INVALID, "stop token %d is outside the vocabulary of %d", token_id, s->m->cfg.vocab);
    if (token_id < 0) token_id = -1;
    if (token_id == s->stop_token) return MLB_OK;
    CU(cudaSetDevice(s->m->device));
    CU(cudaStreamSynchronize(s->stream));
    // the id is an argument of the captured launches: capture again on next use
    for (auto& g : s->graphs) if (g) { cudaGraphExecDestroy(g); g = nullptr; }
    for (auto& g : s->tgraphs) if (g) { cudaGraphExecDestroy(g); g = nullptr; }
    s->stop_token = token_id;
    return MLB_OK;
}

extern "C" int mlb_session_stopped(mlb_session* s, int32_t* out_flags) {
    if (!s || !out_flags) return fail(MLB_E_INVALID, "null argument");
    for (int b = 0; b < s->B; ++b) out_flags[b] = s->h_stopped[b] ? 1 : 0;
    return MLB_OK;
}

namespace mlb {
// Shared body of the decode entry points. step_ms != null times each step.
static int decode_impl(mlb_session* s, const mlb_sampling* sp, int n, const int32_t* in_tokens, int32_t* out_tokens,
                       float* step_ms, float* total_ms, int flush_l2) {
    if (!s || !out_tokens) return fail(MLB_E_INVALID, "null argument");
    if (n < 1) return fail(MLB_E_INVALID, "n must be >= 1");
    CU(cudaSetDevice(s->m->device));
    const int B = s->B;
    bool any = false;
    for (int b = 0; b < B; ++b) any = any || seq_live(s, b);
    if (!any) return fail(MLB_E_CONTEXT_FULL, "every sequence is at max_context %d or has drawn the stop token", s->max_ctx);
    const int n_out = n;                       // ids per sequence in out_tokens; behind max_context steps none is left to take
    n = std::min(n, s->max_ctx);
    int kind, rc;
    if ((rc = apply_sampling(s, sp, &kind))) return rc;
    if ((rc = grow_pages(s, n))) return rc;
    if (in_tokens) {
        const int V = s->m->cfg.vocab;
        for (int b = 0; b < B; ++b) {
            if (in_tokens[b] < 0 || in_tokens[b] >= V) return fail(MLB_E_INVALID, "sequence %d: token %d is outside the vocabulary", b, in_tokens[b]);
            s->pinned_tok[b] = in_tokens[b];
        }
    }
    if (n_out == 1 && !step_ms && !s->use_grid && !s->use_lean) {
        // the one-token call: one graph launch, one synchronisation
        if ((rc = ensure_token_graph(s, kind, in_tokens != nullptr))) return rc;
        // The kernel that advances a sequence writes its id to pinned host memory (the error word first, by
        // sequence 0): the host polls those words instead of synchronising the stream, which wakes it later.
        const bool poll = seq_live(s, 0);
        volatile int* words = s->pinned_out;
        if (poll)
            for (int b = 0; b < B; ++b) words[b] = seq_live(s, b) ? -2 : -1;
        CU(cudaGraphLaunch(s->tgraphs[kind * 2 + (in_tokens ? 1 : 0)], s->stream));
        bool arrived = false;
        if (poll) {
            const auto t0 = std::chrono::steady_clock::now();
            for (unsigned spins = 0; !arrived; ++spins) {
                arrived = true;
                for (int b = 0; b < B; ++b)
                    if (words[b] == -2) { arrived = false; break; }
                if (!arrived && (spins & 0xfffu) == 0xfffu && std::chrono::steady_clock::now() - t0 > std::chrono::seconds(5)) break;
            }
        }
        if (!arrived) CU(cudaStreamSynchronize(s->stream));
        for (int b = 0; b < B; ++b) {
            out_tokens[b] = s->pinned_out[b];
            note_outputs(s, b, &out_tokens[b], 1);
        }
        s->have_logits = true;
        return check_err_readback(s);
    }
    if (n_out == 1 && !step_ms && B == 1 && (s->use_grid || s->use_lean) && seq_live(s, 0)) {
        // The one-token call of the single-kernel step: the pending id travels as a launch argument, the
        // kernel that advances the sequence writes the picked id and the error word to pinned host memory,
        // and the host polls that word instead of synchronising the stream (which costs 5-10 us more).
        if ((rc = ensure_graph(s, kind))) return rc;
        volatile int* word = s->pinned_out;
        *word = -2;
        s->ctl_host_io = 1;
        s->tok_arg = in_tokens ? in_tokens[0] : -1;
        rc = chain_run(s, kind, nullptr, nullptr);
        s->ctl_host_io = 0;
        s->tok_arg = -1;
        if (rc) return rc;
        const auto t0 = std::chrono::steady_clock::now();
        for (unsigned spins = 0; *word == -2; ++spins) {
            if ((spins & 0xffffu) == 0xffffu && std::chrono::steady_clock::now() - t0 > std::chrono::seconds(5)) break;
        }
        if (*word == -2) CU(cudaStreamSynchronize(s->stream));       // a wait ran out on the device, or the launch failed late
        if (*word == -2) return fail(MLB_E_CUDA, "the decode step ended without a token");
        out_tokens[0] = *word;
        note_outputs(s, 0, &out_tokens[0], 1);
        s->have_logits = true;
        return check_err_readback(s);
    }
    if ((rc = ensure_graph(s, kind))) return rc;
    if (in_tokens) CU(cudaMemcpyAsync(s->tok, s->pinned_tok, (size_t)B * 4, cudaMemcpyHostToDevice, s->stream));
    CU(cudaMemsetAsync(s->out_idx, 0, (size_t)B * 4, s->stream));
    std::vector<cudaEvent_t> ev;
    if (step_ms) {
        ev.resize(2 * (size_t)n);
        for (auto& e : ev) CU(cudaEventCreate(&e));
    }
    for (int i = 0; i < n; ++i) {
        if (step_ms) {
            if (flush_l2) {
                l2_flush_kernel<<<1184, 256, 0, s->stream>>>(s->flush_buf, s->flush_n, (float)i);
                CU(cudaGetLastError());
            }
            CU(cudaEventRecord(ev[2 * i], s->stream));
        }
        if ((rc = launch_step(s, kind))) return rc;
        if (step_ms) CU(cudaEventRecord(ev[2 * i + 1], s->stream));
    }
    // result: ring [B][max_ctx] -> out [B][n]
    if ((rc = queue_err_readback(s))) return rc;
    if (n == 1) {
        // one id per sequence: gather through the pinned buffer
        CU(cudaMemcpy2DAsync(s->pinned_tok, 4, s->out_ring, (size_t)s->max_ctx * 4, 4, B, cudaMemcpyDeviceToHost, s->stream));
        CU(cudaStreamSynchronize(s->stream));
        for (int b = 0; b < B; ++b) out_tokens[(size_t)b * n_out] = s->pinned_tok[b];
    } else {
        std::vector<int> ring((size_t)B * n);
        CU(cudaMemcpy2DAsync(ring.data(), (size_t)n * 4, s->out_ring, (size_t)s->max_ctx * 4, (size_t)n * 4, B, cudaMemcpyDeviceToHost, s->stream));
        CU(cudaStreamSynchronize(s->stream));
        for (int b = 0; b < B; ++b) std::memcpy(out_tokens + (size_t)b * n_out, &ring[(size_t)b * n], (size_t)n * 4);
    }
    if (step_ms) {
        std::fill(step_ms + n, step_ms + n_out, 0.f);
        for (int i = 0; i < n; ++i) CU(cudaEventElapsedTime(&step_ms[i], ev[2 * i], ev[2 * i + 1]));
        if (total_ms) CU(cudaEventElapsedTime(total_ms, ev[0], ev[2 * (size_t)n - 1]));
        for (auto& e : ev) cudaEventDestroy(e);
    }
    for (int b = 0; b < B; ++b) {
        note_outputs(s, b, &out_tokens[(size_t)b * n_out], n);
        std::fill(&out_tokens[(size_t)b * n_out] + n, &out_tokens[(size_t)b * n_out] + n_out, -1);
    }
    s->have_logits = true;
    return check_err_readback(s);
}
}  // namespace mlb

extern "C" int mlb_decode_step(mlb_session* s, const mlb_sampling* sp, const int32_t* in_tokens, int32_t* out_tokens) {
    return decode_impl(s, sp, 1, in_tokens, out_tokens, nullptr, nullptr, 0);
}
extern "C" int mlb_decode_n(mlb_session* s, const mlb_sampling* sp, int n, int32_t* out_tokens) {
    return decode_impl(s, sp, n, nullptr, out_tokens, nullptr, nullptr, 0);
}
extern "C" int mlb_decode_timed(mlb_session* s, const mlb_sampling* sp, int n, int flush_l2, float* step_ms, float* total_ms,
                                int32_t* out_tokens) {
    if (!step_ms) return fail(MLB_E_INVALID, "null step_ms");
    return decode_impl(s, sp, n, nullptr, out_tokens, step_ms, total_ms, flush_l2);
}

extern "C" int mlb_profile_decode(mlb_session* s, const mlb_sampling* sp, int n, int flush_l2, mlb_kernel_stat* stats,
                                  int max_stats, int* n_stats) {
    if (!s || !stats || !n_stats) return fail(MLB_E_INVALID, "null argument");
    CU(cudaSetDevice(s->m->device));
    int kind, rc;
    if ((rc = apply_sampling(s, sp, &kind))) return rc;
    if ((rc = grow_pages(s, n))) return rc;
    CU(cudaMemsetAsync(s->out_idx, 0, (size_t)s->B * 4, s->stream));
    Recorder rec;
    rec.st = s->stream;
    for (int i = 0; i < n; ++i) {
        bool any = false;
        for (int b = 0; b < s->B; ++b) any = any || seq_live(s, b);
        if (!any) break;
        if (flush_l2) {
            l2_flush_kernel<<<1184, 256, 0, s->stream>>>(s->flush_buf, s->flush_n, (float)i);
            CU(cudaGetLastError());
        }
        if ((rc = chain_run(s, kind, &rec, nullptr))) return rc;
        for (int b = 0; b < s->B; ++b) if (seq_live(s, b)) s->h_pos[b] += 1;
    }
    CU(cudaStreamSynchronize(s->stream));
    if (s->stop_token >= 0) {
        // no ids came back: take positions and who stopped from the device
        std::vector<int> dp(s->B), dl(s->B);
        CU(cudaMemcpy(dp.data(), s->pos, (size_t)s->B * 4, cudaMemcpyDeviceToHost));
        CU(cudaMemcpy(dl.data(), s->limit_decode, (size_t)s->B * 4, cudaMemcpyDeviceToHost));
        for (int b = 0; b < s->B; ++b) {
            s->h_pos[b] = std::min(dp[b], s->max_ctx);
            s->h_stopped[b] = dl[b] < s->max_ctx;
        }
    }
    s->have_logits = true;
    int count = 0;
    for (auto& r : rec.recs) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, r.e0, r.e1);
        cudaEventDestroy(r.e0);
        cudaEventDestroy(r.e1);
        int j = 0;
        for (; j < count; ++j) if (std::strcmp(stats[j].name, r.name) == 0) break;
        if (j == count) {
            if (count >= max_stats) continue;
            std::memset(&stats[j], 0, sizeof stats[j]);
            std::strncpy(stats[j].name, r.name, sizeof(stats[j].name) - 1);
            ++count;
        }
        stats[j].launches += 1;
        stats[j].total_ms += ms;
        stats[j].bytes += r.bytes;
        stats[j].flops += r.flops;
    }
    *n_stats = count;
    return MLB_OK;
}

extern "C" int mlb_get_logits(mlb_session* s, float* out) {
    if (!s || !out) return fail(MLB_E_INVALID, "null argument");
    if (!s->have_logits) return fail(MLB_E_INVALID, "no decode step has run since the last prefill/reset");
    CU(cudaSetDevice(s->m->device));
    CU(cudaMemcpyAsync(out, s->logits, (size_t)s->B * s->m->cfg.vocab * 4, cudaMemcpyDeviceToHost, s->stream));
    CU(cudaStreamSynchronize(s->stream));
    return MLB_OK;
}

extern "C" int mlb_get_probs_col(mlb_session* s, int seq, float* out) {
    if (!s || !out) return fail(MLB_E_INVALID, "null argument");
    if (seq < 0 || seq >= s->B) return fail(MLB_E_INVALID, "sequence index out of range");
    if (!s->have_logits) return fail(MLB_E_INVALID, "no decode step has run since the last prefill/reset");
    CU(cudaSetDevice(s->m->device));
    const int V = s->m->cfg.vocab;
    softmax_probe_kernel<<<1, 256, 0, s->stream>>>(s->logits + (size_t)seq * V, V, s->probe);
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(out, s->probe, (size_t)V * 4, cudaMemcpyDeviceToHost, s->stream));
    CU(cudaStreamSynchronize(s->stream));
    return MLB_OK;
}

extern "C" int mlb_session_positions(mlb_session* s, int32_t* out) {
    if (!s || !out) return fail(MLB_E_INVALID, "null argument");
    CU(cudaSetDevice(s->m->device));
    CU(cudaMemcpyAsync(out, s->pos, (size_t)s->B * 4, cudaMemcpyDeviceToHost, s->stream));
    CU(cudaStreamSynchronize(s->stream));
    return MLB_OK;
}

extern "C" int mlb_session_step_bytes(mlb_session* s, uint64_t* weights, uint64_t* kv, uint64_t* state, uint64_t* rows) {
    if (!s) return fail(MLB_E_INVALID, "null session");
    const mlb_config& c = s->m->cfg;
    uint64_t kvb = 0, st = 0, rw = 0;
    const uint64_t kv_elt = elt_size(c.kv_dtype), w_elt = elt_size(c.weight_dtype), p_elt = elt_size(ple_dtype(c.weight_dtype));
    for (int b = 0; b < s->B; ++b) {
        if (!seq_live(s, b)) continue;
        for (int i = 0; i < c.layers; ++i) {
            if (c.layer_types[i] == MLB_LAYER_ATTENTION) kvb += 2ull * c.kv_heads * c.head_dim * kv_elt * (s->h_pos[b] + 1);
            else st += 2ull * c.heads * c.dn_key_dim * c.dn_value_dim * 4;
        }
        rw += (uint64_t)c.dim * w_elt + (uint64_t)c.layers * c.ple_dim * p_elt;
    }
    if (weights) *weights = s->m->weight_bytes;   // the tied table is streamed once (LM head)
    if (kv) *kv = kvb;
    if (state) *state = st;
    if (rows) *rows = rw;
    return MLB_OK;
}

extern "C" int mlb_session_grid_timers(mlb_session* s, long long* out, int cap) {
    if (!s || !out) return fail(MLB_E_INVALID, "null argument");
    long long* timers = s->use_lean ? s->lean.timers : (s->use_grid ? s->grid.timers : nullptr);
    if (!timers) return 0;
    CU(cudaSetDevice(s->m->device));
    const int n = s->grid_ctas * kGridTimerSlots;
    if (cap < n) return fail(MLB_E_INVALID, "room for %d counters needed, %d given", n, cap);
    CU(cudaStreamSynchronize(s->stream));
    CU(cudaMemcpy(out, timers, (size_t)n * 8, cudaMemcpyDeviceToHost));
    CU(cudaMemset(timers, 0, (size_t)n * 8));
    return s->grid_ctas;
}

extern "C" int mlb_session_grid_trace(mlb_session* s, long long* out, int cap) {
    if (!s || !out) return fail(MLB_E_INVALID, "null argument");
    if (s->tc_trace) {
        // tensor-core step: 8 words per GEMM launch of the last step (entry, set up, predecessor complete,
        // accumulators complete, epilogue done), 64 launches at most
        if (cap < 512) return fail(MLB_E_INVALID, "room for 512 words needed, %d given", cap);
        CU(cudaSetDevice(s->m->device));
        CU(cudaStreamSynchronize(s->stream));
        CU(cudaMemcpy(out, s->tc_trace, 512 * 8, cudaMemcpyDeviceToHost));
        return 64;
    }
    if (!s->use_lean || !s->lean.trace) return 0;
    CU(cudaSetDevice(s->m->device));
    const int n = s->grid_ctas * kLeanTraceLen;
    if (cap < n) return fail(MLB_E_INVALID, "room for %d events needed, %d given", n, cap);
    CU(cudaStreamSynchronize(s->stream));
    CU(cudaMemcpy(out, s->lean.trace, (size_t)n * 8, cudaMemcpyDeviceToHost));
    return s->grid_ctas;
}

extern "C" int mlb_session_launches_per_step(mlb_session* s) {
    if (!s) return fail(MLB_E_INVALID, "null session");
    int rc = ensure_graph(s, CHAIN_GREEDY);
    if (rc) return rc;
    return s->launches_per_step[CHAIN_GREEDY];
}

extern "C" const char* mlb_session_path(const mlb_session* s, int columns) {
    if (!s || columns < 0) return "none";
    if (columns > 0) {
        int i = 0;
        while (i + 1 < kColSets && (kColMin << i) < columns) ++i;
        const mlb_session* cs = s->cols[i] ? s->cols[i] : (i == 0 ? s->cols_gemv : nullptr);
        return !cs ? "none" : (cs->use_cols ? "cols" : (cs->use_tc ? "tcgen05" : "gemv"));
    }
    if (s->use_lean || s->use_grid) return s->use_lean ? "lean" : "grid";
    return !s->use_tc ? "gemv" : (s->use_dec ? "mma" : "tcgen05");
}

// ---- host-only allocator entry points --------------------------------------------------
extern "C" int mlb_kv_alloc_new(int num_pages, int batch, int max_pages_per_seq, mlb_kv_alloc** out) {
    if (!out || num_pages < 0 || batch < 1 || max_pages_per_seq < 1) return fail(MLB_E_INVALID, "kv allocator: bad argument");
    mlb_kv_alloc* a = new mlb_kv_alloc();
    a->num_pages = num_pages;
    a->max_pages_per_seq = max_pages_per_seq;
    a->seq_pages.assign(batch, {});
    for (int p = num_pages - 1; p >= 0; --p) a->free_list.push_back(p);
    *out = a;
    return MLB_OK;
}
extern "C" int mlb_kv_alloc_ensure(mlb_kv_alloc* a, int seq, int n_positions, int block) { return kv_ensure(a, seq, n_positions, block); }
extern "C" int mlb_kv_alloc_table(const mlb_kv_alloc* a, int seq, int32_t* out, int max_entries) {
    if (!a || !out || seq < 0 || seq >= (int)a->seq_pages.size()) return fail(MLB_E_INVALID, "kv allocator: bad argument");
    const auto& pg = a->seq_pages[seq];
    int n = std::min((int)pg.size(), max_entries);
    for (int i = 0; i < n; ++i) out[i] = pg[i];
    return (int)pg.size();
}
extern "C" int mlb_kv_alloc_free_pages(const mlb_kv_alloc* a) { return a ? (int)a->free_list.size() : fail(MLB_E_INVALID, "null allocator"); }
extern "C" void mlb_kv_alloc_release(mlb_kv_alloc* a, int seq) {
    if (!a || seq < 0 || seq >= (int)a->seq_pages.size()) return;
    for (int pg : a->seq_pages[seq]) a->free_list.push_back(pg);
    a->seq_pages[seq].clear();
}
extern "C" void mlb_kv_alloc_free(mlb_kv_alloc* a) { delete a; }

extern "C" const char* mlb_last_error(void) { return g_err.c_str(); }
extern "C" const char* mlb_version(void) { return "mini-llm-b200 0.1 (sm_100a)"; }
