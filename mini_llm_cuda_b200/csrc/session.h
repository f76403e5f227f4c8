// Model and session of the decode path, and what the host files share: the launch chains of one step (chain.cuh, one
// translation unit per weight type) and everything around them (engine.cu).
#pragma once
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/mlb.h"
#include "errors.h"
#include "step_shapes.h"
#include "attn_decode.cuh"
#include "gemm_tc.cuh"
#include "gemm_dec.cuh"
#include "tc_host.h"
#include "grid_params.h"
#include "lean_params.h"
#include "cols_host.h"

#define CU(expr)                                                                              \
    do {                                                                                      \
        cudaError_t e__ = (expr);                                                             \
        if (e__ != cudaSuccess)                                                               \
            return fail(MLB_E_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), __FILE__, __LINE__); \
    } while (0)

static size_t elt_size(int dt) { return dt == MLB_DT_F32 ? 4 : (dt == MLB_DT_BF16 ? 2 : 1); }
static int ple_dtype(int wdt) { return wdt == MLB_DT_FP8_E4M3 ? MLB_DT_BF16 : wdt; }

struct mlb_kv_alloc {
    std::vector<int> free_list;                 // stack; back() is handed out next
    std::vector<std::vector<int>> seq_pages;
    int max_pages_per_seq = 0;
    int num_pages = 0;
};

namespace mlb {
struct DevLayer {
    int type = MLB_LAYER_ATTENTION;
    float *g1 = nullptr, *g2 = nullptr, *gq = nullptr, *gk = nullptr;
    void* Wqkv = nullptr; float* Sqkv = nullptr; int n_qkv = 0;
    int nq = 0, nk = 0, nv = 0, ng = 0;
    void* Wo = nullptr; float* So = nullptr; int o_in = 0;
    void *W1a = nullptr, *W1b = nullptr, *W2 = nullptr;
    float *S1a = nullptr, *S1b = nullptr, *S2 = nullptr;
    void *pleT = nullptr, *pleP = nullptr;
};

}  // namespace mlb

struct mlb_model {
    mlb_config cfg;
    int device = 0;
    void* E = nullptr; float* Es = nullptr; float* g_final = nullptr; float* rope = nullptr;
    std::vector<mlb::DevLayer> layers;      // execution order
    uint64_t weight_bytes = 0;
    std::vector<void*> allocs;
    // FP8 models: the codes as bf16 (exact; the row scales stay separate), made when the first prompt is taken in by
    // columns and shared by all sessions. A chunk multiplies every weight tile with up to 32 column tiles: widening the
    // codes in the GEMM, once per tile and use, cost more than the MMA.
    struct Wide { void *Wqkv = nullptr, *Wo = nullptr, *W1a = nullptr, *W1b = nullptr, *W2 = nullptr; };
    std::vector<Wide> wide;
    void* wide_E = nullptr;
    std::mutex wide_mutex;
};

namespace mlb {
// widths of the column sets: 64, 128, ... 4096 (a chunk of a prompt takes the narrowest that holds it)
constexpr int kColMin = 64, kColSets = 7, kColMax = kColMin << (kColSets - 1);
constexpr int kPlanSlots = 4;
constexpr int kTcRefCols = 256;
enum ChainKind { CHAIN_PREFILL = 0, CHAIN_GREEDY = 1, CHAIN_TOPK = 2 };

struct LaunchRec {
    const char* name;
    uint64_t bytes, flops;
    cudaEvent_t e0, e1;
};
struct Recorder {
    cudaStream_t st;
    std::vector<LaunchRec> recs;
    int begin(const char* name, uint64_t bytes, uint64_t flops) {
        LaunchRec r{name, bytes, flops, nullptr, nullptr};
        CU(cudaEventCreate(&r.e0));
        CU(cudaEventCreate(&r.e1));
        CU(cudaEventRecord(r.e0, st));
        recs.push_back(r);
        return MLB_OK;
    }
    int end() {
        CU(cudaEventRecord(recs.back().e1, st));
        return MLB_OK;
    }
};
}  // namespace mlb

struct TcShape { int nb, split, stages, group; size_t smem; uint32_t tmem_cols; };
// launch shape of one projection of a column set (gemm_cols.cuh)
struct ColsGemm { int bn, stages, ctas, split, mains, exts, nbuf; uint32_t tmem_cols; bool sums, pair; int w_rows; };      // w_rows: of a CTA's weight tile, one matrix

struct mlb_session {
    mlb_model* m = nullptr;
    int B = 0, max_ctx = 0, max_pages = 0, kv_pages = 0;
    cudaStream_t stream = nullptr;
    int *pos = nullptr, *tok = nullptr, *limit_prefill = nullptr, *limit_decode = nullptr;
    int *prompt = nullptr, *out_ring = nullptr, *out_idx = nullptr, *page_table = nullptr;
    unsigned long long* seeds = nullptr;
    std::vector<unsigned long long> h_seeds;      // what `seeds` holds (empty: nothing yet)
    float *x = nullptr, *qbuf = nullptr, *gbuf = nullptr, *abuf = nullptr, *hbuf = nullptr, *raw = nullptr;
    float *logits = nullptr, *part = nullptr, *part_val = nullptr, *probe = nullptr;
    int *part_idx = nullptr, *attn_ticket = nullptr, *lm_ticket = nullptr;
    std::vector<void*> kpool, vpool;
    std::vector<float*> state;
    std::vector<void*> allocs;
    // host mirrors
    std::vector<int> h_pos;
    std::vector<char> h_stopped;            // the sequence drew the stop token: it takes no further step
    int stop_token = -1;
    std::vector<int> h_table;
    bool table_dirty = true;
    bool have_logits = false;
    mlb_kv_alloc alloc;
    int attn_min_pps = 11;                    // KV pages a flash-decode split must hold before a sequence uses it
    int splits = 1, lm_rows = 32, lm_parts = 1, raw_stride = 0, max_q = 0;
    // graphs
    cudaGraphExec_t graphs[3] = {nullptr, nullptr, nullptr};
    int g_topk = -1; float g_temp = 0.f;
    int cur_topk = 50; float cur_temp = 1.f;
    int launches_per_step[3] = {0, 0, 0};
    // one-token call as ONE graph: upload of the pending ids, the step, read-back of ids and error word
    cudaGraphExec_t tgraphs[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};     // [kind][with input ids]
    int tg_topk[2] = {-1, -1}; float tg_temp[2] = {0.f, 0.f};
    int* pinned_out = nullptr;
    int ctl_host_io = 0;                    // while the one-token graph is captured: 1 = ids and error word to the host, 2 = + ids from the host
    int tok_arg = -1;                       // single-kernel step: the pending id travels with the launch (>= 0), else it is read from `tok`
    float4* flush_buf = nullptr; size_t flush_n = 0;
    int* pinned_tok = nullptr;
    bool use_pdl = true;
    bool use_sgemv = false;                 // TMA-streamed GEMV for very small batches and large matrices
    bool force_sgemv = false;               // MLB_GEMV=stream: also for small matrices (tests)
    int sg_stage_kb = 48, sg_max_stages = 8; // ring geometry of the streamed GEMV (MLB_SG_STAGE_KB, MLB_SG_STAGES)
    int sm_count = 148;
    mlb::StepLayer* step_layers = nullptr;   // device table of per-layer pointers (single-kernel step)
    int* dev_err = nullptr;                 // set by a kernel whose bounded wait ran out
    // whole-GPU single-kernel step (batch 1)
    bool use_grid = false;
    int grid_ctas = 0;
    size_t grid_smem = 0;
    mlb::GridParams grid;
    // the same step with compile-time shapes, for the models it is built for
    bool use_lean = false;
    int lean_idx = -1;
    size_t lean_smem = 0;
    mlb::LeanParams lean;
    // tensor-core projections (bf16 or FP8 weights, batch >= 4)
    bool use_tc = false;
    bool use_dec = false;                     // the step's projections on mma.sync tiles (gemm_dec.cuh) instead of tcgen05 ones
    int tc_nb = 0, tc_stages = 0, tc_stages_swiglu = 0;
    int tc_max_split = 8;                     // largest cluster that may split a GEMM's k-blocks
    bool tc_split_forced = false;             // MLB_TC_SPLIT given: take it as the limit without the k-blocks-per-CTA rule
    int tc_cluster_cap[4] = {0, 0, 0, 0};     // clusters of 1, 2, 4, 8 GEMM CTAs that can be resident at once
    unsigned long long* tc_trace = nullptr;   // MLB_TC_TRACE=1: [64][8] timer stamps of the step's GEMM launches
    int tc_trace_n = 0;
    TcShape tc_shape_down{};                  // launch shape of the down projection (its per-layer embedding map has this batch tile)
    mlb::bf16_t *xn16 = nullptr, *a16 = nullptr, *h16 = nullptr;
    float* rawq = nullptr;
    struct alignas(64) TcLayerMaps { CUtensorMap qkv, o, w1a, w1b, w2, pleP, pleT; };   // pleP / pleT: [d][ple] projection, gathered [B][ple] rows
    float* tc_ssq = nullptr;                 // [B][ceil(d / 128)] partial sums of squares of the residual stream
    mlb::bf16_t* tple16 = nullptr;           // [layers][B][ple] per-layer embedding rows of the step's tokens
    std::vector<TcLayerMaps> tc_maps;
    // activation operand maps per batch tile 16, 32, 64, 128, 256 (index log2(Nb/16))
    // (decode GEMMs of gemm_dec.cuh: per tile of 16, 32, 64 sequences and 1, 2, 4 k-blocks, index gd_index)
    struct alignas(64) TcGlobalMaps { CUtensorMap E, xn[9], a_attn[9], a_dn[9], h[9]; } tc_g;
    int* pinned_err = nullptr;
    // prompt columns: further sets of step buffers, `B` columns wide, that share this session's KV pool, page table,
    // delta-net state and stream; a column is one prompt token of one sequence. A set per power of two of columns,
    // made when first needed.
    mlb_session* cols[mlb::kColSets] = {};  // owned by the session they serve
    size_t cols_bytes = 0, own_bytes = 0;   // device memory of the column sets; in a column set, its own
    bool cols_failed = false;               // they cannot be had here, for another reason than memory
    mlb_session* cols_gemv = nullptr;       // column set of kColMin columns on the GEMV chain, for short prompts of bf16 / FP8 models
    mlb_session* parent = nullptr;          // set in a column set
    int* seq_of = nullptr;                  // [B] in a column set: column -> sequence of the parent
    bool use_cols = false;                  // column set: persistent column GEMMs (else, without the bf16 codes, run_tc)
    bool as_steps = false;                  // column set: on the decode step's kernels throughout (MLB_GEMM=tcgen05)
    bool no_copy = false;                   // column set of an FP8 model that was made without them
    ColsGemm cg_qkv{}, cg_dn{}, cg_o_attn{}, cg_o_dn{}, cg_up{}, cg_down{}, cg_last{}, cg_head{};      // cg_last: the last layer's down projection
    bool few_runs = false;                  // column set: form of the delta-net recurrence in `graphs`; the other form's are other_graphs
    cudaGraphExec_t other_graphs[3] = {nullptr, nullptr, nullptr};
    mlb::ColsPlan plan;                     // column set: what the columns of the current chunk are (one array, plan_dev)
    int* plan_dev = nullptr;
    int* plan_host = nullptr;               // session: pinned ring of kPlanSlots plans of the widest set
    size_t plan_host_ints = 0;              // ints per slot
    cudaEvent_t plan_free[mlb::kPlanSlots] = {};   // the copy out of a slot is done
};

namespace mlb {

// Host mirror of seq_active for the decode chains.
static bool seq_live(const mlb_session* s, int b) { return s->h_pos[b] < s->max_ctx && !s->h_stopped[b]; }

static StepCtl make_ctl(mlb_session* s, int kind) {
    StepCtl c{};
    c.B = s->B;
    c.seq_of = s->seq_of;
    c.n_cols = s->plan.hdr;
    c.vocab = s->m->cfg.vocab;
    c.pos = s->pos;
    c.tok = s->tok;
    c.limit = kind == CHAIN_PREFILL ? s->limit_prefill : s->limit_decode;
    c.stop_token = kind == CHAIN_PREFILL ? -1 : s->stop_token;
    c.prompt = kind == CHAIN_PREFILL ? s->prompt : nullptr;
    c.prompt_stride = s->max_ctx;
    c.out_ring = s->out_ring;
    c.out_idx = s->out_idx;
    c.out_cap = s->parent ? 0 : s->max_ctx;     // a column set has no output ring
    c.tok_src = s->ctl_host_io == 2 ? s->pinned_tok : nullptr;
    c.host_out = s->ctl_host_io ? s->pinned_out : nullptr;
    c.host_err = s->ctl_host_io ? s->pinned_err : nullptr;
    c.dev_err = s->dev_err;
    return c;
}

// Shape of one tensor-core GEMM launch: batch tile (UMMA N), how many CTAs of a cluster split the k-blocks of
// an output tile, and the ring. Measured on B200: a tcgen05.mma of M = 128 costs about 0.1 us whatever its N
// (16..128), so a CTA's k-loop takes 0.4 us per 64-wide k-block (0.8 with two weight tiles) whatever the ring
// depth, and is the time of the kernel unless the k-blocks are spread over CTAs. Exchanging partial
// accumulators through distributed shared memory costs 2-3 us per launch with clusters of 4 and 8, more than
// it saves at cfg1's sizes (8-23 k-blocks per tile); pairs pay off at small batches (cfg1 step at 32 sequences:
// 452 -> 424 us) and are neutral at 256. Larger clusters are taken only where a CTA keeps 8 k-blocks or more
// (cfg4: 32-90 k-blocks per tile and few tiles). MLB_TC_SPLIT sets the limit by hand. One wave of CTAs per
// launch where possible.
static TcShape tc_pick_shape(const mlb_session* s, int B, int N, int nkb_all, int na, bool w8, int nacc) {
    const int tiles_m = (N + kTcM - 1) / kTcM;
    const int cap = std::min(256, (B + 15) / 16 * 16);
    TcShape best{};
    double best_cost = -1.0;
    for (int nb = 16; nb <= cap && nacc * nb <= 512; nb <<= 1) {
        for (int li = 0; li < 4; ++li) {
            const int S = 1 << li;
            if (S > s->tc_max_split || S > nkb_all) break;
            // clusters of 4 and 8 only where a CTA keeps 8 k-blocks or more: their exchange costs 2-3 us
            if (S > 2 && !s->tc_split_forced && (nkb_all + S - 1) / S < 8) break;
            if (S > 1 && (nb % S != 0 || s->tc_cluster_cap[li] <= 0)) continue;
            const size_t stage_bytes = (size_t)na * kTcM * 128 + (size_t)nb * 128;      // FP8 codes land inside the operand tile
            const int kpc = (nkb_all + S - 1) / S;
            int st = (int)std::max<size_t>(1, std::min<size_t>(std::min(kpc, 12), kTcRingBytes / stage_bytes));
            const int g = st >= kpc ? 1 : (st >= 8 ? 4 : (st >= 4 ? 2 : 1));
            st -= st % g;
            const size_t body = std::max((size_t)st * stage_bytes, S > 1 ? (size_t)nacc * nb * kTcM * 4 : (size_t)0);
            const size_t smem = 1024 + kTcHeadBytes + kTcStageBytes + body;
            if (smem > 227 * 1024) continue;
            const long ctas = (long)tiles_m * ((B + nb - 1) / nb) * S;
            const long resident = S == 1 ? s->sm_count : (long)s->tc_cluster_cap[li] * S;
            const long waves = (ctas + resident - 1) / resident;
            const double t_loop = 0.4 * na * kpc;
            const double t_red = S > 2 ? 2.5 + (double)nacc * nb * 512.0 / 65536.0 : (S > 1 ? 0.5 + (double)nacc * nb * 512.0 / 65536.0 : 0.0);
            const double t_epi = 0.25 * ((nb / S + 15) / 16);
            const double cost = (double)waves * (t_loop + t_red + t_epi + 0.5);
            if (best_cost < 0 || cost < best_cost) {
                best_cost = cost;
                uint32_t cols = 32;
                while (cols < (uint32_t)(nacc * nb)) cols <<= 1;
                best = TcShape{nb, S, st, g, smem, cols};
            }
        }
    }
    return best;
}
// Launch shape of a decode GEMM (gemm_dec.cuh).
struct GdShape { int np, split, g, stages, w_bytes; size_t smem; };
static int gd_index(int np, int g) { return (np >> 1) * 3 + (g >> 1); }       // np, g in {1, 2, 4}
// mma.sync multiplies at about 512 a cycle and SM here (k-loop times against sequences per CTA), tcgen05 eight times as fast, so what
// gemm_dec_kernel saves around the products it pays back in them once they are many. Measured per step, tcgen05 -> mma.sync: cfg1 372
// -> 195 us at 4 sequences, 534 -> 455 at 256; cfg4 (gate/up 2 x 5632 x 2048) 2338 -> 1677 at 4, 3112 -> 2760 at 48 (7.5 M products
// per SM in the gate/up projection, the largest), 2735 -> 2739 and behind long prompts 3385 -> 3440 at 64 (10 M). The line lies between.
constexpr long kGdMostProducts = 8L << 20;
static bool gd_small_enough(const mlb_session* s) {
    return s->B <= 256 && 2L * s->m->cfg.ffn_dim * s->m->cfg.dim * s->B / s->sm_count <= kGdMostProducts;
}
// The k-ranges are those of the tcgen05 launch of the same batch (the results are the same bits). Sequences per CTA: the most
// that still leaves 96 CTAs, two thirds of the SMs - fewer CTAs read the activations less often, more of them share the epilogue.
static GdShape gd_pick(const mlb_session* s, int N, int nkb, int mode, bool w8, bool ext) {
    GdShape g;
    const int na = mode == TC_SWIGLU ? 2 : 1;
    const bool ext2 = w8 && mode == TC_RESID;
    g.split = std::max(1, tc_pick_shape(s, s->B, N, nkb, na, w8, na == 2 || ext2 ? 2 : 1).split);
    g.np = 4;
    while (g.np > 1 && (16 * (g.np / 2) >= s->B || (long)((N + kGdF - 1) / kGdF) * ((s->B + 16 * g.np - 1) / (16 * g.np)) < 96)) g.np >>= 1;
    g.w_bytes = kGdF * (w8 && !ext ? 64 : 128);
    const int ct = 16 * g.np;
    const long ctas = (long)((N + kGdF - 1) / kGdF) * ((s->B + 16 * g.np - 1) / (16 * g.np));
    const size_t block = (size_t)g.split * (na * g.w_bytes + ct * 128);      // a stage of one k-block per copy
    const size_t ring = gd_ring(kGdRing, ctas, s->sm_count, mode == TC_SWIGLU, block * std::min(2, (nkb + g.split - 1) / g.split + (ext ? 1 : 0)));
    // k-blocks per copy: as many as leave two stages
    size_t stage = 0;
    int n_iter = 1;
    for (g.g = 4;; g.g >>= 1) {
        stage = block * g.g;
        n_iter = ((nkb + g.split - 1) / g.split + g.g - 1) / g.g + (ext ? 1 : 0);
        if (g.g == 1 || stage * std::min(2, n_iter) <= ring) break;
    }
    g.stages = (int)std::max<size_t>(1, std::min<size_t>(std::min(n_iter, kGdMaxStages), ring / stage));
    const size_t part = (size_t)g.split * (ext2 ? 2 : 1) * ct * (32 * na + 4) * 4;
    g.smem = 1024 + std::max((size_t)g.stages * stage, part);
    return g;
}
static int nb_index(int nb) { return nb == 16 ? 0 : nb == 32 ? 1 : nb == 64 ? 2 : nb == 128 ? 3 : 4; }

// delta-net recurrence of layer i over the columns of a column set
static inline cudaError_t delta_cols(const mlb_session* s, int i, float* out, bf16_t* out16) {
    const mlb_config& cfg = s->m->cfg;
    DeltaColsParams dc;
    dc.raw = s->raw; dc.raw_stride = s->raw_stride; dc.state = s->state[i]; dc.H = cfg.heads; dc.dv = cfg.dn_value_dim;
    dc.out = out; dc.out16 = out16; dc.l2_eps = 1e-6f;
    dc.hdr = s->plan.hdr; dc.runs = reinterpret_cast<const int4*>(s->plan.runs);
    return delta_cols_launch(cfg.dn_key_dim, s->few_runs, s->use_pdl, s->plan.max_runs, s->stream, dc);
}

// ---- the launch chains (chain_f32.cu, chain_bf16.cu, chain_fp8.cu) ------------------------------------
int chain_run_f32(mlb_session* s, int kind, Recorder* rec, int* n_launches);
int chain_run_bf16(mlb_session* s, int kind, Recorder* rec, int* n_launches);
int chain_run_fp8(mlb_session* s, int kind, Recorder* rec, int* n_launches);
// shared-memory limits of the chain's GEMV kernels
int chain_configure_f32(mlb_session* s);
int chain_configure_bf16(mlb_session* s);
int chain_configure_fp8(mlb_session* s);
// shared-memory limits of the tensor-core GEMMs
int tc_allow_big_smem_bf16(int kv_dtype);
int tc_allow_big_smem_fp8(int kv_dtype);
// clusters of `size` GEMM CTAs with `smem` bytes each that can be resident at once
int tc_max_clusters(int size, size_t smem, int* n);
// flash-decode attention over an fp32 K/V cache, one launch
int chain_attn_f32kv(mlb_session* s, const StepCtl& c, const AttnParams& a);

}  // namespace mlb
