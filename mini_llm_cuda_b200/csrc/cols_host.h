// Host entry points of the prompt-column kernels (defined in cols.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include <cuda.h>

#include "ring.cuh"

namespace mlb {

// The plan of one chunk of prompt columns, one int array on the device: header (active columns, runs, attention
// tiles), token / position / limit / sequence per column, then the runs and the tiles. A run is the consecutive
// columns of one sequence, a tile up to attn_cols_queries() of them.
struct ColsPlan {
    const int* hdr = nullptr;      // [4]
    const int* runs = nullptr;     // [max_runs][4]: first column, columns, sequence, position of the first
    const int* tiles = nullptr;    // [max_tiles][4]: the same for a tile
    int max_runs = 0, max_tiles = 0;
};

struct AttnColsParams {
    const bf16_t* kpool; const bf16_t* vpool;        // [page][kv_heads][16][hd]
    const int* page_table; int pt_stride;            // [sequence][pt_stride]
    const float* qbuf; const float* gbuf;            // [column][heads * hd]; gates may be null
    bf16_t* out16;                                   // [column][heads * hd]
    int heads, kv_heads;
    const int* hdr; const int4* tiles;
};
// Query columns of one attention tile for `group` query heads per kv head.
int attn_cols_queries(int group);
cudaError_t attn_cols_launch(int head_dim, int group, bool pdl, int max_tiles, cudaStream_t st, const AttnColsParams& p);

struct DeltaColsParams {
    const float* raw; int raw_stride;                // [column][q (H dk) | k (H dk) | v (H dv) | beta (H) | alpha (H)]
    float* state;                                    // [sequence][H][dv][dk]
    int H, dv;
    float* out; bf16_t* out16;                       // [column][H * dv], either may be null
    float l2_eps;
    const int* hdr; const int4* runs;
};
// Which form a chunk of `columns`, the longest run of `longest`, takes: `few` of delta_cols_launch.
bool delta_cols_serial(int sm_count, int H, int dv, int columns, int longest);
cudaError_t delta_cols_launch(int dk, bool few, bool pdl, int max_runs, cudaStream_t st, const DeltaColsParams& p);

// ---- embedding of a chunk ------------------------------------------------------------------------
struct EmbedColsParams {
    const void* E; const float* escale; int d;       // bf16, or e4m3 codes with row scales
    const StepLayer* layers; int n_layers, ple;      // per-layer embedding tables (bf16)
    const float* gain;                               // of the first layer's norm
    float* x; bf16_t* xg16; float* ssq; int parts;   // residual stream, its operand, sums of squares of 32 features each [column][parts]
    bf16_t* tple16;                                  // [layer][T][ple] rows of the later layers
    int T;
};
cudaError_t embed_cols_launch(bool w8, bool pdl, cudaStream_t st, const StepCtl& c, const EmbedColsParams& p);

// ---- projections of a chunk ----------------------------------------------------------------------
struct GemmColsParams;
struct QkvPostParams;
// Whether launches with `sums` may be made: as the library's compiler left the kernels. The others serve without.
cudaError_t gemm_cols_can_sum(bool* ok);
// `mode` a GemmTcMode; raises the kernel's shared-memory limit on first use.
cudaError_t gemm_cols_launch(int mode, int kv_dtype, bool sums, bool pair, bool pdl, int ctas, cudaStream_t st, const CUtensorMap& x, const CUtensorMap& w,
                             const CUtensorMap& w2, const CUtensorMap& xx, const CUtensorMap& wx, const GemmColsParams& p, const StepCtl& c,
                             const QkvPostParams& q);
// e4m3 codes -> the same values as bf16 (exact), n a multiple of 16
cudaError_t widen_e4m3_launch(const void* codes, bf16_t* out, size_t n, cudaStream_t st);

}  // namespace mlb
