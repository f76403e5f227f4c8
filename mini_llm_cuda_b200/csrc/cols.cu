// Kernels that only a prompt taken in by columns needs: causal attention of many columns of a sequence over its
// paged K/V rows, and the gated delta-net recurrence over a sequence's columns. Everything else of a column step is
// the decode step's own kernels with a column in the place of a sequence.
#include <cstring>
#include <type_traits>

#include "cols_host.h"
#include "cols_math.h"
#include "../../include/mlb.h"
#include "gemm_cols.cuh"

namespace mlb {

template <typename... KArgs>
static cudaError_t launch_pdl_cluster(bool pdl, int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, KArgs... args) {
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename... KArgs>
static cudaError_t launch_pdl(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, KArgs... args) {
    return launch_pdl_cluster(pdl, 1, kernel, grid, block, smem, st, args...);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------------
// Causal attention of prompt columns (inference.cu:510-579 for a block of query columns), with the results of
// attn_decode_kernel to the last bit: the model rounds its activations to bf16 behind every layer, and a sum taken in
// another order ends, some layers later, in other roundings and now and then in another token.
//
// That kernel keeps, per query and head, one running softmax per warp and lane group: stream (w, grp) takes the pages
// w, w + 4, .. and in them the positions of its lane group, four at a time; a score is the sum over HD / 8 lanes of
// eight-element products. Here a CTA takes 32 rows = 32 / G consecutive query columns times the G heads of a kv head, so that
// a K/V row comes from L2 once for 32 rows (once per row before: 9 GB a layer for a 3000-token prompt). A warp
// works on one stream of its rows: four rows and 16 dims (lanes a and a + HD / 16 of the other kernel) per thread as packed
// fp32 pairs, K/V read as bf16 and unpacked once for four rows. The partial scores of the four rows are summed by a butterfly
// that leaves each lane one row, whose exponentials it takes alone and hands to the others. Half of the streams are
// live at a time: the pages of w = 0, 1 first, then those of w = 2, 3.
// What bounds it: 11 instructions per warp, row and position share of 64 under two warps a scheduler (IPC 2.2 an SM, FMA pipe half busy;
// 64 q and 64 accumulator registers a thread leave room for no more warps), not its FMAs (1 and 2 cycles per SM, row and position at
// HD = 64 and 128): 3001 tokens of 16 heads of 128 take 1290 us a layer, 5.2 cycles (1351 with the chunks of a page one after the other and
// a division per score). At HD = 64 a page is one chunk; two pages at once wasted more on odd numbers of pages (256 x 256 tokens of 8
// heads: 185 -> 212 us a launch of 16 columns each).
// ------------------------------------------------------------------------------------------------
constexpr int kAcRows = 32;      // (query, head) rows per CTA
constexpr int kAcThreads = 256;
constexpr int kAcPages = 4;      // pages of a K/V tile: two for each of the two w of a pass

// (a model without attention layers may state any number of heads per kv head)
int attn_cols_queries(int group) { return group <= kAcRows ? kAcRows / group : 1; }

template <int HD>
constexpr size_t attn_cols_smem() {
    constexpr size_t tiles = 2 * 2 * (size_t)kAcPages * kKvBlock * HD * 2;                   // stages, K and V
    constexpr size_t streams = (size_t)(HD == 64 ? 8 : 4) * kAcRows * (HD + 2) * 4;
    return (tiles > streams ? tiles : streams) + (size_t)4 * kAcRows * (HD + 2) * 4 + (size_t)2 * kAcRows * 8 * 4;
}

template <int HD, int G>
__global__ void __launch_bounds__(kAcThreads, 1) attn_cols_kernel(AttnColsParams p) {
    constexpr int L = HD / 16;                      // lanes that share a group of four rows
    constexpr int NG = HD == 64 ? 4 : 2;            // lane groups (positions per warp iteration) of attn_decode_kernel
    constexpr int CPP = 4 / NG;                     // chunks of 4 positions per page and stream
    constexpr int NS = 2 * NG;                      // streams of a pass
    constexpr int W = HD + 2;
    constexpr int TILE = kAcPages * kKvBlock * HD * 2;      // bytes of a K or V tile
    extern __shared__ __align__(128) unsigned char sm[];
    constexpr size_t area = (size_t)4 * TILE > (size_t)NS * kAcRows * W * 4 ? (size_t)4 * TILE : (size_t)NS * kAcRows * W * 4;
    float* sred = reinterpret_cast<float*>(sm);                       // [NS][32][HD + 2] of a pass, over the tiles
    float* wred = reinterpret_cast<float*>(sm + area);                // [4][32][HD + 2]
    float* fac = wred + 4 * kAcRows * W;                              // [2][32][8] factors of the merges
    pdl_launch_dependents();
    const int n_tiles = p.hdr[2];                   // the plan is in place before the step's first kernel starts
    if ((int)blockIdx.x >= n_tiles) return;
    const int4 tl = p.tiles[n_tiles - 1 - (int)blockIdx.x];     // later positions (more K/V rows) first
    const int col0 = tl.x, nq = tl.y, pos0 = tl.w;
    const int kvh = blockIdx.y;
    const int last = pos0 + nq - 1, np = last / kKvBlock + 1;
    const int* pt = p.page_table + (size_t)tl.z * p.pt_stride;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int a = lane % L;
    const int stream = HD == 64 ? warp : warp >> 1, wl = stream / NG, grp = stream % NG;
    const int rbase = (HD == 64 ? 0 : (warp & 1) * 16) + lane / L * 4;          // this thread's rows: rbase .. rbase + 3
    const int own = HD == 64 ? a : a >> 1;                                      // the row of them whose softmax it keeps
    const int own_pos = pos0 + min((rbase + own) / G, nq - 1);
    const int warp_first = pos0 + min((HD == 64 ? 0 : (warp & 1) * 16) / G, nq - 1);
    const int warp_last = pos0 + min(((HD == 64 ? 0 : (warp & 1) * 16) + (HD == 64 ? 31 : 15)) / G, nq - 1);
    const uint32_t sm0 = smem_u32(sm);
    auto load = [&](int pass, int t, int st) {
#pragma unroll
        for (int i = 0; i < kAcPages * kKvBlock * (HD / 8) / kAcThreads; ++i) {
            const int idx = tid + i * kAcThreads, row = idx / (HD / 8), ch = idx % (HD / 8);
            const int sl = row / kKvBlock;           // slot: w_local * 2 + k
            const int pg = 2 * pass + (sl >> 1) + 4 * (2 * t + (sl & 1));
            const bool ok = pg < np && pg * kKvBlock + row % kKvBlock <= last;      // rows behind the tile's last position read as zeros
            const int page = ok ? pt[pg] : 0;
            const size_t off = (((size_t)page * p.kv_heads + kvh) * kKvBlock + (row % kKvBlock)) * HD + ch * 8;
            cp_async16(sm0 + (uint32_t)(st * 2 * TILE + row * HD * 2 + ch * 16), p.kpool + off, ok);
            cp_async16(sm0 + (uint32_t)(st * 2 * TILE + TILE + row * HD * 2 + ch * 16), p.vpool + off, ok);
        }
        cp_async_commit();
    };
    // eight pairs of one K or V row: element e of the other kernel's lanes a and a + L
    auto unpack = [&](const unsigned char* rowp, f32x2* o) {
        const uint4 x = *reinterpret_cast<const uint4*>(rowp + a * 16), y = *reinterpret_cast<const uint4*>(rowp + (a + L) * 16);
        o[0] = pack2u(x.x << 16, y.x << 16); o[1] = pack2u(x.x & 0xffff0000u, y.x & 0xffff0000u);
        o[2] = pack2u(x.y << 16, y.y << 16); o[3] = pack2u(x.y & 0xffff0000u, y.y & 0xffff0000u);
        o[4] = pack2u(x.z << 16, y.z << 16); o[5] = pack2u(x.z & 0xffff0000u, y.z & 0xffff0000u);
        o[6] = pack2u(x.w << 16, y.w << 16); o[7] = pack2u(x.w & 0xffff0000u, y.w & 0xffff0000u);
    };
    pdl_wait();                                     // q and this chunk's K/V rows come from the projection kernel
    load(0, 0, 0);
    f32x2 q[4][8];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int qi = min((rbase + r) / G, nq - 1), h = kvh * G + (rbase + r) % G;
        const float4* qp = reinterpret_cast<const float4*>(p.qbuf + ((size_t)(col0 + qi) * p.heads + h) * HD);
        const float4 x0 = __ldcg(qp + 2 * a), x1 = __ldcg(qp + 2 * a + 1), y0 = __ldcg(qp + 2 * (a + L)), y1 = __ldcg(qp + 2 * (a + L) + 1);
        q[r][0] = pack2(x0.x, y0.x); q[r][1] = pack2(x0.y, y0.y); q[r][2] = pack2(x0.z, y0.z); q[r][3] = pack2(x0.w, y0.w);
        q[r][4] = pack2(x1.x, y1.x); q[r][5] = pack2(x1.y, y1.y); q[r][6] = pack2(x1.z, y1.z); q[r][7] = pack2(x1.w, y1.w);
    }
    auto scaled = [](float x) { return HD == 64 ? x * 0.125f : over_sqrt128(x); };      // x / sqrtf(HD)
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const int n_t = np > 2 * pass ? ((np - 2 * pass + 3) / 4 + 1) / 2 : 0;         // tiles: of the pass's first w, which has the most pages
        f32x2 acc[4][8];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[r][e] = 0ull;
        float m = kNegBig, l = 0.f;
        if (pass == 1 && n_t > 0) load(1, 0, 0);
        // One page of the warp's stream: one or two chunks of four positions. The products, butterflies and exponentials of two chunks
        // depend on one another only by the running maximum and fill one another's waits. `later`: the page may hold positions behind some
        // row of the warp. Their probability is 0, but 0 times a value that is no number is none: their products are left out.
        auto use_page = [&](auto later, const unsigned char* kt, const unsigned char* vt, int cnt) {
            auto row_of = [&](int c, int u) { return (c * 4 + u) * NG + grp; };
            auto valid = [&](int c, int u) { return !decltype(later)::value || row_of(c, u) < cnt; };
            float s[CPP][16];                     // [chunk][row][u]
#pragma unroll
            for (int c = 0; c < CPP; ++c)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    f32x2 kp[8];
                    unpack(kt + row_of(c, u) * HD * 2, kp);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        f32x2 d = 0ull;
#pragma unroll
                        for (int e = 0; e < 8; ++e) d = fma2(q[r][e], kp[e], d);
                        float x, y;
                        unpack2(d, x, y);
                        s[c][r * 4 + u] = x + y;
                    }
                }
            const bool up1 = (a & (L / 2)) != 0, up2 = (a & (L / 4)) != 0;
#pragma unroll
            for (int c = 0; c < CPP; ++c)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float send = up1 ? s[c][j] : s[c][j + 8], keep = up1 ? s[c][j + 8] : s[c][j];
                    s[c][j] = keep + __shfl_xor_sync(0xffffffffu, send, L / 2);
                }
#pragma unroll
            for (int c = 0; c < CPP; ++c)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float send = up2 ? s[c][j] : s[c][j + 4], keep = up2 ? s[c][j + 4] : s[c][j];
                    s[c][j] = keep + __shfl_xor_sync(0xffffffffu, send, L / 4);
                }
            if (HD == 128) {
#pragma unroll
                for (int c = 0; c < CPP; ++c)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[c][j] += __shfl_xor_sync(0xffffffffu, s[c][j], 1);
            }
            // softmax of the own row
            float sc[CPP];
#pragma unroll
            for (int c = 0; c < CPP; ++c) {
                float mn = m;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    s[c][u] = valid(c, u) ? scaled(s[c][u]) : kNegBig;
                    mn = fmaxf(mn, s[c][u]);
                }
                sc[c] = expf(m - mn);
#pragma unroll
                for (int u = 0; u < 4; ++u) s[c][u] = valid(c, u) ? expf(s[c][u] - mn) : 0.f;
                l = __fadd_rn(__fmul_rn(l, sc[c]), s[c][0]);         // (not one fma: the other kernel's roundings)
                l = __fadd_rn(__fadd_rn(__fadd_rn(l, s[c][1]), s[c][2]), s[c][3]);
                m = mn;
            }
            const int src = lane - a;
            const bool moved = __any_sync(0xffffffffu, sc[0] != 1.0f || sc[CPP - 1] != 1.0f);
#pragma unroll
            for (int c = 0; c < CPP; ++c) {
                if (moved) {
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float x = __shfl_sync(0xffffffffu, sc[c], src + (HD == 64 ? r : 2 * r));
                        const f32x2 xx = pack2(x, x);
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[r][e] = mul2(acc[r][e], xx);
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    f32x2 vp[8];
                    unpack(vt + row_of(c, u) * HD * 2, vp);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float x = __shfl_sync(0xffffffffu, s[c][u], src + (HD == 64 ? r : 2 * r));
                        if (decltype(later)::value && x == 0.f) continue;
                        const f32x2 xx = pack2(x, x);
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[r][e] = fma2(xx, vp[e], acc[r][e]);
                    }
                }
            }
        };
#pragma unroll 1
        for (int t = 0; t < n_t; ++t) {
            const int st = t & 1;
            if (t + 1 < n_t) {
                load(pass, t + 1, st ^ 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
#pragma unroll 1
            for (int k = 0; k < 2; ++k) {
                const int pg = 2 * pass + wl + 4 * (2 * t + k);
                if (pg * kKvBlock > warp_last) break;        // behind every row of the warp: the other kernel does not visit it
                const unsigned char* kt = sm + st * 2 * TILE + (wl * 2 + k) * kKvBlock * HD * 2;
                const unsigned char* vt = kt + TILE;
                const int cnt = own_pos + 1 - pg * kKvBlock;
                if (pg * kKvBlock + kKvBlock - 1 > warp_first) use_page(std::true_type(), kt, vt, cnt);
                else use_page(std::false_type(), kt, vt, cnt);
            }
            __syncthreads();                         // the stage is refilled in the next round
        }
        // the pass's streams -> shared memory, merged over the lane groups in the other kernel's order
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float* d = sred + ((size_t)stream * kAcRows + rbase + r) * W;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float x, y;
                unpack2(acc[r][e], x, y);
                d[a * 8 + e] = x;
                d[(a + L) * 8 + e] = y;
            }
        }
        if (HD == 64 || !(a & 1)) {
            float* d = sred + ((size_t)stream * kAcRows + rbase + own) * W;
            d[HD] = m;
            d[HD + 1] = l;
        }
        __syncthreads();
        if (tid < 2 * kAcRows) {
            const int w = tid / kAcRows, row = tid % kAcRows;
            const float* g0 = sred + ((size_t)(w * NG) * kAcRows + row) * W;
            constexpr int GS = kAcRows * W;          // from one group's results to the next
            float* f = fac + tid * 8;
            auto merge = [](float m0, float l0, float m1, float l1, float& mo, float& lo, float& sa, float& sb) {
                const float mn = fmaxf(m0, m1);
                sa = expf(m0 - mn);
                sb = expf(m1 - mn);
                lo = fmaf(l0, sa, __fmul_rn(l1, sb));
                mo = mn;
            };
            float mr, lr;
            merge(g0[HD], g0[HD + 1], g0[GS + HD], g0[GS + HD + 1], mr, lr, f[0], f[1]);
            if (NG == 4) {
                float m2, l2, mo, lo;
                merge(g0[2 * GS + HD], g0[2 * GS + HD + 1], g0[3 * GS + HD], g0[3 * GS + HD + 1], m2, l2, f[2], f[3]);
                merge(mr, lr, m2, l2, mo, lo, f[4], f[5]);
                mr = mo;
                lr = lo;
            }
            float* d = wred + ((size_t)(2 * pass + w) * kAcRows + row) * W;
            d[HD] = mr;
            d[HD + 1] = lr;
        }
        __syncthreads();
        for (int i = tid; i < 2 * kAcRows * HD; i += kAcThreads) {
            const int wr = i / HD, e = i % HD, w = wr / kAcRows, row = wr % kAcRows;
            const float* g0 = sred + ((size_t)(w * NG) * kAcRows + row) * W + e;
            constexpr int GS = kAcRows * W;
            const float* f = fac + wr * 8;
            float x = fmaf(g0[0], f[0], __fmul_rn(g0[GS], f[1]));
            if (NG == 4) {
                const float y = fmaf(g0[2 * GS], f[2], __fmul_rn(g0[3 * GS], f[3]));
                x = fmaf(x, f[4], __fmul_rn(y, f[5]));
            }
            wred[((size_t)(2 * pass + w) * kAcRows + row) * W + e] = x;
        }
        __syncthreads();
    }
    // merge over the four w
    if (tid < kAcRows) {
        float mn = kNegBig, lt = 0.f;
        float* f = fac + tid * 8;
#pragma unroll
        for (int w = 0; w < 4; ++w) mn = fmaxf(mn, wred[((size_t)w * kAcRows + tid) * W + HD]);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float sc = expf(wred[((size_t)w * kAcRows + tid) * W + HD] - mn);
            lt = fmaf(wred[((size_t)w * kAcRows + tid) * W + HD + 1], sc, lt);
            f[w] = sc;
        }
        f[4] = lt;
    }
    __syncthreads();
    for (int i = tid; i < kAcRows * HD / 2; i += kAcThreads) {
        const int row = i / (HD / 2), e = (i % (HD / 2)) * 2, qi = row / G;
        if (qi >= nq) continue;
        const float* f = fac + row * 8;
        float o[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float at = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) at = fmaf(wred[((size_t)w * kAcRows + row) * W + e + j], f[w], at);
            o[j] = at / f[4];
        }
        const size_t at = ((size_t)(col0 + qi) * p.heads + kvh * G + row % G) * HD + e;
        if (p.gbuf) {
            o[0] *= p.gbuf[at];
            o[1] *= p.gbuf[at + 1];
        }
        const __nv_bfloat162 v = __floats2bfloat162_rn(o[0], o[1]);
        *reinterpret_cast<__nv_bfloat162*>(p.out16 + at) = v;
    }
}

template <int HD, int G>
static cudaError_t attn_cols_one(bool pdl, int max_tiles, cudaStream_t st, const AttnColsParams& p) {
    constexpr size_t smem = attn_cols_smem<HD>();
    cudaError_t e = cudaFuncSetAttribute(attn_cols_kernel<HD, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(pdl, attn_cols_kernel<HD, G>, dim3(max_tiles, p.kv_heads), dim3(kAcThreads), smem, st, p);
}

cudaError_t attn_cols_launch(int head_dim, int group, bool pdl, int max_tiles, cudaStream_t st, const AttnColsParams& p) {
    if (head_dim == 64) {
        switch (group) {
            case 1: return attn_cols_one<64, 1>(pdl, max_tiles, st, p);
            case 2: return attn_cols_one<64, 2>(pdl, max_tiles, st, p);
            case 4: return attn_cols_one<64, 4>(pdl, max_tiles, st, p);
            default: return attn_cols_one<64, 8>(pdl, max_tiles, st, p);
        }
    }
    switch (group) {
        case 1: return attn_cols_one<128, 1>(pdl, max_tiles, st, p);
        case 2: return attn_cols_one<128, 2>(pdl, max_tiles, st, p);
        case 4: return attn_cols_one<128, 4>(pdl, max_tiles, st, p);
        default: return attn_cols_one<128, 8>(pdl, max_tiles, st, p);
    }
}

// ------------------------------------------------------------------------------------------------
// Gated delta-net recurrence over the columns of a sequence (no counterpart in the reference): delta_net_kernel's update
//   S <- alpha S,  u = beta (v - S k^),  S <- S + u k^^T,  o = S q^
// walked in order, with that kernel's results to the last bit (see attn_cols_kernel).
//
// It is a serial chain along the columns: at small batch its time is the latency of a column times their number, at
// large batch the instructions. There a warp had a row per instruction and 10 shuffles per row and column. Here eight lanes
// share R rows; a lane holds the elements of four of that kernel's lanes (a, a + 8, a + 16, a + 24), as packed pairs, so
// that the first two steps of a row's 32-lane sum are its own additions and three shuffle steps are left, on values halved from
// step to step; k^ and q^ of a column are read from shared memory once for R rows, as the pairs that the products take. The inputs of 16
// columns at a time come through a cp.async ring and are L2-normalised there, by the walking warps or (R = 1) by others. R = 4 where the
// chunk's runs fill the SMs (fewest instructions per row), else R = 1 (a quarter of the rows, and of the instructions in the chain, per
// warp): delta_cols_serial. Per launch, before the pairs, the output sums under the next column and the preparing warps -> with them: one run of
// 3001 columns, 16 heads of 128 2059 -> 1038 us; 64 runs of 64 columns 363 -> 312, 8 heads of 128 187 -> 164; 128 of 32, 8 heads of 64 54 -> 48.
// ------------------------------------------------------------------------------------------------
constexpr int kDcCols = 16;       // columns per ring stage
constexpr int dc_stages(int rows) { return rows == 1 ? 4 : 3; }
// One row per lane group: four more warps copy and normalise the inputs of the next columns under the walk of these, which is then only the
// recurrence (3001 columns of 16 heads of 128: 1717 -> 1038 us). Where runs fill the SMs other CTAs' walks do that, and the walking warps prepare.
constexpr int dc_threads(int rows) { return 32 * 4 * (rows == 1 ? 2 : 1); }
constexpr int kDcWarps = 4;
constexpr int kDcThreads = 32 * kDcWarps;

template <int DK, int R>
struct DeltaStage {
    float q[kDcCols][DK], k[kDcCols][DK], v[kDcCols][4 * R * kDcWarps];
    float beta[kDcCols], alpha[kDcCols];
};

// this lane's part of a vector of DK floats: element e of lanes a, a + 8 and of a + 16, a + 24 as pairs
template <int DK>
__device__ __forceinline__ void delta_pairs(const float* v, int a, f32x2 (&lo)[DK / 32], f32x2 (&hi)[DK / 32]) {
    if (DK == 128) {
        const float4* p = reinterpret_cast<const float4*>(v);
        const float4 x = p[a], y = p[a + 8], z = p[a + 16], w = p[a + 24];
        lo[0] = pack2(x.x, y.x); lo[1] = pack2(x.y, y.y); lo[2 % (DK / 32)] = pack2(x.z, y.z); lo[3 % (DK / 32)] = pack2(x.w, y.w);
        hi[0] = pack2(z.x, w.x); hi[1] = pack2(z.y, w.y); hi[2 % (DK / 32)] = pack2(z.z, w.z); hi[3 % (DK / 32)] = pack2(z.w, w.w);
    } else {
        const float2* p = reinterpret_cast<const float2*>(v);
        const float2 x = p[a], y = p[a + 8], z = p[a + 16], w = p[a + 24];
        lo[0] = pack2(x.x, y.x); lo[1] = pack2(x.y, y.y);
        hi[0] = pack2(z.x, w.x); hi[1] = pack2(z.y, w.y);
    }
}

// The same pairs from a column that the kernel has normalised: 16-byte pieces of two pairs, piece i of lane a at i * 8 + a (put together from
// the elements' own order, a column cost 16 moves per vector).
template <int DK>
__device__ __forceinline__ void delta_shared_pairs(const float* v, int a, f32x2* lo, f32x2* hi) {
    constexpr int H = DK / 64;                      // pieces of lo, and of hi
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(v) + a;
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const ulonglong2 x = p[8 * i], y = p[8 * (H + i)];
        lo[2 * i] = x.x; lo[2 * i + 1] = x.y;
        hi[2 * i] = y.x; hi[2 * i + 1] = y.y;
    }
}

template <int DK, int R>
__global__ void __launch_bounds__(dc_threads(R)) delta_cols_kernel(DeltaColsParams p) {
    constexpr int EPL = DK / 32;                    // elements per lane of delta_net_kernel
    constexpr int ROWS = 4 * R * kDcWarps;          // rows of S per CTA
    constexpr int kDcStages = dc_stages(R);
    constexpr bool APART = R == 1;                  // warps 4 - 7 prepare, 0 - 3 walk
    extern __shared__ __align__(128) unsigned char sm[];
    DeltaStage<DK, R>* ring = reinterpret_cast<DeltaStage<DK, R>*>(sm);
    pdl_launch_dependents();
    if ((int)blockIdx.z >= p.hdr[1]) return;
    const int4 run = p.runs[blockIdx.z];            // first column, columns, sequence, position of the first
    const int h = blockIdx.y, H = p.H, dv = p.dv;
    const int tid = threadIdx.x & (kDcThreads - 1), lane = tid & 31, warp = tid >> 5, a = lane & 7;
    const bool prepares = !APART || threadIdx.x >= kDcThreads, walks = !APART || !prepares;
    const int row0 = blockIdx.x * ROWS, rloc = warp * 4 * R + (lane >> 3) * R;      // this lane's rows: row0 + rloc .. + R - 1
    const int n_rows = min(ROWS, dv - row0);
    const int n_groups = (run.y + kDcCols - 1) / kDcCols;
    const bool wide = (p.raw_stride & 3) == 0;      // rows of raw start on 16 bytes (an even number of heads), else on 8
    auto load = [&](int g) {
        if (g < n_groups) {
            DeltaStage<DK, R>& s = ring[g % kDcStages];
            const int c0 = run.x + g * kDcCols, n = min(kDcCols, run.y - g * kDcCols);
            auto piece = [&](float (*dst)[DK], int off) {
                if (wide) {
                    for (int i = tid; i < n * (DK / 4); i += kDcThreads) {
                        const int c = i / (DK / 4), e = (i % (DK / 4)) * 4;
                        cp_async16(smem_u32(&dst[c][e]), p.raw + (size_t)(c0 + c) * p.raw_stride + off + e, true);
                    }
                } else {
                    for (int i = tid; i < n * (DK / 2); i += kDcThreads) {
                        const int c = i / (DK / 2), e = (i % (DK / 2)) * 2;
                        cp_async8(smem_u32(&dst[c][e]), p.raw + (size_t)(c0 + c) * p.raw_stride + off + e);
                    }
                }
            };
            piece(s.q, h * DK);
            piece(s.k, (H + h) * DK);
            for (int i = tid; i < n * ROWS; i += kDcThreads) {
                const int c = i / ROWS, e = i % ROWS;
                if (e < n_rows) cp_async4(smem_u32(&s.v[c][e]), p.raw + (size_t)(c0 + c) * p.raw_stride + 2 * H * DK + (size_t)h * dv + row0 + e);
            }
            if (tid < 2 * n) {
                const int c = tid >> 1, which = tid & 1;
                cp_async4(smem_u32(&(which ? s.alpha : s.beta)[c]), p.raw + (size_t)(c0 + c) * p.raw_stride + 2 * H * DK + (size_t)H * dv + which * H + h);
            }
        }
        cp_async_commit();
    };
    f32x2 slo[R][EPL], shi[R][EPL];
    float* Sh = p.state + (((size_t)run.z * H + h) * dv + row0 + rloc) * DK;
    pdl_wait();
    if (prepares) {
        load(0);
        load(1);
        if (APART) load(2);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (walks && rloc + r < n_rows) {
            delta_pairs<DK>(Sh + (size_t)r * DK, a, slo[r], shi[r]);
        } else {
#pragma unroll
            for (int e = 0; e < EPL; ++e) slo[r][e] = shi[r][e] = 0ull;
        }
    }
    // the row whose sums the butterfly leaves in this lane
    const int own = R == 4 ? ((a & 4) ? 2 : 0) + ((a & 2) ? 1 : 0) : 0;
    // sum over the eight lanes of R values per lane, lane a's own row's: steps 4, 2, 1 as in warp_sum
    auto reduce = [&](float (&d)[R]) -> float {
        if (R == 4) {
            const bool up4 = (a & 4) != 0, up2 = (a & 2) != 0;
            float x0 = (up4 ? d[2 % R] : d[0]) + __shfl_xor_sync(0xffffffffu, up4 ? d[0] : d[2 % R], 4);
            float x1 = (up4 ? d[3 % R] : d[1 % R]) + __shfl_xor_sync(0xffffffffu, up4 ? d[1 % R] : d[3 % R], 4);
            x0 = (up2 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, up2 ? x0 : x1, 2);
            return x0 + __shfl_xor_sync(0xffffffffu, x0, 1);
        }
        float x = d[0];
        x += __shfl_xor_sync(0xffffffffu, x, 4);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        return x + __shfl_xor_sync(0xffffffffu, x, 1);
    };
    // a lane's share of a dot product: four-lane chains, then the first two steps of the sum over 32 lanes
    auto dot = [&](const f32x2 (&xl)[EPL], const f32x2 (&xh)[EPL], const f32x2 (&yl)[EPL], const f32x2 (&yh)[EPL]) -> float {
        f32x2 l = 0ull, hh = 0ull;
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            l = fma2(xl[e], yl[e], l);
            hh = fma2(xh[e], yh[e], hh);
        }
        float x, y;
        unpack2(add2(l, hh), x, y);
        return x + y;
    };
    // A column's output is summed over the lanes and written under the next column's dot products: in line it was a second chain of shuffles in
    // a chain that already has one (3001 columns, one row: 1904 -> 1717 us a layer).
    float od[R];
#pragma unroll
    for (int r = 0; r < R; ++r) od[r] = 0.f;
    size_t at = ((size_t)run.x * H + h) * dv + row0 + rloc + own;
    const bool writes = (R == 4 ? (a & 1) == 0 : a == 0) && rloc + own < n_rows;
    auto put = [&](float o) {
        if (writes) {
            if (p.out) p.out[at] = o;
            if (p.out16) p.out16[at] = __float2bfloat16_rn(o);
        }
        at += (size_t)H * dv;
    };
    // L2 norms and gates, as delta_net_kernel takes them
    auto prepare = [&](int g) {
        DeltaStage<DK, R>& sg = ring[g % kDcStages];
        const int n = min(kDcCols, run.y - g * kDcCols);
        for (int c = warp; c < n; c += kDcWarps) {
            float q[EPL], k[EPL], x = 0.f, y = 0.f;
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                q[e] = sg.q[c][lane * EPL + e];
                k[e] = sg.k[c][lane * EPL + e];
                x = fmaf(q[e], q[e], x);
                y = fmaf(k[e], k[e], y);
            }
            x = sqrtf(warp_sum(x) + p.l2_eps);
            y = sqrtf(warp_sum(y) + p.l2_eps);
            __syncwarp();                            // every lane has read its part: the column is rewritten as the pairs that the lanes take
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                const int at = (((lane >> 4) * (EPL / 2) + e / 2) * 8 + (lane & 7)) * 4 + (e & 1) * 2 + ((lane >> 3) & 1);
                sg.q[c][at] = q[e] / x;
                sg.k[c][at] = k[e] / y;
            }
            if (lane < 2) {
                float* gt = (lane ? sg.alpha : sg.beta) + c;
                *gt = 1.0f / (1.0f + expf(-*gt));
            }
        }
    };
    auto walk = [&](int g) {
        DeltaStage<DK, R>& sg = ring[g % kDcStages];
        const int n = min(kDcCols, run.y - g * kDcCols);
        f32x2 kl[EPL], kh[EPL], ql[EPL], qh[EPL];
        delta_shared_pairs<DK>(sg.k[0], a, kl, kh);
        delta_shared_pairs<DK>(sg.q[0], a, ql, qh);
        float alpha = sg.alpha[0], beta = sg.beta[0], v = sg.v[0][rloc + own];
#pragma unroll 2
        for (int c = 0; c < n; ++c) {
            const f32x2 al = pack2(alpha, alpha);
            float d[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int e = 0; e < EPL; ++e) {
                    slo[r][e] = mul2(slo[r][e], al);
                    shi[r][e] = mul2(shi[r][e], al);
                }
                d[r] = dot(slo[r], shi[r], kl, kh);
            }
            // next column's inputs, in flight while this one is summed
            const int cn = c + 1 < n ? c + 1 : c;
            f32x2 nkl[EPL], nkh[EPL], nql[EPL], nqh[EPL];
            delta_shared_pairs<DK>(sg.k[cn], a, nkl, nkh);
            delta_shared_pairs<DK>(sg.q[cn], a, nql, nqh);
            const float nalpha = sg.alpha[cn], nbeta = sg.beta[cn], nv = sg.v[cn][rloc + own];
            const float u = beta * (v - reduce(d)), o = reduce(od);      // (two independent chains of shuffles)
            if (c + g > 0) put(o);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float ur = R == 1 ? u : __shfl_sync(0xffffffffu, u, (lane & 24) + 2 * r);
                const f32x2 uu = pack2(ur, ur);
#pragma unroll
                for (int e = 0; e < EPL; ++e) {
                    slo[r][e] = fma2(uu, kl[e], slo[r][e]);
                    shi[r][e] = fma2(uu, kh[e], shi[r][e]);
                }
                od[r] = dot(slo[r], shi[r], ql, qh);
            }
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                kl[e] = nkl[e];
                kh[e] = nkh[e];
                ql[e] = nql[e];
                qh[e] = nqh[e];
            }
            alpha = nalpha;
            beta = nbeta;
            v = nv;
        }
    };
    if (APART) {
        auto arrived_and_prepared = [&](int g) {     // (each thread has waited for its own copies of the group)
            asm volatile("bar.sync 1, %0;" ::"n"(kDcThreads) : "memory");
            prepare(g);
        };
        if (prepares && n_groups > 0) {
            cp_async_wait<2>();
            arrived_and_prepared(0);
        }
        __syncthreads();
        for (int g = 0; g < n_groups; ++g) {
            if (walks) {
                walk(g);
            } else {
                if (g + 1 < n_groups) {
                    cp_async_wait<1>();
                    arrived_and_prepared(g + 1);
                }
                load(g + 3);                         // into the stage that was walked before the last barrier
            }
            __syncthreads();
        }
    } else {
        for (int g = 0; g < n_groups; ++g) {
            cp_async_wait<1>();
            __syncthreads();
            prepare(g);
            __syncthreads();
            load(g + 2);                             // into the stage whose columns every thread has left behind
            walk(g);
        }
    }
    if (!walks) return;
    if (n_groups > 0) put(reduce(od));
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (rloc + r < n_rows) {
            float x[EPL], y[EPL], z[EPL], w[EPL];
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                unpack2(slo[r][e], x[e], y[e]);
                unpack2(shi[r][e], z[e], w[e]);
            }
            float* d = Sh + (size_t)r * DK;
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                d[a * EPL + e] = x[e];
                d[(a + 8) * EPL + e] = y[e];
                d[(a + 16) * EPL + e] = z[e];
                d[(a + 24) * EPL + e] = w[e];
            }
        }
}

template <int DK, int R>
static cudaError_t delta_cols_one(bool pdl, int max_runs, cudaStream_t st, const DeltaColsParams& p) {
    constexpr int rows = 4 * R * kDcWarps;
    const size_t smem = dc_stages(R) * sizeof(DeltaStage<DK, R>);
    cudaError_t e = cudaFuncSetAttribute(delta_cols_kernel<DK, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(pdl, delta_cols_kernel<DK, R>, dim3((p.dv + rows - 1) / rows, p.H, max_runs), dim3(dc_threads(R)), smem, st, p);
}

// One row per lane group where a chunk is a serial chain rather than a load: columns / longest run sequences side by side, each of H dv rows,
// do not give every SM a CTA of 64 rows. Measured per launch, one row -> four, before the former's preparing warps (now 1038 us): one run of 3000
// columns (dk 128, 16 heads) 2074 -> 3494 us, of 899 (dk 64, 8 heads) 318 -> 424.
bool delta_cols_serial(int sm_count, int H, int dv, int columns, int longest) {
    return (long)columns * H * dv < (long)longest * sm_count * 16 * kDcWarps;
}

cudaError_t delta_cols_launch(int dk, bool few, bool pdl, int max_runs, cudaStream_t st, const DeltaColsParams& p) {
    if (dk == 64) return few ? delta_cols_one<64, 1>(pdl, max_runs, st, p) : delta_cols_one<64, 4>(pdl, max_runs, st, p);
    return few ? delta_cols_one<128, 1>(pdl, max_runs, st, p) : delta_cols_one<128, 4>(pdl, max_runs, st, p);
}

// ------------------------------------------------------------------------------------------------
// Start of a chunk: embed_tc_kernel for many columns. A CTA takes 8 columns and 128 features, so that a row of the first
// layer's per-layer-embedding projection is read once for 8 columns (at 256 columns, one CTA per column and 128 features
// read the 0.5 MB projection of the large model 256 times: 44 us, more than a projection GEMM).
// grid = (ceil(T / 8), ceil(d / 128)), block = 128: one feature per thread.
// ------------------------------------------------------------------------------------------------
constexpr int kEcCols = 8;

template <typename WT>
__global__ void __launch_bounds__(128) embed_cols_kernel(const __grid_constant__ StepCtl c, const __grid_constant__ EmbedColsParams p) {
    extern __shared__ __align__(16) float trow[];    // [8][ple]
    pdl_launch_dependents();
    const int n_cols = *c.n_cols, col0 = blockIdx.x * kEcCols;
    if (col0 >= n_cols) return;
    const int n = min(kEcCols, n_cols - col0), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ple = p.ple;
    const int i = blockIdx.y * 128 + tid;
    if (ple > 0) {
        const bf16_t* T0 = static_cast<const bf16_t*>(p.layers[0].pleT);
        for (int e = tid; e < kEcCols * ple; e += 128) {
            const int u = e / ple, j = e - u * ple;
            trow[e] = u < n ? __bfloat162float(T0[(size_t)c.tok[col0 + u] * ple + j]) : 0.f;
        }
        // 16-byte pieces of the later layers' rows
        const int pieces = ple / 8;
        for (int l = 1 + blockIdx.y; l < p.n_layers; l += gridDim.y) {
            const uint4* Tl = static_cast<const uint4*>(p.layers[l].pleT);
            uint4* dst = reinterpret_cast<uint4*>(p.tple16) + ((size_t)l * p.T + col0) * pieces;
            for (int e = tid; e < n * pieces; e += 128) {
                const int u = e / pieces, j = e - u * pieces;
                dst[e] = __ldg(Tl + (size_t)c.tok[col0 + u] * pieces + j);
            }
        }
        __syncthreads();
    }
    float v[kEcCols];
#pragma unroll
    for (int u = 0; u < kEcCols; ++u) v[u] = 0.f;
    if (i < p.d) {
        if (ple > 0) {
            const bf16_t* prow = static_cast<const bf16_t*>(p.layers[0].pleP) + (size_t)i * ple;
#pragma unroll 2
            for (int j = 0; j < ple; j += 8) {
                float w[8];
                Elem<bf16_t>::load_vec(prow + j, w);
#pragma unroll
                for (int u = 0; u < kEcCols; ++u) {
                    const float4 a = *reinterpret_cast<const float4*>(trow + u * ple + j), b = *reinterpret_cast<const float4*>(trow + u * ple + j + 4);
                    v[u] = fmaf(w[0], a.x, v[u]); v[u] = fmaf(w[1], a.y, v[u]); v[u] = fmaf(w[2], a.z, v[u]); v[u] = fmaf(w[3], a.w, v[u]);
                    v[u] = fmaf(w[4], b.x, v[u]); v[u] = fmaf(w[5], b.y, v[u]); v[u] = fmaf(w[6], b.z, v[u]); v[u] = fmaf(w[7], b.w, v[u]);
                }
            }
        }
        const float g = p.gain[i];
#pragma unroll
        for (int u = 0; u < kEcCols; ++u) {
            if (u < n) {
                const int t = c.tok[col0 + u];
                v[u] = __fadd_rn(__fmul_rn(Elem<WT>::get(static_cast<const WT*>(p.E), (size_t)t * p.d + i), p.escale ? p.escale[t] : 1.0f), v[u]);
            }
        }
        pdl_wait();                                  // nothing before this point is written by an earlier kernel
#pragma unroll
        for (int u = 0; u < kEcCols; ++u) {
            if (u < n) {
                p.x[(size_t)(col0 + u) * p.d + i] = v[u];
                p.xg16[(size_t)(col0 + u) * p.d + i] = __float2bfloat16_rn(v[u] * g);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < kEcCols; ++u) {
        const float ss = warp_sum(i < p.d ? v[u] * v[u] : 0.f);
        if (lane == 0 && u < n) p.ssq[(size_t)(col0 + u) * p.parts + blockIdx.y * 4 + warp] = ss;
    }
}

cudaError_t embed_cols_launch(bool w8, bool pdl, cudaStream_t st, const StepCtl& c, const EmbedColsParams& p) {
    const dim3 grid((p.T + kEcCols - 1) / kEcCols, (p.d + 127) / 128);
    const size_t smem = (size_t)kEcCols * p.ple * 4;
    if (w8) return launch_pdl(pdl, embed_cols_kernel<fp8_t>, grid, dim3(128), smem, st, c, p);
    return launch_pdl(pdl, embed_cols_kernel<bf16_t>, grid, dim3(128), smem, st, c, p);
}

// ------------------------------------------------------------------------------------------------
// Projections (gemm_cols.cuh)
// ------------------------------------------------------------------------------------------------
template <int MODE, typename KVT, bool SUMS, bool PAIR>
static cudaError_t gemm_cols_one(bool pdl, int ctas, cudaStream_t st, const CUtensorMap& x, const CUtensorMap& w, const CUtensorMap& w2,
                                 const CUtensorMap& xx, const CUtensorMap& wx, const GemmColsParams& p, const StepCtl& c, const QkvPostParams& q) {
    cudaError_t e = cudaFuncSetAttribute(gemm_cols_kernel<MODE, KVT, SUMS, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGcSmem);
    if (e != cudaSuccess) return e;
    const size_t smem = 1024 + (size_t)p.stages * (kGcM + (PAIR ? p.BN / 2 : p.BN)) * 128 + gc_staging(MODE);
    return launch_pdl_cluster(pdl, PAIR ? 2 : 1, gemm_cols_kernel<MODE, KVT, SUMS, PAIR>, dim3(ctas), dim3(kGcThreads), smem, st, x, w, w2, xx, wx, p, c, q);
}

template <bool SUMS, bool PAIR>
static cudaError_t gemm_cols_mode(int mode, int kv_dtype, bool pdl, int ctas, cudaStream_t st, const CUtensorMap& x, const CUtensorMap& w,
                                  const CUtensorMap& w2, const CUtensorMap& xx, const CUtensorMap& wx, const GemmColsParams& p, const StepCtl& c,
                                  const QkvPostParams& q) {
    switch (mode) {
        case TC_RAW: return gemm_cols_one<TC_RAW, float, SUMS, PAIR>(pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
        case TC_RESID: return gemm_cols_one<TC_RESID, float, SUMS, PAIR>(pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
        case TC_SWIGLU: return gemm_cols_one<TC_SWIGLU, float, SUMS, PAIR>(pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
        default:
            if (kv_dtype == MLB_DT_F32) return gemm_cols_one<TC_QKV, float, SUMS, PAIR>(pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
            return gemm_cols_one<TC_QKV, bf16_t, SUMS, PAIR>(pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
    }
}

// The register shares of the kernels with sums add up only at kGcRegsLaunch registers a thread, which a compiler chooses: with another count their
// warps would wait for registers without end.
template <int MODE, typename KVT, bool PAIR>
static cudaError_t gemm_cols_shares(bool* ok) {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, gemm_cols_kernel<MODE, KVT, true, PAIR>);
    *ok = *ok && e == cudaSuccess && a.numRegs == kGcRegsLaunch;
    return e;
}
template <bool PAIR>
static cudaError_t gemm_cols_shares_of(bool* ok) {
    cudaError_t e = gemm_cols_shares<TC_RAW, float, PAIR>(ok);
    if (e == cudaSuccess) e = gemm_cols_shares<TC_RESID, float, PAIR>(ok);
    if (e == cudaSuccess) e = gemm_cols_shares<TC_SWIGLU, float, PAIR>(ok);
    if (e == cudaSuccess) e = gemm_cols_shares<TC_QKV, float, PAIR>(ok);
    if (e == cudaSuccess) e = gemm_cols_shares<TC_QKV, bf16_t, PAIR>(ok);
    return e;
}
cudaError_t gemm_cols_can_sum(bool* ok) {
    *ok = true;
    const cudaError_t e = gemm_cols_shares_of<false>(ok);
    return e == cudaSuccess ? gemm_cols_shares_of<true>(ok) : e;
}

cudaError_t gemm_cols_launch(int mode, int kv_dtype, bool sums, bool pair, bool pdl, int ctas, cudaStream_t st, const CUtensorMap& x, const CUtensorMap& w,
                             const CUtensorMap& w2, const CUtensorMap& xx, const CUtensorMap& wx, const GemmColsParams& p, const StepCtl& c,
                             const QkvPostParams& q) {
    if (pair) return sums ? gemm_cols_mode<true, true>(mode, kv_dtype, pdl, ctas, st, x, w, w2, xx, wx, p, c, q)
                          : gemm_cols_mode<false, true>(mode, kv_dtype, pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
    return sums ? gemm_cols_mode<true, false>(mode, kv_dtype, pdl, ctas, st, x, w, w2, xx, wx, p, c, q)
                : gemm_cols_mode<false, false>(mode, kv_dtype, pdl, ctas, st, x, w, w2, xx, wx, p, c, q);
}

static __global__ void __launch_bounds__(256) widen_e4m3_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, size_t n16) {
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n16; i += (size_t)gridDim.x * 256) {
        const uint4 w = __ldg(src + i);
        uint4 a, b;
        a.x = e4m3x2_to_bf16x2(w.x & 0xffffu); a.y = e4m3x2_to_bf16x2(w.x >> 16); a.z = e4m3x2_to_bf16x2(w.y & 0xffffu); a.w = e4m3x2_to_bf16x2(w.y >> 16);
        b.x = e4m3x2_to_bf16x2(w.z & 0xffffu); b.y = e4m3x2_to_bf16x2(w.z >> 16); b.z = e4m3x2_to_bf16x2(w.w & 0xffffu); b.w = e4m3x2_to_bf16x2(w.w >> 16);
        dst[2 * i] = a;
        dst[2 * i + 1] = b;
    }
}
cudaError_t widen_e4m3_launch(const void* codes, bf16_t* out, size_t n, cudaStream_t st) {
    widen_e4m3_kernel<<<1184, 256, 0, st>>>(static_cast<const uint4*>(codes), reinterpret_cast<uint4*>(out), n / 16);
    return cudaGetLastError();
}

}  // namespace mlb
