// Streaming GEMV for BT = 1 .. 3 sequences per CTA row: y[b][row] = sum_k W[row][k] * x[b][k], with the weights
// fed by TMA bulk copies instead of per-thread loads.
//
// The per-thread-load GEMV of kernels.cuh keeps ~30 KB in flight per SM and pays its latency chain
// (activations -> weights -> reduction) once per CTA of 8-16 rows; on multi-MB matrices that caps it
// at a tenth of the HBM bandwidth. Here the matrix is cut into one contiguous slab of rows per CTA
// (about one CTA per SM). A producer warp streams the slab with cp.async.bulk into a ring of
// shared-memory stages guarded by mbarriers - and it starts BEFORE griddepcontrol.wait, because
// weights do not depend on the predecessor kernel - while 31 consumer warps stage and normalise
// the activation vector once, then take dot products out of shared memory two rows at a time.
// Epilogues are the ones of gemv_kernel (same reference citations): plain store, residual (+ the
// next layer's per-layer embedding), SwiGLU of a gate/up slab pair, QKV with per-head norm / RoPE /
// KV append (one head per CTA), LM head with argmax partials and last-CTA pick.
// grid = (slabs, ceil(B / BT)); every mbarrier wait is bounded (Ring::wait).
// A slab is taken for all of a small batch: with a CTA per slab and sequence (one CTA per SM) the 8 MB LM head of three
// sequences went three times through the GPU, 24.4 us.
#pragma once
#include "ring.cuh"

namespace mlb {

struct SgemvGeom {
    int rows_per_cta;
    int n_stages, stage_bytes;
    int off_xs, off_xs2, off_outs, off_pacc, off_red, off_bar, off_ring;   // float offsets
    int xs_stride, xs2_stride, outs_stride, pacc_stride;                   // floats from one sequence's to the next's
    int* err;
};

constexpr int kSgWarps = 31;                       // consumer warps (+ 1 producer warp = 1024 threads, 64 registers each)
constexpr int kSgConsumers = kSgWarps * 32;
constexpr int kSgThreads = kSgConsumers + 32;

// Two rows at a time against BT activation vectors in shared memory (xs_f4_index); one read of a row serves all of them.
template <typename T, int BT>
__device__ __forceinline__ void sg_rows_dot2(const T* row0, const T* row1, int nvec, const float* xs, int xs_stride, int lane, float (&a0)[BT], float (&a1)[BT]) {
    constexpr int EPV = Elem<T>::EPV;
#pragma unroll
    for (int b = 0; b < BT; ++b) a0[b] = a1[b] = 0.f;
#pragma unroll 1
    for (int vi = lane; vi < nvec; vi += 32) {
        float w0[EPV], w1[EPV];
        Elem<T>::unpack(*reinterpret_cast<const uint4*>(row0 + (size_t)vi * EPV), w0);
        Elem<T>::unpack(*reinterpret_cast<const uint4*>(row1 + (size_t)vi * EPV), w1);
#pragma unroll
        for (int b = 0; b < BT; ++b) {
            const float4* xp = reinterpret_cast<const float4*>(xs + b * xs_stride);
#pragma unroll
            for (int q = 0; q < EPV / 4; ++q) {
                const float4 t = xp[q * nvec + vi];
                a0[b] = fmaf(w0[4 * q], t.x, a0[b]); a0[b] = fmaf(w0[4 * q + 1], t.y, a0[b]);
                a0[b] = fmaf(w0[4 * q + 2], t.z, a0[b]); a0[b] = fmaf(w0[4 * q + 3], t.w, a0[b]);
                a1[b] = fmaf(w1[4 * q], t.x, a1[b]); a1[b] = fmaf(w1[4 * q + 1], t.y, a1[b]);
                a1[b] = fmaf(w1[4 * q + 2], t.z, a1[b]); a1[b] = fmaf(w1[4 * q + 3], t.w, a1[b]);
            }
        }
    }
#pragma unroll
    for (int b = 0; b < BT; ++b) {
        a0[b] = warp_sum(a0[b]);
        a1[b] = warp_sum(a1[b]);
    }
}

// A slab of `rows` rows of K elements, or a chunk-interleaved pair: f(local row, dots), f(local row, dots of the first matrix, of the second),
// in every lane of the warp that owns the row.
template <typename T, int BT, typename F>
__device__ __forceinline__ void sg_consume(Ring& r, int rows, int K, const float* xs, int xs_stride, int warp, int lane, F&& f) {
    const int nvec = K / Elem<T>::EPV, rpc = max(1, r.stage_bytes / (K * (int)sizeof(T)));
    for (int r0 = 0; r0 < rows; r0 += rpc) {
        const int n = min(rpc, rows - r0);
        r.wait(r.full0 + 8u * r.idx, r.phase, 2);
        const T* base = reinterpret_cast<const T*>(r.stages + (size_t)r.idx * r.stage_bytes);
        const int two = n >= 2 * kSgWarps ? 1 : 0;     // few long rows in the chunk: one row per warp keeps more warps busy
        for (int i = warp << two; i < n; i += kSgWarps << two) {
            const int i1 = two && i + 1 < n ? i + 1 : i;
            float a0[BT], a1[BT];
            sg_rows_dot2<T, BT>(base + (size_t)i * K, base + (size_t)i1 * K, nvec, xs, xs_stride, lane, a0, a1);
            f(r0 + i, a0);
            if (i1 > i) f(r0 + i1, a1);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(r.empty0 + 8u * r.idx);
        r.advance();
    }
}
template <typename T, int BT, typename F>
__device__ __forceinline__ void sg_consume_pair(Ring& r, int rows, int K, const float* xs, int xs_stride, int warp, int lane, F&& f) {
    const int nvec = K / Elem<T>::EPV, rpc = max(1, r.stage_bytes / (K * (int)sizeof(T)));
    for (int r0 = 0; r0 < rows; r0 += rpc) {
        const int n = min(rpc, rows - r0);
        const int ia = r.idx;
        r.wait(r.full0 + 8u * r.idx, r.phase, 2);
        r.advance();
        const int ib = r.idx;
        r.wait(r.full0 + 8u * r.idx, r.phase, 2);
        r.advance();
        const T* A = reinterpret_cast<const T*>(r.stages + (size_t)ia * r.stage_bytes);
        const T* Bm = reinterpret_cast<const T*>(r.stages + (size_t)ib * r.stage_bytes);
        for (int i = warp; i < n; i += kSgWarps) {
            float a0[BT], a1[BT];
            sg_rows_dot2<T, BT>(A + (size_t)i * K, Bm + (size_t)i * K, nvec, xs, xs_stride, lane, a0, a1);
            f(r0 + i, a0, a1);
        }
        __syncwarp();
        if (lane == 0) { mbar_arrive(r.empty0 + 8u * ia); mbar_arrive(r.empty0 + 8u * ib); }
    }
}

template <typename T, typename T2, typename KVT, int BT, int MODE>
__global__ void __launch_bounds__(kSgThreads, 1) sgemv_kernel(StepCtl c, GemvParams p, SgemvGeom g) {
    extern __shared__ __align__(128) float sg_smem[];
    float* smem = sg_smem;
    float* xs = smem + g.off_xs;
    float* xs2 = smem + g.off_xs2;
    float* outs = smem + g.off_outs;
    float* pacc = smem + g.off_pacc;
    float* red = smem + g.off_red;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b0 = (int)blockIdx.y * BT;
    const int K = p.K, Kp = p.Kp, N = p.N;
    const int esz = (int)sizeof(T);
    const int r_begin = min(N, (int)blockIdx.x * g.rows_per_cta);
    const int r_end = min(N, r_begin + g.rows_per_cta);
    const int rows = r_end - r_begin;

    Ring ring;
    int* dead = reinterpret_cast<int*>(red + kSgWarps);
    ring.full0 = smem_u32(smem + g.off_bar);
    ring.empty0 = ring.full0 + 8u * g.n_stages;
    ring.stages = reinterpret_cast<unsigned char*>(smem + g.off_ring);
    ring.nst = g.n_stages;
    ring.stage_bytes = g.stage_bytes;
    ring.idx = 0;
    ring.phase = 0;
    ring.dead = dead;
    ring.err = g.err;
    ring.backoff_ns = 0;
    if (tid == 0) {
        *dead = 0;
        for (int i = 0; i < g.n_stages; ++i) {
            mbar_init(ring.full0 + 8u * i, 1);
            mbar_init(ring.empty0 + 8u * i, kSgWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kSgWarps) {
        // ---- producer: weights only, nothing here depends on the predecessor kernel ------------
        if (Kp > 0)
            issue_slab(ring, reinterpret_cast<const unsigned char*>(p.P) + (size_t)r_begin * Kp * sizeof(T2), rows,
                       Kp * (int)sizeof(T2), lane);
        if (MODE == GEMV_SWIGLU)
            issue_slab_pair(ring, reinterpret_cast<const unsigned char*>(p.W) + (size_t)r_begin * K * esz,
                            reinterpret_cast<const unsigned char*>(p.Wb) + (size_t)r_begin * K * esz, rows, K * esz, lane);
        else
            issue_slab(ring, reinterpret_cast<const unsigned char*>(p.W) + (size_t)r_begin * K * esz, rows, K * esz, lane);
        return;
    }

    // ---- consumers ------------------------------------------------------------------------------
    pdl_wait();
    bool active[BT];
#pragma unroll
    for (int u = 0; u < BT; ++u) active[u] = seq_active(c, b0 + u);
    // stage (and RMS-normalise) the activation vectors: inference.cu:24-50, :83-95
#pragma unroll 1
    for (int u = 0; u < BT; ++u) {
        const int bg = min(b0 + u, c.B - 1);
        const float* xr = p.xin + (size_t)bg * K;
        float* xu = xs + u * g.xs_stride;
        constexpr int EPV = Elem<T>::EPV;
        const int nvec = K / EPV;
        float ss = 0.f;
        for (int k = tid; k < K; k += kSgConsumers) {
            const float v = xr[k];
            xu[xs_index<EPV>(k, nvec)] = v;              // bank-conflict-free layout for the dot products
            ss = fmaf(v, v, ss);
        }
        if (Kp > 0) {
            const int t = c.tok[bg];
            const T2* trow = reinterpret_cast<const T2*>(p.Ptab) + (size_t)t * Kp;
            for (int k = tid; k < Kp; k += kSgConsumers) xs2[u * g.xs2_stride + xs_index<Elem<T2>::EPV>(k, Kp / Elem<T2>::EPV)] = Elem<T2>::get(trow, k);
        }
        if (p.do_norm) {
            const float tot = consumer_sum<kSgWarps>(ss, red, warp, lane);
            const float r = sqrtf(tot / (float)K + p.eps);
            for (int k = tid; k < K; k += kSgConsumers) {
                const int d = xs_index<EPV>(k, nvec);
                xu[d] = (xu[d] / r) * p.gain[k];
            }
        }
    }
    consumer_sync<kSgWarps>();
    if (Kp > 0) {
        sg_consume<T2, BT>(ring, rows, Kp, xs2, g.xs2_stride, warp, lane, [&](int r, const float (&v)[BT]) {
            if (lane == 0) {
#pragma unroll
                for (int u = 0; u < BT; ++u) pacc[u * g.pacc_stride + r] = v[u];
            }
        });
        consumer_sync<kSgWarps>();
    }

    if (MODE == GEMV_SWIGLU) {
        sg_consume_pair<T, BT>(ring, rows, K, xs, g.xs_stride, warp, lane, [&](int r, const float (&va)[BT], const float (&vb)[BT]) {
            const int row = r_begin + r;
#pragma unroll
            for (int u = 0; u < BT; ++u) {
                float gt = va[u], up = vb[u];
                if (p.wscale) { gt *= p.wscale[row]; up *= p.wscale_b[row]; }
                // applySiluToFFN + hadamardMultiplyFFN, inference.cu:262-281
                if (lane == 0 && active[u]) p.y[(size_t)(b0 + u) * N + row] = (gt / (1.0f + expf(-gt))) * up;
            }
        });
    } else if (MODE == GEMV_RAW || MODE == GEMV_RESID) {
        sg_consume<T, BT>(ring, rows, K, xs, g.xs_stride, warp, lane, [&](int r, const float (&va)[BT]) {
            const int row = r_begin + r;
#pragma unroll
            for (int u = 0; u < BT; ++u) {
                float v = va[u];
                // (no fused multiply-add here and below: every form of the kernel rounds alike)
                if (p.wscale) v = __fmul_rn(v, p.wscale[row]);
                if (Kp > 0) v = __fadd_rn(v, pacc[u * g.pacc_stride + r]);
                if (lane == 0 && active[u]) {
                    // addResidualToOutputProj / addResidualToFFN, inference.cu:252-260, :283-291
                    if (MODE == GEMV_RESID) v = __fadd_rn(v, p.resid[(size_t)(b0 + u) * N + row]);
                    p.y[(size_t)(b0 + u) * N + row] = v;
                }
            }
        });
    } else if (MODE == GEMV_QKV) {
        // a CTA owns whole heads' worth of rows (rows_per_cta == hd) when the per-head norm is on,
        // else a 32-row group inside one head
        sg_consume<T, BT>(ring, rows, K, xs, g.xs_stride, warp, lane, [&](int r, const float (&v)[BT]) {
            if (lane == 0) {
#pragma unroll
                for (int u = 0; u < BT; ++u) outs[u * g.outs_stride + r] = p.wscale ? v[u] * p.wscale[r_begin + r] : v[u];
            }
        });
        consumer_sync<kSgWarps>();
#pragma unroll 1
        for (int u = 0; u < BT; ++u) {
            const int b = b0 + u;
            const float* ou = outs + u * g.outs_stride;
            const int hd = p.hd;
            const int seg_q = p.nq, seg_k = p.nq + p.nk, seg_v = seg_k + p.nv;
            const int seg = r_begin < seg_q ? 0 : (r_begin < seg_k ? 1 : (r_begin < seg_v ? 2 : 3));
            float rs = 1.f;
            if (p.qk_norm && seg < 2) {
                // getRMSColSumsAcrossHeads + applyRMSNormAcrossHeads, inference.cu:52-81, :97-111
                float ss = 0.f;
                for (int r = tid; r < rows; r += kSgConsumers) ss = fmaf(ou[r], ou[r], ss);
                rs = sqrtf(consumer_sum<kSgWarps>(ss, red, warp, lane) / (float)hd + p.eps);
            }
            if (seq_active(c, b)) {
                const int pos = c.pos[b];
                KVT* kpool = reinterpret_cast<KVT*>(p.kpool);
                KVT* vpool = reinterpret_cast<KVT*>(p.vpool);
                for (int pr = tid; pr < rows / 2; pr += kSgConsumers) {
                    const int r = 2 * pr, row = r_begin + r;
                    float a = ou[r], cc = ou[r + 1];
                    if (seg < 2) {
                        const int srow = seg == 0 ? row : row - seg_q;
                        if (p.qk_norm) {
                            const float* gg = seg == 0 ? p.gq : p.gk;
                            a = (a / rs) * gg[srow];
                            cc = (cc / rs) * gg[srow + 1];
                        }
                        // applyRoPE, inference.cu:113-134
                        const int e = srow % hd;                       // position of the pair inside its head
                        const float cs = p.rope[(size_t)pos * hd + e], sn = p.rope[(size_t)pos * hd + e + 1];
                        const float ra = fmaf(cs, a, -__fmul_rn(sn, cc)), rc = fmaf(cs, cc, __fmul_rn(sn, a));
                        if (seg == 0) {
                            p.qbuf[(size_t)b * p.nq + srow] = ra;
                            p.qbuf[(size_t)b * p.nq + srow + 1] = rc;
                        } else {
                            const int kvh = srow / hd;
                            const int page = p.page_table[kv_seq(c, b) * p.pt_stride + pos / kKvBlock];
                            const size_t off = (((size_t)page * p.kv_heads + kvh) * kKvBlock + (pos % kKvBlock)) * hd + e;
                            Elem<KVT>::put(kpool, off, ra);
                            Elem<KVT>::put(kpool, off + 1, rc);
                        }
                    } else if (seg == 2) {
                        const int srow = row - seg_k;
                        const int kvh = srow / hd, e = srow % hd;
                        const int page = p.page_table[kv_seq(c, b) * p.pt_stride + pos / kKvBlock];
                        const size_t off = (((size_t)page * p.kv_heads + kvh) * kKvBlock + (pos % kKvBlock)) * hd + e;
                        Elem<KVT>::put(vpool, off, a);
                        Elem<KVT>::put(vpool, off + 1, cc);
                    } else {
                        const int srow = row - seg_v;
                        p.gbuf[(size_t)b * p.ng + srow] = 1.0f / (1.0f + expf(-a));        // inference.cu:248
                        p.gbuf[(size_t)b * p.ng + srow + 1] = 1.0f / (1.0f + expf(-cc));
                    }
                }
            }
        }
    } else {
        // LM head: logits, argmax partial of this CTA, pick by the last CTA of the sequences
        // (inference.cu:720-743; host qsort of inference_orchestrator.cu:77-84 replaced)
        float bv[BT];
        int bi[BT];
#pragma unroll
        for (int u = 0; u < BT; ++u) { bv[u] = -INFINITY; bi[u] = 0x7fffffff; }
        sg_consume<T, BT>(ring, rows, K, xs, g.xs_stride, warp, lane, [&](int r, const float (&va)[BT]) {
            const int row = r_begin + r;
#pragma unroll
            for (int u = 0; u < BT; ++u) {
                float v = va[u];
                if (p.wscale) v *= p.wscale[row];
                if (lane == 0 && active[u]) p.y[(size_t)(b0 + u) * N + row] = v;
                if (v > bv[u] || (v == bv[u] && row < bi[u])) { bv[u] = v; bi[u] = row; }
            }
        });
        consumer_sync<kSgWarps>();
        if (lane == 0) {
#pragma unroll
            for (int u = 0; u < BT; ++u) {
                outs[u * g.outs_stride + 2 * warp] = bv[u];
                outs[u * g.outs_stride + 2 * warp + 1] = __int_as_float(bi[u]);
            }
        }
        consumer_sync<kSgWarps>();
        __shared__ int is_last;
        const int nparts = gridDim.x;
        // warp u takes sequence b0 + u; one ticket for all of them
        const int b = b0 + warp;
        if (warp < BT && b < c.B) {
            float v = -INFINITY;
            int ix = 0x7fffffff;
            if (lane < kSgWarps) {
                v = outs[warp * g.outs_stride + 2 * lane];
                ix = __float_as_int(outs[warp * g.outs_stride + 2 * lane + 1]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, v, o);
                const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
                if (ov > v || (ov == v && oi < ix)) { v = ov; ix = oi; }
            }
            if (lane == 0) {
                p.part_val[(size_t)b * nparts + blockIdx.x] = v;
                p.part_idx[(size_t)b * nparts + blockIdx.x] = ix;
                __threadfence();
            }
        }
        consumer_sync<kSgWarps>();
        if (tid == 0) is_last = atomicAdd(&p.ticket[blockIdx.y], 1) == nparts - 1;
        consumer_sync<kSgWarps>();
        if (is_last && warp < BT && b < c.B) {
            __threadfence();
            float v2 = -INFINITY;
            int i2 = 0x7fffffff;
            for (int q = lane; q < nparts; q += 32) {
                const float v = __ldcg(&p.part_val[(size_t)b * nparts + q]);
                const int ix = __ldcg(&p.part_idx[(size_t)b * nparts + q]);
                if (v > v2 || (v == v2 && ix < i2)) { v2 = v; i2 = ix; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, v2, o);
                const int oi = __shfl_xor_sync(0xffffffffu, i2, o);
                if (ov > v2 || (ov == v2 && oi < i2)) { v2 = ov; i2 = oi; }
            }
            if (lane == 0) {
                if (warp == 0) p.ticket[blockIdx.y] = 0;
                if (p.do_pick && seq_active(c, b)) advance_seq(c, b, i2);
            }
        }
    }
}

}  // namespace mlb
