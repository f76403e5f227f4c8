// The launch chain for bf16 weights.
#include "chain.cuh"

namespace mlb {

int chain_run_bf16(mlb_session* s, int kind, Recorder* rec, int* n_launches) {
    if (s->m->cfg.kv_dtype == MLB_DT_F32) return Chain<bf16_t, bf16_t, float>::run(s, kind, rec, n_launches);
    return Chain<bf16_t, bf16_t, bf16_t>::run(s, kind, rec, n_launches);
}
int chain_configure_bf16(mlb_session* s) {
    return s->m->cfg.kv_dtype == MLB_DT_F32 ? Chain<bf16_t, bf16_t, float>::configure() : Chain<bf16_t, bf16_t, bf16_t>::configure();
}
int tc_allow_big_smem_bf16(int kv_dtype) { return kv_dtype == MLB_DT_BF16 ? tc_allow_big_smem_t<bf16_t, bf16_t>() : tc_allow_big_smem_t<float, bf16_t>(); }

int tc_max_clusters(int size, size_t smem, int* n) {
    void (*kern)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, GemmTcParams, StepCtl, QkvPostParams) =
        gemm_tc_kernel<TC_RESID, float, bf16_t>;
    CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(1, 1, size);
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = size;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(n, kern, &cfg) != cudaSuccess) { cudaGetLastError(); *n = 0; }
    return MLB_OK;
}

int chain_attn_f32kv(mlb_session* s, const StepCtl& c, const AttnParams& a) {
    const mlb_config& cfg = s->m->cfg;
    const int G = cfg.heads / cfg.kv_heads;
    return cfg.head_dim == 64 ? Chain<bf16_t, bf16_t, float>::attn_g<64>(s, c, a, G) : Chain<bf16_t, bf16_t, float>::attn_g<128>(s, c, a, G);
}

}  // namespace mlb
