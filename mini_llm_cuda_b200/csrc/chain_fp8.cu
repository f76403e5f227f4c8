// The launch chain for FP8 weights.
#include "chain.cuh"

namespace mlb {

int chain_run_fp8(mlb_session* s, int kind, Recorder* rec, int* n_launches) {
    if (s->m->cfg.kv_dtype == MLB_DT_F32) return Chain<fp8_t, bf16_t, float>::run(s, kind, rec, n_launches);
    return Chain<fp8_t, bf16_t, bf16_t>::run(s, kind, rec, n_launches);
}
int chain_configure_fp8(mlb_session* s) {
    return s->m->cfg.kv_dtype == MLB_DT_F32 ? Chain<fp8_t, bf16_t, float>::configure() : Chain<fp8_t, bf16_t, bf16_t>::configure();
}
int tc_allow_big_smem_fp8(int kv_dtype) { return kv_dtype == MLB_DT_BF16 ? tc_allow_big_smem_t<bf16_t, fp8_t>() : tc_allow_big_smem_t<float, fp8_t>(); }

}  // namespace mlb
