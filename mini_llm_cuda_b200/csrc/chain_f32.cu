// The launch chain for fp32 weights.
#include "chain.cuh"

namespace mlb {

int chain_run_f32(mlb_session* s, int kind, Recorder* rec, int* n_launches) {
    if (s->m->cfg.kv_dtype == MLB_DT_F32) return Chain<float, float, float>::run(s, kind, rec, n_launches);
    return Chain<float, float, bf16_t>::run(s, kind, rec, n_launches);
}
int chain_configure_f32(mlb_session* s) {
    return s->m->cfg.kv_dtype == MLB_DT_F32 ? Chain<float, float, float>::configure() : Chain<float, float, bf16_t>::configure();
}

}  // namespace mlb
