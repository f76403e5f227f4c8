"""The projections of batched decode steps at the edges of their tiles: 32 output features, 16 / 32 / 64 sequences, ranges and
copies of 64-wide k-blocks; against the oracle."""
import numpy as np
import pytest

from helpers import TOL_LOWP, load_oracle, logits_error, random_prompts, write_model
from mini_llm_cuda_b200.model_file import ModelSpec, periodic_layer_types

pytestmark = pytest.mark.gpu

MHA = dict(heads=2, head_dim=64, kv_dtype="bfloat16", rms_eps=1e-5, max_context=32)
SPECS = {
    # a per-layer embedding behind the down projection; 21 k-blocks over the ranges; 500 logits end inside a tile
    "bf16_ple": ModelSpec(dim=128, layers=3, ffn_dim=1344, ple_dim=64, vocab=500, layer_types=periodic_layer_types(3, 2), weight_dtype="bfloat16", **MHA),
    # one k-block; gated queries
    "bf16_one": ModelSpec(dim=64, layers=2, ffn_dim=64, vocab=72, query_gating=True, weight_dtype="bfloat16", **{**MHA, "heads": 1}),
    # codes, row scales and the embedding's own accumulators; delta-net rows that end inside a tile of 32
    "fp8_ple": ModelSpec(dim=192, layers=3, ffn_dim=832, ple_dim=128, vocab=500, dn_key_dim=64, dn_value_dim=96, layer_types=periodic_layer_types(3, 3),
                         weight_dtype="float8_e4m3", **MHA),
    "fp8": ModelSpec(dim=512, layers=2, ffn_dim=640, kv_heads=2, vocab=512, weight_dtype="float8_e4m3", **{**MHA, "heads": 8}),
}


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


@pytest.mark.parametrize("name", list(SPECS))
def test_decode_projections_at_tile_edges(api, tmp_path, name):
    spec = SPECS[name]
    path = write_model(tmp_path, spec, seed=61)
    oracle = load_oracle(path)
    texts = random_prompts(spec.vocab, [4] * 11, seed=63)           # eleven texts, so that neighbours in a tile differ
    want = []
    for t in texts:
        st = oracle.new_state()
        want.append([oracle.step(st, int(k)).numpy() for k in t])
    model = api.Model(path)
    for batch in (4, 5, 15, 16, 17, 32, 33, 64, 65, 129, 256):
        sess = api.Session(model, batch)
        assert sess.path() == "mma"
        sess.prefill([texts[b % 11][:1] for b in range(batch)])
        for k in range(4):
            sess.decode_step(in_tokens=np.array([texts[b % 11][k] for b in range(batch)], dtype=np.int32))
        got = sess.logits()
        worst = max(logits_error(got[b], want[b % 11][3]) for b in range(batch))
        assert worst < TOL_LOWP, (batch, worst)
        sess.close()
    model.close()
