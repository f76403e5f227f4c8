"""The generic single-kernel step where its work splits change: vectors of up to 960, 1920 and more words per gather, rows taken in
pairs or one by one, an odd last row, uneven shares; against the oracle."""
import pytest

from helpers import TOL_FP32, TOL_LOWP, load_oracle, logits_error, oracle_rollout, random_prompts, write_model
from mini_llm_cuda_b200.model_file import ModelSpec, periodic_layer_types

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float8_e4m3"])
@pytest.mark.parametrize("dim,heads,ffn,vocab", [(192, 3, 144, 160), (256, 4, 976, 509), (512, 8, 1936, 1000), (1024, 16, 2416, 2400), (2064, 4, 4464, 300)])
def test_single_kernel_step_splits(api, tmp_path, monkeypatch, dtype, dim, heads, ffn, vocab):
    monkeypatch.setenv("MLB_DECODE_PATH", "grid")
    spec = ModelSpec(dim=dim, layers=2, heads=heads, head_dim=64, ffn_dim=ffn, vocab=vocab, max_context=96, ple_dim=48, rms_eps=1e-5,
                     dn_key_dim=64, dn_value_dim=64, layer_types=periodic_layer_types(2, 2), weight_dtype=dtype,
                     kv_dtype="float32" if dtype == "float32" else "bfloat16")
    path = write_model(tmp_path, spec, seed=71)
    oracle = load_oracle(path)
    prompt = random_prompts(spec.vocab, [70], seed=73)[0]
    _, want = oracle_rollout(oracle, prompt, 1)
    model = api.Model(path)
    sess = api.Session(model, 1)
    sess.prefill([prompt])
    sess.decode_step()
    assert logits_error(sess.logits()[0], want[0]) < (TOL_FP32 if dtype == "float32" else TOL_LOWP)
    sess.close()
    model.close()
