"""Prompt columns at the edges of their tiles: column sets of 64 to 4096, attention tiles of 32 (query, head) rows over
64-position K/V tiles, delta-net stages of 16 columns, GEMM tiles of 128 columns; against the oracle."""
import dataclasses
import os

import numpy as np
import pytest

from helpers import TOL_FP32, TOL_LOWP, load_oracle, logits_error, oracle_rollout, random_prompts, write_model
from mini_llm_cuda_b200.model_file import ModelSpec, periodic_layer_types, synth_weights, write_model_bin

pytestmark = pytest.mark.gpu

BF16 = dict(weight_dtype="bfloat16", kv_dtype="bfloat16", rms_eps=1e-5, vocab=512)
SPECS = {
    "mha64": ModelSpec(dim=128, layers=3, heads=2, head_dim=64, ffn_dim=256, ple_dim=32, layer_types=periodic_layer_types(3, 2), **BF16),
    "gqa4_128": ModelSpec(dim=256, layers=2, heads=4, kv_heads=1, head_dim=128, ffn_dim=264, qk_norm=True, query_gating=True, **BF16),
    "gqa8_64": ModelSpec(dim=256, layers=2, heads=8, kv_heads=1, head_dim=64, ffn_dim=256, **BF16),
    "gqa2_128": ModelSpec(dim=256, layers=2, heads=4, kv_heads=2, head_dim=128, ffn_dim=256, **BF16),
    # three heads: the rows of the raw delta-net projection start on 8 bytes; 72 value rows end inside a CTA's 64 and 16
    "dn_odd": ModelSpec(dim=192, layers=2, heads=3, head_dim=64, ffn_dim=256, dn_key_dim=128, dn_value_dim=72,
                        layer_types=periodic_layer_types(2, 1), **BF16),
    "fp8": ModelSpec(dim=256, layers=3, heads=4, kv_heads=1, head_dim=64, ffn_dim=272, ple_dim=24, vocab=512, rms_eps=1e-5,
                     layer_types=periodic_layer_types(3, 3), weight_dtype="float8_e4m3", kv_dtype="bfloat16"),
}


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


@pytest.mark.parametrize("name", list(SPECS))
def test_scored_columns_at_tile_edges(api, tmp_path, name):
    """Every position's logits of texts of 1 to 1025 tokens (one session: the column sets are made as they are needed)."""
    spec = dataclasses.replace(SPECS[name], max_context=1040)
    path = write_model(tmp_path, spec, seed=41)
    oracle = load_oracle(path)
    tokens = random_prompts(spec.vocab, [1025], seed=43)[0]
    st = oracle.new_state()
    want = np.stack([np.asarray(oracle.step(st, int(t))) for t in tokens])
    model = api.Model(path)
    sess = api.Session(model, 1)
    for length in (1, 2, 15, 17, 63, 64, 65, 127, 128, 129, 1025):
        got = sess.score(tokens[:length])
        assert sess.path(length) == "cols"
        worst = max(logits_error(got[i], want[i]) for i in range(length))
        assert worst < TOL_LOWP, (length, worst)
    sess.close()
    model.close()


@pytest.mark.parametrize("name,lens", [("mha64", [2100, 1, 2050]), ("dn_odd", [2048, 2049, 3]), ("gqa4_128", [4099]), ("fp8", [65] * 70), ("mha64", [70, 33, 101] * 29)])
def test_prompts_longer_than_one_chunk(api, tmp_path, monkeypatch, name, lens):
    """More than 4096 prompt tokens: the sequences continue across chunks, in equal shares; many short ones share a chunk, in whole
    attention tiles (87 sequences: shares of 47 become 64, and the last of them wait for the next chunk)."""
    monkeypatch.setenv("MLB_PREFILL", "chunk")
    spec = dataclasses.replace(SPECS[name], max_context=max(lens) + 8)
    path = write_model(tmp_path, spec, seed=45)
    oracle = load_oracle(path)
    prompts = random_prompts(spec.vocab, lens, seed=47)
    model = api.Model(path)
    sess = api.Session(model, len(lens))
    sess.prefill(prompts)
    assert sess.positions().tolist() == [n - 1 for n in lens]
    sess.decode_step()
    got = sess.logits()
    for b in sorted({0, 1 % len(lens), len(lens) - 1}):
        _, want = oracle_rollout(oracle, prompts[b], 1)
        assert logits_error(got[b], want[0]) < TOL_LOWP, b
    sess.close()
    model.close()


@pytest.mark.parametrize("name,lens", [("mha64", [4, 5]), ("gqa4_128", [70]), ("dn_odd", [9, 1, 18, 33, 2]), ("gqa8_64", [65, 64, 63, 8, 1, 16, 17, 130, 3])])
def test_fp32_prompt_columns_match_oracle(api, tmp_path, name, lens):
    """fp32 weights and cache: a prompt of four tokens or more goes through the GEMV chain eight columns to a CTA; the logits behind
    it within the fp32 bound, the ids of the steps that follow identical."""
    spec = dataclasses.replace(SPECS[name], weight_dtype="float32", kv_dtype="float32", max_context=160)
    path = write_model(tmp_path, spec, seed=51)
    oracle = load_oracle(path)
    prompts = random_prompts(spec.vocab, lens, seed=53)
    model = api.Model(path)
    sess = api.Session(model, len(lens))
    for _ in range(2):
        sess.prefill(prompts)
        assert sess.positions().tolist() == [n - 1 for n in lens]
        got = sess.decode(4)
    logits = sess.logits()
    for b in range(len(lens)):
        toks, want = oracle_rollout(oracle, prompts[b], 4)
        assert got[b].tolist() == toks.tolist(), b
        assert logits_error(logits[b], want[-1]) < TOL_FP32, b
    sess.close()
    model.close()


@pytest.mark.parametrize("name", ["mha64", "gqa4_128", "gqa8_64", "dn_odd", "fp8"])
@pytest.mark.parametrize("lens", [[8], [9], [63], [5, 5, 1], [30, 3]])
def test_short_prompts_in_fp32_activations(api, tmp_path, monkeypatch, name, lens):
    """bf16 / FP8 models, one to three sequences, 8 to 63 columns: the GEMV chain; the oracle's logits, and the token
    loop's up to the rounding of single K/V entries."""
    spec = dataclasses.replace(SPECS[name], max_context=96)
    path = write_model(tmp_path, spec, seed=57)
    oracle = load_oracle(path)
    prompts = random_prompts(spec.vocab, lens, seed=59)
    model = api.Model(path)
    got = []
    for mode in ("auto", "step"):
        monkeypatch.setenv("MLB_PREFILL", mode)
        sess = api.Session(model, len(lens))
        sess.prefill(prompts)
        assert sess.positions().tolist() == [n - 1 for n in lens]
        sess.decode_step()
        got.append(sess.logits())
        sess.close()
    model.close()
    assert logits_error(got[0], got[1]) < 2e-3
    for b in range(len(lens)):
        _, want = oracle_rollout(oracle, prompts[b], 1)
        assert logits_error(got[0][b], want[0]) < TOL_LOWP, b


def test_fp8_columns_without_the_bf16_copy(api, tmp_path, monkeypatch):
    """An FP8 model whose bf16 codes cannot be had: its columns run on the decode step's kernels, codes widened tile by tile. At 129
    to 256 columns their k-ranges are those of the column GEMMs, hence the same bits; the copy is used once it can be had."""
    spec = dataclasses.replace(SPECS["fp8"], max_context=700)
    path = write_model(tmp_path, spec, seed=63)
    oracle = load_oracle(path)
    tokens = random_prompts(spec.vocab, [600], seed=65)[0]
    st = oracle.new_state()
    want = np.stack([np.asarray(oracle.step(st, int(t))) for t in tokens])
    model = api.Model(path)
    monkeypatch.setenv("MLB_FP8_COPY", "0")
    sess = api.Session(model, 1)
    got = {}
    for length in (1, 64, 65, 129, 256, 600):
        got[length] = sess.score(tokens[:length])
        assert sess.path(length) == "tcgen05"
        worst = max(logits_error(got[length][i], want[i]) for i in range(length))
        assert worst < TOL_LOWP, (length, worst)
    monkeypatch.delenv("MLB_FP8_COPY")
    copied = {}
    for length in got:
        copied[length] = sess.score(tokens[:length])
        assert sess.path(length) == "cols"
    for length in (129, 256):
        assert np.array_equal(got[length], copied[length]), length
    sess.close()
    model.close()


@pytest.mark.parametrize("name", ["mha64", "gqa4_128", "gqa8_64", "gqa2_128", "fp8"])
def test_columns_do_not_see_later_positions_that_are_no_numbers(api, tmp_path, name):
    """A token whose embedding is infinite makes its K/V rows NaN. Neither the tokens before it in the same chunk nor a later request
    that gets its pages may see them (the token's own logit, from the same row of the tied table, is left out)."""
    spec = dataclasses.replace(SPECS[name], max_context=400, layer_types=["attention"] * SPECS[name].layers)
    weights = synth_weights(spec, seed=67)
    bad = 7
    weights["tokenEmbeddings"][bad] = np.inf
    path = os.path.join(str(tmp_path), "m.bin")
    write_model_bin(path, spec, weights)
    model = api.Model(path)
    text = [t for t in random_prompts(spec.vocab, [320], seed=69)[0] if t != bad]
    fresh = api.Session(model, 1)
    others = np.arange(spec.vocab) != bad
    want = fresh.score(text)[:, others]
    assert np.isfinite(want).all()
    for at in (1, 15, 16, 33, 70, 131, 200):
        got = fresh.score(text[:at] + [bad] * 3 + text[at:])[:, others]
        assert np.array_equal(got[:at], want[:at]), at
        assert np.isnan(got[at]).all()
    fresh.close()
    sess = api.Session(model, 1, max_context=352)
    sess.prefill([[bad] * 350])                               # every page of the pool
    for n in (65, 70, 81, 255):
        sess.prefill([text[:n]])
        sess.decode_step()
        used = sess.logits()[:, others]
        other = api.Session(model, 1, max_context=352)
        other.prefill([text[:n]])
        other.decode_step()
        assert np.isfinite(used).all() and np.array_equal(used, other.logits()[:, others]), n
        other.close()
        sess.prefill([[bad] * 350])
    sess.close()
    model.close()


@pytest.mark.parametrize("weight_dtype", ["bfloat16", "float32"])
def test_prompt_of_a_model_without_attention_whose_heads_state_no_group(api, tmp_path, weight_dtype):
    """64 heads, one kv head, delta-net layers only: no attention tile holds 64 heads, and none is needed."""
    spec = ModelSpec(dim=128, layers=2, heads=64, kv_heads=1, head_dim=64, ffn_dim=256, vocab=128, max_context=96, rms_eps=1e-5, dn_key_dim=64,
                     dn_value_dim=8, layer_types=["delta_net"] * 2, weight_dtype=weight_dtype, kv_dtype="bfloat16")
    path = write_model(tmp_path, spec, seed=71)
    prompt = random_prompts(spec.vocab, [80], seed=73)[0]
    _, want = oracle_rollout(load_oracle(path), prompt, 1)
    model = api.Model(path)
    sess = api.Session(model, 1)
    sess.prefill([prompt])
    sess.decode_step()
    assert logits_error(sess.logits()[0], want[0]) < (TOL_FP32 if weight_dtype == "float32" else TOL_LOWP)
    sess.close()
    model.close()
