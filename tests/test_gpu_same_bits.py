"""Kernels that are built to return the bits of the kernel they replaced, held to it on one model: the projections of a step on mma.sync
and on tcgen05 tiles, the column GEMMs and the column attention against the decode step's kernels, the column form of the delta-net
recurrence (one row of the state per lane group, or four) against the step's."""
import dataclasses

import numpy as np
import pytest

from helpers import random_prompts, write_model
from mini_llm_cuda_b200.model_file import ModelSpec, periodic_layer_types

pytestmark = pytest.mark.gpu

COMMON = dict(kv_dtype="bfloat16", rms_eps=1e-5, max_context=320)
SPECS = {
    # 21 + 1 k-blocks in ranges; a vocabulary that ends inside a tile
    "bf16": ModelSpec(dim=256, layers=4, heads=4, head_dim=64, ffn_dim=1344, ple_dim=64, vocab=500, layer_types=periodic_layer_types(4, 2),
                      weight_dtype="bfloat16", **COMMON),
    "bf16_gqa_gated": ModelSpec(dim=512, layers=2, heads=8, kv_heads=2, head_dim=128, ffn_dim=1408, vocab=512, query_gating=True, weight_dtype="bfloat16", **COMMON),
    "fp8": ModelSpec(dim=512, layers=4, heads=4, kv_heads=1, head_dim=128, ffn_dim=1408, ple_dim=64, vocab=512, layer_types=periodic_layer_types(4, 3),
                     weight_dtype="float8_e4m3", **COMMON),
}
QK_NORM = {
    "bf16_qknorm": ModelSpec(dim=256, layers=2, heads=4, kv_heads=1, head_dim=128, ffn_dim=264, vocab=512, qk_norm=True, query_gating=True,
                             weight_dtype="bfloat16", **COMMON),
}


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


@pytest.mark.parametrize("name", list(SPECS))
def test_step_projections_on_both_tiles(api, tmp_path, monkeypatch, name):
    """Token loop of four tokens, then four greedy steps: ids and logits, 4 to 256 sequences."""
    monkeypatch.setenv("MLB_PREFILL", "step")
    spec = SPECS[name]
    model = api.Model(write_model(tmp_path, spec, seed=101))
    for batch in (4, 17, 37, 64, 130, 256):
        prompts = random_prompts(spec.vocab, [1 + b % 4 for b in range(batch)], seed=103)
        got = {}
        for tiles in ("mma", "tcgen05"):
            monkeypatch.setenv("MLB_GEMM", tiles)
            sess = api.Session(model, batch)
            assert sess.path() == tiles
            names = [k["name"] for k in sess.profile(1, False) if "gemm" in k["name"]]
            assert len(names) >= 4 and all(tiles in n for n in names), names
            sess.prefill(prompts)
            got[tiles] = sess.decode(4), sess.logits()
            sess.close()
        assert np.array_equal(got["mma"][0], got["tcgen05"][0]) and np.array_equal(got["mma"][1], got["tcgen05"][1]), batch
    model.close()


# widths that end 8 and 24 features behind a group of 32 (residual stream) and inside a tile
RAGGED = {
    "bf16_264": ModelSpec(dim=264, layers=2, heads=4, head_dim=64, ffn_dim=328, ple_dim=64, vocab=500, layer_types=periodic_layer_types(2, 2),
                          weight_dtype="bfloat16", **COMMON),
    "bf16_280": ModelSpec(dim=280, layers=2, heads=4, head_dim=64, ffn_dim=1352, vocab=500, weight_dtype="bfloat16", **COMMON),
}


@pytest.mark.parametrize("name", ["bf16", "fp8"])
def test_step_projections_of_more_ctas_than_two_per_sm(api, tmp_path, monkeypatch, name):
    """LM head of 125 or 100 x 3 or 4 CTAs, which run on smaller rings, against the tcgen05 tiles."""
    monkeypatch.setenv("MLB_PREFILL", "step")
    spec = dataclasses.replace(SPECS[name], vocab=4000 if name == "bf16" else 3200)
    model = api.Model(write_model(tmp_path, spec, seed=117))
    for batch in (191, 256):
        prompts = random_prompts(spec.vocab, [1 + b % 2 for b in range(batch)], seed=119)
        got = {}
        for tiles in ("mma", "tcgen05"):
            monkeypatch.setenv("MLB_GEMM", tiles)
            sess = api.Session(model, batch)
            assert sess.path() == tiles
            sess.prefill(prompts)
            got[tiles] = sess.decode(2), sess.logits()
            sess.close()
        assert np.array_equal(got["mma"][0], got["tcgen05"][0]) and np.array_equal(got["mma"][1], got["tcgen05"][1]), batch
    model.close()


@pytest.mark.parametrize("weight_dtype", ["bfloat16", "float8_e4m3"])
def test_wide_step_projections_of_more_ctas_than_two_per_sm(api, tmp_path, monkeypatch, weight_dtype):
    """QKV, delta-net projections, gate/up and residual launches (with and without the next layer's embedding) of 304 to 388 CTAs at 250 and 256
    sequences, stages of one k-block per range, against the tcgen05 tiles."""
    monkeypatch.setenv("MLB_PREFILL", "step")
    spec = ModelSpec(dim=2432, layers=3, heads=16, head_dim=64, ffn_dim=2432, ple_dim=64, vocab=500, max_context=32, rms_eps=1e-5, kv_dtype="bfloat16",
                     layer_types=["attention", "delta_net", "attention"], weight_dtype=weight_dtype)
    model = api.Model(write_model(tmp_path, spec, seed=123))
    for batch in (250, 256):
        prompts = random_prompts(spec.vocab, [1 + b % 2 for b in range(batch)], seed=125)
        got = {}
        for tiles in ("mma", "tcgen05"):
            monkeypatch.setenv("MLB_GEMM", tiles)
            sess = api.Session(model, batch)
            assert sess.path() == tiles
            sess.prefill(prompts)
            got[tiles] = sess.decode(2), sess.logits()
            sess.close()
        assert np.array_equal(got["mma"][0], got["tcgen05"][0]) and np.array_equal(got["mma"][1], got["tcgen05"][1]), batch
    model.close()


@pytest.mark.parametrize("name", [*SPECS, *QK_NORM, *RAGGED])
def test_columns_against_the_decode_steps_kernels(api, tmp_path, monkeypatch, name):
    """129 to 256 columns (one set, whose k-ranges are those that every width takes): every position's logits."""
    spec = {**SPECS, **QK_NORM, **RAGGED}[name]
    model = api.Model(write_model(tmp_path, spec, seed=105))
    text = random_prompts(spec.vocab, [256], seed=107)[0]
    got = {}
    for gemm, path in (("auto", "cols"), ("tcgen05", "tcgen05")):
        monkeypatch.setenv("MLB_GEMM", gemm)
        sess = api.Session(model, 1)
        for n in (129, 200, 256):
            got[gemm, n] = sess.score(text[:n])
            assert sess.path(n) == path
        sess.close()
    for n in (129, 200, 256):
        assert np.array_equal(got["auto", n], got["tcgen05", n]), n
    model.close()


@pytest.mark.parametrize("name", [*SPECS, *QK_NORM, *RAGGED])
def test_column_tiles_over_two_ctas(api, tmp_path, monkeypatch, name):
    """MLB_COLS_PAIR pins the tiles of 256 columns x 256 features of a CTA pair (0: never, 1: wherever they can run): 257 to 1100 columns, the last tile
    of one column, of one CTA's part and nearly whole; every position's logits."""
    spec = dataclasses.replace({**SPECS, **QK_NORM, **RAGGED}[name], max_context=1200)
    model = api.Model(write_model(tmp_path, spec, seed=111))
    text = random_prompts(spec.vocab, [1100], seed=113)[0]
    lens = (257, 384, 500, 512, 513, 1100)
    got = {}
    for pair in "01":
        monkeypatch.setenv("MLB_COLS_PAIR", pair)
        sess = api.Session(model, 1)
        for n in lens:
            got[pair, n] = sess.score(text[:n])
            assert sess.path(n) == "cols"
        sess.close()
    for n in lens:
        assert np.array_equal(got["0", n], got["1", n]), n
    model.close()


@pytest.mark.parametrize("name", ["bf16", "bf16_gqa_gated", "fp8", "fp8_eight_ranges"])
def test_column_gemms_without_sums(api, tmp_path, monkeypatch, name):
    """Kernels with sums in registers may be unusable as a compiler left them: prompts and scores run without them, on column GEMMs that hold every
    range in tensor memory, or where they do not fit on the decode step's (eight ranges of codes and the embedding's)."""
    spec = {**SPECS, "fp8_eight_ranges": dataclasses.replace(SPECS["fp8"], ffn_dim=4096, layers=2, layer_types=["attention"] * 2)}[name]
    model = api.Model(write_model(tmp_path, dataclasses.replace(spec, max_context=700), seed=127))
    text = random_prompts(spec.vocab, [600], seed=129)[0]
    lens = (200,) if name == "fp8_eight_ranges" else (70, 200, 600)
    got = {}
    for sums in (None, "0"):
        if sums:
            monkeypatch.setenv("MLB_COLS_SUMS", sums)
        sess = api.Session(model, 1)
        for n in lens:
            got[sums, n] = sess.score(text[:n])
            assert sess.path(n) == ("tcgen05" if sums and name == "fp8_eight_ranges" else "cols")
        sess.close()
    for n in lens:
        assert np.array_equal(got[None, n], got["0", n]), n
    model.close()


@pytest.mark.parametrize("dk,dv,heads,batch,uneven", [(64, 72, 3, 1, 0), (128, 128, 4, 1, 0), (64, 64, 4, 48, 0), (128, 72, 3, 48, 0), (64, 64, 4, 48, 1),
                                                      (128, 72, 3, 48, 1)])
def test_recurrence_over_columns_against_steps(api, tmp_path, monkeypatch, dk, dv, heads, batch, uneven):
    """fp32 models run prompt columns and steps on the same GEMV chain, so that the recurrence is what differs: one sequence (one row per
    lane group), 48 (four rows), 48 of which one has a long prompt (one row again); twice, in one order and in the other."""
    monkeypatch.setenv("MLB_DECODE_PATH", "chain")
    spec = ModelSpec(dim=192, layers=2, heads=heads, head_dim=64, ffn_dim=256, dn_key_dim=dk, dn_value_dim=dv, vocab=300, max_context=96, rms_eps=1e-5,
                     layer_types=["delta_net"] * 2, weight_dtype="float32", kv_dtype="float32")
    model = api.Model(write_model(tmp_path, spec, seed=109))
    even, one_long = [41 - b % 7 for b in range(batch)], [90 if b == 3 else 2 for b in range(batch)]
    asked = [random_prompts(spec.vocab, lens, seed=111) for lens in ([one_long, even, one_long] if uneven else [even])]
    got = {}
    for mode in ("auto", "step"):
        monkeypatch.setenv("MLB_PREFILL", mode)
        sess = api.Session(model, batch)
        got[mode] = []
        for prompts in asked:
            sess.prefill(prompts)
            assert (sess.path(sum(len(p) - 1 for p in prompts)) != "none") == (mode == "auto")
            sess.decode_step()
            got[mode].append(sess.logits())
        sess.close()
    for a, b in zip(got["auto"], got["step"]):
        assert np.array_equal(a, b)
    model.close()


@pytest.mark.parametrize("name", ["fp8", "bf16", "fp32_qknorm_gated", "fp8_many_heads", "fp32_qknorm_many_heads"])
def test_streamed_gemv_of_several_sequences(api, tmp_path, monkeypatch, name):
    """A CTA of the streamed GEMV takes up to three sequences: each gets the ids and logits that it gets alone. Two to seven
    sequences: whole and ragged groups of one to three; down projections whose input leaves room for fewer (ffn_dim 9216: 108 KB for
    three); QKV cut into so few slabs that a CTA takes one sequence, and into 96 and 128."""
    for key, value in (("MLB_PREFILL", "step"), ("MLB_DECODE_PATH", "chain"), ("MLB_GEMV", "stream"), ("MLB_GEMM", "simt")):
        monkeypatch.setenv(key, value)
    spec = {**SPECS, "fp32_qknorm_gated": ModelSpec(dim=256, layers=2, heads=4, kv_heads=2, head_dim=64, ffn_dim=9216, vocab=500, qk_norm=True, query_gating=True,
                                                    rms_eps=1e-5, max_context=64),
            "fp8_many_heads": dataclasses.replace(SPECS["fp8"], heads=16, kv_heads=4, layers=2, layer_types=["attention"] * 2),
            "fp32_qknorm_many_heads": ModelSpec(dim=128, layers=1, heads=32, head_dim=64, ffn_dim=256, vocab=500, qk_norm=True, query_gating=True,
                                                rms_eps=1e-5, max_context=64)}[name]
    model = api.Model(write_model(tmp_path, spec, seed=113))
    prompts = random_prompts(spec.vocab, [3 + b % 4 for b in range(7)], seed=115)
    sess = api.Session(model, 1)
    want = []
    for p in prompts:
        sess.prefill([p])
        want.append((sess.decode(4)[0], sess.logits()[0]))
    sess.close()
    for batch in (2, 3, 4, 7):
        sess = api.Session(model, batch)
        sess.prefill(prompts[:batch])
        ids, logits = sess.decode(4), sess.logits()
        for b in range(batch):
            assert np.array_equal(ids[b], want[b][0]) and np.array_equal(logits[b], want[b][1]), (batch, b)
        sess.close()
    model.close()
