"""Device memory that is not to be had: what fails, what goes on, and what the calls after it see."""
import dataclasses

import numpy as np
import pytest

from helpers import random_prompts, write_model
from mini_llm_cuda_b200.model_file import ModelSpec, periodic_layer_types

pytestmark = pytest.mark.gpu

# wide enough a vocabulary that the logits of 2048 scored columns take 128 MB
WIDE = ModelSpec(dim=128, layers=2, heads=2, head_dim=64, ffn_dim=256, vocab=16384, max_context=1200, rms_eps=1e-5,
                 layer_types=periodic_layer_types(2, 2), weight_dtype="bfloat16", kv_dtype="bfloat16")
SPEC = ModelSpec(dim=128, layers=3, heads=2, head_dim=64, ffn_dim=256, ple_dim=32, vocab=512, max_context=128, rms_eps=1e-5,
                 layer_types=periodic_layer_types(3, 2), weight_dtype="bfloat16", kv_dtype="bfloat16")


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


def test_refused_session_leaves_the_others_alone(api, tmp_path):
    """A K/V pool of terabytes is refused; the next call of another session, whose launches ask the runtime for its last error,
    must not be blamed for it."""
    model = api.Model(write_model(tmp_path, SPEC, seed=81))
    sess = api.Session(model, 2)
    prompts = [[1, 2, 3], [4, 5]]
    sess.prefill(prompts)
    want = sess.decode(4)
    with pytest.raises(api.MlbError) as e:
        api.Session(model, 1, kv_pages=2 ** 31 - 1)
    assert e.value.status == api.MLB_E_NOMEM
    sess.prefill(prompts)
    assert np.array_equal(sess.decode(4), want)
    sess.close()
    model.close()


def free_mb():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0] / 2 ** 20


@pytest.mark.parametrize("limit", [8, 40])
def test_scoring_takes_narrower_chunks_where_wide_ones_do_not_fit(api, tmp_path, monkeypatch, limit):
    """1100 tokens with room for the logits of 64 or 256 columns only: the same bits in more chunks, and no more memory than allowed."""
    model = api.Model(write_model(tmp_path, WIDE, seed=82))
    text = random_prompts(WIDE.vocab, [1100], seed=83)[0]
    sess = api.Session(model, 1)
    want = sess.score(text)
    sess.close()
    sess = api.Session(model, 1)
    sess.score(text[:1])                                   # the narrowest set and its launches exist
    monkeypatch.setenv("MLB_COLUMNS_MB", str(limit))
    before = free_mb()
    got = sess.score(text)
    assert before - free_mb() < limit + 4                  # (the device hands memory out 2 MB at a time)
    assert np.array_equal(got, want)
    sess.close()
    monkeypatch.setenv("MLB_COLUMNS_MB", "0")
    sess = api.Session(model, 1)
    with pytest.raises(api.MlbError) as e:
        sess.score(text)
    assert e.value.status == api.MLB_E_NOMEM
    monkeypatch.delenv("MLB_COLUMNS_MB")
    assert np.array_equal(sess.score(text), want)
    sess.close()
    model.close()


def test_prompts_go_on_without_memory_for_their_columns(api, tmp_path, monkeypatch):
    """Narrower columns, or a wider set at hand, give the same bits; without any, the token loop takes the prompt; with memory
    again, the next prompt is taken by columns again."""
    model = api.Model(write_model(tmp_path, WIDE, seed=84))
    long, short = random_prompts(WIDE.vocab, [1000, 90], seed=85)

    def logits(sess, prompt):
        sess.prefill([prompt])
        assert sess.positions().tolist() == [len(prompt) - 1]
        sess.decode_step()
        return sess.logits()

    sess = api.Session(model, 1)
    by_columns = logits(sess, long), logits(sess, short)
    monkeypatch.setenv("MLB_PREFILL", "step")
    by_steps = logits(sess, long)
    sess.close()
    monkeypatch.delenv("MLB_PREFILL")
    assert not np.array_equal(by_columns[0], by_steps)     # bf16 activations against fp32 ones
    sess = api.Session(model, 1)
    monkeypatch.setenv("MLB_COLUMNS_MB", "0")
    assert np.array_equal(logits(sess, long), by_steps)
    monkeypatch.setenv("MLB_COLUMNS_MB", "1")              # 64 or 128 columns
    assert np.array_equal(logits(sess, long), by_columns[0])
    monkeypatch.delenv("MLB_COLUMNS_MB")
    assert np.array_equal(logits(sess, long), by_columns[0])
    sess.close()
    sess = api.Session(model, 1)
    assert np.array_equal(logits(sess, long), by_columns[0])
    monkeypatch.setenv("MLB_COLUMNS_MB", "1")              # no room beside the wide set: it serves
    assert np.array_equal(logits(sess, short), by_columns[1])
    sess.close()
    model.close()


def test_column_sets_hold_what_their_kernels_use(api, tmp_path, monkeypatch):
    """4096 columns of this model need per column: x and q (512 bytes each), the raw delta-net projection (1552), bf16 operands (256 +
    256 + 512), sums of squares, plan: 15 MB. Partial results of attention splits and of the LM head's pick would add 37 MB."""
    spec = dataclasses.replace(WIDE, max_context=4200)
    model = api.Model(write_model(tmp_path, spec, seed=86))
    sess = api.Session(model, 1)
    monkeypatch.setenv("MLB_COLUMNS_MB", "16")
    sess.prefill(random_prompts(spec.vocab, [4097], seed=87))
    assert sess.path(4096) == "cols"
    sess.close()
    model.close()
