"""The requests that users of this library send it, as cases that can be timed and compared.

A case is one whole request through the public API on a session that the program keeps: a prompt is
taken in and tokens come back, or a text is scored. Three kinds of request:

``generate``  ``prefill`` then ``decode``: the device picks every token itself, the ids come back together.
``stream``    ``prefill`` then one ``decode_step`` per token, the id of each position given by the caller (a
              server that owns the choice of the token: its own sampler, a grammar, a forced continuation).
              Because the text is the caller's, two correct implementations walk the same text, and the
              logits after the last token can be compared.
``score``     ``score``: the logits of every position of a given text.

The models are the repository's own configurations with seeded N(0, 0.02) weights. A program loads its model
and opens its session once and serves many requests with them, so both are kept here between preparations;
what a seed changes is the request: prompts, given ids, sampling keys.
"""
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

from mini_llm_cuda_b200 import api
from mini_llm_cuda_b200 import model_file

MODELS = ("cfg0", "cfg1_ref", "cfg1", "cfg3", "cfg4")
FP32_MODELS = ("cfg0", "cfg1_ref")


def listed():
    return [
        # the next few words for a text field: one user, one short line, latency of every part of the call counts
        {"name": "completion", "call": "generate", "model": "cfg1", "batch": 1, "prompt": 17, "ragged": False, "new": 6, "top_k": 0},
        # the small fp32 configuration as its own benchmark runs it: 32-token prompt, 64 greedy tokens
        {"name": "tiny fp32", "call": "generate", "model": "cfg0", "batch": 1, "prompt": 32, "ragged": False, "new": 64, "top_k": 0},
        # the latency configuration: 128-token prompt, one user who reads along, every id crosses to the host
        {"name": "latency stream", "call": "stream", "model": "cfg1", "batch": 1, "prompt": 128, "ragged": False, "new": 128, "top_k": 0},
        # the model the reference itself can run (fp32, QK-norm, gating), whole answer at once
        {"name": "fp32 answer", "call": "generate", "model": "cfg1_ref", "batch": 1, "prompt": 128, "ragged": False, "new": 128, "top_k": 0},
        # three users of a small service, short questions of uneven length, sampled answers
        {"name": "three users", "call": "generate", "model": "cfg1", "batch": 3, "prompt": 21, "ragged": True, "new": 96, "top_k": 40},
        # a service at part load: an odd number of users, prompts of 1 to 200 tokens
        {"name": "part load", "call": "stream", "model": "cfg1", "batch": 37, "prompt": 200, "ragged": True, "new": 48, "top_k": 0},
        # the batched configuration: 256 users, 256-token prompts, temperature 1 / top-k 50
        {"name": "full load", "call": "stream", "model": "cfg1", "batch": 256, "prompt": 256, "ragged": False, "new": 128, "top_k": 50},
        # the delta-net configuration: 64 users, 64-token prompts, greedy
        {"name": "delta-net", "call": "stream", "model": "cfg3", "batch": 64, "prompt": 64, "ragged": False, "new": 64, "top_k": 0},
        # the FP8 GQA configuration for one user: 512-token prompt
        {"name": "fp8 one user", "call": "stream", "model": "cfg4", "batch": 1, "prompt": 512, "ragged": False, "new": 128, "top_k": 0},
        # the FP8 GQA configuration for 64 users with 512-token prompts: the largest request
        {"name": "fp8 batch", "call": "stream", "model": "cfg4", "batch": 64, "prompt": 512, "ragged": False, "new": 32, "top_k": 0},
        # summary of a long document: the prompt is most of the work
        {"name": "long document", "call": "stream", "model": "cfg4", "batch": 1, "prompt": 3001, "ragged": False, "new": 32, "top_k": 0},
        # likelihood of a given text (evaluation, reranking): every position's logits come back
        {"name": "score text", "call": "score", "model": "cfg1", "batch": 1, "prompt": 500, "ragged": False, "new": 0, "top_k": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another request of the same ranges: 1 to 256 users (64 on the large models, 8 in fp32), prompts from one token
    to most of the context, a few to 160 new tokens, greedy or top-k, equal or uneven lengths."""
    call = rng.choice(("generate", "generate", "stream", "stream", "stream", "stream", "score"))
    if call == "score":
        model = rng.choice(("cfg1", "cfg1", "cfg3", "cfg4"))
        return {"call": call, "model": model, "batch": 1, "prompt": _log_int(rng, 20, 1024), "ragged": False, "new": 0, "top_k": 0}
    top_k = rng.choice((0, 0, _log_int(rng, 2, 200)))
    if call == "generate":
        model = rng.choice(("cfg0", "cfg1_ref", "cfg1", "cfg1"))
        batch = _log_int(rng, 1, 8) if model in FP32_MODELS else rng.choice((1, 1, 2, 3))
        # bf16 prompts below 64 tokens in all, which run on fp32 activations like the decode steps behind them
        prompt = _log_int(rng, 1, 120) if model in FP32_MODELS else _log_int(rng, 2, 63 // batch)
        new = _log_int(rng, 4, 128)
    else:
        model = rng.choice(("cfg1", "cfg1", "cfg3", "cfg4"))
        batch = _log_int(rng, 1, 256 if model == "cfg1" else 64)
        # no more prompt tokens, attended positions and steps than the largest listed request has
        longest = {"cfg1": 800, "cfg3": 1000, "cfg4": 3500}[model]
        most = min({"cfg1": 65536, "cfg3": 16384, "cfg4": 32768}[model] // batch, int((2 ** 24 / batch) ** 0.5))
        prompt = _log_int(rng, 4, min(longest, most))
        new = max(_log_int(rng, 16, 160), -(-100 // batch))
        if model == "cfg4" and batch > 8:
            new = min(new, 32)
    return {"call": call, "model": model, "batch": batch, "prompt": prompt, "ragged": batch > 1 and rng.random() < 0.5,
            "new": new, "top_k": top_k}


# ---- model and session of the running program -----------------------------------------------------------------
_kept = {}


def _matrix(shape, std, dtype, gen):
    """Bytes of one seeded matrix in the container's encoding of `dtype`."""
    w = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * std
    if dtype == "float32":
        return [w.cpu().numpy()]
    if dtype == "bfloat16":
        return [w.to(torch.bfloat16).view(torch.int16).cpu().numpy()]
    scale = w.abs().amax(dim=1, keepdim=True) / 448.0
    return [(w / scale).to(torch.float8_e4m3fn).view(torch.uint8).cpu().numpy(), scale.cpu().numpy()]


def _write_model(path, spec):
    """A model file of `spec` with N(0, 0.02) matrices and unit gains (delta-net gates N(0, 1/dim)), drawn on the GPU: the
    container of model_file.write_model_bin, whose numpy generator would take a minute for the largest model."""
    gen = torch.Generator(device="cuda").manual_seed(0)
    chunks = []

    def tensor(name, shape):
        if len(shape) == 1:
            dtype = "float32"
            chunks.append(np.ones(shape, dtype=np.float32))
        else:
            dtype = spec.weight_dtype
            if dtype == "float8_e4m3" and name in ("pleTable", "pleProjection"):
                dtype = "bfloat16"
            std = spec.dim ** -0.5 if name in ("betaWeights", "decayWeights") else 0.02
            chunks.extend(_matrix(shape, std, dtype, gen))
        return {"shape": list(shape), "dtype": dtype}

    header = {"tokenEmbeddings": tensor("tokenEmbeddings", (spec.vocab, spec.dim)),
              "finalRMSNormGamma": tensor("finalRMSNormGamma", (spec.dim,)), "transformerBlocks": []}
    for b in range(spec.layers):
        shapes = model_file.block_shapes(spec, b)
        order = [k for k in model_file.BASE_KEYS + model_file.QK_NORM_KEYS + model_file.GATING_KEYS if k in shapes]
        header["transformerBlocks"].append({k: tensor(k, shapes[k]) for k in order})
    header["config"] = spec.config_dict()
    header["ext"] = [{"name": k, "block": b, **tensor(k, s)} for b in range(spec.layers) for k, s in model_file.ext_shapes(spec, b).items()]
    text = json.dumps(header).encode("utf-8")
    with open(path, "wb") as f:
        f.write(struct.pack("<Q", len(text)) + text + b"\0" * (-(8 + len(text)) % 8))
        for c in chunks:
            c.tofile(f)


def _session(name, batch):
    """The program's session of `batch` sequences on the named model, opened on first use. One model and one session are
    held at a time."""
    if _kept.get("model_name") != name:
        _kept.clear()
        spec = model_file.named_spec(name)
        with tempfile.TemporaryDirectory() as tmp:
            path = os.path.join(tmp, name + ".bin")
            _write_model(path, spec)
            torch.cuda.empty_cache()
            _kept.update(model=api.Model(path, device=0), model_name=name)
    if _kept.get("batch") != batch:
        _kept.pop("session", None)
        _kept.update(session=api.Session(_kept["model"], batch), batch=batch)
    return _kept["session"]


# ---- one request ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    B, P, n = case["batch"], case["prompt"], case["new"]
    sess = _session(case["model"], B)
    V = sess.model.config.vocab
    rng = np.random.default_rng(seed)
    lens = rng.integers(1, P + 1, size=B) if case["ragged"] else np.full(B, P)
    prompts = [rng.integers(0, V, size=int(k)).astype(np.int32).tolist() for k in lens]
    given = rng.integers(0, V, size=(n, B)).astype(np.int32)
    if n:
        given[0] = [p[-1] for p in prompts]          # the last prompt token is the input of the first step
    sampling = None
    if case["top_k"]:
        sampling = {"mode": "top_k", "top_k": case["top_k"], "temperature": 1.0,
                    "seeds": rng.integers(0, 1 << 62, size=B).astype(np.uint64)}
    return {"call": case["call"], "session": sess, "prompts": prompts, "given": given, "new": n, "sampling": sampling}


def run(state):
    sess = state["session"]
    if state["call"] == "score":
        return sess.score(state["prompts"][0])
    sess.prefill(state["prompts"])
    if state["call"] == "generate":
        ids = sess.decode(state["new"], state["sampling"])
    else:
        ids = np.stack([sess.decode_step(state["sampling"], in_tokens=row) for row in state["given"]], axis=1)
    return {"ids": ids, "logits": sess.logits()}


# ---- what a request cannot do without ---------------------------------------------------------------------------
def work(case):
    """Weights once for the prompt and once for every further token (a step needs the token before it), every cached
    position's K/V row written once and read once per step and once for the prompt, delta-net state read and written once per step,
    the logits that are returned; two flops per weight and token, four per head element and attended position, six per
    delta-net state element and token."""
    spec = model_file.named_spec(case["model"])
    B, n = case["batch"], case["new"]
    P = (case["prompt"] + 1) / 2 if case["ragged"] else case["prompt"]          # mean length
    w_elt = {"float32": 4, "bfloat16": 2, "float8_e4m3": 1}[spec.weight_dtype]
    p_elt = 2 if spec.weight_dtype == "float8_e4m3" else w_elt
    kv_elt = 4 if spec.kv_dtype == "float32" else 2
    weights = w_bytes = 0
    for b in range(spec.layers):
        for k, s in {**model_file.block_shapes(spec, b), **model_file.ext_shapes(spec, b)}.items():
            if len(s) == 2 and k != "pleTable":
                weights += s[0] * s[1]
                w_bytes += s[0] * s[1] * (p_elt if k == "pleProjection" else w_elt)
    head = spec.vocab * spec.dim
    attn = sum(t == model_file.ATTENTION for t in spec.layer_types)
    kv_row = 2 * attn * spec.kv_heads * spec.head_dim * kv_elt
    state = (spec.layers - attn) * spec.heads * spec.dn_key_dim * spec.dn_value_dim
    row = spec.dim * w_elt + spec.layers * spec.ple_dim * p_elt                  # embedding rows of one token
    if case["call"] == "score":
        tokens, head_tokens, steps, attended, kv_reads, returned = P, P, 0, P * (P + 1) / 2, P, P * spec.vocab * 4
    else:
        tokens, head_tokens, steps = P - 1 + n, n, n
        attended = (P - 1 + n) * (P + n) / 2
        kv_reads = P - 1 + n * P + n * (n - 1) / 2
        returned = spec.vocab * 4 + 4 * n
    prompt_passes = 1 if case["call"] == "score" or P > 1 else 0
    n_bytes = (prompt_passes + steps) * w_bytes + (1 if steps == 0 else steps) * head * w_elt
    n_bytes += B * (kv_row * (tokens + kv_reads) + 8 * state * (prompt_passes + steps) + row * tokens + returned)
    flops = B * (2 * weights * tokens + 2 * head * head_tokens + 4 * attn * spec.heads * spec.head_dim * attended + 6 * state * tokens)
    return {"bytes": n_bytes, "flops": flops}


def tolerance(case):
    """Logits: fp32 models sum in fp32 through their layers; the others round activations or the K/V cache to bf16. Ids are
    argmax or inverse-CDF picks of those logits: near ties may fall either way."""
    return {"rel": 2e-5 if case["model"] in FP32_MODELS else 1e-2, "differ": 0.01}
