"""CPU: the host side of the library - model.bin container, C ABI surface, KV page allocator."""
import json
import os
import re
import struct
import sys

import numpy as np
import pytest

from helpers import write_model
from mini_llm_cuda_b200.model_file import (ModelSpec, named_spec, periodic_layer_types, synth_weights,
                                           write_model_bin)
from oracle.model_bin import read_model_bin

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


def declared_functions(header):
    text = open(os.path.join(ROOT, "include", header)).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(mlb_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol(api):
    L = api.lib()
    names = declared_functions("mlb.h") + declared_functions("mini_llm_compat.h")
    assert len(names) > 40
    for n in names:
        assert hasattr(L, n), f"{n} is declared in include/ but not exported"
    assert b"sm_100a" in L.mlb_version()


def test_reference_named_entry_points_are_exported_with_cxx_linkage():
    """runInferenceLoop & co keep the reference's C++ linkage so that a main written against the
    reference's headers links: check the mangled names in the dynamic symbol table."""
    import subprocess
    from mini_llm_cuda_b200.build import LIB_PATH
    out = subprocess.run(["nm", "-D", "--defined-only", LIB_PATH], capture_output=True, text=True).stdout
    for mangled in ("_Z16runInferenceLoopPKciibb", "_Z12runInferencei", "_Z9loadModelPKc", "_Z9loadVocabPKc",
                    "_Z11vocabLookupPKc", "_Z13vocabGetTokeni", "_Z14allocateMemoryb",
                    "_Z16loadStoryContextPKcii", "_Z23getPreComputedRopeThetaPfi", "seqTokenIndices"):
        assert mangled in out, mangled


def test_no_compute_without_gpu_fails_loudly(api, tmp_path):
    import ctypes as C
    n = C.c_int(0)
    # cudaGetDeviceCount is the first CUDA call of mlb_model_load
    path = write_model(tmp_path, ModelSpec(dim=64, layers=1, heads=1, head_dim=64, ffn_dim=64, vocab=32))
    try:
        m = api.Model(path)
    except api.MlbError as e:
        assert e.status == api.MLB_E_CUDA and "no CPU path" in e.message
    else:
        m.close()      # a GPU is present: loading simply works


def test_writer_reader_round_trip_and_layout(tmp_path):
    spec = named_spec("cfg0")
    w = synth_weights(spec, seed=0)
    path = os.path.join(str(tmp_path), "m.bin")
    write_model_bin(path, spec, w)
    raw = open(path, "rb").read()
    (hlen,) = struct.unpack("<Q", raw[:8])
    header = json.loads(raw[8:8 + hlen])
    assert list(header)[:3] == ["tokenEmbeddings", "finalRMSNormGamma", "transformerBlocks"]
    assert list(header["transformerBlocks"][0])[:9] == [
        "rmsGamma", "queryWeights", "keyWeights", "valueWeights", "outputProjectionWeights", "rmsGamma2",
        "feedForwardWeights1A", "feedForwardWeights1B", "feedForwardWeights2"]
    data_off = 8 + hlen + (8 - (8 + hlen) % 8) % 8
    first = np.frombuffer(raw, dtype="<f4", count=4, offset=data_off)
    assert np.array_equal(first, w["tokenEmbeddings"].ravel()[:4])       # row-major, token row contiguous
    m = read_model_bin(path)
    assert np.array_equal(m["tokenEmbeddings"], w["tokenEmbeddings"])
    for b in range(spec.layers):
        for k, v in w["blocks"][b].items():
            assert np.array_equal(m["blocks"][b][k], v), (b, k)
        for k, v in w["ext"][b].items():
            assert np.array_equal(m["ext"][b][k], v), (b, k)
    # execution order N-1 .. 0: block 0 is the last layer, a delta-net one for cfg0
    assert spec.block_type(0) == "delta_net" and "betaWeights" in m["ext"][0]
    assert m["config"]["layer_types"] == ["attention", "delta_net", "attention", "delta_net"]


def test_converter_gives_a_reference_file_its_config(api, tmp_path):
    """A file as the reference's tools write it (fp32, no config key, QK-norm and gating tensors)
    converted to a bf16 file with an embedded config: the product's own Python reader and the C++
    parser agree with the oracle's reader on it, tensors are the nearest-even bf16 of the source, and
    the command-line form writes the same bytes."""
    import subprocess
    import torch
    from mini_llm_cuda_b200 import model_file as mf
    spec = ModelSpec(dim=128, layers=2, heads=2, head_dim=64, ffn_dim=256, vocab=96, qk_norm=True, query_gating=True)
    w = synth_weights(spec, seed=5, random_gains=True)
    src = os.path.join(str(tmp_path), "ref.bin")
    dst = os.path.join(str(tmp_path), "conv.bin")
    write_model_bin(src, spec, w, with_config=False)
    with pytest.raises(ValueError):
        mf.convert_model_bin(src, dst)                      # heads / head_dim are not in a reference file
    out = mf.convert_model_bin(src, dst, heads=2, head_dim=64, file_dtype="bfloat16", weight_dtype="bfloat16",
                               kv_dtype="bfloat16", rms_eps=1e-8, max_context=256)
    assert out.qk_norm and out.query_gating and out.kv_heads == 2 and out.dim == 128 and out.ffn_dim == 256
    header, got = mf.read_model_bin(dst)
    assert header["config"]["weight_dtype"] == "bfloat16" and header["config"]["max_context"] == 256
    m = read_model_bin(dst)                                  # the oracle's reader
    for k in ("queryWeights", "feedForwardWeights2", "gatedQueryWeights"):
        want = torch.from_numpy(w["blocks"][1][k]).to(torch.bfloat16).float().numpy()
        assert np.array_equal(got["blocks"][1][k], want) and np.array_equal(m["blocks"][1][k], want)
    assert np.array_equal(got["blocks"][0]["queryRMSGamma"], w["blocks"][0]["queryRMSGamma"])     # gains stay fp32
    cfg, nbytes = api.inspect_file(dst)
    assert (cfg.heads, cfg.head_dim, cfg.qk_norm, cfg.query_gating, cfg.max_context) == (2, 64, 1, 1, 256)
    dst2 = os.path.join(str(tmp_path), "conv2.bin")
    r = subprocess.run([sys.executable, "-m", "mini_llm_cuda_b200.model_file", "convert", src, dst2, "--heads", "2",
                        "--head-dim", "64", "--file-dtype", "bfloat16", "--weight-dtype", "bfloat16", "--kv-dtype",
                        "bfloat16", "--max-context", "256"], capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert open(dst, "rb").read() == open(dst2, "rb").read()


def test_bf16_file_rounding_is_nearest_even(tmp_path):
    import torch
    spec = ModelSpec(dim=64, layers=1, heads=1, head_dim=64, ffn_dim=64, vocab=32)
    w = synth_weights(spec, seed=3)
    path = os.path.join(str(tmp_path), "b.bin")
    write_model_bin(path, spec, w, file_dtype="bfloat16")
    m = read_model_bin(path)
    want = torch.from_numpy(w["tokenEmbeddings"]).to(torch.bfloat16).float().numpy()
    assert np.array_equal(m["tokenEmbeddings"], want)


def test_file_inspect_and_format_errors(api, tmp_path):
    spec = named_spec("cfg0")
    path = write_model(tmp_path, spec, seed=0)
    cfg, n = api.inspect_file(path)
    assert (cfg.dim, cfg.layers, cfg.heads, cfg.head_dim, cfg.ffn_dim, cfg.vocab) == (256, 4, 4, 64, 768, 4096)
    assert cfg.ple_dim == 32 and list(cfg.layer_types[:4]) == [0, 1, 0, 1] and abs(cfg.rms_eps - 1e-5) < 1e-12
    m = read_model_bin(path)
    n_want = m["tokenEmbeddings"].size + m["finalRMSNormGamma"].size + \
        sum(v.size for b in m["blocks"] for v in b.values()) + sum(v.size for b in m["ext"] for v in b.values())
    assert n == n_want
    raw = open(path, "rb").read()

    def expect(blob, status, name):
        p = os.path.join(str(tmp_path), name)
        open(p, "wb").write(blob)
        with pytest.raises(api.MlbError) as e:
            api.inspect_file(p)
        assert e.value.status == status, e.value

    with pytest.raises(api.MlbError) as e:
        api.inspect_file(os.path.join(str(tmp_path), "absent.bin"))
    assert e.value.status == api.MLB_E_IO
    expect(b"", api.MLB_E_FORMAT, "empty.bin")
    expect(raw[:4], api.MLB_E_FORMAT, "short.bin")
    expect(struct.pack("<Q", 10 ** 12) + raw[8:], api.MLB_E_FORMAT, "hugeheader.bin")
    expect(raw[:len(raw) - 100], api.MLB_E_FORMAT, "truncated.bin")                 # data runs past the end
    (hlen,) = struct.unpack("<Q", raw[:8])
    bad = raw[8:8 + hlen].replace(b'"float32"', b'"float16"', 1)
    expect(struct.pack("<Q", len(bad)) + bad + raw[8 + hlen:], api.MLB_E_FORMAT, "dtype.bin")
    expect(struct.pack("<Q", 5) + b"{oops" + b"\0" * 3, api.MLB_E_FORMAT, "json.bin")
    # a reference-format file says nothing about heads: an override is required
    base = write_model(tmp_path, ModelSpec(dim=128, layers=2, heads=2, head_dim=64, ffn_dim=128, vocab=64),
                       name="base.bin", with_config=False)
    with pytest.raises(api.MlbError) as e:
        api.inspect_file(base)
    assert e.value.status == api.MLB_E_INVALID
    cfg, _ = api.inspect_file(base, api.make_override(heads=2, head_dim=64))
    assert cfg.kv_heads == 2 and cfg.qk_norm == 0 and abs(cfg.rms_eps - 1e-8) < 1e-15
    # wrong head count for the tensor shapes
    with pytest.raises(api.MlbError) as e:
        api.inspect_file(base, api.make_override(heads=3, head_dim=64))
    assert e.value.status == api.MLB_E_FORMAT


def test_kv_page_allocator(api):
    a = api.KvAllocator(num_pages=6, batch=3, max_pages_per_seq=4)
    assert a.ensure(0, 0) == 0 and a.table(0) == []
    assert a.ensure(0, 1) == 0 and a.table(0) == [0]
    assert a.ensure(1, 17) == 0 and a.table(1) == [1, 2]
    assert a.ensure(0, 33) == 0 and a.table(0) == [0, 3, 4]       # pages of a sequence need not be contiguous
    assert a.free_pages() == 1
    assert a.ensure(2, 32) == api.MLB_E_KV_FULL                   # needs two, one left: fails, keeps what it got
    assert b"exhausted" in api.lib().mlb_last_error()
    assert a.free_pages() == 0 and a.table(2) == [5]
    assert a.ensure(1, 65) == api.MLB_E_CONTEXT_FULL              # beyond the page table
    a.release(0)
    assert a.free_pages() == 3 and a.table(0) == []
    assert a.ensure(2, 32) == 0 and len(a.table(2)) == 2
    assert a.ensure(5, 1) == api.MLB_E_INVALID


def test_rope_table_bitwise_equals_oracle(api):
    from oracle.decode_oracle import rope_table
    for L, hd, base in ((256, 64, 10000.0), (1024, 128, 10000.0), (64, 64, 500000.0)):
        assert np.array_equal(api.rope_table(L, hd, base), rope_table(L, hd, base))
    t = api.rope_table(4, 64, 10000.0)
    assert np.all(t[0, 0::2] == 1.0) and np.all(t[0, 1::2] == 0.0)      # position 0: cos 1, sin 0
    assert abs(t[1, 0] - np.cos(1.0)) < 1e-7 and abs(t[1, 1] - np.sin(1.0)) < 1e-7


def test_pool_sharding_matches_the_python_sharding_and_refuses_bad_arguments(api):
    """Host side of the multi-GPU pool without a GPU: the C shard ranges are those of the torchrun driver's
    shard_range (contiguous, the first n % world shards one longer, together covering every sequence once),
    and mlb_pool_new turns down argument errors before it touches a device."""
    import ctypes as C
    from mini_llm_cuda_b200.sharding import shard_range
    for n in (0, 1, 7, 8, 64, 255, 256):
        for world in (1, 2, 3, 4, 8):
            cover = []
            for r in range(world):
                got = api.shard_range_c(n, world, r)
                assert got == shard_range(n, world, r)
                cover += list(range(*got))
            assert cover == list(range(n))
    with pytest.raises(api.MlbError):
        api.shard_range_c(8, 4, 4)
    with pytest.raises(api.MlbError):
        api.shard_range_c(8, 0, 0)
    L = api.lib()
    h = C.c_void_p()
    dev = np.array([0, -1], dtype=np.int32)
    ptr = dev.ctypes.data_as(C.POINTER(C.c_int32))
    assert L.mlb_pool_new(b"nowhere.bin", ptr, 0, 4, 0, None, C.byref(h)) == api.MLB_E_INVALID
    assert L.mlb_pool_new(b"nowhere.bin", ptr, 2, 4, 0, None, C.byref(h)) == api.MLB_E_INVALID      # negative device
    assert L.mlb_pool_new(b"nowhere.bin", ptr, 1, 0, 0, None, C.byref(h)) == api.MLB_E_INVALID      # empty batch
    assert L.mlb_pool_new(None, ptr, 1, 4, 0, None, C.byref(h)) == api.MLB_E_INVALID
    assert not h


def test_fp8_tensors_in_the_model_file(api, tmp_path):
    """Offline FP8: the converter's e4m3 encoder is the hardware rounding (checked against torch's cast on a
    sweep including subnormals, ties and saturation), a float8_e4m3 file holds codes and per-row scales for the
    matrices (bf16 for the per-layer embedding, float32 for the gains), both readers return code * scale, the
    C parser accepts the file, and the file is about a quarter of the float32 one."""
    import torch
    from mini_llm_cuda_b200 import model_file as mf
    from oracle.model_bin import read_model_bin as oracle_read
    rng = np.random.default_rng(0)
    x = np.concatenate([rng.standard_normal(50000).astype(np.float32) * s for s in (1e-3, 0.02, 1.0, 60.0, 300.0)] +
                       [np.array([0, -0.0, 448, -448, 500, -1e9, 2 ** -9, 2 ** -10, 1.5 * 2 ** -9, 2.5 * 2 ** -9, 447.9, 464,
                                  479.9, 15.5 * 2 ** -9, 2 ** -6, 0.99 * 2 ** -6], dtype=np.float32)])
    ref = torch.from_numpy(np.clip(x, -448, 448)).to(torch.float8_e4m3fn).view(torch.uint8).numpy()
    assert np.array_equal(mf._to_e4m3_bits(x), ref)
    spec = mf.ModelSpec(dim=128, layers=2, heads=2, head_dim=64, ffn_dim=256, vocab=512, max_context=64, ple_dim=32,
                        layer_types=mf.periodic_layer_types(2, 2), weight_dtype="float8_e4m3", kv_dtype="bfloat16")
    w = mf.synth_weights(spec, seed=3)
    p32, p8 = os.path.join(str(tmp_path), "f32.bin"), os.path.join(str(tmp_path), "fp8.bin")
    mf.write_model_bin(p32, spec, w)
    mf.write_model_bin(p8, spec, w, file_dtype="float8_e4m3")
    assert os.path.getsize(p8) < 0.3 * os.path.getsize(p32)
    header, back = mf.read_model_bin(p8)
    assert header["transformerBlocks"][0]["queryWeights"]["dtype"] == "float8_e4m3"
    assert header["transformerBlocks"][0]["rmsGamma"]["dtype"] == "float32"
    assert {e["name"]: e["dtype"] for e in header["ext"]}["pleTable"] == "bfloat16"
    q = w["blocks"][0]["queryWeights"]
    codes, scale = mf.quantize_fp8_rows(q)
    want = mf._e4m3_values()[codes] * scale[:, None]
    assert np.array_equal(back["blocks"][0]["queryWeights"], want)
    assert np.abs(want - q).max() <= np.abs(q).max() / 16            # 3 mantissa bits
    assert np.array_equal(oracle_read(p8)["blocks"][0]["queryWeights"], want)
    cfg, n_params = api.inspect_file(p8)
    cfg32, n32 = api.inspect_file(p32)
    assert n_params == n32 and cfg.weight_dtype == api.DT_FP8
    # the converter: float32 file in, FP8 file out by default when the device type is FP8
    dst = os.path.join(str(tmp_path), "conv.bin")
    spec2 = mf.convert_model_bin(p32, dst, weight_dtype="float8_e4m3")
    assert spec2.weight_dtype == "float8_e4m3" and os.path.getsize(dst) == os.path.getsize(p8)
    # a truncated FP8 tensor is refused like any other
    raw = open(p8, "rb").read()
    short = os.path.join(str(tmp_path), "short.bin")
    open(short, "wb").write(raw[:len(raw) - 64])
    with pytest.raises(api.MlbError):
        api.inspect_file(short)


def run_host_program(tmp_path, includes, body):
    """What a C++ program with `body` as its main prints, built against the library's host headers."""
    import subprocess
    src, exe = os.path.join(str(tmp_path), "p.cc"), os.path.join(str(tmp_path), "p")
    with open(src, "w") as f:
        f.write("".join(f"#include {i}\n" for i in includes) + "int main() {\n" + body + "\nreturn 0; }\n")
    csrc = os.path.join(ROOT, "mini_llm_cuda_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", csrc, src, "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout


def test_sequences_of_a_streamed_gemv_cta(tmp_path):
    """Every sequence has a CTA, no more waves than groups of three need, no group larger than its wave asks for, none at all where
    the CTAs fit side by side."""
    out = run_host_program(tmp_path, ["<cstdio>", '"step_shapes.h"'], """
        for (int b = 1; b <= 64; ++b)
            for (int slabs = 1; slabs <= 148; ++slabs) std::printf("%d %d %d\\n", b, slabs, mlb::sg_sequences(b, slabs, 148));""")
    for batch, slabs, n in (map(int, line.split()) for line in out.splitlines()):
        rows = -(-batch // n)
        assert 1 <= n <= 3 and rows * n >= batch
        assert rows * slabs <= 148 or rows <= -(-batch // 3), (batch, slabs, n)      # more rows than groups of three make only in one wave
        assert n == 1 or rows < -(-batch // (n - 1)), (batch, slabs, n)              # with one sequence less to a CTA there would be more rows
        if batch * slabs <= 148:
            assert n == 1, (batch, slabs, n)
        if slabs > 74 and batch in (2, 3, 4):
            assert n == {2: 2, 3: 3, 4: 2}[batch], (batch, slabs, n)


def test_splits_in_turn_follow_the_devices_sms(tmp_path):
    """One CTA takes a sequence's splits in turn where sequences and groups of heads give every SM of the device a CTA, whatever its number."""
    out = run_host_program(tmp_path, ["<cstdio>", '"step_shapes.h"'], """
        for (int sms : {20, 132, 148, 160})
            for (int splits : {1, 4, 5})
                for (long n : {sms - 1L, (long)sms}) std::printf("%d %ld %d %d\\n", splits, n, sms, (int)mlb::attn_splits_in_turn(splits, n, sms));""")
    lines = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(lines) == 24
    for splits, n, sms, turn in lines:
        assert turn == (splits <= 4 and n >= sms)


def test_attention_ctas_stand_side_by_side(tmp_path):
    """Rings of decode attention over fp32 K/V leave as many CTAs room on an SM as registers do, or as the launch has; whole pages where
    they fit."""
    out = run_host_program(tmp_path, ["<cstdio>", '"step_shapes.h"'], """
        for (int kv : {2, 4})
            for (int hd : {64, 128})
                for (int heads : {1, 2, 4, 8})
                    for (long ctas = 1; ctas <= 1000; ++ctas) {
                        const bool pages = mlb::attn_whole_pages(kv, hd, heads, ctas, 148);
                        std::printf("%d %d %d %ld %d %d %ld %ld\\n", kv, hd, heads, ctas, (int)pages, mlb::attn_resident(heads),
                                    mlb::attn_smem(kv, hd, heads, pages ? 16 : mlb::attn_few_rows(kv, hd, heads)), mlb::attn_smem(kv, hd, heads, 16));
                    }""")
    seen = set()
    for kv, hd, heads, ctas, pages, resident, smem, smem_pages in (map(int, line.split()) for line in out.splitlines()):
        per_sm = min(resident, -(-ctas // 148))
        if kv == 4:
            assert per_sm * (smem + 2048) <= 227 * 1024, (hd, heads, ctas)
            assert pages or per_sm * (smem_pages + 2048) > 227 * 1024, (hd, heads, ctas)
        else:
            assert pages
        seen.add((kv, hd, heads, pages))
    assert len([x for x in seen if not x[3]]) == 4      # fp32: 64 x 1 head, 128 x 1, 2 and 4
    out = run_host_program(tmp_path, ["<cstdio>", '"step_shapes.h"'], """
        std::printf("%ld %ld %ld %ld\\n", mlb::attn_ctas_with_work(64, 10, 64, 11), mlb::attn_ctas_with_work(400, 1, 64, 11),
                    mlb::attn_ctas_with_work(6, 8, 1, 1), mlb::attn_ctas_with_work(6, 8, 100, 0));""")
    assert out.split() == ["128", "400", "6", "48"]


def test_rings_of_decode_gemms_hold_two_stages(tmp_path):
    """A launch of more CTAs than two per SM takes the least of a quarter, half and whole ring in which a copy can run under the products;
    gate/up launches and those of fewer CTAs the whole ring."""
    out = run_host_program(tmp_path, ["<cstdio>", '"step_shapes.h"'], """
        const size_t whole = 108 * 1024;
        for (long ctas : {1, 296, 297, 1024})
            for (int gate_up = 0; gate_up < 2; ++gate_up)
                for (size_t kb = 4; kb <= 160; kb += 2)
                    std::printf("%ld %d %zu %zu\\n", ctas, gate_up, kb, mlb::gd_ring(whole, ctas, 148, gate_up, kb * 1024) / 1024);""")
    for ctas, gate_up, two_stages, ring in (map(int, line.split()) for line in out.splitlines()):
        if ctas <= 296 or gate_up:
            assert ring == 108
        else:
            assert ring in (27, 54, 108) and (ring >= two_stages or ring == 108)
            assert ring == 27 or two_stages > ring // 2


def test_prompt_chunks_are_full(tmp_path):
    """Shares of a chunk, in whole attention tiles where they can be: every chunk but the last is full, so a prompt takes as many chunks as its tokens
    need; equal prompts get whole tiles."""
    out = run_host_program(tmp_path, ["<cstdio>", '"step_shapes.h"'], """
        unsigned state = 1;
        auto rnd = [&](int n) { state = state * 1664525u + 1013904223u; return (int)((state >> 8) % (unsigned)n); };
        for (int round = 0; round < 4000; ++round) {
            const int batches[] = {1, 2, 3, 8, 37, 64, 200, 256}, B = batches[rnd(8)], longest = 1 + rnd(16000 / B), tile = (round % 4) ? 32 >> rnd(4) : 0;
            std::vector<int> rest(B), cursor(B, 0), take;
            long left = 0;
            for (int& r : rest) left += r = rnd(5) ? rnd(longest + 1) : longest;
            while (left > 0) {
                const int want = (int)std::min<long>(left, 4096);
                mlb::cols_shares(rest, cursor, want, tile, take);
                long n = 0;
                int parts = 0, bad = 0;
                for (int b = 0; b < B; ++b) {
                    bad += take[b] < 0 || take[b] > rest[b];
                    parts += tile > 0 && take[b] % tile != 0 && take[b] < rest[b];
                    n += take[b];
                    rest[b] -= take[b];
                    cursor[b] += take[b];
                }
                std::printf("%d %ld %d %d %d\\n", want, n, bad, tile, parts);
                if (n != want) return 0;
                left -= n;
            }
        }""")
    lines = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(lines) > 4000
    for want, n, bad, tile, parts in lines:
        assert n == want and bad == 0
        assert tile == 0 or parts <= 1 or want < 32 * 8, (want, tile, parts)


def test_scores_over_sqrt128_are_the_division(tmp_path):
    """Prompt attention at head size 128 multiplies by a two-word reciprocal: the quotient for every significand, in a middle binade and
    at both ends of the range in which it is meant to be exact; infinities, zeros and what is no number stay."""
    out = run_host_program(tmp_path, ["<cstdio>", "<cstdint>", "<cstring>", "<initializer_list>", '"cols_math.h"'], """
        volatile float divisor = std::sqrt(128.0f);
        const float d = divisor;
        long wrong = 0;
        for (uint32_t exponent : {127u, 127u - 90u, 254u})
            for (uint32_t frac = 0; frac < (1u << 23); ++frac) {
                const uint32_t bits = (exponent << 23) | frac;
                float x;
                std::memcpy(&x, &bits, 4);
                wrong += mlb::over_sqrt128(x) != x / d;
                wrong += mlb::over_sqrt128(-x) != -x / d;
            }
        std::printf("%ld %g %g %g %g %d\\n", wrong, mlb::over_sqrt128(INFINITY), mlb::over_sqrt128(-INFINITY), mlb::over_sqrt128(0.f), mlb::over_sqrt128(-0.f),
                    (int)std::isnan(mlb::over_sqrt128(NAN)));""")
    assert out.split() == ["0", "inf", "-inf", "0", "-0", "1"]
