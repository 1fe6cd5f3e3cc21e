"""GPU parity at the edges of the kernels' tiles and of the rules that choose between them.

Every case compares with the CPU oracle on the same seeded weights (or with an fp64 product), at the sizes where a
kernel hands over to another one or a tile, a slice or a chunk is only partly filled.
"""
import dataclasses

import numpy as np
import pytest

from helpers import BF16_ABS_TOL, assert_logits_close, compare_greedy_stream, dense_pair, quantised_pair, to_bf16_bits, upload_all

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from espresso_b200 import runtime

    runtime.load_library()
    return runtime


def _model(name, n_layer, n_head, n_kv, d, head_dim, hidden, vocab, max_seq):
    from espresso_b200.model_config import MultiModelConfig

    return MultiModelConfig(name, n_layer, n_head, n_kv, d, head_dim, hidden, vocab, max_seq, 1e-5, 10000.0, None, "llama")


@pytest.mark.parametrize("kind", ["f16", "bf16"])
@pytest.mark.parametrize("shape", [(128, 64, 1), (129, 128, 8), (127, 2048, 9), (300, 4096, 16), (640, 1024, 17), (2049, 768, 64), (1000, 704, 65), (257, 2048, 255)])
def test_streamed_product(rt, kind, shape):
    """Rows around the tile widths, ragged output columns, one K block up to many K slices."""
    M, K, N = shape
    rng = np.random.default_rng(M + K + N)
    w = (rng.standard_normal((M, K)) * 0.05).astype(np.float32)
    x = rng.standard_normal((N, K)).astype(np.float32)
    if kind == "f16":
        stored, wr, xr = w.astype(np.float16), w.astype(np.float16).astype(np.float64), x.astype(np.float16).astype(np.float64)
    else:
        stored = to_bf16_bits(w)
        wr, xr = ((b.astype(np.uint32) << np.uint32(16)).view(np.float32).astype(np.float64) for b in (stored, to_bf16_bits(x)))
    y, _ = rt.gemm_tc_bench(kind, stored, M, K, x, warmup=1, iterations=1)
    np.testing.assert_allclose(y, xr @ wr.T, atol=2e-4, rtol=2e-4)


@pytest.mark.parametrize("kind", ["f16", "bf16"])
@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 65, 143, 144, 512, 704, 705])
def test_prompt_rows(rt, oracle_lib, kind, rows):
    """A prompt of 144 rows is the first with the tiled attention (three query heads per KV head), 704 rows the last of the
    streamed products at this width, 705 the first of the paired tiles; hidden 1056 leaves a partial column tile in every product."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-rows", 2, 6, 2, 384, 64, 1056, 520, 768)
    eng, model = dense_pair(rt, oracle_lib, cfg, kind)
    prompt = synthetic_prompt(cfg.vocab, rows)
    eng.prefill(prompt)
    ora = oracle_lib.Runtime(model)
    assert ora.prefill(prompt) == 0
    tol = {} if kind == "f16" else {"abs_tol": BF16_ABS_TOL}
    assert_logits_close(eng.logits(), ora.logits(), f"{kind} {rows} rows", **tol)
    tok = eng.select_greedy_token()
    eng.decode_step(tok)
    assert ora.advance(tok) == 0
    assert_logits_close(eng.logits(), ora.logits(), f"{kind} {rows} rows, one step on", **tol)
    eng.close()


@pytest.mark.parametrize("rows", [768, 832])
def test_query_key_value_product_of_a_prompt(rt, oracle_lib, rows):
    """At 2560 rows of weights 768 is the last prompt whose q/k/v go through the streamed product, 832 the first on the pairs."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-qkv", 1, 20, 10, 1280, 64, 512, 320, 840)
    eng, model = dense_pair(rt, oracle_lib, cfg)
    prompt = synthetic_prompt(cfg.vocab, rows)
    eng.prefill(prompt)
    ora = oracle_lib.Runtime(model)
    assert ora.prefill(prompt) == 0
    assert_logits_close(eng.logits(), ora.logits(), f"{rows} rows")
    eng.close()


@pytest.mark.parametrize("n_head,n_kv,head_dim", [(16, 1, 32), (12, 12, 64), (20, 2, 64), (4, 2, 128), (9, 1, 128)])
@pytest.mark.parametrize("length", [14, 126])
def test_decode_attention_edges(rt, oracle_lib, n_head, n_kv, head_dim, length):
    """Three sequences, contexts that pass a multiple of 16 and of 128 positions; 1 to 16 query heads per KV head."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-attn", 1, n_head, n_kv, n_head * head_dim, head_dim, 512, 320, 160)
    eng, model = dense_pair(rt, oracle_lib, cfg, "f16", 3)
    prompts = np.stack([synthetic_prompt(cfg.vocab, length, stream=s) for s in range(3)])
    streams, _ = eng.generate_batch(prompts, 5)
    for s in range(3):
        compare_greedy_stream(oracle_lib.Runtime(model), prompts[s], streams[s])
    eng.close()


@pytest.mark.parametrize("n_head,head_dim,hidden", [(4, 32, 512), (12, 64, 3072), (3, 128, 1536)])
def test_gpt2_in_the_persistent_kernel(rt, oracle_lib, tmp_models, n_head, head_dim, hidden):
    """One launch for the whole loop, the stream and the state after it equal to the per-stage kernels' and the oracle's."""
    from espresso_b200.model_config import tiny_gpt2
    from espresso_b200.synthetic import synthetic_prompt

    cfg = dataclasses.replace(tiny_gpt2(vocab=515, max_seq=96), nHead=n_head, nKVHead=n_head, headDim=head_dim, dModel=n_head * head_dim, hiddenDim=hidden)
    d = tmp_models(cfg)
    prompt = synthetic_prompt(cfg.vocab, 9)
    ora = oracle_lib.Runtime(oracle_lib.Model.from_dir(d))
    for flags in (0, rt.FLAG_NO_MEGAKERNEL):
        eng = rt.DecodeEngine.build(d, flags=flags)
        eng.prefill(prompt)
        toks, _ = eng.decode(40)
        assert (eng.timings()["kernel_launches"] == 1) == (flags == 0)
        compare_greedy_stream(ora, prompt, toks[0])
        assert ora.prefill(list(prompt) + [int(t) for t in toks[0][:-1]]) == 0
        assert_logits_close(eng.logits(), ora.logits(), f"flags {flags}")
        eng.close()


@pytest.mark.parametrize("kind,n_head,hidden", [("q8_0", 4, 256), ("q8_0", 4, 14592), ("q4_0", 6, 14592)])
def test_quantised_down_projection_in_column_chunks(rt, oracle_lib, kind, n_head, hidden):
    """W2 of the persistent kernel arrives cut along its columns: one short chunk, and chunks with a shorter last one."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-w2", 1, n_head, 2, 128 * n_head, 128, hidden, 300, 48)
    model, uploads = quantised_pair(oracle_lib, cfg, kind)
    eng = rt.DecodeEngine.empty(cfg)
    upload_all(eng, uploads)
    prompt = synthetic_prompt(cfg.vocab, 7)
    res = eng.generate(prompt, 12)
    assert eng.timings()["kernel_launches"] == 1
    compare_greedy_stream(oracle_lib.Runtime(model), prompt, res.tokens)
    eng.close()


@pytest.mark.parametrize("kind,head,n_head,n_kv,head_dim,hidden,vocab", [
    ("f16", "f16", 3, 3, 32, 96, 301),          # fewer K units than warps
    ("f16", "f16", 4, 4, 64, 2048, 600),        # the widest activation vector with cache lines of its own per CTA
    ("f16", "f16", 4, 4, 64, 2080, 600),        # the narrowest compact one
    ("f16", "f16", 6, 2, 64, 2944, 12000),      # gate/up rows in three tiles, the head in two groups
    ("f16", "f16", 12, 12, 64, 7168, 31000),    # gate/up rows in two groups
    ("q8_0", "q8_0", 4, 1, 128, 512, 2000),     # q/k/v rows past one tile
    ("q8_0", "f16", 8, 2, 64, 768, 9000),       # an fp16 head on quantised layers
    ("q4_0", "q4_0", 8, 8, 32, 9728, 26001),    # two groups, a ragged last row
])
def test_row_groups_and_units_of_the_persistent_kernel(rt, oracle_lib, kind, head, n_head, n_kv, head_dim, hidden, vocab):
    """A CTA's gate/up and head rows in one to five tiles and in several groups (q/k/v rows: the test below), K units that do not divide
    among the warps, contexts that pass a warp round (256 positions)."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-groups", 2, n_head, n_kv, n_head * head_dim, head_dim, hidden, vocab, 300)
    if kind == "f16":
        eng, model = dense_pair(rt, oracle_lib, cfg)
    else:
        model, uploads = quantised_pair(oracle_lib, cfg, kind, quantise_head=head != "f16")
        eng = rt.DecodeEngine.empty(cfg)
        upload_all(eng, uploads)
    for length in (9, 250):
        prompt = synthetic_prompt(cfg.vocab, length)
        res = eng.generate(prompt, 14)
        assert eng.timings()["kernel_launches"] == 1
        ora = oracle_lib.Runtime(model)
        compare_greedy_stream(ora, prompt, res.tokens)
        assert_logits_close(eng.logits(), ora.logits(), f"{kind} {length}")
    eng.close()


@pytest.mark.parametrize("kind,n_head,n_kv,head_dim,hidden", [
    ("f16", 4, 4, 128, 32),      # 96 rows in two groups; a CTA's second group takes over from the keys
    ("f16", 10, 5, 128, 64),     # grouped heads, 86 rows: groups of 48 and 38
    ("q8_0", 26, 26, 128, 256),
])
def test_query_key_value_rows_in_several_groups(rt, oracle_lib, kind, n_head, n_kv, head_dim, hidden):
    """A thread of the persistent kernel finishes a rotated pair in one row group and a value pair in the next: decode and the
    two-position pass, the cache that they leave included."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-qkv-groups", 2, n_head, n_kv, n_head * head_dim, head_dim, hidden, 600, 64)
    cfg = dataclasses.replace(cfg, ropeTheta=10.0)  # (the upper pairs of a key turn visibly within a few positions)
    n_cta, qpk = hidden // 2, n_head // n_kv  # (fewer CTAs than SMs: one pair of FFN units each)
    items = (qpk + 2) * head_dim // 2
    rows = 2 * -(-items // (min(n_cta // n_head, items // qpk) * qpk))
    assert 80 < rows <= 160  # five 16-row tiles per group
    if kind == "f16":
        eng, model = dense_pair(rt, oracle_lib, cfg)
    else:
        model, uploads = quantised_pair(oracle_lib, cfg, kind)
        eng = rt.DecodeEngine.empty(cfg)
        upload_all(eng, uploads)
    prompt = synthetic_prompt(cfg.vocab, 9)
    ora = oracle_lib.Runtime(model)
    res = eng.generate(prompt, 14)
    assert eng.timings()["kernel_launches"] == 1
    compare_greedy_stream(ora, prompt, res.tokens)
    assert_logits_close(eng.logits(), ora.logits(), "decode")
    if kind == "f16":
        follow = [int(t) for t in synthetic_prompt(cfg.vocab, 8, stream=1)]
        eng.prefill(prompt)
        assert ora.prefill(prompt) == 0
        for i in range(0, len(follow), 2):
            eng.verify2(follow[i], follow[i + 1])
            assert eng.timings()["kernel_launches"] == 1
            eng.commit(2)
            assert ora.advance(follow[i]) == 0 and ora.advance(follow[i + 1]) == 0
            assert_logits_close(eng.logits(), ora.logits(), f"pair {i // 2}")
    eng.close()


def test_quantised_engines_of_different_widths_take_turns(rt, oracle_lib):
    """A launch finds in shared memory what the other engine's kernel left there: every engine repeats its tokens and logits."""
    from espresso_b200.synthetic import synthetic_prompt

    engines = []
    for kind, n_head, n_kv, hidden in (("q8_0", 8, 4, 1536), ("q8_0", 32, 4, 5632), ("q4_0", 32, 4, 5632)):
        cfg = _model("edge-turns", 2, n_head, n_kv, 64 * n_head, 64, hidden, 2000, 64)
        model, uploads = quantised_pair(oracle_lib, cfg, kind)
        eng = rt.DecodeEngine.empty(cfg)
        upload_all(eng, uploads)
        prompt = synthetic_prompt(cfg.vocab, 11)
        tokens = eng.generate(prompt, 10).tokens
        assert eng.timings()["kernel_launches"] == 1
        logits = eng.logits()
        ora = oracle_lib.Runtime(model)
        compare_greedy_stream(ora, prompt, tokens)
        assert_logits_close(logits, ora.logits(), kind)
        engines.append((eng, prompt, tokens, logits))
    for turn in range(12):
        eng, prompt, tokens, logits = engines[(turn * 5 + turn // 3) % 3]
        np.testing.assert_array_equal(eng.generate(prompt, 10).tokens, tokens)
        np.testing.assert_array_equal(eng.logits(), logits)
    for eng, *_ in engines:
        eng.close()


@pytest.mark.parametrize("kind", ["f16", "q8_0", "q4_0"])
@pytest.mark.parametrize("gain", [1e20, float("nan")])
def test_values_that_overflow_stay_visible(rt, oracle_lib, kind, gain):
    """Gains that overflow the FFN activation: the persistent kernel's last hidden state is not finite, whatever the weights' type."""
    from espresso_b200.synthetic import synthetic_prompt, synthetic_tensors

    cfg = _model("edge-overflow", 1, 4, 2, 256, 64, 512, 320, 32)
    if kind != "f16":
        _, uploads = quantised_pair(oracle_lib, cfg, kind)
    else:
        uploads = [(n, "f16", t.astype(np.float16)) for n, t in synthetic_tensors(cfg, 1234)]
    gains = np.full(cfg.dModel, gain, np.float32)
    eng = rt.DecodeEngine.empty(cfg)
    upload_all(eng, [(n, "f32", gains) if n.endswith("rms_ffn") else (n, k, t) for n, k, t in uploads])
    eng.prefill(synthetic_prompt(cfg.vocab, 5))
    eng.decode(3)
    assert eng.timings()["kernel_launches"] == 1
    assert np.isnan(eng.logits()).all()
    eng.close()


@pytest.mark.parametrize("n_seq", [3, 40, 330])
def test_full_sequence_beside_unfinished_ones(rt, oracle_lib, n_seq):
    """A sequence that has filled its context stays in the batch as an inactive row one position past the rotation table;
    330 rows go through the products on SM pairs."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-full", 2, 4, 2, 256, 64, 512, 320, 24)
    eng, model = dense_pair(rt, oracle_lib, cfg, "f16", n_seq)
    prompts = np.stack([synthetic_prompt(cfg.vocab, 10, stream=s) for s in range(n_seq)])
    eng.prefill_batch(prompts)
    for i in range(cfg.maxSeq - 10):
        eng.decode_step(i % cfg.vocab)  # sequence 0 only
    toks, _ = eng.decode(6, n_seq)
    assert eng.visible_token_count(0) == cfg.maxSeq and len(toks[0]) == 0
    for s in (1, 2, n_seq - 1):
        assert len(toks[s]) == 6
        compare_greedy_stream(oracle_lib.Runtime(model), prompts[s], toks[s])
    eng.close()


def test_failed_prompt_leaves_nothing_to_decode(rt, oracle_lib):
    """A prompt that fails in a later pass: nothing is visible, decode is refused, and the next prompt is served as usual."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-fail", 1, 4, 2, 128, 32, 256, 320, 128)
    n_seq, length = 64, 100  # 6400 rows: two passes
    eng, model = dense_pair(rt, oracle_lib, cfg, "f16", n_seq)
    prompts = np.stack([synthetic_prompt(cfg.vocab, length, stream=s) for s in range(n_seq)])
    bad = prompts.copy()
    bad[-1, -1] = cfg.vocab
    with pytest.raises(rt.RealModelInferenceError):
        eng.prefill_batch(bad)
    assert [eng.visible_token_count(s) for s in range(n_seq)] == [0] * n_seq
    with pytest.raises(rt.RealModelInferenceError):
        eng.decode(2)
    eng.prefill_batch(prompts)
    toks, _ = eng.decode(4, n_seq)
    compare_greedy_stream(oracle_lib.Runtime(model), prompts[-1], toks[-1])
    eng.close()

    model, uploads = quantised_pair(oracle_lib, cfg, "q8_0")
    eng = rt.DecodeEngine.empty(cfg, flags=rt.FLAG_NO_TC_SHADOW)  # row-wise kernels: passes of eight positions
    upload_all(eng, uploads)
    bad = synthetic_prompt(cfg.vocab, 20)
    bad[12] = cfg.vocab
    with pytest.raises(rt.RealModelInferenceError):
        eng.prefill(bad)
    assert eng.visible_token_count() == 0
    with pytest.raises(rt.RealModelInferenceError):
        eng.decode(2)
    prompt = synthetic_prompt(cfg.vocab, 20)
    compare_greedy_stream(oracle_lib.Runtime(model), prompt, eng.generate(prompt, 6).tokens)
    eng.close()


@pytest.mark.parametrize("d_head,offset,spike", [(64, 0.0, 0.0), (64, 32.0, 0.0), (64, 0.0, 30000.0), (1088, 32.0, 0.0)])
def test_gpt2_stream_far_from_zero(rt, oracle_lib, d_head, offset, spike):
    """GPT-2 in the persistent kernel on a residual stream whose mean is a thousand times its deviation, and on one whose largest
    value times its gain is beyond fp16: the LayerNorm has to centre before it squares, and to scale before it rounds.  The stream
    itself is fp32 on both sides: one rounding at 32 is 1e-4 of a deviation of 0.02, well inside the logit tolerances."""
    from espresso_b200.model_config import tiny_gpt2
    from espresso_b200.synthetic import synthetic_prompt, synthetic_tensor
    from espresso_b200.weight_blob import tensor_shapes

    n_head = 3 if d_head == 64 else 17  # 1088: some threads normalise two pairs
    cfg = dataclasses.replace(tiny_gpt2(vocab=515, max_seq=48), nHead=n_head, nKVHead=n_head, headDim=64, dModel=64 * n_head, hiddenDim=256 * n_head)
    eng, model = rt.DecodeEngine.empty(cfg), oracle_lib.Model(cfg.to_metadata())
    for name, shape in tensor_shapes(cfg).items():
        h = synthetic_tensor(cfg, name, shape, 1234).astype(np.float16)
        if name == "embeddings/position":
            h = (h.astype(np.float32) + offset).astype(np.float16)
            h[:, 5] += np.float16(spike)
        if spike and name.endswith("gamma"):
            h[5] = 8.0
        eng.load_tensor(name, "f16", h)
        model.set_tensor(name, h.astype(np.float32))
    eng.finalize()
    prompt = synthetic_prompt(cfg.vocab, 9)
    eng.prefill(prompt)
    toks, _ = eng.decode(12)
    assert eng.timings()["kernel_launches"] == 1
    ora = oracle_lib.Runtime(model)
    compare_greedy_stream(ora, prompt, toks[0])
    assert ora.prefill(list(prompt) + [int(t) for t in toks[0][:-1]]) == 0
    assert_logits_close(eng.logits(), ora.logits(), f"offset {offset} spike {spike}")
    eng.close()


def test_token_rows_receive_their_own_counts(rt, oracle_lib):
    """Behind a sequence's own tokens the caller's buffer keeps what it held, for a batch whose sequences stop at different steps."""
    import ctypes as C

    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-own", 1, 4, 2, 128, 32, 256, 320, 64)
    prompts = np.stack([synthetic_prompt(cfg.vocab, 6, stream=s) for s in range(3)])
    eng, _ = dense_pair(rt, oracle_lib, cfg, "f16", 3)
    free, _ = eng.generate_batch(prompts, 12)
    eng.close()
    # a stop token that ends the sequences at different steps
    at = lambda t: [list(s).index(t) + 1 if t in s else 12 for s in free]
    stop = next(int(t) for t in free[0] if len(set(at(t))) > 1)
    cfg = dataclasses.replace(cfg, eosToken=stop)
    eng, _ = dense_pair(rt, oracle_lib, cfg, "f16", 3)
    eng.prefill_batch(prompts)
    out, n = np.full((3, 12), 0xABCDEF01, np.uint32), np.zeros(3, np.int32)
    rc = eng._lib.esp_cuda_decode(eng._h, 3, 12, out.ctypes.data_as(C.POINTER(C.c_uint32)), n.ctypes.data_as(C.POINTER(C.c_int32)), None)
    assert rc == 0 and list(n) == at(stop)
    for s in range(3):
        assert np.array_equal(out[s, : n[s]], free[s][: n[s]]) and np.all(out[s, n[s] :] == 0xABCDEF01)
    eng.close()


@pytest.mark.parametrize("kind", ["f16", "bf16"])
@pytest.mark.parametrize("rows", [193, 256, 257, 300, 385, 641])
def test_prompt_rows_of_a_wider_model(rt, oracle_lib, kind, rows):
    """d_model 1280: products on 128- and 256-row tiles from 193 rows on, with an almost empty last tile at 257, 385 and 641 rows; the
    residual products are cut along K; hidden 1088 leaves a partial weight tile."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-tiles", 1, 20, 4, 1280, 64, 1088, 320, 700)
    eng, model = dense_pair(rt, oracle_lib, cfg, kind)
    prompt = synthetic_prompt(cfg.vocab, rows)
    eng.prefill(prompt)
    ora = oracle_lib.Runtime(model)
    assert ora.prefill(prompt) == 0
    tol = {} if kind == "f16" else {"abs_tol": BF16_ABS_TOL}
    assert_logits_close(eng.logits(), ora.logits(), f"{kind} {rows} rows", **tol)
    eng.close()


@pytest.mark.parametrize("n_head,head_dim", [(66, 32), (33, 64), (17, 128)])
@pytest.mark.parametrize("rows", [321, 513])
def test_query_key_value_product_on_tiles(rt, oracle_lib, n_head, head_dim, rows):
    """q/k/v with more 128 x 64 tiles than the chip holds: on pairs at 321 rows, on single SMs at 513, RoPE across the columns of a tile."""
    from espresso_b200.synthetic import synthetic_prompt

    cfg = _model("edge-qkv-tiles", 1, n_head, n_head, n_head * head_dim, head_dim, 512, 320, 520)
    eng, model = dense_pair(rt, oracle_lib, cfg)
    prompt = synthetic_prompt(cfg.vocab, rows)
    eng.prefill(prompt)
    ora = oracle_lib.Runtime(model)
    assert ora.prefill(prompt) == 0
    assert_logits_close(eng.logits(), ora.logits(), f"head_dim {head_dim}, {rows} rows")
    eng.close()
