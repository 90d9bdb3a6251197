"""Model-level parity on the GPU: Engine::forward / generate through the C ABI against the CPU oracle,
on identical synthetic weights."""
import numpy as np
import pytest

from conftest import assert_close, make_pair

pytestmark = pytest.mark.gpu

LOGIT_ABS, LOGIT_REL = 1e-2, 1e-3  # the stated bar for logits


def small_spec(layer_type, embed_type, head_type, layers=2, hidden=256, heads=8, kv=2, ffn=512, vocab=1000):
    from leafcutterllm_b200.synth import ModelSpec
    return ModelSpec("small", layers, hidden, heads, kv, ffn, vocab, 10000.0, layer_type, embed_type, head_type)


@pytest.mark.parametrize("types", [(12, 12, 12), (2, 8, 8), (8, 8, 8)])
def test_forward_and_generate_small(gpu, oracle, types):
    from leafcutterllm_b200 import synth
    spec = small_spec(*types)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=128)
    prompt = synth.prompt_tokens(17, spec.vocab_size)
    got = eng.forward(prompt)
    want = om.forward(prompt)
    assert_close(got, want, LOGIT_ABS, LOGIT_REL, "prefill logits")
    assert eng.kv_length() == 17
    assert eng.kv_memory_bytes() == om.kv_memory_bytes()  # rust/src/cache/mod.rs:80-84
    nxt = int(np.argmax(want))
    assert_close(eng.forward([nxt]), om.forward([nxt]), LOGIT_ABS, LOGIT_REL, "decode logits")
    toks = eng.generate(prompt, 24, stop_on_eos=False)
    ref, margins = om.generate(prompt, 24, stop_on_eos=False, want_margins=True)
    assert toks == ref, f"greedy tokens differ; oracle top-2 margins {margins}"
    # per-token callback path and the device-resident loop give the same tokens
    seen = []
    assert eng.generate(prompt, 24, stop_on_eos=False, on_token=seen.append) == ref and seen == ref
    eng.close()


@pytest.mark.parametrize("on_device", [False, True])
def test_q4_k_m_mix_with_generated_weights(gpu, oracle, on_device):
    """Eight layers with the type mix of a "Q4_K_M" file (Q6_K head; Q6_K attn_v and ffn_down in layers 0, 3, 6, 7), weights
    from the generator's own Q4_K and Q6_K quantisers on the host and on the device: prefill logits, a decode step and
    greedy tokens against the oracle."""
    from leafcutterllm_b200 import synth
    from leafcutterllm_b200.synth import ModelSpec
    spec = ModelSpec("small-q4_k_m", 8, 256, 8, 2, 768, 1008, 10000.0, 12, 12, 12, mix="q4_k_m")
    assert [l for l in range(8) if spec.mixed_type(l, "down") == 14] == [0, 3, 6, 7]
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=96, on_device=on_device)
    prompt = synth.prompt_tokens(21, spec.vocab_size, 5)
    want = om.forward(prompt)
    assert_close(eng.forward(prompt), want, LOGIT_ABS, LOGIT_REL, "prefill logits")
    nxt = int(np.argmax(want))
    assert_close(eng.forward([nxt]), om.forward([nxt]), LOGIT_ABS, LOGIT_REL, "decode logits")
    ref, margins = om.generate(prompt, 20, stop_on_eos=False, want_margins=True)
    assert eng.generate(prompt, 20, stop_on_eos=False) == ref, margins
    eng.close()


def test_layer_probes(gpu, oracle):
    spec = small_spec(12, 12, 12, layers=1, hidden=512, heads=8, kv=4, ffn=768)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=64)
    r = np.random.default_rng(0)
    x = r.standard_normal((5, 512)).astype(np.float32)
    assert_close(eng.probe_ffn(0, x), om.ffn(0, x), 1e-5, 1e-4, "ffn")
    assert_close(eng.probe_attention(0, x), om.attention(0, x), 1e-4, 1e-3, "attention (5 tokens)")
    x1 = r.standard_normal((1, 512)).astype(np.float32)
    assert_close(eng.probe_attention(0, x1), om.attention(0, x1), 1e-4, 1e-3, "attention (next token over the cache)")
    eng.close()


@pytest.mark.parametrize("kw", [dict(kv_dtype="f32"), dict(rope_mode="absolute"), dict(kv_page_tokens=4)])
def test_switches(gpu, oracle, kw):
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=96, **kw)
    prompt = synth.prompt_tokens(33, spec.vocab_size, 3)
    assert_close(eng.forward(prompt), om.forward(prompt), LOGIT_ABS, LOGIT_REL, f"prefill {kw}")
    assert eng.generate(prompt, 12, stop_on_eos=False) == om.generate(prompt, 12, stop_on_eos=False)
    eng.close()


def test_chunked_prefill_matches(gpu, oracle):
    """700 tokens in one pass, eleven tiles of prompt attention, call-relative RoPE indices (longer than a pass: test_prompt_longer_than_a_pass)."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=1, hidden=256, heads=4, kv=4, ffn=256, vocab=500)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=800)
    prompt = synth.prompt_tokens(700, spec.vocab_size, 1)
    assert_close(eng.forward(prompt), om.forward(prompt), LOGIT_ABS, LOGIT_REL, "700-token prefill")
    eng.close()


@pytest.mark.parametrize("rows", [16, 63, 65, 130])  # one tile with idle warps, a row short of a tile, one more, two full ones and a short one
@pytest.mark.parametrize("hd,kv_dtype,page", [(32, "f16", 16), (32, "f32", 5), (64, "f32", 16), (64, "f16", 32), (128, "f32", 16), (128, "f16", 8), (256, "f16", 16), (256, "f32", 16)])
def test_prompt_attention_in_tiles(gpu, oracle, monkeypatch, hd, kv_dtype, page, rows):
    """Head sizes, cache types and page sizes that the tensor-core prompt attention does not take; a second run of rows behind the first,
    so that tiles begin past position 0.  The host's and the device's powf differ by an ulp or two, which is 260 * 2^-22 = 6e-5 of an angle at the
    last position and of the scores' order: 2e-4 of the largest output; an f16 cache may round a key or value the other way (2^-11 of it): 1e-3."""
    monkeypatch.setenv("LC_ATTN_ROWS", "1")  # these few heads are faster through the kernel that splits contexts
    spec = small_spec(12, 12, 12, layers=1, hidden=512, heads=512 // hd, kv=max(1, 256 // hd), ffn=256, vocab=64)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=2 * rows, kv_dtype=kv_dtype, kv_page_tokens=page, rope_mode="absolute")
    x = np.random.default_rng(hd + rows).standard_normal((2 * rows, 512)).astype(np.float32)
    for part in (x[:rows], x[rows:]):
        got, want = eng.probe_attention(0, part), om.attention(0, part)
        assert_close(got, want, (2e-4 if kv_dtype == "f32" else 1e-3) * np.abs(want).max(), 0, f"{rows} rows of {hd}")
    eng.close()


@pytest.mark.parametrize("rows,tiles", [(16, False), (128, True)])
def test_prompt_attention_takes_the_faster_kernel(gpu, monkeypatch, rows, tiles):
    """Behind 1,000 tokens: 16 rows of 32 heads are faster with the context split (a tile would walk it alone), 128 rows in two tiles.  The kernels add in different
    orders, so their outputs tell which one ran; sums of 1,128 weights and 2,048 products in f32 differ by 1e-5 of the largest output at most."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=1, hidden=2048, heads=32, kv=4, ffn=256, vocab=64)
    eng = synth.build_engine(spec, 1200, on_device=True, kv_dtype="f32", rope_mode="absolute")
    x = np.random.default_rng(rows).standard_normal((1000 + rows, 2048)).astype(np.float32)

    def run():
        eng.kv_clear()
        eng.probe_attention(0, x[:500])
        eng.probe_attention(0, x[500:1000])
        return eng.probe_attention(0, x[1000:])

    got = run()
    monkeypatch.setenv("LC_ATTN_ROWS", "1")
    by_rows = run()
    monkeypatch.setenv("LC_ATTN_ROWS", "0")
    split = run()
    assert not np.array_equal(by_rows, split)
    assert_close(by_rows, split, 1e-5 * np.abs(split).max(), 0, "the two kernels")
    assert np.array_equal(got, by_rows if tiles else split)
    eng.close()


@pytest.mark.parametrize("tiles", ["1", "0"])
def test_prompt_attention_where_the_first_keys_score_minus_infinity(gpu, oracle, monkeypatch, tiles):
    """The last 20 rows' scores with keys 0 ... 63 fall below f32's range: the softmax over the other keys is what it would be without them.  One head of
    256 whose 100th dim is not rotated (theta^-200/256); there the first rows' keys have -1e34 and the last rows' queries 1e6, elsewhere both next to nothing.  The
    bound is test_prompt_attention_in_tiles's, row by row."""
    monkeypatch.setenv("LC_ATTN_ROWS", tiles)
    from dataclasses import replace
    from leafcutterllm_b200 import synth
    spec = replace(small_spec(12, 12, 12, layers=1, hidden=256, heads=1, kv=1, ffn=256, vocab=64), rope_theta=1e30)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=160, kv_dtype="f32", rope_mode="absolute")
    names = {name: (typ, dims, kind) for name, typ, dims, kind in spec.tensors()}

    def input_for(which, value):  # the row that the layer's matrix turns into `value` in dim 100 and zero elsewhere
        name = f"blk.0.attn_{which}.weight"
        typ, dims, kind = names[name]
        w = oracle.dequantize(typ, synth.tensor_bytes(spec, name, typ, dims, kind, 1234), 256 * 256).reshape(256, 256)
        return np.linalg.solve(w.astype(np.float64), value * np.eye(256)[100])

    r = np.random.default_rng(3)
    scale = lambda n: 1 + r.random((n, 1))
    first = np.concatenate([input_for("k", -1e34) * scale(64), 1e-6 * r.standard_normal((64, 256))]).astype(np.float32)
    last = (input_for("q", 1e6) * scale(20)).astype(np.float32)
    om.attention(0, first)
    want = om.attention(0, last)
    assert np.isfinite(want).all()
    eng.probe_attention(0, first)
    got = eng.probe_attention(0, last)
    for i in range(20):
        assert_close(got[i], want[i], 2e-4 * np.abs(want[i]).max(), 0, f"row {i}")
    eng.close()


def test_a_piece_that_begins_with_scores_of_minus_infinity(gpu, oracle, monkeypatch):
    """As above, but only keys 0, 1 and 2 of a piece fall below f32's range, the first that three groups of lanes meet: the other keys of the piece keep their weights."""
    monkeypatch.setenv("LC_ATTN_ROWS", "0")
    from dataclasses import replace
    from leafcutterllm_b200 import synth
    spec = replace(small_spec(12, 12, 12, layers=1, hidden=256, heads=1, kv=1, ffn=256, vocab=64), rope_theta=1e30)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=160, kv_dtype="f32", rope_mode="absolute")
    names = {name: (typ, dims, kind) for name, typ, dims, kind in spec.tensors()}

    def input_for(which, value):
        name = f"blk.0.attn_{which}.weight"
        typ, dims, kind = names[name]
        w = oracle.dequantize(typ, synth.tensor_bytes(spec, name, typ, dims, kind, 1234), 256 * 256).reshape(256, 256)
        return np.linalg.solve(w.astype(np.float64), value * np.eye(256)[100])

    r = np.random.default_rng(4)
    first = np.concatenate([input_for("k", -1e34) * (1 + r.random((3, 1))), 1e-6 * r.standard_normal((61, 256))]).astype(np.float32)
    last = (input_for("q", 1e6) * (1 + r.random((20, 1)))).astype(np.float32)
    om.attention(0, first)
    want = om.attention(0, last)
    assert np.isfinite(want).all()
    eng.probe_attention(0, first)
    got = eng.probe_attention(0, last)
    for i in range(20):
        assert_close(got[i], want[i], 2e-4 * np.abs(want[i]).max(), 0, f"row {i}")
    eng.close()


@pytest.mark.parametrize("types,heads", [((12, 12, 12), 2), ((2, 8, 8), 8)])
def test_prompt_longer_than_a_pass(gpu, oracle, types, heads):
    """2,100 tokens: a full pass of 2,048 and a short one behind it; heads of 128 (tiles on the tensor cores) and of 32 (tiles in f32, then the kernel that
    splits contexts)."""
    from leafcutterllm_b200 import synth
    spec = small_spec(*types, layers=1, hidden=256, heads=heads, kv=heads, ffn=256, vocab=300)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=2112)
    prompt = synth.prompt_tokens(2100, spec.vocab_size, 1)
    assert_close(eng.forward(prompt), om.forward(prompt), LOGIT_ABS, LOGIT_REL, "2100-token prefill")
    eng.close()


def test_many_short_runs_attend_in_slices(gpu, oracle):
    """130 sequences of five tokens are 650 tokens in tiles of five, too few for tiled attention: the split-context kernel takes 512 tokens and then 138
    (sequence 102 lies on the border), with one scratch and one set of counters for both.  Then five more tokens each, behind the first."""
    from leafcutterllm_b200 import synth
    spec = small_spec(2, 8, 8, layers=2, hidden=256, heads=8, kv=8, ffn=256, vocab=300)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=16, max_seqs=130)
    ids = list(range(130))
    calls = [[synth.prompt_tokens(5, spec.vocab_size, 1000 * c + i).tolist() for i in ids] for c in range(2)]
    got = [eng.forward_batch(ids, parts)[0] for parts in calls]
    for i in (0, 1, 50, 101, 102, 103, 128, 129):
        om.kv_clear()
        for c in range(2):
            assert_close(got[c][i], om.forward(calls[c][i]), LOGIT_ABS, LOGIT_REL, f"sequence {i}, call {c}")
    eng.close()


def test_batched_sequences_match_single(gpu, oracle):
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=64, max_seqs=5)
    prompts = [synth.prompt_tokens(n, spec.vocab_size, i).tolist() for i, n in enumerate([3, 20, 1, 9, 16])]
    logits, nxt = eng.forward_batch([0, 1, 2, 3, 4], prompts)
    for i, p in enumerate(prompts):
        om.kv_clear()
        want = om.forward(p)
        assert_close(logits[i], want, LOGIT_ABS, LOGIT_REL, f"sequence {i}")
        assert nxt[i] == oracle.argmax(want)
    # four decode steps for all five sequences on the device == four oracle steps each
    toks, _ms = eng.decode_loop([0, 1, 2, 3, 4], nxt, 4)
    for i, p in enumerate(prompts):
        ref = om.generate(p, 5, stop_on_eos=False)
        assert [int(nxt[i])] + toks[:, i].tolist() == ref
    assert eng.counters()["kv_pages_in_use"] == sum((len(p) + 4 + 15) // 16 for p in prompts)
    eng.kv_clear(1)
    assert eng.kv_length(1) == 0 and eng.kv_length(0) == 3 + 4
    eng.close()


def test_many_sequences_decode_through_the_tensor_core_gemm(gpu, oracle):
    """Twelve sequences: the ragged prefill (49 tokens in one call) and every decode step (12 tokens) go through the
    many-token tcgen05 product instead of the matrix-vector kernels; tokens must still equal the oracle's, sequence by
    sequence, and a second engine must reproduce the first bit for bit (one issuing order, no atomics)."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=2, hidden=512, heads=4, kv=2, ffn=768, vocab=640)
    lens = [3, 7, 1, 9, 2, 5, 4, 6, 1, 3, 2, 6]
    ids = list(range(12))
    prompts = [synth.prompt_tokens(n, spec.vocab_size, 40 + i).tolist() for i, n in enumerate(lens)]
    runs = []
    for _ in range(2):
        eng, om = make_pair(gpu, oracle, spec, max_seq_len=48, max_seqs=12)
        logits, nxt = eng.forward_batch(ids, prompts)
        toks, _ms = eng.decode_loop(ids, nxt, 6)
        runs.append((logits.copy(), nxt.copy(), toks.copy()))
        if len(runs) == 1:
            for i, p in enumerate(prompts):
                om.kv_clear()
                assert_close(logits[i], om.forward(p), LOGIT_ABS, LOGIT_REL, f"sequence {i}")
                ref, margins = om.generate(p, 7, stop_on_eos=False, want_margins=True)
                assert [int(nxt[i])] + toks[:, i].tolist() == ref, (i, margins)
        eng.close()
    assert np.array_equal(runs[0][0].view(np.uint32), runs[1][0].view(np.uint32))
    assert np.array_equal(runs[0][2], runs[1][2])


def test_batched_decode_attention_over_several_context_pieces(gpu, oracle):
    """80 sequences x 8 heads of 128 dims = 640 (token, head) pairs: past four per SM, so the batched decode step runs
    the split-context attention kernel with the context cut into 1024-key pieces and the pieces merged through the
    scratch partials.  Contexts sit on both sides of the piece edges (1023 / 1024 / 1025, 2047 / 2049, 4090) and most are
    short, so many (pair, piece) CTAs have no key at all and leave at once.  Prefill logits and four decode steps are
    compared with the oracle sequence by sequence."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=1, hidden=1024, heads=8, kv=2, ffn=512, vocab=512)
    special = [5, 1023, 1024, 1025, 2047, 2049, 2500, 4090]
    r = np.random.default_rng(5)
    lens = special + [int(v) for v in r.integers(1, 200, 80 - len(special))]
    ids = list(range(80))
    steps = 4
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=4096, max_seqs=80, kv_pool_tokens=sum((n + steps + 15) // 16 * 16 for n in lens))
    prompts = [synth.prompt_tokens(n, spec.vocab_size, 100 + i).tolist() for i, n in enumerate(lens)]
    logits, nxt = eng.forward_batch(ids, prompts)
    step_logits, cur = [], nxt.copy()
    for _ in range(steps):  # every sequence advances by one token per call: the 80-token batched decode step
        lg, cur = eng.forward_batch(ids, [[int(t)] for t in cur])
        step_logits.append(lg.copy())
    for i, p in enumerate(prompts):
        if i >= len(special) and i % 6:  # every special context and a sample of the short ones go through the oracle
            continue
        om.kv_clear()
        want = om.forward(p)
        assert_close(logits[i], want, LOGIT_ABS, LOGIT_REL, f"prefill of sequence {i} ({lens[i]} tokens)")
        for s_ in range(steps):
            tok = int(oracle.argmax(want))
            want = om.forward([tok])
            assert_close(step_logits[s_][i], want, LOGIT_ABS, LOGIT_REL, f"sequence {i} (context {lens[i]}), decode step {s_}")
    eng.close()


def test_results_stay_what_they_are_while_somebody_holds_them(gpu, oracle):
    """Logits lie in blocks that the handle lends.  Four results held at once (more than it has), views of them, and one that outlives its handle keep their
    values; blocks come back when the last view goes."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=1)
    eng = synth.build_engine(spec, 64, max_seqs=3)
    ids, steps = [0, 1, 2], [[[7], [8], [9]], [[1], [2], [3]], [[4], [5], [6]], [[10], [11], [12]]]
    held = [eng.forward_batch(ids, s)[0] for s in steps]
    again = synth.build_engine(spec, 64, max_seqs=3)
    kept = [again.forward_batch(ids, s)[0].copy() for s in steps]
    for a, b in zip(held, kept):
        assert np.array_equal(a, b)
    lent = {a.ctypes.data for a in held}
    view = held[0][1:, ::2]
    del held
    reused = [again.forward_batch(ids, s)[0] for s in steps[:2]] + [eng.forward_batch(ids, s)[0] for s in steps[:1]]
    assert reused[-1].ctypes.data in lent and np.array_equal(view, kept[0][1:, ::2])
    last = eng.forward_batch(ids, steps[0])[0]
    want = last.copy()
    eng.close()
    again.forward_batch(ids, steps[1])
    assert np.array_equal(last, want) and np.array_equal(view, kept[0][1:, ::2])
    again.close()


@pytest.mark.parametrize("rows,vocab", [(3, 512), (9, 32000)])
def test_a_copy_that_begins_before_a_result_is_dropped(gpu, rows, vocab):
    """A caller starts asynchronous copies of results to the GPU behind work that takes a while, and drops the results; the calls that follow leave what is copied alone."""
    import torch
    from leafcutterllm_b200 import synth
    eng = synth.build_engine(small_spec(12, 12, 12, layers=1, vocab=vocab), 64, max_seqs=rows)
    ids, steps = list(range(rows)), [[[7 * i + j] for j in range(rows)] for i in range(6)]
    side, want, got = torch.cuda.Stream(), [], []
    for s in steps[:3]:
        logits = eng.forward_batch(ids, s)[0]
        want.append(logits.copy())
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)
            got.append(torch.from_numpy(logits).to("cuda", non_blocking=True))
        del logits
    for s in steps[3:]:
        eng.forward_batch(ids, s)
    torch.cuda.synchronize()
    eng.close()
    for a, b in zip(got, want):
        assert np.array_equal(a.cpu().numpy(), b)


@pytest.mark.parametrize("heads,kv", [(4, 4), (4, 2), (4, 1), (8, 1)])
def test_batched_decode_attention_as_one_stream(gpu, oracle, heads, kv):
    """The (token, kv head, page) items of a decode step cut into one run per warp: contexts on both sides of a page's edge, a first token, one that many runs
    share (38 pages), for 1, 2, 4 and 8 query heads per kv head, with rotation by position.  Against the oracle: keys and values of both are
    rounded to f16 (2^-11 at most), so results that differ by more than four times that (2-norm) are wrong."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=1, hidden=128 * heads, heads=heads, kv=kv, ffn=512, vocab=512)
    lens = [15, 16, 600, 1, 31, 33, 128]
    ids = list(range(len(lens)))
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=640, max_seqs=len(lens), rope_mode="absolute")
    prompts = [synth.prompt_tokens(n, spec.vocab_size, 400 + i).tolist() for i, n in enumerate(lens)]
    fed = np.random.default_rng(heads + kv).integers(0, spec.vocab_size, (3, len(lens)))
    eng.forward_batch(ids, prompts, want_logits=False)
    got = [eng.forward_batch(ids, [[int(t)] for t in row])[0].copy() for row in fed]
    eng.close()
    for i, p in enumerate(prompts):
        om.kv_clear()
        om.forward(p)
        for step, row in enumerate(fed):
            want = np.asarray(om.forward([int(row[i])]), np.float64)
            err = np.linalg.norm(got[step][i] - want) / np.linalg.norm(want)
            assert err < 4 * 2.0 ** -11, (i, step, err)


@pytest.mark.parametrize("typ", [12, 14])
@pytest.mark.parametrize("n", [1, 3, 7])
def test_norm_of_rows_near_the_ends_of_f32(gpu, typ, n):
    """The matrix-vector kernels multiply by the norm's factor at the end.  Hidden rows of 1e-26 keep their 22 bits on the way there (bound: what f32 sums of 512 products leave, a few
    1e-7), and rows whose squares leave f32's range have a factor of zero, so that q, k, v and logits are zero and not NaN, though the sums may leave it as well."""
    from leafcutterllm_b200 import synth
    from leafcutterllm_b200.synth import ModelSpec
    H, V = 512, 64
    spec = ModelSpec("ends", 1, H, 4, 4, 512, V, 10000.0, typ, 0, typ)
    r = np.random.default_rng(typ + n)
    embed = (r.standard_normal((V, H)) * np.where(np.arange(V) < 32, 1e-26, 3e37)[:, None]).astype(np.float32)
    eng = gpu.Engine(H, 1, 4, 4, 512, V, max_seq_len=32, max_seqs=n, kv_dtype="f32")
    w = {}
    for name, t, dims, kind in spec.tensors():
        data = embed if name.startswith("token_embd") else synth.tensor_bytes(spec, name, t, dims, kind, 77)
        eng.set_tensor(name, t, dims, data)
        if t == typ:
            w[name.split(".")[-2]] = gpu.dequantize(typ, data, int(np.prod(dims))).reshape(dims[1], dims[0]).astype(np.float64)
    eng.finalize()
    ids = list(range(n))
    got = eng.forward_batch(ids, [[i] for i in ids])[0]  # the first token of each sequence: the attention's result is its value
    for i in ids:
        x = embed[i].astype(np.float64)
        h = x + w["attn_output"] @ (w["attn_v"] @ (x / np.sqrt(1e-5)))
        want = w["output"] @ (h / np.sqrt(1e-5))
        assert np.linalg.norm(got[i] - want) < 2e-6 * np.linalg.norm(want)
    eng.kv_clear()
    assert (eng.forward_batch(ids, [[32 + i] for i in ids])[0] == 0).all()
    eng.close()


@pytest.mark.parametrize("heads,kv,n", [(8, 2, 128), (8, 2, 127), (8, 2, 5), (8, 2, 4), (8, 4, 4), (4, 4, 9)])
def test_batched_decode_attention_without_rotation(gpu, oracle, heads, kv, n):
    """Steps that rotate by nothing, on both sides of the lines between the kernels (1,024 heads of all sequences; up to four sequences, four heads per kv head; no kv groups).
    Bound as in the test above."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=2, hidden=128 * heads, heads=heads, kv=kv, ffn=256, vocab=256)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=80, max_seqs=n)
    prompts = [synth.prompt_tokens(1 + (7 * i) % 40, spec.vocab_size, 600 + i).tolist() for i in range(n)]
    fed = np.random.default_rng(n).integers(0, spec.vocab_size, (2, n))
    eng.forward_batch(list(range(n)), prompts, want_logits=False)
    got = [eng.forward_batch(list(range(n)), [[int(t)] for t in row])[0].copy() for row in fed]
    eng.close()
    for i in range(0, n, 1 if n < 16 else 13):
        om.kv_clear()
        om.forward(prompts[i])
        for step, row in enumerate(fed):
            want = np.asarray(om.forward([int(row[i])]), np.float64)
            err = np.linalg.norm(got[step][i] - want) / np.linalg.norm(want)
            assert err < 4 * 2.0 ** -11, (i, step, err)


def test_batched_decode_attention_adds_in_32_bits(gpu):
    """16 sequences of 3,700 random tokens, small queries: the weights are nearly equal, but not to 2^-11, and values positive, so that an error of the sums adds up.  Keys and values
    are f16 numbers (permutations of one row, so that one gain brings the norm back to the row itself; keys in dims that do not turn at this theta); the output projection adds
    the even dims alone to the residual, so the last norm does not hide a common factor.  f32 sums, and the head's 4,096 products, leave 1.9e-7 -
    2.9e-7 of the logits (the kernel that adds with f32 FMAs the same); sums in the matrix unit's accumulators, which truncate, 1.6e-6 - 2.6e-6.  6e-7 lies between."""
    from leafcutterllm_b200.synth import ModelSpec
    H, heads, F, V, n, ctx = 4096, 32, 256, 64, 16, 3700
    r = np.random.default_rng(5)
    base = np.exp2(r.uniform(-4, 1, H)).astype(np.float16).astype(np.float32)
    embed = np.stack([r.permutation(base) for _ in range(V)])
    gain = np.float32(np.sqrt((base.astype(np.float64) ** 2).mean() + 1e-5))
    even, still = np.arange(H) % 2 == 0, np.arange(H) % 64 >= 32
    head = r.standard_normal((V, H)).astype(np.float32)
    made = {"token_embd": embed, "output": head, "attn_q": np.diag(np.where(still, 0.02, 0)).astype(np.float32), "attn_k": np.diag(still.astype(np.float32)), "attn_v": np.eye(H, dtype=np.float32),
            "attn_output": np.diag(even.astype(np.float32)),
            "attn_norm": np.full(H, gain, np.float32), "ffn_norm": np.ones(H, np.float32), "output_norm": np.ones(H, np.float32)}
    spec = ModelSpec("flat", 1, H, heads, heads, F, V, 10000.0, 0, 0, 0)
    eng = gpu.Engine(H, 1, heads, heads, F, V, max_seq_len=ctx + 16, rope_theta=1e30, max_seqs=n, kv_pool_tokens=n * (ctx + 32), rope_mode="absolute")
    for name, typ, dims, _ in spec.tensors():
        eng.set_tensor(name, typ, dims, made.get(name.split(".")[-2], np.zeros(int(np.prod(dims)), np.float32)))
    eng.finalize()
    ids = list(range(n))
    tokens = r.integers(0, V, (n, ctx + 3))
    eng.forward_batch(ids, tokens[:, :ctx].tolist(), want_logits=False)
    for step in range(ctx, ctx + 3):
        got = eng.forward_batch(ids, tokens[:, step:step + 1].tolist())[0]
        for i in ids:
            of = embed.astype(np.float64).reshape(V, heads, 128)
            q = np.where(still, np.float32(0.02), 0) * of[tokens[i, step]].ravel()
            w = np.bincount(tokens[i, :step + 1], minlength=V) * np.exp(np.einsum("hd,vhd->hv", q.reshape(heads, 128), of) / np.sqrt(128))
            h = embed[tokens[i, step]] + np.where(even, np.einsum("hv,vhd->hd", w / w.sum(1, keepdims=True), of).ravel(), 0.0)
            want = head.astype(np.float64) @ (h / np.sqrt((h * h).mean() + 1e-5))
            assert np.linalg.norm(got[i] - want) < 6e-7 * np.linalg.norm(want), np.linalg.norm(got[i] - want) / np.linalg.norm(want)
    eng.close()


@pytest.mark.parametrize("heads,kv", [(4, 4), (4, 1)])
def test_batched_decode_attention_of_keys_beyond_f16(gpu, oracle, heads, kv):
    """One token's keys have an element beyond f16's range: minus or plus infinity in the cache.  Queries that give them scores of minus infinity give them no weight, whatever the signs
    of the halves that queries are cut into; the others' results are NaN in the oracle too.  Bound as in the test above it."""
    from leafcutterllm_b200.synth import ModelSpec
    H, V, n, at = 128 * heads, 256, 7, 40  # dim 40 of a head does not turn at this theta
    r = np.random.default_rng(heads + kv)
    embed = r.standard_normal((V, H)).astype(np.float32)
    embed[:, at::128] = 0.0
    embed[5, at::128] = 90.0  # token 5's keys are infinite there (weights beyond 100 count as zero, so it takes three factors) ...
    gain = np.ones(H, np.float32)
    gain[at] = 100.0
    wq = (r.standard_normal((H, H)) / np.sqrt(H)).astype(np.float32)
    wk, wv, wo = [(r.standard_normal(s) / np.sqrt(H)).astype(np.float32) for s in ((128 * kv, H), (128 * kv, H), (H, H))]
    wq[:, at::128] = wk[:, at::128] = 0.0
    for h in range(kv):
        wk[128 * h + at, at] = 100.0
    made = {"token_embd": embed, "output": r.standard_normal((V, H)).astype(np.float32), "attn_q": wq, "attn_k": wk, "attn_v": wv, "attn_output": wo,
            "attn_norm": gain, "ffn_norm": np.ones(H, np.float32), "output_norm": np.ones(H, np.float32)}
    spec = ModelSpec("wild", 1, H, heads, kv, 256, V, 1e30, 0, 0, 0)
    eng = gpu.Engine(H, 1, heads, kv, 256, V, max_seq_len=256, rope_theta=1e30, max_seqs=n, rope_mode="absolute")
    om = oracle.OracleModel(H, 1, heads, kv, 256, V, max_seq_len=256, rope_theta=1e30, rope_absolute=True)
    for name, typ, dims, _ in spec.tensors():
        w = made.get(name.split(".")[-2], np.zeros(int(np.prod(dims)), np.float32))
        eng.set_tensor(name, typ, dims, w)
        om.set_tensor(name, typ, dims, np.ascontiguousarray(w).view(np.uint8).ravel())
    eng.finalize()
    prompts = [[5 if j % 37 == i else int(t) for j, t in enumerate(r.integers(6, V, 3 + 33 * i))] for i in range(n)]
    # ... and these queries have there what makes all scores with them minus infinity: tokens whose q is negative there for every head
    scores = (embed @ wq.T)[:, at::128]
    fed = [int(t) for t in np.flatnonzero((scores < 0).all(1)) if t > 5][:3]
    assert len(fed) == 3
    eng.forward_batch(list(range(n)), prompts, want_logits=False)
    got = [eng.forward_batch(list(range(n)), [[t]] * n)[0].copy() for t in fed]
    eng.close()
    for i in range(n):
        om.kv_clear()
        om.forward(prompts[i])
        for step, t in enumerate(fed):
            want = np.asarray(om.forward([t]), np.float64)
            assert np.isfinite(want).all()
            err = np.linalg.norm(got[step][i] - want) / np.linalg.norm(want)
            assert err < 4 * 2.0 ** -11, (i, step, err)


def test_batched_decode_attention_whose_waits_run_out(gpu, monkeypatch):
    """Every wait for a page gives up before it looks (LC_ATTN_WAITS=0, a step's launches are made anew for another number of sequences): the call ends with an error, and
    the handle is usable: the tickets of segments that several warps share are back at zero, so the next steps give what a handle gives that never failed."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=2, hidden=512, heads=4, kv=1, ffn=512, vocab=512)
    lens = [600, 16, 300, 1, 128, 33]
    prompts = [synth.prompt_tokens(n, spec.vocab_size, 500 + i).tolist() for i, n in enumerate(lens)]

    def steps(eng, n):
        eng.kv_clear()
        eng.forward_batch(list(range(n)), prompts[:n], want_logits=False)
        return [eng.forward_batch(list(range(n)), [[7 + i] for i in range(n)])[0].copy() for _ in range(2)]

    eng = synth.build_engine(spec, 640, max_seqs=len(lens), rope_mode="absolute")
    want = steps(eng, 5)
    eng.close()
    eng = synth.build_engine(spec, 640, max_seqs=len(lens), rope_mode="absolute")
    monkeypatch.setenv("LC_ATTN_WAITS", "0")
    with pytest.raises(gpu.LeafcutterError, match="a bounded wait ran out"):
        steps(eng, 6)
    monkeypatch.delenv("LC_ATTN_WAITS")
    for a, b in zip(steps(eng, 5), want):
        assert np.array_equal(a, b)
    eng.close()


def close_to(got, want, what):
    """Keys and values of both sides are rounded to f16 (2^-11 at most): results that differ by more than four times that (2-norm) are wrong."""
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err < 4 * 2.0 ** -11, (what, err)


@pytest.mark.parametrize("heads,kv", [(4, 4), (4, 1)])
def test_batched_decode_attention_of_later_layers(gpu, oracle, heads, kv):
    """Layers behind the first read positions and page tables, and request cached pages, ahead of the kernel before them.  40 sequences, three layers, rotation by position: page
    counts of more than 32 tokens, page-table entries reloaded every 32 pages, one context of 257 pages that about 30 runs share; contexts that step over a page's edge.
    Steps alone, then a loop of captured steps, then a step alone again."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=3, hidden=128 * heads, heads=heads, kv=kv, ffn=256, vocab=256)
    n, looped = 40, 6
    lens = [600, 1, 15, 511] + [1 + (11 * i) % 60 for i in range(n - 5)] + [4095]
    ids, checked = list(range(n)), [0, 1, 2, 3, 9, 32, 33, n - 1]
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=4112, max_seqs=n, kv_pool_tokens=sum(lens) + 32 * n, rope_mode="absolute")
    prompts = [synth.prompt_tokens(m, spec.vocab_size, 700 + i).tolist() for i, m in enumerate(lens)]
    fed = np.random.default_rng(heads + kv).integers(0, spec.vocab_size, (4, n))
    eng.forward_batch(ids, prompts, want_logits=False)
    got = [eng.forward_batch(ids, [[int(t)] for t in row])[0].copy() for row in fed[:2]]
    picks, _ = eng.decode_loop(ids, fed[2], looped)
    last = eng.forward_batch(ids, [[int(t)] for t in fed[3]])[0].copy()
    eng.close()
    for i in checked:
        om.kv_clear()
        om.forward(prompts[i])
        for step in range(2):
            close_to(got[step][i], np.asarray(om.forward([int(fed[step][i])]), np.float64), (i, step))
        for t, pick in zip([int(fed[2][i])] + picks[:-1, i].tolist(), picks[:, i]):
            logits = np.asarray(om.forward([t]), np.float64)
            assert logits.max() - logits[pick] < 8 * 2.0 ** -11 * np.linalg.norm(logits), (i, t, pick)  # the pick's and the largest's errors
        close_to(last[i], np.asarray(om.forward([int(fed[3][i])]), np.float64), (i, "last"))


@pytest.mark.parametrize("n", [3, 7])
@pytest.mark.parametrize("heads,kv,hidden,cache,mix", [(4, 4, 512, "f16", "q4_k_m"), (4, 2, 512, "f16", "q4_k_m"), (4, 4, 512, "f32", "q4_k_m"), (4, 2, 256, "f16", ""), (8, 4, 256, "f32", "")])
def test_batched_decode_turned_by_position(gpu, oracle, n, heads, kv, hidden, cache, mix):
    """Several sequences at unequal positions, each turned by its own row of the step's table, in every kernel that a step of several tokens has: heads of 128 without kv groups
    (staged at 3, one stream at 7), with them, an f32 cache, heads of 64 and 32 (split contexts).  With a mix of types the last layers' q, k and v are three
    products, whose rows lie apart by other strides than a fused product's."""
    from dataclasses import replace
    from leafcutterllm_b200 import synth
    spec = replace(small_spec(12, 12, 12, layers=3, hidden=hidden, heads=heads, kv=kv, ffn=512, vocab=512), mix=mix)
    lens = [37, 5, 130, 1, 16, 64, 250][:n]
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=272, max_seqs=n, kv_dtype=cache, rope_mode="absolute", on_device=True)
    prompts = [synth.prompt_tokens(m, spec.vocab_size, 800 + i).tolist() for i, m in enumerate(lens)]
    fed = np.random.default_rng(heads + n).integers(0, spec.vocab_size, (3, n))
    eng.forward_batch(list(range(n)), prompts, want_logits=False)
    got = [eng.forward_batch(list(range(n)), [[int(t)] for t in row])[0].copy() for row in fed]
    eng.close()
    for i in range(n):
        om.kv_clear()
        om.forward(prompts[i])
        for step, row in enumerate(fed):
            close_to(got[step][i], np.asarray(om.forward([int(row[i])]), np.float64), (i, step))


@pytest.mark.parametrize("heads,kv,cache", [(8, 2, "f32"), (16, 4, "f16")])
def test_batched_decode_attention_split_into_pieces(gpu, oracle, heads, kv, cache):
    """80 sequences over a cache in f32, and with heads of 64: kernels of split contexts.  1,024-key pieces merged through scratch, the new key in one of them,
    contexts on both sides of their edges, most pieces empty; turned by position."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=2, hidden=1024, heads=heads, kv=kv, ffn=256, vocab=256)
    n, special = 80, [5, 1022, 1023, 1024, 2047, 2049, 2500, 4090]
    lens = special + [1 + (13 * i) % 90 for i in range(n - len(special))]
    ids = list(range(n))
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=4096, max_seqs=n, kv_pool_tokens=sum(lens) + 32 * n, kv_dtype=cache, rope_mode="absolute")
    prompts = [synth.prompt_tokens(m, spec.vocab_size, 900 + i).tolist() for i, m in enumerate(lens)]
    fed = np.random.default_rng(heads).integers(0, spec.vocab_size, (3, n))
    eng.forward_batch(ids, prompts, want_logits=False)
    got = [eng.forward_batch(ids, [[int(t)] for t in row])[0].copy() for row in fed]
    eng.close()
    for i in list(range(len(special))) + [20, 79]:
        om.kv_clear()
        om.forward(prompts[i])
        for step, row in enumerate(fed):
            close_to(got[step][i], np.asarray(om.forward([int(row[i])]), np.float64), (i, step))


def test_prefill_attention_on_tensor_cores_ragged(gpu, oracle):
    """head_dim 128, f16 cache: calls of 16 tokens and more run the tiled tensor-core prefill attention.  Four sequences of
    70, 16, 129 and 33 tokens in ONE call (tiles end where a sequence ends; 129 = two full tiles and a one-token tile), then a
    second call that appends 20 to 40 tokens to each cache (tiles that start in the middle of a page and attend to keys of
    the earlier call), grouped-query heads (4 query heads over 2 kv heads).  Logits per sequence against the oracle."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=2, hidden=512, heads=4, kv=2, ffn=512, vocab=600)
    lens, more = [70, 16, 129, 33], [20, 40, 25, 31]
    ids = [0, 1, 2, 3]
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=192, max_seqs=4)
    p1 = [synth.prompt_tokens(n, spec.vocab_size, 200 + i).tolist() for i, n in enumerate(lens)]
    p2 = [synth.prompt_tokens(n, spec.vocab_size, 300 + i).tolist() for i, n in enumerate(more)]
    l1, _ = eng.forward_batch(ids, p1)
    l2, _ = eng.forward_batch(ids, p2)
    for i in ids:
        om.kv_clear()
        assert_close(l1[i], om.forward(p1[i]), LOGIT_ABS, LOGIT_REL, f"sequence {i}, first call")
        assert_close(l2[i], om.forward(p2[i]), LOGIT_ABS, LOGIT_REL, f"sequence {i}, second call over the cache of the first")
    eng.close()


def test_a_second_model_does_not_disturb_a_captured_decode_step(gpu, oracle):
    """Scratch that a captured decode graph points at belongs to its model: a small model captures its step, then a
    model with more heads is created on the same device (which used to regrow a shared buffer), and the small model
    must keep decoding the oracle's tokens."""
    from leafcutterllm_b200 import synth
    small = small_spec(12, 12, 12, layers=2, hidden=256, heads=2, kv=2, ffn=512, vocab=900)
    big = small_spec(12, 12, 12, layers=1, hidden=2048, heads=16, kv=16, ffn=512, vocab=600)
    eng, om = make_pair(gpu, oracle, small, max_seq_len=96)
    prompt = synth.prompt_tokens(20, small.vocab_size, 3)
    ref, margins = om.generate(prompt, 30, stop_on_eos=False, want_margins=True)
    assert eng.generate(prompt, 10, stop_on_eos=False) == ref[:10], margins   # captures the one-sequence step
    eng2 = synth.build_engine(big, 64, on_device=True)
    assert len(eng2.generate(synth.prompt_tokens(9, big.vocab_size, 4), 6, stop_on_eos=False)) == 6
    assert eng.generate(prompt, 30, stop_on_eos=False) == ref, margins         # replays the graph captured before eng2 existed
    eng2.close()
    assert eng.generate(prompt, 30, stop_on_eos=False) == ref, margins
    eng.close()


@pytest.mark.parametrize("other", [12, 13, 14])
def test_mixed_quant_types_like_q4_k_m(gpu, oracle, other):
    """A "Q4_K_M" file keeps attn_v and ffn_down in Q6_K while q, k, o, gate and up are Q4_K: the three projections of a
    layer then cannot be one matrix (three products per layer); the Q6_K matrices run through the int8 tensor-core kernel
    (fused norm, residual epilogue), the 8-token tiles of the prefill as two passes of it.
    other = 14: every matrix is Q6_K (one fused q/k/v matrix, SiLU(gate) * up epilogue on Q6_K); other = 13: the Q5_K + Q6_K
    mix of a "Q5_K_M" file (Q5_K through the Q4_K kernel's fifth-bit variant).
    Prefill (17 tokens: the unfused parts are interleaved into the q/k/v rows), decode and greedy tokens against the oracle."""
    from leafcutterllm_b200 import Engine, synth
    H, Fd, V, nh, nkv, L = 256, 512, 384, 2, 1, 2
    r = np.random.default_rng(8)

    def q6k(rows, cols):  # random blocks with small scales (no host quantiser for Q6_K): |w| stays below ~0.3
        raw = r.integers(0, 256, (rows * cols // 256, 210), dtype=np.uint8)
        raw[:, 192:208] = r.integers(-40, 41, (raw.shape[0], 16)).astype(np.int8).view(np.uint8)
        d = np.float16(r.uniform(2e-5, 2e-4, raw.shape[0])).view(np.uint16)
        raw[:, 208] = d & 0xFF
        raw[:, 209] = d >> 8
        return raw.ravel()

    def q5k(rows, cols):  # random blocks: 6-bit scales and mins as they come, small d and dmin
        raw = r.integers(0, 256, (rows * cols // 256, 176), dtype=np.uint8)
        for at in (0, 2):
            d = np.float16(r.uniform(2e-5, 2e-4, raw.shape[0])).view(np.uint16)
            raw[:, at] = d & 0xFF
            raw[:, at + 1] = d >> 8
        return raw.ravel()

    eng = Engine(H, L, nh, nkv, Fd, V, max_seq_len=64)
    om = oracle.OracleModel(H, L, nh, nkv, Fd, V, max_seq_len=64)
    hd = H // nh
    tensors = [("token_embd.weight", 12, (H, V)), ("output_norm.weight", 0, (H,)), ("output.weight", 14, (H, V))]
    for l in range(L):
        p = f"blk.{l}."
        tensors += [(p + "attn_norm.weight", 0, (H,)), (p + "attn_q.weight", other, (H, nh * hd)), (p + "attn_k.weight", other, (H, nkv * hd)),
                    (p + "attn_v.weight", 14, (H, nkv * hd)), (p + "attn_output.weight", other, (nh * hd, H)), (p + "ffn_norm.weight", 0, (H,)),
                    (p + "ffn_gate.weight", other, (H, Fd)), (p + "ffn_up.weight", other, (H, Fd)), (p + "ffn_down.weight", 14, (Fd, H))]
    for name, typ, dims in tensors:
        n = int(np.prod(dims))
        data = np.ones(n, np.float32).view(np.uint8) if typ == 0 else (q6k(dims[1], dims[0]) if typ == 14 else (q5k(dims[1], dims[0]) if typ == 13 else synth.host_tensor(typ, 21, name, n)))
        eng.set_tensor(name, typ, dims, data)
        om.set_tensor(name, typ, list(dims), data)
    eng.finalize()
    prompt = synth.prompt_tokens(17, V, 2)
    assert_close(eng.forward(prompt), om.forward(prompt), LOGIT_ABS, LOGIT_REL, "prefill logits, mixed types")
    nxt = 5
    assert_close(eng.forward([nxt]), om.forward([nxt]), LOGIT_ABS, LOGIT_REL, "decode logits, mixed types")
    ref, margins = om.generate(prompt, 10, stop_on_eos=False, want_margins=True)
    assert eng.generate(prompt, 10, stop_on_eos=False) == ref, margins
    eng.close()


def test_error_paths(gpu):
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=1)
    eng = gpu.Engine(spec.hidden_size, 1, spec.num_heads, spec.num_kv_heads, spec.intermediate_size, spec.vocab_size, max_seq_len=32)
    with pytest.raises(gpu.LeafcutterError) as e:
        eng.forward([1])
    assert e.value.status == -7  # not finalized
    with pytest.raises(gpu.LeafcutterError) as e:
        eng.finalize()
    assert e.value.status == -6  # missing tensors (the reference panics: engine.rs:84,97,101)
    eng.close()
    eng = synth.build_engine(spec, 32, on_device=True)
    with pytest.raises(gpu.LeafcutterError) as e:
        eng.forward(list(range(33)))
    assert e.value.status == -5  # KV capacity
    with pytest.raises(gpu.LeafcutterError) as e:
        eng.generate([1, 2], 4, temperature=0.7)
    assert e.value.status == -2
    out = eng.forward([10 ** 6])  # engine.rs:137-141: out-of-range id -> zero embedding row, still finite
    assert np.isfinite(out).all()
    eng.close()


def test_tiny_shape_reduced_depth(gpu, oracle):
    """TinyLlama-1.1B dims (hidden 2048, 32 q / 4 kv heads, FFN 5632, vocab 32000, Q4_0 + Q8_0), 3 layers."""
    from leafcutterllm_b200 import synth
    spec = synth.TINY.with_layers(3)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=64, on_device=True)
    prompt = synth.prompt_tokens(32, spec.vocab_size)
    assert_close(eng.forward(prompt), om.forward(prompt), LOGIT_ABS, LOGIT_REL, "prefill")
    toks = eng.generate(prompt, 16, stop_on_eos=False)
    ref, margins = om.generate(prompt, 16, stop_on_eos=False, want_margins=True)
    assert toks == ref, margins
    eng.close()


@pytest.mark.parametrize("layers,heads,kv", [(2, 4, 2), (3, 2, 2), (3, 4, 4), (3, 8, 2)])
def test_single_sequence_decode_head_dim_128(gpu, oracle, layers, heads, kv):
    """head_dim 128 + Q4_K + f16 cache: single-sequence decode steps run the streaming attention kernel and the
    tensor-core matrix-vector kernel from a captured graph.  Same tokens as the oracle through the device-resident
    loop, and the oracle's logits step by step through the host API."""
    from leafcutterllm_b200 import synth
    spec = small_spec(12, 12, 12, layers=layers, hidden=128 * heads, heads=heads, kv=kv, ffn=768, vocab=1500)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=160)
    prompt = synth.prompt_tokens(40, spec.vocab_size, 5)
    ref, margins = om.generate(prompt, 48, stop_on_eos=False, want_margins=True)
    toks = eng.generate(prompt, 48, stop_on_eos=False)
    assert toks == ref, margins
    eng.kv_clear()
    om.kv_clear()
    got = eng.forward(prompt)
    want = om.forward(prompt)
    for step in range(6):
        nxt = int(np.argmax(want))
        got, want = eng.forward([nxt]), om.forward([nxt])
        assert_close(got, want, LOGIT_ABS, LOGIT_REL, f"step {step}")
    eng.close()


def test_decode_ignores_unwritten_cache_rows(gpu, oracle):
    """The rows of a KV page beyond the current position hold whatever the pool's memory held before (the pools are
    not cleared).  Their softmax weight is zero, but 0 * NaN is NaN: kernels must not touch them.  Device memory is
    poisoned with f16 NaNs and released just before the model is built, and decoding crosses page boundaries."""
    import ctypes as C
    from leafcutterllm_b200 import synth, _capi
    lib = _capi.load()
    bufs = []
    poison = np.full(64 << 20, 0xFF, np.uint8)
    for _ in range(6):
        p = C.c_void_p()
        _capi.check(lib.lc_dev_alloc(poison.nbytes, C.byref(p)))
        _capi.check(lib.lc_dev_upload(p, poison.ctypes.data_as(C.c_void_p), poison.nbytes))
        bufs.append(p)
    for p in bufs:
        lib.lc_dev_free(p)
    spec = small_spec(12, 12, 12, layers=2, hidden=256, heads=2, kv=2, ffn=768, vocab=1500)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=160)
    prompt = synth.prompt_tokens(30, spec.vocab_size, 9)
    ref, margins = om.generate(prompt, 40, stop_on_eos=False, want_margins=True)
    toks = eng.generate(prompt, 40, stop_on_eos=False)
    assert toks == ref, margins
    eng.close()


def test_ffn_probe_of_more_rows_than_the_cache_holds(gpu, oracle):
    """A pass is 512 rows at least, whatever the sequences' capacity."""
    spec = small_spec(12, 12, 12, layers=1, hidden=256, heads=2, kv=2, ffn=512, vocab=64)
    eng, om = make_pair(gpu, oracle, spec, max_seq_len=32)
    x = np.random.default_rng(3).standard_normal((512, 256)).astype(np.float32)
    want = om.ffn(0, x)
    # SiLU(gate) * up of two many-token products (2e-5 of the largest each, tested with the product), then a third
    assert_close(eng.probe_ffn(0, x), want, 1e-4 * np.abs(want).max(), 1e-4, "512 rows")
    eng.close()
