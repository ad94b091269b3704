"""Engine-level parity on a B200 through the C ABI: whole decode steps against the CPU
checker holding byte-identical weights.

The engine keeps every f32 operation in the CPU path's order, so for dense models the bar is
bit identity: residual stream after every layer, logits, KV rows and every greedy token equal the
checker's.  (Acceptance gates, for reference: per-layer hidden states and logits within max-abs
2e-2 and relative 1e-2; greedy token ids equal for at least the first 32 generated tokens.)
"""
import numpy as np
import pytest

from helpers import ModelPair, greedy_match, hidden_gate

pytestmark = pytest.mark.gpu


class Lcg:
    """The reference tests' generator (src/cuda_resident/tests.rs:3700-3717)."""

    def __init__(self, seed):
        self.s = seed

    def f32(self, n):
        out = np.empty(n, np.float32)
        for i in range(n):
            self.s = (self.s * 6364136223846793005 + 1442695040888963407) & 0xFFFFFFFFFFFFFFFF
            out[i] = np.float32(np.float32(self.s >> 40) / np.float32(1 << 24)) * np.float32(2.0) - np.float32(1.0)
        return out


# full_forward_token_matches_cpu (src/cuda_resident/tests.rs:2962-3134): the reference's own
# tiny Llama (2 layers, hidden 64, 2 heads / 1 kv head, head_dim 32, ffn 128, vocab 96), Q8_0
# weights from its LCG, norm weights 1 +- 0.2, four positions fed as embeddings; token ids
# must be equal.
def test_reference_tiny_model_token_identity(cm, orc):
    L, hidden, heads, kv, hd, ffn, vocab, max_pos = 2, 64, 2, 1, 32, 128, 96, 16
    rng = Lcg(0xABCDEF)
    cfg = cm.EngineConfig(n_layers=L, n_heads=heads, n_kv_heads=kv, head_dim=hd, hidden=hidden, ffn_dim=ffn, max_pos=max_pos,
                          vocab=vocab, rope_dim=hd, eps=1e-5, rope_theta=10000.0)
    eng = cm.ResidentDecode(cfg)
    ref = orc.OracleModel(cfg.oracle_dict())
    shapes = {"q": (heads * hd, hidden), "k": (kv * hd, hidden), "v": (kv * hd, hidden), "o": (hidden, heads * hd),
              "gate": (ffn, hidden), "up": (ffn, hidden), "down": (hidden, ffn)}
    for layer in range(L):
        projs = {n: (8, orc.quantize(8, rng.f32(r * c))) for n, (r, c) in shapes.items()}
        an = rng.f32(hidden) * np.float32(0.2) + np.float32(1.0)
        fn = rng.f32(hidden) * np.float32(0.2) + np.float32(1.0)
        eng.set_layer(layer, projs, an, fn)
        ref.set_layer(layer, projs, an, fn)
    fnorm = rng.f32(hidden) * np.float32(0.2) + np.float32(1.0)
    out_w = orc.quantize(8, rng.f32(vocab * hidden))
    eng.set_output(fnorm, (8, out_w))
    ref.set_output(fnorm, 8, out_w)
    assert eng.weights_ready() and eng.n_layers() == L and eng.max_pos() == max_pos
    scale = float(np.float32(1.0) / np.sqrt(np.float32(hd)))
    for position in range(4):
        emb = rng.f32(hidden)
        c, s = orc.rope_table(position, hd, 10000.0)
        logits, _, _ = ref.forward(emb, position)
        tok = eng.forward_token(emb, c, s, position, scale, True)
        assert tok == orc.argmax(logits), position
        eng.set_filled(position + 1)
    assert eng.filled() == 4


@pytest.fixture(scope="module", params=["q8_0", "q4_k_m"])
def pair(request, cm):
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny", max_pos=160, max_seqs=4)
    return ModelPair(cfg, request.param, seed=20261125)


def test_per_layer_hidden_logits_and_kv_are_bit_identical(pair, orc):
    eng, ref, cfg = pair.engine, pair.oracle, pair.cfg
    toks = orc.synth_tokens(1, 1, 12, cfg.vocab)
    for pos, t in enumerate(toks):
        emb = ref.embedding(int(t))
        c, s = pair.rope(pos)
        ref_logits, ref_hidden, ref_taps = ref.forward(emb, pos, want_taps=True)
        hidden, taps = eng.forward_token_hidden(emb, c, s, pos, pair.scale, taps=True)
        for layer in range(cfg.n_layers):
            assert np.array_equal(taps[layer].view(np.uint32), ref_taps[layer].view(np.uint32)), (pos, layer, hidden_gate(taps[layer], ref_taps[layer]))
        assert np.array_equal(hidden.view(np.uint32), ref_hidden.view(np.uint32))
        logits = eng.forward_token_logits(emb, c, s, pos, pair.scale)
        assert np.array_equal(logits.view(np.uint32), ref_logits.view(np.uint32)), (pos, hidden_gate(logits, ref_logits))
    for layer in range(cfg.n_layers):
        ck, cv = eng.read_kv_layer(layer, len(toks))
        rk, rv = ref.read_kv_layer(layer, len(toks))
        assert np.array_equal(ck, rk) and np.array_equal(cv, rv), layer


def test_greedy_tokens_match_checker(pair, orc):
    eng, ref, cfg = pair.engine, pair.oracle, pair.cfg
    n_gen = 48
    runs = []
    for prompt_seed in (2, 3, 4, 5):
        prompt = orc.synth_tokens(prompt_seed, 1, 9, cfg.vocab)
        ref_tokens, _, gaps = ref.generate(prompt, n_gen, want_gaps=True)
        first = eng.prefill_tokens(0, prompt, 0)
        out = eng.decode_greedy([0], [first], [len(prompt)], n_gen - 1)
        got = np.concatenate([[first], out[:, 0]])
        runs.append(greedy_match(got, ref_tokens, gaps))
    assert all(n == n_gen for n, _ in runs), runs  # every token of every prompt
    ms, launches = eng.last_timing()
    assert ms > 0 and launches > 0


def test_batched_rows_equal_serial_bitwise(pair, orc):
    """phase7_independent_paged_batch*_matches_*_serial_forwards and
    verify_batch_matches_sequential (src/cuda_resident/tests.rs:6267, :3947)."""
    eng, cfg = pair.engine, pair.cfg
    prompts = [orc.synth_tokens(3, s, 6 + s, cfg.vocab) for s in range(4)]
    firsts = [eng.prefill_tokens(s, prompts[s], 0) for s in range(4)]
    # serial: each sequence alone
    serial_logits = []
    for s in range(4):
        _, lg, _ = eng.step_batch([s], [firsts[s]], [len(prompts[s])], want_logits=True)
        serial_logits.append(lg[0])
    # batched: the same four rows in one step (KV rows are rewritten with identical values)
    toks, lg, _ = eng.step_batch([0, 1, 2, 3], firsts, [len(p) for p in prompts], want_logits=True)
    for s in range(4):
        assert np.array_equal(lg[s], serial_logits[s]), s
        assert toks[s] == int(np.argmax(serial_logits[s]))
    # verify_batch: k consecutive positions of one sequence in one pass == k serial forward_token calls
    ref = pair.oracle
    embs = np.stack([ref.embedding(int(t)) for t in prompts[0][:5]])
    cs = [pair.rope(p) for p in range(5)]
    cos_all, sin_all = np.stack([c for c, _ in cs]), np.stack([s for _, s in cs])
    serial = [eng.forward_token(embs[p], cos_all[p], sin_all[p], p, pair.scale, True) for p in range(5)]
    k0, v0 = eng.read_kv_layer(1, 5)
    batch = eng.verify_batch(embs, cos_all, sin_all, 0, 5, pair.scale)
    k1, v1 = eng.read_kv_layer(1, 5)
    assert list(batch) == serial
    assert np.array_equal(k0, k1) and np.array_equal(v0, v1)
    # prefill (embedding form) leaves the same KV as serial calls
    eng.prefill(embs, cos_all, sin_all, 5, pair.scale)
    k2, v2 = eng.read_kv_layer(1, 5)
    assert np.array_equal(k0, k2) and np.array_equal(v0, v2)


def staged_launches(monkeypatch, tmp_path, cm, orc, hidden, ffn, rows):
    """(matrices, paired) of every launch of the staged matvec in one Q8_0 step of `rows` rows, whose logits are the checker's."""
    import csv

    cfg = cm.EngineConfig(n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, hidden=hidden, ffn_dim=ffn, vocab=512, max_pos=32, max_seqs=4)
    monkeypatch.setenv("CMLD_TRACE", str(tmp_path / "trace"))
    pair = ModelPair(cfg, "q8_0", seed=64)
    tokens = orc.synth_tokens(5, 1, rows, cfg.vocab)
    _, logits, _ = pair.engine.step_batch(list(range(rows)), tokens, [0] * rows, want_logits=True)
    for b in range(rows):
        want = pair.oracle.forward(pair.oracle.embedding(int(tokens[b])), 0)[0]
        assert np.array_equal(logits[b].view(np.uint32), want.view(np.uint32)), b
    pair.engine.close()
    with open(tmp_path / "trace.0") as f:
        return [(int(r["jobs"]), int(r["paired"])) for r in csv.DictReader(f)]


@pytest.mark.parametrize("hidden, ffn, rows, paired", [(288, 576, 1, 1), (288, 576, 2, 1), (288, 576, 3, 0), (1024, 1056, 1, 1)])
def test_gate_and_up_pair_where_the_staged_kernel_runs_them(monkeypatch, tmp_path, cm, orc, hidden, ffn, rows, paired):
    """Widths that the row-batched kernel does not take."""
    assert (2, paired) in staged_launches(monkeypatch, tmp_path, cm, orc, hidden, ffn, rows)


@pytest.mark.parametrize("hidden, rows, staged", [(512, 1, True), (512, 2, False), (768, 1, False)])
def test_one_row_of_a_narrow_model_runs_on_the_staged_kernel(monkeypatch, tmp_path, cm, orc, hidden, rows, staged):
    launches = staged_launches(monkeypatch, tmp_path, cm, orc, hidden, 1024, rows)
    assert ((3, 0) in launches and (2, 1) in launches) if staged else not any(n > 1 for n, _ in launches)


def test_seed_layer_round_trip_and_continue(pair, orc):
    eng, cfg = pair.engine, pair.cfg
    prompt = orc.synth_tokens(4, 1, 10, cfg.vocab)
    first = eng.prefill_tokens(0, prompt, 0)
    saved = [eng.read_kv_layer(l, len(prompt)) for l in range(cfg.n_layers)]
    cont = eng.decode_greedy([0], [first], [len(prompt)], 4)[:, 0]
    eng.prefill_tokens(0, orc.synth_tokens(5, 1, 10, cfg.vocab), 0)  # overwrite the cache
    for l, (ck, cv) in enumerate(saved):
        eng.seed_layer(l, ck, cv, len(prompt))
    again = eng.decode_greedy([0], [first], [len(prompt)], 4)[:, 0]
    assert np.array_equal(cont, again)


def test_error_paths_do_not_touch_the_device(pair, cm):
    eng, cfg = pair.engine, pair.cfg
    with pytest.raises(cm.CmldError) as ei:
        eng.decode_greedy([0], [0], [cfg.max_pos - 1], 5)
    assert ei.value.code == 7
    with pytest.raises(cm.CmldError):
        eng.step_batch([9], [0], [0])
    with pytest.raises(cm.CmldError):
        eng.step_batch([0], [cfg.vocab], [0])
    with pytest.raises(cm.CmldError):
        eng.set_layer(0, {"q": (8, np.zeros(10, np.uint8))}, np.ones(cfg.hidden), np.ones(cfg.hidden))
    with pytest.raises(cm.CmldError) as ei:
        eng.set_layer(0, {n: (2, np.zeros(18, np.uint8)) for n in ("q", "k", "v", "o", "gate", "up", "down")},
                      np.ones(cfg.hidden), np.ones(cfg.hidden))
    assert ei.value.code == 3  # Q4_0 is outside the path


def test_generic_and_staged_matvec_paths_agree(cm, orc):
    """The engine built with CMLD_FLAG_DIRECT_GEMV (separate quantise kernels + the generic matvec),
    the default engine (staged matvec with fused prologues), the engine with separate preparation
    kernels and no graphs, and the plain reference-order engine (CMLD_FLAG_EXACT_ORDER) all keep the
    CPU path's order of operations: identical logits."""
    from camelid_b200 import synth

    for shape, mix in (("tiny", "q8_0"), ("tiny", "q4_k_m"), ("small", "q4_k_m")):
        cfg = synth.engine_config(shape, max_pos=64)
        a = ModelPair(cfg, mix, seed=9)
        b = ModelPair(synth.engine_config(shape, max_pos=64, flags=2), mix, seed=9)
        c = ModelPair(synth.engine_config(shape, max_pos=64, flags=8 | 1 | 4), mix, seed=9)  # separate prep kernels, no graph, no PDL
        d = ModelPair(synth.engine_config(shape, max_pos=64, flags=16), mix, seed=9)
        prompt = orc.synth_tokens(8, 1, 8, cfg.vocab)
        fa, fb, fc, fd = (m.engine.prefill_tokens(0, prompt, 0) for m in (a, b, c, d))
        _, la, _ = a.engine.step_batch([0], [fa], [8], want_logits=True)
        _, lb, _ = b.engine.step_batch([0], [fb], [8], want_logits=True)
        _, lc, _ = c.engine.step_batch([0], [fc], [8], want_logits=True)
        _, ld, _ = d.engine.step_batch([0], [fd], [8], want_logits=True)
        assert fa == fb == fc == fd
        assert np.array_equal(la, lb) and np.array_equal(la, lc) and np.array_equal(la, ld)
        _, launches_a = a.engine.last_timing()
        _, launches_c = c.engine.last_timing()
        if shape == "small":  # wide enough for the staged kernel, whose fused prologues (the default) save kernels
            assert launches_a < launches_c
        for m in (a, b, c, d):
            m.engine.close()


def test_wire_upload_path_equals_device_generated(cm, orc):
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny", max_pos=64)
    a = ModelPair(cfg, "q4_k_m", seed=5, via="device")
    b = ModelPair(cfg, "q4_k_m", seed=5, via="wire")
    prompt = orc.synth_tokens(6, 1, 8, cfg.vocab)
    fa, fb = a.engine.prefill_tokens(0, prompt, 0), b.engine.prefill_tokens(0, prompt, 0)
    _, la, _ = a.engine.step_batch([0], [fa], [8], want_logits=True)
    _, lb, _ = b.engine.step_batch([0], [fb], [8], want_logits=True)
    assert fa == fb and np.array_equal(la, lb)


def test_mixtral_shaped_moe_parity(cm, orc):
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny-moe", max_pos=96, max_seqs=2)
    pair = ModelPair(cfg, "q4_k_m", seed=31)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(7, 1, 6, cfg.vocab)
    for pos, t in enumerate(prompt):
        emb = ref.embedding(int(t))
        c, s = pair.rope(pos)
        ref_logits, ref_hidden, ref_taps = ref.forward(emb, pos, want_taps=True)
        hidden, taps = eng.forward_token_hidden(emb, c, s, pos, pair.scale, taps=True)
        for layer in range(cfg.n_layers):
            assert np.array_equal(taps[layer].view(np.uint32), ref_taps[layer].view(np.uint32)), (pos, layer, hidden_gate(taps[layer], ref_taps[layer]))
        logits = eng.forward_token_logits(emb, c, s, pos, pair.scale)
        assert np.array_equal(logits.view(np.uint32), ref_logits.view(np.uint32)), hidden_gate(logits, ref_logits)
    ref_tokens, _, gaps = ref.generate(prompt, 40, want_gaps=True)
    first = eng.prefill_tokens(1, prompt, 0)
    got = np.concatenate([[first], eng.decode_greedy([1], [first], [len(prompt)], 39)[:, 0]])
    n_match, gap = greedy_match(got, ref_tokens, gaps)
    assert n_match == 40, (n_match, gap)


@pytest.mark.parametrize("qt", [12, 14])  # Q4_K, Q6_K experts
@pytest.mark.parametrize("n", [9, 11, 37, 150, 301])
def test_moe_prompts_equal_the_serial_path(cm, orc, qt, n):
    """Prompts that give an expert 1 to 100 and more assignments, on a shape with few row tiles: the row product (9 tokens), and
    one and two assignments per thread of the tiled product in many passes."""
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny-moe", max_pos=352)
    pair = ModelPair(cfg, "q4_k_m", seed=33)
    eng, ref = pair.engine, pair.oracle
    for layer in range(cfg.n_layers):
        router = np.random.default_rng(layer).normal(0, 0.1, (cfg.n_experts, cfg.hidden)).astype(np.float32)
        exps = [(qt, orc.synth_tensor(qt, 41, 10 * layer + i, cfg.n_experts * r, c, 0.02))
                for i, (r, c) in enumerate([(cfg.ffn_dim, cfg.hidden), (cfg.ffn_dim, cfg.hidden), (cfg.hidden, cfg.ffn_dim)])]
        eng.set_layer_moe(layer, router, *exps)
        ref.set_moe(layer, router, *exps)
    prompt = orc.synth_tokens(8, 1, n, cfg.vocab)
    for pos, t in enumerate(prompt):
        want, _, _ = ref.forward(ref.embedding(int(t)), pos)
    token, logits = eng.extend(0, prompt, 0, want=[n - 1])
    assert np.array_equal(logits[0].view(np.uint32), want.view(np.uint32)), hidden_gate(logits[0], want)
    assert token == orc.argmax(want)


@pytest.mark.parametrize("qt", [12, 14])  # Q4_K, Q6_K experts
def test_moe_prompts_on_a_wide_shape(cm, orc, qt):
    """Enough row tiles that gate and up keep the largest passes: prompts whose experts have about 6 to 60 assignments go through
    every number of assignments per thread (1 to 6) and through passes that split an expert's.  The width leaves the router a
    short last chunk."""
    cfg = cm.EngineConfig(n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, hidden=1280, ffn_dim=4864, vocab=256, max_pos=256, n_experts=8, n_experts_used=2)
    pair = ModelPair(cfg, "q4_k_m", seed=33)
    eng, ref = pair.engine, pair.oracle
    router = np.random.default_rng(0).normal(0, 0.1, (cfg.n_experts, cfg.hidden)).astype(np.float32)
    exps = [(qt, orc.synth_tensor(qt, 41, i, cfg.n_experts * r, c, 0.02))
            for i, (r, c) in enumerate([(cfg.ffn_dim, cfg.hidden), (cfg.ffn_dim, cfg.hidden), (cfg.hidden, cfg.ffn_dim)])]
    eng.set_layer_moe(0, router, *exps)
    ref.set_moe(0, router, *exps)
    prompt = orc.synth_tokens(8, 1, 200, cfg.vocab)
    want = np.stack([ref.forward(ref.embedding(int(t)), pos)[0] for pos, t in enumerate(prompt)])
    for n in (3, 24, 45, 66, 97, 130, 163, 200):
        token, logits = eng.extend(0, prompt[:n], 0, want=list(range(n)))
        bad = np.nonzero((logits.view(np.uint32) != want[:n].view(np.uint32)).any(axis=1))[0]
        assert bad.size == 0, (n, bad, hidden_gate(logits, want[:n]))
        assert token == orc.argmax(want[n - 1])


@pytest.mark.parametrize("n", [150, 600])  # one long step
def test_logits_of_long_steps_by_row(cm, orc, n):
    """The rows of a long step whose logits are asked for are gathered 32 at a time: more of them than one pass takes, lists with
    and without the last token (whose greedy token is returned either way), none at all; and the draw from
    the logits of the last token afterwards."""
    cfg = cm.EngineConfig(n_layers=2, n_heads=8, n_kv_heads=4, head_dim=64, hidden=256, ffn_dim=512, vocab=512, max_pos=640)
    pair = ModelPair(cfg, "q4_k_m", seed=61)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(9, 1, n, cfg.vocab)
    all_logits = np.stack([ref.forward(ref.embedding(int(t)), pos)[0] for pos, t in enumerate(prompt)])
    rng = np.random.default_rng(n)
    some = lambda k: sorted(int(i) for i in rng.choice(n - 1, k, replace=False))
    lists = [list(range(n)), list(range(n - 1)), some(32), some(33), some(31) + [n - 1], some(64), some(65), [0], [n - 1], [], list(range(n - 40, n - 1))]
    for want in lists:
        token, logits = eng.extend(0, prompt, 0, want=want)
        assert np.array_equal(logits.view(np.uint32), all_logits[want].view(np.uint32)), want
        assert token == orc.argmax(all_logits[n - 1]), want
        assert eng.sample(1e-6, 7) == token, want  # so cold that the draw is the greedy token


def test_prompt_of_two_long_steps(cm, orc):
    """1100 tokens: steps of 1024 and 76 rows.  Logits at places in both, and the K/V rows, are the checker's."""
    n = 1100
    cfg = cm.EngineConfig(n_layers=2, n_heads=8, n_kv_heads=4, head_dim=64, hidden=256, ffn_dim=512, vocab=512, max_pos=1152)
    pair = ModelPair(cfg, "q4_k_m", seed=63)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(9, 1, n, cfg.vocab)
    all_logits = np.stack([ref.forward(ref.embedding(int(t)), pos)[0] for pos, t in enumerate(prompt)])
    for want in ([0, 127, 128, 1023, 1024, 1099], [500], list(range(1000, 1060)), []):
        token, logits = eng.extend(0, prompt, 0, want=want)
        assert np.array_equal(logits.view(np.uint32), all_logits[want].view(np.uint32)), want
        assert token == orc.argmax(all_logits[n - 1]), want
    for layer in range(cfg.n_layers):
        for got, kept in zip(eng.read_kv_layer(layer, n), ref.read_kv_layer(layer, n)):
            assert np.array_equal(got, kept), layer


def test_long_prefill_from_embeddings_leaves_the_serial_kv(cm, orc):
    """Embedding rows in, long steps of 1024 and 76 rows and a start past row 0: the K/V rows are the checker's."""
    n = 1100
    cfg = cm.EngineConfig(n_layers=2, n_heads=8, n_kv_heads=4, head_dim=64, hidden=256, ffn_dim=512, vocab=512, max_pos=1152)
    pair = ModelPair(cfg, "q4_k_m", seed=62)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(9, 1, n, cfg.vocab)
    embs = np.stack([ref.embedding(int(t)) for t in prompt])
    for pos in range(n):
        ref.forward(embs[pos], pos, want_logits=False)
    cos, sin = (np.stack(t) for t in zip(*[pair.rope(pos) for pos in range(n)]))
    for start in (0, 3):
        eng.prefill_from(embs, cos, sin, n, pair.scale, start)
        for layer in range(cfg.n_layers):
            for got, want in zip(eng.read_kv_layer(layer, n), ref.read_kv_layer(layer, n)):
                assert np.array_equal(got, want), (start, layer)


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 10])  # ten rows give every expert enough assignments for the tiled product
def test_infinite_superblock_scales_give_the_cpus_infinities(cm, orc, rows):
    """Q4_K experts with an infinite scale: a code above 0 stands for an infinity, a code of 0 for NaN, in both expert
    products.  The activations of the down projection are made equal, so that the infinities of a row have one sign."""
    from camelid_b200 import synth

    cfg = cm.EngineConfig(n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, hidden=256, ffn_dim=512, vocab=256, max_pos=32, n_experts=4,
                          n_experts_used=2, max_seqs=rows)
    pair = ModelPair(cfg, "q4_k_m", seed=3)
    eng, ref = pair.engine, pair.oracle
    rng = np.random.default_rng(0)
    router = rng.normal(0, 0.1, (4, 256)).astype(np.float32)
    gate, up = (np.tile(orc.synth_tensor(12, 41, i, 1, 256, 0.02), 4 * 512) for i in range(2))
    down = orc.synth_tensor(12, 41, 2, 4 * 256, 512, 0.02).copy()
    blocks = down.reshape(4, 256, 2, 144)
    blocks[:, 3:6, 1, 4:16] = 0x11   # scales and mins above 0
    blocks[:, 3:6, 1, 16:] |= 0x11   # codes above 0
    blocks[:, 3, 1, 0:2] = [0, 0x7C]  # +inf
    blocks[:, 4, 1, 0:2] = [0, 0xFC]  # -inf
    blocks[:, 5, 1, 0:2] = [0, 0x7C]
    blocks[:, 5, 1, 77] = 0x10
    for m in (eng.set_layer_moe, ref.set_moe):
        m(0, router, (12, gate), (12, up), (12, down))
    with np.errstate(all="ignore"):
        _, want, _ = ref.forward(ref.embedding(7), 0)
    assert np.isinf(want[3]) and want[4] == -want[3] and np.isnan(want[5]) and np.isfinite(np.delete(want, [3, 4, 5])).all()
    _, _, hidden = eng.step_batch(list(range(rows)), [7] * rows, [0] * rows, want_hidden=True)
    for got in hidden:
        assert np.array_equal(got, want, equal_nan=True), (got[3:6], want[3:6])


@pytest.mark.parametrize("heads,kv,hd,first,n", [(16, 16, 64, 0, 150), (16, 8, 64, 3, 150), (8, 4, 128, 0, 300), (12, 4, 64, 0, 301), (12, 4, 64, 900, 301),
                                                  (12, 4, 128, 30, 299), (32, 8, 64, 5, 77), (16, 4, 64, 1400, 150), (16, 4, 128, 0, 161), (32, 4, 64, 100, 75),
                                                  (16, 2, 128, 0, 149), (16, 4, 128, 10, 40), (12, 4, 128, 800, 301), (16, 4, 128, 1300, 161),
                                                  (32, 4, 64, 1300, 150), (32, 4, 128, 1300, 150), (8, 4, 64, 1200, 301), (16, 16, 64, 1300, 150)])
def test_long_prompt_steps_equal_the_serial_path(cm, orc, heads, kv, hd, first, n):
    """Steps of more than 32 rows of one sequence, whose attention serves neighbouring rows together: every group size and
    head dimension, row counts that leave the last group short, contexts that end inside a tile, a start past position 0, long
    contexts (fewer queries per thread, or outputs with three heads per KV head, at both head dimensions), and a step too short
    for it."""
    cfg = cm.EngineConfig(n_layers=2, n_heads=heads, n_kv_heads=kv, head_dim=hd, hidden=256, ffn_dim=512, vocab=512, max_pos=1600)
    pair = ModelPair(cfg, "q4_k_m", seed=61)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(9, 1, first + n, cfg.vocab)
    places = {first + n // 2: None, first + n - 2: None, first + n - 1: None}
    for pos, t in enumerate(prompt):
        lg, _, _ = ref.forward(ref.embedding(int(t)), pos)
        if pos in places:
            places[pos] = np.array(lg)
    if first:
        eng.extend(0, prompt[:first], 0)
    _, logits = eng.extend(0, prompt[first:], first, want=[p - first for p in places])
    for got, want in zip(logits, places.values()):
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), hidden_gate(got, want)


def test_long_prompt_steps_whose_scores_go_by_groups(cm, orc):
    """64 heads without sharing at 2100 positions: the second and third step's scores do not fit the scratch at once.  Against the plain
    reference-order kernels, bit for bit, at places in every step."""
    from camelid_b200 import synth

    def engine(flags):
        cfg = cm.EngineConfig(n_layers=1, n_heads=64, n_kv_heads=64, head_dim=64, hidden=256, ffn_dim=512, vocab=512, max_pos=4096, flags=flags)
        return synth.build_engine(cfg, "q4_k_m", 5)

    prompt = orc.synth_tokens(4, 1, 2100, 512)
    want = [5, 1023, 1024, 1500, 2040, 2047, 2048, 2099]
    (t1, got), (t2, ref) = (engine(flags).extend(0, prompt, 0, want=want) for flags in (0, 16))
    assert t1 == t2 and np.array_equal(got.view(np.uint32), ref.view(np.uint32))


def test_engines_open_on_a_nearly_full_card(monkeypatch, cm, orc):
    """Without room for the prompt attention's scratch, and without room for the rows of the longest steps: the same logits."""
    import torch

    from camelid_b200 import synth
    from camelid_b200.engine import DeviceBuffer

    cfg = cm.EngineConfig(n_layers=1, n_heads=64, n_kv_heads=64, head_dim=64, hidden=4096, ffn_dim=14336, vocab=512, max_pos=4096)
    prompt, want = orc.synth_tokens(4, 1, 1100, 512), [5, 511, 1023, 1024, 1099]
    free = lambda: torch.cuda.mem_get_info()[0]

    def run(eng):
        token, logits = eng.extend(0, prompt, 0, want=want)
        launches = eng.last_timing()[1]
        eng.close()
        return token, logits.view(np.uint32), launches

    run(synth.build_engine(cfg, "q4_k_m", 5))  # (what the library itself loads is in place)
    before = free()
    eng = cm.ResidentDecode(cfg)
    opened = before - free()
    eng.close()
    eng = synth.build_engine(cfg, "q4_k_m", 5)
    held = before - free()
    token, logits, launches = run(eng)
    full = DeviceBuffer(free() - held + (256 << 20))  # half of the scratch is missing
    eng = synth.build_engine(cfg, "q4_k_m", 5)
    del full
    fewer = run(eng)
    assert fewer[0] == token and np.array_equal(fewer[1], logits) and fewer[2] < launches  # one kernel of attention a step in place of three
    full = DeviceBuffer(free() - opened + (64 << 20))
    eng = cm.ResidentDecode(cfg)
    del full
    monkeypatch.setattr(synth, "ResidentDecode", lambda cfg: eng)
    shorter = run(synth.build_engine(cfg, "q4_k_m", 5))
    assert shorter[0] == token and np.array_equal(shorter[1], logits) and shorter[2] > launches  # three steps in place of two


@pytest.mark.parametrize("n", [513, 520, 521])  # 512 and a rest of its own, and the first that is one step
def test_prompts_just_beyond_512_rows(cm, orc, n):
    cfg = cm.EngineConfig(n_layers=2, n_heads=8, n_kv_heads=4, head_dim=64, hidden=256, ffn_dim=512, vocab=512, max_pos=640)
    pair = ModelPair(cfg, "q4_k_m", seed=65)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(9, 1, n, cfg.vocab)
    all_logits = np.stack([ref.forward(ref.embedding(int(t)), pos)[0] for pos, t in enumerate(prompt)])
    launches = {}
    for want in (sorted({0, 511, 512, n - 1}), [511], [512], []):
        token, logits = eng.extend(0, prompt, 0, want=want)
        launches[n] = eng.last_timing()[1]
        assert np.array_equal(logits.view(np.uint32), all_logits[want].view(np.uint32)), want
        assert token == orc.argmax(all_logits[n - 1]), want
    eng.extend(0, prompt[:512], 0)
    assert (launches[n] > eng.last_timing()[1]) == (n <= 520)  # (no logits but the last token's)
    for layer in range(cfg.n_layers):
        eng.extend(0, prompt, 0)
        for got, kept in zip(eng.read_kv_layer(layer, n), ref.read_kv_layer(layer, n)):
            assert np.array_equal(got, kept), layer


@pytest.mark.parametrize("rows, first, kernels", [(36, 2000, 1), (40, 2000, 3), (40, 1000, 1), (36, 6000, 1), (80, 100, 3)])
def test_attention_of_some_rows_at_long_contexts(cm, rows, first, kernels):
    """The row kernel where it is done in two rounds of the machine, the three prompt kernels beyond: as many launches a layer more than with one
    kernel, the same logits as from the plain reference-order kernels."""
    from camelid_b200 import synth

    def engine(layers, flags):
        cfg = cm.EngineConfig(n_layers=layers, n_heads=32, n_kv_heads=8, head_dim=128, hidden=256, ffn_dim=512, vocab=512, max_pos=8192, flags=flags)
        return synth.build_engine(cfg, "q4_k_m", 5)

    def run(eng, tokens, start):
        token, logits = eng.extend(0, tokens, start, want=[0, len(tokens) - 1])
        return token, logits.view(np.uint32), eng.last_timing()[1]

    prompt = np.arange(rows, dtype=np.int32)
    per_layer = run(engine(2, 0), prompt, first)[2] - run(engine(1, 0), prompt, first)[2]
    short = np.arange(36, dtype=np.int32)  # (at a short context always one kernel)
    base = run(engine(2, 0), short, 100)[2] - run(engine(1, 0), short, 100)[2]
    assert per_layer - base == kernels - 1
    got, ref = run(engine(1, 0), prompt, first), run(engine(1, 16), prompt, first)
    assert got[0] == ref[0] and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("slots", [40, 64, 512])
def test_prompts_take_the_same_steps_whatever_the_number_of_slots(cm, orc, slots):
    """A prompt's steps are chosen by its rows: an engine of many slots launches what an engine of one launches (no logits of
    rows that nobody asked for) and gives its bits, the second time as the first (long steps are not captured)."""
    from camelid_b200 import synth

    def engine(n_slots):
        cfg = cm.EngineConfig(n_layers=2, n_heads=8, n_kv_heads=4, head_dim=64, hidden=512, ffn_dim=512, vocab=512, max_pos=1152, max_seqs=n_slots)
        return synth.build_engine(cfg, "q4_k_m", 5)

    one, many = engine(1), engine(slots)
    for n in (40, 200, 600, 1100):
        prompt = orc.synth_tokens(3, 1, n, 512)
        for want in ([], [], [], [0, n // 2, n - 2]):  # a step was captured at its second call and replayed from the third on
            t1, l1 = one.extend(0, prompt, 0, want=want)
            launches = one.last_timing()[1]
            t2, l2 = many.extend(slots - 1, prompt, 0, want=want)
            assert t1 == t2 and np.array_equal(l1.view(np.uint32), l2.view(np.uint32)), (n, want)
            assert many.last_timing()[1] == launches, (n, want)


def test_tensor_batch_flag_moves_small_batches_to_the_tensor_core_kernel(cm, orc):
    """CMLD_FLAG_TENSOR_BATCH (64): steps of 5..32 rows use the int8 mma.sync matvec.  Same integers, f32 terms
    added in another order: logits within the acceptance gate of the default engine's, and the rows of such a
    step do not depend on their neighbours."""
    from camelid_b200 import synth
    from helpers import hidden_gate

    cfg = synth.engine_config("tiny", max_pos=64, max_seqs=6)
    base = synth.build_engine(cfg, "q4_k_m", 5)
    fast = synth.build_engine(synth.engine_config("tiny", max_pos=64, max_seqs=6, flags=64), "q4_k_m", 5)
    toks = [3, 7, 11, 19, 23, 29]
    seqs = list(range(6))
    _, l0, h0 = base.step_batch(seqs, toks, [0] * 6, want_logits=True, want_hidden=True)
    _, l1, h1 = fast.step_batch(seqs, toks, [0] * 6, want_logits=True, want_hidden=True)
    ok, max_abs, rel = hidden_gate(l1, l0)
    assert ok, (max_abs, rel)
    _, l2, _ = fast.step_batch(seqs[::-1], toks[::-1], [0] * 6, want_logits=True)
    assert np.array_equal(l2[::-1], l1)
    base.close()
    fast.close()


# Continuous batching (ContinuousBatch::run_round, src/api/continuous_batch.rs:86-104): a round is N
# independent serial token steps, so the oracle for a 16- or 32-row step is N single-sequence runs of
# the checker.  "small" is wide enough (hidden 4096) for every matvec to take the staged kernel.
@pytest.mark.parametrize("shape,mix,rows", [("small", "q4_k_m", 16), ("small", "q4_k_m", 32), ("small", "q8_0", 32),
                                             ("tiny-moe", "q4_k_m", 16), ("tiny-moe", "q4_k_m", 32)])
def test_steps_of_16_and_32_rows_equal_independent_sequences(cm, orc, shape, mix, rows):
    from camelid_b200 import synth

    cfg = synth.engine_config(shape, max_pos=48, max_seqs=rows)
    pair = ModelPair(cfg, mix, seed=77)
    eng, ref = pair.engine, pair.oracle
    prompts = [orc.synth_tokens(50 + s, 1, 3 + s % 5, cfg.vocab) for s in range(rows)]
    firsts = [eng.prefill_tokens(s, prompts[s], 0) for s in range(rows)]
    # the checker, one sequence at a time: prompt, then the logits of the step that follows it
    want_first, want_logits = [], []
    for s in range(rows):
        for pos, t in enumerate(prompts[s]):
            lg, _, _ = ref.forward(ref.embedding(int(t)), pos)
        want_first.append(orc.argmax(lg))
        lg, _, _ = ref.forward(ref.embedding(want_first[-1]), len(prompts[s]))
        want_logits.append(lg)
    assert firsts == want_first
    toks, lg, _ = eng.step_batch(list(range(rows)), firsts, [len(p) for p in prompts], want_logits=True)
    for s in range(rows):
        assert np.array_equal(lg[s].view(np.uint32), want_logits[s].view(np.uint32)), (s, hidden_gate(lg[s], want_logits[s]))
        assert toks[s] == orc.argmax(want_logits[s])
    # rows do not depend on their neighbours: the same rows in another order
    order = list(range(rows))[::-1]
    _, lg2, _ = eng.step_batch(order, [firsts[s] for s in order], [len(prompts[s]) for s in order], want_logits=True)
    assert np.array_equal(lg2[::-1], lg)


def test_prefill_of_40_rows_leaves_the_serial_kv(cm, orc):
    """prefill_then_decode_matches_sequential (src/cuda_resident/tests.rs:3143): a 40-token prompt ingested in
    one step leaves the KV rows, and gives the next token, of token-by-token steps — which are the checker's."""
    from camelid_b200 import synth

    cfg = synth.engine_config("small", max_pos=64, max_seqs=2)
    pair = ModelPair(cfg, "q4_k_m", seed=78)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(9, 1, 40, cfg.vocab)
    first = eng.prefill_tokens(0, prompt, 0)
    tok = None
    for pos, t in enumerate(prompt):  # serial steps on the second sequence
        tok, _, _ = eng.step_batch([1], [int(t)], [pos])
        lg, _, _ = ref.forward(ref.embedding(int(t)), pos)
    assert first == int(tok[0]) == orc.argmax(lg)
    for layer in range(cfg.n_layers):
        rk, rv = ref.read_kv_layer(layer, len(prompt))
        k0, v0 = eng.read_kv_layer(layer, len(prompt))
        assert np.array_equal(k0, rk) and np.array_equal(v0, rv), layer


def test_verify_tree_predicts_what_a_linear_decode_of_each_path_predicts(cm, orc):
    """verify_tree (src/cuda_resident.rs:22944): every node of a draft tree in one batched pass.  The token predicted
    after node i equals the CPU checker's greedy token after prompt + the tokens on the path to node i (lossless
    speculation, :4343-4352); after compact_tree_kv_path the cache is that of a linear decode of the accepted path,
    so decoding on gives the checker's tokens."""
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny", max_pos=96)
    pair = ModelPair(cfg, "q4_k_m", seed=41)
    eng, ref = pair.engine, pair.oracle
    prompt = orc.synth_tokens(41, 5, 7, cfg.vocab)
    base = len(prompt)
    root = eng.prefill_tokens(0, prompt, 0)
    truth, _ = ref.generate(prompt, 8)  # the greedy continuation: truth[0] is the root token
    assert root == truth[0]
    # breadth-first tree: node 0 = root; one branch follows the greedy continuation for three steps, others do not
    parents = [-1, 0, 0, 0, 1, 1, 2, 4, 4, 7, 7, 9]
    rng = np.random.default_rng(9)
    tokens = [int(root)] + [int(t) for t in rng.integers(0, cfg.vocab, len(parents) - 1)]
    tokens[2] = int(truth[1])           # child of the root on the greedy path
    tokens[6] = int(truth[2])           # its child
    depth = [0] * len(parents)
    for i, par in enumerate(parents):
        if par >= 0:
            depth[i] = depth[par] + 1
    emb = np.stack([ref.embedding(t) for t in tokens])
    cs = [pair.rope(base + d) for d in depth]
    got = eng.verify_tree(emb, np.stack([c for c, _ in cs]), np.stack([s for _, s in cs]), parents, base, pair.scale)
    for i in range(len(parents)):
        path, j = [], i
        while j >= 0:
            path.append(tokens[j])
            j = parents[j]
        seq = np.concatenate([prompt, np.array(path[::-1], np.int32)])
        want, _ = ref.generate(seq, 1)
        assert got[i] == want[0], (i, got[i], want[0])
    # accept the longest path whose tokens are the model's own predictions: 0 -> 2 -> 6
    accepted = [0]
    while True:
        nxt = [j for j, par in enumerate(parents) if par == accepted[-1] and tokens[j] == got[accepted[-1]]]
        if not nxt:
            break
        accepted.append(nxt[0])
    assert accepted == [0, 2, 6]
    eng.compact_tree_kv_path(accepted, base)
    n_acc = len(accepted)
    cont = eng.decode_greedy([0], [int(got[accepted[-1]])], [base + n_acc], 4)[:, 0]
    assert int(got[accepted[-1]]) == truth[n_acc] and np.array_equal(cont, truth[n_acc + 1: n_acc + 5]), (cont, truth)
    # argument checks: a node may not name a later node, rows must be base + index
    with pytest.raises(cm.CmldError):
        eng.verify_tree(emb[:2], np.stack([cs[0][0], cs[1][0]]), np.stack([cs[0][1], cs[1][1]]), [-1, 0], cfg.max_pos - 1, pair.scale)


def test_forward_token_sample_draws_from_the_steps_own_logits(cm, orc):
    """forward_token_sample (src/cuda_resident.rs:20163): the token drawn on the device is the checker's draw over the
    logits of the very same forward pass (bit-identical to the CPU path's), with and without the min-p filter."""
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny", max_pos=64)
    pair = ModelPair(cfg, "q4_k_m", seed=3)
    eng, ref = pair.engine, pair.oracle
    tok = 5
    for pos in range(6):
        emb = ref.embedding(tok)
        c, s = pair.rope(pos)
        ref_logits, _, _ = ref.forward(emb, pos)
        if pos % 2 == 0:
            got = eng.forward_token_sample(emb, c, s, pos, pair.scale, 0.9, 1000 + pos)
            want, scores = orc.sample_gumbel(ref_logits, np.float32(1.0) / np.float32(0.9), 1000 + pos)
        else:
            got = eng.forward_token_sample(emb, c, s, pos, pair.scale, 0.9, 1000 + pos, min_p=0.05)
            want, scores = orc.sample_gumbel_filtered(ref_logits, 0.9, 0.05, 1000 + pos)
        if isinstance(got, tuple):  # the filter handed the row back: the logits come with it, bit for bit
            assert got[0] is None and np.array_equal(got[1].view(np.uint32), ref_logits.view(np.uint32))
            got = want if want >= 0 else int(np.argmax(ref_logits))
        else:
            assert want >= 0 and (got == want or abs(float(scores[got]) - float(scores[want])) <= 1e-5 * max(1.0, abs(float(scores[want]))))
        tok = int(got)


def test_q8_0_kv_cache_follows_the_cpu_lanes_scalar_arithmetic(cm, orc):
    """CMLD_FLAG_KV_Q8_0 (new_with_kv_quant, src/cuda_resident.rs:15748): K and V rows are kept as Q8_0 blocks
    (quantize_block_q8_0, src/tensor/kv_quant.rs:123) and attention runs over the blocks in the order of the CPU
    lane's scalar path (vec_dot_row_q8_0 :180, axpy_row_q8_0 :203).  Against the checker holding its cache the same
    way: residual stream, logits, cache rows and greedy tokens are bit-identical.  (The reference's AVX2 path adds in
    another order; its own test holds the two to 1e-5.)"""
    from camelid_b200 import synth

    cfg = synth.engine_config("tiny", max_pos=64, flags=256)
    pair = ModelPair(cfg, "q4_k_m", seed=19)
    eng, ref = pair.engine, pair.oracle
    ref.set_kv_q8(True)
    prompt = orc.synth_tokens(19, 5, 9, cfg.vocab)
    for pos in range(5):
        emb = ref.embedding(int(prompt[pos]))
        c, s = pair.rope(pos)
        ref_logits, _, ref_taps = ref.forward(emb, pos, want_taps=True)
        _, taps = eng.forward_token_hidden(emb, c, s, pos, pair.scale, taps=True)
        logits = eng.forward_token_logits(emb, c, s, pos, pair.scale)
        assert np.array_equal(taps.view(np.uint32), ref_taps.view(np.uint32)), pos
        assert np.array_equal(logits.view(np.uint32), ref_logits.view(np.uint32)), pos
    # the cache rows read back dequantised (code * d): what the blocks hold is what the checker's blocks hold
    ck, cv = eng.read_kv_layer(1, 5)
    nb = cfg.head_dim // 32
    kq, vq = ref.read_kv_layer(1, 5)          # the checker keeps codes (as floats) ...
    assert np.all(np.abs(kq) <= 127) and np.array_equal(kq, np.round(kq))
    ratio = np.where(kq != 0, ck / np.where(kq != 0, kq, 1), 0).reshape(cfg.n_kv_heads, 5, nb, 32)
    for blk in ratio.reshape(-1, 32):          # ... so every block's values are one scale times its codes
        nz = blk[blk != 0]
        assert nz.size == 0 or np.all(nz == nz[0])
    # a full generation: prompt through the 32-row chunks, then greedy steps
    ref2 = ModelPair(cfg, "q4_k_m", seed=19)
    ref2.oracle.set_kv_q8(True)
    want, _ = ref2.oracle.generate(prompt, 24)
    first = ref2.engine.prefill_tokens(0, prompt, 0)
    rest = ref2.engine.decode_greedy([0], [first], [len(prompt)], 23)[:, 0]
    assert np.array_equal(np.concatenate([[first], rest]), want)
    # seeding quantises rows exactly like an append does
    rows = np.random.default_rng(2).standard_normal((cfg.n_kv_heads, 3, cfg.head_dim)).astype(np.float32)
    eng.seed_layer(0, rows, rows * 0.5, 3)
    back_k, back_v = eng.read_kv_layer(0, 3)
    import ctypes as C
    for kh in range(cfg.n_kv_heads):
        for p in range(3):
            for b in range(nb):
                codes = np.empty(32, np.float32)
                blk = np.ascontiguousarray(rows[kh, p, 32 * b: 32 * b + 32])
                d = orc.lib().orc_kv_q8_0_quantize_block(blk.ctypes.data_as(C.c_void_p), codes.ctypes.data_as(C.c_void_p))
                assert np.array_equal(back_k[kh, p, 32 * b: 32 * b + 32], (codes * np.float32(d)).astype(np.float32))
