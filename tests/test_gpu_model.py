"""GPU parity of the resident decode model against the oracle's decode loop.

A small Qwen3MoE-shaped model (2 layers, 8 experts, 2 active) is decoded token
by token on both sides from the same seeded weights. Expert ids and greedy
token ids must be identical; hidden states, K/V and logits are compared bit
for bit where no exp() is upstream, and at the reference's named tolerances
(crates/llamd-core/src/tolerance.rs) after one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYER = 1e-4      # tolerance.rs:100
LOGITS = 2e-3     # tolerance.rs:109
ATTENTION = 1e-5  # tolerance.rs:97


def max_dev(a, b):
    """llamd_core::tolerance::max_deviation (tolerance.rs:135-151)."""
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.max(np.abs(a - b) / np.maximum(np.maximum(np.abs(a), np.abs(b)), 1.0)))


@pytest.fixture(scope="module")
def tiny():
    from llamd_rs_b200 import backend, synth
    from llamd_rs_b200.model import CudaModel
    import oracle

    if not backend.available():
        pytest.fail("no CUDA device: the GPU tests must run on a GPU box")
    hp = synth.TINY
    w = synth.make_model(hp, seed=7)
    gm = CudaModel.load_batched(hp, w, max_kv=64, max_seq=4)
    om = oracle.Model(hp, w, threads=4)
    yield hp, w, gm, om
    gm.free()


def test_bad_arguments_are_refused(tiny):
    from llamd_rs_b200 import backend
    from llamd_rs_b200.model import CudaModel

    hp, w, gm, om = tiny
    with pytest.raises(backend.Malformed):
        CudaModel(hp, 0)
    with pytest.raises(backend.Malformed):
        CudaModel(hp, 16, backend.MAX_BATCH + 1)
    with pytest.raises(backend.Malformed):
        gm.forward(1, 64)
    with pytest.raises(backend.Other):
        gm.forward(hp["n_vocab"], 0)
    assert gm.weight_bytes() > 0 and gm.hparams()["n_layer"] == 2


def test_first_token_layer_by_layer(tiny):
    """Position 0: softmax over one key is exactly 1, so nothing upstream of the
    router depends on exp(); the routing itself does."""
    hp, w, gm, om = tiny
    om.kv_new(64)
    gm.set_trace(True)
    tok = 17
    got_tok = gm.forward(tok, 0)
    gx, gids = gm.read_trace()
    gm.set_trace(False)
    import oracle

    x = oracle.dequantize(oracle.Q6K, w["tok_embd"][tok * hp["n_embd"] // 256 * 210:], hp["n_embd"])
    for il in range(hp["n_layer"]):
        x, tr = om.forward_layer(il, x, 0)
        assert gids[il, 0].tolist() == tr["experts"].tolist(), f"layer {il} expert ids"
        assert max_dev(gx[il, 0], x) <= LAYER, f"layer {il} hidden state"
        gk, gv = gm.read_kv(il, 1)
        ok, ov = om.kv_layer(il, 1)
        assert np.array_equal(gv.view(np.uint32), ov.view(np.uint32)) or il > 0, "layer 0 V is exp-free: bit-exact"
        assert max_dev(gk, ok) <= ATTENTION and max_dev(gv, ov) <= ATTENTION
    om.kv_new(64)
    logits = om.forward(tok, 0)
    assert max_dev(gm.logits()[0], logits) <= LOGITS
    assert got_tok == oracle.argmax(logits)


def test_greedy_decode_matches_token_for_token(tiny):
    """Prompt of 6 ids, then 10 greedy tokens: ids EXACT, logits at LOGITS."""
    import oracle
    from llamd_rs_b200 import synth

    hp, w, gm, om = tiny
    prompt = synth.token_ids(6, hp["n_vocab"], 3, "prompt").tolist()
    om.kv_new(64)
    want, got = [], []
    worst = 0.0
    tok_o = tok_g = None
    for pos in range(16):
        t_in_o = prompt[pos] if pos < len(prompt) else tok_o
        t_in_g = prompt[pos] if pos < len(prompt) else tok_g
        lo = om.forward(t_in_o, pos)
        tok_o = oracle.argmax(lo)
        tok_g = gm.forward(t_in_g, pos)
        worst = max(worst, max_dev(gm.logits()[0], lo))
        want.append(tok_o)
        got.append(tok_g)
        assert tok_g == tok_o, f"token {pos}: gpu {got} cpu {want}"
    assert worst <= LOGITS, f"logits deviate by {worst}"


def test_graph_replay_equals_plain_queueing(tiny):
    hp, w, gm, om = tiny
    gm.use_graph = False
    a = [gm.forward(5 + p, p) for p in range(5)]
    la = gm.logits()[0]
    gm.use_graph = True
    b = [gm.forward(5 + p, p) for p in range(5)]
    lb = gm.logits()[0]
    assert a == b and np.array_equal(la.view(np.uint32), lb.view(np.uint32))


def test_batch_equals_single(tiny):
    """crates/llamd-testing/tests/batch_decode.rs:102-125: N sequences in one
    pass give the tokens (and here the logits, bit for bit) of N single passes."""
    hp, w, gm, om = tiny
    seqs = [[3, 9, 27], [100, 200, 300], [7, 7, 7], [511, 0, 255]]
    single_tokens, single_logits = [], []
    for s in seqs:
        toks = []
        for pos, t in enumerate(s):
            toks.append(gm.forward(t, pos))
        single_tokens.append(toks)
        single_logits.append(gm.logits()[0].copy())
    # batched: all four sequences advance together (each in its own KV slot)
    for pos in range(3):
        out = gm.forward_batch([s[pos] for s in seqs], [pos] * 4)
        assert out.tolist() == [st[pos] for st in single_tokens]
    lb = gm.logits(4)
    for i in range(4):
        assert np.array_equal(lb[i].view(np.uint32), single_logits[i].view(np.uint32)), f"sequence {i} logits"


def test_fused_tails_change_nothing(tiny):
    """The decode pass with the attention-quantize and SiLU-quantize tails inside their producers (option
    fuse_tails) and with the separate launches (default): same tokens, same logits, bit for bit."""
    hp, w, gm, om = tiny
    runs = {}
    for fuse in (0, 1, 0):
        gm.set_option("fuse_tails", fuse)
        toks, tok = [], 3
        for pos in range(6):
            tok = gm.forward(tok, pos)
            toks.append(tok)
        runs.setdefault(fuse, []).append((toks, gm.logits()[0].copy()))
    gm.set_option("fuse_tails", 0)
    ref_t, ref_l = runs[1][0]
    for t, l in runs[0]:
        assert t == ref_t and np.array_equal(l.view(np.uint32), ref_l.view(np.uint32))


@pytest.mark.parametrize("option", ["fuse_norm_router", "fuse_rope_attn", "fuse_norm_qkv", "fuse_silu_down", "early_loads", "fuse_attn_quant", "sort_slots", "head_gemm", "dense_gemm"])
def test_fused_launches_change_nothing(tiny, option):
    """The decode pass with the FFN norm and the router as one launch (option fuse_norm_router), with QK-norm, RoPE and
    the KV store inside the attention-scores launch (option fuse_rope_attn), and with the attention norm and the MoE combine
    inside the QKV matvec (option fuse_norm_qkv; off by default), and with the loads that do not depend on the launch in
    front issued before the dependency wait (option early_loads), and with the expert launches taking their slots in expert
    order (option sort_slots), and with the output projection, or the attention projections, on the integer GEMM over folded
    copies of their matrices (options head_gemm, dense_gemm) -- against the separate launches, the late loads, the slots in routing order and the output matvec: same tokens, same hidden states after every layer, same routed experts, same logits and cache rows, bit for
    bit; one and four sequences. (Positions beyond a 64-position tile, where the token's own row moves from tile to tile, are
    covered by the 768-position run against the CPU fixture, which uses the defaults.)"""
    hp, w, gm, om = tiny
    runs = {}
    default = 0 if option in ("fuse_norm_qkv", "fuse_silu_down", "fuse_attn_quant") else 1  # (measured no faster, so off unless asked for)
    if option == "sort_slots":
        default = 8  # (the number of sequences from which the expert launches take their slots in expert order; 1: always)
    if option == "head_gemm":
        default = 4  # (the number of sequences from which the output projection runs on the integer GEMM; 1: always)
    if option == "dense_gemm":
        default = 8  # (the same for the attention projections)
    for fuse in (1, 0, 1):
        gm.set_option(option, fuse)
        gm.set_trace(True)
        toks, tok, traces = [], 3, []
        for pos in range(6):
            tok = gm.forward(tok, pos)
            toks.append(tok)
            x, ids = gm.read_trace()
            traces.append((x.copy(), ids.copy()))
        gm.set_trace(False)
        batch = [gm.forward_batch([5 + pos, 9, 100 + pos, 7], [pos] * 4).tolist() for pos in range(3)]
        kv = [gm.read_kv(il, 3) for il in range(hp["n_layer"])]
        runs.setdefault(fuse, []).append((toks, traces, gm.logits(4).copy(), batch, kv))
    gm.set_option(option, default)
    ref = runs[0][0]
    for toks, traces, logits, batch, kv in runs[1]:
        assert toks == ref[0] and batch == ref[3]
        assert np.array_equal(logits.view(np.uint32), ref[2].view(np.uint32))
        for (k, v), (rk, rv) in zip(kv, ref[4]):
            assert np.array_equal(k.view(np.uint32), rk.view(np.uint32)) and np.array_equal(v.view(np.uint32), rv.view(np.uint32))
        for (x, ids), (rx, rids) in zip(traces, ref[1]):
            assert np.array_equal(x.view(np.uint32), rx.view(np.uint32)) and np.array_equal(ids, rids)


@pytest.mark.parametrize("kv_f16", [0, 1])
def test_attention_output_leaves_its_launch_quantized(kv_f16):
    """Heads of 128: the eight CTAs that make a 256-element block of the attention output form a cluster, exchange their
    largest magnitudes through distributed shared memory and write the block's Q8_K form themselves (option fuse_attn_quant;
    off by default, measured slower) -- against the separate quantize launch: the same tokens, hidden states, experts, logits and cache rows, bit
    for bit; one and four sequences; against the oracle for the first tokens. Also with the loads before the wait off."""
    import oracle
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(n_layer=2, n_embd=256, n_head=4, n_head_kv=2, head_dim=128, n_expert=8, n_expert_used=2, n_ff_expert=256, n_vocab=512,
              rope_freq_base=1e7, rms_eps=1e-6)
    w = synth.make_model(hp, seed=11)
    gm = CudaModel.load_batched(hp, w, max_kv=96, max_seq=4)
    try:
        if kv_f16:
            gm.set_option("kv_f16", 1)
        runs = []
        for fuse, early in ((1, 1), (0, 1), (1, 0), (1, 1)):
            gm.set_option("fuse_attn_quant", fuse)
            gm.set_option("early_loads", early)
            gm.set_trace(True)
            toks, tok, traces = [], 3, []
            for pos in range(70):  # (past one 64-position tile of the scores launch)
                tok = gm.forward(tok, pos)
                toks.append(tok)
                if pos < 6 or pos > 62:
                    x, ids = gm.read_trace()
                    traces.append((x.copy(), ids.copy()))
            gm.set_trace(False)
            batch = [gm.forward_batch([5 + pos, 9, 100 + pos, 7], [pos] * 4).tolist() for pos in range(3)]
            runs.append((toks, traces, gm.logits(4).copy(), batch, [gm.read_kv(il, 3) for il in range(hp["n_layer"])]))
        ref = runs[1]
        for toks, traces, logits, batch, kv in (runs[0], runs[2], runs[3]):
            assert toks == ref[0] and batch == ref[3]
            assert np.array_equal(logits.view(np.uint32), ref[2].view(np.uint32))
            for (k, v), (rk, rv) in zip(kv, ref[4]):
                assert np.array_equal(k.view(np.uint32), rk.view(np.uint32)) and np.array_equal(v.view(np.uint32), rv.view(np.uint32))
            for (x, ids), (rx, rids) in zip(traces, ref[1]):
                assert np.array_equal(x.view(np.uint32), rx.view(np.uint32)) and np.array_equal(ids, rids)
        if not kv_f16:
            om = oracle.Model(hp, w, threads=4)
            om.kv_new(96)
            tok = 3
            for pos in range(8):
                tok = oracle.argmax(om.forward(tok, pos))
                assert tok == ref[0][pos], f"position {pos}"
    finally:
        gm.free()


@pytest.mark.parametrize("kv_f16", [0, 1])
def test_batch_attention_per_kv_head(kv_f16):
    """Eight query heads of 128 per kv head: a batch of sequences runs attention as one CTA per kv head for all of them
    (option attn_gqa, the default, from four sequences on). Sequences at different positions, across the 64-position score tiles and the
    256-position value tiles: each sequence's tokens, logits and cache rows equal a single-sequence run's, bit for bit, and
    the per-head kernels' on the same batch."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(n_layer=2, n_embd=256, n_head=8, n_head_kv=1, head_dim=128, n_expert=8, n_expert_used=2, n_ff_expert=256, n_vocab=512,
              rope_freq_base=1e7, rms_eps=1e-6)
    w = synth.make_model(hp, seed=13)
    gm = CudaModel.load_batched(hp, w, max_kv=320, max_seq=4)
    try:
        if kv_f16:
            gm.set_option("kv_f16", 1)
        lens = [300, 70, 5, 130]  # the sequences end at different positions
        prompts = [synth.token_ids(n, hp["n_vocab"], 40 + i, "gqa").tolist() for i, n in enumerate(lens)]
        single = []
        for s_, pr in enumerate(prompts):
            for pos, t in enumerate(pr):
                tok = gm.forward(t, pos)
            single.append((tok, gm.logits()[0].copy(), [gm.read_kv(il, len(pr)) for il in range(hp["n_layer"])]))
        runs = {}
        for gqa in (1, 0):
            gm.set_option("attn_gqa", gqa)
            # the four sequences advance together while they last; a finished one repeats its last token at its last position
            for step in range(max(lens)):
                toks = [pr[min(step, len(pr) - 1)] for pr in prompts]
                poss = [min(step, len(pr) - 1) for pr in prompts]
                out = gm.forward_batch(toks, poss)
            runs[gqa] = (out.tolist(), gm.logits(4).copy())
        gm.set_option("attn_gqa", 1)
        assert runs[1][0] == runs[0][0] and np.array_equal(runs[1][1].view(np.uint32), runs[0][1].view(np.uint32))
        for s_ in range(4):  # (a finished sequence repeated its last position: the same row, the same logits)
            assert runs[1][0][s_] == single[s_][0], f"sequence {s_}"
            assert np.array_equal(runs[1][1][s_].view(np.uint32), single[s_][1].view(np.uint32)), f"sequence {s_}: logits"
            for il in range(hp["n_layer"]):
                k, v = gm.read_kv(il, lens[s_], s_)
                rk, rv = single[s_][2][il]
                assert np.array_equal(k.view(np.uint32), rk.view(np.uint32)) and np.array_equal(v.view(np.uint32), rv.view(np.uint32))
    finally:
        gm.free()


@pytest.mark.parametrize("n", [1, 8, 9, 12, 13, 56, 57])
def test_small_tiles_equal_gemm_tiles(tiny, n):
    """A tile's matrices run on the decode pass's launches up to matvec_batch_max tokens and on the tile GEMMs beyond: the
    same logits and cache rows on both sides of the line, and the same picks from a verification."""
    from llamd_rs_b200 import synth

    hp, w, gm, om = tiny
    prompt = synth.token_ids(n, hp["n_vocab"], 11, "prefill").tolist()
    runs = []
    for line in (8, 256):
        gm.set_option("matvec_batch_max", line)
        tok = gm.prefill(prompt, 0)
        runs.append((tok, gm.logits()[0].view(np.uint32).copy(), gm.read_kv(hp["n_layer"] - 1, n), list(gm.verify(prompt, 0))))
    gm.set_option("matvec_batch_max", 56)
    a, b = runs
    assert a[0] == b[0] and np.array_equal(a[1], b[1]) and a[3] == b[3] and a[3][-1] == a[0]
    assert np.array_equal(a[2][0].view(np.uint32), b[2][0].view(np.uint32)) and np.array_equal(a[2][1].view(np.uint32), b[2][1].view(np.uint32))


@pytest.mark.parametrize("kv16", [0, 1])
def test_small_tile_attention_equals_the_tile_kernels(kv16):
    """Eight heads of 128 per kv head: a small tile's attention runs on the kernels that take a kv head's query heads together.
    Against the tile kernels (option attn_gqa off) across the 64-position score tiles and the 224- and 256-position value tiles."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_head=8, n_head_kv=1, head_dim=128)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=9), max_kv=400, max_seq=1)
    try:
        if kv16:
            gm.set_option("kv_f16", 1)
        toks = synth.token_ids(400, hp["n_vocab"], 3, "small tile").tolist()
        gm.prefill(toks[:340], 0)
        for base, n in [(0, 1), (0, 9), (60, 9), (200, 56), (220, 8), (250, 40), (340, 37)]:
            runs = []
            for gqa in (1, 0):
                gm.set_option("attn_gqa", gqa)
                runs.append((list(gm.verify(toks[base:base + n], base)), gm.prefill(toks[base:base + n], base), gm.logits()[0].view(np.uint32).copy()))
            assert runs[0][:2] == runs[1][:2] and np.array_equal(runs[0][2], runs[1][2]), f"{n} tokens from {base}"
    finally:
        gm.free()


def test_prefill_equals_sequential_decode(tiny):
    """crates/llamd-testing/tests/vulkan_prefill.rs:48-136: prefill gives the token (and here the logits and the
    K/V cache, bit for bit) of sequential decode, for (tile, length) pairs that straddle tile and chunk boundaries."""
    from llamd_rs_b200 import backend, synth

    hp, w, gm, om = tiny
    prompt = synth.token_ids(37, hp["n_vocab"], 5, "prefill").tolist()
    seq_tok, seq_logits = {}, {}
    for pos, t in enumerate(prompt):
        seq_tok[pos + 1] = gm.forward(t, pos)
        seq_logits[pos + 1] = gm.logits()[0].copy()
    kv_ref = [gm.read_kv(il, len(prompt)) for il in range(hp["n_layer"])]
    for tile, length in [(1, 1), (1, 5), (2, 5), (4, 4), (4, 5), (8, 7), (8, 8), (8, 9), (8, 17), (16, 33), (16, 37), (64, 37), (512, 37)]:
        gm.prefill_tile = tile
        for gemm, attn in ((True, True), (False, True), (True, False)):  # integer tensor path / dp4a; tiled / per-token attention
            gm.set_prefill_gemm(gemm)
            gm.set_prefill_attn(attn)
            got = gm.prefill(prompt[:length], 0)
            assert got == seq_tok[length], f"tile {tile} length {length} gemm {gemm} attn {attn}"
            assert np.array_equal(gm.logits()[0].view(np.uint32), seq_logits[length].view(np.uint32)), f"tile {tile} length {length}: logits"
    gm.set_prefill_gemm(True)
    gm.set_prefill_attn(True)
    # the expert matrices folded once and kept (option prefill_prefold): the grouped GEMM copies operands instead of
    # folding them, the same bits
    gm.set_option("prefill_prefold", 1)
    for tile, length in [(4, 5), (8, 17), (16, 37), (512, 37)]:
        gm.prefill_tile = tile
        got = gm.prefill(prompt[:length], 0)
        assert got == seq_tok[length], f"prefold: tile {tile} length {length}"
        assert np.array_equal(gm.logits()[0].view(np.uint32), seq_logits[length].view(np.uint32)), f"prefold: tile {tile} length {length}: logits"
    gm.set_option("prefill_prefold", 0)
    gm.prefill_tile = 512
    assert gm.prefill(prompt, 0) == seq_tok[len(prompt)]
    for il in range(hp["n_layer"]):
        k, v = gm.read_kv(il, len(prompt))
        assert np.array_equal(k.view(np.uint32), kv_ref[il][0].view(np.uint32)) and np.array_equal(v.view(np.uint32), kv_ref[il][1].view(np.uint32))
    # chunked: a later call continues at base_pos, and decode continues after a prefill
    gm.prefill_tile = 8
    gm.prefill(prompt[:20], 0)
    assert gm.prefill(prompt[20:], 20) == seq_tok[37]
    gm.prefill(prompt[:12], 0)
    assert gm.forward(prompt[12], 12) == seq_tok[13]
    with pytest.raises(backend.Other):
        gm.prefill(prompt, 40)  # runs past the 64 allocated positions
    with pytest.raises(backend.Malformed):
        gm.prefill([], 0)
    gm.prefill_tile = 512


class _FullDevice:
    """All but `leave` bytes of the device's free memory taken, in as few allocations as it allows."""

    def __init__(self, leave):
        from llamd_rs_b200 import backend
        from llamd_rs_b200._lib import lib

        self.L, self.held = lib(), []
        for size in (8 << 30, 1 << 30, 128 << 20, 16 << 20, 2 << 20):
            while backend.free_memory() >= leave + size:
                p = self.L.llamd_fwd_alloc(size)
                if not p:
                    self.L.llamd_fwd_last_error()  # (refused: smaller pieces)
                    break
                self.held.append(p)

    def release(self):
        for p in self.held:
            self.L.llamd_fwd_free(p)
        self.held = []


def test_prefill_after_a_failed_growth():
    """Tile buffers that could not grow for a long prompt: the call is refused, and the next prompt, whose tile is no larger
    than the old one, allocates again instead of running on what was released."""
    from llamd_rs_b200 import backend, synth
    from llamd_rs_b200._lib import lib
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_ff_expert=2048)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=9), max_kv=4096, max_seq=1)
    try:
        toks = synth.token_ids(4096, hp["n_vocab"], 3, "growth").tolist()
        gm.prefill_tile = 16
        want = gm.prefill(toks[:20], 0), gm.logits()[0].view(np.uint32).copy()
        gm.verify(toks[:9], 0)
        gm.prefill_tile = 4096
        full = _FullDevice(96 << 20)  # (the buffers of 4096 tokens take 300 MB)
        try:
            with pytest.raises(backend.Other):
                gm.prefill(toks, 0)
        finally:
            full.release()
        lib().llamd_fwd_last_error()
        gm.prefill_tile = 16
        got = gm.prefill(toks[:20], 0), gm.logits()[0].view(np.uint32).copy()
        assert got[0] == want[0] and np.array_equal(got[1], want[1])
        assert gm.verify(toks[:20], 0)[-1] == want[0]
    finally:
        gm.free()


def test_verify_buffers_do_not_follow_the_prompt_tile():
    """A verification keeps the logits of at most 64 tokens, however large the tile of the prompt before it was."""
    from llamd_rs_b200 import backend, synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_vocab=32768)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=9), max_kv=2048, max_seq=1)
    try:
        toks = synth.token_ids(2048, hp["n_vocab"], 3, "verify memory").tolist()
        gm.set_option("head_gemm", 0)
        gm.set_option("dense_gemm", 0)  # (no folded copies of the projections in the figures below)
        gm.prefill(toks[:80], 0)
        want = list(gm.verify(toks[:80], 0))
        gm.prefill(toks, 0)  # one tile of 2048
        free = backend.free_memory()
        assert list(gm.verify(toks[:80], 0)) == want
        assert free - backend.free_memory() <= 64 * 4 * hp["n_vocab"] + (8 << 20)
    finally:
        gm.free()


def test_automatic_tile_counts_the_score_buffer():
    """A long context's score buffer is most of what a tile takes. With memory for a tile of 512 tokens but not of 2048, a
    prompt that never chose a tile runs, and gives what it gives with memory to spare."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_embd=512, n_head=16, n_head_kv=1, n_expert_used=8, n_ff_expert=1024)
    w = synth.make_model(hp, seed=9)
    toks = synth.token_ids(2000, hp["n_vocab"], 3, "score buffer").tolist()
    runs = []
    for tight in (False, True):
        gm = CudaModel.load_batched(hp, w, max_kv=40000, max_seq=1)
        # (scores 1.31 GB, the rest of a tile of 512 tokens 0.08 GB, of 2048 0.31 GB)
        full = _FullDevice(1540 << 20) if tight else None
        try:
            runs.append((gm.prefill(toks, 0), gm.logits()[0].view(np.uint32).copy()))
        finally:
            if full:
                full.release()
            gm.free()
    assert runs[0][0] == runs[1][0] and np.array_equal(runs[0][1], runs[1][1])


@pytest.mark.parametrize("tight", [False, True])
def test_folded_copies_leave_room_for_a_tile(tight):
    """A prompt makes the folded copies of the attention projections only where a full tile's buffers still fit beside them,
    and gives the same bits with and without them."""
    from llamd_rs_b200 import backend, synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=8, n_embd=512, n_head=16, n_head_kv=1)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=9), max_kv=40000, max_seq=1)
    try:
        toks = synth.token_ids(20, hp["n_vocab"], 3, "fold room").tolist()
        gm.set_option("dense_gemm", 0)
        want = gm.prefill(toks, 0), gm.logits()[0].view(np.uint32).copy()
        gm.set_option("dense_gemm", 8)
        full = _FullDevice(2 << 30) if tight else None  # (1 GB besides; a full tile's scores are 1.3 GB)
        try:
            free = backend.free_memory()
            got = gm.prefill(toks, 0), gm.logits()[0].view(np.uint32).copy()
            took = free - backend.free_memory()
        finally:
            if full:
                full.release()
        assert got[0] == want[0] and np.array_equal(got[1], want[1])
        assert took == 0 if tight else took > 0
    finally:
        gm.free()


@pytest.mark.parametrize("kv16", [0, 1])
def test_near_and_far_contexts(kv16):
    """The scores launch changes with the context (one sequence at 512 positions, two at 256), and each kind has its graph: the
    same tokens and logits as the per-head launches on both sides of the line, across it inside one decode call, and back."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_head=8, n_head_kv=1, head_dim=128)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=9), max_kv=640, max_seq=2)
    try:
        if kv16:
            gm.set_option("kv_f16", 1)
        toks = synth.token_ids(600, hp["n_vocab"], 3, "near").tolist()
        gm.prefill(toks, 0)
        runs = []
        for gqa, graph in ((0, True), (1, True), (1, False)):
            gm.set_option("attn_gqa", gqa)
            gm.use_graph = graph
            got = [gm.decode(toks[505], 505, 16)[0].tolist(), gm.logits()[0].view(np.uint32).tolist()]
            for pos in (3, 510, 511, 512, 513, 90, 599):
                got += [gm.forward(toks[pos], pos), gm.logits()[0].view(np.uint32).tolist()]
            for a, b in ((255, 10), (256, 10), (7, 254), (511, 512)):
                got += [gm.forward_batch([toks[a], toks[b]], [a, b]).tolist(), gm.logits(2).view(np.uint32).tolist()]
            gm.prefill(toks[500:530], 500)  # (the rows that the decode call wrote)
            runs.append(got)
        assert runs[0] == runs[1] == runs[2]
    finally:
        gm.use_graph = True
        gm.free()


@pytest.mark.parametrize("kv16", [0, 1])
def test_automatic_tiles_equal_sequential_decode(kv16):
    """prefill_tile never set: one tile up to 2048 tokens, two equal ones beyond, attention 512 tokens at a time. Tokens, logits and
    K/V rows are those of one token after the other, from position 0 and behind a context; and on the tile GEMMs alone for the
    lengths that otherwise run on the decode pass's launches."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = synth.TINY
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=7), max_kv=2112, max_seq=1)
    try:
        if kv16:
            gm.set_option("kv_f16", 1)
        toks = synth.token_ids(2049, hp["n_vocab"], 5, "automatic tile").tolist()
        ends, want = (37, 57, 193, 512, 513, 1025, 2048, 2049), {}
        for pos, t in enumerate(toks):
            tok = gm.forward(t, pos)
            if pos + 1 in ends:
                want[pos + 1] = tok, gm.logits()[0].view(np.uint32).copy()
        rows = [[x.view(np.uint32).copy() for x in gm.read_kv(il, len(toks))] for il in range(hp["n_layer"])]
        kvd = hp["n_head_kv"] * hp["head_dim"]
        for gemm_only in (False, True):
            gm.set_option("matvec_batch_max", 8 if gemm_only else 56)
            gm.set_option("dense_gemm", 0 if gemm_only else 8)
            for end in ends:
                for base in (0, 20):
                    gm.prefill(toks[:base] or toks[:1], 0)
                    tok = gm.prefill(toks[base:end], base)
                    what = f"{end - base} tokens from {base}, GEMMs only: {gemm_only}"
                    assert tok == want[end][0] and np.array_equal(gm.logits()[0].view(np.uint32), want[end][1]), what
                    for il in range(hp["n_layer"]):
                        for got, ref in zip(gm.read_kv(il, end), rows[il]):
                            assert np.array_equal(got.view(np.uint32), ref[:end * kvd]), what
    finally:
        gm.free()


def test_tile_gemms_equal_sequential_decode_at_wide_rows():
    """The benchmark's widths (8 blocks in, 16 out of attention, heads of 128, eight to a kv head, 8 experts of 16 used): the tile
    GEMMs without folded copies against one token after the other."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.QWEN3MOE_30B, n_layer=1, n_expert=16, n_vocab=1024)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=7), max_kv=320, max_seq=1)
    try:
        toks = synth.token_ids(300, hp["n_vocab"], 5, "wide rows").tolist()
        ends, want = (9, 40, 65, 300), {}
        for pos, t in enumerate(toks):
            tok = gm.forward(t, pos)
            if pos + 1 in ends:
                want[pos + 1] = tok, gm.logits()[0].view(np.uint32).copy()
        rows = [x.view(np.uint32).copy() for x in gm.read_kv(0, len(toks))]
        kvd = hp["n_head_kv"] * hp["head_dim"]
        for line, dense in ((8, 0), (56, 8)):
            gm.set_option("matvec_batch_max", line)
            gm.set_option("dense_gemm", dense)
            for end in ends:
                tok = gm.prefill(toks[:end], 0)
                what = f"{end} tokens, matvec launches up to {line}"
                assert tok == want[end][0] and np.array_equal(gm.logits()[0].view(np.uint32), want[end][1]), what
                assert all(np.array_equal(g.view(np.uint32), r[:end * kvd]) for g, r in zip(gm.read_kv(0, end), rows)), what
                if end <= 65:
                    assert gm.verify(toks[:end], 0)[-1] == tok, what
    finally:
        gm.free()
