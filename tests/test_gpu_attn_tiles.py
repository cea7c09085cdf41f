"""The register-tiled attention of prompts at the edges of its tiles: 64 tokens by 128 positions for the scores, four positions a
lane in the softmax, 16 tokens by stages of 16 positions for the values. The per-token kernels are the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd,n_head,n_head_kv", [(128, 4, 1), (64, 4, 2)])
@pytest.mark.parametrize("base,ntok", [(0, 1), (0, 15), (111, 17), (126, 3), (128, 64), (191, 65), (0, 129), (1000, 33)])
@pytest.mark.parametrize("scale", [1.0, 300.0])
def test_tile_edges(hd, n_head, n_head_kv, base, ntok, scale):
    """`scale` 300: logits thousands apart, so that most weights are 0 and some rows hold one weight of 1."""
    from llamd_rs_b200 import ops, synth

    n_rows, kv_dim = base + ntok, n_head_kv * hd
    max_kv = (n_rows + 3) & ~3
    q = (synth.normal_f32(ntok * n_head * hd, 7, "tiles.q", hd, base) * np.float32(scale)).reshape(ntok, -1)
    k = synth.normal_f32(n_rows * kv_dim, 7, "tiles.k", hd, base)
    v = synth.normal_f32(n_rows * kv_dim, 7, "tiles.v", hd, base)
    pos = np.random.default_rng(ntok).permutation(np.arange(base, n_rows, dtype=np.int32))
    got = ops.attention_prefill(q, k, v, pos, n_head, n_head_kv, hd, max_kv)
    want = ops.attention_prefill(q, k, v, pos, n_head, n_head_kv, hd, max_kv, tiled=False)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("kv_f16", [False, True])
def test_per_kv_head_forms_by_ctas(kv_f16):
    """Tiles and batches on either side of 518 value CTAs (32 and 33 tokens at four kv heads), contexts around 8 and 16
    positions and the value tile of 128: logits and tokens are those of one token after the other."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_embd=512, n_head=32, n_head_kv=4, head_dim=128, n_vocab=512)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=6), max_kv=200, max_seq=40)
    try:
        if kv_f16:
            gm.set_option("kv_f16", 1)
        toks = synth.token_ids(180, hp["n_vocab"], 6, "ctas").tolist()
        want, logits = [], []
        for pos, t in enumerate(toks):
            want.append(gm.forward(t, pos))
            logits.append(gm.logits()[0].view(np.uint32).copy())
        for base in (0, 100, 124):
            for n in (9, 16, 17, 32, 33, 56):
                assert list(gm.verify(toks[base : base + n], base)) == want[base : base + n], f"draft of {n} at {base}"
                assert gm.prefill(toks[base : base + n], base) == want[base + n - 1], f"turn of {n} at {base}"
                assert np.array_equal(gm.logits()[0].view(np.uint32), logits[base + n - 1]), f"turn of {n} at {base}"
        for n in (32, 33, 40):  # every sequence behind the same context
            for pos in range(20):
                got = gm.forward_batch([toks[pos]] * n, [pos] * n)
                rows = gm.logits(n).view(np.uint32)
                assert list(got) == [want[pos]] * n and all(np.array_equal(r, logits[pos]) for r in rows), f"{n} sequences at {pos}"
    finally:
        gm.free()


@pytest.mark.parametrize("kv_f16", [False, True])
def test_small_tiles_around_the_longest_rows(kv_f16):
    """Drafts and turns whose rows end around 4352 positions (nine tokens of four kv heads are the most that stay with the launches
    by kv head behind them), around 5376, and around the four-CTA form's last row of 768: as one token after the other."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_embd=512, n_head=32, n_head_kv=4, head_dim=128, n_vocab=512)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=8), max_kv=5440, max_seq=1)
    try:
        if kv_f16:
            gm.set_option("kv_f16", 1)
        toks = synth.token_ids(5440, hp["n_vocab"], 8, "rows").tolist()
        gm.prefill(toks, 0)
        for base, counts in ((728, (40, 41)), (4320, (9, 32, 33, 37)), (4343, (9, 10)), (5360, (9, 16, 17))):
            want, logits = [], []
            for pos in range(base, base + max(counts)):
                want.append(gm.forward(toks[pos], pos))
                logits.append(gm.logits()[0].view(np.uint32).copy())
            for n in counts:
                assert list(gm.verify(toks[base : base + n], base)) == want[:n], f"draft of {n} at {base}"
                assert gm.prefill(toks[base : base + n], base) == want[n - 1], f"turn of {n} at {base}"
                assert np.array_equal(gm.logits()[0].view(np.uint32), logits[n - 1]), f"turn of {n} at {base}"
    finally:
        gm.free()
