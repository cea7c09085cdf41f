"""The integer GEMM's forms -- few tokens, token tiles by the team, folded rows shared by warps -- at the edges of their tiles,
against the oracle and against one token after the other. Everything is bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from llamd_rs_b200 import backend

    backend.stream_init()
    return backend


def _largest(w, n):
    """The first n blocks of w with the largest products: codes 0 or 63, scales -128 or 127."""
    b = w.reshape(-1, 210)
    rng = np.random.default_rng(n)
    b[:n, :192] = rng.integers(0, 2, (n, 192)) * 255
    b[:n, 192:208] = np.where(rng.integers(0, 2, (n, 16)), -128, 127).astype(np.int8).view(np.uint8)
    return w


# blocks per row: every split of a row's blocks over warps, whole tiles of 32 blocks and not; rows: part of a row tile, one row more
@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 5, 8, 9, 16, 17, 24])
@pytest.mark.parametrize("rows", [5, 33])
def test_dense_forms(be, blocks, rows):
    import oracle as orc
    from llamd_rs_b200 import ops, synth

    k, most = 256 * blocks, 65 if blocks > 9 else 130
    w = _largest(synth.q6k_blocks(rows * blocks, 91, "forms", blocks).copy(), rows * blocks // 3)
    dw = be.DeviceWeights.upload(w, rows, blocks)
    x = synth.normal_f32(most * k, 91, "forms.x", blocks).reshape(most, k)
    x[1] = np.where(x[1] < 0, -1, 1)  # quants of +-127 throughout
    want = np.stack([orc.matvec_q6k(w, x[t], k, rows) for t in range(most)]).view(np.uint32)
    for ntok in (1, 7, 8, 9, 16, 17, 24, 25, 33, 48, 49, 63, 64, 65, 130):
        if ntok <= most:
            (got,) = ops.matvec_tokens([dw], x[:ntok], gemm=True)
            assert np.array_equal(got.view(np.uint32), want[:ntok]), f"{ntok} tokens"
    for nseq in range(1, 9):
        assert np.array_equal(dw.matvec_f32(x[:nseq].ravel(), nseq).view(np.uint32).reshape(nseq, rows), want[:nseq]), f"{nseq} sequences"


# around the number of sequences from which such a matrix runs on the GEMM, with part of a row tile at the end
@pytest.mark.parametrize("rows,blocks,counts", [(2047, 12, (2, 3, 8)), (1030, 16, (3, 4)), (1030, 24, (5, 6))])
def test_products_of_several_sequences(be, rows, blocks, counts):
    import oracle as orc
    from llamd_rs_b200 import synth

    k, most = 256 * blocks, max(counts)
    w = synth.q6k_blocks(rows * blocks, 94, "products", blocks)
    dw = be.DeviceWeights.upload(w, rows, blocks)
    x = synth.normal_f32(most * k, 94, "products.x", blocks).reshape(most, k)
    want = np.stack([orc.matvec_q6k(w, x[t], k, rows) for t in range(most)]).view(np.uint32)
    for n in counts:
        assert np.array_equal(dw.matvec_f32(x[:n].ravel(), n).view(np.uint32).reshape(n, rows), want[:n]), f"{n} sequences"


@pytest.mark.parametrize("blocks", [2, 4, 5, 24, 25, 26])
def test_grouped_token_counts(be, blocks):
    """Groups of no token, one, a tile and its neighbours, two tiles of teams and one more."""
    from llamd_rs_b200 import ops, synth

    counts, rows, k = (0, 1, 7, 8, 9, 63, 64, 65, 129), 40, 256 * blocks
    ids = np.repeat(np.arange(len(counts), dtype=np.int32), counts).reshape(-1, 1)
    ids = np.ascontiguousarray(ids[np.random.default_rng(blocks).permutation(len(ids))])
    w = _largest(synth.q6k_blocks(len(counts) * rows * blocks, 92, "counts", blocks).copy(), rows * blocks)
    dw = be.DeviceWeights.upload(w, len(counts) * rows, blocks)
    x = synth.normal_f32(len(ids) * k, 92, "counts.x", blocks).reshape(len(ids), k)
    (want,) = ops.expert_major([dw], x, ids, rows)
    (got,) = ops.expert_major([dw], x, ids, rows, gemm=True)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("embd,ffe,n_expert,n_used", [(1280, 768, 64, 4), (512, 1536, 64, 4), (512, 768, 8, 2)])
def test_expert_forms_by_tokens_per_expert(embd, ffe, n_expert, n_used):
    """64 experts, 4 per token: tiles of 30 to 400 tokens are 2 to 25 tokens per expert, where the experts go from matvecs over
    the few-token forms to the teams; batches likewise. They change over at 36, 39 and 32 tokens. Tokens and logits are those of
    one token after the other."""
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_embd=embd, n_ff_expert=ffe, n_expert=n_expert, n_expert_used=n_used, n_vocab=512)
    gm = CudaModel.load_batched(hp, synth.make_model(hp, seed=5), max_kv=400, max_seq=64)
    try:
        toks = synth.token_ids(400, hp["n_vocab"], 5, "forms").tolist()
        want, logits = [], []
        for pos, t in enumerate(toks):
            want.append(gm.forward(t, pos))
            logits.append(gm.logits()[0].view(np.uint32).copy())
        for n in (26, 30, 31, 32, 33, 35, 36, 38, 39, 56, 100, 200, 400):
            assert gm.prefill(toks[:n], 0) == want[n - 1] and np.array_equal(gm.logits()[0].view(np.uint32), logits[n - 1]), f"prompt of {n}"
            assert list(gm.verify(toks[:n], 0)) == want[:n], f"draft of {n}"
        for n in (3, 4, 9, 30, 31, 32, 35, 36, 38, 39, 56, 64):  # one position of n sequences
            got = gm.forward_batch(toks[:n], [0] * n)
            rows = gm.logits(n).view(np.uint32)
            for s in range(n):
                assert got[s] == gm.forward(toks[s], 0) and np.array_equal(gm.logits()[0].view(np.uint32), rows[s]), f"sequence {s} of {n}"
    finally:
        gm.free()


# blocks per row around the rows one thread adds up by itself (3); rows around what one CTA of 256 (row, block) units covers
@pytest.mark.parametrize("blocks", [1, 2, 3, 4, 7, 24, 256])
def test_matvec_tails(be, blocks):
    """One activation: dense and grouped products, with quants of -128 and 127 and the largest weights, against the oracle."""
    import oracle as orc
    from llamd_rs_b200 import synth

    k, per_cta = 256 * blocks, 256 // blocks
    rng = np.random.default_rng(blocks)
    for rows in sorted({1, per_cta, per_cta + 1, 2 * per_cta - 1}):
        w = _largest(synth.q6k_blocks(2 * rows * blocks, 93, "tails", blocks, rows).copy(), rows * blocks // 2 + 1)
        qs, d = rng.integers(-128, 128, k).astype(np.int8), rng.random(blocks, dtype=np.float32)
        qs[:256] = np.where(qs[:256] < 0, -128, 127)
        want = orc.matvec_q6k_q8k(w, qs, d, k, 2 * rows).view(np.uint32)
        dw = be.DeviceWeights.upload(w, 2 * rows, blocks)
        assert np.array_equal(dw.matvec(qs, d).view(np.uint32), want)
        got = dw.matvec_grouped(qs, d, [1, 0, 1], rows).view(np.uint32)
        assert np.array_equal(got, want.reshape(2, rows)[[1, 0, 1]])
