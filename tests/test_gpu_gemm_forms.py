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


COUNTS = (0, 1, 7, 8, 9, 63, 64, 65, 129)


def _groups(be, blocks, rows, matrices):
    """One expert per entry of COUNTS, its pairs scattered over the tokens, and what expert_major makes of them."""
    from llamd_rs_b200 import ops, synth

    k = 256 * blocks
    ids = np.repeat(np.arange(len(COUNTS), dtype=np.int32), COUNTS).reshape(-1, 1)
    ids = np.ascontiguousarray(ids[np.random.default_rng(blocks).permutation(len(ids))])
    ws = [be.DeviceWeights.upload(_largest(synth.q6k_blocks(len(COUNTS) * rows * blocks, 92 + i, "counts", blocks).copy(), rows * blocks),
                                  len(COUNTS) * rows, blocks) for i in range(matrices)]
    x = synth.normal_f32(len(ids) * k, 92, "counts.x", blocks).reshape(len(ids), k)
    return ids, ws, x, ops.expert_major(ws, x, ids, rows)


@pytest.mark.parametrize("blocks", [2, 4, 5, 24, 25, 26])
def test_grouped_token_counts(be, blocks):
    """Groups of no token, one, a tile and its neighbours, two tiles of teams and one more, in the form that the entry point takes
    for 64 tokens per group."""
    from llamd_rs_b200 import ops

    ids, ws, x, want = _groups(be, blocks, 40, 1)
    got = ops.expert_major(ws, x, ids, 40, gemm=True)
    assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))


# rows: experts that begin with a tile of 32 blocks, and (part of a row tile at the end) that do not
@pytest.mark.parametrize("blocks", [1, 3, 4, 5, 8, 24])
@pytest.mark.parametrize("rows", [64, 33])
def test_grouped_forms_meet_any_count(be, blocks, rows):
    """The form follows the mean of the groups; each is given groups of none to 129 tokens, two matrices at a time."""
    import ctypes as C
    from llamd_rs_b200._lib import lib
    from llamd_rs_b200.backend import DevBuf

    vp = C.c_void_p
    scatter = lib()._ZN5llamd19expert_gemm_scatterEPKvS1_PKiS3_S3_S3_S1_PKfPfS6_iiiiPKS6_iS1_S1_  # (as the model's passes call it)
    scatter.restype, scatter.argtypes = None, [vp] * 10 + [C.c_int] * 4 + [vp, C.c_int, vp, vp]
    ids, ws, x, want = _groups(be, blocks, rows, 2)
    n, ne = len(ids), len(COUNTS)
    dx, dq, dd, di = DevBuf.from_array(x), DevBuf(x.size), DevBuf(n * blocks * 4), DevBuf.from_array(ids)
    lib().llamd_fwd_quantize(dx.ptr, dq.ptr, dd.ptr, n * blocks)
    drm = DevBuf(x.size)
    lib().llamd_fwd_q8k_residue_major(dq.ptr, drm.ptr, n * blocks)
    gs, gc, pt, ps = DevBuf(ne * 4), DevBuf(ne * 4), DevBuf(n * 4), DevBuf(n * 4)
    work, n_work = DevBuf((n // 8 + ne + 1) * 12), DevBuf.zeroed(4)
    lib().llamd_fwd_moe_group_work(di.ptr, ne, 1, n, gs.ptr, gc.ptr, pt.ptr, ps.ptr, work.ptr, n_work.ptr)
    for per_group in (1, 9, 17, 25, 41, 129):
        outs = [DevBuf.zeroed(n * rows * 4) for _ in ws]
        scatter(ws[0].ptr, ws[1].ptr, gs.ptr, gc.ptr, pt.ptr, ps.ptr, drm.ptr, dd.ptr, outs[0].ptr, outs[1].ptr, blocks, rows, ne,
                per_group * ne, None, 1, None, None)
        be.sync()
        for o, w in zip(outs, want):
            assert np.array_equal(o.download_f32(n * rows).view(np.uint32), w.view(np.uint32).ravel()), f"{per_group} tokens per group"


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
