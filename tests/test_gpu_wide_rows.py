"""Rows around the widest that the integer GEMM takes, and around the widest that keep folded copies: models of one layer, tiles
and batches against one token after the other. Everything is bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(max_seq, **hp):
    from llamd_rs_b200 import synth
    from llamd_rs_b200.model import CudaModel

    hp = dict(synth.TINY, n_layer=1, n_head_kv=2, head_dim=128, n_expert=4, **hp)
    return CudaModel.load_batched(hp, synth.make_model(hp, seed=11), max_kv=200, max_seq=max_seq), hp


def _one_by_one(gm, toks):
    want, logits = [], []
    for pos, t in enumerate(toks):
        want.append(gm.forward(t, pos))
        logits.append(gm.logits()[0].view(np.uint32).copy())
    return want, logits


def _check_batch(gm, toks, n):
    got = gm.forward_batch(toks[:n], [0] * n)
    rows = gm.logits(n).view(np.uint32)
    for s in range(n):
        assert got[s] == gm.forward(toks[s], 0) and np.array_equal(gm.logits()[0].view(np.uint32), rows[s]), f"sequence {s} of {n}"


# 24 blocks: images that leave room for the rings of four token tiles only; 50 heads: an output projection of 25, the widest
@pytest.mark.parametrize("blocks,n_head", [(24, 48), (23, 46), (2, 50)])
def test_folded_rows(blocks, n_head):
    """Tiles of up to 192 tokens and batches multiply with folded copies of the projections: up to four token tiles, and more."""
    from llamd_rs_b200 import synth

    gm, hp = _model(33, n_embd=256 * blocks, n_head=n_head)
    try:
        toks = synth.token_ids(192, hp["n_vocab"], 11, "wide").tolist()
        want, logits = _one_by_one(gm, toks)
        for n in (32, 33, 56, 64, 192):
            assert gm.prefill(toks[:n], 0) == want[n - 1] and np.array_equal(gm.logits()[0].view(np.uint32), logits[n - 1]), f"prompt of {n}"
        _check_batch(gm, toks, 33)
    finally:
        gm.free()


# gate and up, and down, of 1 to 5 blocks a row (images are taken from 24 or 48 tokens per expert on), and wider (they are not)
@pytest.mark.parametrize("blocks,down_blocks", [(1, 2), (3, 4), (5, 5), (6, 3), (24, 1)])
def test_prefolded_experts(blocks, down_blocks):
    """prefill_prefold: 2 to 96 tokens per expert."""
    from llamd_rs_b200 import synth

    gm, hp = _model(1, n_embd=256 * blocks, n_head=2, n_ff_expert=256 * down_blocks)
    try:
        gm.set_option("prefill_prefold", 1)
        toks = synth.token_ids(192, hp["n_vocab"], 11, "wide").tolist()
        want, logits = _one_by_one(gm, toks)
        for n in (4, 32, 48, 50, 64, 65, 98, 130, 192):
            assert gm.prefill(toks[:n], 0) == want[n - 1] and np.array_equal(gm.logits()[0].view(np.uint32), logits[n - 1]), f"prompt of {n}"
    finally:
        gm.free()


@pytest.mark.parametrize("which", ["T_FFN_GATE_EXPS", "T_FFN_UP_EXPS", "T_FFN_DOWN_EXPS"])
def test_prefolded_experts_follow_their_tensor(which):
    """An expert tensor set after a prompt with prefill_prefold: the next prompt multiplies with the new bytes."""
    from llamd_rs_b200 import model, synth

    gm, hp = _model(1, n_embd=512, n_head=4, n_ff_expert=512)
    try:
        gm.set_option("prefill_prefold", 1)
        toks = synth.token_ids(130, hp["n_vocab"], 11, "wide").tolist()
        before = gm.prefill(toks, 0), gm.logits()[0].view(np.uint32).copy()
        gm.set_tensor(0, getattr(model, which), synth.q6k_blocks(hp["n_expert"] * 512 * 512 // 256, 12, "other"))
        want, logits = _one_by_one(gm, toks)
        assert not np.array_equal(before[1], logits[-1])
        assert gm.prefill(toks, 0) == want[-1] and np.array_equal(gm.logits()[0].view(np.uint32), logits[-1])
    finally:
        gm.free()


@pytest.mark.parametrize("n_head", [52, 64])
def test_projections_wider_than_the_gemm_takes(n_head):
    """An output projection of 26 and 32 blocks a row: batches, drafts and short prompts run on the matvecs, from the first pass on."""
    from llamd_rs_b200 import synth

    for first in ("batch", "prompt"):
        gm, hp = _model(9, n_embd=512, n_head=n_head)
        try:
            toks = synth.token_ids(9, hp["n_vocab"], 11, "wide").tolist()
            if first == "batch":
                for n in (8, 4, 9):
                    _check_batch(gm, toks, n)
            want, logits = _one_by_one(gm, toks)  # (a batch writes position 0 of sequence 0)
            for n in (9, 4):
                assert gm.prefill(toks[:n], 0) == want[n - 1] and np.array_equal(gm.logits()[0].view(np.uint32), logits[n - 1]), f"prompt of {n}"
                assert list(gm.verify(toks[:n], 0)) == want[:n], f"draft of {n}"
        finally:
            gm.free()


def test_narrower_rows_after_a_refused_form():
    """Folded rows of 24 blocks and more than 32 tokens, whether or not a form takes them, leave those of 23 as they were."""
    from llamd_rs_b200 import backend, synth
    from llamd_rs_b200._lib import lib

    for blocks in (24, 23):
        gm, hp = _model(1, n_embd=256 * blocks, n_head=2 * blocks)
        try:
            toks = synth.token_ids(33, hp["n_vocab"], 11, "wide").tolist()
            want, logits = _one_by_one(gm, toks)
            try:
                got = gm.prefill(toks, 0)
            except backend.Other:
                assert blocks == 24
                lib().llamd_fwd_last_error()
                continue
            assert got == want[-1] and np.array_equal(gm.logits()[0].view(np.uint32), logits[-1])
        finally:
            gm.free()
