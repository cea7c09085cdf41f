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
