"""GPU parity of the f32 ops around the matvecs (router, norms, RoPE,
attention, SiLU, combine, argmax, scatter plan) against the oracle.

Everything without an exponential is bit-exact. Where exp() is involved the
device rounds a double-precision exponential once while the oracle calls the
host libm; the two differ by one ulp on a small fraction of inputs, so those
outputs are compared at tolerance::ATTENTION (1e-5, crates/llamd-core/src/tolerance.rs:97)
and the discrete results (expert ids) must still match on these inputs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ATTENTION = 1e-5
F32_ULP = 1.2e-7


@pytest.fixture(scope="module")
def ops():
    from llamd_rs_b200 import backend, ops

    if not backend.available():
        pytest.fail("no CUDA device: the GPU tests must run on a GPU box")
    backend.stream_init()
    return ops


@pytest.fixture(scope="module")
def synth():
    from llamd_rs_b200 import synth

    return synth


def bit_equal(a, b):
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return a.shape == b.shape and np.array_equal(a.view(np.uint32), b.view(np.uint32))


def max_dev(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.max(np.abs(a - b) / np.maximum(np.maximum(np.abs(a), np.abs(b)), 1.0)))


@pytest.mark.parametrize("n", [768, 772, 1024, 2048, 4096, 4100, 6144])
@pytest.mark.parametrize("kind", ["normal", "ties", "mixed", "tiny", "huge"])
def test_sum_of_squares_in_runs_is_the_chain(ops, orc, n, kind):
    """The CTA-wide ordered sum against the oracle's chain: from the longest sum that is walked as it is to several passes of
    the scratch, with terms that tie, vanish against the sum, stay subnormal, or overflow."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal((16, n))
    if kind == "ties":
        x = np.exp2(-rng.integers(0, 14, (16, n))) * rng.integers(1, 4, (16, n))
    elif kind == "mixed":
        x = x * np.exp2(rng.integers(-20, 20, (16, n))) * (rng.random((16, n)) < 0.7)
    elif kind == "tiny":
        x = x * 2.0 ** -70
    elif kind == "huge":
        x = x * 2.0 ** 62
    x = x.astype(np.float32)
    with np.errstate(all="ignore"):
        want = orc.rms_norm(x, 1e-6)
    assert bit_equal(ops.rms_norm_mul(x, np.ones(n, np.float32), 1e-6), want)


def test_rms_norm_is_bit_exact(ops, orc, synth):
    x = synth.normal_f32(3 * 2048, 1, "rms").reshape(3, 2048)
    w = synth.normal_f32(2048, 1, "rms.w")
    want = orc.mul(orc.rms_norm(x, 1e-6), np.tile(w, 3)).reshape(3, 2048)
    assert bit_equal(ops.rms_norm_mul(x, w, 1e-6), want)
    out, qs, d = ops.rms_norm_quant(x, w, 1e-6)
    assert bit_equal(out, want)
    hq, hd, _ = orc.quantize_q8k(want)
    assert np.array_equal(qs, hq) and bit_equal(d, hd)
    r = synth.normal_f32(3 * 2048, 1, "rms.r").reshape(3, 2048)
    out, qs, d, s = ops.rms_norm_quant(x, w, 1e-6, residual=r)
    assert bit_equal(s, orc.add(x, r).reshape(3, 2048))
    assert bit_equal(out, orc.mul(orc.rms_norm(s, 1e-6), np.tile(w, 3)).reshape(3, 2048))
    # crates/llamd-cpu/src/lib.rs:237-244
    got = ops.rms_norm_mul(np.array([3.0, 4.0, 0.0, 0.0], np.float32), np.ones(4, np.float32), 0.0)
    assert bit_equal(got, orc.rms_norm(np.array([3.0, 4.0, 0.0, 0.0], np.float32), 0.0))


def test_head_norm_and_rope_are_bit_exact(ops, orc, synth):
    n_head, hd = 8, 128
    x = synth.normal_f32(n_head * hd, 2, "rope")
    w = synth.normal_f32(hd, 2, "rope.w")
    normed = orc.rms_norm(x.reshape(n_head, hd), 1e-6) * 0 + orc.mul(orc.rms_norm(x.reshape(n_head, hd), 1e-6).ravel(), np.tile(w, n_head)).reshape(n_head, hd)
    assert bit_equal(ops.head_rms_norm_mul(x, w, n_head, hd, 1e-6), normed.ravel())
    for pos in (0, 1, 37, 700):
        want = orc.rope(normed.reshape(1, -1), [pos], hd, 1e7)[0]
        assert bit_equal(ops.norm_rope(x, w, n_head, hd, pos, 1e7, 1e-6), want), f"pos {pos}"
        assert bit_equal(ops.norm_rope(x, None, n_head, hd, pos, 1e7, 1e-6), orc.rope(x.reshape(1, -1), [pos], hd, 1e7)[0])
    # crates/llamd-cpu/src/lib.rs:314-322: position 0 is the identity
    assert bit_equal(ops.norm_rope(x, None, n_head, hd, 0, 1e4, 0.0), x)
    tab = ops.rope_table(5, 8, 1e7)
    s, c = orc.rope_angles(3, 8, 1e7)
    assert bit_equal(tab[3, :, 0], s) and bit_equal(tab[3, :, 1], c)


@pytest.mark.parametrize("n_kv", [1, 7, 64, 65, 200, 513])
def test_attention_matches(ops, orc, synth, n_kv):
    n_head, n_head_kv, hd = 32, 4, 128
    q = synth.normal_f32(n_head * hd, 3, "att.q", n_kv)
    k = synth.normal_f32(n_kv * n_head_kv * hd, 3, "att.k", n_kv)
    v = synth.normal_f32(n_kv * n_head_kv * hd, 3, "att.v", n_kv)
    want = orc.attend(q, k, v, n_kv, n_head, n_head_kv, hd)
    got = ops.attention(q, k, v, n_kv, n_head, n_head_kv, hd)
    if n_kv == 1:
        assert bit_equal(got, want), "a single key gives exactly its value"
    assert max_dev(got, want) <= ATTENTION
    split = ops.attention(q, k, v, n_kv, n_head, n_head_kv, hd, scores=True)
    assert bit_equal(split, got), "the split-over-CTAs variant keeps every sum in order"


@pytest.mark.parametrize("n_head,n_head_kv,hd,base,ntok,max_kv", [
    (8, 2, 128, 0, 70, 128),      # ragged token and position tiles, first tile of a prompt
    (4, 2, 64, 37, 33, 96),       # a later tile: 37 positions of context before it
    (4, 1, 128, 100, 1, 104),     # a single token with context
    (4, 4, 64, 0, 96, 100),       # no grouping
    (4, 2, 96, 0, 9, 16),         # a head_dim the tiled kernels do not cover: falls through
    (4, 2, 64, 0, 9, 18),         # max_kv not a multiple of 4: falls through
])
def test_attention_prefill_tile(ops, orc, synth, n_head, n_head_kv, hd, base, ntok, max_kv):
    """The register-tiled prefill attention equals the per-token kernels bit for bit and `attend` per token."""
    n_rows = base + ntok
    kv_dim = n_head_kv * hd
    q = synth.normal_f32(ntok * n_head * hd, 5, "attp.q", hd, ntok).reshape(ntok, -1)
    k = synth.normal_f32(n_rows * kv_dim, 5, "attp.k", hd, ntok)
    v = synth.normal_f32(n_rows * kv_dim, 5, "attp.v", hd, ntok)
    pos = np.arange(base, base + ntok, dtype=np.int32)
    got = ops.attention_prefill(q, k, v, pos, n_head, n_head_kv, hd, max_kv)
    per_token = ops.attention_prefill(q, k, v, pos, n_head, n_head_kv, hd, max_kv, tiled=False)
    assert bit_equal(got, per_token)
    for i in (0, ntok // 2, ntok - 1):
        n_kv = int(pos[i]) + 1
        want = orc.attend(q[i], k[: n_kv * kv_dim], v[: n_kv * kv_dim], n_kv, n_head, n_head_kv, hd)
        assert max_dev(got[i], want) <= ATTENTION
    # positions need not be consecutive or increasing
    perm = np.random.default_rng(1).permutation(ntok)
    got2 = ops.attention_prefill(q[perm], k, v, pos[perm], n_head, n_head_kv, hd, max_kv)
    assert bit_equal(got2, got[perm])


def test_attention_reference_kats(ops, orc):
    """crates/llamd-runtime/src/attention.rs:140-213"""
    out = ops.attention([0.5] * 4, [0.25] * 4, [7, 8, 9, 10], 1, 1, 1, 4)
    assert out.tolist() == [7.0, 8.0, 9.0, 10.0]
    out = ops.attention([1, 0, 0, 0] * 4, [1, 0, 0, 0, 1, 0, 0, 0], [100] * 4 + [200] * 4, 1, 4, 2, 4)
    assert out[0] == 100 and out[4] == 100 and out[8] == 200 and out[12] == 200, "GQA maps by integer division"
    out = ops.attention([2, 0, 0, 0], [2, 0, 0, 0, 0, 2, 0, 0], [1, 0, 0, 0, 0, 0, 0, 0], 2, 1, 1, 4)
    assert abs(out[0] - np.exp(2.0) / (np.exp(2.0) + 1.0)) < ATTENTION
    out = ops.attention([100.0] * 4, [100.0] * 4 + [-100.0] * 4, [1.0] * 4 + [2.0] * 4, 2, 1, 1, 4)
    assert np.all(np.isfinite(out)) and abs(out[0] - 1.0) < ATTENTION
    from llamd_rs_b200 import backend

    with pytest.raises(backend.Malformed):
        ops.attention([0.0] * 4, [0.0] * 4, [0.0] * 4, 1, 3, 2, 2)  # 3 does not group into 2
    with pytest.raises(backend.ShapeError):
        ops.attention([0.0] * 3, [0.0] * 4, [0.0] * 4, 1, 1, 1, 4)
    with pytest.raises(backend.Malformed):
        ops.attention([0.0] * 4, [], [], 0, 1, 1, 4)
    with pytest.raises(backend.Malformed):
        ops.attention([0.0] * 6, [0.0] * 4, [0.0] * 4, 1, 3, 2, 2)


def test_router_matches_route(ops, orc, synth):
    logits = synth.normal_f32(5 * 128, 4, "router").reshape(5, 128) * np.float32(2.0)
    ids, w, probs = ops.router(logits, 8)
    for s in range(5):
        r = orc.route(logits[s], 8)
        assert ids[s].tolist() == r["experts"].tolist(), f"sequence {s}"
        assert max_dev(w[s], r["weights"]) <= ATTENTION and max_dev(probs[s], r["probs"]) <= ATTENTION


def test_router_reference_kats(ops, orc):
    """crates/llamd-models/src/moe.rs:120-246"""
    from llamd_rs_b200 import backend

    assert ops.router([0.1, 5.0, 0.2, 3.0, 0.3], 2)[0][0].tolist() == [1, 3]
    ids, w, _ = ops.router([10.0, 9.0, 0.0, 0.0], 2)
    assert abs(w[0][0] - 0.7310586) < ATTENTION and abs(w[0][1] - 0.2689414) < ATTENTION
    for _ in range(4):
        assert ops.router([1.0, 1.0, 1.0, 1.0], 2)[0][0].tolist() == [0, 1], "ties break toward the lower index"
    ids, w, _ = ops.router([0.0, -800.0, -800.0, -800.0], 3)
    assert np.all(np.isfinite(w)) and ids[0][0] == 0
    assert ids[0].tolist() == [0, 1, 2], "equal (zero) probabilities are taken in index order"
    logits = (np.sin(np.arange(128, dtype=np.float32) * np.float32(0.37)) * np.float32(3.0)).astype(np.float32)
    ids, w, _ = ops.router(logits, 8)
    assert ids[0].tolist() == orc.route(logits, 8)["experts"].tolist() and len(set(ids[0].tolist())) == 8
    for bad in (0, 3):
        with pytest.raises(backend.Malformed):
            ops.router([1.0, 2.0], bad)


def test_router_matvec_logits_are_bit_exact(ops, orc, synth):
    ne, k = 128, 2048
    w = synth.normal_f32(ne * k, 5, "rw", std=0.02).reshape(ne, k)
    x = synth.normal_f32(3 * k, 5, "rx").reshape(3, k)
    logits, ids, wts = ops.router_matvec(w, x, 8)
    for s in range(3):
        want = orc.matvec_dequant(orc.F32, w, x[s], k, ne)
        assert bit_equal(logits[s], want), "router logits: sequential f32 dot"
        r = orc.route(want, 8)
        assert ids[s].tolist() == r["experts"].tolist()
        assert max_dev(wts[s], r["weights"]) <= ATTENTION
    assert bit_equal(ops.matvec_f32(w, x), np.stack([orc.matvec_dequant(orc.F32, w, x[s], k, ne) for s in range(3)]))


@pytest.mark.parametrize("hd,heads,kv_heads,n,shift,kv16,own_caches,norms", [
    (128, 7, 1, 513, 0, 0, False, "qk"),   # 4104 vectors: the last CTA holds 8
    (64, 6, 2, 512, 0, 1, False, "qk"),    # 4096, binary16 cache
    (256, 12, 4, 513, 0, 0, True, "q"),    # 8208, a cache per sequence, keys not normed
    (20, 30, 10, 131, 0, 1, True, ""),     # 5240, no norm weights
    (128, 7, 1, 513, 4, 0, False, "qk"),   # queries and keys off the 16-byte boundary
    (128, 7, 1, 511, 0, 0, False, "k"),    # 4088: a CTA per head
])
def test_norm_rope_of_many_vectors(ops, orc, synth, hd, heads, kv_heads, n, shift, kv16, own_caches, norms):
    """QK-norm, RoPE and the K/V store of a tile on both sides of the line where a CTA takes 32 vectors: queries, keys and cache
    rows against the oracle, the other cache rows untouched."""
    from llamd_rs_b200.backend import DevBuf, sync
    from llamd_rs_b200._lib import lib

    q, k, v = (synth.normal_f32(n * h * hd, 91, "many", what).reshape(n, h * hd) for what, h in (("q", heads), ("k", kv_heads), ("v", kv_heads)))
    w = {c: synth.normal_f32(hd, 91, "many.w", c) if c in norms else None for c in "qk"}
    max_kv, first = (160 if own_caches else 520), 3
    pos = np.array([(7 * i) % max_kv if own_caches else first + i for i in range(n)], np.int32)
    rows = np.arange(n) * max_kv + pos if own_caches else pos  # of a cache
    want = {}
    for c, x, h in (("q", q, heads), ("k", k, kv_heads)):
        if w[c] is not None:
            x = orc.mul(orc.rms_norm(x.reshape(-1, hd), 1e-6).ravel(), np.tile(w[c], n * h))
        want[c] = np.asarray(orc.rope(np.asarray(x, np.float32).reshape(n, h * hd), pos.tolist(), hd, 1e7)).reshape(n, h * hd)

    def moved(x):  # `shift` bytes into a buffer
        b = DevBuf.from_array(np.concatenate([np.zeros(shift // 4, np.float32), x.ravel()]))
        return b, b.ptr + shift

    (bq, pq), (bk, pk) = moved(q), moved(k)
    dv, tab = DevBuf.from_array(v), DevBuf.from_array(ops.rope_table(max_kv, hd, 1e7))
    dw = {c: DevBuf.from_array(x) if x is not None else None for c, x in w.items()}
    meta = DevBuf.from_array(np.stack([np.zeros(n, np.int32), pos], 1))
    n_rows = (n if own_caches else 1) * max_kv
    elem = np.float16 if kv16 else np.float32
    cache = [DevBuf.zeroed(n_rows * kv_heads * hd * np.dtype(elem).itemsize) for _ in range(2)]
    args = [pq, dw["q"].ptr if dw["q"] else None, pk, dw["k"].ptr if dw["k"] else None, dv.ptr, cache[0].ptr, cache[1].ptr, heads, kv_heads, hd,
            meta.ptr, tab.ptr, 1e-6, n] + ([max_kv] if own_caches else [])
    getattr(lib(), "llamd_fwd_qk_norm_rope_store" + ("" if own_caches else "_tile") + ("_kv16" if kv16 else ""))(*args)
    sync()
    assert bit_equal(bq.download_f32(shift // 4 + q.size)[shift // 4:].reshape(q.shape), want["q"])
    assert bit_equal(bk.download_f32(shift // 4 + k.size)[shift // 4:].reshape(k.shape), want["k"])
    for buf, x in ((cache[0], want["k"]), (cache[1], v)):
        full = np.zeros((n_rows, kv_heads * hd), elem)
        full[rows] = x.astype(elem)
        got = buf.download_f32(buf.nbytes // 4).view(elem).reshape(full.shape)
        assert np.array_equal(got.view(np.uint8), full.view(np.uint8))


@pytest.mark.parametrize("rows,k,ntok", [(128, 2048, 37), (8, 256, 1), (50, 100, 19), (33, 68, 16), (33, 772, 129), (128, 640, 593),
                                         (33, 260, 592), (33, 260, 593), (65, 324, 1180), (65, 324, 1601)])
def test_matmul_f32_tokens(ops, orc, synth, rows, k, ntok):
    """The tile form of the f32 matvec: every output is the same -0.0-seeded left-to-right sum."""
    w = synth.normal_f32(rows * k, 5, "mm.w", rows, k, std=0.02).reshape(rows, k)
    x = synth.normal_f32(ntok * k, 5, "mm.x", rows, k).reshape(ntok, k)
    got = ops.matmul_f32_tokens(w, x)
    want = np.stack([orc.matvec_dequant(orc.F32, w, x[t], k, rows) for t in range(ntok)])
    assert bit_equal(got, want)
    z = ops.matmul_f32_tokens(-np.abs(w), np.zeros_like(x))
    assert np.all(np.signbit(z)), "an all -0.0 sum keeps its sign: no padding term enters a chain"


@pytest.mark.parametrize("ntok", [5, 300])
def test_matmul_f32_tokens_of_a_launch_in_front(ops, synth, ntok):
    """The matrix may be what the launch in front on the stream writes: the same bits as with a wait between the two."""
    from llamd_rs_b200.backend import DevBuf, sync
    from llamd_rs_b200._lib import lib

    k0, k, rows = 4096, 512, 96
    w0, x0 = (DevBuf.from_array(synth.normal_f32(n * k0, 92, "front", n, std=0.02)) for n in (k, rows))
    x, w, out = DevBuf.from_array(synth.normal_f32(ntok * k, 92, "front.x")), DevBuf(rows * k * 4), DevBuf(ntok * rows * 4)
    got = []
    for wait in (True, False, False, False):
        lib().llamd_fwd_memset(w.ptr, 0, w.nbytes)
        sync()
        lib().llamd_fwd_matmul_f32_tokens(w0.ptr, x0.ptr, w.ptr, k0, k, rows)  # w [rows][k]
        if wait:
            sync()
        lib().llamd_fwd_matmul_f32_tokens(w.ptr, x.ptr, out.ptr, k, rows, ntok)
        sync()
        got.append(out.download_f32(ntok * rows))
    assert np.any(got[0] != 0) and all(bit_equal(got[0], g) for g in got[1:])


def test_silu_mul_and_quant(ops, orc, synth):
    g = synth.normal_f32(8 * 768, 6, "g") * np.float32(3.0)
    u = synth.normal_f32(8 * 768, 6, "u")
    want = orc.mul(orc.silu(g), u)
    got = ops.silu_mul(g, u)
    assert max_dev(got, want) <= ATTENTION
    ulp = np.abs(got.view(np.int32).astype(np.int64) - want.view(np.int32).astype(np.int64))
    assert ulp.max() <= 2 and np.mean(ulp > 0) < 0.01, "exp differs from the host libm by at most an ulp, rarely"
    out, qs, d = ops.silu_mul_quant(g, u)
    assert bit_equal(out, got)
    hq, hd, _ = orc.quantize_q8k(got)  # the quantizer itself is exact on the device's own activations
    assert np.array_equal(qs, hq) and bit_equal(d, hd)
    # crates/llamd-cpu/src/lib.rs:282-290
    s = ops.silu_mul([0.0, 1.0, -1.0], [1.0, 1.0, 1.0])
    assert s[0] == 0.0 and abs(s[1] - 1.0 / (1.0 + np.exp(-1.0))) < F32_ULP * 2 and -1.0 < s[2] < 0.0


def test_moe_combine_is_bit_exact(ops, orc, synth):
    nseq, nu, E = 2, 8, 2048
    down = synth.normal_f32(nseq * nu * E, 7, "down").reshape(nseq, nu, E)
    w = np.abs(synth.normal_f32(nseq * nu, 7, "cw")).reshape(nseq, nu)
    res = synth.normal_f32(nseq * E, 7, "res").reshape(nseq, E)
    want = np.zeros((nseq, E), np.float32)
    for s in range(nseq):
        acc = np.zeros(E, np.float32)
        for e in range(nu):
            acc = (acc + (w[s, e] * down[s, e]).astype(np.float32)).astype(np.float32)
        want[s] = res[s] + acc
    assert bit_equal(ops.moe_combine_add(down, w, res), want)


def test_argmax_lowest_index_on_ties(ops, orc, synth):
    x = synth.normal_f32(2 * 151936, 8, "amax").reshape(2, 151936)
    x[0, 777] = x[0, 150000] = 9.0
    x[1, 151935] = 12.0
    assert ops.argmax(x).tolist() == [777, 151935]
    assert ops.argmax(np.zeros(1000, np.float32)).tolist() == [0]
    assert ops.argmax(x[0])[0] == orc.argmax(x[0])


def test_moe_group_is_a_stable_counting_sort(ops, synth):
    n_expert, n_used, nseq = 128, 8, 37
    rng = np.random.default_rng(9)
    ids = np.stack([rng.permutation(n_expert)[:n_used] for _ in range(nseq)]).astype(np.int32)
    g = ops.moe_group(ids, n_expert, n_used)
    flat = ids.ravel()
    assert g["gcount"].tolist() == np.bincount(flat, minlength=n_expert).tolist()
    assert g["gstart"].tolist() == (np.cumsum(g["gcount"]) - g["gcount"]).tolist()
    order = np.argsort(flat, kind="stable")
    assert g["pslot"].tolist() == order.tolist(), "pairs of an expert in ascending pair order"
    assert g["ptoken"].tolist() == (order // n_used).tolist()
    covered = []
    for e, first, cnt in g["work"].tolist():
        assert 1 <= cnt <= 8 and g["gstart"][e] <= first and first + cnt <= g["gstart"][e] + g["gcount"][e]
        covered.extend(range(first, first + cnt))
    assert covered == list(range(flat.size)), "the work list covers every pair once"
    empty = ops.moe_group(np.zeros((0, n_used), np.int32), n_expert, n_used)
    assert not empty["gcount"].any() and empty["work"].shape[0] == 0


@pytest.mark.parametrize("n_expert,n_used,nseq,hot", [
    (128, 8, 512, None),    # a full prefill tile
    (128, 8, 5120, None),   # the largest tile one launch takes: 40960 pairs
    (1024, 2, 33, None),    # the most experts, most of them empty
    (8, 1, 1, None),        # a single pair
    (16, 4, 300, 5),        # every token also picks expert 5: one group far longer than a warp's chunk
])
def test_moe_group_edges(ops, n_expert, n_used, nseq, hot):
    rng = np.random.default_rng(n_expert + nseq)
    ids = np.stack([rng.permutation(n_expert)[:n_used] for _ in range(nseq)]).astype(np.int32)
    if hot is not None:
        ids[:, 0] = hot
    g = ops.moe_group(ids, n_expert, n_used)
    flat = ids.ravel()
    order = np.argsort(flat, kind="stable")
    assert g["gcount"].tolist() == np.bincount(flat, minlength=n_expert).tolist()
    assert g["gstart"].tolist() == (np.cumsum(g["gcount"]) - g["gcount"]).tolist()
    assert np.array_equal(g["pslot"], order) and np.array_equal(g["ptoken"], order // n_used)
    work = g["work"]
    assert work.shape[0] == int(np.sum((g["gcount"] + 7) // 8))
    assert int(work[:, 2].sum()) == flat.size and work[:, 2].min() >= 1 and work[:, 2].max() <= 8


def test_embed_is_a_dequantized_row(ops, orc, synth):
    from llamd_rs_b200 import backend

    rows, blocks = 50, 3
    w = synth.q6k_blocks(rows * blocks, 10, "embd")
    t = backend.DeviceWeights.upload(w, rows, blocks)
    full = orc.dequantize(orc.Q6K, w, rows * blocks * 256).reshape(rows, blocks * 256)
    for tok in (0, 17, 49):
        assert bit_equal(ops.embed(t, tok), full[tok])
    with pytest.raises(backend.Malformed):
        ops.embed(t, 50)


@pytest.mark.parametrize("nseq", [1, 3])
def test_gate_up_with_the_silu_quant_tail(ops, orc, synth, nseq):
    """The slot's last CTA produces silu(gate)*up and its Q8_K form: same bits as the two separate launches."""
    from llamd_rs_b200 import backend

    n_expert, rows, k, n_used = 10, 512, 512, 4
    wa = synth.q6k_blocks(n_expert * rows * k // 256, 94, "tail.a")
    wb = synth.q6k_blocks(n_expert * rows * k // 256, 94, "tail.b")
    da = backend.DeviceWeights.upload(wa, n_expert * rows, k // 256)
    db = backend.DeviceWeights.upload(wb, n_expert * rows, k // 256)
    rng = np.random.default_rng(nseq)
    ids = np.stack([rng.permutation(n_expert)[:n_used] for _ in range(nseq)]).astype(np.int32)
    x = synth.normal_f32(nseq * k, 94, "tail.x", nseq).reshape(nseq, k)
    for _ in range(2):  # twice: the counters must be reusable
        got = ops.matvec_grouped_x2_silu_quant(da, db, ids, x, rows)
    want = ops.matvec_grouped_x2_silu_quant(da, db, ids, x, rows, fused=False)
    assert bit_equal(got[0], want[0]) and bit_equal(got[1], want[1])
    assert np.array_equal(got[2], want[2]) and bit_equal(got[3], want[3])


def test_attention_with_the_quantize_tail(ops, synth):
    n_head, n_head_kv, hd, max_kv = 8, 2, 64, 48
    pos = np.array([5, 47, 0], dtype=np.int32)
    kvd = n_head_kv * hd
    q = synth.normal_f32(3 * n_head * hd, 95, "atq.q")
    k = synth.normal_f32(3 * max_kv * kvd, 95, "atq.k")
    v = synth.normal_f32(3 * max_kv * kvd, 95, "atq.v")
    for _ in range(2):
        got = ops.attention_meta_quant(q, k, v, pos, n_head, n_head_kv, hd, max_kv)
    want = ops.attention_meta_quant(q, k, v, pos, n_head, n_head_kv, hd, max_kv, fused=False)
    assert bit_equal(got[0], want[0]) and np.array_equal(got[1], want[1]) and bit_equal(got[2], want[2])
