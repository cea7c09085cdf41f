"""Performance cases: the work that a program built on this library has it do, through its public entry points.

Every model case is the benchmark architecture (synth.QWEN3MOE_30B, random-init Q6_K weights of the benchmark's
distribution). A program loads a model once and then sends it requests, so a model, and the context that its requests
continue from, is made once per process and kept; what a seed makes is the request: the prompt, the next token of every
sequence, the draft, or for the single products the matrix and the activations.

Requests leave the context they continue from intact: a sequence only ever writes at and behind its own position.
"""
import json
import math

import numpy as np
import torch

from llamd_rs_b200 import backend, model, synth

HP = synth.QWEN3MOE_30B
N_LAYER = HP["n_layer"]
MAX_CTX = 2304       # positions of the single-sequence model (f32 cache)
MAX_CTX_F16 = 4224   # positions of the long-context model (binary16 cache)
LONG_LAYERS = 12     # layers of the long-context model: a quarter of the stack, every layer launches the same kernels
MAX_BATCH = 160      # sequences of the batch model
BATCH_CTX = 288      # positions per sequence of the batch model


def listed():
    return [
        # the headline: greedy decoding of one sequence behind a 512-token prompt, tokens fed back on the device
        dict(name="decode_greedy", kind="decode", pos=512, n=4),
        # one token of one long conversation over a binary16 cache, and its logits to the host for a sampler
        dict(name="decode_long_sampled", kind="sample", pos=4001),
        # a small, a middle and a large serving batch, every sequence at its own position; the small one's caller samples,
        # so it takes the logits too
        dict(name="batch_8", kind="batch", nseq=8, sampled=True),
        dict(name="batch_32", kind="batch", nseq=32, sampled=False),
        dict(name="batch_128", kind="batch", nseq=128, sampled=False),
        # the benchmark's prompt; a long ragged prompt of several tiles; a chat turn that continues a conversation
        dict(name="prefill_512", kind="prefill", n=512, base=0),
        dict(name="prefill_1999", kind="prefill", n=1999, base=0),
        dict(name="prefill_turn_37", kind="prefill", n=37, base=300),
        # a draft of eight tokens checked in one pass (speculative decoding)
        dict(name="verify_9", kind="verify", n=9, base=512),
        # single products through the host-facing calls: the smallest projection (latency), the largest matrix for a few
        # sequences, and the Q8_0 type
        dict(name="matvec_q6k_small", kind="matvec", type="q6k", rows=512, k=2048, nseq=1),
        dict(name="matvec_q6k_head_4", kind="matvec", type="q6k", rows=151936, k=2048, nseq=4),
        dict(name="matvec_q8_0_2", kind="matvec", type="q8_0", rows=4096, k=2048, nseq=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "sample", "batch", "batch", "prefill", "prefill", "verify", "matvec"])
    if kind == "decode":
        return dict(kind=kind, pos=_log_int(rng, 8, 2000), n=rng.randint(1, 6))
    if kind == "sample":
        return dict(kind=kind, pos=_log_int(rng, 64, 4200))
    if kind == "batch":
        nseq = _log_int(rng, 2, MAX_BATCH)
        return dict(kind=kind, nseq=nseq, sampled=nseq <= 8 and rng.random() < 0.5)
    if kind == "prefill":
        return dict(kind=kind, n=_log_int(rng, 4, 1999), base=rng.choice([0, rng.randint(1, 300)]))
    if kind == "verify":
        return dict(kind=kind, n=_log_int(rng, 2, 40), base=_log_int(rng, 8, 2000))
    if rng.random() < 0.6:
        return dict(kind=kind, type="q6k", rows=_log_int(rng, 64, 151936), k=256 * rng.choice([1, 3, 5, 8, 8, 16]), nseq=rng.randint(1, 8))
    return dict(kind=kind, type="q8_0", rows=_log_int(rng, 64, 20000), k=32 * rng.choice([24, 33, 64, 64, 128]), nseq=rng.randint(1, 8))


# ---- what a program keeps ----------------------------------------------------------------------------------------------

_staging = None  # pinned host memory that weights go through
_models = {}     # key -> the loaded model
_context = {}    # key -> what its caches hold, as far as that is known


def _q6k_blocks(n, gen):
    """n Q6_K blocks of synth.q6k_blocks' distribution, made on the GPU, as a host array (valid until the next call)."""
    global _staging
    b = torch.randint(0, 256, (n, synth.Q6K_BLOCK_BYTES), dtype=torch.uint8, device="cuda", generator=gen)
    b[:, 192:208] = ((b[:, 192:208] & 63).to(torch.int16) - 32).to(torch.int8).view(torch.uint8)
    b[:, 208:210] = (torch.randn(n, device="cuda", generator=gen).abs() * 1e-3).half().view(torch.uint8).view(n, 2)
    if _staging is None or _staging.numel() < b.numel():
        _staging = torch.empty(max(b.numel(), HP["n_vocab"] * HP["n_embd"] // synth.QK_K * synth.Q6K_BLOCK_BYTES), dtype=torch.uint8, pin_memory=True)
    host = _staging[:b.numel()]
    host.copy_(b.view(-1))
    return host.numpy()


def _q8_0_blocks(n, gen):
    b = torch.empty((n, synth.Q8_0_BLOCK_BYTES), dtype=torch.uint8, device="cuda")
    b[:, 2:] = torch.randint(-127, 128, (n, 32), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
    b[:, :2] = (torch.randn(n, device="cuda", generator=gen).abs() * 1e-2).half().view(torch.uint8).view(n, 2)
    return b.view(-1).cpu().numpy()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _load(n_layer, max_kv, max_seq):
    hp = dict(HP, n_layer=n_layer)
    E, H, ffe, gen = hp["n_embd"], hp["head_dim"], hp["n_ff_expert"], _gen(1)
    qd, kvd = hp["n_head"] * H, hp["n_head_kv"] * H
    m = model.CudaModel(hp, max_kv, max_seq)

    def q6k(layer, which, elements):
        m.set_tensor(layer, which, _q6k_blocks(elements // synth.QK_K, gen))

    q6k(-1, model.T_TOK_EMBD, hp["n_vocab"] * E)
    q6k(-1, model.T_OUTPUT, hp["n_vocab"] * E)
    m.set_tensor(-1, model.T_OUTPUT_NORM, np.ones(E, np.float32))
    for il in range(n_layer):
        for which, n in ((model.T_ATTN_NORM, E), (model.T_FFN_NORM, E), (model.T_ATTN_Q_NORM, H), (model.T_ATTN_K_NORM, H)):
            m.set_tensor(il, which, np.ones(n, np.float32))
        for which, rows, k in ((model.T_ATTN_Q, qd, E), (model.T_ATTN_K, kvd, E), (model.T_ATTN_V, kvd, E), (model.T_ATTN_OUT, E, qd)):
            q6k(il, which, rows * k)
        m.set_tensor(il, model.T_FFN_GATE_INP, (torch.randn(hp["n_expert"] * E, device="cuda", generator=gen) * 0.02).cpu().numpy())
        for which in (model.T_FFN_GATE_EXPS, model.T_FFN_UP_EXPS, model.T_FFN_DOWN_EXPS):
            q6k(il, which, hp["n_expert"] * ffe * E)
    torch.cuda.synchronize()
    return m


def _model(key):
    if key not in _models:
        if key == "batch":
            m = _load(N_LAYER, BATCH_CTX, MAX_BATCH)
        elif key == "long":
            m = _load(LONG_LAYERS, MAX_CTX_F16, 1)
            m.set_option("kv_f16", 1)
        else:
            m = _load(N_LAYER, MAX_CTX, 1)
        _models[key] = m
    return _models[key]


def _tokens(seed, n, what):
    return synth.token_ids(n, HP["n_vocab"], seed, "perf", what).astype(np.int32)


def _batch_len(s):
    """Positions that sequence s of the batch model has behind it: a few long conversations, many short ones."""
    if s < 8:
        return 264 - s
    return 96 - (s - 8) // 4 if s < 64 else 40 - (s - 64) // 12


def _fill_batch(m):
    toks = np.stack([_tokens(7, MAX_BATCH, "context %d" % p) for p in range(_batch_len(0))])
    for p in range(_batch_len(0)):
        n = sum(_batch_len(s) > p for s in range(MAX_BATCH))  # (the lengths do not grow with s)
        m.forward_batch(toks[p, :n], np.full(n, p, np.int32))


def _with_context(key, case, n):
    """The model behind `key` with n positions of context in sequence 0 (or the batch model's own contexts)."""
    m, want = _model(key), "batch" if key == "batch" else json.dumps(case, sort_keys=True)
    if _context.get(key) != want:
        if key == "batch":
            _fill_batch(m)
        elif n:
            m.prefill(_tokens(7, n, "context"), 0)
        _context[key] = want
    return m


# ---- the five functions --------------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "sample"):
        m = _with_context("long" if kind == "sample" else "single", case, case["pos"])
        return dict(case, m=m, token=int(_tokens(seed, 1, "next")[0]))
    if kind == "batch":
        n = case["nseq"]
        return dict(case, m=_with_context("batch", case, 0), tokens=_tokens(seed, n, "next"),
                    positions=np.array([_batch_len(s) for s in range(n)], np.int32))
    if kind in ("prefill", "verify"):
        return dict(case, m=_with_context("single", case, case["base"]), tokens=_tokens(seed, case["n"], "prompt"))
    gen, rows, k = _gen(seed), case["rows"], case["k"]
    if case["type"] == "q6k":
        w = backend.DeviceWeights.upload(_q6k_blocks(rows * k // 256, gen), rows, k // 256)
    else:
        w = backend.Q80Weights.upload(_q8_0_blocks(rows * k // 32, gen), rows, k // 32)
    return dict(case, w=w, x=torch.randn(case["nseq"] * k, device="cuda", generator=gen).cpu().numpy())


def run(s):
    kind = s["kind"]
    if kind == "decode":
        return s["m"].decode(s["token"], s["pos"], s["n"])[0]
    if kind == "sample":
        return {"token": s["m"].forward(s["token"], s["pos"]), "logits": s["m"].logits()}
    if kind == "batch":
        tokens = s["m"].forward_batch(s["tokens"], s["positions"])
        return {"tokens": tokens, "logits": s["m"].logits(s["nseq"])} if s["sampled"] else tokens
    if kind == "prefill":
        return {"token": s["m"].prefill(s["tokens"], s["base"]), "logits": s["m"].logits()}
    if kind == "verify":
        return s["m"].verify(s["tokens"], s["base"])
    return s["w"].matvec_f32(s["x"], s["nseq"])


def _pass_work(n_layer, tokens, heads, kv_rows, kv_pairs, kv_bytes):
    """One pass of `tokens` tokens: attention reads kv_rows cached rows (K and V) and computes kv_pairs (token, position)
    pairs; the head runs for `heads` tokens. An expert's weights are read once if any token of the pass chose it."""
    E, H, ne, nu, ffe, V = HP["n_embd"], HP["head_dim"], HP["n_expert"], HP["n_expert_used"], HP["n_ff_expert"], HP["n_vocab"]
    qd, kvd = HP["n_head"] * H, HP["n_head_kv"] * H
    q6k = synth.Q6K_BLOCK_BYTES / synth.QK_K
    dense, expert = E * (2 * qd + 2 * kvd), 3 * E * ffe
    experts = ne * (1 - (1 - nu / ne) ** tokens)
    per_layer = q6k * (dense + experts * expert) + 4 * ne * E + 2 * kvd * kv_bytes * (kv_rows + tokens)
    flops = 2 * (n_layer * (tokens * (dense + nu * expert + ne * E) + 2 * kv_pairs * qd) + heads * V * E)
    return n_layer * per_layer + (q6k * V * E + 4 * heads * V if heads else 0) + tokens * E * q6k, flops


def work(case):
    kind = case["kind"]
    if kind == "decode":
        got = [_pass_work(N_LAYER, 1, 1, case["pos"] + i, case["pos"] + i + 1, 4) for i in range(case["n"])]
        return dict(bytes=sum(b for b, _ in got), flops=sum(f for _, f in got))
    if kind == "sample":
        b, f = _pass_work(LONG_LAYERS, 1, 1, case["pos"], case["pos"] + 1, 2)
    elif kind == "batch":
        rows = sum(_batch_len(s) for s in range(case["nseq"]))
        b, f = _pass_work(N_LAYER, case["nseq"], case["nseq"], rows, rows + case["nseq"], 4)
    elif kind in ("prefill", "verify"):
        n, base = case["n"], case["base"]
        b, f = _pass_work(N_LAYER, n, n if kind == "verify" else 1, base, n * base + n * (n + 1) // 2, 4)
    else:
        rows, k, n = case["rows"], case["k"], case["nseq"]
        b = rows * k * (synth.Q6K_BLOCK_BYTES / 256 if case["type"] == "q6k" else synth.Q8_0_BLOCK_BYTES / 32) + 4 * n * (k + rows)
        f = 2 * n * rows * k
    return dict(bytes=b, flops=f)


def tolerance(case):
    # every path performs the reference's operations in the reference's order: tokens, logits and products are bit for bit
    # the same whatever kernel computes them
    return "exact"
