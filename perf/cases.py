"""Workloads for timing the framework and comparing two builds of it.

A case is one call path of a step as a host drives it: a sublayer of the ragged continuous-batching step through the C
ABI (include/q38_kernels.h), the launchers in the order in which the step issues them, or a whole step of a slice of the
model through the engine's runner. Geometries are those of the 27B model and of the "small" and "medium" design
benchmarks; batch sizes, contexts and step lengths span a single interactive request up to full serving batches.

    listed()            the standard cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) weights, caches, states and inputs on the GPU, from the seed alone
    run(state)          one pass; returns the device buffers (or host logits) that it wrote
    exact(case, seed)   the same outputs in float64, by plain torch
    work(case)          bytes and FLOPs the pass cannot do without
    tolerance(case)     error that another correct implementation at the same precision may show
"""

from __future__ import annotations

import ctypes as C
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

HD, PAGE, CHUNK_MIN = 256, 64, 16  # head size, tokens per KV page, shortest run the engine gives to the chunked recurrence
DEV = "cuda"

# Hybrid geometries: hidden, feed-forward, q / kv heads of the attention layers, k / v heads of the Gated DeltaNet layers.
HYBRID = {
    "27b": dict(H=5120, I=17408, nq=24, nkv=4, nk=16, nv=48),
    "medium": dict(H=4096, I=11008, nq=16, nkv=4, nk=16, nv=32),
    "small": dict(H=2048, I=5632, nq=8, nkv=2, nk=8, nv=16),
}
RECIPES = {
    "default": dict(qkvg=5, o=5, qkvz=5, out=5, gate_up=4, down=5, head=8),
    "lean": dict(qkvg=4, o=4, qkvz=4, out=4, gate_up=4, down=4, head=6),
    "quality": dict(qkvg=5, o=6, qkvz=5, out=6, gate_up=4, down=6, head=8),
}
DESIGN = {
    "medium": dict(W=4096, heads=32, kv_heads=8),
    "small": dict(W=2048, heads=16, kv_heads=4),
}
VOCAB_27B = 248320
EPS = 1e-6


def listed():
    return [
        # one interactive request, a token at a time: latency of the whole step (4 of the 64 layers, 1/16 of the vocabulary)
        dict(name="decode_1", kind="decode", seqs=1, context=1000),
        # the first chunk of a prompt, the engine's default step of 512 tokens, up to the logits of its last token
        dict(name="prompt_512", kind="prompt", tokens=512),
        # feed-forward of a handful of concurrent requests
        dict(name="mlp_5", kind="mlp", geo="27b", recipe="default", m=5),
        # feed-forward of the serving batch the repository's benchmark uses
        dict(name="mlp_64", kind="mlp", geo="27b", recipe="default", m=64),
        # linear-attention mixer of that batch: state streaming
        dict(name="gdn_decode_64", kind="gdn", geo="27b", recipe="default", seqs=64, tokens=64),
        # the same mixer over a step that packs three prompts of uneven length
        dict(name="gdn_prefill_1531", kind="gdn", geo="27b", recipe="default", seqs=3, tokens=1531),
        # attention mixer of the serving batch over mixed contexts of up to 8192 tokens
        dict(name="attn_decode_64", kind="attn", geo="27b", recipe="default", seqs=64, tokens=64, context=8192, kv="int8"),
        # one chunk of a long document behind 32 K tokens of context
        dict(name="attn_prefill_32k", kind="attn", geo="27b", recipe="default", seqs=1, tokens=512, context=32768, kv="int8"),
        # logits over the full vocabulary and the sampler for the serving batch
        dict(name="head_64", kind="head", geo="27b", recipe="default", m=64),
        # attention with mixed heads, last chunk of a 2048-token prompt
        dict(name="mixed_prefill_512", kind="mixed", geo="medium", seqs=1, tokens=512, context=1536),
        # retention over one 2048-token prompt step
        dict(name="retention_prefill_2048", kind="retention", geo="medium", seqs=1, tokens=2048),
        # latent attention of the serving batch at 2048 tokens of context
        dict(name="latent_decode_64", kind="latent", geo="medium", seqs=64, tokens=64, context=2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "prompt", "mlp", "mlp", "gdn", "gdn", "attn", "attn", "head", "mixed", "retention", "latent"])
    geo, recipe = rng.choice(["27b", "27b", "medium", "small"]), rng.choice(["default", "default", "lean", "quality"])
    if kind == "decode":
        return dict(kind=kind, seqs=_log(rng, 1, 16), context=_log(rng, 64, 2000))
    if kind == "prompt":
        return dict(kind=kind, tokens=_log(rng, 16, 512))
    if kind == "mlp":
        return dict(kind=kind, geo=geo, recipe=recipe, m=_log(rng, 1, 2048))
    if kind == "head":
        return dict(kind=kind, geo=geo, recipe=recipe, m=_log(rng, 1, 64))
    if kind == "gdn":
        if rng.random() < 0.4:
            n = _log(rng, 1, 64)
            return dict(kind=kind, geo=geo, recipe=recipe, seqs=n, tokens=n)
        n = rng.randint(1, 4)
        return dict(kind=kind, geo=geo, recipe=recipe, seqs=n, tokens=_log(rng, 64, 1531))
    if kind == "attn":
        kv = rng.choice(["int8", "int8", "bf16"])
        if rng.random() < 0.5:
            n = _log(rng, 1, 64)
            return dict(kind=kind, geo=geo, recipe=recipe, seqs=n, tokens=n, context=_log(rng, 256, 8192), kv=kv)
        n = rng.randint(1, 3)
        return dict(kind=kind, geo=geo, recipe=recipe, seqs=n, tokens=_log(rng, 64, 512), context=_log(rng, 64, 16384), kv=kv)
    design = rng.choice(["medium", "small"])
    if rng.random() < 0.5:
        n = _log(rng, 1, 64)
        case = dict(kind=kind, geo=design, seqs=n, tokens=n)
    else:
        case = dict(kind=kind, geo=design, seqs=rng.randint(1, 3), tokens=_log(rng, 64, 512 if kind == "mixed" else 2048))
    if kind != "retention":
        case["context"] = _log(rng, 64, 2048)
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------------
class State:
    """Everything a pass touches, by name; `calls` issues its launches."""


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _ragged(case, seed):
    """(lengths, contexts before the step) of the sequences: uneven runs that add up to the step, contexts log-uniform up to
    the case's. The seed decides which sequence gets which."""
    n, total, top = case["seqs"], case["tokens"], case.get("context", 0)
    if n == total:
        lens = [1] * n
    else:
        share = np.random.default_rng(total).dirichlet([4.0] * n)
        lens = [max(CHUNK_MIN, int(s * total)) for s in share]
        lens[int(np.argmax(lens))] += total - sum(lens)
    if n == 1:
        ctx = [top]
    else:
        ctx = [int(v) for v in np.exp(np.linspace(math.log(64), math.log(max(65, top)), n))] if top else [0] * n
    order = np.random.default_rng(seed).permutation(n)
    return [lens[i] for i in order], [ctx[i] for i in order]


class _Batch:
    def __init__(self, lens, pos0, slots):
        mk = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
        start = [0]
        for n in lens:
            start.append(start[-1] + n)
        self.keep = (mk(start), mk(slots), mk(pos0), mk([p + i for p, n in zip(pos0, lens) for i in range(n)]),
                     mk([b for b, n in enumerate(lens) for _ in range(n)]))
        self.desc = pkg.BatchDesc(len(lens), start[-1], max(lens), *[pkg.ptr(t) for t in self.keep])


class _Bq:
    """Random codes and scales in the layout of a model file; weights of standard deviation 1 / sqrt(k)."""

    def __init__(self, g, rows, k, bits):
        n = (rows + 127) // 128 * 128
        self.n, self.k, self.bits, self.rows = n, k, bits, rows
        byte = lambda c: torch.randint(0, 256, (c,), dtype=torch.uint8, device=DEV, generator=g)  # noqa: E731
        self.lo = byte(n * k // 2)
        self.hi = byte(n * k * (bits - 4) // 8) if bits > 4 else None
        s = math.sqrt(12.0 / k) / (1 << bits)
        self.sc = (s * (0.75 + 0.5 * torch.rand(n * k // 64, device=DEV, generator=g))).to(torch.bfloat16)
        self.desc = pkg.BQWeight(pkg.ptr(self.lo), pkg.ptr(self.hi), pkg.ptr(self.sc), bits, n, k, rows)

    @property
    def bytes(self):
        return _bq_bytes(self.rows, self.k, self.bits)


def _bq_bytes(n, k, bits):
    return n * k * bits / 8 + n * k / 32


def _dense(g, n, k, bias=False):
    w = (torch.randn((n, k), generator=g, device=DEV) / math.sqrt(k)).to(torch.bfloat16)
    b = 0.1 * torch.randn(n, generator=g, device=DEV) if bias else None
    return w, b, pkg.DenseWeight(pkg.ptr(w), pkg.ptr(b), n, k, k)


def _workspace(tokens):
    floats = 2 * pkg.kernels().q38_num_sms() * 128 * tokens
    part, count = torch.empty(floats, device=DEV), torch.zeros(65536, dtype=torch.int32, device=DEV)
    return part, count, pkg.GemmWorkspace(pkg.ptr(part), floats, pkg.ptr(count), 65536)


def _hidden(S, g, m, H):
    """The residual stream before a sublayer: fp32 rows, their bf16 copy and the sums of squares of their 128-column blocks."""
    S.residual = torch.randn((m, H), generator=g, device=DEV)
    S.x = S.residual.to(torch.bfloat16)
    S.norm_in = (S.residual ** 2).view(m, H // 128, 128).sum(-1)
    S.x_out, S.norm_out = torch.empty_like(S.x), torch.empty_like(S.norm_in)


def _into_residual(S):
    return pkg.GemmEpilogue(pkg.EPI_RESIDUAL, None, 0, 0, pkg.ptr(S.residual), pkg.ptr(S.x_out), pkg.ptr(S.norm_out), None, 0, 0.0, None)


def _from_norm(S, kind, out, ldo, n_store, H):
    return pkg.GemmEpilogue(kind, pkg.ptr(out), ldo, n_store, None, None, None, pkg.ptr(S.norm_in), H, EPS, None)


def _gemm(S, a, m, w, ep):
    pkg.check(S.K.q38_qgemm(pkg.ptr(a), m, C.byref(w.desc), C.byref(ep), C.byref(S.ws), _stream(), -1))


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ---- hybrid sublayers --------------------------------------------------------------------------------------------------
def _prepare_mlp(S, case, g):
    d, bits, m = HYBRID[case["geo"]], RECIPES[case["recipe"]], case["m"]
    _hidden(S, g, m, d["H"])
    S.up, S.down = _Bq(g, 2 * d["I"], d["H"], bits["gate_up"]), _Bq(g, d["H"], d["I"], bits["down"])
    S.act = torch.empty((m, d["I"]), dtype=torch.bfloat16, device=DEV)
    e1, e2 = _from_norm(S, pkg.EPI_SWIGLU, S.act, d["I"], 0, d["H"]), _into_residual(S)

    def calls():
        _gemm(S, S.x, m, S.up, e1)
        _gemm(S, S.act, m, S.down, e2)
        return {"residual": S.residual, "x": S.x_out, "norm": S.norm_out}
    return calls


def _prepare_gdn(S, case, g):
    d, bits = HYBRID[case["geo"]], RECIPES[case["recipe"]]
    H, nk, nv, m = d["H"], d["nk"], d["nv"], case["tokens"]
    conv_dim = (2 * nk + nv) * 128
    ld = conv_dim + nv * 128
    lens, _ = _ragged(case, S.seed)
    S.lens = lens
    S.batch = _Batch(lens, [64] * len(lens), list(range(len(lens))))
    _hidden(S, g, m, H)
    S.w_in, S.w_out = _Bq(g, ld, H, bits["qkvz"]), _Bq(g, H, nv * 128, bits["out"])
    S.w_ab = (torch.randn((2 * nv, H), generator=g, device=DEV) / math.sqrt(H)).to(torch.bfloat16)
    S.conv_w = 0.4 * torch.randn((conv_dim, 4), generator=g, device=DEV)
    S.A = -(0.5 + 7.5 * torch.rand(nv, generator=g, device=DEV))
    S.dt = 0.5 * torch.randn(nv, generator=g, device=DEV)
    S.gain = 1.0 + 0.2 * torch.randn(128, generator=g, device=DEV)
    S.state = 0.1 * torch.randn((len(lens), 1, nv, 128, 128), generator=g, device=DEV)
    S.conv = torch.randn((len(lens), 1, 3, conv_dim), generator=g, device=DEV).to(torch.bfloat16)
    S.proj = torch.empty((m, ld), dtype=torch.bfloat16, device=DEV)
    S.ab = torch.empty((m, 2 * nv), device=DEV)
    S.qkv = torch.empty((m, conv_dim), device=DEV)
    S.mix = torch.empty((m, nv * 128), dtype=torch.bfloat16, device=DEV)
    chunked = max(lens) >= CHUNK_MIN
    need = int(S.K.q38_gdn_chunk_scratch_floats(m, len(lens), nv)) if chunked else 0
    S.scratch = torch.empty(max(need, 1), device=DEV)
    dims, st = pkg.GdnDims(nk, nv, conv_dim, ld), pkg.GdnStateDesc(pkg.ptr(S.state), pkg.ptr(S.conv), 1)
    cp = pkg.GdnConvParams(pkg.ptr(S.proj), pkg.ptr(S.conv_w), pkg.ptr(S.qkv), 0)
    rp = pkg.GdnRecurrenceParams(pkg.ptr(S.qkv), pkg.ptr(S.ab), pkg.ptr(S.A), pkg.ptr(S.dt), pkg.ptr(S.proj) + 2 * conv_dim, ld,
                                 pkg.ptr(S.gain), EPS, pkg.ptr(S.mix), 0)
    e1, e2 = _from_norm(S, pkg.EPI_STORE_BF16, S.proj, ld, ld, H), _into_residual(S)
    D, B, T = C.byref(dims), C.byref(S.batch.desc), C.byref(st)

    def calls():
        s = _stream()
        _gemm(S, S.x, m, S.w_in, e1)
        pkg.check(S.K.q38_gdn_ab(pkg.ptr(S.x), m, H, pkg.ptr(S.w_ab), 2 * nv, pkg.ptr(S.norm_in), EPS, pkg.ptr(S.ab), s))
        pkg.check(S.K.q38_gdn_conv(C.byref(cp), D, B, T, s))
        if chunked:
            pkg.check(S.K.q38_gdn_recurrence_chunked(C.byref(rp), D, B, T, pkg.ptr(S.scratch), need, s))
        else:
            pkg.check(S.K.q38_gdn_recurrence(C.byref(rp), D, B, T, s))
        _gemm(S, S.mix, m, S.w_out, e2)
        return {"residual": S.residual, "x": S.x_out, "norm": S.norm_out, "mix": S.mix, "gates": S.ab, "state": S.state,
                "conv": S.conv}
    return calls


def _kv_pool(S, g, kv, nkv, lens, ctx):
    """Pages of all sequences in shuffled order, filled with keys and values of about unit size."""
    pages = [(c + n + PAGE - 1) // PAGE for c, n in zip(ctx, lens)]
    total, widest = sum(pages) + 1, max(pages)
    half = nkv * PAGE * HD
    code = pkg.KV_INT8 if kv == "int8" else pkg.KV_BF16
    page_bytes = int(S.K.q38_kv_page_bytes(code, nkv))
    if kv == "int8":
        S.pool = torch.randint(0, 256, (total, page_bytes), dtype=torch.uint8, device=DEV, generator=g)
        scale = (torch.rand((total, nkv * PAGE * 8), device=DEV, generator=g) * 0.008 + 0.008).to(torch.float16)
        S.pool[:, 2 * half:] = scale.view(torch.uint8)
    else:
        S.pool = torch.randn((total, 2 * half), device=DEV, generator=g).to(torch.bfloat16).view(torch.uint8)
    order = np.random.default_rng(S.seed + 1).permutation(total - 1) + 1
    table, at = np.zeros((len(lens), widest), dtype=np.int32), 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
    S.table = torch.from_numpy(table).to(DEV)
    return pkg.KvCacheDesc(pkg.ptr(S.pool), code, nkv, total, page_bytes, total * page_bytes, pkg.ptr(S.table), widest)


def _prepare_attn(S, case, g):
    d, bits = HYBRID[case["geo"]], RECIPES[case["recipe"]]
    H, nq, nkv, m = d["H"], d["nq"], d["nkv"], case["tokens"]
    lens, ctx = _ragged(case, S.seed)
    S.lens, S.ctx = lens, ctx
    ld, q_dim = (2 * nq + 2 * nkv) * HD, nq * HD
    S.batch = _Batch(lens, ctx, list(range(len(lens))))
    _hidden(S, g, m, H)
    S.w_in, S.w_out = _Bq(g, ld, H, bits["qkvg"]), _Bq(g, H, q_dim, bits["o"])
    S.q_norm = 1.0 + 0.2 * torch.randn(HD, generator=g, device=DEV)
    S.k_norm = 1.0 + 0.2 * torch.randn(HD, generator=g, device=DEV)
    kv = _kv_pool(S, g, case["kv"], nkv, lens, ctx)
    S.proj = torch.empty((m, ld), dtype=torch.bfloat16, device=DEV)
    S.q = torch.empty((m, q_dim), dtype=torch.float16, device=DEV)
    S.mix = torch.empty((m, q_dim), dtype=torch.bfloat16, device=DEV)
    decode = max(lens) == 1
    # the engine's scratch: 64 splits for each of up to 65 rows; a prefill step reads it as one row per token
    rows, splits = (len(lens), 64) if decode else (m, min(64, 65 * 64 // m))
    S.scratch = torch.empty(rows * nq * splits * (HD + 2), device=DEV)
    rp = pkg.QkNormRopeParams(pkg.ptr(S.proj), ld, pkg.ptr(S.q_norm), pkg.ptr(S.k_norm), EPS, 1e7, nq, nkv, pkg.ptr(S.q), 0)
    ap = pkg.AttentionParams(pkg.ptr(S.q), pkg.ptr(S.proj) + 2 * q_dim, ld, pkg.ptr(S.mix), nq, nkv, 0, pkg.ptr(S.scratch), splits,
                             0 if decode or splits < 2 else m)
    e1, e2 = _from_norm(S, pkg.EPI_STORE_BF16, S.proj, ld, ld, H), _into_residual(S)
    B, V = C.byref(S.batch.desc), C.byref(kv)
    attend = S.K.q38_attention_decode if decode else S.K.q38_attention_prefill

    def calls():
        s = _stream()
        _gemm(S, S.x, m, S.w_in, e1)
        pkg.check(S.K.q38_qk_norm_rope_append(C.byref(rp), B, V, s))
        pkg.check(attend(C.byref(ap), B, V, s))
        _gemm(S, S.mix, m, S.w_out, e2)
        return {"residual": S.residual, "x": S.x_out, "norm": S.norm_out, "mix": S.mix, "pages": S.pool}
    return calls


def _prepare_head(S, case, g):
    d, bits, m = HYBRID[case["geo"]], RECIPES[case["recipe"]], case["m"]
    vocab = VOCAB_27B if case["geo"] == "27b" else 32768
    _hidden(S, g, m, d["H"])
    S.w = _Bq(g, vocab, d["H"], bits["head"])
    S.logits = torch.empty((m, vocab), device=DEV)
    S.tokens, S.logprob = torch.empty(m, dtype=torch.int32, device=DEV), torch.empty(m, device=DEV)
    S.history, S.history_len = torch.zeros((m, 4096), dtype=torch.int32, device=DEV), torch.zeros(m, dtype=torch.int32, device=DEV)
    S.slot, S.step = torch.arange(m, dtype=torch.int32, device=DEV), torch.full((m,), 7, dtype=torch.int32, device=DEV)
    one = pkg.SamplingParamsDev(1.0, 20, 0.95, 0.0, 0.0, 1.0, S.seed)  # the engine's default sampling
    S.params = torch.frombuffer(bytearray(bytes((pkg.SamplingParamsDev * m)(*[one] * m))), dtype=torch.uint8).to(DEV)
    sa = pkg.SamplingArgs(pkg.ptr(S.logits), vocab, vocab, pkg.ptr(S.params), pkg.ptr(S.slot), pkg.ptr(S.history),
                          pkg.ptr(S.history_len), 4096, pkg.ptr(S.step), pkg.ptr(S.tokens), pkg.ptr(S.logprob))
    ep = _from_norm(S, pkg.EPI_STORE_F32, S.logits, vocab, vocab, d["H"])

    def calls():
        _gemm(S, S.x, m, S.w, ep)
        pkg.check(S.K.q38_sample(C.byref(sa), m, _stream()))
        return {"logits": S.logits, "tokens": S.tokens, "logprob": S.logprob}
    return calls


# ---- layer-list sublayers ----------------------------------------------------------------------------------------------
def _dense_call(S, x, ldx, m, w, kind, out, ldo, gate=None, ld_gate=0):
    ep = pkg.DenseEpilogue(kind, pkg.ptr(out), ldo, 0.0, 0.0, gate, ld_gate)
    x, W = pkg.ptr(x), w[2]
    return lambda s: pkg.check(S.K.q38_dense_gemm(x, ldx, pkg.ACT_BF16, m, C.byref(W), C.byref(ep), C.byref(S.ws), s, -1))


def _grouped_call(S, x, ldx, m, w, groups, kind, out, ldo, gate=None, ld_gate=0):
    ep = pkg.DenseEpilogue(kind, pkg.ptr(out), ldo, 0.0, 0.0, gate, ld_gate)
    x, W = pkg.ptr(x), w[2]
    return lambda s: pkg.check(S.K.q38_dense_gemm_grouped(x, ldx, pkg.ACT_BF16, m, C.byref(W), C.byref(groups), C.byref(ep),
                                                          C.byref(S.ws), s, -1))


def _layer_pages(S, g, heads, k_dim, v_dim, lens, ctx):
    pages = [(c + n + PAGE - 1) // PAGE for c, n in zip(ctx, lens)]
    total, widest = sum(pages) + 1, max(pages)
    S.pages = torch.randn((total, heads * PAGE * (k_dim + v_dim)), device=DEV, generator=g).to(torch.bfloat16)
    order = np.random.default_rng(S.seed + 1).permutation(total - 1) + 1
    table, at = np.zeros((len(lens), widest), dtype=np.int32), 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
    S.table = torch.from_numpy(table).to(DEV)
    page_bytes = heads * PAGE * (k_dim + v_dim) * 2
    return pkg.KvLayerDesc(pkg.ptr(S.pages), pkg.KV_BF16, heads, k_dim, v_dim, total, page_bytes, pkg.ptr(S.table), widest)


def _prepare_mixed(S, case, g):
    d, m, dim = DESIGN[case["geo"]], case["tokens"], 128
    W, N, G = d["W"], d["heads"], d["kv_heads"]
    lens, ctx = _ragged(case, S.seed)
    S.lens, S.ctx = lens, ctx
    S.batch = _Batch(lens, ctx, list(range(len(lens))))
    kv = _layer_pages(S, g, G, dim, dim, lens, ctx)
    bf = lambda *s: torch.empty(s, dtype=torch.bfloat16, device=DEV)  # noqa: E731
    ld = (N + 2 * G) * dim
    S.x = torch.randn((m, W), generator=g, device=DEV).to(torch.bfloat16)
    S.w_in, S.w_out = _dense(g, ld, W, True), _dense(g, W, N * dim, True)
    S.talk = (torch.eye(N, device=DEV) + torch.randn((N, N), generator=g, device=DEV) / N).contiguous()
    S.freq = torch.tensor([10000.0 ** (-2.0 * i / 64) for i in range(32)], dtype=torch.float64, device=DEV)
    S.proj, S.q, S.mix, S.y = bf(m, ld), bf(m, N * dim), bf(m, N * dim), torch.empty((m, W), device=DEV)
    decode = max(lens) == 1
    S.stats = torch.empty(8 * m * N * 2, device=DEV)
    S.scores = torch.empty(kv.num_pages * N * PAGE if decode else 1, device=DEV)
    S.parts = torch.empty(len(lens) * 64 * N * (dim + 2) if decode else 1, device=DEV)
    rp = pkg.RopeAppendParams(pkg.ptr(S.proj), ld, pkg.ACT_BF16, N, G, dim, dim, 64, pkg.ptr(S.freq), pkg.ptr(S.q), None, None, None)
    ap = pkg.MixedAttentionParams(pkg.ptr(S.q), pkg.ACT_BF16, N, dim, dim ** -0.5, pkg.ptr(S.talk), pkg.ptr(S.mix), N * dim,
                                  pkg.ptr(S.stats), 8, pkg.ptr(S.scores) if decode else None, pkg.ptr(S.parts), 64)
    c1 = _dense_call(S, S.x, W, m, S.w_in, pkg.DENSE_STORE, S.proj, ld)
    c2 = _dense_call(S, S.mix, N * dim, m, S.w_out, pkg.DENSE_STORE_F32, S.y, W)
    attend = S.K.q38_mixed_attention_decode if decode else S.K.q38_mixed_attention_prefill
    B, V = C.byref(S.batch.desc), C.byref(kv)

    def calls():
        s = _stream()
        c1(s)
        pkg.check(S.K.q38_rope_append(C.byref(rp), B, V, s))
        pkg.check(attend(C.byref(ap), B, V, s))
        c2(s)
        return {"y": S.y, "mix": S.mix, "pages": S.pages}
    return calls


def _decays(N):
    return [1.0 - 2.0 ** -(5 + 5 * h / N) for h in range(N)]


def _prepare_retention(S, case, g):
    W, m, dim = DESIGN[case["geo"]]["W"], case["tokens"], 128
    N, ld = W // 128, 4 * W
    lens, _ = _ragged(case, S.seed)
    S.lens = lens
    S.batch = _Batch(lens, [128] * len(lens), list(range(len(lens))))
    S.x = torch.randn((m, W), generator=g, device=DEV).to(torch.bfloat16)
    S.w_in, S.w_out = _dense(g, ld, W), _dense(g, W, W)
    S.state = 0.3 * torch.randn((len(lens), N, dim, dim), generator=g, device=DEV)
    S.freq = torch.tensor([10000.0 ** (-2.0 * i / dim) for i in range(dim // 2)], dtype=torch.float64, device=DEV)
    S.pow = torch.tensor([[a ** i for i in range(pkg.RETENTION_CHUNK + 1)] for a in _decays(N)], dtype=torch.float32, device=DEV)
    S.proj = torch.empty((m, ld), dtype=torch.bfloat16, device=DEV)
    S.qk = torch.empty(int(S.K.q38_retention_qk_bytes(m, N, dim, pkg.ACT_BF16)), dtype=torch.uint8, device=DEV)
    S.o, S.mix, S.y = torch.empty((m, W), device=DEV), torch.empty((m, W), dtype=torch.bfloat16, device=DEV), torch.empty((m, W), device=DEV)
    p = pkg.RetentionParams(pkg.ptr(S.proj), ld, pkg.ACT_BF16, N, dim, dim, dim, pkg.ptr(S.freq), pkg.ptr(S.pow), dim ** -0.5, EPS,
                            pkg.ptr(S.qk), pkg.ptr(S.o), pkg.ptr(S.mix), W)
    st = pkg.RecurrentStateDesc(pkg.ptr(S.state), None, N * dim * dim * 4)
    c1 = _dense_call(S, S.x, W, m, S.w_in, pkg.DENSE_STORE, S.proj, ld)
    c2 = _dense_call(S, S.mix, W, m, S.w_out, pkg.DENSE_STORE_F32, S.y, W)

    def calls():
        s = _stream()
        c1(s)
        pkg.check(S.K.q38_retention(C.byref(p), C.byref(S.batch.desc), C.byref(st), s))
        c2(s)
        return {"y": S.y, "mix": S.mix, "state": S.state}
    return calls


def _packs(lens, rank, own):
    """Whether the engine makes keys and values from the latents for this step (long runs) or stays in the latent space."""
    return max(lens) > 1 and sum(lens) / len(lens) * 1.5 * (2.0 * rank - own) > 0.5 * rank * own


def _prepare_latent(S, case, g):
    d, m, dim, rank = DESIGN[case["geo"]], case["tokens"], 128, 512
    W, N, qr = d["W"], d["heads"], 3 * d["W"] // 8
    lens, ctx = _ragged(case, S.seed)
    S.lens, S.ctx = lens, ctx
    S.batch = _Batch(lens, ctx, list(range(len(lens))))
    kv = _layer_pages(S, g, 1, rank, 0, lens, ctx)
    bf = lambda *s: torch.empty(s, dtype=torch.bfloat16, device=DEV)  # noqa: E731
    ld, Nd = qr + rank + N * dim, N * dim
    S.x = torch.randn((m, W), generator=g, device=DEV).to(torch.bfloat16)
    S.w_in, S.w_q, S.w_out = _dense(g, ld, W), _dense(g, Nd, qr), _dense(g, W, Nd)
    S.w_kv = _dense(g, 2 * Nd, rank)  # the heads' key rows, then their value rows
    S.q_gain = 1.0 + 0.2 * torch.randn(qr, generator=g, device=DEV)
    S.kv_gain = 1.0 + 0.2 * torch.randn(rank, generator=g, device=DEV)
    S.proj, S.ql, S.qh, S.mix, S.y = bf(m, ld), bf(m, qr), bf(m, Nd), bf(m, Nd), torch.empty((m, W), device=DEV)
    lp = pkg.LatentAppendParams(pkg.ptr(S.proj), ld, pkg.ACT_BF16, qr, rank, pkg.ptr(S.q_gain), pkg.ptr(S.kv_gain), EPS, pkg.ptr(S.ql), qr)
    gate = pkg.ptr(S.proj) + 2 * (qr + rank)
    B, V = C.byref(S.batch.desc), C.byref(kv)
    steps = [_dense_call(S, S.x, W, m, S.w_in, pkg.DENSE_STORE, S.proj, ld),
             lambda s: pkg.check(S.K.q38_latent_append(C.byref(lp), B, V, s)),
             _dense_call(S, S.ql, qr, m, S.w_q, pkg.DENSE_STORE, S.qh, Nd)]
    if _packs(lens, rank, 2 * dim):
        rows = sum((c + n + PAGE - 1) // PAGE * PAGE for c, n in zip(ctx, lens))
        longest = max(c + n for c, n in zip(ctx, lens))
        S.lat, S.kvp = bf(rows, rank), bf(rows, 2 * Nd)
        pp = pkg.PackedAttentionParams(pkg.ptr(S.qh), Nd, dim, pkg.ptr(S.kvp), pkg.ptr(S.kvp) + 2 * Nd, 2 * Nd, dim, dim, N, dim, dim,
                                       dim ** -0.5, gate, ld, pkg.ptr(S.mix), Nd)
        steps += [lambda s: pkg.check(S.K.q38_latent_gather(B, V, longest, rows, pkg.ptr(S.lat), s)),
                  _dense_call(S, S.lat, rank, rows, S.w_kv, pkg.DENSE_STORE, S.kvp, 2 * Nd),
                  lambda s: pkg.check(S.K.q38_packed_attention(C.byref(pp), B, s))]
    else:
        wk, wv = S.w_kv[0][:Nd].view(N, dim, rank).transpose(1, 2).contiguous(), S.w_kv[0][Nd:]
        S.wk = wk, None, pkg.DenseWeight(pkg.ptr(wk), None, rank, dim, dim)
        S.wv = wv, None, pkg.DenseWeight(pkg.ptr(wv), None, dim, rank, rank)
        S.qa, S.ol = bf(m, N * rank), bf(m, N * rank)
        floats = int(S.K.q38_latent_attention_partial_floats(rank))
        S.parts = torch.empty(floats, device=DEV)
        ap = pkg.LatentAttentionParams(pkg.ptr(S.qa), pkg.ACT_BF16, N, dim ** -0.5, pkg.ptr(S.ol), pkg.ptr(S.parts), floats)
        steps += [_grouped_call(S, S.qh, Nd, m, S.wk, pkg.DenseGroups(N, dim, rank), pkg.DENSE_STORE, S.qa, N * rank),
                  lambda s: pkg.check(S.K.q38_latent_attention(C.byref(ap), B, V, s)),
                  _grouped_call(S, S.ol, N * rank, m, S.wv, pkg.DenseGroups(N, rank, dim), pkg.DENSE_GATE_SIGMOID, S.mix, Nd, gate, ld)]
    steps.append(_dense_call(S, S.mix, Nd, m, S.w_out, pkg.DENSE_STORE_F32, S.y, W))

    def calls():
        s = _stream()
        for f in steps:
            f(s)
        return {"y": S.y, "mix": S.mix, "pages": S.pages}
    return calls


# ---- the runner --------------------------------------------------------------------------------------------------------
SLICE_LAYERS, SLICE_VOCAB = 4, VOCAB_27B // 16 // 128 * 128


def _model_file(seed):
    """A slice of the 27B model as a file: one period of its layers (three Gated DeltaNet, one attention) and the same share
    of its vocabulary, random weights."""
    from q38b200 import synth
    cfg = synth.model_config(**dict(synth.CONFIG_27B, layers=SLICE_LAYERS, vocab=SLICE_VOCAB, eos=(1, 2)))
    torch.manual_seed(seed)
    f = tempfile.NamedTemporaryFile(prefix="perf_cases_", suffix=".q38", dir="/dev/shm" if os.path.isdir("/dev/shm") else None, delete=False)
    f.close()
    synth.write_random_planes_q38(f.name, cfg, seed=seed)
    return f.name


class _Served:
    """A loaded model with a runner; given back when the state goes."""

    def __init__(self, path, seqs, tokens):
        from q38b200 import engine
        self.engine, self.model, self.runner = engine, engine.Model(path), None
        self.runner = engine.Runner(self.model, engine.default_runner_options(
            max_batch=max(seqs, 1), prefill_chunk=512, verbose=0, kv_tokens=seqs * (tokens + 128), max_context=tokens + 64))

    def __del__(self):
        if self.runner is not None:
            self.runner.close()
        self.model.close()


def _step_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ids = lambda n: rng.integers(0, SLICE_VOCAB, n).astype(np.int32)  # noqa: E731
    if case["kind"] == "prompt":
        return [ids(case["tokens"])]
    return [ids(n + 1) for n in _contexts(case, seed)]


def _contexts(case, seed):
    n, top = case["seqs"], case["context"]
    ctx = [top] if n == 1 else [int(v) for v in np.exp(np.linspace(math.log(32), math.log(top), n))]
    return [ctx[i] for i in np.random.default_rng(seed + 5).permutation(n)]


def _prepare_runner(S, case):
    S.rows = _step_inputs(case, S.seed)
    path = _model_file(S.seed)
    try:
        S.served = _Served(path, len(S.rows), max(len(r) for r in S.rows))
    finally:
        os.unlink(path)
    r, g = S.served.runner, S.served.engine.greedy()
    for slot, t in enumerate(S.rows):
        r.reset_slot(slot)
        if not r.kv_ensure(slot, len(t)):
            raise RuntimeError("KV cache too small")
    if case["kind"] == "prompt":
        def calls():
            r.reset_slot(0)
            return {"logits": r.step_logits([(0, 0, S.rows[0], None, 0)], [(0, len(S.rows[0]) - 1)])}
        return calls
    for slot, t in enumerate(S.rows):
        for at in range(0, len(t) - 1, 512):
            r.prefill([(slot, at, t[at:min(at + 512, len(t) - 1)], None, 0)])
    step = [(slot, len(t) - 1, int(t[-1]), g, 1) for slot, t in enumerate(S.rows)]

    def calls():
        r.decode(step)
        return {"logits": r.last_logits(len(step))}
    return calls


# ---- the interface -----------------------------------------------------------------------------------------------------
SUBLAYERS = {"mlp": _prepare_mlp, "gdn": _prepare_gdn, "attn": _prepare_attn, "head": _prepare_head, "mixed": _prepare_mixed,
             "retention": _prepare_retention, "latent": _prepare_latent}


def prepare(case, seed):
    S = State()
    S.seed, S.K = int(seed), pkg.kernels()
    if case["kind"] in ("decode", "prompt"):
        S.calls = _prepare_runner(S, case)
        return S
    S.part, S.count, S.ws = _workspace(512)
    S.calls = SUBLAYERS[case["kind"]](S, case, _gen(seed))
    return S


def run(state):
    return state.calls()


# ---- float64 -----------------------------------------------------------------------------------------------------------
def _plane_codes(lo, hi, bits, n, k):
    """Signed codes [n][k] of the packed planes: 16 x 64 slabs, lane 4 g + t owns column 8 j + g and rows 2 t + 8 h + e."""
    def nibbles(p):
        b = p.view(n // 64, k // 16, 8, 4, 4, 2, 2)  # nb kb g t word e byte: pair 4 word + 2 byte + nibble
        u = torch.stack([b & 15, b >> 4], -1)
        return u.permute(0, 4, 6, 2, 1, 7, 3, 5).reshape(n, k)
    u = nibbles(lo).to(torch.int16)
    if bits == 5:
        b = hi.view(n // 64, k // 16, 8, 4, 2, 2)  # nb kb g t e byte: pair 8 byte + bit
        v = torch.stack([(b >> i) & 1 for i in range(8)], -1).view(n // 64, k // 16, 8, 4, 2, 2, 4, 2)
        u += v.permute(0, 5, 6, 2, 1, 7, 3, 4).reshape(n, k).to(torch.int16) << 4
    elif bits == 6:
        b = hi.view(n // 64, k // 16, 8, 4, 2, 2, 2)  # nb kb g t word e byte: pair 8 word + 4 byte + field
        v = torch.stack([(b >> (2 * i)) & 3 for i in range(4)], -1).view(n // 64, k // 16, 8, 4, 2, 2, 2, 2, 2)
        u += v.permute(0, 4, 6, 7, 2, 1, 8, 3, 5).reshape(n, k).to(torch.int16) << 4
    elif bits == 8:
        u += nibbles(hi).to(torch.int16) << 4
    return u - (1 << (bits - 1))


def _weights(w):
    """float64 [rows][k] of a packed tensor: bf16(code * scale)."""
    sc = w.sc.view(w.n // 64, w.k // 64, 8, 8).permute(0, 3, 2, 1).reshape(w.n, w.k // 64).float()
    code = _plane_codes(w.lo, w.hi, w.bits, w.n, w.k).float().view(w.n, w.k // 64, 64)
    return (code * sc[:, :, None]).to(torch.bfloat16).double().view(w.n, w.k)[:w.rows]


def _product(x, w):
    """x w^T in float64, a slice of the rows of w at a time."""
    full = isinstance(w, _Bq)
    if not full:
        return x @ w.double().T
    if w.rows <= 40000:
        return x @ _weights(w).T
    W, out = _Slice(w), []
    for lo in range(0, w.n, 32768):
        out.append(x @ W.rows(lo, min(w.n, lo + 32768)).T)
    return torch.cat(out, 1)[:, :w.rows]


class _Slice:
    """Rows of a packed tensor as a packed tensor of their own (64-row blocks are contiguous in every plane)."""

    def __init__(self, w):
        self.w = w

    def rows(self, lo, hi):
        w, s = self.w, State()
        cut = lambda p: p[p.numel() // w.n * lo:p.numel() // w.n * hi]  # noqa: E731
        s.n, s.k, s.bits, s.rows = hi - lo, w.k, w.bits, hi - lo
        s.lo, s.hi, s.sc = cut(w.lo), None if w.hi is None else cut(w.hi), cut(w.sc)
        return _weights(s)


def _silu(x):
    return x * torch.sigmoid(x)


def _exact_mlp(x, rs, up, down):
    c = _product(x, up) * rs
    return _product(_silu(c[:, 0::2]) * c[:, 1::2], down)


def _exact_gdn(x, rs, w_in, w_ab, conv_w, A, dt, gain, w_out, nk, nv, lens, state, conv):
    """(mixer rows, their projection, gates, states, conv states) of runs of `lens` tokens."""
    conv_dim = (2 * nk + nv) * 128
    proj, ab = _product(x, w_in) * rs, x @ w_ab.double().T * rs
    state, conv = state.clone().double(), conv.clone().double()  # [seq][nv][128 dv][128 dk], [seq][3][conv_dim]
    mix, at = [], 0
    for b, n in enumerate(lens):
        rows = torch.cat([conv[b], proj[at:at + n, :conv_dim]])
        act = _silu(sum(rows[j:j + n] * conv_w[:, j].double() for j in range(4)))
        conv[b] = rows[-3:]
        q, k, v = act[:, :nk * 128].view(n, nk, 128), act[:, nk * 128:2 * nk * 128].view(n, nk, 128), act[:, 2 * nk * 128:].view(n, nv, 128)
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q = (unit(q) * 128 ** -0.5).repeat_interleave(nv // nk, 1)
        k = unit(k).repeat_interleave(nv // nk, 1)
        beta = torch.sigmoid(ab[at:at + n, :nv])
        decay = torch.exp(A.double() * torch.nn.functional.softplus(ab[at:at + n, nv:] + dt.double()))
        s, o = state[b], torch.empty((n, nv, 128), dtype=torch.float64, device=x.device)
        for t in range(n):
            s = s * decay[t, :, None, None]
            delta = beta[t, :, None] * (v[t] - torch.einsum("hvk,hk->hv", s, k[t]))
            s = s + delta[:, :, None] * k[t, :, None, :]
            o[t] = torch.einsum("hvk,hk->hv", s, q[t])
        state[b] = s
        o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + EPS) * gain.double()
        mix.append((o * _silu(proj[at:at + n, conv_dim:].view(n, nv, 128))).view(n, nv * 128))
        at += n
    mix = torch.cat(mix)
    return mix, _product(mix, w_out), ab, state, conv


def _turn(x, pos, dims, base):
    """x [t][heads][d]: dimension i of the leading `dims` turns with i + dims / 2."""
    half = dims // 2
    ang = pos.double()[:, None] * base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _causal(q, k, v, first, scale, talk=None):
    """q [t][H][d] at positions first ..., k [T][G][d], v [T][G][dv]: softmax per head, mixed by `talk` if given."""
    t, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty((t, H, v.shape[2]), dtype=torch.float64, device=q.device)
    hide = torch.arange(k.shape[0], device=q.device)[None, :] > first + torch.arange(t, device=q.device)[:, None]
    if talk is None:
        for h in range(H):
            s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill_(hide, -math.inf)
            out[:, h] = torch.softmax(s, -1) @ v[:, h * G // H]
        return out
    p = torch.stack([torch.softmax((q[:, h] @ k[:, h * G // H].T * scale).masked_fill_(hide, -math.inf), -1) for h in range(H)])
    for h in range(H):
        out[:, h] = torch.einsum("g,gij->ij", talk[h].double(), p) @ v[:, h * G // H]
    return out


def _stored(x):
    """int8 codes with an fp16 scale per 64 values, as the cache keeps them."""
    y = x.reshape(-1, 64)
    s = (y.abs().amax(1, keepdim=True) / 127).to(torch.float16).double()
    return (torch.where(s > 0, torch.clamp(torch.round(y / s), -127, 127), 0.0) * s).reshape(x.shape)


def _history(S, b, n, nkv, kv):
    """Keys and values [n][nkv][256] of sequence b's first n cached tokens."""
    pages, half = S.pool[S.table[b, :(n + PAGE - 1) // PAGE].long()], nkv * PAGE * HD
    if kv == "int8":
        code = pages[:, :2 * half].contiguous().view(torch.int8).double().view(-1, 2, nkv, PAGE, 4, 64)
        x = (code * pages[:, 2 * half:].contiguous().view(torch.float16).double().view(-1, 2, nkv, PAGE, 4, 1)).view(-1, 2, nkv, PAGE, HD)
    else:
        x = pages.contiguous().view(torch.bfloat16).double().view(-1, 2, nkv, PAGE, HD)
    x = x.permute(1, 0, 3, 2, 4).reshape(2, -1, nkv, HD)[:, :n]
    return x[0], x[1]


def _exact_attn(x, rs, w_in, w_out, q_norm, k_norm, nq, nkv, lens, ctx, past, store):
    """past(b) -> keys and values before the step; store: what the cache makes of a row."""
    proj = _product(x, w_in) * rs
    q_dim, mix, at = nq * HD, [], 0
    unit = lambda t, w: t / torch.sqrt((t * t).mean(-1, keepdim=True) + EPS) * w.double()  # noqa: E731
    for b, (n, p) in enumerate(zip(lens, ctx)):
        row, pos = proj[at:at + n], torch.arange(p, p + n, device=x.device)
        q = _turn(unit(row[:, :q_dim].reshape(n, nq, HD), q_norm), pos, 64, 1e7)
        k = _turn(unit(row[:, 2 * q_dim:2 * q_dim + nkv * HD].reshape(n, nkv, HD), k_norm), pos, 64, 1e7)
        v = row[:, 2 * q_dim + nkv * HD:].reshape(n, nkv, HD)
        k0, v0 = past(b)
        o = _causal(q, torch.cat([k0, store(k)]), torch.cat([v0, store(v)]), p, HD ** -0.5)
        mix.append(o.reshape(n, q_dim) * torch.sigmoid(row[:, q_dim:2 * q_dim]))
        at += n
    mix = torch.cat(mix)
    return mix, _product(mix, w_out)


def _scale(norm, H):
    return 1.0 / torch.sqrt(norm.double().sum(1, keepdim=True) / H + EPS)


def _residual_out(S, delta):
    r = S.residual.double() + delta
    return {"residual": r, "x": r, "norm": (r * r).view(r.shape[0], -1, 128).sum(-1)}


def _exact_layer_list(S, case):
    x, m, dim = S.x.double(), case["tokens"], 128
    lin = lambda a, w: a @ w[0].double().T + (0 if w[1] is None else w[1].double())  # noqa: E731
    d = DESIGN[case["geo"]]
    proj, mix, at, unit = lin(x, S.w_in), [], 0, lambda t, w=1.0: t / torch.sqrt((t * t).mean(-1, keepdim=True) + EPS) * w
    if case["kind"] == "retention":
        N, state = d["W"] // dim, S.state.double()
        decay = torch.tensor(_decays(N), dtype=torch.float64, device=DEV)[:, None, None]
        for b, n in enumerate(S.lens):
            q, k, v, gate = proj[at:at + n].view(n, 4, N, dim).unbind(1)
            pos = torch.arange(128, 128 + n, device=DEV)
            q, k = _turn(q, pos, dim, 10000.0), _turn(k, pos, dim, 10000.0) * dim ** -0.5
            s, o = state[b], torch.empty((n, N, dim), dtype=torch.float64, device=DEV)
            for t in range(n):
                s = decay * s + k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hdv,hd->hv", s, q[t])
            state[b] = s
            mix.append((unit(o) * _silu(gate)).reshape(n, -1))
            at += n
        mix = torch.cat(mix)
        return {"y": lin(mix, S.w_out), "mix": mix, "state": state}
    N = d["heads"]
    for b, (n, p) in enumerate(zip(S.lens, S.ctx)):
        row, pos = proj[at:at + n], torch.arange(p, p + n, device=DEV)
        used = S.pages[S.table[b, :(p + PAGE - 1) // PAGE].long()].double()
        if case["kind"] == "mixed":
            G = d["kv_heads"]
            q, k, v = row.split([N * dim, G * dim, G * dim], 1)
            q, k = _turn(q.reshape(n, N, dim), pos, 64, 10000.0), _turn(k.reshape(n, G, dim), pos, 64, 10000.0)
            k0 = used[:, :G * PAGE * dim].view(-1, G, PAGE, dim).permute(0, 2, 1, 3).reshape(-1, G, dim)[:p]
            v0 = used[:, G * PAGE * dim:].view(-1, G, dim, PAGE).permute(0, 3, 1, 2).reshape(-1, G, dim)[:p]
            o = _causal(q, torch.cat([k0, k]), torch.cat([v0, v.reshape(n, G, dim)]), p, dim ** -0.5, S.talk)
            mix.append(o.reshape(n, -1))
        else:
            qr, rank = 3 * d["W"] // 8, 512
            ql, c, gate = row.split([qr, rank, N * dim], 1)
            q = lin(unit(ql, S.q_gain.double()), S.w_q).view(n, N, dim)
            c = torch.cat([used.view(-1, rank)[:p], unit(c, S.kv_gain.double())])
            k, v = lin(c, S.w_kv).view(-1, 2, N, dim).unbind(1)
            mix.append(_causal(q, k, v, p, dim ** -0.5).reshape(n, -1) * torch.sigmoid(gate))
        at += n
    mix = torch.cat(mix)
    return {"y": lin(mix, S.w_out), "mix": mix, "pages": None}


class _File:
    """Tensors of a model file on the GPU."""

    def __init__(self, path):
        with open(path, "rb") as f:
            f.seek(8)
            (n,) = struct.unpack("<Q", f.read(8))
            self.tensors = json.loads(f.read(n))["tensors"]
            self.start = (16 + n + 4095) // 4096 * 4096
        self.map = np.memmap(path, dtype=np.uint8, mode="r")

    def raw(self, at, size):
        return torch.from_numpy(np.array(self.map[self.start + at:self.start + at + size])).to(DEV)

    def packed(self, name):
        t, w = self.tensors[name], _Bq.__new__(_Bq)
        w.bits, (w.n, w.k) = int(t["dtype"][2:]), t["shape"]
        w.rows = t.get("rows", w.n)
        w.lo, w.sc = self.raw(*t["planes"]["lo"]), self.raw(*t["planes"]["scales"]).view(torch.bfloat16)
        w.hi = self.raw(*t["planes"]["hi"]) if "hi" in t["planes"] else None
        return w

    def plain(self, name):
        t = self.tensors[name]
        return self.raw(t["offset"], t["bytes"]).view(torch.bfloat16 if t["dtype"] == "bf16" else torch.float32).view(t["shape"])


def _exact_runner(case, seed):
    path = _model_file(seed)
    f = _File(path)
    d, rows = HYBRID["27b"], _step_inputs(case, seed)
    lens = [len(r) for r in rows]
    r = f.plain("embed").double()[torch.from_numpy(np.concatenate(rows)).long().to(DEV)]
    none = torch.empty((0, d["nkv"], HD), dtype=torch.float64, device=DEV)
    for i in range(SLICE_LAYERS):
        rs = _scale(r * r, d["H"])
        if f"{i}.attn.o" in f.tensors:
            _, y = _exact_attn(r, rs, f.packed(f"{i}.attn.qkvg"), f.packed(f"{i}.attn.o"), f.plain(f"{i}.attn.q_norm"),
                               f.plain(f"{i}.attn.k_norm"), d["nq"], d["nkv"], lens, [0] * len(lens), lambda b: (none, none), _stored)
        else:
            p = f"{i}.gdn."
            state = torch.zeros((len(lens), d["nv"], 128, 128), device=DEV)
            conv = torch.zeros((len(lens), 3, (2 * d["nk"] + d["nv"]) * 128), device=DEV)
            y = _exact_gdn(r, rs, f.packed(p + "qkvz"), f.plain(p + "ab"), f.plain(p + "conv"), f.plain(p + "A"), f.plain(p + "dt_bias"),
                           f.plain(p + "norm"), f.packed(p + "out"), d["nk"], d["nv"], lens, state, conv)[1]
        r = r + y
        r = r + _exact_mlp(r, _scale(r * r, d["H"]), f.packed(f"{i}.mlp.gate_up"), f.packed(f"{i}.mlp.down"))
    last = r[torch.tensor(np.cumsum(lens) - 1, device=DEV)]
    out = _product(last, f.packed("lm_head")) * _scale(last * last, d["H"])
    os.unlink(path)
    return {"logits": out}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        if kind == "decode" and sum(_contexts(case, int(seed))) > 6000:
            return None
        return _exact_runner(case, int(seed))
    S = prepare(case, seed)
    if kind in ("mixed", "retention", "latent"):
        return _exact_layer_list(S, case)
    d = HYBRID[case["geo"]]
    x, rs = S.x.double(), _scale(S.norm_in, d["H"])
    if kind == "mlp":
        return _residual_out(S, _exact_mlp(x, rs, S.up, S.down))
    if kind == "head":
        return {"logits": _product(x, S.w) * rs, "tokens": None, "logprob": None}
    if kind == "gdn":
        mix, y, ab, state, conv = _exact_gdn(x, rs, S.w_in, S.w_ab, S.conv_w, S.A, S.dt, S.gain, S.w_out, d["nk"], d["nv"], S.lens,
                                             S.state[:, 0], S.conv[:, 0])
        return dict(_residual_out(S, y), mix=mix, gates=ab, state=state[:, None], conv=conv[:, None])
    past = lambda b: _history(S, b, S.ctx[b], d["nkv"], case["kv"])  # noqa: E731
    store = _stored if case["kv"] == "int8" else (lambda t: t)
    mix, y = _exact_attn(x, rs, S.w_in, S.w_out, S.q_norm, S.k_norm, d["nq"], d["nkv"], S.lens, S.ctx, past, store)
    return dict(_residual_out(S, y), mix=mix, pages=None)


# ---- work --------------------------------------------------------------------------------------------------------------
def _rows_work(m, H):
    return m * H * 10  # the residual read and written in fp32, its bf16 copy written


def _pairs(lens, ctx):
    return sum(n * c + n * (n + 1) / 2 for n, c in zip(lens, ctx))


def _typical(case):
    """Lengths and contexts for counting work: the runs in equal parts, contexts at the mean of their distribution."""
    n, top = case["seqs"], case.get("context", 0)
    mean = top if n == 1 else (top - 64) / math.log(top / 64) if top > 64 else top
    return [case["tokens"] / n] * n, [mean] * n


def _w_mlp(d, bits, m):
    return (_bq_bytes(2 * d["I"], d["H"], bits["gate_up"]) + _bq_bytes(d["H"], d["I"], bits["down"]) + m * d["H"] * 2 + _rows_work(m, d["H"]),
            6.0 * m * d["H"] * d["I"])


def _w_gdn(d, bits, m, seqs):
    conv = (2 * d["nk"] + d["nv"]) * 128
    n = conv + d["nv"] * 128
    by = (_bq_bytes(n, d["H"], bits["qkvz"]) + _bq_bytes(d["H"], d["nv"] * 128, bits["out"]) + 4 * d["nv"] * d["H"]
          + seqs * (2 * d["nv"] * 65536 + 12 * conv) + m * d["H"] * 2 + m * d["nv"] * 256 + _rows_work(m, d["H"]))
    return by, 2.0 * m * d["H"] * (n + d["nv"] * 128 + 2 * d["nv"]) + 6.0 * m * d["nv"] * 16384


def _w_attn(d, bits, lens, ctx, kv):
    m, n, q = sum(lens), (2 * d["nq"] + 2 * d["nkv"]) * HD, d["nq"] * HD
    row = d["nkv"] * (2 * HD + 16 if kv == "int8" else 4 * HD)
    by = (_bq_bytes(n, d["H"], bits["qkvg"]) + _bq_bytes(d["H"], q, bits["o"]) + (sum(ctx) + sum(lens)) * row + m * d["H"] * 2 + m * q * 2
          + _rows_work(m, d["H"]))
    return by, 2.0 * m * d["H"] * (n + q) + 4.0 * q * _pairs(lens, ctx)


def work(case):
    kind = case["kind"]
    if kind in ("mixed", "retention", "latent"):
        d, m = DESIGN[case["geo"]], case["tokens"]
        W, N, dim = d["W"], d["heads"], 128
        lens, ctx = _typical(case)
        if kind == "mixed":
            G = d["kv_heads"]
            n, own = (N + 2 * G) * dim, N * dim
            by = 2 * W * (n + own) + m * W * 6 + (sum(ctx) + m) * G * dim * 4
            fl = 2.0 * m * W * (n + own) + 2.0 * N * (2 * dim + N) * _pairs(lens, ctx)
        elif kind == "retention":
            by, fl = 2 * 5 * W * W + m * W * 6 + case["seqs"] * 8 * W * dim, 10.0 * m * W * W + 4.0 * m * W * dim
        else:
            qr, rank = 3 * W // 8, 512
            n, own = qr + rank + N * dim, N * dim
            by = 2 * (W * (n + own) + own * qr + 2 * own * rank) + m * W * 6 + (sum(ctx) + m) * rank * 2
            new = sum(lens) + (sum(ctx) if _packs(lens, rank, 2 * dim) else 0)
            fl = 2.0 * m * (W * (n + own) + own * qr) + 4.0 * new * own * rank + 4.0 * N * dim * _pairs(lens, ctx)
        return {"bytes": by, "flops": fl}
    if kind in ("decode", "prompt"):
        d, bits = HYBRID["27b"], RECIPES["default"]
        seqs, m = case.get("seqs", 1), case.get("tokens", case.get("seqs", 1))
        lens, ctx = [m / seqs] * seqs, [case.get("context", 0) * (1 if seqs == 1 else 0.4)] * seqs
        parts = [_w_gdn(d, bits, m, seqs)] * 3 + [_w_attn(d, bits, lens, ctx, "int8")] + [_w_mlp(d, bits, m)] * 4
        parts.append((_bq_bytes(SLICE_VOCAB, d["H"], bits["head"]) + seqs * SLICE_VOCAB * 4, 2.0 * seqs * d["H"] * SLICE_VOCAB))
    else:
        d, bits = HYBRID[case["geo"]], RECIPES[case["recipe"]]
        if kind == "mlp":
            parts = [_w_mlp(d, bits, case["m"])]
        elif kind == "head":
            vocab = VOCAB_27B if case["geo"] == "27b" else 32768
            parts = [(_bq_bytes(vocab, d["H"], bits["head"]) + case["m"] * (2 * d["H"] + 4 * vocab), 2.0 * case["m"] * d["H"] * vocab)]
        elif kind == "gdn":
            parts = [_w_gdn(d, bits, case["tokens"], case["seqs"])]
        else:
            parts = [_w_attn(d, bits, *_typical(case), case["kv"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """Activations are bf16 between the launches, sums fp32: a different order of a sum moves single roundings of the
    intermediate rows. `differ` allows cache bytes and sampled tokens next to a tie."""
    if case["kind"] == "head":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.01}  # fp32 logits of equal products
    if case["kind"] in ("decode", "prompt"):
        return {"rel": 0.02, "max": 0.3}
    return {"rel": 0.01, "max": 0.3, "differ": 0.01}
