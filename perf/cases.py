"""Performance cases: the calls that carry serving and scoring, over the sizes they meet.

Every case goes through entry points that a program can call: the tensor-level ops of
``orinfer_b200.ops.functional`` for single layers, and ``ModelRunner`` (replayed from a CUDA
graph over static buffers, as the engine does) for whole calls.  Geometries are the presets of
``orinfer_b200.config``.  ``exact`` restates each path in 64-bit torch, with the quantisation
steps that define it (INT8 rows, INT8 KV, FP16 layer boundaries).
"""

from __future__ import annotations

import dataclasses
import math

import torch

from orinfer_b200.config import PRESETS
from orinfer_b200.models.runner import KVPool, ModelRunner, Packet
from orinfer_b200.models.weights import LayerWeights, ModelWeights, QLinear
from orinfer_b200.ops import functional as F
from orinfer_b200.ops import native

PAGE = 128
Q4_STD, Q2_STD = 13.0, 3.2            # spread of the integer weights of uniformly drawn codes


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one token of one request through the widest projection of a 4B-class layer
        dict(name="linear_decode", kind="linear", m=1, n=19456, k=2560, fmt="q4"),
        # the same projection for a prefill chunk
        dict(name="linear_prefill", kind="linear", m=2048, n=19456, k=2560, fmt="q4"),
        # attention of a full decode batch with short conversations
        dict(name="attn_decode_batch", kind="attn_decode", rows=128, ctx=640, qh=32, kvh=8, d=128),
        # a few requests far into long documents
        dict(name="attn_decode_long", kind="attn_decode", rows=6, ctx=24000, qh=32, kvh=8, d=128),
        # one long prompt of a dense model
        dict(name="attn_prefill", kind="attn_prefill", chunks=1, rows=4096, past=0, qh=32, kvh=8,
             d=128, gated=False),
        # chunks of two prompts that already have a cached prefix, gated heads of 256 channels
        dict(name="attn_prefill_gated", kind="attn_prefill", chunks=2, rows=777, past=3000, qh=16,
             kvh=2, d=256, gated=True),
        # recurrent mixer of a hybrid layer: a packet with two prompts, one of them continued
        dict(name="gdn_prefill", kind="gdn", segs=2, rows=2100, hk=16, hv=32, d=128),
        # the same mixer for one decode step of a batch
        dict(name="gdn_decode", kind="gdn", segs=64, rows=64, hk=16, hv=32, d=128),
        # routed experts of a prompt chunk, 35B-A3B class
        dict(name="moe_prefill", kind="moe", rows=2048, hidden=2048, ffn=768, experts=128, top_k=8,
             fmt="q4", shared=0),
        # routed experts and the shared expert of a decode batch, 80B-A3B class
        dict(name="moe_decode", kind="moe", rows=16, hidden=2048, ffn=512, experts=512, top_k=10,
             fmt="q2", shared=512),
        # whole call: one decode step of eight requests, two layers and the head of the 4B class
        dict(name="model_decode", kind="model", rows=8, ctx=900, prefill=False, layers=2),
        # whole call: a 512-token prompt up to its logits (one layer: see ``tolerance``)
        dict(name="model_prefill", kind="model", rows=512, ctx=0, prefill=True, layers=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "attn_decode", "attn_prefill", "gdn", "moe", "model"])
    if kind == "linear":
        n, k = rng.choice([(19456, 2560), (6144, 2560), (2560, 4096), (2560, 9728), (5120, 2048),
                           (12288, 2048), (2048, 4096)])
        return dict(kind=kind, m=_log(rng, 1, 2048), n=n, k=k, fmt=rng.choice(["q4", "q4", "w8", "q2"]))
    if kind == "attn_decode":
        qh, kvh, d = rng.choice([(32, 8, 128), (40, 8, 128), (32, 4, 128), (16, 2, 256)])
        rows = _log(rng, 1, 128)
        return dict(kind=kind, rows=rows, ctx=_log(rng, 40, min(24000, 144000 // rows)), qh=qh,
                    kvh=kvh, d=d)
    if kind == "attn_prefill":
        qh, kvh, d, gated = rng.choice([(32, 8, 128, False), (40, 8, 128, False),
                                        (32, 4, 128, False), (16, 2, 256, True)])
        chunks = rng.choice([1, 1, 2, 3])
        return dict(kind=kind, chunks=chunks, rows=_log(rng, 17, 2800 // chunks),
                    past=rng.choice([0, _log(rng, 1, 1000)]), qh=qh, kvh=kvh, d=d, gated=gated)
    if kind == "gdn":
        if rng.random() < 0.5:
            segs = _log(rng, 1, 64)
            return dict(kind=kind, segs=segs, rows=segs, hk=16, hv=32, d=128)
        segs = rng.choice([1, 1, 2, 3])
        return dict(kind=kind, segs=segs, rows=_log(rng, 40 * segs, 1050 * segs), hk=16, hv=32,
                    d=128)
    if kind == "moe":
        if rng.random() < 0.5:
            return dict(kind=kind, rows=_log(rng, 1, 2048), hidden=2048, ffn=768, experts=128,
                        top_k=8, fmt="q4", shared=0)
        return dict(kind=kind, rows=_log(rng, 1, 512), hidden=2048, ffn=512, experts=512, top_k=10,
                    fmt="q2", shared=512)
    if rng.random() < 0.5:
        return dict(kind="model", rows=rng.randint(1, 16), ctx=_log(rng, 30, 3000), prefill=False,
                    layers=rng.choice([1, 2]))
    return dict(kind="model", rows=_log(rng, 20, 512), ctx=0, prefill=True, layers=1)


# ----------------------------------------------------------------------------- inputs
class _Rand:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(1000003 * (seed % 1000000007) + 17)

    def normal(self, *shape, std=1.0, dtype=torch.float32):
        return (torch.randn(*shape, generator=self.g, device="cuda") * std).to(dtype)

    def ints(self, lo, hi, shape, dtype):
        return torch.randint(lo, hi, shape, generator=self.g, device="cuda", dtype=dtype)

    def int8(self, *shape):
        """Gaussian INT8 values whose absolute maximum is about 127."""
        t = torch.randn(*shape, generator=self.g, device="cuda", dtype=torch.float16)
        return (t * 33).clamp_(-127, 127).round_().to(torch.int8)

    def signs(self, k):
        return self.ints(0, 2, (k,), torch.int8) * 2 - 1

    def codes(self, fmt, *lead, n, k, std=0.02):
        """(codes, FP16 row scales) of a projection in one of the checkpoint formats."""
        if fmt == "w8":
            w, unit = self.int8(*lead, n, k), 33.0
        elif fmt == "q4":
            w = self.ints(-2 ** 31, 2 ** 31, (*lead, k // 128, n, 16), torch.int32)
            unit = Q4_STD
        else:
            w = self.ints(-2 ** 15, 2 ** 15, (*lead, k // 128, n, 16), torch.int16)
            unit = Q2_STD
        scale = (torch.rand(*lead, n, generator=self.g, device="cuda") * 0.5 + 0.75) * (std / unit)
        return w, scale.to(torch.float16)

    def linear(self, fmt, n, k, signs):
        w, s = self.codes(fmt, n=n, k=k)
        return QLinear(fmt, n, k, w, s, signs)


def _lens(count, ctx):
    """Ragged context lengths between half of ctx and ctx."""
    return [max(1, int(ctx * (0.5 + 0.5 * ((0.618034 * i) % 1.0)))) if i else ctx
            for i in range(count)]


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _paged(r, lens, kvh, d):
    """Page table (pages in random order) and filled INT8 caches for requests of these lengths."""
    need = [(n + PAGE - 1) // PAGE for n in lens]
    total, width = sum(need), max(need) + 1
    order = (torch.randperm(total, generator=r.g, device="cuda") + 1).to(torch.int32)
    table, at = torch.zeros(len(lens), width, dtype=torch.int32, device="cuda"), 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    cache = lambda: r.int8(total + 1, PAGE, kvh, d)
    scale = lambda: ((torch.rand(total + 1, PAGE, kvh, d // 64, generator=r.g, device="cuda") + 0.5)
                     * (1.0 / 33)).to(torch.float16)
    return dict(table=table, k=cache(), v=cache(), ks=scale(), vs=scale())


def prepare(case, seed):
    native.init()
    return dict(_PREPARE[case["kind"]](case, _Rand(seed)), kind=case["kind"], case=case)


def _prep_linear(c, r):
    w, s = r.codes(c["fmt"], n=c["n"], k=c["k"])
    return dict(a=r.int8(c["m"], c["k"]), a_scale=torch.rand(c["m"], generator=r.g, device="cuda")
                * 0.02 + 0.02, w=w, w_scale=s,
                out=torch.empty(c["m"], c["n"], dtype=torch.float16, device="cuda"))


def _prep_attn_decode(c, r):
    lens = _lens(c["rows"], c["ctx"])
    kv = _paged(r, lens, c["kvh"], c["d"])
    rows = c["rows"]
    return dict(q=r.normal(rows, c["qh"], c["d"], dtype=torch.float16), req=_i32(list(range(rows))),
                pos=_i32([n - 1 for n in lens]),
                scratch=torch.empty(512 * c["qh"] * (c["d"] + 2), device="cuda"),
                out=torch.empty(rows, c["qh"] * c["d"], dtype=torch.float16, device="cuda"), **kv)


def _chunk_rows(c):
    """Rows of every chunk (ragged) of a packet of ``chunks`` prompts."""
    return [max(1, c["rows"] - 131 * i) for i in range(c["chunks"])]


def _prep_attn_prefill(c, r):
    sizes, spec, at = _chunk_rows(c), [], 0
    for i, n in enumerate(sizes):
        spec.append([at, n, c["past"], i])
        at += n
    kv = _paged(r, [n + c["past"] for n in sizes], c["kvh"], c["d"])
    shape = (at, c["qh"], c["d"])
    return dict(q=r.normal(*shape, dtype=torch.float16),
                gate=r.normal(*shape, dtype=torch.float16) if c["gated"] else None,
                chunks=_i32(spec), longest=max(sizes),
                out=torch.empty(at, c["qh"] * c["d"], dtype=torch.float16, device="cuda"), **kv)


def _seg_rows(c):
    base = c["rows"] // c["segs"]
    return [c["rows"] - base * (c["segs"] - 1)] + [base] * (c["segs"] - 1)


def _prep_gdn(c, r):
    hk, hv, d, rows = c["hk"], c["hv"], c["d"], c["rows"]
    conv = (2 * hk + hv) * d
    sizes, segs, first, slot, pos, at = _seg_rows(c), [], [], [], [], 0
    for i, n in enumerate(sizes):
        start = 0 if i == 1 else 300 + i               # the second request is a fresh prompt
        segs.append([at, n, 0, 0])
        first += [at] * n
        slot += [i] * n
        pos += list(range(start, start + n))
        at += n
    return dict(proj=r.normal(rows, conv + hv * d, dtype=torch.float16),
                ab=r.normal(rows, 2 * hv), weight=r.normal(conv, 4, std=0.3, dtype=torch.float16),
                hist=r.normal(c["segs"], 3, conv, dtype=torch.float16),
                state=r.normal(c["segs"], hv, d, d, std=0.05),
                a_log=r.normal(hv, std=0.5) - 1.0, dt_bias=r.normal(hv, std=0.5) - 2.0,
                norm=(r.normal(d, std=0.1) + 1).to(torch.float16),
                segs=_i32(segs), first=_i32(first), slot=_i32(slot), pos=_i32(pos),
                y=torch.empty(rows, conv, dtype=torch.float16, device="cuda"),
                o=torch.empty(rows, hv, d, device="cuda"),
                mix=torch.empty(rows, hv * d, dtype=torch.float16, device="cuda"))


def _prep_moe(c, r):
    rows, h, f, e = c["rows"], c["hidden"], c["ffn"], c["experts"]
    up, up_s = r.codes(c["fmt"], e, n=2 * f, k=h)
    dn, dn_s = r.codes(c["fmt"], e, n=h, k=f)
    half = lambda *s: torch.empty(*s, dtype=torch.float16, device="cuda")
    st = dict(x=r.normal(rows, h, dtype=torch.float16),
              norm=(r.normal(h, std=0.1) + 1).to(torch.float16), signs=r.signs(h),
              signs_mid=r.signs(f), up=up, up_s=up_s, dn=dn, dn_s=dn_s,
              router=r.normal(e + (1 if c["shared"] else 0), h, std=0.02, dtype=torch.float16),
              scratch=F.MoeScratch(rows, c["top_k"], e, h, f, torch.device("cuda")),
              q8=torch.empty(rows, h, dtype=torch.int8, device="cuda"),
              s8=torch.empty(rows, device="cuda"), y16=half(rows, h), out=half(rows, h))
    if c["shared"]:
        fs = c["shared"]
        st.update(sh_up=r.linear("q4", 2 * fs, h, None), sh_dn=r.linear("q4", h, fs, None),
                  sh_signs=r.signs(fs), sh_gu=half(rows, 2 * fs),
                  sh_q=torch.empty(rows, fs, dtype=torch.int8, device="cuda"),
                  sh_s=torch.empty(rows, device="cuda"), sh_out=half(rows, h))
    return st


def _model_config(c):
    return dataclasses.replace(PRESETS["qwen3.5-4b-class"], layers=c["layers"], mtp_layers=0)


def _model_weights(cfg, r):
    h, qd, sign = cfg.hidden, cfg.q_heads * cfg.head_dim, {}
    for k in (h, qd, cfg.ffn):
        sign.setdefault(k, r.signs(k))
    norm = lambda n: (r.normal(n, std=0.1) + 1).to(torch.float16)
    layers = []
    for _ in range(cfg.layers):
        lw = LayerWeights("attn", norm(h), norm(h))
        lw.qkv = r.linear("q4", qd + 2 * cfg.kv_dim, h, sign[h])
        lw.q_norm, lw.k_norm = norm(cfg.head_dim), norm(cfg.head_dim)
        lw.o = r.linear("q4", h, qd, sign[qd])
        lw.gate_up = r.linear("q4", 2 * cfg.ffn, h, sign[h])
        lw.down = r.linear("q4", h, cfg.ffn, sign[cfg.ffn])
        layers.append(lw)
    table, scale = r.codes("w8", n=cfg.vocab, k=h, std=0.5)
    head = QLinear("w8", cfg.vocab, h, table, scale, None)
    return ModelWeights(cfg, table, scale, layers, norm(h), head, sign)


def _prep_model(c, r):
    cfg, rows = _model_config(c), c["rows"]
    w = _model_weights(cfg, r)
    lens = [rows] if c["prefill"] else _lens(rows, c["ctx"])
    pools = [_paged(r, lens, cfg.kv_heads, cfg.head_dim) for _ in range(cfg.layers)]
    table = pools[0]["table"]
    for p in pools[1:]:
        p["table"] = table                      # one page table addresses every layer's cache
    kv = KVPool([p["k"] for p in pools], [p["v"] for p in pools], [p["ks"] for p in pools],
                [p["vs"] for p in pools], pools[0]["k"].shape[0])
    runner = ModelRunner(w, kv, rows)
    ids = r.ints(0, cfg.vocab, (rows,), torch.int32)
    if c["prefill"]:
        packet = Packet(ids, _i32([0] * rows), _i32(list(range(rows))), table, rows, rows,
                        torch.tensor([rows - 1], device="cuda"), chunks=_i32([[0, rows, 0, 0]]),
                        max_q_len=rows)
    else:
        packet = Packet(ids, _i32(list(range(rows))), _i32([n - 1 for n in lens]), table, rows,
                        max(lens))
    logits = torch.empty(1 if c["prefill"] else rows, cfg.vocab, device="cuda")
    runner.logits(packet, logits)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        runner.logits(packet, logits)
    return dict(graph=graph, runner=runner, packet=packet, logits=logits)


_PREPARE = dict(linear=_prep_linear, attn_decode=_prep_attn_decode, attn_prefill=_prep_attn_prefill,
                gdn=_prep_gdn, moe=_prep_moe, model=_prep_model)


# ------------------------------------------------------------------------------- one pass
def run(s):
    return _RUN[s["kind"]](s, s["case"])


def _run_linear(s, c):
    return F.qgemm(s["a"], s["a_scale"], s["w"], s["w_scale"], c["fmt"], c["n"], out=s["out"])


def _run_attn_decode(s, c):
    rows = c["rows"]
    splits = min(F.attention_splits(c["ctx"], rows, c["kvh"]), max(512 // rows, 1))
    return F.attention(s["q"], None, s["req"], s["pos"], s["table"], s["k"], s["v"], s["ks"],
                       s["vs"], splits=splits, scratch=s["scratch"] if splits > 1 else None,
                       out=s["out"])


def _run_attn_prefill(s, c):
    if not F.attention_prefill(s["q"], s["gate"], s["chunks"], s["longest"], s["table"], s["k"],
                               s["v"], s["ks"], s["vs"], out=s["out"]):
        raise RuntimeError("no prefill kernel for this head size")
    return s["out"]


def _run_gdn(s, c):
    hk, hv, d, rows = c["hk"], c["hv"], c["d"], c["rows"]
    conv = (2 * hk + hv) * d
    F.gdn_conv(s["proj"], s["weight"], s["hist"], s["first"], s["slot"], s["pos"], s["segs"],
               c["segs"], rows, hk, hv, d, out=s["y"])
    F.gdn_scan(s["y"], s["ab"], s["a_log"], s["dt_bias"], s["segs"], c["segs"], s["slot"],
               s["pos"], hk, hv, d, s["state"], out=s["o"])
    F.gdn_gated_norm(s["o"], s["proj"][:, conv:], s["norm"], 1e-6, rows, hv, d, out=s["mix"])
    return dict(mix=s["mix"], state=s["state"], history=s["hist"])


def _run_moe(s, c):
    rows, h, f, e, sc = c["rows"], c["hidden"], c["ffn"], c["experts"], s["scratch"]
    F.act_prep(s["x"], None, s["norm"], s["signs"], q_out=s["q8"], scale_out=s["s8"],
               y_out=s["y16"])
    F.router_topk(s["y16"], s["router"], e, c["top_k"], rows=rows, ids=sc.ids, probs=sc.probs,
                  gate=sc.gate)
    F.moe_dispatch(sc.ids, s["q8"], s["s8"], e, sc, rows)
    total = rows * c["top_k"]
    F.qgemm_grouped(sc.q8, sc.scale, s["up"], s["up_s"], c["fmt"], 2 * f, sc.gate_up, sc, total)
    F.act_prep_limited(sc.gate_up, s["signs_mid"], sc.offsets[e:], swiglu=True, rows=total,
                       q_out=sc.q8_mid, scale_out=sc.scale_mid)
    F.qgemm_grouped(sc.q8_mid, sc.scale_mid, s["dn"], s["dn_s"], c["fmt"], h, sc.down, sc, total)
    shared = None
    if c["shared"]:
        up, dn = s["sh_up"], s["sh_dn"]
        F.qgemm(s["q8"], s["s8"], up.codes, up.scale, up.fmt, up.n, out=s["sh_gu"])
        F.act_prep(s["sh_gu"], None, None, s["sh_signs"], swiglu=True, q_out=s["sh_q"],
                   scale_out=s["sh_s"])
        shared = F.qgemm(s["sh_q"], s["sh_s"], dn.codes, dn.scale, dn.fmt, dn.n, out=s["sh_out"])
    F.moe_combine(sc.down, sc.slots, sc.probs, shared, sc.gate if c["shared"] else None, s["out"],
                  rows)
    return dict(out=s["out"], ids=sc.ids, probs=sc.probs)


def _run_model(s, c):
    s["graph"].replay()
    return dict(logits=s["logits"], hidden=s["runner"].final_hidden(c["rows"]))


_RUN = dict(linear=_run_linear, attn_decode=_run_attn_decode, attn_prefill=_run_attn_prefill,
            gdn=_run_gdn, moe=_run_moe, model=_run_model)


# ------------------------------------------------------------------------- work, tolerance
_BITS = {"q4": 0.5, "q2": 0.25, "w8": 1.0}


def _linear_work(m, n, k, fmt, out=2):
    return dict(bytes=m * k + 4 * m + n * k * _BITS[fmt] + 2 * n + out * m * n,
                flops=2.0 * m * n * k)


def _kv_row(kvh, d):
    return 2 * kvh * d + 4 * kvh * (d // 64)


def _add(*parts):
    return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))


def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        return _linear_work(c["m"], c["n"], c["k"], c["fmt"])
    if kind == "attn_decode":
        keys = sum(_lens(c["rows"], c["ctx"]))
        return dict(bytes=keys * _kv_row(c["kvh"], c["d"]) + 4.0 * c["rows"] * c["qh"] * c["d"],
                    flops=4.0 * keys * c["qh"] * c["d"])
    if kind == "attn_prefill":
        sizes = _chunk_rows(c)
        pairs = sum(n * c["past"] + n * (n + 1) // 2 for n in sizes)
        cells = sum(sizes) * c["qh"] * c["d"]
        return dict(bytes=sum(n + c["past"] for n in sizes) * _kv_row(c["kvh"], c["d"]) +
                    cells * (6.0 if c["gated"] else 4.0), flops=4.0 * pairs * c["qh"] * c["d"])
    if kind == "gdn":
        hk, hv, d, rows = c["hk"], c["hv"], c["d"], c["rows"]
        conv = (2 * hk + hv) * d
        return dict(bytes=rows * (2.0 * conv + 4 * hv * d + 8 * hv) +
                    c["segs"] * (8.0 * hv * d * d + 12 * conv),
                    flops=rows * (6.0 * hv * d * d + 8 * conv))
    if kind == "moe":
        rows, h, f, e, k = c["rows"], c["hidden"], c["ffn"], c["experts"], c["top_k"]
        hit = e * (1.0 - (1.0 - k / e) ** rows)              # experts that get a row
        parts = [dict(bytes=4.0 * rows * h + 2.0 * e * h + 8.0 * rows * k, flops=2.0 * rows * e * h),
                 dict(bytes=hit * 3 * f * h * _BITS[c["fmt"]], flops=6.0 * rows * k * f * h)]
        if c["shared"]:
            parts.append(dict(bytes=3.0 * c["shared"] * h * 0.5,
                              flops=6.0 * rows * c["shared"] * h))
        return _add(*parts)
    cfg, rows = _model_config(c), c["rows"]
    h, qd, n_out = cfg.hidden, cfg.q_heads * cfg.head_dim, 1 if c["prefill"] else rows
    weights = (qd + 2 * cfg.kv_dim) * h + h * qd + 3 * cfg.ffn * h
    if c["prefill"]:
        keys, pairs = rows, rows * (rows + 1) // 2
    else:
        keys = pairs = sum(_lens(rows, c["ctx"]))
    layer = dict(bytes=0.5 * weights + keys * _kv_row(cfg.kv_heads, cfg.head_dim),
                 flops=2.0 * rows * weights + 4.0 * pairs * qd)
    return _add(*[layer] * cfg.layers, _linear_work(n_out, cfg.vocab, h, "w8", 4),
                dict(bytes=(h + 4.0 * h) * rows, flops=0.0))


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 8e-4}           # exact integer sums, two FP32 scales, one FP16 rounding
    if kind == "attn_decode":
        return {"rel": 1e-3}           # FP32 throughout, one FP16 rounding
    if kind == "attn_prefill":
        return {"rel": 2e-3}           # FP16 keys, values and probabilities in the products
    if kind == "gdn":
        return {"rel": 1e-3}           # FP32 recurrence between FP16 inputs and outputs
    if kind == "moe":
        return {"rel": 5e-3, "differ": 2e-3}      # INT8 rows: a code at a tie may step
    # INT8 steps are about 3 % of a row's spread: a change of FP16 rounding moves some codes, and
    # through the four quantisations of a layer (and those of its keys and values, which only a
    # prefill computes) the difference grows towards that step
    return {"rel": 3e-2 if case["prefill"] else 2e-2}


# ------------------------------------------------------------------------------- 64 bits
_H128 = None


def _basis():
    """The 256 x 8 lattice basis of the E8P code, from its definition."""
    rows, digits = [], torch.cartesian_prod(*[torch.tensor([2, 6, 10])] * 8)
    rows.append(digits[(digits * digits).sum(1) <= 160])
    five = torch.combinations(torch.arange(8), 5)
    outer = torch.full((29, 8), 2)
    for i in range(29):
        outer[i, five[i * len(five) // 29]] = 6
    table = torch.cat([rows[0], outer])
    odd = (table.sum(1) // 4) % 2 == 1
    table[odd, 7] *= -1
    return table.to(torch.int16).cuda()


def _coords(code, table):
    """INT32 tensor of 16-bit codes [...] -> coordinates [..., 8]."""
    low = code & 0xFF
    par = low ^ (low >> 4)
    par = par ^ (par >> 2)
    par = (par ^ (par >> 1)) & 1
    flips = low ^ par
    bits = torch.tensor([0, 4, 1, 5, 2, 6, 3, 7], device=code.device, dtype=torch.int32)
    neg = ((flips[..., None] >> bits) & 1).to(torch.int16)
    return table[(code >> 8).long()] * (1 - 2 * neg) + (1 - 2 * par.to(torch.int16))[..., None]


def _weights64(w, fmt):
    """Integer weights [N, K] of one projection as FP64."""
    if fmt == "w8":
        return w.double()
    table, kb, n = _basis(), w.shape[0], w.shape[1]
    c = w.to(torch.int32)
    if fmt == "q4":
        v = 4 * _coords(c & 0xFFFF, table) + _coords((c >> 16) & 0xFFFF, table)
    else:
        v = _coords(c & 0xFFFF, table)
    return v.permute(1, 0, 2, 3).reshape(n, kb * 128).double()


def _f16(x):
    return x.to(torch.float16).double()


def _linear64(q, s, w, ws, fmt):
    return (q.double() @ _weights64(w, fmt).t()) * ws.double()[None] * s.double()[:, None]


def _rotate64(y, signs):
    global _H128
    if _H128 is None:
        h = torch.ones(1, 1, dtype=torch.float64, device="cuda")
        for _ in range(7):
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)])
        _H128 = h / math.sqrt(128.0)
    return ((y * signs.double()).reshape(y.shape[0], -1, 128) @ _H128).reshape(y.shape)


def _a8(y, signs):
    """Rotation and per-row INT8 codes of FP16-valued rows."""
    z = y if signs is None else _rotate64(y, signs)
    amax = z.abs().amax(1)
    scale = _f16(torch.where(amax > 0, (amax / 127.0).clamp(min=2.0 ** -24), torch.ones_like(amax)))
    return torch.clamp(torch.round(z / scale[:, None]), -127, 127), scale


def _norm64(x, w, eps=1e-6):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _swiglu64(gu):
    g, u = gu.chunk(2, dim=1)
    return _f16(g * torch.sigmoid(g) * u)


def _gather64(s, key, req, length):
    """Dequantised cache rows [length, KVH, D] of a request."""
    pages = s["table"][req, :(length + PAGE - 1) // PAGE].long()
    q, sc = s[key][pages], s[key + "s"][pages]
    q = q.reshape(-1, *q.shape[2:])[:length].double()
    sc = sc.reshape(-1, *sc.shape[2:])[:length].double()
    return (q.reshape(*q.shape[:2], -1, 64) * sc[..., None]).reshape(q.shape)


def _attend64(q, k, v, first):
    """Causal attention of rows at positions first.. over keys 0..: [Tq, QH * D]."""
    rep, out = q.shape[1] // k.shape[1], torch.empty_like(q, dtype=torch.float64)
    keys = torch.arange(k.shape[0], device=q.device)
    pos = first + torch.arange(q.shape[0], device=q.device)
    hide = keys[None] > pos[:, None]
    for h in range(q.shape[1]):
        sc = q[:, h].double() @ k[:, h // rep].t() / math.sqrt(q.shape[2])
        out[:, h] = torch.softmax(sc.masked_fill(hide, -math.inf), 1) @ v[:, h // rep]
    return out.reshape(q.shape[0], -1)


def exact(case, seed):
    if case["kind"] == "model":
        native.init()
        return _exact_model(case, _Rand(seed))
    return _EXACT[case["kind"]](prepare(case, seed), case)


def _exact_linear(s, c):
    return _linear64(s["a"], s["a_scale"], s["w"], s["w_scale"], c["fmt"])


def _exact_attn_decode(s, c):
    out = []
    for i, n in enumerate(_lens(c["rows"], c["ctx"])):
        out.append(_attend64(s["q"][i:i + 1], _gather64(s, "k", i, n), _gather64(s, "v", i, n),
                             n - 1))
    return torch.cat(out)


def _exact_attn_prefill(s, c):
    out, at = [], 0
    for i, n in enumerate(_chunk_rows(c)):
        kv = [_gather64(s, key, i, n + c["past"]) for key in "kv"]
        out.append(_attend64(s["q"][at:at + n], *kv, c["past"]))
        at += n
    out = torch.cat(out)
    if s["gate"] is not None:
        out = out * torch.sigmoid(s["gate"].double()).reshape(out.shape)
    return out


def _exact_gdn(s, c):
    hk, hv, d = c["hk"], c["hv"], c["d"]
    dk, conv, rep = hk * d, (2 * hk + hv) * d, hv // hk
    mix, states, hists, at = [], [], [], 0
    w = s["weight"].double()
    decay_all = torch.exp(-torch.exp(s["a_log"].double()) *
                          torch.nn.functional.softplus(s["ab"][:, :hv].double() +
                                                       s["dt_bias"].double(), threshold=50))
    beta_all = torch.sigmoid(s["ab"][:, hv:].double())
    for i, n in enumerate(_seg_rows(c)):
        fresh = int(s["pos"][at]) == 0
        x = s["proj"][at:at + n].double()
        full = torch.cat([s["hist"][i].double() * (0.0 if fresh else 1.0), x[:, :conv]])
        y = sum(full[j:j + n] * w[:, j] for j in range(4))
        y = _f16(y * torch.sigmoid(y))
        qk = y[:, :2 * dk].reshape(n, 2 * hk, d)
        qk = _f16(qk * torch.rsqrt((qk * qk).sum(-1, keepdim=True) + 1e-6))
        q = qk[:, :hk].repeat_interleave(rep, 1) / math.sqrt(d)
        k, v = qk[:, hk:].repeat_interleave(rep, 1), y[:, 2 * dk:].reshape(n, hv, d)
        st = s["state"][i].double() * (0.0 if fresh else 1.0)
        o = torch.empty(n, hv, d, dtype=torch.float64, device="cuda")
        for t in range(n):
            st = st * decay_all[at + t][:, None, None]
            delta = beta_all[at + t][:, None] * (v[t] - torch.bmm(k[t][:, None], st)[:, 0])
            st = torch.baddbmm(st, k[t][:, :, None], delta[:, None])
            o[t] = torch.bmm(q[t][:, None], st)[:, 0]
        z = x[:, conv:].reshape(n, hv, d)
        mix.append((_norm64(o, s["norm"]) * z * torch.sigmoid(z)).reshape(n, -1))
        states.append(st)
        hists.append(full[-3:])
        at += n
    return dict(mix=torch.cat(mix), state=torch.stack(states), history=torch.stack(hists))


def _exact_moe(s, c):
    e, k, rows = c["experts"], c["top_k"], c["rows"]
    y = _f16(_norm64(s["x"].double(), s["norm"]))
    q, sc = _a8(y, s["signs"])
    logits = y @ s["router"].double().t()
    prob, ids = torch.softmax(logits[:, :e], 1).topk(k, 1)
    prob = prob / prob.sum(1, keepdim=True)
    out = torch.zeros(rows, c["hidden"], dtype=torch.float64, device="cuda")
    for ex in ids.unique().tolist():
        row, slot = (ids == ex).nonzero(as_tuple=True)
        gu = _f16(_linear64(q[row], sc[row], s["up"][ex], s["up_s"][ex], c["fmt"]))
        qm, sm = _a8(_swiglu64(gu), s["signs_mid"])
        dn = _f16(_linear64(qm, sm, s["dn"][ex], s["dn_s"][ex], c["fmt"]))
        out.index_add_(0, row, dn * prob[row, slot][:, None])
    if c["shared"]:
        gu = _f16(_linear64(q, sc, s["sh_up"].codes, s["sh_up"].scale, "q4"))
        qm, sm = _a8(_swiglu64(gu), s["sh_signs"])
        dn = _f16(_linear64(qm, sm, s["sh_dn"].codes, s["sh_dn"].scale, "q4"))
        out += torch.sigmoid(logits[:, e])[:, None] * dn
    return dict(out=out, ids=None, probs=prob)


def _rope64(x, w, pos, theta):
    half = x.shape[-1] // 2
    y = _f16(_norm64(x, w))
    inv = theta ** (-torch.arange(half, dtype=torch.float64, device="cuda") / half)
    ang = pos.double()[:, None] * inv
    co, si = ang.cos()[:, None], ang.sin()[:, None]
    a, b = y[..., :half], y[..., half:]
    return _f16(torch.cat([a * co - b * si, b * co + a * si], -1))


def _kv8(x):
    g = x.reshape(*x.shape[:-1], -1, 64)
    scale = _f16((g.abs().amax(-1) / 127.0).clamp(min=2.0 ** -24))
    return (torch.clamp(torch.round(g / scale[..., None]), -127, 127) *
            scale[..., None]).reshape(x.shape)


def _exact_model(c, r):
    """The two-layer decoder: the same draws as ``_prep_model`` makes, in the same order."""
    cfg, rows = _model_config(c), c["rows"]
    w = _model_weights(cfg, r)
    lens = [rows] if c["prefill"] else _lens(rows, c["ctx"])
    pools = [_paged(r, lens, cfg.kv_heads, cfg.head_dim) for _ in range(cfg.layers)]
    ids = r.ints(0, cfg.vocab, (rows,), torch.int32).long()
    pos = torch.arange(rows, device="cuda") if c["prefill"] else _i32([n - 1 for n in lens])
    qd, kvd, d = cfg.q_heads * cfg.head_dim, cfg.kv_dim, cfg.head_dim
    lin = lambda x, p: _f16(_linear64(*_a8(x, p.signs), p.codes, p.scale, p.fmt))
    resid = _f16(w.embed_q[ids].double() * w.embed_s[ids].double()[:, None])
    for lw, pool in zip(w.layers, pools):
        pool["table"] = pools[0]["table"]
        qkv = lin(_f16(_norm64(resid, lw.in_norm, cfg.eps)), lw.qkv)
        q = _rope64(qkv[:, :qd].reshape(rows, -1, d), lw.q_norm, pos, cfg.rope_theta)
        k = _kv8(_rope64(qkv[:, qd:qd + kvd].reshape(rows, -1, d), lw.k_norm, pos, cfg.rope_theta))
        v = _kv8(qkv[:, qd + kvd:].reshape(rows, -1, d))
        if c["prefill"]:
            att = _attend64(q, k, v, 0)
        else:
            att = []
            for i, n in enumerate(lens):
                ki = torch.cat([_gather64(pool, "k", i, n)[:n - 1], k[i:i + 1]])
                vi = torch.cat([_gather64(pool, "v", i, n)[:n - 1], v[i:i + 1]])
                att.append(_attend64(q[i:i + 1], ki, vi, n - 1))
            att = torch.cat(att)
        resid = resid + lin(_f16(att), lw.o)
        gu = lin(_f16(_norm64(resid, lw.post_norm, cfg.eps)), lw.gate_up)
        resid = resid + lin(_swiglu64(gu), lw.down)
    y = _f16(_norm64(resid, w.final_norm, cfg.eps))
    sel = y[-1:] if c["prefill"] else y
    return dict(logits=_linear64(*_a8(sel, None), w.head.codes, w.head.scale, "w8"), hidden=resid)


_EXACT = dict(linear=_exact_linear, attn_decode=_exact_attn_decode,
              attn_prefill=_exact_attn_prefill, gdn=_exact_gdn, moe=_exact_moe)
