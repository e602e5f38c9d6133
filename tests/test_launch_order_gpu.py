"""Kernels that start before the ones in front of them have ended (launch_early): every mixer of a
layer in a loop over its own buffers, each round reading what the round before wrote and overwriting
what it read, without a wait and in a graph, against the same calls with a wait after each."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROUNDS = 6


@pytest.fixture(scope="module")
def dev(cuda):
    from orinfer_b200.ops import native
    native.init()
    return cuda


def _weight(fmt, n, k, g, dev, lead=()):
    """Random codes with row scales that keep outputs near one."""
    if fmt == "w8":
        w = torch.randint(-127, 128, (*lead, n, k), generator=g, dtype=torch.int8)
        unit = 73.0
    else:
        w = torch.randint(-2 ** 31, 2 ** 31, (*lead, k // 128, n, 16), generator=g,
                          dtype=torch.int64).to(torch.int32)
        unit = 13.0
    s = torch.full((*lead, n), 1.0 / (unit * k ** 0.5), dtype=torch.float16)
    return w.to(dev), s.to(dev)


def _same_without_waits(calls, live, first):
    """`calls(round)` yields after each call; `live` tensors start as `first`."""
    def chain(wait):
        for t, t0 in zip(live, first):
            t.copy_(t0)
        for i in range(ROUNDS):
            for _ in calls(i):
                if wait:
                    torch.cuda.synchronize()

    chain(True)
    torch.cuda.synchronize()
    want = [t.clone() for t in live]
    assert all(bool(t.isfinite().all()) for t in want if t.is_floating_point())
    assert any(not torch.equal(t, t0) for t, t0 in zip(want, first))
    for _ in range(10):
        chain(False)
        assert all(torch.equal(t, w) for t, w in zip(live, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(False)
    for _ in range(10):
        graph.replay()
        assert all(torch.equal(t, w) for t, w in zip(live, want))


@pytest.mark.parametrize("qh,kvh,d", [(8, 2, 64), (16, 8, 128), (8, 1, 256)])
@pytest.mark.parametrize("form", ["rows", "split", "prefill"])
def test_attention_behind_its_cache_writes(dev, qh, kvh, d, form):
    """A round writes the slots behind those of the round before, whose scales lie in cache lines
    that the attention of that round has read."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(d + qh)
    n = 150 if form == "prefill" else 24
    past = 120                                           # the second round crosses a page
    width = (qh + 2 * kvh) * d
    step = n if form == "prefill" else 1
    pages = (past + ROUNDS * step + 127) // 128
    reqs = 1 if form == "prefill" else n
    table = (torch.arange(reqs * pages, dtype=torch.int32) + 1).reshape(reqs, pages).to(dev)
    w, ws = _weight("w8", width, qh * d, g, dev)
    total = reqs * pages + 1
    cache = lambda: torch.randint(-127, 128, (total, 128, kvh, d), generator=g,
                                  dtype=torch.int8).to(dev)
    scale = lambda: (torch.rand(total, 128, kvh, d // 64, generator=g) * 0.01 + 0.01).half().to(dev)
    first = [torch.randn(n, width, generator=g).half().to(dev), cache(), cache(), scale(), scale()]
    live = [torch.empty_like(t) for t in first]
    qkv, kc, vc, ks, vs = live
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    req = i32([0] * n if form == "prefill" else list(range(n)))
    pos = [i32([past + i * step + (r if form == "prefill" else 0) for r in range(n)])
           for i in range(ROUNDS)]
    chunk = [i32([[0, n, past + i * n, 0]]) for i in range(ROUNDS)]
    cos = torch.empty(n, d // 2, device=dev)
    sin = torch.empty_like(cos)
    q, out = (torch.empty(n, qh * d, dtype=torch.float16, device=dev) for _ in range(2))
    q = q.view(n, qh, d)
    q8, s8 = torch.empty(n, qh * d, dtype=torch.int8, device=dev), torch.empty(n, device=dev)
    splits = 3 if form == "split" else 1
    scratch = torch.empty(n * qh * splits * (d + 2), device=dev)

    def calls(i):
        yield F.rope_table(pos[i], d, 1e6, cos, sin)
        yield F.qk_rope_kv(qkv, None, None, cos, sin, req, pos[i], table, kc, vc, ks, vs, qh=qh,
                           kvh=kvh, head_dim=d, q_out=q)
        if form == "prefill":
            yield F.attention_prefill(q, None, chunk[i], n, table, kc, vc, ks, vs, out=out)
        else:
            yield F.attention(q, None, req, pos[i], table, kc, vc, ks, vs, splits=splits,
                              scratch=scratch if splits > 1 else None, out=out)
        yield F.act_prep(out, None, None, None, q_out=q8, scale_out=s8)
        yield F.qgemm(q8, s8, w, ws, "w8", width, out=qkv)

    _same_without_waits(calls, live, first)


@pytest.mark.parametrize("fmt", ["w8", "q4"])
@pytest.mark.parametrize("rows,experts,top_k,h,ffn", [
    (5, 8, 2, 512, 256), (40, 16, 4, 512, 256), (300, 8, 2, 512, 256), (600, 48, 8, 2048, 256)])
def test_experts_behind_their_router(dev, fmt, rows, experts, top_k, h, ffn):
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(rows + experts)
    up, up_s = _weight(fmt, 2 * ffn, h, g, dev, (experts,))
    dn, dn_s = _weight(fmt, h, ffn, g, dev, (experts,))
    router = (torch.randn(experts, h, generator=g) * 0.05).half().to(dev)
    norm = torch.ones(h, dtype=torch.float16, device=dev)
    signs = torch.ones(ffn, dtype=torch.int8, device=dev)
    sc = F.MoeScratch(rows, top_k, experts, h, ffn, dev)
    first = [torch.randn(rows, h, generator=g).half().to(dev)]
    x = torch.empty_like(first[0])
    y16, q8 = torch.empty_like(x), torch.empty(rows, h, dtype=torch.int8, device=dev)
    s8, total = torch.empty(rows, device=dev), rows * top_k

    def calls(_):
        yield F.act_prep(x, None, norm, None, q_out=q8, scale_out=s8, y_out=y16)
        yield F.router_topk(y16, router, experts, top_k, rows=rows, ids=sc.ids, probs=sc.probs)
        yield F.moe_dispatch(sc.ids, q8, s8, experts, sc, rows)
        yield F.qgemm_grouped(sc.q8, sc.scale, up, up_s, fmt, 2 * ffn, sc.gate_up, sc, total)
        yield F.act_prep_limited(sc.gate_up, signs, sc.offsets[experts:], swiglu=True, rows=total,
                                 q_out=sc.q8_mid, scale_out=sc.scale_mid)
        yield F.qgemm_grouped(sc.q8_mid, sc.scale_mid, dn, dn_s, fmt, h, sc.down, sc, total)
        yield F.moe_combine(sc.down, sc.slots, sc.probs, None, None, x, rows)

    _same_without_waits(calls, [x], first)


@pytest.mark.parametrize("segs,rows,hk,hv,d", [(24, 24, 2, 4, 128), (1, 90, 2, 4, 128),
                                               (3, 36, 4, 4, 64)])
def test_recurrent_mixer_behind_its_projection(dev, segs, rows, hk, hv, d):
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(rows + d)
    conv, width = (2 * hk + hv) * d, (2 * hk + 2 * hv) * d
    w, ws = _weight("q4", width, hv * d, g, dev)
    per = rows // segs
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    seg = i32([[s * per, per, 0, 0] for s in range(segs)])
    row_first = i32([r // per * per for r in range(rows)])
    slot = i32([r // per for r in range(rows)])
    pos = i32([200 + r % per for r in range(rows)])
    f16 = lambda *s: torch.randn(*s, generator=g).half().to(dev)
    weight, norm = f16(conv, 4) * 0.3, torch.ones(d, dtype=torch.float16, device=dev)
    ab = torch.randn(rows, 2 * hv, generator=g).to(dev)
    a_log, dt = torch.randn(hv, generator=g).to(dev) - 1, torch.randn(hv, generator=g).to(dev) - 2
    first = [f16(rows, width), f16(segs, 3, conv),
             (torch.randn(segs, hv, d, d, generator=g) * 0.05).to(dev)]
    live = [torch.empty_like(t) for t in first]
    proj, hist, state = live
    y = torch.empty(rows, conv, dtype=torch.float16, device=dev)
    o, mix = torch.empty(rows, hv, d, device=dev), y.new_empty(rows, hv * d)
    q8, s8 = torch.empty(rows, hv * d, dtype=torch.int8, device=dev), torch.empty(rows, device=dev)

    def calls(_):
        yield F.gdn_conv(proj, weight, hist, row_first, slot, pos, seg, segs, rows, hk, hv, d,
                         out=y)
        yield F.gdn_scan(y, ab, a_log, dt, seg, segs, slot, pos, hk, hv, d, state, out=o)
        yield F.gdn_gated_norm(o, proj[:, conv:], norm, 1e-6, rows, hv, d, out=mix)
        yield F.act_prep(mix, None, None, None, q_out=q8, scale_out=s8)
        yield F.qgemm(q8, s8, w, ws, "q4", width, out=proj)

    _same_without_waits(calls, live, first)
