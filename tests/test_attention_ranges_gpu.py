"""Attention kernels at the edges of their tiles and ranges, against 64-bit statements."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(cuda):
    from orinfer_b200.ops import native
    native.init()
    return cuda


def _unaligned(t):
    """A contiguous copy whose address is two bytes past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)
    out = flat[1:1 + t.numel()].view(t.shape)
    out.copy_(t)
    return out


def _attention64(q, k, v, ks, vs, gate=None):
    """q [QH, D] against every row of k, v [T, KVH, D] with group scales [T, KVH, D / 64]."""
    qh, d = q.shape
    kk = (k.double().reshape(*k.shape[:2], -1, 64) * ks.double()[..., None]).reshape(k.shape)
    vv = (v.double().reshape(*v.shape[:2], -1, 64) * vs.double()[..., None]).reshape(v.shape)
    rep = qh // k.shape[1]
    s = torch.einsum("hd,thd->ht", q.double(), kk.repeat_interleave(rep, 1)) / math.sqrt(d)
    o = torch.einsum("ht,thd->hd", torch.softmax(s, 1), vv.repeat_interleave(rep, 1))
    return o if gate is None else o * torch.sigmoid(gate.double())


# contexts around the 16- / 32-key blocks, the pages and the splits
@pytest.mark.parametrize("qh,kvh,d", [(2, 2, 64), (4, 2, 64), (16, 2, 64), (3, 3, 128), (4, 2, 128),
                                      (8, 2, 128), (10, 2, 128), (8, 1, 128), (2, 1, 256),
                                      (8, 1, 256), (4, 1, 256)])
@pytest.mark.parametrize("splits,wide", [(1, True), (5, True), (3, False)])
def test_attention_rows_at_block_edges(dev, qh, kvh, d, splits, wide):
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(qh * 1000 + d + splits)
    lens = [1, 2, 15, 16, 17, 31, 33, 127, 128, 129, 160, 257, 700]
    pages = sum((n + 127) // 128 for n in lens) + 1
    table = torch.zeros(len(lens), 6, dtype=torch.int32)
    at = 1
    for i, n in enumerate(lens):
        for j in range((n + 127) // 128):
            table[i, j] = at
            at += 1
    kc = torch.randint(-127, 128, (pages, 128, kvh, d), generator=g, dtype=torch.int8).to(dev)
    vc = torch.randint(-127, 128, (pages, 128, kvh, d), generator=g, dtype=torch.int8).to(dev)
    # value scales over many binades: the weights are rescaled as larger ones turn up
    ks = (torch.rand(pages, 128, kvh, d // 64, generator=g) * 0.02 + 1e-3).half().to(dev)
    vs = torch.exp2(torch.rand(pages, 128, kvh, d // 64, generator=g) * 18 - 14).half().to(dev)
    for i, n in enumerate(lens):                    # slots never written hold anything
        last = int(table[i, (n - 1) // 128])
        ks[last, (n - 1) % 128 + 1:] = float("nan")
        vs[last, (n - 1) % 128 + 1:] = float("inf")
    q = torch.randn(len(lens), qh, d, generator=g).half().to(dev)
    gate = torch.randn(len(lens), qh, d, generator=g).half().to(dev) if d == 256 else None
    if not wide:
        q, ks, vs = _unaligned(q), _unaligned(ks), _unaligned(vs)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    out = F.attention(q, gate, t(list(range(len(lens)))), t([n - 1 for n in lens]), table.to(dev),
                      kc, vc, ks, vs, splits=splits)
    for i, n in enumerate(lens):
        pg = table[i, :(n + 127) // 128].long().to(dev)
        rows = lambda c: c[pg].reshape(-1, *c.shape[2:])[:n]
        ref = _attention64(q[i], rows(kc), rows(vc), rows(ks), rows(vs),
                           None if gate is None else gate[i]).reshape(-1)
        # one FP16 rounding (2^-11 of the value) on top of FP32 sums over terms that may cancel:
        # a few 2^-22 of the largest value
        lim = ref.abs() * 2.0 ** -11 + 2.0 ** -18 * ref.abs().max() + 2.0 ** -25
        assert bool(((out[i].double() - ref).abs() <= lim).all()), (n, float((out[i] - ref).abs().max()))


def _short_rows(dev, rows, qh, kvh, d, lens):
    """One request per length, each attended by rows / len(lens) equal query rows."""
    g = torch.Generator().manual_seed(rows + d)
    n = len(lens)
    table = torch.arange(1, 2 * n + 1, dtype=torch.int32).view(n, 2).to(dev)
    shape = (2 * n + 1, 128, kvh)
    kc = torch.randint(-127, 128, (*shape, d), generator=g, dtype=torch.int8).to(dev)
    vc = torch.randint(-127, 128, (*shape, d), generator=g, dtype=torch.int8).to(dev)
    ks = (torch.rand(*shape, d // 64, generator=g) * 0.02 + 1e-3).half().to(dev)
    vs = (torch.rand(*shape, d // 64, generator=g) * 0.02 + 1e-3).half().to(dev)
    q = torch.randn(n, qh, d, generator=g).half().to(dev)
    req = torch.arange(rows, device=dev, dtype=torch.int32) % n
    pos = torch.tensor(lens, dtype=torch.int32, device=dev)[req.long()] - 1
    return q, req, pos, table, kc, vc, ks, vs


# launches of less than one to more than four waves of CTAs, lengths around the limits of each;
# the last warps of a CTA have no head where the KV heads are no multiple of four
@pytest.mark.parametrize("qh,kvh,d", [(8, 8, 64), (7, 7, 64), (5, 5, 128), (40, 8, 128), (8, 4, 256)])
@pytest.mark.parametrize("waves", [0.9, 1.1, 2.1, 3.5, 4.2])
@pytest.mark.parametrize("wide", [True, False])
def test_attention_rows_of_short_contexts(dev, qh, kvh, d, waves, wide):
    from orinfer_b200.ops import functional as F
    lens = [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65, 96, 97, 127, 128, 129, 160, 256]
    rows = int(waves * 148 * {64: 4, 128: 3, 256: 2}[d] / kvh)
    q, req, pos, table, kc, vc, ks, vs = _short_rows(dev, rows, qh, kvh, d, lens)
    gate = torch.randn_like(q.float()).half() if d == 256 else None
    for i, n in enumerate(lens):                    # slots never written hold anything
        if n % 128:
            page = table[i, (n - 1) // 128].long()
            ks[page, (n - 1) % 128 + 1:] = float("nan")
            vs[page, (n - 1) % 128 + 1:] = float("inf")
    if not wide:
        ks, vs = _unaligned(ks), _unaligned(vs)
    out = F.attention(q[req.long()].contiguous(), None if gate is None else gate[req.long()], req,
                      pos, table, kc, vc, ks, vs, splits=1).view(rows, qh * d)
    for i, n in enumerate(lens[:rows]):
        pick = lambda c: c[table[i].long()].reshape(-1, *c.shape[2:])[:n]
        ref = _attention64(q[i], pick(kc), pick(vc), pick(ks), pick(vs),
                           None if gate is None else gate[i]).reshape(-1)
        # as above: one FP16 rounding and FP32 sums over terms that may cancel
        lim = ref.abs() * 2.0 ** -11 + 2.0 ** -18 * ref.abs().max() + 2.0 ** -25
        got = out[i::len(lens)].double()
        assert bool(((got - ref).abs() <= lim).all()), n


def test_attention_rows_fill_the_chip_with_short_contexts(dev):
    """A warp without a block costs as much as one with: contexts of one block are clearly quicker
    than contexts of four."""
    from orinfer_b200.ops import functional as F
    us = []
    for n in (30, 110):
        q, req, pos, table, kc, vc, ks, vs = _short_rows(dev, 512, 16, 16, 128, [n] * 512)
        times = []
        for _ in range(15):
            b, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            b.record()
            for _ in range(10):
                F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=1)
            e.record()
            e.synchronize()
            times.append(b.elapsed_time(e) * 100)
        us.append(sorted(times)[7])
    assert us[0] < 0.75 * us[1], us                 # about 0.6; 0.83 with a CTA to each head


@pytest.mark.parametrize("qh,kvh,d,gated", [(2, 2, 64, False), (8, 1, 64, False), (3, 3, 128, False),
                                            (8, 2, 128, True), (10, 2, 128, False),
                                            (16, 1, 128, False), (8, 1, 256, True),
                                            (4, 4, 256, False)])
@pytest.mark.parametrize("spec", [[(1, 0)], [(63, 0), (65, 64), (1, 200)], [(129, 127), (257, 5)],
                                  [(400, 1000)], [(5200, 0), (1, 70)]])
def test_attention_prefill_at_tile_edges(dev, qh, kvh, d, gated, spec):
    """Chunks that end inside the first or second query tile of a CTA, one or two tiles per CTA,
    pages cut by the first position, against the 64-bit statement."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(qh * d + spec[0][0])
    width = max((n + p + 127) // 128 for n, p in spec)
    need = sum((n + p + 127) // 128 for n, p in spec)
    table = torch.zeros(len(spec), width, dtype=torch.int32)
    at = 1
    for i, (n, p) in enumerate(spec):
        for j in range((n + p + 127) // 128):
            table[i, j] = at
            at += 1
    kc = torch.randint(-127, 128, (need + 1, 128, kvh, d), generator=g, dtype=torch.int8).to(dev)
    vc = torch.randint(-127, 128, (need + 1, 128, kvh, d), generator=g, dtype=torch.int8).to(dev)
    ks = (torch.rand(need + 1, 128, kvh, d // 64, generator=g) * 0.02 + 1e-3).half().to(dev)
    vs = (torch.rand(need + 1, 128, kvh, d // 64, generator=g) * 0.02 + 1e-3).half().to(dev)
    for i, (n, p) in enumerate(spec):               # slots never written hold anything
        last, used = int(table[i, (n + p - 1) // 128]), (n + p - 1) % 128 + 1
        ks[last, used:] = float("nan")
        vs[last, used:] = float("inf")
    rows = sum(n for n, _ in spec)
    q = torch.randn(rows, qh, d, generator=g).half().to(dev)
    gate = torch.randn(rows, qh, d, generator=g).half().to(dev) if gated else None
    chunks, first = [], 0
    for i, (n, p) in enumerate(spec):
        chunks.append([first, n, p, i])
        first += n
    out = torch.full((rows, qh * d), float("nan"), dtype=torch.float16, device=dev)
    assert F.attention_prefill(q, gate, torch.tensor(chunks, dtype=torch.int32, device=dev),
                               max(n for n, _ in spec), table.to(dev), kc, vc, ks, vs, out=out)
    for i, (n, p) in enumerate(spec):
        pg = table[i, :(n + p + 127) // 128].long().to(dev)
        flat = lambda c: c[pg].reshape(-1, *c.shape[2:])
        for r in sorted({0, 1, n // 2, n - 2, n - 1} & set(range(n))):
            seen = p + r + 1
            ref = _attention64(q[chunks[i][0] + r], flat(kc)[:seen], flat(vc)[:seen],
                               flat(ks)[:seen], flat(vs)[:seen],
                               None if gate is None else gate[chunks[i][0] + r]).reshape(-1)
            got = out[chunks[i][0] + r].double()
            # FP16 keys, values and weights (2^-11 each, scores up to about 20): 2^-8 of the
            # largest value
            assert float((got - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max()), (n, p, r)


@pytest.mark.parametrize("d,kvh,qh", [(64, 2, 4), (128, 1, 5), (256, 1, 8)])
@pytest.mark.parametrize("rows", [40, 300])
def test_attention_prefill_largest_weight_is_exact(dev, d, kvh, qh, rows):
    """A late key that dominates by up to 2^8, the only one with a value: its weight is the row's
    largest, 1 in FP16 whatever the earlier pages held, so only the output is rounded."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(d + rows)
    past, peak = 300, 270
    pages = (rows + past + 127) // 128
    kc = torch.zeros(pages + 1, 128, kvh, d, dtype=torch.int8)
    vc = torch.zeros_like(kc)
    table = torch.arange(1, pages + 1, dtype=torch.int32)[None]
    kc[1:, :, :, 0] = torch.randint(0, 60, (pages, 128, kvh), generator=g, dtype=torch.int8)
    kc[1 + peak // 128, peak % 128, :, 0] = 127
    vc[1 + peak // 128, peak % 128] = torch.randint(20, 127, (kvh, d), generator=g, dtype=torch.int8)
    scale = lambda v: torch.full((pages + 1, 128, kvh, d // 64), v, dtype=torch.float16, device=dev)
    q = torch.zeros(rows, qh, d)
    # the peak is above the others by 2^0.5 .. 2^8 of the softmax weight
    q[:, :, 0] = torch.linspace(0.5, 8, rows * qh).reshape(rows, qh) * math.sqrt(d) * math.log(2) * 127 / 67
    q = q.half().to(dev)
    kc, vc, ks, vs = kc.to(dev), vc.to(dev), scale(1 / 128), scale(1 / 64)
    out = torch.empty(rows, qh * d, dtype=torch.float16, device=dev)
    chunk = torch.tensor([[0, rows, past, 0]], dtype=torch.int32, device=dev)
    assert F.attention_prefill(q, None, chunk, rows, table.to(dev), kc, vc, ks, vs, out=out)
    flat = lambda c: c[1:].reshape(-1, *c.shape[2:])
    for r in range(rows):
        n = past + r + 1
        ref = _attention64(q[r], flat(kc)[:n], flat(vc)[:n], flat(ks)[:n], flat(vs)[:n]).reshape(-1)
        # one FP16 rounding of the output (2^-11); scores of up to 2^4 in FP32, a sum of up to 600
        # FP32 weights and their exponentials: below 2^-17
        assert bool(((out[r].double() - ref).abs() <= ref.abs() * (2.0 ** -11 + 2.0 ** -17)).all()), r


@pytest.mark.parametrize("d,kvh,qh", [(64, 2, 4), (128, 1, 5), (256, 1, 8)])
@pytest.mark.parametrize("rows", [128, 5200])
def test_attention_prefill_adds_weights_in_the_order_of_keys(dev, d, kvh, qh, rows):
    """Two keys of weight 1 at the start of a step and about 2^-26 for the others, which vanish one
    pair after the other in a sum of 2 (ulp 2^-22) and in FP16 weights: the sum is exactly 2 and the
    output the FP16 tie (1 + 1 + 3 * 2^-10) / 2, to even upwards.  Sums of their own over the later
    keys would reach 2^-21 and more, and tip the tie downwards."""
    from orinfer_b200.ops import functional as F
    step = 64 if d == 256 else 128                             # keys per step
    pages = (rows + 127) // 128
    table = torch.arange(1, pages + 1, dtype=torch.int32, device=dev)[None]
    kc = torch.zeros(pages + 1, 128, kvh, d, dtype=torch.int8, device=dev)
    vc = torch.ones_like(kc)
    ks = torch.full((pages + 1, 128, kvh, d // 64), 2.0, dtype=torch.float16, device=dev)
    vs = torch.ones_like(ks)
    # scores are q . k / sqrt(d), weights their exponentials: q . k of -26 * ln 2 * sqrt(d)
    kc[:, :, :, 0] = -round(26 * math.log(2) * math.sqrt(d) / (4 if d == 256 else 2))
    kc[1, :2, :, 0] = 0
    vs[1, 0], vs[1, 1] = 1 + 2.0 ** -10, 1 + 2.0 ** -9
    q = torch.zeros(rows, qh, d, dtype=torch.float16, device=dev)
    q[:, :, 0] = 2 if d == 256 else 1
    out = torch.empty(rows, qh * d, dtype=torch.float16, device=dev)
    chunk = torch.tensor([[0, rows, 0, 0]], dtype=torch.int32, device=dev)
    assert F.attention_prefill(q, None, chunk, rows, table, kc, vc, ks, vs, out=out)
    assert bool((out[1:step] == 1 + 2.0 ** -9).all())


def _walk(dev, n, qh, kvh, d, seed, grow=0.0):
    """One request of n keys whose scores and value scales grow along the context."""
    g = torch.Generator().manual_seed(seed)
    pages = (n + 127) // 128
    table = (torch.randperm(pages, generator=g) + 1).to(torch.int32)[None].to(dev)
    shape = (pages + 1, 128, kvh)
    kc = torch.randint(-127, 128, (*shape, d), generator=g, dtype=torch.int8).to(dev)
    vc = torch.randint(-127, 128, (*shape, d), generator=g, dtype=torch.int8).to(dev)
    up = torch.zeros(shape[:2])
    up[table[0].long().cpu()] = (torch.arange(pages * 128).view(pages, 128) / n * grow)
    ks = ((torch.rand(*shape, d // 64, generator=g) * 0.02 + 1e-3) * (1 + up)[..., None, None])
    vs = torch.rand(*shape, d // 64, generator=g) * 0.02 * torch.exp2(up)[..., None, None]
    q = torch.randn(1, qh, d, generator=g).half().to(dev)
    one = torch.zeros(1, dtype=torch.int32, device=dev)
    return q, one, one + n - 1, table, kc, vc, ks.half().to(dev), vs.half().to(dev)


def _in_digits(qh, kvh, d, table, splits):
    from orinfer_b200.ops import native
    return bool(native.lib().orinfer_attention_in_digits(qh, kvh, d, table.shape[1], splits))


# contexts of a warp around 32 blocks, where it fetches the next page ids, references that move with
# the context, an odd and an even number of heads
@pytest.mark.parametrize("qh,kvh,d", [(4, 1, 128), (6, 3, 64), (4, 2, 64), (3, 3, 128), (8, 1, 128)])
@pytest.mark.parametrize("n", [3713, 3968, 4096, 4129, 8257, 12400])
@pytest.mark.parametrize("grow,splits", [(0.0, 1), (6.0, 1), (6.0, 5)])
def test_attention_rows_walk_many_pages(dev, qh, kvh, d, n, grow, splits):
    from orinfer_b200.ops import functional as F
    q, req, pos, table, kc, vc, ks, vs = _walk(dev, n, qh, kvh, d, n + qh, grow)
    assert _in_digits(qh, kvh, d, table, splits) == (qh // kvh <= 4)
    out = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=splits).view(-1)
    pick = lambda c: c[table[0].long()].reshape(-1, *c.shape[2:])[:n]
    ref = _attention64(q[0], pick(kc), pick(vc), pick(ks), pick(vs)).reshape(-1)
    lim = ref.abs() * 2.0 ** -11 + 2.0 ** -18 * ref.abs().max() + 2.0 ** -25
    assert bool(((out.double() - ref).abs() <= lim).all())


# value scales of one group far below those of the other, a key of huge value scale whose weight is
# nil or not, and both against the group's own values: each keeps the bits of FP32 products
@pytest.mark.parametrize("qh,kvh,n,splits", [(4, 1, 900, 1), (8, 2, 4129, 1), (4, 2, 3000, 3)])
@pytest.mark.parametrize("what", ["group", "nil", "heavy"])
@pytest.mark.parametrize("k", [6, 10, 14])
def test_attention_rows_keep_the_bits_of_small_value_scales(dev, qh, kvh, n, splits, what, k):
    from orinfer_b200.ops import functional as F
    d, rep = 128, qh // kvh
    q, req, pos, table, kc, vc, ks, vs = _walk(dev, n, qh, kvh, d, n + k)
    assert _in_digits(qh, kvh, d, table, splits)
    vs = (vs.float() * 2.0 ** 10).half()                  # (2^-14 of it is a normal FP16 number)
    if what == "group":
        vs[..., 1] = (vs[..., 1].float() * 2.0 ** -k).half()
    else:
        vs = (vs.float() * 2.0 ** -k).half()
        page, slot = int(table[0, 2]), 77                 # key 333
        vs[page, slot] = 16.0
        if what == "nil":                                 # far below every head's maximum
            q = q.view(kvh, rep, d)[:, :1].expand(kvh, rep, d).reshape(1, qh, d).contiguous()
            kc[page, slot] = -(q[0, ::rep].sign() * 127).to(torch.int8)
            ks[page, slot] = 0.5
    out = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=splits).view(qh, -1, 64)
    pick = lambda c: c[table[0].long()].reshape(-1, *c.shape[2:])[:n]
    ref = _attention64(q[0], pick(kc), pick(vc), pick(ks), pick(vs)).reshape(qh, -1, 64)
    # one FP16 rounding, and FP32 sums of terms that may cancel: a few 2^-22 of the group's largest;
    # outputs below the smallest normal FP16 number are rounded at 2^-25
    lim = ref.abs() * 2.0 ** -11 + 2.0 ** -20 * ref.abs().amax(-1, keepdim=True) + 2.0 ** -25
    assert bool(((out.double() - ref).abs() <= lim).all())


# scores that leap by many binades from block to block, up or down, over tiny value scales: references
# move, units follow as far as they go
@pytest.mark.parametrize("leap", [5, 20, 70, 130])
@pytest.mark.parametrize("up", [True, False])
@pytest.mark.parametrize("d", [64, 128])
def test_attention_rows_of_scores_that_leap(dev, leap, up, d):
    from orinfer_b200.ops import functional as F
    n, qh = 128 * 6, 4
    q, req, pos, table, kc, vc, ks, vs = _walk(dev, n, qh, 1, d, leap)
    assert _in_digits(qh, 1, d, table, 1)
    step = torch.arange(n, device=dev) // 128               # a block of each warp per step
    kc[table[0].long()] = torch.randint(-9, 10, (6, 128, 1, d), device=dev, dtype=torch.int8)
    flat = (table[0].long()[:, None] * 128 + torch.arange(128, device=dev)).flatten()
    kc.view(-1, 1, d)[flat, :, 0] = (20 * (step if up else 5 - step))[:, None].to(torch.int8)
    ks[:] = 1 / 64
    q[..., 0] = leap * math.log(2) * math.sqrt(d) * 64 / 20
    vs.view(-1, 1, d // 64)[flat] = (vs.view(-1, 1, d // 64)[flat].float() + 0.01).half()
    small = step % 2 == (0 if up else 1)                     # every other step's scales are tiny
    vs.view(-1, 1, d // 64)[flat[small]] *= 2.0 ** -9
    out = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=1).view(-1)
    pick = lambda c: c[table[0].long()].reshape(-1, *c.shape[2:])[:n]
    ref = _attention64(q[0], pick(kc), pick(vc), pick(ks), pick(vs)).reshape(-1)
    # one FP16 rounding; scores of up to 650 binades in FP32, 2^-15 of a weight
    lim = ref.abs() * (2.0 ** -11 + 2.0 ** -14) + 2.0 ** -14 * ref.abs().max() + 2.0 ** -25
    assert bool(((out.double() - ref).abs() <= lim).all())


# a group of query values far below the other, whose keys make up for it: seen in the records of the
# splits, which no FP16 rounding hides
@pytest.mark.parametrize("k", [8, 16, 22])
@pytest.mark.parametrize("group", [0, 1])
def test_attention_rows_keep_the_bits_of_small_query_groups(dev, k, group):
    from orinfer_b200.ops import functional as F
    n, qh, d, splits = 700, 4, 128, 2
    g = torch.Generator().manual_seed(k)
    q, req, pos, table, kc, vc, ks, vs = _walk(dev, n, qh, 1, d, n + k)
    assert _in_digits(qh, 1, d, table, splits)
    q = torch.randn(1, qh, 2, 64, generator=g)
    q[:, :, group] *= 2.0 ** (k // 2 - k)
    q[:, :, 1 - group] *= 2.0 ** (k // 2)
    q = q.view(1, qh, d).half().to(dev)
    ks[..., group] = (ks[..., group].float() * 2.0 ** (k - k // 2)).half()
    ks[..., 1 - group] = (ks[..., 1 - group].float() * 2.0 ** -(k // 2)).half()
    scratch = torch.empty(qh * splits * (d + 2), device=dev)
    F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=splits, scratch=scratch)
    rec = scratch.view(qh, splits, d + 2).double()
    part = torch.exp2(rec[..., 0] - rec[..., 0].amax(1, keepdim=True))[..., None]
    out = (rec[..., 2:] * part).sum(1) / (rec[..., 1:2] * part).sum(1)
    pick = lambda c: c[table[0].long()].reshape(-1, *c.shape[2:])[:n]
    ref = _attention64(q[0], pick(kc), pick(vc), pick(ks), pick(vs))
    # scores of up to 2^4 in FP32, whose error is the weights': 2^-19
    assert float((out - ref).norm() / ref.norm()) < 2.0 ** -19


# equal weights, which round the same way at every step of a sum
def test_attention_rows_add_a_block_of_weights_at_a_time(dev):
    from orinfer_b200.ops import functional as F
    n, d, splits = 240_000, 128, 2
    pages = (n + 127) // 128
    table = torch.arange(pages, dtype=torch.int32, device=dev)[None]
    kc = torch.zeros(pages, 128, 1, d, dtype=torch.int8, device=dev)
    kc[..., 0] = 1
    for k in range(0, n, n // splits):                    # every warp begins with weights of 1
        kc.view(-1, d)[k:k + 128] = 0
    vc = torch.full_like(kc, 100)
    s = torch.ones(pages, 128, 1, 2, device=dev).half()
    one = torch.zeros(1, dtype=torch.int32, device=dev)
    scratch = torch.empty(4 * splits * (d + 2), device=dev)
    assert _in_digits(4, 1, d, table, splits)
    err = []
    for i in range(24):                                   # weights from 0.51 to 0.99, a head each
        q = torch.zeros(1, 4, d, device=dev)
        q[0, :, 0] = -torch.linspace(0.01 + i / 25, 0.045 + i / 25, 4) * math.log(2) * math.sqrt(d)
        F.attention(q.half(), None, one, one + n - 1, table, kc, vc, s, s, splits=splits, scratch=scratch)
        rec = scratch.view(4, splits, d + 2).double()
        err.append(float((rec[..., 2:] / rec[..., 1:2] / 100 - 1).abs().max()))
    # a sum of as many terms as a warp has blocks of 32 keys, each step within 2^-24 of the sum so
    # far, half of the last one on average; 2^-21 for the rest
    blocks = n // splits // 32 // 4
    assert max(err) <= blocks / 2 * 2.0 ** -24 + 2.0 ** -21, max(err)


def test_attention_rows_sums_of_a_long_context_do_not_overflow(dev):
    """Where a weight of 1 times the scale has 27 bits, 1.125 * 2^26 has the digits 5, -128, 0 and 0, and
    128 x 127 a key passes 2^31 after 132 105 of a warp's 150 000 keys, were the sums not scaled down
    on the way (with a bit less or more 1.25 and 1.0625 have them).  Weights and their sum are exact,
    so only the output is rounded."""
    from orinfer_b200.ops import functional as F
    n, kvh, d = 600_000, 1, 64
    pages = (n + 127) // 128
    table = torch.arange(pages, dtype=torch.int32, device=dev)[None]
    assert _in_digits(4, kvh, d, table, 1)
    for value, size in ((127, 1.125), (-127, 1.125), (127, 1.25), (-127, 1.0625)):
        kc = torch.zeros(pages, 128, kvh, d, dtype=torch.int8, device=dev)
        vc = torch.full_like(kc, value)
        s = torch.full((pages, 128, kvh, 1), size * 2.0 ** -7, device=dev).half()
        q = torch.ones(1, 4, d, device=dev).half()
        one = torch.zeros(1, dtype=torch.int32, device=dev)
        out = F.attention(q, None, one, one + n - 1, table, kc, vc, s, s, splits=1)
        want = value * size * 2.0 ** -7
        # one FP16 rounding, a few FP32 ones
        lim = abs(want) * (2.0 ** -11 + 2.0 ** -20)
        assert bool(((out.double() - want).abs() <= lim).all()), out


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("splits", [1, 2])
def test_attention_rows_keep_the_other_group_of_a_bad_value_scale(dev, bad, splits):
    from orinfer_b200.ops import functional as F
    q, req, pos, table, kc, vc, ks, vs = _walk(dev, 700, 8, 2, 128, 5)
    assert _in_digits(8, 2, 128, table, splits)
    good = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=splits).view(2, 4, 2, 64)
    vs[int(table[0, 1]), 50, 1, 0] = bad                  # KV head 1, its lower group
    out = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=splits).view(2, 4, 2, 64)
    assert bool(out[1, :, 0].isnan().all())
    assert torch.equal(out[0], good[0]) and torch.equal(out[1, :, 1], good[1, :, 1])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_attention_rows_keep_the_other_heads_of_a_bad_query(dev, bad):
    from orinfer_b200.ops import functional as F
    q, req, pos, table, kc, vc, ks, vs = _walk(dev, 300, 8, 2, 128, 5)
    assert _in_digits(8, 2, 128, table, 1)
    good = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=1).view(8, 128)
    q[0, 2, 77] = bad
    out = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=1).view(8, 128)
    keep = torch.arange(8, device=dev) != 2
    assert torch.equal(out[keep], good[keep])
    assert not torch.equal(out[2], good[2])


# a query whose values span all of FP16, down to the smallest: rounded at 2^-31 of the largest
def test_attention_rows_of_a_query_of_many_binades(dev):
    from orinfer_b200.ops import functional as F
    for top in (0.0, 12.0):
        q, req, pos, table, kc, vc, ks, vs = _walk(dev, 800, 4, 1, 128, 9)
        assert _in_digits(4, 1, 128, table, 2)
        g = torch.Generator().manual_seed(1)
        q = (q.float() * torch.exp2(top - torch.rand(q.shape, generator=g).to(dev) * 30)).half()
        ks = (ks.float() * 2.0 ** -top).half()
        out = F.attention(q, None, req, pos, table, kc, vc, ks, vs, splits=2).view(-1)
        pick = lambda c: c[table[0].long()].reshape(-1, *c.shape[2:])[:800]
        ref = _attention64(q[0], pick(kc), pick(vc), pick(ks), pick(vs)).reshape(-1)
        lim = ref.abs() * 2.0 ** -11 + 2.0 ** -18 * ref.abs().max() + 2.0 ** -25
        assert bool(((out.double() - ref).abs() <= lim).all())


# the forms of short contexts again, with a page table wide enough for the digit form
@pytest.mark.parametrize("qh,kvh,d", [(8, 8, 64), (14, 7, 64), (5, 5, 128), (32, 8, 128)])
@pytest.mark.parametrize("waves", [0.9, 1.1, 2.1, 4.2])
def test_attention_rows_of_short_contexts_in_digits(dev, qh, kvh, d, waves):
    from orinfer_b200.ops import functional as F
    lens = [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65, 96, 97, 127, 128, 129, 160, 256]
    rows = int(waves * 148 * {64: 4, 128: 3}[d] / kvh)
    q, req, pos, table, kc, vc, ks, vs = _short_rows(dev, rows, qh, kvh, d, lens)
    for i, n in enumerate(lens):                    # slots never written hold anything
        if n % 128:
            page = table[i, (n - 1) // 128].long()
            ks[page, (n - 1) % 128 + 1:] = float("nan")
            vs[page, (n - 1) % 128 + 1:] = float("inf")
    wide = torch.cat([table, torch.zeros_like(table)], 1)
    assert _in_digits(qh, kvh, d, wide, 1)
    out = F.attention(q[req.long()].contiguous(), None, req, pos, wide, kc, vc, ks, vs,
                      splits=1).view(rows, qh * d)
    for i, n in enumerate(lens[:rows]):
        pick = lambda c: c[table[i].long()].reshape(-1, *c.shape[2:])[:n]
        ref = _attention64(q[i], pick(kc), pick(vc), pick(ks), pick(vs)).reshape(-1)
        lim = ref.abs() * 2.0 ** -11 + 2.0 ** -18 * ref.abs().max() + 2.0 ** -25
        got = out[i::len(lens)].double()
        assert bool(((got - ref).abs() <= lim).all()), n


# gates at any address, and as large as they come
@pytest.mark.parametrize("qh,kvh,d,rows", [(8, 1, 256, 37), (4, 2, 128, 70), (16, 2, 256, 300),
                                           (2, 2, 64, 33)])
@pytest.mark.parametrize("aligned", [True, False])
def test_attention_prefill_gates(dev, qh, kvh, d, rows, aligned):
    from orinfer_b200.ops import functional as F
    _, req, pos, table, kc, vc, ks, vs = _walk(dev, rows + 90, qh, kvh, d, rows)
    g = torch.Generator().manual_seed(d)
    q = torch.randn(rows, qh, d, generator=g).half().to(dev)
    size = torch.exp2(torch.rand(rows, qh, d, generator=g) * 14)
    gate = torch.randn(rows, qh, d, generator=g) * size
    gate[0, 0, :4] = torch.tensor([math.inf, -math.inf, 90.0, -90.0])
    gate = gate.half().to(dev)
    if not aligned:
        gate = _unaligned(gate)
    out = torch.empty(rows, qh * d, dtype=torch.float16, device=dev)
    chunks = torch.tensor([[0, rows, 90, 0]], dtype=torch.int32, device=dev)
    assert F.attention_prefill(q, gate, chunks, rows, table, kc, vc, ks, vs, out=out)
    plain = torch.empty_like(out)
    assert F.attention_prefill(q, None, chunks, rows, table, kc, vc, ks, vs, out=plain)
    want = plain.double() * torch.sigmoid(gate.double()).view(rows, -1)
    # the ungated output has one FP16 rounding (2^-11), the gated one another
    lim = want.abs() * 2.0 ** -10 + 2.0 ** -24
    assert bool(((out.double() - want).abs() <= lim).all())


# tiles whose keys are cut over a cluster: as few as the rows have, ragged chunks (clusters without a
# tile), parts without a step, slots never written
@pytest.mark.parametrize("rows,past,qh,kvh,parts", [(16, 4000, 8, 1, 8), (33, 900, 16, 2, 4),
                                                    (64, 1000, 16, 2, 4), (150, 2000, 16, 2, 4),
                                                    (230, 1700, 8, 1, 4), (400, 1500, 16, 2, 2),
                                                    (5, 3000, 2, 2, 8)])
@pytest.mark.parametrize("gated", [True, False])
def test_attention_prefill_cut_over_a_cluster(dev, rows, past, qh, kvh, parts, gated):
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    d, g = 256, torch.Generator().manual_seed(rows)
    sizes, pasts = [rows, max(1, rows // 3)], [past, 5]
    pages = [(n + p + 127) // 128 for n, p in zip(sizes, pasts)]
    table = torch.zeros(2, max(pages), dtype=torch.int32)
    order = torch.randperm(sum(pages), generator=g) + 1
    table[0, :pages[0]], table[1, :pages[1]] = order[:pages[0]], order[pages[0]:]
    shape = (sum(pages) + 1, 128, kvh)
    kc = torch.randint(-127, 128, (*shape, d), generator=g, dtype=torch.int8)
    vc = torch.randint(-127, 128, (*shape, d), generator=g, dtype=torch.int8)
    ks = (torch.rand(*shape, 4, generator=g) * 0.02 + 1e-3).half()
    vs = (torch.rand(*shape, 4, generator=g) * 0.02 + 1e-3).half()
    for i in range(2):
        n = sizes[i] + pasts[i]
        ks[table[i, pages[i] - 1], (n - 1) % 128 + 1:] = math.nan
        vs[table[i, pages[i] - 1], (n - 1) % 128 + 1:] = math.inf
    total = sum(sizes)
    q = torch.randn(total, qh, d, generator=g).half()
    gate = torch.randn(total, qh, d, generator=g).half() if gated else None
    tile_rows = 128 // (qh // kvh)
    tiles = min((rows + tile_rows - 1) // tile_rows * 2, total // tile_rows + 2)
    assert native.lib().orinfer_attention_prefill_parts(tiles * kvh, table.shape[1]) == parts
    out = torch.empty(total, qh * d, dtype=torch.float16, device=dev)
    chunks = torch.tensor([[0, sizes[0], past, 0], [sizes[0], sizes[1], 5, 1]], dtype=torch.int32)
    on = lambda t: None if t is None else t.to(dev)
    assert F.attention_prefill(on(q), on(gate), on(chunks), rows, on(table), on(kc), on(vc), on(ks),
                               on(vs), out=out)
    assert native.read_status() == 0
    at = 0
    for i in range(2):
        pick = lambda c: c[table[i, :pages[i]].long()].reshape(-1, *c.shape[2:])[:sizes[i] + pasts[i]]
        for r in range(0, sizes[i], max(1, sizes[i] // 7)):
            n = pasts[i] + r + 1
            ref = _attention64(q[at + r], pick(kc)[:n], pick(vc)[:n], pick(ks)[:n], pick(vs)[:n],
                               None if gate is None else gate[at + r]).reshape(-1)
            # keys, values and weights in FP16 (2^-11 each) under a softmax of many terms, FP16 output
            err = (out[at + r].cpu().double() - ref).norm() / ref.norm()
            assert float(err) < 2e-3, (i, r, float(err))
        at += sizes[i]


# the page table of a serving engine is as wide as the longest context there may be: which launch a
# packet gets, and with it the bits, depends on the context alone
@pytest.mark.parametrize("rows,past", [(17, 0), (64, 0), (64, 330), (130, 400), (64, 1000)])
def test_attention_prefill_of_a_packet_does_not_depend_on_the_width_of_its_table(dev, rows, past):
    cfg = dict(q_heads=8, kv_heads=1, head_dim=256, gated_attention=True)
    out = _packet_of_one_layer(dev, cfg, rows, past, prefill=True)
    assert torch.equal(out[1], out[3]) and torch.equal(out[0], out[2])


@pytest.mark.parametrize("rows,past", [(1, 100), (1, 900), (6, 1500), (3, 4000)])
def test_attention_of_a_decode_packet_does_not_depend_on_the_width_of_its_table(dev, rows, past):
    cfg = dict(q_heads=8, kv_heads=2, head_dim=128)
    out = _packet_of_one_layer(dev, cfg, rows, past, prefill=False)
    assert torch.equal(out[1], out[3]) and torch.equal(out[0], out[2])


def _packet_of_one_layer(dev, geometry, rows, past, prefill):
    """Logits and attention outputs of a packet of one request, a prefill chunk or verification rows,
    with a page table that fits and one of 256 pages."""
    import dataclasses
    from orinfer_b200.config import PRESETS
    from orinfer_b200.models.runner import KVPool, ModelRunner, Packet
    from orinfer_b200.models.weights import random_model
    cfg = dataclasses.replace(PRESETS["tiny"], layers=1, **geometry)
    w = random_model(cfg, seed=0).to(dev)
    g = torch.Generator().manual_seed(rows + past)
    pages = (rows + past + 127) // 128
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    runner = ModelRunner(w, KVPool.allocate(cfg, pages + 1, dev), max_rows=rows)
    kv = runner.kv
    for c in (kv.k[0], kv.v[0]):
        c.copy_(torch.randint(-127, 128, c.shape, generator=g, dtype=torch.int8))
    for c in (kv.ks[0], kv.vs[0]):
        c.copy_((torch.rand(c.shape, generator=g) * 0.02 + 1e-3).half())
    ids = torch.randint(0, cfg.vocab, (rows,), generator=g).int().to(dev)
    out = []
    for width in (pages, 256):
        table = torch.zeros(1, width, dtype=torch.int32, device=dev)
        table[0, :pages] = torch.arange(1, pages + 1)
        p = Packet(ids, t([0] * rows), t(list(range(past, past + rows))), table, rows, past + rows,
                   chunks=t([[0, rows, past, 0]]) if prefill else None, max_q_len=rows)
        out.append(runner.greedy(p, need_logits=True)[1].clone())
        out.append(runner.ws.attn[:rows].clone())
    return out
