"""Routing, dispatch and expert projections at the edges of their ranges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(cuda):
    from orinfer_b200.ops import native
    native.init()
    return cuda


def _int_weight(fmt, n, k, g):
    """(codes, FP16 scales, integer weights) of a random projection."""
    from orinfer_b200.models.weights import QLinear
    if fmt == "w8":
        codes = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8)
    elif fmt == "q4":
        codes = torch.randint(-2 ** 31, 2 ** 31, (k // 128, n, 16), generator=g, dtype=torch.int32)
    else:
        codes = torch.randint(-2 ** 15, 2 ** 15, (k // 128, n, 16), generator=g, dtype=torch.int16)
    scale = (torch.rand(n, generator=g) * 0.01 + 1e-3).half()
    return codes, scale, QLinear(fmt, n, k, codes, scale, None).integers()


def _int_weight_of(fmt, codes, scale, n, k):
    from orinfer_b200.models.weights import QLinear
    return QLinear(fmt, n, k, codes, scale, None).integers()


def _scaled(a, sa, w, ws):
    """The integer product with its two FP32 scales, in the kernels' order."""
    acc = (a.double() @ w.double().t()).float()
    return (acc * ws.float()[None]) * sa.float()[:, None]


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 50])
@pytest.mark.parametrize("hidden,experts,top_k,shared", [
    (256, 3, 2, False), (256, 64, 4, True), (512, 128, 8, False), (2048, 191, 8, True),
    (256, 192, 8, True), (2048, 512, 10, True), (256, 576, 6, False), (256, 576, 6, True),
    (264, 128, 8, False), (4096, 9, 2, False), (2304, 16, 3, True)])
def test_router_topk_forms(dev, rows, hidden, experts, top_k, shared):
    """Tensor-core and general router at the edges of their expert and row tiles."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(experts + rows)
    y = torch.randn(rows, hidden, generator=g).half().to(dev)
    w = (torch.randn(experts + int(shared), hidden, generator=g) * 0.1).half().to(dev)
    w[experts - 1] = w[0]                                  # an exact tie: the lower id first
    ids, probs, gate = F.router_topk(y, w, experts, top_k)
    logits = y.double() @ w.double().t()
    p, order = torch.softmax(logits[:, :experts], 1).sort(dim=1, descending=True, stable=True)
    p, order = p[:, :top_k], order[:, :top_k]
    p = p / p.sum(1, keepdim=True)
    # FP32 sums of up to 2048 products: the logits are within 1e-5 of exact, the weights with them
    assert bool(((probs.double() - p).abs() <= 4e-5 * p + 1e-7).all())
    picked = torch.gather(logits, 1, ids.long())
    assert bool(((picked - torch.gather(logits, 1, order)).abs() <= 2e-5).all())
    for r in range(rows):
        chosen = ids[r].tolist()
        assert len(set(chosen)) == top_k
        if experts - 1 in chosen:
            assert 0 in chosen and chosen.index(0) < chosen.index(experts - 1)
    if shared:
        assert torch.allclose(gate.double(), torch.sigmoid(logits[:, experts]), atol=1e-5)


@pytest.mark.parametrize("hidden,experts,shared", [(512, 64, False), (2048, 128, False),
                                                   (2048, 512, True), (4096, 256, True)])
def test_router_sums_keep_fp32_accuracy(dev, hidden, experts, shared):
    """Probabilities against 64 bits: no further than rounded FP32 sums in blocks would be."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(hidden)
    y = torch.randn(1024, hidden, generator=g).half().to(dev)
    w = (torch.randn(experts + int(shared), hidden, generator=g) * 0.02).half().to(dev)
    ids, probs, _ = F.router_topk(y, w, experts, 6, renorm=False)
    p = torch.softmax((y.double() @ w.double().t())[:, :experts], 1)
    p = torch.gather(p, 1, ids.long())
    # logits of about 0.02 sqrt(hidden) with a few roundings of 2^-25 each in the mean, and as many
    # again in the exponential, the sum over the experts and the division
    limit = 2.0 ** -25 * (4 + 0.02 * hidden ** 0.5 * 3)
    assert float((probs.double() - p).norm() / p.norm()) < limit


@pytest.mark.parametrize("rows,hidden,experts,top_k,shared,form", [
    (512, 2048, 128, 8, False, 64), (513, 2048, 135, 8, True, 64), (575, 1536, 43, 40, False, 64),
    (1100, 3072, 97, 6, True, 64), (640, 4096, 129, 1, False, 64), (700, 2048, 33, 33, False, 64),
    (575, 1536, 40, 40, False, 1), (40, 2048, 64, 35, True, 16)])
def test_router_rows_form_and_long_choices(dev, rows, hidden, experts, top_k, shared, form):
    """The form for many rows at the edges of its row and expert tiles and both spans of four and
    eight CTAs, and choices past the 32nd in all forms."""
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    assert native.lib().orinfer_router_form(rows, hidden, experts, int(shared)) == form
    g = torch.Generator(device=dev).manual_seed(experts + rows)
    y = torch.randn(rows, hidden, generator=g, device=dev).half()
    w = (torch.randn(experts + int(shared), hidden, generator=g, device=dev) * 0.02).half()
    w[experts - 1] = w[0]                                  # an exact tie: the lower id first
    logits = y.double() @ w.double().t()
    p, order = torch.softmax(logits[:, :experts], 1).sort(dim=1, descending=True, stable=True)
    p, order = p[:, :top_k], order[:, :top_k]
    for renorm in (True, False):
        ids, probs, gate = F.router_topk(y, w, experts, top_k, renorm=renorm)
        want = p / p.sum(1, keepdim=True) if renorm else p
        # FP32 sums of up to 4096 products, as above
        assert bool(((probs.double() - want).abs() <= 4e-5 * want + 1e-7).all())
        picked = torch.gather(logits, 1, ids.long())
        assert bool(((picked - torch.gather(logits, 1, order)).abs() <= 2e-5).all())
        assert bool((ids.sort(1).values.diff(dim=1) > 0).all())            # no expert twice
        first, last = ((ids == e).int().argmax(1) for e in (0, experts - 1))
        both = (ids == 0).any(1) & (ids == experts - 1).any(1)
        assert bool((first[both] < last[both]).all())
        if shared:
            assert torch.allclose(gate.double(), torch.sigmoid(logits[:, experts]), atol=1e-5)


@pytest.mark.parametrize("experts,rows,top_k,k", [(1, 1, 1, 128), (8, 5, 2, 256), (3, 300, 1, 128),
                                                  (128, 2048, 8, 2048), (512, 16, 10, 2048),
                                                  (512, 700, 10, 512)])
@pytest.mark.parametrize("part", [False, True])
def test_moe_dispatch_numbers_and_copies(dev, experts, rows, top_k, k, part):
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(rows)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(rows)])
    ids = (ids // 2 if experts == 8 else ids).to(torch.int32)      # some experts get no row
    q8 = torch.randint(-127, 128, (rows, k), generator=g, dtype=torch.int8).to(dev)
    scale = torch.rand(rows, generator=g).to(dev)
    base, local = (experts // 3, max(experts // 2, 1)) if part else (0, experts)
    if base + local > experts:
        local = experts - base
    sc = F.MoeScratch(rows, top_k, experts, k, 64, dev)
    sc.tiles.fill_(-7)
    F.moe_dispatch(ids.to(dev), q8, scale, experts, sc, rows, base, local)
    flat = ids.flatten().long() - base
    flat = torch.where((flat >= 0) & (flat < local), flat, local)
    order = torch.sort(flat, stable=True).indices
    want = torch.full((rows * top_k,), -1, dtype=torch.int64)
    kept = int((flat < local).sum())
    want[order[:kept]] = torch.arange(kept)
    counts = torch.bincount(flat, minlength=local + 1)[:local]
    assert torch.equal(sc.slots.cpu().long(), want)
    assert torch.equal(sc.counts[:local].cpu().long(), counts)
    offs = torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)])
    assert torch.equal(sc.offsets[:local + 1].cpu().long(), offs)
    tiles = [[e, int(offs[e]) + r, min(128, int(counts[e]) - r), r // 128]
             for e in range(local) for r in range(0, int(counts[e]), 128)]
    assert int(sc.meta[0]) == len(tiles)
    assert sc.tiles[:len(tiles)].cpu().tolist() == tiles
    src = order[:kept] // top_k
    assert torch.equal(sc.q8[:kept].cpu(), q8.cpu()[src])
    assert torch.equal(sc.scale[:kept].cpu(), scale.cpu()[src])


@pytest.mark.parametrize("local", [4, 12])
@pytest.mark.parametrize("k", [16, 2048, 4112])
def test_moe_dispatch_of_a_mostly_free_buffer(dev, local, k):
    """One slot a row, most of them free (-1) or of another rank: the free rows' values and
    scales, here never written, go nowhere."""
    from orinfer_b200.ops import functional as F
    rows, base = 700, 0 if local == 12 else 3
    g = torch.Generator().manual_seed(k)
    ids = torch.full((rows, 1), -1, dtype=torch.int32)
    live = torch.randperm(rows, generator=g)[:30]
    ids[live, 0] = torch.randint(0, 12, (30,), generator=g, dtype=torch.int32)
    q8 = torch.full((rows, k), -128, dtype=torch.int8)
    scale = torch.full((rows,), float("nan"))
    q8[live] = torch.randint(-127, 128, (30, k), generator=g, dtype=torch.int8)
    scale[live] = torch.rand(30, generator=g)
    sc = F.MoeScratch(rows, 1, 12, k, 64, dev)
    sc.q8.fill_(7)
    sc.scale.fill_(7.0)
    F.moe_dispatch(ids.to(dev), q8.to(dev), scale.to(dev), 12, sc, rows, base, local)
    flat = ids.flatten() - base
    flat = torch.where((flat >= 0) & (flat < local) & (ids.flatten() >= 0), flat, local)
    kept = int((flat < local).sum())
    order = torch.sort(flat, stable=True).indices[:kept]
    assert torch.equal(sc.q8[:kept].cpu(), q8[order])
    assert torch.equal(sc.scale[:kept].cpu(), scale[order])
    assert bool((sc.q8[kept:] == 7).all()) and bool((sc.scale[kept:] == 7.0).all())


# few rows per expert (small-M kernel, K shared by several warps or not), a tile of rows and
# several tiles of rows per expert (one, two or four row tiles per CTA)
@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("counts", [[1, 0, 2, 7, 8, 9, 0, 1, 3, 0, 0, 0, 1, 1, 1, 1],
                                    [0] * 30 + [16, 17, 33], [0] * 40 + [129] + [0] * 9,
                                    [1, 1, 0, 1], [40, 0, 13, 1], [300, 0, 129, 128, 5, 256],
                                    [513, 257, 300]])
@pytest.mark.parametrize("n,k", [(128, 128), (384, 640), (256, 4096)])
def test_grouped_projection_is_exact(dev, fmt, counts, n, k):
    from orinfer_b200.ops import functional as F
    experts, s = len(counts), sum(counts)
    g = torch.Generator().manual_seed(s)
    banks = [_int_weight(fmt, n, k, g) for _ in range(experts)]
    a = torch.randint(-127, 128, (s, k), generator=g, dtype=torch.int8)
    sa = torch.rand(s, generator=g) * 0.05 + 1e-3
    ids = torch.tensor([e for e, c in enumerate(counts) for _ in range(c)], dtype=torch.int32)
    sc = F.MoeScratch(s, 1, experts, k, 64, dev)
    F.moe_dispatch(ids[:, None].to(dev), a.to(dev), sa.to(dev), experts, sc, s)
    out = torch.full((s, n), float("nan"), dtype=torch.float16, device=dev)
    F.qgemm_grouped(sc.q8, sc.scale, torch.stack([b[0] for b in banks]).to(dev),
                    torch.stack([b[1] for b in banks]).to(dev), fmt, n, out, sc, s)
    at = 0
    for e, c in enumerate(counts):                       # the rows are in expert order already
        if c:
            want = _scaled(a[at:at + c].to(dev), sa[at:at + c].to(dev), banks[e][2].to(dev),
                           banks[e][1].to(dev))
            assert torch.equal(out[at:at + c], want.half()), e
        at += c


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("experts,rows,top_k,tall", [
    (1100, 40, 3, [5]), (1100, 300, 2, [0, 1, 600, 1024, 1099]), (64, 25, 4, [3, 63]),
    (64, 17, 4, [3, 63]), (16, 100, 1, [9]), (40, 130, 2, [0, 39])])
@pytest.mark.parametrize("expected", [None, 1])
def test_grouped_projection_splits_by_tile_height(dev, fmt, experts, rows, top_k, tall, expected):
    """Few rows per expert but many for some: every row is written, by one kernel or the other,
    over tile lists of more entries than a CTA has threads and experts of several tiles."""
    from orinfer_b200.ops import functional as F
    n = k = 128
    g = torch.Generator().manual_seed(experts + rows)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(rows)])
    for r in range(rows - 3):                              # most rows go to the tall experts too
        e = tall[r % len(tall)]
        if e not in ids[r]:
            ids[r, 0] = e
    codes, ws, _ = _int_weight(fmt, experts * n, k, g)
    split = [codes[i * n:(i + 1) * n] if fmt == "w8" else codes[:, i * n:(i + 1) * n]
             for i in range(experts)]
    ints = _int_weight_of(fmt, codes, ws, experts * n, k).to(dev)
    a = torch.randint(-127, 128, (rows, k), generator=g, dtype=torch.int8).to(dev)
    sa = (torch.rand(rows, generator=g) * 0.05 + 1e-3).to(dev)
    sc = F.MoeScratch(rows, top_k, experts, k, 64, dev)
    F.moe_dispatch(ids.to(torch.int32).to(dev), a, sa, experts, sc, rows)
    out = torch.full((rows * top_k, n), float("nan"), dtype=torch.float16, device=dev)
    F.qgemm_grouped(sc.q8, sc.scale, torch.stack(split).contiguous().to(dev),
                    ws.view(experts, n).to(dev), fmt, n, out, sc, rows * top_k, expected)
    flat = ids.flatten()
    order = torch.sort(flat, stable=True).indices.to(dev)
    flat = flat.to(dev)
    src = a[order // top_k].double()
    acc = torch.einsum("rk,rnk->rn", src, ints.view(experts, n, k)[flat[order]].double()).float()
    want = acc * ws.view(experts, n).to(dev)[flat[order]].float() * sa[order // top_k, None]
    assert torch.equal(out, want.half())


@pytest.mark.parametrize("short,tall", [(383, 200), (384, 256), (383, 129)])
def test_walked_tile_lists_of_several_passes(dev, short, tall):
    """More INT8 experts than the 384 threads of the walking kernel, so that its CTAs list the tiles
    in two passes, and an expert of two tiles across the seam (codes have more threads than room
    for tiles)."""
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    n, k, fmt = 128, 128, "w8"
    counts = [120] * (short - 1) + [97, tall, 1, 0, 128]
    experts, s = len(counts), sum(counts)
    g = torch.Generator().manual_seed(short + tall)
    codes, ws, _ = _int_weight(fmt, experts * n, k, g)
    codes, ws = codes.view(experts, n, k).to(dev), ws.view(experts, n).to(dev)
    a = torch.randint(-127, 128, (s, k), generator=g, dtype=torch.int8).to(dev)
    sa = (torch.rand(s, generator=g) * 0.05 + 1e-3).to(dev)
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts)).to(torch.int32)
    sc = F.MoeScratch(s, 1, experts, k, 64, dev)
    F.moe_dispatch(ids[:, None].to(dev), a, sa, experts, sc, s)
    tiles = int(sc.meta[0])
    assert tiles > 384
    assert native.lib().orinfer_qgemm_grouped_form(F.FMT[fmt], s, experts, sc.tiles.shape[0], s,
                                                   s) == 3
    out = torch.full((s, n), float("nan"), dtype=torch.float16, device=dev)
    F.qgemm_grouped(sc.q8, sc.scale, codes, ws, fmt, n, out, sc, s)
    at = 0
    for e, c in enumerate(counts):                       # the rows are in expert order already
        want = _scaled(a[at:at + c], sa[at:at + c], codes[e], ws[e])
        assert torch.equal(out[at:at + c], want.half()), e
        at += c


@pytest.mark.parametrize("fmt", ["q4", "q2"])
def test_walked_experts_of_many_row_tiles(dev, fmt):
    """Codes of experts with three row tiles and more, which the walking kernel takes two at a time:
    odd numbers of them, a single row in the last, experts without rows."""
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    n, k = 256, 256
    counts = [257, 600, 0, 385, 128, 1025, 512, 300, 1, 640, 513, 256, 129, 900, 383, 300]
    experts, s = len(counts), sum(counts)
    assert s >= 256 * experts
    g = torch.Generator().manual_seed(s)
    codes, ws, _ = _int_weight(fmt, experts * n, k, g)
    split = [codes[:, i * n:(i + 1) * n] for i in range(experts)]
    ints = _int_weight_of(fmt, codes, ws, experts * n, k).to(dev).view(experts, n, k)
    ws = ws.view(experts, n).to(dev)
    a = torch.randint(-127, 128, (s, k), generator=g, dtype=torch.int8).to(dev)
    sa = (torch.rand(s, generator=g) * 0.05 + 1e-3).to(dev)
    ids = torch.repeat_interleave(torch.arange(experts), torch.tensor(counts)).to(torch.int32)
    sc = F.MoeScratch(s, 1, experts, k, 64, dev)
    F.moe_dispatch(ids[:, None].to(dev), a, sa, experts, sc, s)
    form = native.lib().orinfer_qgemm_grouped_form
    assert form(F.FMT[fmt], s, experts, sc.tiles.shape[0], s, s) == 3
    assert form(F.FMT[fmt], 4096, 8, sc.tiles.shape[0], 4096, 512) == 2      # few: one wave
    out = torch.full((s, n), float("nan"), dtype=torch.float16, device=dev)
    banks = torch.stack(split).contiguous().to(dev)
    F.qgemm_grouped(sc.q8, sc.scale, banks, ws, fmt, n, out, sc, s)
    at = 0
    for e, c in enumerate(counts):                       # the rows are in expert order already
        want = _scaled(a[at:at + c], sa[at:at + c], ints[e], ws[e])
        assert torch.equal(out[at:at + c], want.half()), e
        at += c


def _grouped_us(dev, ids, experts, n, k, fmt, banks):
    from orinfer_b200.ops import functional as F
    rows, top_k = ids.shape
    sc = F.MoeScratch(rows, top_k, experts, k, 64, dev)
    a = torch.randint(-127, 128, (rows, k), dtype=torch.int8, device=dev)
    F.moe_dispatch(ids.to(torch.int32).to(dev), a, torch.rand(rows, device=dev), experts, sc, rows)
    out = torch.empty(rows * top_k, n, dtype=torch.float16, device=dev)
    times = []
    for _ in range(15):
        b, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        b.record()
        for _ in range(10):
            F.qgemm_grouped(sc.q8, sc.scale, banks[0], banks[1], fmt, n, out, sc, rows * top_k)
        e.record()
        e.synchronize()
        times.append(b.elapsed_time(e) * 100)
    return sorted(times)[len(times) // 2]


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
def test_grouped_projection_takes_skew(dev, fmt):
    """Rows that crowd on a few experts read fewer weights than evenly spread ones: they take no
    longer.  (A kernel that walks each expert's weights once per sixteen rows took 2.5 times as
    long; the margin is for the clock.)"""
    experts, n, k, rows, top_k = 128, 1536, 2048, 110, 8
    g = torch.Generator().manual_seed(1)
    codes, ws, _ = _int_weight(fmt, n, k, g)
    banks = (codes[None].expand(experts, *codes.shape).contiguous().to(dev),
             ws[None].expand(experts, n).contiguous().to(dev))
    even = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(rows)])
    weight = 1.0 / torch.arange(1, experts + 1).float() ** 1.2
    skew = torch.stack([torch.multinomial(weight, top_k, generator=g) for _ in range(rows)])
    t = [_grouped_us(dev, i, experts, n, k, fmt, banks) for i in (even, skew)]
    assert t[1] < 1.25 * t[0], t


def test_grouped_projection_follows_expected_rows():
    """The choice of kernels follows the rows to be expected, not the room for them."""
    from orinfer_b200.ops import native
    lib = native.lib()
    # 16 experts, room for 4096 rows of top 8: tensor cores alone (one launch) ...
    assert lib.orinfer_qgemm_grouped_launches(1, 4096, 16, 48, 4096, 512) == 1
    # ... with 64 expected both kernels, and one where no expert can have many
    assert lib.orinfer_qgemm_grouped_launches(1, 4096, 16, 48, 64, 512) == 2
    assert lib.orinfer_qgemm_grouped_launches(1, 128, 16, 48, 64, 16) == 1
