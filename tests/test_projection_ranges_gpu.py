"""Projections and row preparation at the edges of their tiles."""
import math

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


def _scaled(a, sa, w, ws):
    """The integer product with its two FP32 scales, in the kernels' order."""
    acc = (a.double() @ w.double().t()).float()
    return (acc * ws.float()[None]) * sa.float()[:, None]


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n,k", [(8, 128), (24, 384), (16, 1152), (2560, 1024), (2376, 512),
                                 (40000, 256), (3976, 2176), (6152, 2176), (264, 8448)])
def test_small_row_projections_are_exact(dev, fmt, m, n, k):
    """Row groups of sixteen cut by N, single k-blocks, K splits and several groups per CTA, on both
    sides of the lines between the dp4a, row-per-warp and MMA forms."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(m * n + k)
    codes, ws, w = _int_weight(fmt, n, k, g)
    a = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    sa = torch.rand(m, generator=g) * 0.05 + 1e-3
    want = _scaled(a, sa, w, ws)
    for f32 in (False, True):
        out = F.qgemm(a.to(dev), sa.to(dev), codes.to(dev), ws.to(dev), fmt, n, out_f32=f32, path=1)
        assert torch.equal(out.cpu(), want if f32 else want.half())


@pytest.mark.parametrize("m", [1, 2, 3, 8])
@pytest.mark.parametrize("n,k", [(93752, 256), (187504, 128), (23440, 1024), (7512, 3200),
                                 (24008, 1024)])
def test_streamed_int8_projections_are_exact(dev, m, n, k):
    """From 24 million weights on: short rows and the longest that keep three ring stages, a last
    tile of eight rows, CTAs with one tile more than others."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator(device=dev).manual_seed(m * n + k)
    w = torch.randint(-127, 128, (n, k), generator=g, device=dev, dtype=torch.int8)
    ws = (torch.rand(n, generator=g, device=dev) * 0.01 + 1e-3).half()
    a = torch.randint(-127, 128, (m, k), generator=g, device=dev, dtype=torch.int8)
    sa = torch.rand(m, generator=g, device=dev) * 0.05 + 1e-3
    want = _scaled(a, sa, w, ws)
    for f32 in (False, True) * 5:            # repeated: stages are refilled while others run
        out = F.qgemm(a, sa, w, ws, "w8", n, out_f32=f32, path=1)
        assert torch.equal(out, want if f32 else want.half())


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m,n", [(260, 19456), (600, 19456), (1024, 19456), (1500, 6400),
                                 (2047, 9728), (2048, 19456)])
def test_peeled_tail_tiles_are_exact(dev, fmt, m, n):
    """Grids a few CTAs past a whole number of waves, M tiles cut by the last row."""
    import ctypes
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    plan = (ctypes.c_int * 4)()
    native.lib().orinfer_qgemm_plan(F.FMT[fmt], m, n, 1024, 0, plan)
    assert plan[3] > 0                                # these shapes do peel tiles
    g = torch.Generator().manual_seed(m)
    codes, ws, w = _int_weight(fmt, n, 1024, g)
    a = torch.randint(-127, 128, (m, 1024), generator=g, dtype=torch.int8)
    sa = torch.rand(m, generator=g) * 0.05 + 1e-3
    want = _scaled(a.to(dev), sa.to(dev), w.to(dev), ws.to(dev))
    for f32 in (False, True):
        out = F.qgemm(a.to(dev), sa.to(dev), codes.to(dev), ws.to(dev), fmt, n, out_f32=f32)
        assert torch.equal(out, want if f32 else want.half())


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m,n,k", [(9, 25600, 128), (128, 25560, 384), (129, 25560, 1152),
                                   (255, 40000, 640), (256, 25608, 2560), (385, 25560, 384),
                                   (1030, 12200, 768)])
def test_walked_tiles_are_exact(dev, fmt, m, n, k):
    """More tiles than SMs: one row tile and two, the last of them cut, columns cut inside an
    eight-row piece of a tile, single k-blocks, fewer k-blocks than ring stages; repeated, since its
    warps run ahead of each other."""
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    lib = native.lib()
    g = torch.Generator().manual_seed(m + n + k)
    codes, ws, w = _int_weight(fmt, n, k, g)
    a = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    sa = torch.rand(m, generator=g) * 0.05 + 1e-3
    want = _scaled(a.to(dev), sa.to(dev), w.to(dev), ws.to(dev)).half()
    a, sa, codes, ws = a.to(dev), sa.to(dev), codes.to(dev), ws.to(dev)
    if m > 256 and fmt != "w8":                            # codes: two row tiles, not four
        assert not lib.orinfer_qgemm_walks(F.FMT[fmt], m, n, k, 0)
        assert lib.orinfer_qgemm_set_variant(F.FMT[fmt], m, m, n, k, 2, 128, 1) == 0
    try:
        assert lib.orinfer_qgemm_walks(F.FMT[fmt], m, n, k, 0)
        for _ in range(5):
            assert torch.equal(F.qgemm(a, sa, codes, ws, fmt, n), want)
    finally:
        lib.orinfer_qgemm_clear_variants()


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m", [129, 300, 513, 1100])
@pytest.mark.parametrize("n,k", [(1000, 2048), (2568, 4096), (6144, 2048), (12296, 2176)])
def test_plans_of_least_cost_are_exact(dev, fmt, m, n, k):
    """Plans chosen by their cost: narrow and wide tiles, K splits and walked tiles, columns that no
    tile width divides; without a tuned table."""
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    from orinfer_b200.tuning import tables
    lib = native.lib()
    g = torch.Generator().manual_seed(m + n + k)
    codes, ws, w = _int_weight(fmt, n, k, g)
    a = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    sa = torch.rand(m, generator=g) * 0.05 + 1e-3
    want = _scaled(a.to(dev), sa.to(dev), w.to(dev), ws.to(dev)).half()
    lib.orinfer_qgemm_clear_variants()
    try:
        for _ in range(2):
            out = F.qgemm(a.to(dev), sa.to(dev), codes.to(dev), ws.to(dev), fmt, n)
            assert torch.equal(out, want)
    finally:
        tables.load_default(lib)


@pytest.mark.parametrize("rows", [1, 7, 149, 300, 2049])
@pytest.mark.parametrize("k", [128, 384, 768, 2176, 6144, 6272, 9728, 16384])
@pytest.mark.parametrize("mode", ["norm", "plain", "swiglu", "bare"])
def test_act_prep_row_splits(dev, rows, k, mode):
    """Blocks of a row over one to 32 warps, uneven splits, against the torch statement: INT8
    codes may differ by one where a value sits on a rounding boundary."""
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ref import ops_ref as R
    if rows * k > 1 << 23:
        rows = (1 << 23) // k
    g = torch.Generator(device=dev).manual_seed(rows + k)
    x = torch.randn(rows, 2 * k if mode == "swiglu" else k, generator=g, device=dev).half()
    signs = (1 - 2 * torch.randint(0, 2, (k,), generator=g, device=dev)).to(torch.int8)
    resid = torch.randn(rows, k, generator=g, device=dev) if mode == "norm" else None
    w = (1 + 0.1 * torch.randn(k, generator=g, device=dev)).half() if mode == "norm" else None
    if mode == "bare":
        signs = None
    ref_q, ref_s, ref_r, ref_y = R.act_prep(x, resid, w, signs, swiglu=mode == "swiglu")
    y = torch.empty(rows, k, dtype=torch.float16, device=dev)
    q, s = F.act_prep(x, resid, w, signs, swiglu=mode == "swiglu", y_out=y)
    diff = (q.int() - ref_q.int()).abs()
    assert int(diff.max()) <= 1 and float((diff > 0).float().mean()) < 0.01
    assert bool(((s - ref_s).abs() <= ref_s * 2.0 ** -10).all())      # one FP16 step
    assert bool(((y.float() - ref_y).abs() <= ref_y.abs() * 2.0 ** -10 + 1e-7).all())
    if resid is not None:
        assert torch.equal(resid, ref_r)


@pytest.mark.parametrize("rows,k,fused", [(300, 4096, False), (8, 16384, False), (8, 4096, True)])
def test_swiglu_sigmoid_keeps_fp32_accuracy(dev, rows, k, fused):
    """Strongly negative gates times large values: the FP32 product under the FP16 rounding."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator(device=dev).manual_seed(k)
    y = torch.empty(rows, k, dtype=torch.float16, device=dev)
    for _ in range(8 if rows > 8 else 60):
        gate = -21 + 6 * torch.rand(rows, k, generator=g, device=dev)
        x = torch.cat([gate, 2e4 + 4e4 * torch.rand(rows, k, generator=g, device=dev)], 1).half()
        if fused:
            codes, ws, _ = _int_weight("q4", 8, k, torch.Generator().manual_seed(1))
            assert F.qgemv_fused(F.PRE_SWIGLU, x, None, None, None, codes.to(dev), ws.to(dev), "q4",
                                 8, k, rows, y_out=y,
                                 out=torch.empty(rows, 8, dtype=torch.float16, device=dev))
        else:
            F.act_prep(x, None, None, None, swiglu=True, y_out=y)
        a, u = x.double().chunk(2, 1)
        ref = a * torch.sigmoid(a) * u
        half_ulp = torch.exp2(torch.floor(torch.log2(ref.abs())) - 11)
        # e^-x within one step (2^-23), then a sum, a reciprocal and two products (2^-24 each)
        assert bool(((y.double() - ref).abs() <= half_ulp + ref.abs() * 3 * 2.0 ** -23).all())


@pytest.mark.parametrize("fmt", ["q4", "q2"])
@pytest.mark.parametrize("m,n,k", [(2, 24, 384), (4, 2376, 512), (8, 1040, 1152), (5, 9736, 2560),
                                   (8, 9736, 2560)])
def test_fused_projection_forms_equal_separate_kernels(dev, fmt, m, n, k):
    """dp4a and MMA forms with a row preparation give the bits of act_prep and qgemm."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(m * n + k)
    codes, ws, _ = _int_weight(fmt, n, k, g)
    codes, ws = codes.to(dev), ws.to(dev)
    signs = (1 - 2 * torch.randint(0, 2, (k,), generator=g)).to(torch.int8).to(dev)
    for pre, width in ((F.PRE_PLAIN, k), (F.PRE_SWIGLU, 2 * k)):
        x = torch.randn(m, width, generator=g).half().to(dev)
        q8, sc = F.act_prep(x, None, None, signs, swiglu=pre == F.PRE_SWIGLU)
        want = F.qgemm(q8, sc, codes, ws, fmt, n)
        out = torch.empty_like(want)
        assert F.qgemv_fused(pre, x, None, None, signs, codes, ws, fmt, n, k, m, out=out)
        assert torch.equal(out, want)


@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m", [1, 8, 40, 300])
def test_kernels_that_start_early_keep_the_stream_order(dev, fmt, m):
    """Row preparations and projections one behind the other, each reading what the one before wrote
    and overwriting what an earlier one read, weights copied right before their use: eagerly without
    a wait and in a graph, against the same calls with a wait after each."""
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(m)
    k, n = 1024, 2048
    up, ups, _ = _int_weight(fmt, n, k, g)
    down, downs, _ = _int_weight(fmt, k, n // 2, g)
    banks = [t.to(dev) for t in (up, ups, down, downs)]
    live = [torch.empty_like(t) for t in banks]
    x0 = torch.randn(m, k, generator=g).half().to(dev)
    x, gu = torch.empty_like(x0), torch.empty(m, n, dtype=torch.float16, device=dev)
    norm = torch.ones(k, dtype=torch.float16, device=dev)
    q8, s8 = torch.empty(m, k, dtype=torch.int8, device=dev), torch.empty(m, device=dev)
    qm = torch.empty(m, n // 2, dtype=torch.int8, device=dev)

    def chain(wait):
        step = torch.cuda.synchronize if wait else (lambda: None)
        x.copy_(x0)
        for i in range(4):
            for to, bank in zip(live, banks):
                to.copy_(bank.roll(i, 0) if bank.dim() > 1 else bank)
            step()
            F.act_prep(x, None, norm, None, q_out=q8, scale_out=s8)
            step()
            F.qgemm(q8, s8, live[0], live[1], fmt, n, out=gu)
            step()
            F.act_prep(gu, None, None, None, swiglu=True, q_out=qm, scale_out=s8)
            step()
            F.qgemm(qm, s8, live[2], live[3], fmt, k, out=x)
            step()

    chain(True)
    want = x.clone()
    assert bool(want.isfinite().all())
    for _ in range(10):
        chain(False)
        assert torch.equal(x, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(False)
    for _ in range(10):
        graph.replay()
        assert torch.equal(x, want)


# rows of a warp each, which larger packets take, against the same rows in small packets
@pytest.mark.parametrize("k", [128, 256, 384, 512, 640, 768, 896, 1024, 1152])
@pytest.mark.parametrize("signed", [True, False])
def test_swiglu_rows_of_large_packets_have_the_bits_of_small_ones(dev, k, signed):
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(k)
    rows = 1024 + 5 * k // 128
    x = torch.randn(rows, 2 * k, generator=g) * torch.exp2(torch.randint(-13, 5, (rows, 1), generator=g))
    x[3] = 0                                           # an empty row
    x[5, :k] = -300                                    # sigmoids below the normal numbers
    x[7, 2], x[9, k + 1], x[11, 0] = math.nan, math.inf, -math.inf
    x[13, :k], x[13, k:] = 2.0 ** -9, 2.0 ** -14       # scales among FP16's subnormal numbers
    x = x.half().to(dev)
    signs = (torch.randint(0, 2, (k,), generator=g) * 2 - 1).to(torch.int8).to(dev) if signed else None
    y = torch.empty(rows, k, dtype=torch.float16, device=dev)
    q, s = F.act_prep(x, None, None, signs, swiglu=True, y_out=y)
    for at in range(0, rows, 512):
        part = x[at:at + 512].contiguous()
        y1 = torch.empty(part.shape[0], k, dtype=torch.float16, device=dev)
        q1, s1 = F.act_prep(part, None, None, signs, swiglu=True, y_out=y1)
        same = lambda a, b: torch.equal(torch.nan_to_num(a.float(), 1e9), torch.nan_to_num(b.float(), 1e9))
        assert same(y[at:at + 512], y1) and same(s[at:at + 512], s1)
        assert torch.equal(q[at:at + 512], q1)
    # a count on the device limits the rows
    q2, s2 = torch.full_like(q, 77), torch.full_like(s, 77)
    F.act_prep_limited(x, signs, torch.tensor([1025], dtype=torch.int32, device=dev), swiglu=True,
                       rows=rows, q_out=q2, scale_out=s2)
    assert torch.equal(q2[:1025], q[:1025]) and bool((q2[1025:] == 77).all())
    assert bool((s2[1025:] == 77).all())


# nine to sixteen rows on the small-M kernels: row groups cut by N, K splits (their workspace halved
# in width), the shortest and longest rows they take, and one past each
@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m", [9, 12, 16])
@pytest.mark.parametrize("n,k,small", [(8, 1024, True), (24, 1152, True), (2376, 1024, True),
                                       (264, 6144, True), (2560, 4096, True), (6152, 2176, True),
                                       (40000, 1024, True), (512, 896, False), (264, 6272, False)])
def test_sixteen_row_projections_are_exact(dev, fmt, m, n, k, small):
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    assert native.lib().orinfer_qgemm_small_rows(F.FMT[fmt], m, n, k) == int(small)
    assert not native.lib().orinfer_qgemm_small_rows(F.FMT[fmt], 17, n, k)
    g = torch.Generator().manual_seed(m * n + k)
    codes, ws, w = _int_weight(fmt, n, k, g)
    a = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    sa = torch.rand(m, generator=g) * 0.05 + 1e-3
    want = _scaled(a, sa, w, ws)
    for f32 in (False, True, False):                   # repeated: the workspace is left empty
        out = F.qgemm(a.to(dev), sa.to(dev), codes.to(dev), ws.to(dev), fmt, n, out_f32=f32)
        assert torch.equal(out.cpu(), want if f32 else want.half())


@pytest.mark.parametrize("m", [9, 13, 16])
@pytest.mark.parametrize("n,k", [(97664, 1024), (100008, 1152), (32008, 3200)])
def test_streamed_int8_projections_of_sixteen_rows_are_exact(dev, m, n, k):
    from orinfer_b200.ops import functional as F
    g = torch.Generator(device=dev).manual_seed(m * n + k)
    w = torch.randint(-127, 128, (n, k), generator=g, device=dev, dtype=torch.int8)
    ws = (torch.rand(n, generator=g, device=dev) * 0.01 + 1e-3).half()
    a = torch.randint(-127, 128, (m, k), generator=g, device=dev, dtype=torch.int8)
    sa = torch.rand(m, generator=g, device=dev) * 0.05 + 1e-3
    want = _scaled(a, sa, w, ws)
    for f32 in (False, True) * 5:            # repeated: stages are refilled while others run
        out = F.qgemm(a, sa, w, ws, "w8", n, out_f32=f32)
        assert torch.equal(out, want if f32 else want.half())


# operands that TMA cannot read are refused by the host, on either side of the rule for few rows
@pytest.mark.parametrize("fmt", ["w8", "q4", "q2"])
@pytest.mark.parametrize("m", [9, 16, 17])
@pytest.mark.parametrize("what", ["a", "codes"])
def test_unaligned_operands_of_nine_rows_and_more_are_refused(dev, fmt, m, what):
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    n, k = 2376, 1024
    codes, ws, _ = _int_weight(fmt, n, k, torch.Generator().manual_seed(m))
    a = torch.ones(m, k, dtype=torch.int8)

    def off(t):                                        # eight bytes past a 16-byte boundary
        by = 8 // t.element_size()
        return torch.cat([t.flatten()[:by], t.flatten()]).to(dev)[by:].view(t.shape)

    assert off(a).data_ptr() % 16 == 8 and torch.equal(off(codes).cpu(), codes)
    with pytest.raises(native.KernelError):
        F.qgemm(off(a) if what == "a" else a.to(dev), torch.ones(m, device=dev),
                off(codes) if what == "codes" else codes.to(dev), ws.to(dev), fmt, n)
