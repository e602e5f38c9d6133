"""Recurrent-mixer kernels at the edges of their ranges, against 64-bit statements."""
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


def _recurrence64(q, k, v, g, beta, s):
    o = torch.empty_like(v)
    for i in range(v.shape[0]):
        s = s * torch.exp(g[i])[:, None, None]
        delta = beta[i][:, None] * (v[i] - torch.einsum("hk,hkv->hv", k[i], s))
        s = s + k[i][:, :, None] * delta[:, None, :]
        o[i] = torch.einsum("hk,hkv->hv", q[i], s)
    return o, s


@pytest.mark.parametrize("lens", [[39], [40], [41, 39], [64], [63, 65], [5, 96, 1, 97],
                                  [200, 2, 64, 129], [333]])
@pytest.mark.parametrize("strength", [0.3, 4.0])
def test_gdn_scan_long_and_short_runs(dev, lens, strength):
    """Runs on both sides of the chunked kernel's limit, ragged tails, fresh and continued
    states, mild and very strong decay (running sums of log decays down to several thousand)."""
    from orinfer_b200.ops import functional as F
    torch.manual_seed(sum(lens))
    hk, hv, d = 2, 4, 128
    rows = sum(lens)
    a_log = (torch.randn(hv) * 0.5 + strength).to(dev)
    dt = (torch.randn(hv) * 0.5 - 2).to(dev)
    ab = torch.randn(rows, 2 * hv, device=dev)
    qk = torch.nn.functional.normalize(torch.randn(rows, 2 * hk, d, device=dev), dim=-1)
    v = torch.randn(rows, hv, d, device=dev) * 3
    qkv = torch.cat([qk.reshape(rows, -1), v.reshape(rows, -1)], 1).half()
    state = torch.randn(len(lens) + 2, hv, d, d, device=dev) * 0.2
    start = state.double()
    segs, slot, pos, at = [], [], [], 0
    for i, n in enumerate(lens):
        segs.append([at, n, 0, 0])
        slot += [i + 1] * n
        pos += list(range(0 if i % 2 else 50, (0 if i % 2 else 50) + n))
        at += n
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    out = F.gdn_scan(qkv, ab, a_log, dt, t(segs), len(lens), t(slot), t(pos), hk, hv, d, state)
    q64 = qkv[:, :hk * d].double().reshape(rows, hk, d).repeat_interleave(2, 1) / math.sqrt(d)
    k64 = qkv[:, hk * d:2 * hk * d].double().reshape(rows, hk, d).repeat_interleave(2, 1)
    v64 = qkv[:, 2 * hk * d:].double().reshape(rows, hv, d)
    g = -torch.exp(a_log.double()) * torch.nn.functional.softplus(ab[:, :hv].double() + dt.double(),
                                                                  threshold=60)
    beta = torch.sigmoid(ab[:, hv:].double())
    for i, n in enumerate(lens):
        sl = slice(segs[i][0], segs[i][0] + n)
        s0 = start[i + 1] * (0.0 if i % 2 else 1.0)
        ref, s = _recurrence64(q64[sl], k64[sl], v64[sl], g[sl], beta[sl], s0)
        # FP32 sums and 22-bit splits over at most 333 steps; the decays carry the FP32 rounding
        # of g itself (2^-24 of up to 400 per step, summed over the steps a value lives)
        tol = 1e-5 if strength < 1 else 1e-4
        assert float((out[sl].double() - ref).norm() / ref.norm()) < tol, n
        assert float((state[i + 1].double() - s).norm() / s.norm().clamp(min=1e-9)) < tol, n
    assert torch.equal(state[0].double(), start[0]) and torch.equal(state[-1].double(), start[-1])


@pytest.mark.parametrize("d,hk,hv", [(64, 1, 2), (128, 1, 2), (128, 2, 5), (64, 3, 5)])
@pytest.mark.parametrize("rows,segments", [(5, 5), (37, 3), (4801, 3)])
def test_gdn_conv_forms_agree(dev, d, hk, hv, rows, segments):
    """Eight-channel strips, single rows and the general form give the same rows and history
    as the 64-bit convolution; strips cross run boundaries inside the packet."""
    from orinfer_b200.ops import functional as F
    torch.manual_seed(rows + d)
    conv = (2 * hk + hv) * d
    x = torch.randn(rows, conv + 2 * d, device=dev).half()
    w = (torch.randn(conv, 4, device=dev) * 0.4).half()
    hist = torch.randn(segments, 3, conv, device=dev).half()
    base = rows // segments
    lens = [rows - base * (segments - 1)] + [base] * (segments - 1)
    segs, first, slot, pos, at = [], [], [], [], 0
    for i, n in enumerate(lens):
        p0 = 0 if i == 1 else 9
        segs.append([at, n, 0, 0])
        first += [at] * n
        slot += [i] * n
        pos += list(range(p0, p0 + n))
        at += n
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    args = (t(first), t(slot), t(pos), t(segs), segments, rows, hk, hv, d)
    h_vec, h_gen = hist.clone(), _unaligned(hist)
    y = F.gdn_conv(x, w, h_vec, *args)
    y_gen = F.gdn_conv(_unaligned(x), w, h_gen, *args)
    assert torch.equal(h_vec, h_gen)
    at = 0
    for i, n in enumerate(lens):
        prev = hist[i].double() * (0.0 if i == 1 else 1.0)
        full = torch.cat([prev, x[at:at + n, :conv].double()])
        ref = sum(full[j:j + n] * w[:, j].double() for j in range(4))
        ref = (ref * torch.sigmoid(ref)).half().double()
        qk = ref[:, :2 * hk * d].reshape(n, -1, d)
        ref[:, :2 * hk * d] = (qk * torch.rsqrt((qk * qk).sum(-1, keepdim=True) + 1e-6)).reshape(n, -1)
        # two FP16 roundings; the first may fall the other way (one more step)
        for got in (y[at:at + n], y_gen[at:at + n]):
            assert bool(((got.double() - ref).abs() <= ref.abs() * 2.0 ** -9 + 1e-6).all())
        assert torch.equal(h_vec[i].double(), full[-3:])
        at += n


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("rows,hv", [(1, 1), (3, 5), (130, 4), (384, 4), (700, 3)])
def test_gdn_gated_norm_forms_agree(dev, d, rows, hv):
    from orinfer_b200.ops import functional as F
    torch.manual_seed(rows)
    o = torch.randn(rows, hv, d, device=dev)
    proj = torch.randn(rows, 8 + hv * d, device=dev).half()
    w = (1 + 0.1 * torch.randn(d, device=dev)).half()
    for z in (proj[:, 8:], proj[:, 3:3 + hv * d]):
        for sig in (False, True):
            y = F.gdn_gated_norm(o, z, w, 1e-6, rows, hv, d, sigmoid_gate=sig)
            oo, zz = o.double(), z.double().reshape(rows, hv, d)
            gate = torch.sigmoid(zz) * (1.0 if sig else zz)
            ref = oo * torch.rsqrt((oo * oo).mean(-1, keepdim=True) + 1e-6) * w.double() * gate
            lim = ref.reshape(rows, -1).abs() * 2.0 ** -10 + 1e-7
            assert bool(((y.double() - ref.reshape(rows, -1)).abs() <= lim).all())
            one = F.gdn_gated_norm(o[:1], z[:1], w, 1e-6, 1, hv, d, sigmoid_gate=sig)
            assert torch.equal(one, y[:1])               # a row alone gives the same bits


@pytest.mark.parametrize("d", [64, 128])
def test_gdn_gated_norm_sigmoid_keeps_fp32_accuracy(dev, d):
    """Rows whose norm is exactly one, strongly negative gates and large weights: only the sigmoid
    and its product stand under the FP16 rounding."""
    from orinfer_b200.ops import functional as F
    torch.manual_seed(d)
    rows, hv = 4000, 8
    o = torch.full((rows, hv, d), 4.0, device=dev)
    z = (-19 + 4 * torch.rand(rows, hv * d, device=dev)).half()
    w = (2e4 + 4e4 * torch.rand(d, device=dev)).half()      # products above the subnormals
    for form in (z, _unaligned(z)):
        y = F.gdn_gated_norm(o, form, w, 0.0, rows, hv, d, sigmoid_gate=True).double()
        ref = (torch.sigmoid(z.double().reshape(rows, hv, d)) * w.double()).reshape(rows, -1)
        half_ulp = torch.exp2(torch.floor(torch.log2(ref)) - 11)
        # e^-x within one step (2^-23), then a sum, a reciprocal and a product (2^-24 each); the
        # square root's reciprocal of a power of two within one step
        assert bool(((y - ref).abs() <= half_ulp + ref * 3.5 * 2.0 ** -23).all())


@pytest.mark.parametrize("strength", [-4.0, -1.0])
@pytest.mark.parametrize("spread", [0, 12])
def test_gdn_chunks_keep_fp32_accuracy(dev, strength, spread):
    """Long and medium memory, value channels of equal size and over twelve binades: the chunked
    products against the 64-bit recurrence, channel by channel."""
    from orinfer_b200.ops import functional as F
    torch.manual_seed(7 + spread)
    hk, hv, d, rows = 2, 4, 128, 333
    a_log = (torch.randn(hv) * 0.5 + strength).to(dev)
    dt = (torch.randn(hv) * 0.5 - 2).to(dev)
    ab = torch.randn(rows, 2 * hv, device=dev)
    qk = torch.nn.functional.normalize(torch.randn(rows, 2 * hk, d, device=dev), dim=-1)
    size = torch.exp2(-torch.rand(1, hv, d, device=dev) * spread)
    v = torch.randn(rows, hv, d, device=dev) * size
    qkv = torch.cat([qk.reshape(rows, -1), v.reshape(rows, -1)], 1).half()
    state = torch.randn(1, hv, d, d, device=dev) * 0.2 * size[:, :, None, :]
    s0 = state[0].double()
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    out = F.gdn_scan(qkv, ab, a_log, dt, t([[0, rows, 0, 0]]), 1, t([0] * rows),
                     t(list(range(50, 50 + rows))), hk, hv, d, state)
    part = lambda i: qkv[:, i * hk * d:(i + 1) * hk * d].double().reshape(rows, hk, d)
    g = -torch.exp(a_log.double()) * torch.nn.functional.softplus(ab[:, :hv].double() + dt.double())
    ref, s = _recurrence64(part(0).repeat_interleave(2, 1) / math.sqrt(d),
                           part(1).repeat_interleave(2, 1),
                           qkv[:, 2 * hk * d:].double().reshape(rows, hv, d), g,
                           torch.sigmoid(ab[:, hv:].double()), s0)
    err = lambda x, y, dims: ((x - y).square().sum(dims) / y.square().sum(dims)).sqrt()
    # a handful of FP32 roundings (2^-25 each in the mean) between the inputs and an output
    assert float(err(out.double(), ref, (0,)).mean()) < 2.0 ** -22
    assert float(err(state[0].double(), s, (1,)).mean()) < 2.0 ** -22


@pytest.mark.parametrize("what", ["v_nan", "v_inf", "q_nan", "k_nan", "beta_nan", "decay_zero"])
@pytest.mark.parametrize("row", [1, 13, 40, 94])
def test_gdn_chunks_contain_non_finite_rows(dev, what, row):
    """A run of 100 rows with one non-finite value, or with a log decay of minus infinity: as in
    the recurrence, rows before it and channels beside it do not see it."""
    from orinfer_b200.ops import functional as F
    torch.manual_seed(row)
    hk, hv, d, rows = 2, 4, 128, 100
    a_log = (torch.randn(hv) * 0.5 - 1).to(dev)
    dt = (torch.randn(hv) * 0.5 - 2).to(dev)
    ab = torch.randn(rows, 2 * hv, device=dev)
    qk = torch.nn.functional.normalize(torch.randn(rows, 2 * hk, d, device=dev), dim=-1)
    qkv = torch.cat([qk.reshape(rows, -1), torch.randn(rows, hv * d, device=dev)], 1).half()
    head, channel = 1, 37
    if what[0] == "v":
        qkv[row, 2 * hk * d + head * d + channel] = math.inf if what == "v_inf" else math.nan
    elif what == "q_nan":
        qkv[row, 5] = math.nan
    elif what == "k_nan":
        qkv[row, hk * d + 5] = math.nan
    elif what == "beta_nan":
        ab[row, hv + head] = math.nan
    else:
        ab[row, head] = math.inf                       # softplus and with it the log decay
    state = torch.randn(1, hv, d, d, device=dev) * 0.2
    s0 = state[0].double()
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    out = F.gdn_scan(qkv, ab, a_log, dt, t([[0, rows, 0, 0]]), 1, t([0] * rows),
                     t(list(range(50, 50 + rows))), hk, hv, d, state)
    part = lambda i: qkv[:, i * hk * d:(i + 1) * hk * d].double().reshape(rows, hk, d)
    g = -torch.exp(a_log.double()) * torch.nn.functional.softplus(ab[:, :hv].double() + dt.double())
    ref, s = _recurrence64(part(0).repeat_interleave(2, 1) / math.sqrt(d),
                           part(1).repeat_interleave(2, 1),
                           qkv[:, 2 * hk * d:].double().reshape(rows, hv, d), g,
                           torch.sigmoid(ab[:, hv:].double()), s0)
    for got, want in ((out, ref), (state[0], s)):
        fine = torch.isfinite(want)
        assert torch.equal(torch.isfinite(got), fine)
        diff = (got.double() - want)[fine]
        assert float(diff.norm() / want[fine].norm()) < 1e-6


def _runs(dev, lens, hv, strength, seed):
    """A packet of runs, every other one continued: the arguments of a scan and its 64-bit answer."""
    g = torch.Generator().manual_seed(seed)
    rand = lambda *n: torch.randn(*n, generator=g).to(dev)
    hk, d, rows = max(1, hv // 2), 128, sum(lens)
    a_log, dt = rand(hv) * 0.5 + strength, rand(hv) * 0.5 - 2
    ab = rand(rows, 2 * hv)
    qk = torch.nn.functional.normalize(rand(rows, 2 * hk, d), dim=-1)
    qkv = torch.cat([qk.reshape(rows, -1), rand(rows, hv * d)], 1).half()
    state = rand(len(lens), hv, d, d) * 0.2
    segs, slot, pos, at = [], [], [], 0
    for i, n in enumerate(lens):
        segs.append([at, n, 0, 0])
        slot += [i] * n
        pos += list(range(50 * (i % 2), 50 * (i % 2) + n))
        at += n
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    part = lambda i: qkv[:, i * hk * d:(i + 1) * hk * d].double().reshape(rows, hk, d)
    log_decay = -torch.exp(a_log.double()) * torch.nn.functional.softplus(
        ab[:, :hv].double() + dt.double(), threshold=60)

    def exact(i):
        sl = slice(segs[i][0], segs[i][0] + lens[i])
        return _recurrence64(part(0)[sl].repeat_interleave(hv // hk, 1) / math.sqrt(d),
                             part(1)[sl].repeat_interleave(hv // hk, 1),
                             qkv[sl, 2 * hk * d:].double().reshape(lens[i], hv, d), log_decay[sl],
                             torch.sigmoid(ab[sl, hv:].double()),
                             start[i].double() * (i % 2)) + (sl,)

    start = state.clone()
    args = (qkv, ab, a_log, dt, t(segs), len(lens), t(slot), t(pos), hk, hv, d, state)
    return args, state, exact


# both chunked kernels over the same lengths: alone on their SMs, and with more CTAs than SMs
@pytest.mark.parametrize("n", [40, 63, 64, 65, 95, 97, 129, 257, 383, 384])
@pytest.mark.parametrize("many", [False, True])
def test_gdn_chunked_kernels_over_their_lengths(dev, n, many):
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    hv = 8
    lens = [n, 41] if not many else [n, 41, 64] * 4
    assert native.lib().orinfer_gdn_pipelined(hv, len(lens), sum(lens)) == int(not many)
    args, state, exact = _runs(dev, lens, hv, -1.0, n)
    out = F.gdn_scan(*args)
    for i in range(len(lens)):
        ref, s, sl = exact(i)
        # as in test_gdn_chunks_keep_fp32_accuracy, over a whole run
        assert float((out[sl].double() - ref).norm() / ref.norm()) < 2.0 ** -21
        assert float((state[i].double() - s).norm() / s.norm()) < 2.0 ** -21


# a state and outputs at any FP32 address, in both forms of long runs and the scan
@pytest.mark.parametrize("lens", [[100], [257, 41], [96] * 12, [33]])
@pytest.mark.parametrize("what", ["state", "out"])
def test_gdn_scan_at_any_address(dev, lens, what):
    from orinfer_b200.ops import functional as F

    def off(t):
        return torch.cat([t.flatten()[:1], t.flatten()])[1:].view(t.shape)

    args, state, exact = _runs(dev, lens, 8, -1.0, len(lens))
    out = torch.empty(sum(lens), 8, 128, device=dev)
    if what == "state":
        state = off(state)
    else:
        out = off(out)
    assert (state if what == "state" else out).data_ptr() % 8 == 4
    F.gdn_scan(*args[:-1], state, out=out)
    for i in range(len(lens)):
        ref, s, sl = exact(i)
        # as in test_gdn_chunks_keep_fp32_accuracy, over a whole run
        assert float((out[sl].double() - ref).norm() / ref.norm()) < 2.0 ** -21
        assert float((state[i].double() - s).norm() / s.norm()) < 2.0 ** -21


@pytest.mark.parametrize("row", [3, 45, 95])
def test_gdn_many_runs_contain_non_finite_rows(dev, row):
    from orinfer_b200.ops import functional as F
    lens = [96] * 12
    args, state, _ = _runs(dev, lens, 8, -1.0, row)
    fine = F.gdn_scan(*[a.clone() if torch.is_tensor(a) else a for a in args])
    args[0][96 * 5 + row, 2 * 4 * 128 + 2 * 128 + 9] = math.inf           # a value of run 5, head 2
    out = F.gdn_scan(*args)
    bad = torch.zeros_like(out, dtype=torch.bool)
    bad[96 * 5 + row:96 * 6, 2, 9] = True
    assert torch.equal(torch.isfinite(out), ~bad)
    # the sums of its warp are made in another order
    assert float((out - fine)[~bad].norm() / fine[~bad].norm()) < 1e-6


# small elements of a state beside large ones that a chunk's rows overwrite with changing signs, so
# that a bound of the state stands far above it: rows of queries that read the small ones alone
@pytest.mark.parametrize("n", [64, 200])
@pytest.mark.parametrize("small", [2.0 ** -8, 2.0 ** -16])
def test_gdn_small_elements_of_a_state_keep_their_bits(dev, n, small):
    from orinfer_b200.ops import functional as F
    from orinfer_b200.ops import native
    hv, d = 2, 128
    assert native.lib().orinfer_gdn_pipelined(hv, 1, n)
    g = torch.Generator().manual_seed(n)
    q, k, v = torch.zeros(n, 1, d), torch.zeros(n, 1, d), torch.ones(n, hv, d)
    q[..., 2:] = torch.nn.functional.normalize(torch.randn(n, 1, d - 2, generator=g), dim=-1)
    k[..., 1] = 1
    v[1::2] = -1
    qkv = torch.cat([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1)], 1).half().to(dev)
    state = torch.randn(1, hv, d, d, generator=g) * small
    state[:, :, :2] = 1
    state = state.to(dev)
    s0 = state[0].double()
    ab = torch.randn(n, 2 * hv, generator=g).to(dev)
    ab[:, hv:] = 3.0
    a_log, dt = torch.full((hv,), -5.0, device=dev), torch.zeros(hv, device=dev)
    t = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    out = F.gdn_scan(qkv, ab, a_log, dt, t([[0, n, 0, 0]]), 1, t([0] * n),
                     t(list(range(9, 9 + n))), 1, hv, d, state)
    part = lambda i: qkv[:, i * d:(i + 1) * d].double().reshape(n, 1, d).repeat_interleave(hv, 1)
    decay = -torch.exp(a_log.double()) * torch.nn.functional.softplus(ab[:, :hv].double())
    ref, s = _recurrence64(part(0) / math.sqrt(d), part(1),
                           qkv[:, 2 * d:].double().reshape(n, hv, d), decay,
                           torch.sigmoid(ab[:, hv:].double()), s0)
    # as in test_gdn_chunks_keep_fp32_accuracy, over a whole run
    assert float((out.double() - ref).norm() / ref.norm()) < 2.0 ** -20
    assert float((state[0].double() - s).norm() / s.norm()) < 2.0 ** -20


def test_gdn_keys_of_any_size(dev):
    """The state is scaled by a bound that takes the keys' size into account."""
    from orinfer_b200.ops import functional as F
    for size in (2.0 ** -6, 0.5, 1.4):               # above sqrt(2) the recurrence itself diverges
        args, state, exact = _runs(dev, [150], 4, -1.0, 3)
        args[0][:, 2 * 128:4 * 128] *= size
        out = F.gdn_scan(*args)
        ref, s, sl = exact(0)
        assert float((out.double() - ref).norm() / ref.norm()) < 2.0 ** -20
        assert float((state[0].double() - s).norm() / s.norm()) < 2.0 ** -20


# strips of one row, of a few, and as many as fit the machine, with runs that begin anywhere in one
@pytest.mark.parametrize("rows", [1, 73, 75, 149, 297, 1187])
@pytest.mark.parametrize("hk,hv", [(1, 2), (8, 24)])
def test_gdn_conv_strips(dev, rows, hk, hv):
    from orinfer_b200.ops import functional as F
    g = torch.Generator().manual_seed(rows + hk)
    d, conv = 128, (2 * hk + hv) * 128
    x = (torch.randn(rows, conv + 64, generator=g) * 2).half().to(dev)
    w = (torch.randn(conv, 4, generator=g) * 0.4).half().to(dev)
    lens = [n for n in (rows // 3, 1, 2, rows - rows // 3 - 3) if n > 0] if rows > 6 else [rows]
    hist = torch.randn(len(lens), 3, conv, generator=g).half().to(dev)
    segs, first, slot, pos, at = [], [], [], [], 0
    for i, n in enumerate(lens):
        segs.append([at, n, 0, 0])
        first += [at] * n
        slot += [i] * n
        pos += list(range(7 * (i % 2), 7 * (i % 2) + n))
        at += n
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    args = (t(first), t(slot), t(pos), t(segs), len(lens), rows, hk, hv, d)
    y = F.gdn_conv(x, w, hist.clone(), *args)
    y_gen = F.gdn_conv(_unaligned(x), w, hist.clone(), *args)
    for (at, n, _, _), h, i in zip(segs, hist, range(len(lens))):
        full = torch.cat([h.double() * (i % 2), x[at:at + n, :conv].double()])
        ref = sum(full[j:j + n] * w[:, j].double() for j in range(4))
        ref = (ref * torch.sigmoid(ref)).half().double()
        qk = ref[:, :2 * hk * d].reshape(n, -1, d)
        ref[:, :2 * hk * d] = (qk * torch.rsqrt((qk * qk).sum(-1, keepdim=True) + 1e-6)).reshape(n, -1)
        for got in (y, y_gen):                        # as in test_gdn_conv_forms_agree
            assert bool(((got[at:at + n].double() - ref).abs() <= ref.abs() * 2.0 ** -9 + 1e-6).all())


def test_gdn_gates_and_values_at_the_ends_of_their_range(dev):
    """Infinities, NaNs and arguments whose exponential leaves FP32, in the two-value sigmoid."""
    from orinfer_b200.ops import functional as F
    z = torch.tensor([math.inf, -math.inf, math.nan, 0.0, 60000.0, -60000.0, -87.0, -89.0, 89.0,
                      -20.0, 20.0, -104.0], device=dev).half()
    rows, hv, d = 400, 4, 128
    proj = z.repeat(rows, 43)[:, :hv * d].contiguous()
    o = torch.ones(rows, hv, d, device=dev)
    w = torch.full((d,), 4.0, device=dev).half()
    for sig in (True, False):
        y = F.gdn_gated_norm(o, proj, w, 0.0, rows, hv, d, sigmoid_gate=sig)
        zz = proj.double()
        ref = (torch.sigmoid(zz) * (1.0 if sig else zz) * 4).half()
        got, want = y.double(), ref.double()
        if not sig:                                   # minus infinity times a sigmoid of zero
            want = torch.where(proj == -math.inf, math.nan, want)
        same = (got == want) | (got.isnan() & want.isnan()) | ((got - want).abs() <= want.abs() * 2.0 ** -10)
        assert bool(same.all()), (proj[~same][:4], got[~same][:4], want[~same][:4])


def test_both_sigmoids_keep_their_accuracy(dev):
    """Every 61st float between 2^-30 and 87 of both signs, against 64 bits."""
    from orinfer_b200.ops import native
    bits = torch.arange(0x30800000, 0x42AE0000, 61, dtype=torch.int32, device=dev)
    x = bits.view(torch.float32)
    x = torch.cat([x, -x, torch.tensor([0.0, -0.0], device=dev)])
    one, pair = torch.empty_like(x), torch.empty_like(x)
    run = lambda n: native.check(native.lib().orinfer_sigmoids(
        x.data_ptr(), one.data_ptr(), pair.data_ptr(), n, torch.cuda.current_stream().cuda_stream), "")
    run(x.numel())
    want = torch.sigmoid(x.double())
    rel = lambda got: float(((got.double() - want) / want).abs().max())
    # half a step of the result, one and a half of the exponential and its argument's rounding
    assert rel(pair) < 2.0 ** -22.3 and rel(one) < 2.0 ** -22.1, (rel(pair), rel(one))
    x[:8] = torch.tensor([-87.5, -88.5, -90.0, -110.0, -1e30, -math.inf, math.inf, math.nan], device=dev)
    run(8)
    for got in (one, pair):
        assert bool((got[:6].abs() <= 2.0 ** -125).all()) and float(got[6]) == 1 and got[7].isnan()


# how often an FP16 value of the convolution is not the correctly rounded one
def test_gdn_conv_values_are_rounded_as_the_sigmoid_allows(dev):
    from orinfer_b200.ops import functional as F
    g = torch.Generator(device=dev).manual_seed(7)
    rows, hk, hv, d = 2000, 1, 30, 128
    conv = (2 * hk + hv) * d
    x = torch.randn(rows, conv, generator=g, device=dev).half()
    w = (torch.randn(conv, 4, generator=g, device=dev) * 0.3).half()
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    y = F.gdn_conv(x, w, torch.zeros(1, 3, conv, device=dev).half(), t([0] * rows), t([0] * rows),
                   t(list(range(rows))), t([[0, rows, 0, 0]]), 1, rows, hk, hv, d)
    full = torch.cat([torch.zeros(3, conv, device=dev), x]).double()
    acc = sum(full[j:j + rows] * w[:, j].double() for j in range(4))
    want = (acc * torch.sigmoid(acc)).half()
    off = (y != want)[:, 2 * hk * d:].double().mean()
    # a value is off if it lies nearer to a tie than its error: steps of 2^-10 to 2^-11 of the value
    # and errors of 2^-23 to 2^-22 (four products, the sigmoid, a product)
    assert 0 < float(off) < 2.0 ** -12
