"""The kernels that a rule on sizes or alignment chooses, at the edges of their tiles, against the general kernel of
the same operation (bit for bit where the sums have the same order) or a float64 reference."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.0 ** -24  # half a unit in the last place of float32


@pytest.fixture(scope="module")
def ops32():
    from fastgen_b200.csrc.ops import Ops
    return Ops(torch.float32, DEV)


@pytest.fixture(scope="module")
def ops16():
    from fastgen_b200.csrc.ops import Ops
    return Ops(torch.bfloat16, DEV)


def _randn(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(DEV)


# -- the float32 product ----------------------------------------------------------------------------

@pytest.mark.parametrize("m,n,k", [
    (1, 16, 4), (7, 17, 132), (8, 2051, 128), (8, 40, 1028),           # few rows, a row a lane
    (9, 33, 100), (31, 200, 2048), (33, 5120, 36), (64, 15, 260),      # few rows, four a lane
    (9, 5200, 36), (24, 5300, 68), (32, 9001, 32),                     # small blocks of 2, 3 and 4 warps
    (65, 64, 4), (97, 65, 100), (160, 2047, 64), (321, 63, 33 * 4), (64, 9000, 36),  # small blocks of 4
    (65, 7001, 32), (200, 5121, 40), (777, 2050, 28),                  # 128 columns by 3, 4 and 6 warps
    (33, 28672, 36), (49, 28672, 36), (57, 28672, 36),                 # ... by 5, 7 and 8
    (33, 37889, 16), (65, 19201, 20), (777, 3100, 36),                 # 64 x 128 tiles
])
def test_float32_product_routes(ops32, m, n, k):
    """Every kernel gives the bits of the general one (taken for rows that are no multiple of 16 bytes)."""
    g = torch.Generator().manual_seed(m * 7 + n)
    x, w, bias = _randn(g, m, k), _randn(g, n, k), _randn(g, n)
    odd_x, odd_w = torch.empty(m, k + 1, device=DEV)[:, :k], torch.empty(n, k + 3, device=DEV)[:, :k]
    odd_x.copy_(x)
    odd_w.copy_(w)
    got, want = ops32.linear(x, w), ops32.linear(odd_x, odd_w)
    assert torch.equal(got, want)
    assert torch.equal(ops32.linear(x, w, bias=bias), ops32.linear(odd_x, odd_w, bias=bias))
    wide = torch.full((m, n + 5), 3.0, device=DEV)  # rows of the result that are no multiple of 16 bytes
    ops32.linear(x, w, out=wide[:, :n])
    assert torch.equal(wide[:, :n], want) and bool((wide[:, n:] == 3.0).all())
    ref = x.double() @ w.double().T
    bound = k * EPS * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - ref).abs() <= bound + 1e-30).all())


@pytest.mark.parametrize("m,n,k", [
    (1, 1024, 1024), (16, 1025, 1028), (5, 2100, 8192),                  # one tile of 16 rows, shared by 8, 8 and 4 blocks
    (9, 9000, 1024), (3, 37889, 1024),                                   # ... by 2, and a tile to a block
    (17, 2050, 1100), (32, 10241, 1024), (32, 60000, 1024),              # a tile of 32
    (33, 1024, 1024), (64, 19000, 1088),                                 # of 64
    (65, 1024, 2052), (113, 1500, 1028), (225, 9600, 1024),              # of 112
    (160, 19000, 1028), (400, 5121, 1024),                               # of 160
])
def test_float32_product_on_tensor_cores(ops32, m, n, k):
    """Weights from 1,024 x 1,024 on: no further from float64 than the multiply-adds of the general kernel, the same bits for
    a row whatever is beside it (other rows, other tiles, other numbers of blocks), and its infinities and NaNs."""
    g = torch.Generator().manual_seed(m * 5 + n)
    x, w, bias = _randn(g, m, k), _randn(g, n, k), _randn(g, n)
    odd_x = torch.empty(m, k + 1, device=DEV)[:, :k]  # rows off 16 bytes: the general kernel
    odd_x.copy_(x)
    got, other = ops32.linear(x, w), ops32.linear(odd_x, w)
    ref = x.double() @ w.double().T
    assert bool(((got.double() - ref).abs() <= k * EPS * (x.double().abs() @ w.double().abs().T)).all())
    assert _relative(got, ref) <= _relative(other, ref)
    for row in (0, m // 2, m - 1):
        assert torch.equal(ops32.linear(x[row : row + 1], w)[0], got[row])
    assert torch.equal(ops32.linear(x[: min(m, 40)], w), got[:40])
    assert torch.equal(ops32.linear(x, w, bias=bias), got + bias)
    wide = torch.full((m, n + 5), 3.0, device=DEV)
    ops32.linear(x, w, out=wide[:, :n])
    assert torch.equal(wide[:, :n], got) and bool((wide[:, n:] == 3.0).all())
    x[0, 3], x[m // 2, 1], w[n - 1, k - 1], w[7, 5] = float("inf"), float("nan"), -float("inf"), 3e38
    x[m - 1, :] *= 2.0
    odd_x.copy_(x)
    got, other = ops32.linear(x, w), ops32.linear(odd_x, w)
    finite = torch.isfinite(other)
    assert torch.equal(torch.isnan(got), torch.isnan(other)) and torch.equal(torch.isposinf(got), torch.isposinf(other))
    assert torch.equal(torch.isfinite(got), finite) and int(ops32.status.flatten()[0]) == 0
    bound = 2 * k * EPS * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - other.double()).abs() <= bound)[finite].all())


@pytest.mark.parametrize("m,n,k", [(5, 1100, 1024), (20, 1024, 2052), (300, 1500, 1028), (700, 19000, 1024)])
def test_float32_product_of_few_or_unusual_numbers(ops32, m, n, k):
    """Rows of few numbers that are not zero, of numbers at either end of float32's range and of very different ones: no further
    from float64 than the multiply-adds of the general kernel."""
    g = torch.Generator().manual_seed(m + k)
    x, w = _randn(g, m, k), _randn(g, n, k)
    odd = torch.empty(m, k + 1, device=DEV)[:, :k]  # rows off 16 bytes: the general kernel

    def both(x, w):
        odd.copy_(x)
        return ops32.linear(x, w), ops32.linear(odd, w)

    for count in (1, 2, 4, 8, 32):
        at = torch.stack([torch.randperm(k, generator=g)[:count] for _ in range(m)]).to(DEV)
        few = torch.zeros_like(x).scatter_(1, at, x.gather(1, at))
        got, other = both(few, w)
        ref = few.double() @ w.double().T
        # With z numbers, none in the segment of another, z segments and their z - 1 sums are rounded, of multiply-adds z
        # results: sqrt(2) of the error at most, and longer chains of multiply-adds make up for it.  The three products of
        # parts left out come to 2^-24 of a product at most, a fifth of a rounding on average.
        assert _relative(got, ref) <= (2.0 ** 0.5 if count < 32 else 1.0) * _relative(other, ref), count
        if count == 1:
            assert bool(((got.double() - ref).abs() <= (2 + 2.0 ** -6) * EPS * ref.abs()).all())
    mixed = x * torch.exp2(torch.randint(-40, 41, (m, k), generator=g).float()).to(DEV)
    for scaled, weights in ((x * 2.0 ** -120, w * 2.0 ** 100), (x * 2.0 ** 100, w * 2.0 ** -125), (x * 2.0 ** -130, w * 2.0 ** 120),
                            (x.abs() * 2.0 ** -118, w.abs() * 2.0 ** 90), (mixed, w)):
        got, other = both(scaled, weights)
        ref = scaled.double() @ weights.double().T
        assert _relative(got, ref) <= _relative(other, ref) * (1.0 if scaled is not mixed else 2.0 ** 0.5)
    # results below float32's normal range: one rounding to their spacing, the general kernel's are many
    got, other = both(x * 2.0 ** -70, w * 2.0 ** -72)
    ref = (x * 2.0 ** -70).double() @ (w * 2.0 ** -72).double().T
    assert bool(((got.double() - ref).abs() <= 2.0 ** -149).all())
    # numbers that the split does not take (2^111 and more): the general kernel's bits
    got, other = both(x * 2.0 ** 112, w * 2.0 ** -20)
    large = ((x * 2.0 ** 112).abs() >= 2.0 ** 112).any(1)
    assert bool(large.any()) and torch.equal(got[large], other[large]) and bool(torch.isfinite(got).all())
    assert int(ops32.status.flatten()[0]) == 0


@pytest.mark.parametrize("m,n,k", [(5, 1100, 8192), (3, 37889, 1024), (32, 1024, 1100), (40, 19000, 1088), (113, 1500, 14336), (777, 4100, 2048)])
def test_float32_product_of_an_infinite_column(ops32, m, n, k):
    """An infinity in every row: all elements are computed again, behind the block's waits; the general kernel's bits."""
    g = torch.Generator().manual_seed(m * 3 + n)
    x, w, bias = _randn(g, m, k), _randn(g, n, k), _randn(g, n)
    x[:, k // 3], w[n // 2, k // 3] = float("inf"), 0.0
    bias[1] = float("-inf")
    odd_x = torch.empty(m, k + 1, device=DEV)[:, :k]
    odd_x.copy_(x)
    wide = torch.full((m, n + 5), 3.0, device=DEV)
    bits = lambda v: v.contiguous().view(torch.int32)
    for b in (None, bias):
        want = ops32.linear(odd_x, w, bias=b)
        assert torch.equal(bits(ops32.linear(x, w, bias=b)), bits(want)) and not bool(torch.isfinite(want).any())
        ops32.linear(x, w, bias=b, out=wide[:, :n])
        assert torch.equal(bits(wide[:, :n]), bits(want)) and bool((wide[:, n:] == 3.0).all())
    assert int(ops32.status.flatten()[0]) == 0


def _relative(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


# -- convolution, gate and norms -----------------------------------------------------------------------

def _sequences(lengths, pad=0, slots=None):
    """A step's arrays for sequences of these lengths, ``pad`` tokens of slot -1 behind them."""
    slots = slots or list(range(len(lengths)))
    req, start = [], [0]
    for n, s in zip(lengths, slots):
        req += [s] * n
        start.append(start[-1] + n)
    to = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return SimpleNamespace(req=to(req + [-1] * pad), seq_slot=to(slots), seq_start=to(start), n_seqs=len(lengths),
                           n_tokens=len(req) + pad)


@pytest.mark.parametrize("act", ["silu", None])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths,pad", [([1], 0), ([2, 3, 1, 1], 2), ([40], 0), ([11, 1, 8, 30], 5), ([3, 8, 9, 64], 0)])
def test_convolution_four_channels_at_a_time(ops32, ops16, dtype, lengths, pad, act):
    """Aligned channels against the same channels one column further (the kernel of one channel a thread)."""
    ops = ops32 if dtype == torch.float32 else ops16
    channels, taps = 136, 4
    ctx = _sequences(lengths, pad, slots=list(range(1, len(lengths) + 1)))
    g = torch.Generator().manual_seed(sum(lengths))
    t = ctx.n_tokens
    rows = _randn(g, t, channels).to(dtype)
    w, bias = _randn(g, channels, taps), _randn(g, channels)
    state = _randn(g, len(lengths) + 2, 8 + (taps - 1) * channels)
    outs = []
    for shift in (0, 1):
        proj = torch.zeros(t, channels + 4, dtype=dtype, device=DEV)
        proj[:, shift : shift + channels] = rows
        st = state.clone()
        out = ops.time_conv(proj, shift, channels, w, bias, st, 8, taps, ctx, act=act, out_dtype=dtype)
        live = ctx.req >= 0
        outs.append((out[live], st))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("part,parts", [(128, 3), (256, 1), (512, 8), (1024, 2), (96, 2), (640, 1)])
def test_gate_and_norm_in_parts(ops32, ops16, dtype, part, parts):
    ops = ops32 if dtype == torch.float32 else ops16
    ctx = _sequences([5, 12], 2)
    t, width = ctx.n_tokens, part * parts
    g = torch.Generator().manual_seed(part)
    y, w = _randn(g, t, width), 1 + _randn(g, width, scale=0.1)
    proj = _randn(g, t, width + 24).to(dtype)
    z = proj[:, 8 : 8 + width]
    got = ops.gated_part_norm(y, z, w, parts, 1e-5, ctx)[:17].double()
    v = (y.double() * torch.nn.functional.silu(z.double())).reshape(t, parts, part)
    ref = (v * torch.rsqrt((v * v).mean(-1, keepdim=True) + 1e-5)).reshape(t, width) * w.double()
    ref = ref[:17]
    # float32: the sum of squares and a handful of operations; bfloat16: one rounding more
    rel = (part + 16) * EPS + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert bool(((got - ref).abs() <= rel * ref.abs() + 1e-6).all())


@pytest.mark.parametrize("kind", ["layer", "rms"])
@pytest.mark.parametrize("streams,dim", [(1, 4), (2, 2047), (2, 2048), (3, 2049), (4, 4096), (2, 4097), (5, 100)])
def test_stream_norm_rows_in_registers(ops32, streams, dim, kind):
    g = torch.Generator().manual_seed(dim + streams)
    t = 5
    h, delta = _randn(g, t, streams, dim), _randn(g, t, dim).to(torch.bfloat16)
    mix, oc, ic = torch.rand(streams, streams, generator=g).to(DEV), torch.rand(streams, generator=g).to(DEV), torch.rand(streams, generator=g).to(DEV)
    w, b = 1 + _randn(g, dim, scale=0.1), _randn(g, dim, scale=0.1)
    want = torch.einsum("ast,nsd->ntd", mix.double()[None], h.double()) + oc.double()[:, None] * delta.double()[:, None]
    u = (ic.double()[:, None] * want).sum(1)
    if kind == "layer":
        c = u - u.mean(-1, keepdim=True)
        ref = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-5) * w.double() + b.double()
    else:
        ref = u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-5) * w.double()
    out = torch.empty(t, dim, dtype=torch.float32, device=DEV)
    rows = torch.tensor([3, 0], dtype=torch.int32, device=DEV)
    some = torch.empty(2, dim, dtype=torch.float32, device=DEV)
    args = dict(delta=delta, mix=mix, out_coef=oc, in_coef=ic, bias=b if kind == "layer" else None, eps=1e-5, rms=kind == "rms")
    _stream_norm(ops32, h, w, some, rows=rows, **args)
    _stream_norm(ops32, h, w, out, **args)
    bound = (dim + 32) * EPS
    assert float((h.double() - want).abs().max()) <= 8 * EPS * float(want.abs().max()) * (streams + 1)
    assert float((out.double() - ref).abs().max()) <= bound * float(ref.abs().max())
    assert torch.equal(some, out[rows.long()])


@pytest.mark.parametrize("streams,dim", [(1, 1535), (1, 1536), (2, 1023), (2, 1280), (2, 2560), (2, 3585), (3, 1024), (4, 1793), (4, 2049)])
def test_stream_norm_routes_by_rows(ops32, streams, dim):
    """Few rows and many take different kernels at these sizes: the same bits for a row."""
    g = torch.Generator().manual_seed(dim + streams)
    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    h, delta = _randn(g, n, streams, dim), _randn(g, n, dim).to(torch.bfloat16)
    mix, oc, ic = torch.rand(streams, streams, generator=g).to(DEV), torch.rand(streams, generator=g).to(DEV), torch.rand(streams, generator=g).to(DEV)
    w, b = 1 + _randn(g, dim, scale=0.1), _randn(g, dim, scale=0.1)
    args = dict(mix=mix, out_coef=oc, in_coef=ic, bias=b, eps=1e-5, rms=False)
    many, few = h.clone(), h[:7].clone()
    outs = [torch.empty(x.shape[0], dim, dtype=torch.float32, device=DEV) for x in (many, few)]
    for x, out in zip((many, few), outs):
        _stream_norm(ops32, x, w, out, delta=delta[: x.shape[0]], **args)
    assert torch.equal(outs[0][:7], outs[1]) and torch.equal(many[:7], few)


def _stream_norm(ops, h, w, out, delta, mix, out_coef, in_coef, bias, eps, rms, rows=None):
    from fastgen_b200.csrc.ops import _check, _code, _ptr, _stream
    n = out.shape[0]
    _check(ops.lib, ops.lib.fg_stream_norm(_ptr(h), h.shape[1], _ptr(delta), _code(delta.dtype), _ptr(mix), _ptr(out_coef),
                                           _ptr(in_coef), _ptr(w), _ptr(bias), _ptr(out), _code(out.dtype), _ptr(rows), n,
                                           h.shape[2], eps, int(rms), _stream()))


# -- block tables ----------------------------------------------------------------------------------------

@pytest.mark.parametrize("n", [1, 480, 481, 1300])
def test_table_entries_in_launch_arguments(ops32, n):
    g = torch.Generator().manual_seed(n)
    table = torch.randint(0, 99, (7, 300), generator=g, dtype=torch.int32).to(DEV)
    want = table.clone()
    at = torch.randperm(table.numel(), generator=g)[:n]
    value = torch.randint(-1, 1 << 20, (n,), generator=g, dtype=torch.int32)
    want.view(-1)[at.to(DEV)] = value.to(DEV)
    ops32.set_table_entries(table, at.numpy(), value.numpy())
    assert torch.equal(table, want)


# -- attention ----------------------------------------------------------------------------------------------

def _attention_step(lengths, cached, page, heads, kv, hd, dtype, seed):
    """Queries of sequences that bring ``lengths`` tokens behind ``cached`` ones, and pools that hold random entries."""
    from fastgen_b200.engine.step import StepContext
    g = torch.Generator().manual_seed(seed)
    width = max(-(-(c + n) // page) for c, n in zip(cached, lengths))
    n_pages = width * len(lengths) + 3
    order = torch.randperm(n_pages, generator=g)[: width * len(lengths)].reshape(len(lengths), width)
    ctx = StepContext(torch.device(DEV))
    ctx.host_seq_slot, ctx.host_seq_cached = list(range(len(lengths))), list(cached)
    ctx.host_seq_start = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    pos = [c + i for c, n in zip(cached, lengths) for i in range(n)]
    ctx.pos = torch.tensor(pos, dtype=torch.int32, device=DEV)
    ctx.n_tokens, ctx.n_seqs = len(pos), len(lengths)
    q = _randn(g, len(pos), heads * hd).to(dtype)
    pools = [_randn(g, n_pages, kv, page, hd).to(dtype) for _ in range(2)]
    return ctx, q, pools, order.to(DEV, torch.int32)


@pytest.mark.parametrize("hd,heads,kv", [(64, 8, 2), (16, 3, 3), (48, 20, 1), (160, 4, 2), (256, 4, 2)])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 0), (40, 5), (-37, 0)])
def test_float32_attention_on_asynchronous_copies(ops32, hd, heads, kv, window, keep):
    """The bits of the kernel that loads a number at a time (taken for pools that do not start on 16 bytes)."""
    from fastgen_b200.csrc.ops import SIMT_ROWS, _check, _code, _ptr, _stream, attention_tiling, attn
    ctx, q, pools, table = _attention_step([1, 33, 7], [130, 0, 31], 8, heads, kv, hd, torch.float32, hd + window)
    sinks = torch.linspace(-1, 1, heads, device=DEV)
    tiles = ctx.attention_tiles(attention_tiling(heads, kv, SIMT_ROWS), 1)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = []
    for shift in (0, 1):
        moved = []
        for pool in pools:
            room = torch.empty(pool.numel() + 4, device=DEV)
            moved.append(room[shift : shift + pool.numel()].view(pool.shape))
            moved[-1].copy_(pool)
        out = torch.full_like(q, float("nan"))
        lib = attn(hd)
        _check(lib, lib.fg_attention_simt(
            _ptr(q), q.stride(0), _ptr(out), out.stride(0), _code(q.dtype), _ptr(moved[0]), _ptr(moved[1]), _ptr(table),
            table.shape[1], 8, pools[0].shape[0], _ptr(ctx.pos), _ptr(tiles.req), _ptr(tiles.tok0), _ptr(tiles.ntok), tiles.n,
            heads, kv, hd, window, keep, hd ** -0.5, 3.0 if keep else 0.0, _ptr(sinks), _ptr(status), _stream()))
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0]).all()) and int(status) == 0


@pytest.mark.parametrize("hd,heads,kv", [(64, 8, 2), (16, 3, 3), (48, 20, 1), (128, 9, 3), (256, 4, 2), (80, 1, 1)])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 0), (40, 5), (300, 70), (-37, 0)])
def test_float32_attention_by_tokens(ops32, hd, heads, kv, window, keep):
    """Prompts in tiles of 64 rows and single tokens eight tiles at a time, beside each other: the bits of the kernel that
    walks 16 rows (taken for pools off 16 bytes), and what lies behind a row's keys never reaches it."""
    from types import SimpleNamespace
    ctx, q, pools, table = _attention_step([1, 130, 1, 7, 1, 1, 2], [0, 0, 700, 31, 255, 31, 330], 16, heads, kv, hd,
                                           torch.float32, hd + window)
    slots = [s for s, n in zip(ctx.host_seq_slot, torch.tensor(ctx.host_seq_start).diff().tolist()) for _ in range(n)]
    ctx.req = torch.tensor(slots, dtype=torch.int32, device=DEV)
    how = dict(window=max(window, 0) or None, scale=hd ** -0.5, keep_first=keep, softcap=3.0 if keep == 5 else None,
               sinks=torch.linspace(-1, 1, heads, device=DEV) if window else None, chunk=-window if window < 0 else None)
    outs = []
    for shift in (0, 1):
        moved = []
        for pool in pools:
            room = torch.empty(pool.numel() + 4, device=DEV)
            moved.append(room[shift : shift + pool.numel()].view(pool.shape))
            moved[-1].copy_(pool)
        memory = SimpleNamespace(k_pages=moved[0], v_pages=moved[1], block_table=table, page_size=16)
        out = torch.full_like(q, float("nan"))
        ops32.attention(q, out, memory, ctx, heads, kv, hd, **how)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0]).all()) and int(ops32.status) == 0
    if hd > 128:
        return  # (such prompts stay on the kernel of 16 rows)
    # the entry of position 129 of the request of 130 tokens: only its last token sees it
    moved[0][int(table[1, 8]), :, 1], moved[1][int(table[1, 8]), :, 1] = float("nan"), float("inf")
    aligned = [p.clone() for p in moved]
    memory = SimpleNamespace(k_pages=aligned[0], v_pages=aligned[1], block_table=table, page_size=16)
    again = torch.empty_like(q)
    ops32.attention(q, again, memory, ctx, heads, kv, hd, **how)
    keepers = torch.ones(q.shape[0], dtype=torch.bool, device=DEV)
    keepers[130] = False
    assert torch.equal(again[keepers], outs[0][keepers]) and not bool(torch.isfinite(again[130]).all())


@pytest.mark.parametrize("hd,heads,kv", [(64, 8, 2), (16, 3, 3), (48, 20, 1), (128, 9, 3)])
@pytest.mark.parametrize("window,keep", [(0, 0), (40, 5), (300, 70), (-37, 0)])
def test_float32_prompts_in_tiles_of_16_and_of_64_rows(ops32, hd, heads, kv, window, keep):
    """Both kernels of prompts on the same steps, few and many tokens: the same bits, and what lies behind a row's keys reaches
    neither; the rule takes blocks of 16 rows where 64 rows would leave SMs idle or be mostly empty."""
    from fastgen_b200.csrc.ops import F32_PROMPT_ROWS, SIMT_ROWS, _check, _code, _ptr, _stream, attention_tiling, attn
    lib, sms = attn(hd), torch.cuda.get_device_properties(0).multi_processor_count
    tiling = {rows: attention_tiling(heads, kv, rows) for rows in (SIMT_ROWS, F32_PROMPT_ROWS)}
    assert lib.fg_attention_f32_prompt_rows(sms // kv // 2, 1, heads, kv) == SIMT_ROWS
    assert lib.fg_attention_f32_prompt_rows(8 * sms, 2 * sms, heads, kv) == F32_PROMPT_ROWS
    assert lib.fg_attention_f32_prompt_rows(8 * sms, 8 * sms, heads, kv) == (SIMT_ROWS if heads // kv <= 16 else F32_PROMPT_ROWS)
    for lengths, cached in (([2, 3, 9, 16, 17], [130, 0, 31, 700, 5]), ([64, 63, 65, 200], [0, 330, 31, 12])):
        ctx, q, pools, table = _attention_step(lengths, cached, 16, heads, kv, hd, torch.float32, hd + window)
        sinks = torch.linspace(-1, 1, heads, device=DEV)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)

        def run(rows):
            tiles = ctx.attention_tiles(tiling[rows], 2)
            assert ctx.count_tiles(tiling[rows], 2) == tiles.n
            out = torch.full_like(q, 3.0)
            kernel, dtype = (lib.fg_attention_simt, (_code(q.dtype),)) if rows == SIMT_ROWS else (lib.fg_attention_f32_prompt, ())
            _check(lib, kernel(
                _ptr(q), q.stride(0), _ptr(out), out.stride(0), *dtype, _ptr(pools[0]), _ptr(pools[1]), _ptr(table),
                table.shape[1], 16, pools[0].shape[0], _ptr(ctx.pos), _ptr(tiles.req), _ptr(tiles.tok0), _ptr(tiles.ntok), tiles.n,
                heads, kv, hd, window, keep, hd ** -0.5, 3.0 if keep == 5 else 0.0, _ptr(sinks), _ptr(status), _stream()))
            return out

        few, many = run(SIMT_ROWS), run(F32_PROMPT_ROWS)
        assert torch.equal(few, many) and bool(torch.isfinite(few).all())
        last = cached[-1] + lengths[-1] - 1  # only the last token sees its entry
        page, place = int(table[-1, last // 16]), last % 16
        pools[0][page, :, place], pools[1][page, :, place] = float("nan"), float("inf")
        again = [run(rows) for rows in (SIMT_ROWS, F32_PROMPT_ROWS)]
        assert all(torch.equal(v[:-1], few[:-1]) and not bool(torch.isfinite(v[-1]).any()) for v in again) and int(status) == 0


@pytest.mark.parametrize("hd,heads,kv,n", [
    (64, 32, 8, 18), (64, 32, 8, 19), (64, 32, 8, 55), (64, 32, 8, 56), (64, 20, 4, 140),  # runs of 8, 4, 4, 2 and 2 tiles
    (16, 9, 3, 99), (16, 9, 3, 400), (32, 5, 5, 140), (48, 40, 5, 90), (48, 40, 5, 130), (80, 24, 24, 13), (80, 24, 24, 20),
    (128, 32, 8, 40), (160, 8, 4, 80), (256, 4, 2, 90)])
@pytest.mark.parametrize("window,keep", [(0, 0), (100, 40), (-37, 0)])
def test_float32_single_tokens_by_their_number(ops32, hd, heads, kv, n, window, keep):
    """More blocks than fit the chip at once walk their keys in shorter runs: the bits of the kernel that walks tile after tile
    (taken for pools off 16 bytes), padding tokens zeroed."""
    from fastgen_b200.engine.step import SingleTokens
    ctx, q, pools, table = _attention_step([1] * n, [(37 * i) % 90 + 300 * (i % 7 == 3) for i in range(n)], 16, heads, kv, hd,
                                           torch.float32, hd + n)
    ctx.req = torch.arange(n, dtype=torch.int32, device=DEV)
    how = dict(window=max(window, 0) or None, scale=hd ** -0.5, keep_first=keep, softcap=3.0 if keep else None,
               sinks=torch.linspace(-1, 1, heads, device=DEV) if window else None, chunk=-window if window < 0 else None)
    outs = []
    for shift in (0, 1):
        moved = []
        for pool in pools:
            room = torch.empty(pool.numel() + 4, device=DEV)
            moved.append(room[shift : shift + pool.numel()].view(pool.shape))
            moved[-1].copy_(pool)
        memory = SimpleNamespace(k_pages=moved[0], v_pages=moved[1], block_table=table, page_size=16)
        out = torch.full_like(q, float("nan"))
        ops32.attention(q, out, memory, ctx, heads, kv, hd, **how)
        outs.append(out)
        if shift == 0:  # as in a captured step: the last token belongs to no request
            padded = torch.full_like(q, float("nan"))
            ctx.req[-1] = -1
            ctx._singles = SingleTokens(ctx.req.clone(), torch.arange(n, dtype=torch.int32, device=DEV), n, 400)
            ops32.attention(q, padded, memory, ctx, heads, kv, hd, **how)
            ctx._singles, ctx.req[-1] = None, n - 1
    assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0]).all()) and int(ops32.status) == 0
    assert torch.equal(padded[:-1], outs[0][:-1]) and not bool(padded[-1].any())


@pytest.mark.parametrize("page", [8, 64, 128])
@pytest.mark.parametrize("keep,window", [(1, 64), (4, 100), (70, 130), (200, 65)])
def test_kept_positions_in_the_tensor_memory_kernel(ops16, keep, window, page):
    """Prompt portions against a float64 reference; pages between the kept positions and the window are given back."""
    from fastgen_b200.cache.manager import LayerMemory
    heads, kv, hd = 8, 2, 64
    lengths, cached = [200, 3, 64], [0, 390, 130]
    ctx, q, pools, table = _attention_step(lengths, cached, page, heads, kv, hd, torch.bfloat16, keep + page)
    keys = []
    for i, (n, c) in enumerate(zip(lengths, cached)):
        rows = [torch.cat([p[int(t)] for t in table[i]], dim=1)[:, : c + n].double() for p in pools]  # [kv, keys, hd]
        keys.append(rows)
        first, kept = max(0, c - window + 1) // page, -(-keep // page)
        table[i, kept:first] = -1
    memory = LayerMemory(k_pages=pools[0], v_pages=pools[1], block_table=table, page_size=page,
                         tensor_maps=ops16.make_kv_tensor_maps(pools[0][None], pools[1][None], page), layer_index=0)
    out = torch.empty_like(q)
    ops16.attention(q, out, memory, ctx, heads, kv, hd, window, hd ** -0.5, keep_first=keep)
    ops16.check_status()
    for i, (n, c) in enumerate(zip(lengths, cached)):
        a = ctx.host_seq_start[i]
        qq = q[a : a + n].double().reshape(n, heads, hd)
        k, v = (r.repeat_interleave(heads // kv, 0) for r in keys[i])
        s = torch.einsum("thd,hkd->htk", qq, k) * hd ** -0.5
        p, j = torch.arange(c, c + n, device=DEV)[:, None], torch.arange(c + n, device=DEV)[None, :]
        seen = (j <= p) & ((p - j < window) | (j < keep))
        ref = torch.einsum("htk,hkd->thd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), v)
        # probabilities and outputs are rounded to bfloat16 (2^-8 each)
        assert _relative(out[a : a + n], ref.reshape(n, heads * hd)) <= 2.0 ** -7


@pytest.mark.parametrize("hd,length,cached,window,keep", [(64, 700, 0, 300, 4), (64, 90, 1500, 1024, 70), (128, 333, 200, 128, 64)])
@pytest.mark.parametrize("deviation", [0.8, 3.0])
def test_kept_positions_lose_no_precision(ops16, hd, length, cached, window, keep, deviation):
    """Against float64, and no further from it than the mma.sync kernel on the same inputs (with sharp scores
    a weight of almost one that is rounded on its own counts)."""
    from fastgen_b200.cache.manager import LayerMemory
    from fastgen_b200.csrc.ops import Ops
    heads, kv, page = 16, 4, 64
    other = Ops(torch.bfloat16, DEV)
    other.use_tcgen05 = False
    ctx, q, pools, table = _attention_step([length], [cached], page, heads, kv, hd, torch.bfloat16, hd + keep)
    q = (q.float() * deviation).to(torch.bfloat16)
    memory = LayerMemory(k_pages=pools[0], v_pages=pools[1], block_table=table, page_size=page,
                         tensor_maps=ops16.make_kv_tensor_maps(pools[0][None], pools[1][None], page), layer_index=0)
    k, v = (torch.cat([p[int(t)] for t in table[0]], dim=1)[:, : cached + length].double().repeat_interleave(heads // kv, 0)
            for p in pools)
    s = torch.einsum("thd,hkd->htk", q.double().reshape(length, heads, hd), k) * hd ** -0.5
    p, j = torch.arange(cached, cached + length, device=DEV)[:, None], torch.arange(cached + length, device=DEV)[None, :]
    seen = (j <= p) & ((p - j < window) | (j < keep))
    ref = torch.einsum("htk,hkd->thd", torch.softmax(s.masked_fill(~seen, float("-inf")), -1), v).reshape(length, -1)
    errors = []
    for ops in (ops16, other):
        out = torch.empty_like(q)
        ops.attention(q, out, memory, ctx, heads, kv, hd, window, hd ** -0.5, keep_first=keep)
        ops.check_status()
        errors.append(_relative(out, ref))
    # Both round the same weights and outputs: their errors are means over the same 90,000 or more values, equal to
    # 1 % (a tile's maximum is found at other places of the walk).
    assert errors[0] <= 1.01 * errors[1]


def _attention_reference(q, pools, table, heads, kv, hd, cached, seen, sinks=None):
    """One sequence's queries in float64; ``seen`` [queries, keys]."""
    n, keys = seen.shape
    k, v = (torch.cat([p[int(t)] for t in table], dim=1)[:, :keys].double().repeat_interleave(heads // kv, 0) for p in pools)
    s = (torch.einsum("thd,hkd->htk", q.double().reshape(n, heads, hd), k) * hd ** -0.5).masked_fill(~seen, float("-inf"))
    if sinks is not None:
        s = torch.cat([s, sinks.double()[:, None, None].expand(heads, n, 1)], -1)
    w = torch.softmax(s, -1)[..., :keys]
    return torch.einsum("htk,hkd->thd", w, v).reshape(n, heads * hd)


# tiles of 64 keys, the kept ones, then the window's, in parts of equal length of eight tiles or more
@pytest.mark.parametrize("keep,window,length", [
    (4, 1100, 40),     # 1 + 19 tiles in two parts
    (600, 1100, 40),   # 10 + 19 in three parts of ten: the second begins at the seam
    (640, 600, 30),    # 10 + 11 in two parts: the seam lies inside the first
    (1250, 400, 7),    # 20 + 7 in three parts: inside the last
])
@pytest.mark.parametrize("hd,page,with_sinks", [(64, 16, False), (64, 128, True), (128, 64, True), (128, 128, False)])
def test_kept_positions_of_items_in_parts(ops16, hd, page, with_sinks, keep, window, length):
    """A few tokens on a long context: their items are worked on in parts, which start at any of their tiles."""
    from fastgen_b200.cache.manager import LayerMemory
    heads, kv, cached = 4, 2, 3000
    ctx, q, pools, table = _attention_step([length], [cached], page, heads, kv, hd, torch.bfloat16, keep + hd)
    whole = table.clone()
    table[0, -(-keep // page) : (cached - window + 1) // page] = -1
    sinks = torch.linspace(0, 6, heads, device=DEV) if with_sinks else None
    memory = LayerMemory(k_pages=pools[0], v_pages=pools[1], block_table=table, page_size=page,
                         tensor_maps=ops16.make_kv_tensor_maps(pools[0][None], pools[1][None], page), layer_index=0)
    ops16._split.pop(hd, None)  # so that the flags hold nothing of an earlier launch
    out = torch.empty_like(q)
    ops16.attention(q, out, memory, ctx, heads, kv, hd, window, hd ** -0.5, keep_first=keep, sinks=sinks)
    ops16.check_status()
    flags = ops16._split[hd][1].view(-1, 2)
    assert int(flags[:, 1].max()) >= 2 and not bool(flags[:, 0].any())  # parts of an item; all of them counted
    p, j = torch.arange(cached, cached + length, device=DEV)[:, None], torch.arange(cached + length, device=DEV)[None, :]
    seen = (j <= p) & ((p - j < window) | (j < keep))
    ref = _attention_reference(q, pools, whole[0], heads, kv, hd, cached, seen, sinks)
    # probabilities and outputs are rounded to bfloat16 (2^-8 each)
    assert _relative(out, ref) <= 2.0 ** -7


@pytest.mark.parametrize("hd,heads,kv,page", [(64, 20, 4, 64), (128, 24, 8, 16), (48, 20, 5, 8)])
@pytest.mark.parametrize("form", ["whole", "window", "kept", "chunk", "sinks", "turned"])
def test_merge_of_splits_in_half_blocks(ops16, hd, heads, kv, page, form):
    """Single tokens of more heads x requests than full blocks are resident at once: the bits of the same requests a few
    at a time, and padding lanes between them stay untouched."""
    from fastgen_b200.cache.manager import LayerMemory
    from fastgen_b200.engine.step import SingleTokens
    n = 42
    g = torch.Generator().manual_seed(hd)
    cached = [int(x) for x in torch.randint(0, 1400, (n,), generator=g)]
    cached[:6] = [0, 127, 128, 255, 256, 1399]  # on both sides of where splits of 128 keys begin
    ctx, q, pools, table = _attention_step([1] * n, cached, page, heads, kv, hd, torch.bfloat16, hd + 1)
    memory = LayerMemory(k_pages=pools[0], v_pages=pools[1], block_table=table, page_size=page,
                         tensor_maps=ops16.make_kv_tensor_maps(pools[0][None], pools[1][None], page), layer_index=0)
    kw = dict(window=dict(window=300), kept=dict(window=300, keep_first=5), chunk=dict(window=None, chunk=500),
              sinks=dict(window=None, sinks=torch.linspace(-2, 4, heads, device=DEV)),
              turned=dict(window=None, out_freqs=torch.linspace(0.01, 1, hd // 2, device=DEV)), whole=dict(window=None))[form]

    def run(lanes):
        """Outputs of the requests in ``lanes`` (None: a padding lane, whose token index is any row's)."""
        out = torch.full_like(q, 7.0)
        to = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        singles = SingleTokens(to([-1 if i is None else i for i in lanes]), to([0 if i is None else i for i in lanes]),
                               len(lanes), 1400, None, n * 1400)
        ctx.single_tokens = lambda: singles
        ops16.attention(q, out, memory, ctx, heads, kv, hd, scale=hd ** -0.5, **kw)
        ops16.check_status()
        return out

    lanes = [i for k in range(n) for i in ((None, k) if k % 5 == 2 else (k,))]
    assert heads * len(lanes) > 592 and heads * 6 < 592
    together = run(lanes)
    for a in range(0, n, 6):
        few = run(list(range(a, a + 6)))
        assert torch.equal(together[a : a + 6], few[a : a + 6])
        assert bool((few[a + 6 :] == 7.0).all()) and bool((few[:a] == 7.0).all())
    assert bool((run(lanes[:20])[20:] == 7.0).all())
    if form in ("whole", "window", "sinks"):
        for i in (0, 1, 5, 30):
            c = cached[i]
            seen = torch.arange(c + 1, device=DEV)[None, :] > c - kw["window"] if kw["window"] else torch.ones(1, c + 1, dtype=torch.bool, device=DEV)
            ref = _attention_reference(q[i : i + 1], pools, table[i], heads, kv, hd, c, seen, kw.get("sinks"))
            assert _relative(together[i : i + 1], ref) <= 2.0 ** -7


def test_rotation_and_attention_start_early(ops16):
    """Projection, rotation with the page write, and single-token attention as programmatic launches behind one another in
    a graph, where splits that end before the new position are read while the rotation runs: the bits of the same
    launches with a wait after each.  New positions at both ends of splits of 128 keys and of pages."""
    from fastgen_b200.cache.manager import LayerMemory
    from fastgen_b200.engine.step import SingleTokens
    heads, kv, hd, page, n, dim = 8, 2, 64, 64, 8, 512
    first = [0, 63, 64, 127, 128, 129, 255, 511]
    steps = 3
    ctx, _, pools, table = _attention_step([steps] * n, first, page, heads, kv, hd, torch.bfloat16, 3)
    g = torch.Generator().manual_seed(4)
    w = _randn(g, (heads + 2 * kv) * hd, dim, scale=dim ** -0.5).to(torch.bfloat16)
    xs = [_randn(g, n + 1, dim).to(torch.bfloat16) for _ in range(steps)]
    freqs = torch.linspace(1, 0.01, hd // 2, device=DEV)
    to = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    req = to(list(range(n)) + [-1])  # (the last token is padding)
    singles = SingleTokens(req, to(list(range(n + 1))), n + 1, 1024, None, n * 1024)
    ctx.single_tokens = lambda: singles
    ctx.attention_tiles = lambda tpt, least=1: SimpleNamespace(n=0)

    def layer(x, out, pos, pool, wait):
        ctx.pos = pos
        memory = LayerMemory(k_pages=pool[0], v_pages=pool[1], block_table=table, page_size=page,
                             tensor_maps=ops16.make_kv_tensor_maps(pool[0][None], pool[1][None], page), layer_index=0)
        qkv = ops16.linear(x, w)
        wait()
        q, k, v = qkv[:, : heads * hd], qkv[:, heads * hd : (heads + kv) * hd], qkv[:, (heads + kv) * hd :]
        ops16.rope_kv_write(q, k, v, pos, req, freqs, pool[0], pool[1], table, page, heads, kv, hd)
        wait()
        ops16.attention(q, out, memory, ctx, heads, kv, hd, None, hd ** -0.5)
        wait()

    results = []
    for graph in (False, True):
        pool = [p.clone() for p in pools]
        x, out, pos = xs[0].clone(), torch.zeros(n + 1, heads * hd, dtype=torch.bfloat16, device=DEV), to(first + [0])
        if graph:
            layer(x, out, to([c for c in first] + [0]), [p.clone() for p in pool], lambda: None)  # loads and sizes
            stream, replay = torch.cuda.Stream(), torch.cuda.CUDAGraph()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                replay.capture_begin()
                layer(x, out, pos, pool, lambda: None)
                replay.capture_end()
            torch.cuda.current_stream().wait_stream(stream)
        got = []
        for s in range(steps):
            x.copy_(xs[s])
            pos.copy_(to([c + s for c in first] + [0]))
            replay.replay() if graph else layer(x, out, pos, pool, torch.cuda.synchronize)
            got.append(out[:n].clone())
        ops16.check_status()
        results.append(got + pool)
    assert all(torch.equal(a, b) for a, b in zip(*results))


def _graph_against_waits(ops, run, inputs, keep):
    """``run(wait)`` step by step with ``inputs`` (pairs of a buffer and its contents a step): launches with a wait after each
    against one graph of them, from the same ``keep`` (buffers that steps change); the results and buffers of both."""
    first, results = [k.clone() for k in keep], []
    for graph in (False, True):
        if graph:
            stream, replay = torch.cuda.Stream(), torch.cuda.CUDAGraph()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                replay.capture_begin()
                out = run(lambda: None)
                replay.capture_end()
            torch.cuda.current_stream().wait_stream(stream)
        for k, v in zip(keep, first):
            k.copy_(v)
        got = []
        for step in range(len(inputs[0][1])):
            for buffer, contents in inputs:
                buffer.copy_(contents[step])
            if graph:
                replay.replay()
            else:
                out = run(torch.cuda.synchronize)
            got.append(out.clone())
        ops.check_status()
        results.append(got + [k.clone() for k in keep])
    return results


def test_state_space_layers_start_early(ops16):
    """Projection, convolution, its state, the recurrence and the gated norm of two layers as programmatic launches behind one
    another in a graph: the bits of the same launches with a wait after each."""
    heads, groups, n_state, p, dim, taps, n = 8, 2, 128, 64, 512, 4, 5
    inner, channels, floats = heads * p, heads * p + 2 * groups * n_state, heads * n_state * p
    ctx = _sequences([1] * n, slots=[3, 0, -1, 4, 1])
    ctx.longest, ctx.req = 1, ctx.seq_slot
    g = torch.Generator().manual_seed(8)
    layers = [SimpleNamespace(
        w_in=_randn(g, inner + channels + heads, dim, scale=dim ** -0.5).to(torch.bfloat16),
        wo=_randn(g, dim, inner, scale=inner ** -0.5).to(torch.bfloat16),
        conv=_randn(g, channels, taps, scale=0.5), bias=_randn(g, channels), dt_bias=torch.rand(heads, generator=g).to(DEV) * 3.5 - 3,
        a_log=torch.rand(heads, generator=g).to(DEV) * 2.5 - 1, d=_randn(g, heads), norm=1 + _randn(g, inner, scale=0.1),
        state=_randn(g, 6, floats + (taps - 1) * channels)) for _ in range(2)]
    x = torch.zeros(n, dim, dtype=torch.bfloat16, device=DEV)

    def run(wait):
        h = x
        for l in layers:
            proj = ops16.linear(h, l.w_in)
            wait()
            xbc = ops16.mamba2_conv(proj, inner, channels, l.conv, l.bias, l.state, floats, taps, ctx)
            wait()
            y = ops16.mamba2_scan(xbc, proj, inner + channels, l.dt_bias, l.a_log, l.d, l.state, ctx, heads, groups, n_state, p)
            wait()
            h = ops16.linear(ops16.gated_part_norm(y, proj[:, :inner], l.norm, groups, 1e-5, ctx), l.wo)
            wait()
        return h

    xs = [_randn(g, n, dim).to(torch.bfloat16) for _ in range(6)]
    live = ctx.req >= 0
    a, b = _graph_against_waits(ops16, run, [(x, xs)], [l.state for l in layers])
    assert all(torch.equal(u[live] if u.shape[0] == n else u, v[live] if v.shape[0] == n else v) for u, v in zip(a, b))


def _latent_step(g, first, page, width, entry):
    """Single tokens at the positions ``first`` and one of no request, and a pool of random entries."""
    from fastgen_b200.engine.step import AttentionTiles
    n, n_pages = len(first), len(first) * width + 2
    to = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    req, tok = to(list(range(n)) + [-1]), to(list(range(n + 1)))
    ctx = SimpleNamespace(req=req, pos=to(first + [0]), n_tokens=n + 1, n_seqs=n + 1)
    ctx.attention_tiles = lambda tpt, least=1: AttentionTiles(req, tok, torch.ones_like(req), n + 1)
    table = torch.randperm(n_pages, generator=g)[: n * width].reshape(n, width).to(DEV, torch.int32)
    pool = _randn(g, n_pages, 1, page, entry).to(torch.bfloat16)
    return ctx, SimpleNamespace(k_pages=pool, block_table=table, page_size=page)


def test_latent_layers_start_early(ops16):
    """Projection, cache entry and query norm, query projection, rotation, attention in stretches and their merge, two layers
    behind one another in a graph: the bits of the same launches with a wait after each."""
    R, r, heads, hd, q_rank, dim, page = 256, 32, 8, 64, 128, 512, 16
    g = torch.Generator().manual_seed(9)
    first = [0, 15, 16, 63, 200, 330]
    n, qk = len(first), hd + r
    layers = []
    for _ in range(2):
        ctx, memory = _latent_step(g, first, page, 22, R + r)
        layers.append(SimpleNamespace(
            memory=memory, down=_randn(g, q_rank + R + r, dim, scale=dim ** -0.5).to(torch.bfloat16),
            up=_randn(g, heads * qk, q_rank, scale=q_rank ** -0.5).to(torch.bfloat16),
            uk=_randn(g, heads, hd, R, scale=hd ** -0.5).to(torch.bfloat16), qn=1 + _randn(g, q_rank, scale=0.1),
            kn=1 + _randn(g, R, scale=0.1), back=_randn(g, dim, heads * R, scale=R ** -0.5).to(torch.bfloat16)))
    freqs = torch.linspace(1, 0.01, r // 2, device=DEV)
    x = torch.zeros(n + 1, dim, dtype=torch.bfloat16, device=DEV)
    lat = torch.zeros(n + 1, heads, R, dtype=torch.bfloat16, device=DEV)

    def run(wait):
        h = x
        for l in layers:
            down = ops16.linear(h, l.down)
            wait()
            q = ops16.latent_prepare(down[:, q_rank:], l.kn, 1e-5, freqs, 1.0, l.memory, ctx, R, r, down[:, :q_rank], q_norm=l.qn,
                                     n_heads=heads, head_size=qk)
            wait()
            q = ops16.linear(q, l.up)
            wait()
            ops16.rotate_part(q, ctx, freqs, 1.0, heads, qk, hd, r)
            wait()
            q = q.view(n + 1, heads, qk)
            qa = ops16.head_products(q[:, :, :hd], l.uk)
            wait()
            ops16.latent_attention(qa, q[:, :, hd:], lat.permute(1, 0, 2), None, l.memory, ctx, heads, R, r, qk ** -0.5)
            wait()
            h = ops16.linear(lat.view(n + 1, heads * R), l.back)
            wait()
        return h

    steps = 6
    xs = [_randn(g, n + 1, dim).to(torch.bfloat16) for _ in range(steps)]
    pos = [torch.tensor([f + s for f in first] + [0], dtype=torch.int32, device=DEV) for s in range(steps)]
    a, b = _graph_against_waits(ops16, run, [(x, xs), (ctx.pos, pos)], [l.memory.k_pages for l in layers])
    assert all(torch.equal(u[:n] if u.shape[0] == n + 1 else u, v[:n] if v.shape[0] == n + 1 else v) for u, v in zip(a, b))
    assert all(bool(torch.isfinite(u[:n]).all()) for u in a[:steps])


@pytest.mark.parametrize("rank,rot", [(256, 32), (512, 64), (256, 0)])
@pytest.mark.parametrize("tokens", [1, 3])
def test_latent_queries_off_16_bytes(ops16, rank, rot, tokens):
    """Queries whose rows lie on 16 bytes are copied in pieces of 16, others in pieces of 4: the same bits."""
    heads, page, n = 6, 16, 5
    g = torch.Generator().manual_seed(rank + rot + tokens)
    cached = [0, 15, 40, 129, 200]
    ctx, _, pools, table = _attention_step([tokens] * n, cached, page, 1, 1, rank + rot, torch.bfloat16, rank + tokens)
    memory = SimpleNamespace(k_pages=pools[0], block_table=table, page_size=page)
    t = n * tokens
    qa, qt = _randn(g, heads, t, rank).to(torch.bfloat16), _randn(g, t, heads, rot).to(torch.bfloat16)
    outs = []
    for a_shift, t_shift in ((0, 0), (2, 0), (0, 6), (4, 2)):
        wide_a = torch.full((heads, t, rank + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
        wide_t = torch.full((t, heads, rot + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
        wide_a[:, :, a_shift : a_shift + rank], wide_t[:, :, t_shift : t_shift + rot] = qa, qt
        out = torch.full((heads, t, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops16.latent_attention(wide_a[:, :, a_shift : a_shift + rank], wide_t[:, :, t_shift : t_shift + rot], out, None, memory, ctx,
                               heads, rank, rot, rank ** -0.5)
        ops16.check_status()
        outs.append(out)
    assert bool(torch.isfinite(outs[0]).all()) and all(torch.equal(o, outs[0]) for o in outs[1:])


# -- recurrences, chunk by chunk ---------------------------------------------------------------------------

LENGTHS = [([64], 0), ([65, 1, 63], 3), ([95, 96, 97], 0), ([2, 130, 64], 1), ([20, 30], 14), ([300], 0),
           ([111, 112, 113], 0), ([127, 128, 129], 1), ([79], 80), ([80], 79), ([95, 96], 96)]


@pytest.mark.parametrize("n_state,p", [(128, 64), (64, 40), (128, 4)])
@pytest.mark.parametrize("lengths,pad", LENGTHS)
def test_state_space_recurrence(ops16, lengths, pad, n_state, p):
    """Sequences on both sides of the length from which chunks are walked, in one step."""
    heads, groups = 6, 2
    slots = [3, 0, 2][: len(lengths)]
    ctx = _sequences(lengths, pad, slots)
    t = ctx.n_tokens
    g = torch.Generator().manual_seed(sum(lengths) + p)
    inner, bc = heads * p, groups * n_state
    xbc = _randn(g, t, inner + 2 * bc, scale=0.5)
    proj = _randn(g, t, 16 + heads).to(torch.bfloat16)
    dt_bias, a_log = torch.rand(heads, generator=g).to(DEV) * 3.5 - 3, torch.rand(heads, generator=g).to(DEV) * 2.5 - 1
    d = _randn(g, heads)
    state = _randn(g, 5, heads * n_state * p + 12)
    before = state.clone()
    y = ops16.mamba2_scan(xbc, proj, 16, dt_bias, a_log, d, state, ctx, heads, groups, n_state, p)
    per = heads // groups
    for i, (n, slot) in enumerate(zip(lengths, slots)):
        a = int(ctx.seq_start[i])
        rows = xbc[a : a + n].double()
        x = rows[:, :inner].reshape(n, heads, p)
        b = rows[:, inner : inner + bc].reshape(n, groups, n_state).repeat_interleave(per, 1)
        c = rows[:, inner + bc :].reshape(n, groups, n_state).repeat_interleave(per, 1)
        dt = torch.nn.functional.softplus(proj[a : a + n, 16:].double() + dt_bias.double(), threshold=1e9)
        decay = torch.exp(-torch.exp(a_log.double()) * dt)
        S = before[slot, : heads * n_state * p].double().reshape(heads, p, n_state).clone()
        ref = torch.empty(n, heads, p, dtype=torch.float64, device=DEV)
        for s in range(n):
            S = decay[s][:, None, None] * S + (dt[s][:, None] * x[s])[:, :, None] * b[s][:, None, :]
            ref[s] = (S * c[s][:, None, :]).sum(-1) + d.double()[:, None] * x[s]
        bound = (n_state + 2 * 32 + 64) * EPS  # the sums of a row and of a chunk, the decays of a chunk
        assert _relative(y[a : a + n], ref.reshape(n, inner)) <= bound
        assert _relative(state[slot, : heads * n_state * p], S.reshape(-1)) <= bound
        assert torch.equal(state[slot, heads * n_state * p :], before[slot, heads * n_state * p :])
    for slot in {0, 1, 2, 3, 4} - set(slots):
        assert torch.equal(state[slot], before[slot])


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 31, 45, 64, 99])
def test_state_space_chunks_are_causal(ops16, at, value):
    """A number that is not finite changes nothing before its token, and no other column at all."""
    heads, groups, n_state, p, n = 4, 2, 128, 40, 150
    ctx = _sequences([n, 130], 2)
    g = torch.Generator().manual_seed(at)
    inner, bc = heads * p, groups * n_state
    xbc = _randn(g, ctx.n_tokens, inner + 2 * bc, scale=0.5)
    proj = _randn(g, ctx.n_tokens, 16 + heads).to(torch.bfloat16)
    dt_bias, a_log, d = torch.rand(heads, generator=g).to(DEV) - 1, torch.rand(heads, generator=g).to(DEV) - 1, _randn(g, heads)
    column = 2 * p + 35
    outs, states = [], []
    for x in (None, value):
        rows, state = xbc.clone(), torch.zeros(2, heads * n_state * p, device=DEV)
        if x is not None:
            rows[at, column] = x
        outs.append(ops16.mamba2_scan(rows, proj, 16, dt_bias, a_log, d, state, ctx, heads, groups, n_state, p))
        states.append(state)
    want, got = outs
    other = torch.ones(inner, dtype=torch.bool, device=DEV)
    other[column] = False
    # (a chunk that holds such a number sums in another order)
    assert torch.allclose(got[:n, other], want[:n, other], rtol=0, atol=2e-5)
    assert torch.allclose(got[:at, column], want[:at, column], rtol=0, atol=2e-5)
    assert not bool(torch.isfinite(got[at:n, column]).any())
    assert torch.equal(got[n : n + 130], want[n : n + 130]) and torch.equal(states[0][1], states[1][1])
    finite = torch.isfinite(states[1][0].view(heads * p, n_state)).all(1)
    assert bool(finite[other].all()) and not bool(finite[column])


def _portions(n, most=63):
    """The cut of ``n`` tokens into portions that the token kernels take."""
    return [(a, min(a + most, n)) for a in range(0, n, most)]


@pytest.mark.parametrize("n_state,p", [(128, 64), (64, 64)])
def test_state_space_chunks_lose_no_precision(ops16, n_state, p):
    """One long sequence whole (chunks) and in portions of 63 tokens (the token kernel) against float64."""
    heads, groups, n = 64, 8, 600
    g = torch.Generator().manual_seed(n_state)
    inner, bc = heads * p, groups * n_state
    xbc = _randn(g, n, inner + 2 * bc, scale=0.5)
    proj = _randn(g, n, 16 + heads).to(torch.bfloat16)
    dt_bias, a_log = torch.rand(heads, generator=g).to(DEV) * 3.5 - 3, torch.rand(heads, generator=g).to(DEV) * 2.5 - 1
    d, first = _randn(g, heads), _randn(g, 1, heads * n_state * p)
    per, rows = heads // groups, xbc.double()
    x = rows[:, :inner].reshape(n, heads, p)
    b = rows[:, inner : inner + bc].reshape(n, groups, n_state).repeat_interleave(per, 1)
    c = rows[:, inner + bc :].reshape(n, groups, n_state).repeat_interleave(per, 1)
    dt = torch.nn.functional.softplus(proj[:, 16:].double() + dt_bias.double(), threshold=1e9)
    decay = torch.exp(-torch.exp(a_log.double()) * dt)
    S = first.double().reshape(heads, p, n_state).clone()
    ref = torch.empty(n, heads, p, dtype=torch.float64, device=DEV)
    for s in range(n):
        S = decay[s][:, None, None] * S + (dt[s][:, None] * x[s])[:, :, None] * b[s][:, None, :]
        ref[s] = (S * c[s][:, None, :]).sum(-1) + d.double()[:, None] * x[s]
    errors = []
    for cuts in ([(0, n)], _portions(n)):
        state = first.clone()
        y = torch.cat([ops16.mamba2_scan(xbc[a:z], proj[a:z], 16, dt_bias, a_log, d, state, _sequences([z - a]), heads, groups,
                                         n_state, p) for a, z in cuts])
        errors.append((_relative(y, ref.reshape(n, inner)), _relative(state, S.reshape(1, -1))))
    # means over 64 heads, whose decays (rounded alike on both sides) differ: equal to a few per cent
    assert errors[0][0] <= 1.05 * errors[1][0] and errors[0][1] <= 1.05 * errors[1][1], errors


@pytest.mark.parametrize("d,dv", [(64, 64), (40, 24), (128, 12), (100, 130)])
@pytest.mark.parametrize("lengths,pad", LENGTHS)
def test_delta_rule_with_one_decay_a_head(ops16, lengths, pad, d, dv):
    heads, kv = 4, 2
    slots = [1, 3, 0][: len(lengths)]
    ctx = _sequences(lengths, pad, slots)
    t = ctx.n_tokens
    g = torch.Generator().manual_seed(sum(lengths) + d)
    qkv = _randn(g, t, 2 * kv * d + heads * dv)
    proj = _randn(g, t, 2 * heads).to(torch.bfloat16)
    a, b = proj[:, :heads], proj[:, heads:]
    dt_bias, a_log = torch.rand(heads, generator=g).to(DEV) * 3.5 - 3, torch.rand(heads, generator=g).to(DEV) * 2.5 - 2
    state = _randn(g, 4, heads * d * dv + 8, scale=0.3)
    before = state.clone()
    out = ops16.delta_scan(qkv, a, b, dt_bias, a_log, state, ctx, heads, kv, d, dv, head_decay=True)
    for i, (n, slot) in enumerate(zip(lengths, slots)):
        o = int(ctx.seq_start[i])
        rows = qkv[o : o + n].double()
        q = rows[:, : kv * d].reshape(n, kv, d).repeat_interleave(heads // kv, 1)
        k = rows[:, kv * d : 2 * kv * d].reshape(n, kv, d).repeat_interleave(heads // kv, 1)
        v = rows[:, 2 * kv * d :].reshape(n, heads, dv)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        gate = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a[o : o + n].double() + dt_bias.double(), threshold=1e9))
        beta = torch.sigmoid(b[o : o + n].double())
        S = before[slot, : heads * d * dv].double().reshape(heads, dv, d).clone()
        ref = torch.empty(n, heads, dv, dtype=torch.float64, device=DEV)
        for s in range(n):
            S = gate[s][:, None, None] * S
            u = beta[s][:, None] * (v[s] - (S * k[s][:, None, :]).sum(-1))
            S = S + u[:, :, None] * k[s][:, None, :]
            ref[s] = (S * q[s][:, None, :]).sum(-1)
        bound = (2 * d + 4 * 32 + 64) * EPS  # a row's sums, the chunk's triangular system and its decays
        assert _relative(out[o : o + n], ref.reshape(n, heads * dv)) <= bound
        assert _relative(state[slot, : heads * d * dv], S.reshape(-1)) <= bound
    for slot in {0, 1, 2, 3} - set(slots):
        assert torch.equal(state[slot], before[slot])


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("part", ["v", "k", "q"])
@pytest.mark.parametrize("at", [0, 31, 45, 99])
def test_delta_chunks_are_causal(ops16, at, part, value):
    """A number that is not finite changes nothing before its token, and nothing of other columns (a value's) or heads."""
    heads, kv, d, dv, n = 4, 2, 64, 40, 150
    ctx = _sequences([n, 130], 2)
    g = torch.Generator().manual_seed(at)
    qkv = _randn(g, ctx.n_tokens, 2 * kv * d + heads * dv)
    proj = _randn(g, ctx.n_tokens, 2 * heads).to(torch.bfloat16)
    a, b = proj[:, :heads], proj[:, heads:]
    dt_bias, a_log = torch.rand(heads, generator=g).to(DEV) - 1, torch.rand(heads, generator=g).to(DEV) - 1
    # the second value head's 7th value, or the first key head's 5th key or query
    column = {"v": 2 * kv * d + dv + 7, "k": kv * d + 5, "q": 5}[part]
    hit = torch.zeros(heads, dv, dtype=torch.bool, device=DEV)
    if part == "v":
        hit[1, 7] = True
    else:
        hit[:2] = True
    hit = hit.view(-1)
    outs = []
    for x in (None, value):
        rows, state = qkv.clone(), torch.zeros(2, heads * d * dv, device=DEV)
        if x is not None:
            rows[at, column] = x
        outs.append(ops16.delta_scan(rows, a, b, dt_bias, a_log, state, ctx, heads, kv, d, dv, head_decay=True))
    want, got = outs
    assert torch.allclose(got[:n, ~hit], want[:n, ~hit], rtol=0, atol=2e-6)
    assert torch.allclose(got[:at, hit], want[:at, hit], rtol=0, atol=2e-6)
    bad = got[at:n, hit] if part != "q" else got[at, hit]
    assert not bool(torch.isfinite(bad).any())
    if part == "q":
        assert torch.allclose(got[at + 1 : n, hit], want[at + 1 : n, hit], rtol=0, atol=2e-6)
    assert torch.equal(got[n : n + 130], want[n : n + 130])


@pytest.mark.parametrize("d", [64, 128])
def test_delta_chunks_lose_no_precision(ops16, d):
    """One long sequence whole (chunks) and in portions of 63 tokens (the token kernel) against float64."""
    heads, kv, dv, n = 32, 8, 64, 600
    g = torch.Generator().manual_seed(d)
    qkv = _randn(g, n, 2 * kv * d + heads * dv)
    proj = _randn(g, n, 2 * heads).to(torch.bfloat16)
    a, b = proj[:, :heads], proj[:, heads:]
    dt_bias, a_log = torch.rand(heads, generator=g).to(DEV) * 3.5 - 3, torch.rand(heads, generator=g).to(DEV) * 2.5 - 2
    first = _randn(g, 1, heads * d * dv, scale=0.3)
    rows = qkv.double()
    q = rows[:, : kv * d].reshape(n, kv, d).repeat_interleave(heads // kv, 1)
    k = rows[:, kv * d : 2 * kv * d].reshape(n, kv, d).repeat_interleave(heads // kv, 1)
    v = rows[:, 2 * kv * d :].reshape(n, heads, dv)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    gate = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(a.double() + dt_bias.double(), threshold=1e9))
    beta = torch.sigmoid(b.double())
    S = first.double().reshape(heads, dv, d).clone()
    ref = torch.empty(n, heads, dv, dtype=torch.float64, device=DEV)
    for s in range(n):
        S = gate[s][:, None, None] * S
        u = beta[s][:, None] * (v[s] - (S * k[s][:, None, :]).sum(-1))
        S = S + u[:, :, None] * k[s][:, None, :]
        ref[s] = (S * q[s][:, None, :]).sum(-1)
    errors = []
    for cuts in ([(0, n)], _portions(n)):
        state = first.clone()
        out = torch.cat([ops16.delta_scan(qkv[y:z], a[y:z], b[y:z], dt_bias, a_log, state, _sequences([z - y]), heads, kv, d,
                                          dv, head_decay=True) for y, z in cuts])
        errors.append((_relative(out, ref.reshape(n, -1)), _relative(state, S.reshape(1, -1))))
    # means over 32 heads, whose decays, unit vectors and step sizes are rounded alike on both sides: equal to a few per cent
    assert errors[0][0] <= 1.05 * errors[1][0] and errors[0][1] <= 1.05 * errors[1][1], errors


@pytest.mark.parametrize("places,lengths", [(1, [130]), (300, [128]), (300, [63, 200, 0, 129, 1]), (300, [128 + i % 9 for i in range(90)])])
def test_chunks_of_sequences_among_empty_places(ops16, places, lengths):
    """A captured step has a place for every request: sequences behind one another or with empty places between
    them, fewer and more (sequence, part) items than blocks, against each sequence by itself, bit for bit."""
    heads, groups, n_state, p, kv, d, dv = 6, 2, 128, 40, 2, 64, 20
    g = torch.Generator().manual_seed(places + len(lengths))
    t = sum(lengths) + 3
    slots = torch.randperm(len(lengths), generator=g).tolist()
    ctx = _sequences(lengths, 3, slots)
    at, step = [], max(1, places // len(lengths) - 1) if places > 1 else 1
    slot_of, start = [-1] * max(places, len(lengths)), []
    for i in range(len(slot_of)):
        if i % step == 0 and len(at) < len(lengths):
            slot_of[i] = slots[len(at)]
            at.append(i)
    for i in range(len(slot_of) + 1):  # a place without a sequence has no tokens
        start.append(sum(n for n, place in zip(lengths, at) if place < i))
    ctx.seq_slot, ctx.seq_start = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in (slot_of, start))
    ctx.n_seqs = len(slot_of)
    xbc, proj = _randn(g, t, heads * p + 2 * groups * n_state, scale=0.5), _randn(g, t, 2 * heads).to(torch.bfloat16)
    qkv, vec = _randn(g, t, 2 * kv * d + heads * dv), _randn(g, heads, scale=0.5)
    states = [_randn(g, len(lengths), heads * n_state * p), _randn(g, len(lengths), heads * d * dv)]

    def run(ctx, rows, first, second):
        return (ops16.mamba2_scan(xbc[rows], proj[rows], 0, vec, vec, vec, first, ctx, heads, groups, n_state, p),
                ops16.delta_scan(qkv[rows], proj[rows, :heads], proj[rows, heads:], vec, vec, second, ctx, heads, kv, d, dv,
                                 head_decay=True))

    together, alone = [s.clone() for s in states], [s.clone() for s in states]
    outs = run(ctx, slice(0, t), *together)
    begin = 0
    for n, slot in zip(lengths, slots):
        if n:
            one = run(_sequences([n], 0, [slot]), slice(begin, begin + n), *alone)
            assert all(torch.equal(a[begin : begin + n], b) for a, b in zip(outs, one))
        begin += n
    assert all(torch.equal(a, b) for a, b in zip(together, alone))


@pytest.mark.parametrize("lengths", [[4097], [4200, 128, 63, 4000], [130] * 40])
def test_delta_chunks_in_stretches(ops16, lengths):
    """More chunks than there is room for: the room does not grow with them, and the bits are those of each sequence in
    portions of whole chunks that need one stretch."""
    from fastgen_b200.csrc.ops import FG_BF16, delta_rule
    heads, kv, d, dv = 3, 1, 64, 24
    slots = list(range(len(lengths)))
    ctx = _sequences(lengths, 0, slots)
    t = ctx.n_tokens
    g = torch.Generator().manual_seed(t)
    qkv, proj = _randn(g, t, 2 * kv * d + heads * dv), _randn(g, t, 2 * heads).to(torch.bfloat16)
    vec = _randn(g, heads, scale=0.5)
    state = _randn(g, len(lengths), heads * d * dv)
    alone = state.clone()

    def run(a, z, ctx, state):
        return ops16.delta_scan(qkv[a:z], proj[a:z, :heads], proj[a:z, heads:], vec, vec, state, ctx, heads, kv, d, dv,
                                head_decay=True)

    out = run(0, t, ctx, state)
    at = 0
    for n, slot in zip(lengths, slots):
        for a in range(0, n, 2048):
            z = min(a + 2048, n)
            if z - a < 128:  # (the token kernel's)
                assert _relative(out[at + a : at + z], run(at + a, at + z, _sequences([z - a], 0, [slot]), alone).double()) < 1e-5
            else:
                assert torch.equal(out[at + a : at + z], run(at + a, at + z, _sequences([z - a], 0, [slot]), alone))
        at += n
    assert _relative(state, alone.double()) < 1e-5
    sizes = [delta_rule().fg_delta_scan_scratch_floats(n, n, 256, 32, 32, 128, 128, FG_BF16, 1) -
             delta_rule().fg_delta_scan_scratch_floats(n, n, 256, 32, 32, 128, 128, FG_BF16, 0) for n in (8192, 16384)]
    # beside what the tokens take: 128 chunks of 2.2 MB
    assert all(4 * x < 300e6 for x in sizes)


def test_decode_buckets_launch_no_chunks(ops16):
    """A captured step of many single tokens runs the token kernels alone."""
    from fastgen_b200.csrc.ops import Ops
    from fastgen_b200.engine.decode_graph import _Bucket
    g = torch.Generator().manual_seed(5)
    heads, groups, n_state, p, d = 4, 2, 64, 32, 64

    def launches(n, longest):
        ctx = _Bucket(n, 100, 1000, DEV).context(torch.device(DEV))
        assert ctx.longest == 1
        ctx.longest = longest
        ctx.seq_slot.copy_(torch.arange(n, dtype=torch.int32, device=DEV))
        proj = _randn(g, n, 2 * heads).to(torch.bfloat16)
        vec = torch.zeros(heads, device=DEV)
        before = Ops.launches
        ops16.mamba2_scan(_randn(g, n, heads * p + 2 * groups * n_state), proj, 0, vec, vec, vec,
                          torch.zeros(n, heads * n_state * p, device=DEV), ctx, heads, groups, n_state, p)
        between = Ops.launches
        ops16.delta_scan(_randn(g, n, 2 * groups * d + heads * p), proj[:, :heads], proj[:, heads:], vec, vec,
                         torch.zeros(n, heads * d * p, device=DEV), ctx, heads, groups, d, p, head_decay=True)
        return between - before, Ops.launches - between

    assert launches(128, 1) == launches(63, None) == (1, 2)
    assert launches(128, None) == (3, 4)


# -- embedding --------------------------------------------------------------------------------------------

@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim,copies", [(8, 1), (504, 2), (512, 1), (1016, 1), (1024, 2), (2040, 2), (2048, 1), (4104, 3), (8192, 1), (100, 2)])
def test_embedding_rows(ops32, dtype, dim, copies):
    from fastgen_b200.csrc.ops import _check, _code, _ptr, _stream
    g = torch.Generator().manual_seed(dim)
    table = _randn(g, 50, dim).to(dtype)
    tokens = torch.tensor([49, 0, 7, 50, -1], dtype=torch.int32, device=DEV)  # the last two are no tokens
    out = torch.full((5, copies, dim), float("nan"), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    _check(ops32.lib, ops32.lib.fg_embedding(_ptr(table), _code(dtype), _ptr(tokens), _ptr(out), _code(torch.float32), 5, dim, 50,
                                             0.7, copies, _ptr(status), _stream()))
    want = torch.zeros(5, dim, device=DEV)
    want[:3] = table[tokens[:3].long()].float() * torch.tensor(0.7, device=DEV)
    assert torch.equal(out, want[:, None].expand(5, copies, dim)) and int(status) == 2  # STATUS_BAD_TOKEN


# -- the selective scan -------------------------------------------------------------------------------------

@pytest.mark.parametrize("inner,N", [(70, 16), (33, 5), (256, 16), (2048, 16)])
def test_selective_scan_however_cut(ops16, inner, N):
    """A sequence's outputs and state have the same bits in one step and in portions, whatever is beside it; an infinity stays
    in the state that it reached."""
    g = torch.Generator().manual_seed(inner + N)
    lengths, order = [767, 768, 0, 1501, 1, 1153], [4, 0, -1, 5, 1, 2]
    starts = [0]
    for n in lengths:
        starts.append(starts[-1] + n)
    t = starts[-1]
    x, dt, z, low = (_randn(g, t, n).to(torch.bfloat16) for n in (inner, inner, inner, 2 * N + 8))
    bias, skip = _randn(g, inner) - 2.0, _randn(g, inner)
    a = -_randn(g, inner, N).exp()
    if N == 16:  # (numbers that fill the lanes up would turn NaN)
        a[3] = -4.0  # (over some hundred tokens these decays multiply up to zero, one by one they do not)
        x[starts[3] + 100, 3] = float("inf")
    state0 = _randn(g, 6, inner * N + 12)

    def run(state, parts):
        """``parts``: (first token, tokens, slot) of a step's sequences."""
        begin, end = parts[0][0], parts[-1][0] + parts[-1][1]
        ctx = SimpleNamespace(n_seqs=len(parts), longest=None,
                              seq_slot=torch.tensor([p[2] for p in parts], dtype=torch.int32, device=DEV),
                              seq_start=torch.tensor([p[0] - begin for p in parts] + [end - begin], dtype=torch.int32, device=DEV))
        rows = slice(begin, end)
        return ops16.selective_scan(x[rows], dt[rows], low[rows], 8, z[rows], bias, a, skip, state, ctx, N)

    whole, cut = state0.clone(), state0.clone()
    # (the lanes a channel, and with them the order of an output's sum, go by channels and sequences of a launch: one by one)
    groups = [[i] for i, n in enumerate(lengths) if n] if inner > 256 else [list(range(len(lengths)))]
    y = torch.cat([run(whole, [(starts[i], lengths[i], order[i]) for i in group]) for group in groups])
    bits = lambda v: v.contiguous().view(torch.int16)
    for s, n, slot in zip(starts, lengths, order):
        for at in range(0, n, 700):
            m = min(700, n - at)
            assert torch.equal(bits(run(cut, [(s + at, m, slot)])), bits(y[s + at : s + at + m])), (s, at)
    assert torch.equal(whole.view(torch.int32), cut.view(torch.int32))
    assert torch.equal(whole[3], state0[3]) and torch.equal(whole[:, inner * N :], state0[:, inner * N :])
    assert N != 16 or bool(torch.isinf(whole[5].flatten()[3 * N : 4 * N]).all())


@pytest.mark.parametrize("rows,ffn", [(1, 4), (3, 8), (5, 1020), (777, 1028), (70000, 16), (9, 8192)])
@pytest.mark.parametrize("act", ["silu", "relu"])
def test_float32_gate_in_fours(ops32, rows, ffn, act):
    """Rows on 16 bytes take four elements a thread, others one: the same numbers."""
    gen = torch.Generator().manual_seed(rows + ffn)
    x = _randn(gen, rows, 2 * ffn, scale=4.0)
    moved = torch.empty(x.numel() + 1, device=DEV)[1:].view(x.shape)
    moved.copy_(x)
    scale, index = _randn(gen, rows), torch.randperm(rows, generator=gen).to(DEV, torch.int32)
    count = torch.tensor([rows - rows // 3], dtype=torch.int32, device=DEV)
    for interleave in (0, 8) if ffn % 8 == 0 else (0,):
        for more in ((), (scale, index, count)):
            outs = []
            for v in (x, moved):
                out = torch.full((rows, ffn), 7.0, device=DEV)
                ops32.silu_gate(v, out, interleave, act, *more)
                outs.append(out)
            assert torch.equal(*outs)
            assert not more or bool((outs[0][int(count):] == 7.0).all())
