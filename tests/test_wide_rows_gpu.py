"""Row kernels that take 16 bytes a thread for long steps, beside the kernels that take a number a thread: the same rows in one
step of three sequences and in steps of fewer than 128 rows must leave the same outputs, cache rows and records.  Both compute
in 32 bits and differ in the order of one sum over a head, 2^-22 of it, so a bfloat16 result may differ by one rounding (2^-7)."""

import pytest
import torch

from starter_b200.cache import Cache, KVRequest, StateRequest
from test_nifalorn_gpu import context, runtime

pytestmark = pytest.mark.gpu
LENGTHS = [141, 2, 77]


def rand(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).cuda()


def same(a, b, what):
    assert a.shape == b.shape and bool(torch.isfinite(a.float()).all()), what
    d = (a.float() - b.float()).abs()
    assert bool((d <= 2.0 ** -7 * b.float().abs() + 1e-6).all()), f"{what}: {float(d.max())}"


def both_ways(requests, call):
    """call(ops, ctx, layer cache, first row of the piece, one past its last row) for one step of all sequences, and for pieces
    of each: [(outputs, cache)] of both."""
    rt = runtime("bfloat16")
    res = []
    for whole in (True, False):
        cache = Cache([requests], n_slots=4, max_tokens=64 * 16, dtype=rt.dtype, device="cuda")
        cache.alloc()
        slots = [cache.alloc() for _ in LENGTHS]
        starts = [sum(LENGTHS[:i]) for i in range(len(LENGTHS))]
        outs = [None] * len(LENGTHS)
        steps = [list(zip(slots, LENGTHS))] if whole else [[(s, min(100, n - at))] for s, n in zip(slots, LENGTHS) for at in range(0, n, 100)]
        done = dict.fromkeys(slots, 0)
        for step in steps:
            ctx = context(rt, cache, [s for s, _ in step], [n for _, n in step])
            first = starts[slots.index(step[0][0])] + done[step[0][0]]
            out = call(rt.ops, ctx, cache.layers[0], first, first + sum(n for _, n in step))
            rt.ops.advance_lengths(ctx)
            at = 0
            for s, n in step:
                i = slots.index(s)
                outs[i] = out[at:at + n] if outs[i] is None else torch.cat([outs[i], out[at:at + n]])
                cache.advance_host(s, n)
                done[s] += n
                at += n
            assert int(ctx.status.item()) == 0
        res.append((torch.cat(outs), cache))
    return res


@pytest.mark.parametrize("D, V, nq, G, vh, rot, halves", [(64, 128, 8, 4, 2, 64, True), (128, 128, 6, 2, 1, 64, True), (128, 64, 3, 3, 3, 16, True),
                                                          (64, 64, 4, 2, 2, 64, False), (24, 8, 5, 1, 1, 8, False), (72, 40, 2, 2, 2, 48, True),
                                                          (64, 64, 2, 2, 1, 0, True), (40, 16, 2, 1, 1, 24, True)])
def test_rotated_rows(D, V, nq, G, vh, rot, halves):
    rows = sum(LENGTHS)
    p = rand((rows, nq * D + G * D + vh * V + 8), 1).bfloat16()
    freqs = torch.tensor([10000.0 ** (-2.0 * i / max(rot, 1)) for i in range(rot // 2)], dtype=torch.float32, device="cuda") if rot else None
    request = KVRequest(num_kv_heads=G, head_dim=D, v_dim=V, v_heads=vh)

    def call(ops, ctx, lc, a, b):
        x = p[a:b]
        return ops.rotate_store(ctx, x[:, :nq * D].unflatten(1, (nq, D)), x[:, nq * D:(nq + G) * D].unflatten(1, (G, D)),
                                x[:, (nq + G) * D:(nq + G) * D + vh * V], lc, freqs, rot, 1.1, halves)
    (o1, c1), (o2, c2) = both_ways(request, call)
    same(o1, o2, "queries")
    same(c1.layers[0].k, c2.layers[0].k, "keys")
    assert torch.equal(c1.layers[0].v, c2.layers[0].v)


@pytest.mark.parametrize("D, H, G, taps, bias, norm", [(128, 5, 2, 4, True, True), (64, 4, 4, 3, False, True), (128, 2, 1, 2, True, False),
                                                       (64, 1, 1, 1, True, True), (64, 3, 1, 4, True, True)])
def test_convolved_rows(D, H, G, taps, bias, norm):
    rows = sum(LENGTHS)
    p = rand((rows, (H + G) * D + 4), 2).bfloat16()
    w = dict(q_bias=rand((H * D,), 3, 0.2) if bias else None, k_bias=rand((G * D,), 4, 0.2) if bias else None,
             q_conv=rand((H * D, taps), 5, 0.5), k_conv=rand((G * D, taps), 6, 0.5),
             q_norm=rand((D,), 7) if norm else None, k_norm=rand((D,), 8) if norm else None)
    kv = KVRequest(num_kv_heads=G, head_dim=D, v_dim=D)
    request = (kv, StateRequest((taps - 1, (H + G) * D))) if taps > 1 else kv

    def call(ops, ctx, lc, a, b):
        x = p[a:b]
        return ops.conv_qk_store(ctx, x[:, :H * D], x[:, H * D:(H + G) * D], lc, lc.aux.state if taps > 1 else None, H, w["q_bias"], w["k_bias"],
                                 w["q_conv"], w["k_conv"], w["q_norm"], w["k_norm"], 1e-5, 0.2, 16)
    (o1, c1), (o2, c2) = both_ways(request, call)
    same(o1, o2, "queries")
    same(c1.layers[0].k, c2.layers[0].k, "keys")
    same(c1.layers[0].v, c2.layers[0].v, "keys before the norm")
    if taps > 1:
        assert torch.equal(c1.layers[0].aux.state, c2.layers[0].aux.state)


@pytest.mark.parametrize("V", [64, 128, 40, 12])
@pytest.mark.parametrize("pad", [0, 3, 8])
def test_rows_that_are_joined_gated_and_biased(V, pad):
    """Widths and strides that the 16-byte kernels take and ones that they do not, against the formula in 64 bits."""
    ops, rows, H, G = runtime("bfloat16").ops, 37, 4, 2
    a, gate = rand((rows, 2 * H * V), 11).bfloat16(), rand((rows, H * V + pad), 12).bfloat16()
    x = a.double().reshape(rows, G, 2, H // G, V)
    o = x[:, :, 0] - 0.3 * x[:, :, 1]
    o = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * 0.5).reshape(rows, H * V)
    for g in (None, gate[:, :H * V]):
        want = o if g is None else o * torch.sigmoid(g.double())
        got = ops.diff_combine(a, H, G, V, 0.3, 1e-5, 0.5, gate=g).double()
        assert float((got - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    z, b = rand((rows, H + pad), 13), rand((H * V,), 14)
    y = a[:, :H * V].contiguous()
    wide = torch.zeros((rows, H * V + pad), dtype=torch.bfloat16, device="cuda")
    got = ops.head_gate(y, z, pad, H, 0.7, out=wide[:, :H * V]).double()
    want = y.double() * torch.sigmoid(z[:, pad:].double()).repeat_interleave(V, 1) * 0.7
    assert float((got - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    want = y.double() + b.double()
    assert float((ops.add_bias(y.clone(), b).double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    assert torch.equal(ops.relu2(y), (torch.relu(y.float()) ** 2).bfloat16())


@pytest.mark.parametrize("rows", [1023, 1024, 1500])
@pytest.mark.parametrize("width", [2048, 2044, 1024, 516, 64, 2052])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_layer_norms_of_many_rows(rows, width, dtype):
    """A warp per row from 1,024 rows of up to 2,048 columns on: 32-bit sums, one rounding to the output's type (bfloat16: half a unit
    in the last of 8 bits, 2^-8 of the value at most; the 32-bit error of the sums, 2e-6, beside it)."""
    ops, dt = runtime(dtype).ops, getattr(torch, dtype)
    x, d, w, b = rand((rows, width), 21, 2.0) + 0.5, rand((rows, width), 22).to(dt), rand((width,), 23), rand((width,), 24)
    for delta in (None, d):
        y = x.clone()
        got = ops.layernorm(y, delta, w, b, 1e-5, dt).double()
        s = x.double() if delta is None else x.double() + d.double()
        c = s - s.mean(-1, keepdim=True)
        want = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-5) * w.double() + b.double()
        assert float((y.double() - s).abs().max()) <= 2.0 ** -23 * float(s.abs().max())
        assert float((got - want).abs().max()) <= ((2.0 ** -8 if dtype == "bfloat16" else 0.0) + 2e-6) * float(want.abs().max())


@pytest.mark.parametrize("D, G, H, taps", [(64, 2, 4, 4), (128, 1, 2, 3), (64, 3, 3, 2)])
def test_unit_heads_of_many_rows(D, G, H, taps):
    """Runs of 8 rows from 512 rows on, sequences that begin inside a run and records from an earlier step, beside steps of fewer rows."""
    ops, C = runtime("bfloat16").ops, (2 * G + H) * D
    counts = [300, 1, 2, 221]
    p, w = rand((sum(counts), C + 8), 31).bfloat16(), rand((taps, C), 32, 0.5)
    inner = rand((sum(counts), 11), 33)
    state0 = rand((6, taps - 1, C), 34)
    slots = [4, 0, 3, 1]

    def step(seqs, rows, state):
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
        from types import SimpleNamespace
        ns = [counts[s] for s in seqs]
        cu = [sum(ns[:i]) for i in range(len(ns) + 1)]
        ctx = SimpleNamespace(seq_slot=i32([slots[s] for s in seqs]), cu_q=i32(cu), row_seq=i32([i for i, n in enumerate(ns) for _ in range(n)]),
                              lengths=i32([0] * 6), n_seqs=len(ns), n_rows=cu[-1], max_q_len=max(ns), cache=SimpleNamespace(null_slot=5), scratch={})
        return ops.conv_unit_heads(ctx, p[rows, :C], w, state, G, D, 0.3, inner[rows], 7, 16)
    s1, s2 = state0.clone(), state0.clone()
    whole = step([0, 1, 2, 3], slice(None), s1)
    at = 0
    for i, n in enumerate(counts):
        part = step([i], slice(at, at + n), s2)
        assert float((whole[0][at:at + n] - part[0]).abs().max()) <= 1e-6 * float(part[0].abs().max())
        assert torch.equal(whole[1][at:at + n], part[1])
        at += n
    assert torch.equal(s1, s2)


LONGER = [441, 2, 277]      # beyond the rows from which the kernels of this file take the whole step


@pytest.mark.parametrize("D, V, nq, G, vh, rot, halves", [(64, 128, 8, 4, 2, 64, True), (128, 64, 3, 3, 3, 16, True), (64, 64, 4, 2, 2, 64, False),
                                                          (24, 8, 5, 1, 1, 8, False), (72, 40, 2, 2, 2, 48, True), (64, 64, 2, 2, 1, 0, True),
                                                          (40, 16, 2, 1, 1, 24, True)])
def test_rotated_rows_of_longer_steps(monkeypatch, D, V, nq, G, vh, rot, halves):
    monkeypatch.setitem(globals(), "LENGTHS", LONGER)
    test_rotated_rows(D, V, nq, G, vh, rot, halves)


@pytest.mark.parametrize("D, H, G, taps, bias, norm", [(128, 5, 2, 4, True, True), (64, 4, 4, 3, False, True), (128, 2, 1, 2, True, False),
                                                       (64, 1, 1, 1, True, True), (64, 3, 1, 4, True, True)])
def test_convolved_rows_of_longer_steps(monkeypatch, D, H, G, taps, bias, norm):
    monkeypatch.setitem(globals(), "LENGTHS", LONGER)
    test_convolved_rows(D, H, G, taps, bias, norm)


@pytest.mark.parametrize("D, taps", [(128, 4), (64, 3)])
def test_convolved_rows_of_many_sequences(D, taps):
    """One row a sequence: runs of eight rows from 768 (heads of 128) and 1,536 (of 64) on, beside steps of 100."""
    rt, n, H, G = runtime("bfloat16"), 1600, 2, 1
    p, w = rand((n, (H + G) * D), 41).bfloat16(), [rand((h * D, taps), 42 + h, 0.5) for h in (H, G)]
    record, res = rand((n + 1, taps - 1, (H + G) * D), 45), []
    for size in (n, 100):
        cache = Cache([(KVRequest(num_kv_heads=G, head_dim=D, v_dim=D), StateRequest((taps - 1, (H + G) * D)))], n_slots=n, max_tokens=64 * n,
                      dtype=rt.dtype, device="cuda")
        slots = [cache.alloc() for _ in range(n)]
        lc, outs = cache.layers[0], []
        lc.aux.state.copy_(record)
        for at in range(0, n, size):
            ctx = context(rt, cache, slots[at:at + size], [1] * size)
            x = p[at:at + size]
            outs.append(rt.ops.conv_qk_store(ctx, x[:, :H * D], x[:, H * D:], lc, lc.aux.state, H, None, None, *w, None, None, 1e-5, 0.0, 0))
            assert int(ctx.status.item()) == 0
        res.append((torch.cat(outs), cache))
    same(res[0][0], res[1][0], "queries")
    same(res[0][1].layers[0].k, res[1][1].layers[0].k, "keys")
    assert torch.equal(res[0][1].layers[0].aux.state, res[1][1].layers[0].aux.state)


def test_gated_gelu_rounds_a_row_as_its_other_forms_do():
    """Every finite bfloat16 number through the kernel of 16 bytes a thread: the 32-bit kernel's result, rounded once; and that result
    against 64 bits: up to eight roundings of 2^-24, and four of them times the exponent where that is large."""
    ops = runtime("bfloat16").ops
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    g = g[torch.isfinite(g)].cuda()
    g = g[:g.numel() // 8 * 8].view(1, -1)
    u = rand(g.shape, 51).bfloat16()
    wide, narrow = ops.gated_gelu(torch.cat([g, u], 1).float()), ops.gated_gelu(torch.cat([g, u], 1))
    assert torch.equal(narrow, wide.bfloat16())
    z = g.double()
    exponent = -2.0 * (2.0 / torch.pi) ** 0.5 * (z + 0.044715 * z ** 3)
    want = z / (1.0 + torch.exp(exponent)) * u.double()
    error = (wide.double() - want).abs()
    sound = (want.abs() > 1e-30) & (want.abs() < 1e30)
    assert bool((error <= want.abs() * (4.0 + 2.0 * exponent.clamp(min=0.0)) * 2.0 ** -23)[sound].all())


def test_the_clamped_activation_rounds_a_row_as_its_other_forms_do():
    """Every finite bfloat16 number through the kernel of 16 bytes a thread: the 32-bit kernel's result, rounded once."""
    ops = runtime("bfloat16").ops
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    g = g[torch.isfinite(g)].cuda()
    g = g[:g.numel() // 8 * 8].view(1, -1)
    for seed in (52, 53, 54):
        u = rand(g.shape, seed, 3.0).bfloat16()
        wide, narrow = ops.gated_clamp(torch.cat([g, u], 1).float(), 1.702, 7.0), ops.gated_clamp(torch.cat([g, u], 1), 1.702, 7.0)
        assert torch.equal(narrow, wide.bfloat16())
