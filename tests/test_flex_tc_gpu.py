"""The tcgen05 attention for prompts (cache pages and rows of the step itself) against the attention in 64 bits, at tile,
page, window, chunk and ring borders, with every option of the call and with stale values around a sequence's keys."""

import math

import pytest
import torch

from starter_b200.cache import Cache, KVRequest
from starter_b200.engine.context import Runtime, StepContext

pytestmark = pytest.mark.gpu
F = torch.float64


def runtime():
    from starter_b200.csrc.ops import get_ops
    return Runtime(dtype=torch.bfloat16, device=torch.device("cuda"), ops=get_ops(verbose=False))


def describe(rt, cache, slots, held, q_lens):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    cu = [0]
    for n in q_lens:
        cu.append(cu[-1] + n)
    return StepContext(runtime=rt, cache=cache, n_seqs=len(slots), n_rows=cu[-1], max_q_len=max(q_lens),
                       kv_bound=max(a + n for a, n in zip(held, q_lens)), seq_slot=i32(slots), cu_q=i32(cu),
                       row_seq=i32([b for b, n in enumerate(q_lens) for _ in range(n)]), lengths=cache.lengths,
                       status=torch.zeros(1, dtype=torch.int32, device="cuda"), first=not any(held))


def oracle(q, k, v, first, scale, v_of, temp=None, slopes=None, chunk=None, window=None, sink=None):
    """q [T, H, D] at positions first.., k [n, G, D], v [n, Gv, V] at 0..; in 64 bits."""
    T, H, _ = q.shape
    n, G = k.shape[0], k.shape[1]
    i, j = torch.arange(first, first + T, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
    seen = j <= i
    if window:
        seen = seen & (i - j < window)
    if chunk:
        seen = seen & (i // chunk == j // chunk)
    out = []
    for h in range(H):
        s = (q[:, h].to(F) @ k[:, h * G // H].to(F).T) * scale
        if temp is not None:
            s = s * temp[h].to(F)
        if slopes is not None:
            s = s - slopes[h].to(F) * (i - j)
        s = s.masked_fill(~seen, -math.inf)
        top = s.amax(-1, keepdim=True)
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink[h].to(F) - top)
        out.append((e / total) @ v[:, v_of(h)].to(F))
    return torch.stack(out, 1)


def close(got, want, what):
    """The result is rounded once to bfloat16 (2^-9 of a value); the weights keep 16 bits, sums are 32-bit."""
    got = got.reshape(want.shape).to(F)
    err = float((got - want).norm() / want.norm())
    worst = float((got - want).abs().max() / want.abs().max())
    assert err < 2.5e-3 and worst < 8e-3, f"{what}: {err:.3g}, worst {worst:.3g}"


@pytest.mark.parametrize("D, V, H, G, Gv", [(64, 64, 6, 2, 1), (128, 128, 8, 4, 4), (64, 128, 4, 4, 2), (128, 64, 3, 1, 1)])
@pytest.mark.parametrize("options", ["plain", "biased", "window", "chunk", "sink", "ring"])
@pytest.mark.parametrize("held, q_lens", [([0, 0], [129, 64]), ([0, 70, 3], [257, 130, 1]), ([191], [128])])
def test_pages(D, V, H, G, Gv, options, held, q_lens):
    rt = runtime()
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()   # noqa: E731
    window = {"window": 50, "ring": 150}.get(options)
    cache = Cache([KVRequest(G, D, window=150 if options == "ring" else None, v_dim=V, v_heads=Gv)], n_slots=4, max_tokens=64 * 40,
                  dtype=torch.bfloat16, device="cuda", max_seq_tokens=640, max_step_tokens=260)
    layer = cache.layers[0]
    layer.k.fill_(float("nan")), layer.v.fill_(float("inf"))     # whatever a page's former owner left
    cache.alloc()
    slots = [cache.alloc() for _ in q_lens]
    total = [a + n for a, n in zip(held, q_lens)]
    keys, values = [rnd(n, G, D) for n in total], [rnd(n, Gv, V) for n in total]
    for s, n in zip(slots, total):
        cache.reserve(s, n)
    cache.flush()
    group = layer.group
    for s, n, k, v in zip(slots, total, keys, values):
        for pos in range(n):
            lp = pos // 64
            if group.ring_pages:
                if lp + group.ring_pages <= (n - 1) // 64:
                    continue     # turned over by a later page
                lp %= group.ring_pages
            page = int(group.table_host[s, lp])
            layer.k[page, :, pos % 64], layer.v[page, :, pos % 64] = k[pos], v[pos]
    for s, a in zip(slots, held):
        cache.lengths[s] = a
    ctx = describe(rt, cache, slots, held, q_lens)
    wide = rnd(sum(q_lens), H, D + 8)
    q = wide[:, :, :D]                       # a view of wider rows
    more = {}
    if options == "biased":
        more = dict(head_scale=torch.linspace(-0.5, 2.0, H, device="cuda"), slopes=torch.linspace(0.2, 0.001, H, device="cuda"))
    elif options == "chunk":
        more = dict(chunk=100)
    elif options == "sink":
        more = dict(sink=torch.linspace(-3.0, 4.0, H, device="cuda"))
    elif window:
        more = dict(window=window)
    p = rt.ops._flex(layer, q, H, D ** -0.5, V, False, more.get("sink"), more.get("head_scale"), more.get("slopes"), more.get("chunk"), window)
    assert rt.ops._flex_takes_tc(ctx, q, p) == (max(q_lens) * (H // G) >= rt.ops.FLEX_TC_MIN_ROWS)
    got = rt.ops.flex_attention(ctx, q, layer, D ** -0.5, v_dim=V, **more)
    assert rt.ops.read_kernel_status() == 0
    at = 0
    for b, n in enumerate(q_lens):
        want = oracle(q[at:at + n], keys[b], values[b], held[b], D ** -0.5, lambda h: (h * G // H) // (G // Gv), more.get("head_scale"),
                      more.get("slopes"), more.get("chunk"), window, more.get("sink"))
        close(got[at:at + n], want, f"sequence {b}")
        at += n


@pytest.mark.parametrize("D, R, V, H", [(64, 32, 64, 3), (128, 64, 128, 2)])
@pytest.mark.parametrize("q_lens", [[64], [1, 200, 65, 128], [511, 3]])
@pytest.mark.parametrize("with_sink", [False, True])
def test_rows_of_the_step(D, R, V, H, q_lens, with_sink):
    rt = runtime()
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()   # noqa: E731
    cache = Cache([KVRequest(1, 64)], n_slots=4, max_tokens=64 * 16, dtype=torch.bfloat16, device="cuda")
    rows = sum(q_lens)
    ctx = describe(rt, cache, [cache.alloc() for _ in q_lens], [0] * len(q_lens), q_lens)
    q, kv, latent = rnd(rows, H, D + R), rnd(rows, H * (D + V)), rnd(rows, 40 + R)
    sink = torch.linspace(-2.0, 3.0, H, device="cuda") if with_sink else None
    got = rt.ops.rows_attention(ctx, q, kv[:, :H * D], latent[:, 40:], kv[:, H * D:], 0.11, sink=sink)
    assert rt.ops.read_kernel_status() == 0
    at = 0
    for b, n in enumerate(q_lens):
        piece = slice(at, at + n)
        k = torch.cat([kv[piece, :H * D].view(n, H, D), latent[piece, None, 40:].expand(n, H, R)], -1)
        close(got[piece], oracle(q[piece], k, kv[piece, H * D:].view(n, H, V), 0, 0.11, lambda h: h, sink=sink), f"sequence {b}")
        at += n


def long_context(rt, G, D, V, held, rows, seed=11):
    """One sequence of ``held`` + ``rows`` tokens on pages in a shuffled order, every other page full of other numbers."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()   # noqa: E731
    total = held + rows
    cache = Cache([KVRequest(G, D, v_dim=V)], n_slots=2, max_tokens=64 * 260, dtype=torch.bfloat16, device="cuda", max_seq_tokens=total,
                  max_step_tokens=rows)
    layer, slot = cache.layers[0], cache.alloc()
    layer.k.copy_(rnd(*layer.k.shape)), layer.v.copy_(rnd(*layer.v.shape))
    cache.reserve(slot, total)
    cache.flush()
    pages = -(-total // 64)
    ids = layer.group.table[slot, :pages].clone()
    ids = ids[torch.randperm(pages, generator=g, device="cuda")]
    layer.group.table[slot, :pages] = ids
    cache.lengths[slot] = held
    k, v = (t[ids.long()].transpose(1, 2).reshape(pages * 64, G, -1)[:total] for t in (layer.k, layer.v))
    return describe(rt, cache, [slot], [held], [rows]), layer, k, v, rnd


@pytest.mark.parametrize("held", [64 * 128 - 130, 9300, 13000])     # 128 pages exactly; one refill of the page ids; two, and a wrap
@pytest.mark.parametrize("options", ["plain", "biased", "window"])
def test_more_pages_than_the_kernel_keeps_ids_for(held, options):
    rt, rows, H, G, D, V = runtime(), 130, 4, 2, 64, 128
    ctx, layer, k, v, rnd = long_context(rt, G, D, V, held, rows)
    more = {"plain": {}, "window": dict(window=held - 70),
            "biased": dict(head_scale=torch.linspace(-0.5, 2.0, H, device="cuda"), slopes=torch.linspace(1e-2, 1e-5, H, device="cuda"))}[options]
    q = rnd(rows, H, D)
    got = rt.ops.flex_attention(ctx, q, layer, D ** -0.5, v_dim=V, **more)
    assert rt.ops.read_kernel_status() == 0
    want = oracle(q, k, v, held, D ** -0.5, lambda h: h * G // H, more.get("head_scale"), more.get("slopes"), None, more.get("window"))
    close(got, want, f"{held} tokens held")


@pytest.mark.parametrize("held", [9300, 13000])
def test_the_plain_prompt_kernel_far_into_a_long_context(held):
    rt, rows, H, G, D = runtime(), 140, 4, 2, 128
    ctx, layer, k, v, rnd = long_context(rt, G, D, D, held, rows)
    q = rnd(rows, H * D)
    got = rt.ops.attention(ctx, q, layer, H, D ** -0.5, None)
    assert rt.ops.read_kernel_status() == 0
    want = oracle(q.view(rows, H, D), k, v, held, D ** -0.5, lambda h: h * G // H)
    # that kernel's weights meet the values rounded to bfloat16: 2^-9 each, averaging out over thousands of keys
    got = got.view(rows, H, D).to(F)
    assert float((got - want).norm() / want.norm()) < 5e-3 and float((got - want).abs().max() / want.abs().max()) < 2e-2


@pytest.mark.parametrize("D, V", [(128, 64), (128, 128), (64, 64)])
@pytest.mark.parametrize("held, rows", [(0, 129), (70, 257)])
def test_values_inside_the_key_rows(D, V, held, rows):
    rt, H, G = runtime(), 6, 2
    ctx, layer, k, _, rnd = long_context(rt, G, D, D, held, rows)
    q = rnd(rows, H, D)
    p = rt.ops._flex(layer, q, H, D ** -0.5, V, True)
    assert rt.ops._flex_takes_tc(ctx, q, p)
    got = rt.ops.flex_attention(ctx, q, layer, D ** -0.5, v_dim=V, values_in_keys=True)
    assert rt.ops.read_kernel_status() == 0
    close(got, oracle(q, k, k[:, :, :V], held, D ** -0.5, lambda h: h * G // H), f"values of {V} columns in keys of {D}")
