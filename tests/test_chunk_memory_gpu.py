"""The recurrences of the wkv, gla and mlstm mixers over whole chunks (chunk_memory.cu), against the recurrence in 64 bits token by
token and beside the kernels that walk token by token in 32 bits.

Bounds.  State: every entry is a sum of terms that pass at most T decays, T multiplications and additions of 2^-24 each; T is
at most 450 here, so 450 * 2^-23 = 5.4e-5 of the sum of magnitudes covers it, the decays' own rounding included.  Outputs are rounded
to bfloat16 (2^-9 of each at most), the rest is far below that."""

import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
F = torch.float64
EPS = 1e-5


def batch_of(counts, slots, n_slots):
    cu = [0]
    for n in counts:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device="cuda")
    rows = [s for s, n in enumerate(counts) for _ in range(n)]
    return SimpleNamespace(seq_slot=torch.tensor(slots, **i32), cu_q=torch.tensor(cu, **i32), row_seq=torch.tensor(rows, **i32),
                           lengths=torch.zeros(n_slots + 1, **i32), n_seqs=len(counts), n_rows=cu[-1], max_q_len=max(counts),
                           cache=SimpleNamespace(null_slot=n_slots), scratch={}), cu


def unit(o):
    return o / torch.sqrt((o * o).mean(-1, keepdim=True) + EPS)


def walk(kind, q, k, v, a, b, S, u=None):
    """One sequence in 64 bits: q, k [T, H, D], v [T, H, V], a, b broadcastable to [T, H, D]; S [H, D, V] is changed."""
    out = []
    for t in range(q.shape[0]):
        kv = (b[t] * k[t])[:, :, None] * v[t][:, None, :]
        if kind == "wkv":
            out.append(torch.einsum("hd,hdv->hv", q[t], S + u[:, :, None] * kv))
            S.mul_(a[t][:, :, None]).add_(kv)
        else:
            S.mul_(a[t][:, :, None]).add_(kv)
            out.append(torch.einsum("hd,hdv->hv", q[t], S))
    return torch.stack(out) if out else torch.zeros(0, q.shape[1], v.shape[2], dtype=F)


def rel(got, want):
    return float((got.double().cpu() - want).norm() / want.norm())


def run_kind(kind, H, D, V, counts, strong, pad, seed=0):
    """(outputs, state, their 64-bit values) from the chunks and from the walk."""
    from starter_b200.csrc.ops import get_ops
    ops = get_ops(verbose=False)
    g = torch.Generator().manual_seed(seed)
    n_slots, slots = len(counts) + 2, [len(counts) - i for i in range(len(counts))]
    rows = sum(counts)
    ctx, cu = batch_of(counts, slots, n_slots)

    def rand(*shape, scale=1.0):
        return torch.randn(*shape, generator=g) * scale

    # q | k | v | g side by side in rows that `pad` columns more make longer
    p = rand(rows, 2 * H * D + 2 * H * V + pad).bfloat16().cuda()
    cols = [H * D, H * D, H * V, H * V]
    views, at = [], 0
    for c in cols:
        views.append(p[:, at:at + c])
        at += c
    extra = H * D + H if kind == "mlstm" else 0
    state0 = rand(n_slots + 1, H * D * V + extra, scale=0.5)
    if kind == "mlstm":
        state0[:, -H:] = rand(n_slots + 1, H)
    results = []
    q, k, v, gate = (t.double().cpu().reshape(rows, H, -1) for t in views)
    want_state = state0.double().clone()
    if kind == "wkv":
        prev = H * D * V
        state0 = torch.cat([state0, rand(n_slots + 1, 24)], 1)
        want_state = state0.double().clone()
        pre, w0, u = rand(rows, H * D, scale=strong), rand(H * D) - 1.0, rand(H * D)
        norm, h = rand(H * D, scale=0.1) + 1.0, rand(rows, 24).bfloat16()
        flat = [t.contiguous() for t in views]
        args = lambda st: ops.wkv_scan(ctx, *flat, pre.cuda(), w0.cuda(), u.cuda(), norm.cuda(), EPS, h.cuda(), st, H, D, prev)
        a = torch.exp(-torch.exp(pre.double() + w0.double())).reshape(rows, H, D)
        b = torch.ones(rows, H, 1, dtype=F)
    elif kind == "gla":
        z, bias, norm, tau = rand(rows, H * D, scale=4 * strong), rand(H * D), rand(V, scale=0.1) + 1.0, 8.0
        args = lambda st: ops.gla_scan(ctx, *views, z.cuda(), bias.cuda(), norm.cuda(), EPS, tau, D ** -0.5, st, H, D, V)
        a = (torch.nn.functional.logsigmoid(z.double() + bias.double()) / tau).exp().reshape(rows, H, D)
        b = torch.ones(rows, H, 1, dtype=F)
        q = q * D ** -0.5
    else:
        z, bi, bf, cap = rand(rows, 2 * H + 1, scale=5 * strong), rand(H), rand(H) + 2.0, 15.0
        norm = rand(H * V, scale=0.1) + 1.0
        args = lambda st: ops.mlstm_scan(ctx, *views, z.cuda(), 1, 1 + H, bi.cuda(), bf.cuda(), cap, norm.cuda(), EPS, D ** -0.5, st, H, D, V,
                                         out_scale=0.7)
        zd = z.double()
        log_i = cap * torch.tanh((zd[:, 1:1 + H] + bi.double()) / cap)
        log_f = torch.nn.functional.logsigmoid(cap * torch.tanh((zd[:, 1 + H:] + bf.double()) / cap))
        q = q * D ** -0.5
    want = torch.zeros(rows, H, V, dtype=F)
    for s, slot in enumerate(slots):
        r = slice(cu[s], cu[s + 1])
        if kind == "mlstm":
            rec = want_state[slot]
            m, aa, bb, em = rec[-H:].clone(), [], [], []
            for t in range(cu[s], cu[s + 1]):
                new = torch.maximum(log_f[t] + m, log_i[t])
                aa.append(torch.exp(log_f[t] + m - new))
                bb.append(torch.exp(log_i[t] - new))
                em.append(torch.exp(-new))
                m = new
            S = torch.cat([rec[:H * D * V].reshape(H, D, V), rec[H * D * V:-H].reshape(H, D, 1)], 2).clone()
            if aa:
                aa, bb, em = torch.stack(aa)[..., None], torch.stack(bb)[..., None], torch.stack(em)[..., None]
                o = walk(kind, q[r], k[r], torch.cat([v[r], torch.ones(len(aa), H, 1, dtype=F)], 2), aa.expand(-1, -1, D), bb, S)
                want[r] = o[..., :V] / (torch.maximum(o[..., V:].abs(), em) + 1e-6)
            rec[:H * D * V], rec[H * D * V:-H], rec[-H:] = S[..., :V].reshape(-1), S[..., V].reshape(-1), m
        else:
            S = want_state[slot][:H * D * V].reshape(H, D, V).clone()
            want[r] = walk(kind, q[r], k[r], v[r], a[r], b[r], S, u.double().reshape(H, D) if kind == "wkv" else None)
            want_state[slot][:H * D * V] = S.reshape(-1)
            if kind == "wkv" and counts[s]:
                want_state[slot][prev:] = h[cu[s + 1] - 1].double()
    want = unit(want)
    if kind == "gla":
        want = want * norm.double()
    else:
        want = want * norm.double().reshape(H, V)
    want = want * torch.sigmoid(gate) * (0.7 if kind == "mlstm" else gate)
    for chunks in (True, False):
        ops.force_chunk_memory = chunks
        try:
            before = ops.launches
            st = state0.clone().cuda()
            y = args(st)
            torch.cuda.synchronize()
            assert (ops.launches - before >= 3) == chunks
        finally:
            del ops.force_chunk_memory
        results.append((y, st))
    return results, want.reshape(rows, H * V), want_state


CASES = [  # H, D, V, rows of each sequence, how strong the decays are, extra columns
    (2, 64, 64, [64], 1.0, 0), (3, 64, 64, [129, 1, 63, 0, 65], 1.0, 8), (2, 32, 32, [200], 2.5, 0), (1, 128, 128, [70, 300], 1.0, 0),
    (2, 64, 64, [450], 3.0, 0), (2, 24, 24, [100, 16], 1.0, 0), (1, 7, 7, [81], 1.0, 3), (33, 64, 64, [17, 15, 16], 1.0, 0),
    (2, 100, 100, [130], 1.0, 4), (2, 64, 64, [80] * 35, 1.0, 0),
]
WIDE = [(2, 64, 128, [129, 40], 1.0, 0), (1, 128, 64, [65], 1.0, 0), (2, 32, 128, [450], 3.0, 0), (3, 16, 72, [90, 5], 1.0, 0), (1, 9, 101, [77], 1.0, 1)]


@pytest.mark.parametrize("kind, case", [(k, c) for k in ("wkv", "gla", "mlstm") for c in CASES + (WIDE if k != "wkv" else [])],
                         ids=lambda x: x if isinstance(x, str) else "x".join(map(str, x[:3])) + "-" + str(len(x[3])) + "-" + str(max(x[3])))
def test_chunks_against_the_recurrence_in_64_bits(kind, case):
    H, D, V, counts, strong, pad = case
    ((y, st), (y_walk, st_walk)), want, want_state = run_kind(kind, H, D, V, counts, strong, pad)
    print(f"{kind} {case[:3]} outputs {rel(y, want):.2e} (walk {rel(y_walk, want):.2e}), state {rel(st, want_state):.2e} (walk {rel(st_walk, want_state):.2e})")
    assert bool(torch.isfinite(y.float()).all())
    assert rel(y, want) < 2 ** -8
    assert rel(st, want_state) < 5.4e-5
    assert math.isfinite(float(st.abs().max()))


@pytest.mark.parametrize("H, D, V, counts", [(16, 64, 128, [1] * 130), (16, 64, 128, [16] * 33 + [3, 70]), (20, 32, 72, [2] * 200), (9, 128, 200, [1, 40] * 60)])
def test_a_walk_of_many_sequences_leaves_what_each_alone_does(H, D, V, counts):
    """Heads whose value channels several blocks share out: more blocks than the GPU holds at a time, so that one starts from the
    record when another of its head has long ended.  A sequence's outputs and record are the same numbers as alone."""
    from starter_b200.csrc.ops import get_ops
    ops = get_ops(verbose=False)
    g = torch.Generator(device="cuda").manual_seed(2)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    n, rows = len(counts), sum(counts)
    p, z = rand(rows, 2 * H * D + 2 * H * V).bfloat16(), rand(rows, 2 * H) * 4
    bi, bf, norm, state = rand(H), rand(H) + 2.0, rand(H * V), rand(n + 1, H * D * V + H * D + H)

    def run(ctx, lo, hi, st):
        at, views = 0, []
        for c in (H * D, H * D, H * V, H * V):
            views.append(p[lo:hi, at:at + c])
            at += c
        return ops.mlstm_scan(ctx, *views, z[lo:hi], 0, H, bi, bf, 15.0, norm, EPS, D ** -0.5, st, H, D, V)

    ops.force_chunk_memory = False
    try:
        ctx, cu = batch_of(counts, list(range(n)), n)
        together = state.clone()
        y = run(ctx, 0, rows, together)
        for s in range(n):
            alone = state[s:s + 1].clone()
            one, _ = batch_of(counts[s:s + 1], [0], 1)
            assert torch.equal(run(one, cu[s], cu[s + 1], alone), y[cu[s]:cu[s + 1]]), f"outputs of sequence {s}"
            assert torch.equal(alone[0], together[s]), f"record of sequence {s}"
    finally:
        del ops.force_chunk_memory
    assert torch.equal(together[n], state[n])


@pytest.fixture
def little_room(monkeypatch):
    """Once called, the allocator has no room for more than 60 MB of floats at a time."""
    empty = torch.empty

    def limited(*size, dtype=None, **kwargs):
        if dtype == torch.float32 and len(size) == 1 and isinstance(size[0], int) and 4 * size[0] > 60 * 2 ** 20:
            raise torch.OutOfMemoryError("no room")
        return empty(*size, dtype=dtype, **kwargs)
    return lambda: monkeypatch.setattr(torch, "empty", limited)


def test_a_step_without_room_for_the_chunks_is_walked(little_room):
    from starter_b200.csrc.ops import get_ops
    ops, H, D, V, rows = get_ops(verbose=False), 16, 64, 128, 3333
    ctx, _ = batch_of([rows], [0], 1)
    g = torch.Generator(device="cuda").manual_seed(4)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    p = rand(rows, 2 * H * (D + V)).bfloat16()
    views = p.split([H * D, H * D, H * V, H * V], 1)
    z, bias, norm = rand(rows, 2 * H), rand(H), rand(H * V)
    states = [torch.zeros(2, H * D * V + H * D + H, device="cuda") for _ in range(2)]
    run = lambda st: ops.mlstm_scan(ctx, *views, z, 0, H, bias, bias, 15.0, norm, EPS, D ** -0.5, st, H, D, V)   # noqa: E731
    assert 4 * ops.lib.sb_chunk_memory_floats(ops.CHUNK_MLSTM, rows, 1, H, D, V, ops.chunk_head_floats) > 60 * 2 ** 20
    ops.force_chunk_memory = False
    try:
        want = run(states[0])
    finally:
        del ops.force_chunk_memory
    little_room()
    assert ops.chunk_memory_pays(1, rows, rows, H, V)
    assert torch.equal(run(states[1]), want) and torch.equal(states[0], states[1])


def test_a_product_without_room_for_its_chunks_of_k_takes_them_in_order(little_room):
    from starter_b200.csrc.ops import get_ops
    ops, (M, N, K) = get_ops(verbose=False), (300, 19456, 2560)
    g = torch.Generator(device="cuda").manual_seed(4)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    assert 4 * ops.lib.sb_gemm_general_scratch(0, M, N, K) > 60 * 2 ** 20
    want = ops.linear(a, w)
    little_room()
    assert torch.equal(ops.linear(a, w), want)


@pytest.mark.parametrize("kind", ["wkv", "gla", "mlstm"])
@pytest.mark.parametrize("together", [1, 2, 4])
def test_heads_in_groups(monkeypatch, kind, together):
    """A workspace for fewer heads than the layer has: the same numbers as with all heads at once, the last group smaller."""
    from starter_b200.csrc.ops import get_ops
    ops, H, D, V, counts = get_ops(verbose=False), 5, 64, 64, [150, 3, 70]
    ((y, st), _), _, _ = run_kind(kind, H, D, V, counts, 1.0, 0)
    cells = sum(counts) // 64 + len(counts)
    monkeypatch.setattr(ops, "chunk_head_floats", together * cells * (D * V + 3 * D * V // 2 + 2 * D))
    codes = (sum(counts), len(counts), H, D, V, ops.chunk_head_floats)
    code = {"wkv": ops.CHUNK_WKV, "gla": ops.CHUNK_GLA, "mlstm": ops.CHUNK_MLSTM}[kind]
    assert ops.lib.sb_chunk_memory_launches(code, *codes) == -(-H // together) * (4 if kind == "mlstm" else 3)
    ((few, st_few), _), _, _ = run_kind(kind, H, D, V, counts, 1.0, 0)
    assert torch.equal(few, y) and torch.equal(st_few, st)
