"""Decode attention whose blocks start with the longest sequence: the order itself, and the results it must not change."""

import pytest
import torch

from starter_b200.cache import Cache, KVRequest
from starter_b200.engine.context import Runtime, StepContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, splits, most", [(2, 1, 130), (40, 1, 130), (40, 2, 130), (133, 1, 60), (1024, 1, 130)])
def test_the_longest_first(monkeypatch, n, splits, most):
    from starter_b200.csrc.ops import get_ops
    ops, (G, H, D) = get_ops(verbose=False), (8, 16, 64)
    g = torch.Generator().manual_seed(n)
    lengths = torch.randint(0, most, (n,), generator=g).tolist()
    cache = Cache([KVRequest(G, D)], n_slots=n, max_tokens=64 * 3 * n, dtype=torch.bfloat16, device="cuda", max_seq_tokens=192)
    slots = [cache.alloc() for _ in range(n)]
    for s, length in zip(slots, lengths):
        cache.assume_length(s, length)
        cache.reserve(s, length + 1)
    cache.flush()
    layer = cache.layers[0]
    fill = torch.Generator(device="cuda").manual_seed(1)
    k0, v0 = (torch.randn(t.shape, generator=fill, device="cuda").bfloat16() for t in (layer.k, layer.v))
    qkv = torch.randn(n, (H + 2 * G) * D, generator=fill, device="cuda").bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    monkeypatch.setattr(ops, "decode_splits", lambda *a: splits)
    monkeypatch.setattr(ops, "decode_resident", lambda d: 1)

    def run(ranked):
        layer.k.copy_(k0), layer.v.copy_(v0)
        ctx = StepContext(runtime=Runtime(torch.bfloat16, torch.device("cuda"), ops), cache=cache, n_seqs=n, n_rows=n, max_q_len=1, kv_bound=192,
                          seq_slot=i32(slots), cu_q=i32(list(range(n + 1))), row_seq=i32(list(range(n))), lengths=cache.lengths, status=i32([0]))
        if ranked:
            ops.begin_step(ctx)
        out = ops.qk_attention(ctx, qkv, layer, H, G, D, None, None, 1e-5, None, D ** -0.5, None)
        return ctx, out, layer.k.clone(), layer.v.clone()

    ctx, *got = run(True)
    rows = [[s, slots[s], lengths[s], s] for s in range(n)]
    assert ctx.scratch["length_places"].tolist() == sorted(rows, key=lambda r: (-r[2], r[0]))
    plain, *want = run(False)
    assert "length_places" not in plain.scratch and all(torch.equal(a, b) for a, b in zip(got, want))
    ctx.uneven = True      # very unequal lengths go to the kernel of equal shares: nothing is ranked, and an old table is dropped
    ops.begin_step(ctx)
    assert "length_places" not in ctx.scratch
