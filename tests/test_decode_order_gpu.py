"""Decode attention of more (sequence, kv head) pairs than the GPU holds blocks: longest sequences first, every row its own result.
Against 64-bit attention over the same cache pages; the kernel rounds weights to bfloat16 (2^-9 each) and the result (2^-9)."""

import pytest
import torch

from starter_b200.cache import Cache, KVRequest
from test_nifalorn_gpu import context, runtime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D, G, H, lengths", [
    (128, 8, 16, [1 + (37 * i) % 230 for i in range(50)]),     # unequal
    (128, 8, 8, [70] * 40),                                    # all alike: the order of the sequences
    (64, 16, 32, [130 - i for i in range(60)]),                # falling
    (128, 3, 6, [64 + i % 2 for i in range(128)]),             # as many sequences as are ordered
    (128, 3, 6, [64 + i % 3 for i in range(129)]),             # one more
])
def test_every_sequence_meets_its_own_keys(D, G, H, lengths):
    rt = runtime("bfloat16")
    g = torch.Generator().manual_seed(3)
    cache = Cache([KVRequest(num_kv_heads=G, head_dim=D)], n_slots=len(lengths), max_tokens=64 * sum(n // 64 + 2 for n in lengths), dtype=rt.dtype,
                  device="cuda", max_seq_tokens=320)
    slots = [cache.alloc() for _ in lengths]
    lc = cache.layers[0]
    lc.k.copy_(torch.randn(lc.k.shape, generator=g))
    lc.v.copy_(torch.randn(lc.v.shape, generator=g))
    for s, n in zip(slots, lengths):
        cache.reserve(s, n)
    cache.flush()
    for s, n in zip(slots, lengths):
        cache.lengths[s] = n - 1
        cache.lengths_host[s] = n - 1
    ctx = context(rt, cache, slots, [1] * len(lengths))
    q = torch.randn((len(lengths), H * D), generator=g).bfloat16().cuda()
    got = rt.ops.attention(ctx, q, lc, H, D ** -0.5, None).double()
    k, v, table = lc.k.double(), lc.v.double(), lc.group.table_host
    for i, (s, n) in enumerate(zip(slots, lengths)):
        pages = table[s, :(n + 63) // 64].long().cuda()
        kk, vv = (t[pages].transpose(0, 1).reshape(G, -1, D)[:, :n].repeat_interleave(H // G, 0) for t in (k, v))
        w = torch.softmax(torch.einsum("hd,hnd->hn", q[i].double().reshape(H, D), kk) * D ** -0.5, -1)
        want = torch.einsum("hn,hnd->hd", w, vv).reshape(-1)
        assert float((got[i] - want).norm() / want.norm()) < 2 ** -7, f"sequence {i} of {n} tokens"
