"""The experts of a step of few rows (moe_few.cu) against 64-bit products of the same bfloat16 numbers, rounded where the kernels
round: gate, up and the activation to bfloat16 before the next product (2^-9 each, 2^-8 with the sum's own rounding)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [None, 1.702])
@pytest.mark.parametrize("E, width, ff, counts, identity", [
    (4, 32, 32, [1, 8, 9, 0], 3),              # one read of 32 inputs for the first warp only; full and ragged groups of 8 pairs
    (3, 544, 96, [16, 17, 40], 0),             # inputs beyond one turn of all warps, several groups of 16 pairs
    (5, 160, 544, [2, 0, 0, 33, 1], 2),
    (2, 1024, 512, [31, 5], 0),
    (64, 64, 64, [1] * 64, 1),
])
def test_every_expert_serves_its_pairs(E, width, ff, counts, identity, alpha):
    from starter_b200.csrc.ops import get_ops
    ops = get_ops(verbose=False)
    g = torch.Generator().manual_seed(7)

    def rand(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g) * scale).bfloat16().cuda()

    picks = [e for e, n in enumerate(counts) for _ in range(n)] + [E] * identity
    picks = [picks[i] for i in torch.randperm(len(picks), generator=g)]
    top = 1 if len(picks) % 2 else 2
    chosen = torch.tensor(picks, dtype=torch.int32, device="cuda").reshape(-1, top)
    rows = chosen.shape[0]
    h, base = rand(rows, width), rand(rows, width)
    weight = torch.rand(rows, top, generator=g).cuda()
    gu, down = rand(E, 2 * ff, width, scale=width ** -0.5), rand(E, width, ff, scale=ff ** -0.5)
    want = base.double()
    for r in range(rows):
        for k in range(top):
            e = picks[r * top + k]
            if e >= E:
                want[r] += weight[r, k].double() * h[r].double()
                continue
            z = (gu[e].double() @ h[r].double()).bfloat16().double()
            a, b = z[:ff], z[ff:]
            if alpha is None:
                act = a * torch.sigmoid(a) * b
            else:
                a, b = a.clamp(max=3.0), b.clamp(-3.0, 3.0)
                act = a * torch.sigmoid(alpha * a) * (b + 1.0)
            want[r] += weight[r, k].double() * (down[e].double() @ act.bfloat16().double())
    takes = ops._moe_takes_few
    calls = []
    ops._moe_takes_few = lambda *a: calls.append(1) or True
    try:
        got = ops.moe_experts(h, chosen, weight, gu, down, E, alpha, 3.0, base)
    finally:
        ops._moe_takes_few = takes
    assert calls and float((got.double() - want).abs().max()) <= 2 ** -7 * float(want.abs().max())


def test_the_rule_between_pairs_experts_and_grouped_products():
    from starter_b200.csrc.ops import get_ops
    ops = get_ops(verbose=False)
    h, w = torch.zeros(8, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(8, dtype=torch.bfloat16, device="cuda")
    assert [ops._moe_takes_few(h, n, 16, 64, 64, w, w) for n in (15, 16, 512, 513)] == [False, True, True, False]
    assert [ops._moe_takes_few(h, n, 4, 64, 64, w, w) for n in (4, 128, 129)] == [True, True, False]
    assert [ops._moe_takes_few(h, n, 300, 64, 64, w, w) for n in (64, 65)] == [False, True]
    assert not ops._moe_takes_few(h.float(), 32, 16, 64, 64, w, w) and not ops._moe_takes_few(h, 32, 16, 64, 40, w, w)
    assert not ops._moe_takes_few(h, 32, 16, 64, 64, w[1:], w)
