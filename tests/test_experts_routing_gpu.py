"""The routing of a decode step's tokens and the plan of its pairs, as dependents of the kernel in front: numbers of experts around
the warps of a block and the lanes of the scan, identity experts, experts without a pair and with several row tiles."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 3, 31, 32, 33, 70])
@pytest.mark.parametrize("P,top", [(1, 1), (32, 2), (33, 3), (127, 1), (128, 2), (1024, 4)])
def test_plan_is_the_stable_sort(E, P, top):
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(E + P)
    choice = torch.randint(0, E + 2, (P,), generator=g)                    # two identity experts
    choice[torch.rand(P, generator=g) < 0.5] = E // 2                      # one expert with half of the pairs
    plan = ops.moe_plan(choice.view(-1, top).to(torch.int32).cuda(), E, 64)
    order = [p for e in range(E) for p in range(P) if choice[p] == e]
    place = [-1] * P
    for at, p in enumerate(order):
        place[p] = at
    tiles, at = [], 0
    for e in range(E):
        n = int((choice == e).sum())
        tiles += [[e, at + q, min(64, n - q)] for q in range(0, n, 64)]
        at += n
    assert int(plan.n_tiles) == len(tiles) and int(plan.n_rows) == len(order)
    assert plan.sorted[:len(order)].tolist() == order and plan.place_of.tolist() == place
    assert plan.table.view(-1, 3)[:len(tiles)].tolist() == tiles


@pytest.mark.parametrize("E", [2, 5, 16, 17, 40])
@pytest.mark.parametrize("T,K,dtype", [(1, 8, torch.bfloat16), (9, 264, torch.bfloat16), (127, 1024, torch.bfloat16), (128, 96, torch.bfloat16),
                                       (3, 33, torch.float32)])
def test_router(E, T, K, dtype):
    """Behind a kernel that has only just made its rows, against float64.  A logit is a sum of K products in at most K / 32 + 5 rounded
    steps, each off by at most 2^-24 of a partial sum, itself at most 6 here: 1.4e-5 at K = 1,024; a weight moves in proportion to no
    more than its logit and the others' mean move."""
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(E * T + K)
    src = torch.randn(T, K, generator=g).to(dtype).cuda()
    wr = (torch.randn(E, K, generator=g) * K ** -0.5).to(dtype).cuda()
    scores = torch.softmax(src.double() @ wr.double().T, 1)
    for _ in range(3):
        h = src.flip(0).flip(0)
        idx, w = ops.moe_router(h, wr, 2)
        h.zero_()
        assert torch.allclose(scores.gather(1, idx.long()), w.double(), rtol=3e-5, atol=0)
        assert torch.allclose(scores.topk(2, 1).values, w.double(), rtol=3e-5, atol=0)      # (a close call may fall the other way)
