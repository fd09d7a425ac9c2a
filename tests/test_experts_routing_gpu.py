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


@pytest.mark.parametrize("T", [1, 8, 40])
def test_a_layer_behind_a_kernel_that_lets_it_start(T):
    """The kernels of a layer one behind the other, the first behind an RMSNorm that lets its dependents start before it has written a row:
    new numbers in the same buffers in every pass, the rows poisoned in between, launched one by one and from a graph.  A read ahead of a
    wait would show against passes in which every kernel is waited for; those are held against float64."""
    from fellm_b200 import ops
    E, top, d, ff, passes = 8, 2, 1024, 768, 6
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    wr = (rnd(E + 2, d) * 2 * d ** -0.5).bfloat16()                         # (two identity experts)
    gate, up = ((rnd(E, ff, d) * d ** -0.5).bfloat16() for _ in range(2))
    both = torch.stack([ops.interleave_gate_up(gate[e], up[e]) for e in range(E)]).contiguous()
    down = (rnd(E, d, ff) * ff ** -0.5).bfloat16()
    ones = torch.ones(d, device="cuda")
    xs = [rnd(T, d) for _ in range(passes)]
    x, h, out = torch.empty(T, d, device="cuda"), torch.empty(T, d, dtype=torch.bfloat16, device="cuda"), torch.empty(T, d, device="cuda")

    def layer(wait=lambda: None):
        h.fill_(float("nan"))
        ops.rmsnorm(x, ones, 1e-5, torch.bfloat16, out=h)
        wait()
        idx, score = ops.moe_router(h, wr, top)
        wait()
        plan = ops.moe_plan(idx, E, ops.moe_row_tile(idx.numel(), True, True))
        wait()
        a = ops.moe_gemm(h, both, plan, gated=True, gather=True, interleaved=True)
        wait()
        y = ops.moe_gemm(a, down, plan, gated=False, gather=False)
        wait()
        ops.moe_combine(out, y, plan, score, store=True, identity=h)
        return idx, score

    want = []
    for p in range(passes):
        x.copy_(xs[p])
        idx, score = layer(torch.cuda.synchronize)
        torch.cuda.synchronize()
        want.append(out.clone())
        hd = h.double()
        logits = torch.softmax(hd @ wr.double().T, 1)
        assert torch.allclose(logits.gather(1, idx.long()), score.double(), rtol=3e-5, atol=0)
        ref = torch.zeros(T, d, dtype=torch.float64, device="cuda")
        for t in range(T):
            for e, s in zip(idx[t].tolist(), score[t].double()):
                act = torch.nn.functional.silu(gate[e].double() @ hd[t]) * (up[e].double() @ hd[t]) if e < E else None
                ref[t] += s * (down[e].double() @ act if e < E else hd[t])
        # (the activations are rounded to 8 bits of mantissa, their errors add up at random over ff of them)
        assert float((out - ref).norm()) < 2.0 ** -8 * float(ref.norm())
    for p in range(passes):
        x.copy_(xs[p])
        layer()
        assert torch.equal(out, want[p])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer()
    for p in range(passes):
        x.copy_(xs[p])
        graph.replay()
        assert torch.equal(out, want[p])
