"""The grouped product of a handful of pairs (a warp a slab of 16 weight rows on mma.sync, K in slices of a block's warps) against
float64: sizes that fill no slab, no chunk and no slice, experts without a row and with more than eight, both gate layouts."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(8, 8), (24, 264), (40, 520), (13, 1032), (136, 3328), (1024, 32)])
@pytest.mark.parametrize("gated,interleaved", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("tokens", [1, 7, 30])
def test_few_pairs(N, K, gated, interleaved, tokens):
    from fellm_b200 import ops
    if interleaved and N % 8:
        return
    g = torch.Generator().manual_seed(N + K + tokens)
    E, top = 5, 2
    idx = torch.stack([torch.randperm(E - 1, generator=g)[:top] for _ in range(tokens)]).to(torch.int32)       # the last expert is nobody's
    if tokens > 8:
        idx[:, 0], idx[:, 1] = 1, 2                                     # two experts with every row
    plan = ops.moe_plan(idx.cuda(), E)
    a = torch.randn(tokens, K, generator=g).bfloat16().cuda()
    w = (torch.randn(E, (2 if gated else 1) * N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    got = ops.moe_gemm(a, w, plan, gated=gated, gather=True, interleaved=interleaved).double()
    order = plan.sorted.long()
    x, e = a.double()[order // top], idx.cuda().reshape(-1).long()[order]
    y = torch.einsum("pk,pnk->pn", x, w.double()[e])
    if gated:
        if interleaved:
            y = y.view(-1, N // 8, 2, 8)
            gate, up = y[:, :, 0].reshape(-1, N), y[:, :, 1].reshape(-1, N)
        else:
            gate, up = y[:, :N], y[:, N:]
        gate, up = gate.float().bfloat16().double(), up.float().bfloat16().double()
        y = torch.nn.functional.silu(gate) * up
    # float32 sums of K exact products; gated: gate and up round to bfloat16 (2^-9 each), their product once more
    assert float((got - y).norm() / y.norm()) < (6e-3 if gated else 2e-6)


@pytest.mark.parametrize("N,K,tokens", [(1024, 1024, 8), (1024, 3328, 8), (1024, 3328, 30), (2048, 6144, 8)])
def test_sums_are_rounded_not_truncated(N, K, tokens):
    """Float32 results: as near float64 as float32 multiply-adds are (0.7 to 1.1e-7 at these sizes; one chain of accumulating MMAs, which
    truncate, is 2.4 to 7.4e-7 away)."""
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(N + K + tokens)
    E, top = 8, 2
    idx = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(tokens)]).to(torch.int32).cuda()
    plan = ops.moe_plan(idx, E)
    a = torch.randn(tokens, K, generator=g).bfloat16().cuda()
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    got = ops.moe_gemm(a, w, plan, gated=False, gather=True).double()
    order = plan.sorted.long()
    want = torch.einsum("pk,pnk->pn", a.double()[order // top], w.double()[idx.reshape(-1).long()[order]])
    assert float((got - want).norm() / want.norm()) < 1.3e-7
