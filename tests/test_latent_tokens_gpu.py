"""Latent attention of single tokens: a token's keys shared out in portions of 16 over the blocks of a cluster, or over blocks that leave
their sums in memory, against float64, at the edges of portions, tiles, windows and shares."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rk,dr,H", [(512, 64, 8), (512, 64, 16), (64, 16, 4), (64, 16, 24)])
@pytest.mark.parametrize("window,contexts", [(None, (1, 16, 17, 64, 65, 300)), (100, (1, 99, 101, 513)), (1024, (1500, 1039, 64)), (64, (63, 64, 128, 1000)),
                                             (None, (3100,))])
@pytest.mark.parametrize("share", [0, 10, 100])
def test_a_token_over_its_keys(monkeypatch, rk, dr, H, window, contexts, share):
    from fellm_b200 import ops
    monkeypatch.setattr(ops, "LATENT_CLUSTER_TO", share)             # 0: always through memory, 100: always a cluster
    D, PT, n = rk + dr, 64, len(contexts)
    g = torch.Generator().manual_seed(rk + H + n)
    pages = [-(-c // PT) for c in contexts]
    pool = torch.randn(sum(pages) + 1, 1, PT, D, generator=g).bfloat16()
    table = torch.full((n, max(pages) + 1), -1, dtype=torch.int32)
    for i, (p, c) in enumerate(zip(pages, contexts)):
        table[i, :p] = torch.randperm(p, generator=g) + 1 + sum(pages[:i])
        pool[table[i, p - 1], 0, (c - 1) % PT + 1:] = float("nan")   # behind the last key: a freed page's bits
        if window is not None:
            table[i, :max(0, c - window) // PT] = -1                 # pages wholly behind the window are given back
    q = (torch.randn(n, H, D, generator=g) * 0.5).bfloat16()
    sinks = torch.randn(H, generator=g)
    scale = D ** -0.5
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32)
    got = ops.latent_attention(q.reshape(n, H * D).cuda(), H, rk, dr, pool.cuda(), table.cuda(), pos.cuda(), torch.arange(n, dtype=torch.int32).cuda(),
                               torch.arange(n + 1, dtype=torch.int32).cuda(), n, 1, max(contexts), 0, PT, scale, window=window, sinks=sinks.cuda())
    got = got.double().cpu().view(n, H, rk)
    for i, c in enumerate(contexts):
        first = 0 if window is None else max(0, c - window)
        at = torch.arange(first, c)
        rows = pool[table[i, at // PT].long(), 0, at % PT].double()
        s = q[i].double() @ rows.T * scale
        m = torch.maximum(s.max(-1).values, sinks.double())
        p = torch.exp(s - m[:, None])
        want = p @ rows[:, :rk] / (p.sum(-1) + torch.exp(sinks.double() - m))[:, None]
        # probabilities rounded to bfloat16 (2^-9 each) of values of size ~1, then the result
        room = 2.0 ** -8 * (p @ rows[:, :rk].abs() / p.sum(-1, keepdim=True)) + 2.0 ** -8 * want.abs() + 1e-4
        assert ((got[i] - want).abs() <= room).all(), (c, float(((got[i] - want).abs() / room).max()))


@pytest.mark.parametrize("rk,dr,H", [(512, 64, 8), (64, 16, 24), (96, 16, 4)])
@pytest.mark.parametrize("window,contexts", [(None, (1, 40, 129, 700)), (1024, (1500,) * 3 + (1039, 64) + (1100,) * 3), (1024, (2000,) * 17), (None, (3100,))])
def test_how_the_shares_are_put_together_is_not_in_the_bits(monkeypatch, rk, dr, H, window, contexts):
    """A cluster or memory and a second kernel: the shares are the same whole tiles and are added in the same order."""
    from fellm_b200 import ops
    D, PT, n = rk + dr, 64, len(contexts)
    g = torch.Generator().manual_seed(rk + n)
    pages = [-(-c // PT) for c in contexts]
    pool = torch.randn(sum(pages) + 1, 1, PT, D, generator=g).bfloat16().cuda()
    table = torch.zeros((n, max(pages)), dtype=torch.int32)
    for i, p in enumerate(pages):
        table[i, :p] = torch.arange(p) + 1 + sum(pages[:i])
    q = (torch.randn(n, H * D, generator=g) * 0.5).bfloat16().cuda()
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32).cuda()
    sinks = torch.randn(H, generator=g).cuda()

    def run(share):
        monkeypatch.setattr(ops, "LATENT_CLUSTER_TO", share)
        return ops.latent_attention(q, H, rk, dr, pool, table.cuda(), pos, torch.arange(n, dtype=torch.int32).cuda(),
                                    torch.arange(n + 1, dtype=torch.int32).cuda(), n, 1, max(contexts), 0, PT, D ** -0.5, window=window, sinks=sinks)
    assert torch.equal(run(0), run(100))


@pytest.mark.parametrize("n", [1, 8, 140])
def test_directly_behind_the_kernel_that_writes_the_cache(n):
    """Without cache_ready nothing of a step is read before the kernel in front has ended: this one writes the step's own rows, and lets its
    dependents start before it does.  New rows in every pass, a context of one key beside others: a row not yet written would show."""
    from types import SimpleNamespace
    from fellm_b200 import ops
    rk, dr, H, PT, rq = 512, 64, 8, 64, 768
    D = rk + dr
    contexts = [1 + 37 * i % 200 for i in range(n)]
    g = torch.Generator().manual_seed(n)
    pool = torch.randn(4 * n + 1, 1, PT, D, generator=g).bfloat16().cuda()
    table = (torch.arange(4 * n, dtype=torch.int32).view(n, 4) + 1).cuda()
    pos = torch.tensor([c - 1 for c in contexts], dtype=torch.int32).cuda()
    slot, starts = torch.arange(n, dtype=torch.int32).cuda(), torch.arange(n + 1, dtype=torch.int32).cuda()
    cache = SimpleNamespace(pool=pool, block_table=table, page_tokens=PT, layer=0)
    wq, wc = torch.ones(rq).cuda(), torch.ones(rk).cuda()
    freq = (0.5 ** torch.arange(dr // 2)).cuda()
    q = torch.randn(n, H * D, generator=g).bfloat16().cuda()
    z = [torch.randn(n, rq + D, generator=g).cuda() for _ in range(8)]

    def step(i, wait):
        ops.latent_prep(z[i], 0, rq, rq, rk, rq + rk, dr, wq, wc, 1e-5, freq, dr, 1.0, pos, slot, cache, torch.bfloat16)
        if wait:
            torch.cuda.synchronize()
        return ops.latent_attention(q, H, rk, dr, pool, table, pos, slot, starts, n, 1, max(contexts), 0, PT, D ** -0.5)
    want = [step(i, True) for i in range(8)]
    torch.cuda.synchronize()
    got = [step(i, False) for i in range(8)]
    assert all(torch.equal(a, b) for a, b in zip(got, want))
