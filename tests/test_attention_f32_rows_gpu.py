"""The 32-bit engine's attention: how many neighbouring rows a block takes is a matter of speed; every row has the bits it has alone, and
those of the attention in float64 up to the float32 sums' rounding."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [1, 2, 4])
@pytest.mark.parametrize("rows,before", [((33,), (0,)), ((31, 1, 8), (70, 0, 33)), ((201, 60), (300, 5)), ((1100,), (2,))])
def test_rows_have_the_bits_they_have_alone(R, rows, before):
    from fellm_b200 import ops
    G, PT, n = 4, 16, len(rows)
    H, pages = G * R, [-(-(a + b) // PT) for a, b in zip(rows, before)]
    g = torch.Generator().manual_seed(sum(rows) + R)
    pool = torch.randn(sum(pages) + 1, 1, 2, G, PT, 64, generator=g).cuda()
    table = torch.full((n, max(pages) + 1), -1, dtype=torch.int32)
    for i, p in enumerate(pages):
        table[i, :p] = torch.arange(sum(pages[:i]) + 1, sum(pages[:i + 1]) + 1)
    pos = torch.cat([torch.arange(b, a + b) for a, b in zip(rows, before)]).int()
    slot = torch.repeat_interleave(torch.arange(n), torch.tensor(rows)).int()
    q = torch.randn(sum(rows), H, 64, generator=g).cuda()
    args = lambda at: (q[at].contiguous(), pool, table.cuda(), pos[at].cuda(), slot[at].cuda(), 0, 0.125)  # noqa: E731
    got = ops.paged_attention_simt(*args(slice(None)))
    for t in range(0, sum(rows), 7):
        assert torch.equal(got[t], ops.paged_attention_simt(*args(slice(t, t + 1)))[0])
    for t in (0, rows[0] - 1, sum(rows) - 1):
        i, p = int(slot[t]), int(pos[t])
        kv = pool[table[i, :pages[i]].long().cuda(), 0].transpose(0, 1).transpose(1, 2).reshape(2, G, -1, 64)[:, :, :p + 1].double()
        s = torch.einsum("grd,gkd->grk", q[t].double().view(G, R, 64), kv[0]) * 0.125
        want = torch.einsum("grk,gkd->grd", s.softmax(-1), kv[1]).reshape(-1)
        # scores: 64 products of 2^-24 each, as a factor of the exponential; p + 1 probabilities and products
        room = 2.0 ** -24 * (64 * 8 + p + 64) * kv[1].abs().max()
        assert float((got[t].double() - want).abs().max()) <= room
