"""Attention kernels of portions and of single rows that a layer's sizes choose: tcgen05 with chunks, biases, temperatures,
gates and values that are the keys; keys and values per head out of cached latents; and rows whose keys are dealt out over
a cluster.  Against float64 over whole contexts, at the edges of pages, windows, chunks and of a
block's 128 rows."""
from __future__ import annotations

import math
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def attend(q, k, v, pos, scale, window=None, chunk=None, cap=None, slopes=None, temp=None, sinks=None):
    """q [n, H, dk] at positions pos [n]; k, v [len, G, .] -> [n, H, dv], all float64."""
    H, G = q.shape[1], k.shape[1]
    j = torch.arange(k.shape[0])
    see = j[None] <= pos[:, None]
    if window:
        see &= pos[:, None] - j[None] < window
    if chunk:
        see &= pos[:, None] // chunk == j[None] // chunk
    if temp:
        q = q * (1 + temp[0] * torch.log(torch.floor((pos.double() + 1) / temp[1]) + 1))[:, None, None]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64)
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * (pos[:, None] - j[None])
        s = s.masked_fill(~see, -math.inf)
        m = s.max(-1, keepdim=True).values
        if sinks is not None:
            m = m.clamp(min=float(sinks[h]))
        p = torch.exp(s - m)
        out[:, h] = (p / (p.sum(-1, keepdim=True) + (torch.exp(sinks[h] - m) if sinks is not None else 0))) @ v[:, h // (H // G)]
    return out


class Pages:
    """Requests with the given numbers of tokens, their keys and values in pages handed out in a mixed order; what no request
    wrote is NaN."""

    def __init__(self, lens, G, hd, vd, page, seed):
        g = torch.Generator().manual_seed(seed)
        self.lens, self.page = lens, page
        n_pages = [-(-n // page) for n in lens]
        order = torch.randperm(sum(n_pages), generator=g).tolist()
        self.k = [torch.randn(n, G, hd, generator=g).bfloat16() for n in lens]
        self.v = [torch.randn(n, G, vd, generator=g).bfloat16() for n in lens] if vd else self.k
        width = max(n_pages) + 1
        self.table = torch.full((len(lens), width), -1, dtype=torch.int32)
        pool = torch.full((len(order), 2, G * page * (hd + vd)), float("nan"), dtype=torch.bfloat16)
        for r, n in enumerate(lens):
            for i in range(n_pages[r]):
                p = order.pop()
                self.table[r, i] = p
                part = slice(i * page, min(n, (i + 1) * page))
                m = part.stop - part.start
                rec = pool[p, 1]
                rec[:G * page * hd].view(G, page, hd)[:, :m] = self.k[r][part].transpose(0, 1)
                if vd:
                    rec[G * page * hd:].view(G, page, vd)[:, :m] = self.v[r][part].transpose(0, 1)
        self.pool = pool.cuda()

    def five(self, G, hd):
        return self.pool.view(self.pool.shape[0], 2, 2, G, self.page, hd)


def close(got, want):
    # bfloat16 probabilities and results: 2^-8 of the result's size each, with room for the sums
    assert float((got.double().cpu() - want).norm() / want.norm()) < 6e-3
    assert float((got.double().cpu() - want).abs().max() / want.pow(2).mean().sqrt()) < 0.06


FORMS = [dict(window=70), dict(chunk=48), dict(window=100, slopes=True, temp=(0.25, 16)), dict(cap=4.0, chunk=100, gate=True), dict(slopes=True),
         dict(window=1, temp=(0.5, 128)), dict(window=64, out_gate=True), dict(),
         # a cap and a temperature that is 1.6 to 2.5 at most of these positions: of the scores inside the cap
         dict(cap=2.0, temp=(0.5, 16)), dict(cap=4.0, temp=(0.5, 16), slopes=True, window=100)]


def form(spec, T, H, g, hd=64):
    kw = dict(spec)
    slopes = torch.rand(H, generator=g) * 0.2 if kw.pop("slopes", False) else None
    gate = torch.randn(T, H + 3, generator=g) if kw.pop("gate", False) else None
    out_gate = torch.randn(T, H * hd + 8, generator=g).bfloat16() if kw.pop("out_gate", False) else None
    return kw, slopes, gate, out_gate


def gated(want, H, gate, out_gate):
    if gate is not None:
        want = want * torch.sigmoid(gate[:, :H].double())[:, :, None]
    want = want.reshape(want.shape[0], -1)
    return want if out_gate is None else want * torch.sigmoid(out_gate[:, :want.shape[1]].double())


@pytest.mark.parametrize("spec", FORMS)
@pytest.mark.parametrize("H,G,keys_alone", [(4, 1, True), (4, 2, False), (8, 8, False)])
def test_portions_on_tcgen05(spec, H, G, keys_alone):
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(H + G)
    lens, rows = [200, 64, 300, 1], [37, 64, 130, 1]                   # tokens of every request, of which the last `rows` are the step's
    pages = Pages(lens, G, 64, 0 if keys_alone else 64, 64, 3)
    T = sum(rows)
    q = torch.randn(T, H * 64 + 24, generator=g).bfloat16()
    pos = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, rows)])
    kw, slopes, gate, out_gate = form(spec, T, H, g)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    starts = [sum(rows[:i]) for i in range(len(rows) + 1)]
    got = ops.attention_prefill_general(
        q.cuda(), H, pages.pool if keys_alone else pages.five(G, 64), pages.table.cuda(), i32(pos), i32([r for r, m in enumerate(rows) for _ in range(m)]),
        i32(starts), len(rows), max(rows), 1, 0.125, window=kw.get("window"), chunk=kw.get("chunk"), softcap=kw.get("cap"), q_temp=kw.get("temp"),
        slopes=None if slopes is None else slopes.cuda(), gate=None if gate is None else gate.cuda(),
        out_gate=None if out_gate is None else out_gate.cuda()[:, :H * 64], values_are_keys=(G, 64, 64) if keys_alone else None)
    ops.check_umma_status(torch.device("cuda"))
    for r in range(len(rows)):
        at = slice(starts[r], starts[r + 1])
        want = attend(q[at, :H * 64].double().view(-1, H, 64), pages.k[r].double(), pages.v[r].double(), pos[at], 0.125,
                      slopes=None if slopes is None else slopes.double(), **kw)
        close(got[at], gated(want, H, None if gate is None else gate[at], None if out_gate is None else out_gate[at]))


@pytest.mark.parametrize("spec", FORMS)
@pytest.mark.parametrize("H,G,hd,page,keys_alone,cluster", [(4, 1, 64, 64, True, 8), (4, 2, 64, 16, False, 2), (3, 3, 128, 64, False, 4),
                                                           (8, 2, 64, 256, False, 1), (8, 2, 128, 32, True, 8)])
def test_rows_over_a_cluster(spec, H, G, hd, page, keys_alone, cluster, monkeypatch):
    from fellm_b200 import ops
    monkeypatch.setattr(ops, "attention_rows_cluster", lambda *a: cluster)
    g = torch.Generator().manual_seed(H + G)
    lens = [1, 31, 33, 130, 700]
    vd = 0 if keys_alone else hd
    pages = Pages(lens, G, hd, vd, page, 5)
    T = len(lens)
    q = torch.randn(T, (H + 2 * G) * hd + 8, generator=g).bfloat16()
    for r in range(T):                                                 # the step's own keys and values lie in the rows
        pages.k[r][-1] = q[r, H * hd:(H + G) * hd].view(G, hd)
        if vd:
            pages.v[r][-1] = q[r, (H + G) * hd:(H + 2 * G) * hd].view(G, hd)
    pos = torch.tensor([n - 1 for n in lens])
    kw, slopes, gate, out_gate = form(spec, T, H, g, hd)
    pool = pages.pool if keys_alone else pages.five(G, hd)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def call(write, with_gate=True):
        return ops.paged_attention_general(
            q.cuda(), H, hd, vd, pool, pages.table.cuda(), i32(pos), i32(range(T)), 1, page, G, hd ** -0.5, window=kw.get("window"),
            chunk=kw.get("chunk"), softcap=kw.get("cap"), q_temp=kw.get("temp"), slopes=None if slopes is None else slopes.cuda(),
            gate=None if gate is None else gate.cuda(), write_new=write,
            out_gate=out_gate.cuda()[:, :H * hd] if out_gate is not None and with_gate else None)
    write = (H * hd, (H + G) * hd, status)
    assert ops.attention_rows_takes(q.cuda(), pool, H, G, hd, vd, page, write)
    got = call(write)
    assert int(status) == 0
    again = call(None, with_gate=False)          # the CUDA-core kernel, which reads the rows' keys and values from their pages now
    if out_gate is not None:
        assert torch.equal(call(None), got)      # and this kernel, reading them from there
    for r in range(T):
        want = attend(q[r:r + 1, :H * hd].double().view(1, H, hd), pages.k[r].double(), pages.v[r].double(), pos[r:r + 1], hd ** -0.5,
                      slopes=None if slopes is None else slopes.double(), **kw)
        whole = gated(want, H, None if gate is None else gate[r:r + 1], None if out_gate is None else out_gate[r:r + 1])
        # float32 throughout, one rounding to bfloat16 at the end: 2^-9 of an element at most
        assert float((got[r:r + 1].double().cpu() - whole).norm() / whole.norm()) < 2.5e-3
        plain = gated(want, H, None if gate is None else gate[r:r + 1], None)
        assert float((again[r:r + 1].double().cpu() - plain).norm() / plain.norm()) < 2.5e-3
    pages.table[2, (lens[2] - 1) // page] = -1                          # no page for the row's position: nothing written, a status
    before = pool.clone()
    call(write)
    torch.cuda.synchronize()
    assert int(status) == 2 and torch.equal(before.view(torch.int16), pool.view(torch.int16))


@pytest.mark.parametrize("window,chunk,G", [(None, None, 4), (1024, None, 4), (300, None, 2), (1024, 512, 8)])
def test_a_row_keeps_its_bits_in_every_batch(window, chunk, G):
    """However many rows decode together: the blocks that share a row's keys follow the batch, the order of its sums does not."""
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(G)
    lens = [1, 33, 700, 1500, 2100]
    H, hd, page = 2 * G, 64, 64
    pages = Pages(lens, G, hd, hd, page, 7)
    T = 330
    slots = torch.arange(T) % len(lens)
    pos = torch.tensor(lens)[slots] - 1
    q, gate = torch.randn(T, H * hd, generator=g).bfloat16().cuda(), torch.randn(T, H * hd, generator=g).bfloat16().cuda()
    i32 = lambda x: x.to(torch.int32).cuda()  # noqa: E731

    def call(n):
        assert ops.attention_rows_takes(q[:n], pages.five(G, hd), H, G, hd, hd, page)
        return ops.paged_attention_general(q[:n], H, hd, hd, pages.five(G, hd), pages.table.cuda(), i32(pos[:n]), i32(slots[:n]), 1, page, G, 0.125,
                                           window=window, chunk=chunk, out_gate=gate[:n])
    whole = call(T)
    sizes = (1, 5, 12, 40, 80, 200)
    clusters = {ops.attention_rows_cluster(n * G, window, chunk) for n in sizes + (T,)}
    assert len(clusters) > 1
    for n in sizes:
        assert torch.equal(call(n), whole[:n])
    for r in range(len(lens)):
        want = attend(q[r:r + 1].double().cpu().view(1, H, hd), pages.k[r].double(), pages.v[r].double(), pos[r:r + 1], 0.125, window=window, chunk=chunk)
        want = want.reshape(1, -1) * torch.sigmoid(gate[r:r + 1].double().cpu())
        assert float((whole[r:r + 1].double().cpu() - want).norm() / want.norm()) < 2.5e-3


@pytest.mark.parametrize("window,sink", [(64, True), (100, False), (1, True)])
def test_latents_taken_out_per_head(window, sink):
    from fellm_b200 import ops
    H, rk, dr = 3, 128, 64
    g = torch.Generator().manual_seed(window)
    lens, rows = [200, 130, 64, 300], [65, 130, 1, 128]
    pages = Pages(lens, 1, rk + dr, 0, 64, 4)
    T = sum(rows)
    q = torch.randn(T, H * 192, generator=g).bfloat16()
    wk, wv = ((torch.randn(H, 128, rk, generator=g) * rk ** -0.5).bfloat16() for _ in range(2))
    sinks = torch.randn(H, generator=g) if sink else None
    pos = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, rows)])
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).cuda()  # noqa: E731
    starts = [sum(rows[:i]) for i in range(len(rows) + 1)]
    freq = torch.tensor([10000.0 ** (-2 * i / 32) for i in range(16)])                  # half of the rotated part turns
    ctx = types.SimpleNamespace(positions=i32(pos), row_slot=i32([r for r, m in enumerate(rows) for _ in range(m)]), item_start=i32(starts),
                                n_items=len(rows), max_item_rows=max(rows))
    cache = types.SimpleNamespace(pool=pages.pool, block_table=pages.table.cuda(), page_tokens=64, layer=1)
    key_rows = -(-(window - 1 + 63 + max(rows)) // 64) * 64
    qd = q.cuda()
    lat, rope = ops.latent_gather(qd, H, 128, dr, freq.cuda(), 32, 1.5, rk, cache, ctx, window, key_rows)
    kv = (lat.float() @ torch.cat([wk, wv], 1).reshape(H * 256, rk).cuda().float().T).bfloat16()
    assert torch.isfinite(kv).all()
    got = ops.latent_expanded_attention(qd, H, kv, rope, key_rows, ctx, 0.1, window, None if sinks is None else sinks.cuda())
    ops.check_umma_status(torch.device("cuda"))
    a = (pos.float()[:, None] * freq[None]).double()
    q64 = q.double().view(T, H, 192).clone()
    u, v = q64[..., 128:160:2].clone(), q64[..., 129:160:2].clone()
    c, s = (torch.cos(a) * 1.5)[:, None], (torch.sin(a) * 1.5)[:, None]
    q64[..., 128:160:2], q64[..., 129:160:2] = u * c - v * s, v * c + u * s
    for r in range(len(rows)):
        at = slice(starts[r], starts[r + 1])
        row = pages.k[r][:, 0].double()
        k = torch.cat([torch.einsum("nr,hdr->nhd", row[:, :rk], wk.double()), row[:, None, rk:].expand(-1, H, dr)], -1)
        want = attend(q64[at], k, torch.einsum("nr,hdr->nhd", row[:, :rk], wv.double()), pos[at], 0.1, window=window,
                      sinks=None if sinks is None else sinks.double())
        # (keys, values and rotated queries are rounded once more than in `close`'s other callers)
        assert float((got[at].double().cpu() - want.reshape(rows[r], -1)).norm() / want.norm()) < 1e-2


@pytest.mark.parametrize("H,G,page,window", [(4, 4, 16, None), (4, 2, 64, None), (8, 2, 32, None), (4, 2, 64, 40), (3, 3, 64, 1)])
def test_float32_rows_share_their_keys(H, G, page, window):
    """The 32-bit attention: near float64, and a row's bits whatever else is in the launch."""
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(H * G)
    lens, rows = [131, 64, 300, 1, 33], [37, 64, 5, 1, 33]
    pages = Pages(lens, G, 64, 64, page, 6)
    pool = pages.five(G, 64).float()
    T = sum(rows)
    q = torch.randn(T, H, 64, generator=g)
    pos = torch.cat([torch.arange(n - m, n) for n, m in zip(lens, rows)])
    slot = torch.tensor([r for r, m in enumerate(rows) for _ in range(m)])
    i32 = lambda x: x.to(torch.int32).cuda()  # noqa: E731
    got = ops.paged_attention_simt(q.cuda(), pool, pages.table.cuda(), i32(pos), i32(slot), 1, 0.125, window)
    for r in range(len(rows)):
        at = slice(sum(rows[:r]), sum(rows[:r + 1]))
        want = attend(q[at].double(), pages.k[r].double(), pages.v[r].double(), pos[at], 0.125, window=window).reshape(rows[r], -1)
        # scores of 64 products, sums of up to 300 terms, each rounded to 2^-24, exponentials to 2^-22
        assert float((got[at].double().cpu() - want).norm() / want.norm()) < 2e-6
    for part in (slice(0, 40), slice(7, 8), slice(36, 75), slice(100, T)):
        one = ops.paged_attention_simt(q[part].cuda(), pool, pages.table.cuda(), i32(pos[part]), i32(slot[part]), 1, 0.125, window)
        assert torch.equal(one, got[part])
