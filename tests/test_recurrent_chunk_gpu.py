"""Recurrences over portions in chunks of 32 tokens (csrc/recurrent_chunk.cu) against the recurrences walked token by
token in float64, at the edges of a chunk, with several requests of unequal lengths in a step."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

MODES = ("delta", "channel_delta", "decay_bonus", "gated_write")


def walk(S, A, B, G, K, v, beta, c, delta):
    """u = beta (v - S^T A) or v; o = S^T B + c u; S = G S + K u^T (one head, float64).  -> (o [T, dv], S)"""
    out = []
    for t in range(v.shape[0]):
        u = beta[t] * (v[t] - S.T @ A[t]) if delta else v[t]
        out.append(S.T @ B[t] + c[t] * u)
        S = G[t][:, None] * S + K[t][:, None] * u[None]
    return (torch.stack(out) if out else v), S


class Step:
    """Inputs of one step of a mode, the call of its kernel, and the oracle."""

    def __init__(self, mode, lens, H, G, dk, dv, seed=0, dtype=torch.float32, decay_zero=False):
        g = torch.Generator().manual_seed(seed)
        rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
        T = sum(lens)
        self.mode, self.lens, self.H, self.G, self.dk, self.dv = mode, lens, H, G, dk, dv
        self.starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
        self.slots = list(range(len(lens)))[::-1]
        self.state = 0.3 * rnd(len(lens), H, dv, dk)                       # column by column, as the kernels keep it
        self.q, self.k, self.v = rnd(T, G * dk), rnd(T, G * dk), rnd(T, H * dv)
        self.b, self.a = rnd(T, H), rnd(T, H)
        self.A_log, self.dt = 0.5 * rnd(H), rnd(H)
        self.gch = torch.exp(-torch.exp(rnd(T, H * dk)))
        if decay_zero:
            self.gch[torch.rand(T, H * dk, generator=g) < 0.05] = 0.0
        self.bonus, self.lower, self.fb = rnd(H, dk), torch.rand(H * dk, generator=g) * 0.9, rnd(H * dk)
        if mode == "decay_bonus":
            self.q, self.k, self.v = (x.to(dtype).float() for x in (self.q, self.k, self.v))
        self.dtype = dtype

    def run(self, chunk_rows, offset=0):
        from fellm_b200 import ops
        dev = lambda t: t.cuda().contiguous()  # noqa: E731
        H, G, dk, dv, n = self.H, self.G, self.dk, self.dv, len(self.lens)
        state = dev(self.state).view(n, H, dk, dv)
        starts = torch.tensor(self.starts, dtype=torch.int32, device="cuda")
        slots = torch.tensor(self.slots, dtype=torch.int32, device="cuda")
        kw = dict(max_item_rows=max(self.lens), chunk_rows=chunk_rows)

        def rows(*parts):              # a matrix whose rows start `offset` elements behind a 16-byte boundary
            m = torch.cat(parts, 1)
            wide = torch.zeros(m.shape[0], m.shape[1] + 16)
            wide[:, offset:offset + m.shape[1]] = m
            return dev(wide.to(self.dtype if self.mode == "decay_bonus" else torch.float32))[:, offset:offset + m.shape[1]]
        if self.mode in ("delta", "channel_delta"):
            o = ops.delta_scan(rows(self.q, self.k, self.v), G * dk, 2 * G * dk, dev(torch.cat([self.b, self.a], 1)), 0, H, dev(self.A_log),
                               dev(self.dt) if self.mode == "delta" else None, None if self.mode == "delta" else dev(self.gch), state,
                               starts, slots, n, H, G, dk, dv, **kw)
        elif self.mode == "decay_bonus":
            m = rows(self.q, self.k, self.v)
            o = ops.decay_bonus_scan(m[:, :H * dk], m[:, H * dk:2 * H * dk], m[:, 2 * H * dk:3 * H * dk], dev(self.gch), dev(self.bonus), state,
                                     starts, slots, n, H, dk, **kw)
        else:
            o = ops.gated_write_scan(rows(self.q, self.k, self.v), H * dk, 2 * H * dk, dev(self.lower), dev(self.fb), state, starts, slots,
                                     n, H, dk, dv, **kw)
        torch.cuda.synchronize()
        return o.double().cpu(), state.view(n, H, dv, dk).double().cpu()

    def oracle(self):
        H, G, dk, dv = self.H, self.G, self.dk, self.dv
        out, states = torch.zeros(sum(self.lens), H * dv, dtype=torch.float64), self.state.double().clone()
        for i, n in enumerate(self.lens):
            at = slice(self.starts[i], self.starts[i] + n)
            for h in range(H):
                hk, hv = slice(h * dk, (h + 1) * dk), slice(h * dv, (h + 1) * dv)
                g = h // (H // G)
                gk = slice(g * dk, (g + 1) * dk)
                q, k, v = self.q[at, gk].double(), self.k[at, gk].double(), self.v[at, hv].double()
                if "delta" in self.mode:
                    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
                    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
                    if self.mode == "delta":
                        soft = torch.nn.functional.softplus(self.a[at, h].double() + self.dt[h].double())
                        Gd = torch.exp(-torch.exp(self.A_log[h].double()) * soft)[:, None].expand(n, dk)
                    else:
                        Gd = self.gch[at, hk].double()
                    A, B, K, c, beta = Gd * k, Gd * q, k, (k * q).sum(-1), torch.sigmoid(self.b[at, h].double())
                elif self.mode == "decay_bonus":
                    A, B, Gd, K, beta = q, q, self.gch[at, hk].double(), k, torch.ones(n)
                    c = (q * self.bonus[h].double() * k).sum(-1)
                else:
                    f = self.lower[hk].double() + (1 - self.lower[hk].double()) * torch.sigmoid(k + self.fb[hk].double())
                    q = torch.nn.functional.silu(q)
                    A, B, Gd, K, c, beta = q, f * q, f, 1 - f, ((1 - f) * q).sum(-1), torch.ones(n)
                o, S = walk(states[self.slots[i], h].T.clone(), A, B, Gd, K, v, beta, c, "delta" in self.mode)
                out[at, hv] = o
                states[self.slots[i], h] = S.T
        return out, states


def near(got, want):
    # a result is a sum of up to dk + 32 products (their factors: products of up to 32 rounded decays), each rounded to 2^-24,
    # through a substitution of 32 steps: 2^-24 (dk + 64) of the sums' size bounds it; 128 + 64 -> 1.2e-5 of the root mean square
    return float((got - want).norm() / want.norm().clamp(min=1e-30)) < 1.2e-5


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens,H,G,dk,dv", [((32,), 2, 1, 128, 128), ((33,), 1, 1, 64, 16), ((31, 64, 1, 65), 4, 2, 64, 48), ((97, 40), 2, 2, 128, 32)])
def test_chunks_are_the_walk(mode, lens, H, G, dk, dv):
    if mode == "decay_bonus":
        dv = dk
    if not mode.endswith("delta"):
        G = H
    for zero in (False, True):
        s = Step(mode, lens, H, G, dk, dv, seed=len(lens) + dk, decay_zero=zero,
                 dtype=torch.bfloat16 if mode == "decay_bonus" and zero else torch.float32)
        o, st = s.run(32)
        want, want_state = s.oracle()
        assert near(o, want) and near(st, want_state)


@pytest.mark.parametrize("mode", MODES)
def test_short_items_keep_the_scan(mode):
    """Items below the limit give the bits of the scan, whatever else is in the step; all items do where an alignment is refused."""
    H = 2
    s = Step(mode, (5, 70, 31), H, H, 64, 64, seed=9)
    o, st = s.run(32)
    o0, st0 = s.run(0)
    for i in (0, 2):
        at = slice(s.starts[i], s.starts[i + 1])
        assert torch.equal(o[at], o0[at]) and torch.equal(st[s.slots[i]], st0[s.slots[i]])
    assert not torch.equal(o, o0) and near(o, o0)
    o1, st1 = s.run(32, offset=1)
    assert torch.equal(o1, s.run(0, offset=1)[0]) and near(st1, st0)


@pytest.mark.parametrize("mode", MODES)
def test_a_later_token_leaves_earlier_ones_alone(mode):
    s = Step(mode, (64,), 2, 2, 64, 64, seed=4)
    clean, _ = s.run(32)
    for what, value in (("v", float("nan")), ("k", float("inf")), ("q", float("nan"))):
        x = getattr(s, what)
        kept = x[50].clone()
        x[50] = value
        got, _ = s.run(32)
        x[50] = kept
        assert torch.equal(got[:50], clean[:50])


@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("mode", MODES)
def test_chunks_are_no_less_exact_than_the_walk(mode, alike):
    """Errors against float64 of the chunks and of the token-by-token scan, both float32.  Means over the elements of three seeds: a
    tenth of room for the draw (float32 sums throughout were 1.2 to 1.7 times the scan's in the delta rule)."""
    err = {0: [0.0, 0.0], 32: [0.0, 0.0]}
    for seed in range(3):
        s = Step(mode, (160, 96), 2, 2, 128, 128, seed=seed)
        if alike:                                  # keys that differ by a tenth, and almost all of the old value written over
            s.k = torch.randn(1, s.k.shape[1], generator=torch.Generator().manual_seed(seed)) + 0.1 * s.k
            s.b = torch.full_like(s.b, 4.6)
        want, want_state = s.oracle()
        for rows, e in err.items():
            o, st = s.run(rows)
            e[0] += float(((o - want).norm() / want.norm()) ** 2)
            e[1] += float(((st - want_state).norm() / want_state.norm()) ** 2)
    for scan, chunk in zip(err[0], err[32]):
        assert chunk <= 1.1 ** 2 * scan
