"""The all-float32 product fed by cp.async against the general one: the same k-ordered chains, so the same bits, for every tile
and at its remainders."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 40, 4), (16, 33, 36), (17, 2048, 64), (33, 70, 100), (65, 4800, 132), (201, 1024, 1024), (64, 9600, 32)])
@pytest.mark.parametrize("act", [None, "relu2", "add"])
def test_same_bits_as_the_general_product(M, N, K, act):
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    a, w, bias = (torch.randn(*s, generator=g).cuda() for s in ((M, K), (N, K), (N,)))
    off = torch.zeros(M, K + 1, device="cuda")[:, 1:]                   # rows that do not start on 16 bytes: the general kernel
    off.copy_(a)
    out = [torch.randn(M, N, generator=torch.Generator().manual_seed(1)).cuda() for _ in range(2)]
    for x, o in zip((a, off), out):
        ops.gemm_simt(x, w, bias, out=o, accumulate=act == "add", act=act if act == "relu2" else None)
    assert torch.equal(out[0], out[1])
    want = a.double() @ w.double().T + bias.double()
    if act is None:
        # K products rounded to 2^-24 each, in one chain
        assert float((out[0].double() - want).abs().max()) <= 2.0 ** -24 * (K + 2) * float((a.abs().double() @ w.abs().double().T + bias.abs()).max())
