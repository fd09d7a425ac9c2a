"""A product per head for a handful of rows (slabs of 16 weight rows, csrc/gemm_tiled.cu) against the tile that takes more
rows, bit for bit, and against float64."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("H,N,K,a_head,out_head", [(3, 8, 8, 8, 24), (2, 40, 24, 32, 40), (16, 256, 64, 96, 256), (5, 72, 520, 528, 80)])
def test_few_rows_are_the_tile_s(T, H, N, K, a_head, out_head):
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(T + N)
    a = torch.randn(40, H * a_head, generator=g).bfloat16()
    w = (torch.randn(H, N, K, generator=g) * 0.2).bfloat16()
    full = torch.full((40, H * out_head), 7.0, dtype=torch.bfloat16, device="cuda")
    few = full[:T].clone()
    ops.head_gemm(a.cuda(), w.cuda(), full, a_head=a_head, out_head=out_head)
    ops.head_gemm(a[:T].cuda(), w.cuda(), few, a_head=a_head, out_head=out_head)
    assert torch.equal(few, full[:T])
    for h in range(H):
        x, m = a[:T, h * a_head:h * a_head + K].double(), w[h].double()
        got = few[:, h * out_head:h * out_head + N].double().cpu()
        # K float32 sums and one rounding to 8 significant bits (half a unit in the last place: 2^-8 of the value at most)
        assert bool(((got - x @ m.T).abs() <= 2.0 ** -8 * (x @ m.T).abs() * 1.01 + K * 2.0 ** -23 * (x.abs() @ m.abs().T) + 1e-30).all())


@pytest.mark.parametrize("T", [5, 40])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_matrices_in_a_wider_block(T, dtype):
    """A head's matrix may be part of a larger block per head: the bits of the same matrices side by side."""
    from fellm_b200 import ops
    g = torch.Generator().manual_seed(T)
    H, N, K = 3, 40, 64
    block = torch.randn(H, N + 24, K, generator=g).to(dtype).cuda()
    a = torch.randn(T, H * K, generator=g).to(dtype).cuda()
    out = [torch.empty(T, H * N, dtype=dtype, device="cuda") for _ in range(2)]
    ops.head_gemm(a, block[:, 24:], out[0], a_head=K, out_head=N)
    ops.head_gemm(a, block[:, 24:].contiguous(), out[1], a_head=K, out_head=N)
    assert torch.equal(*out)
