"""What the tcgen05 products of many rows write: every epilogue at rows and columns that end inside a tile, a warp's 32 rows, a chunk of 32
columns and a 16-byte piece of a row, into outputs whose rows or first element are not on 16 bytes, beside what must stay."""
from __future__ import annotations

import pytest
import torch

DEV = "cuda"


def _near(got, a, b, want, out_bf16):
    """K products of bfloat16 numbers summed in float32 in any order, truncating (K 2^-23 of the sum of magnitudes), then one rounding to
    the output's type; a gated or squared output multiplies two such sums: four times that."""
    K = a.shape[1]
    room = 4 * K * 2.0 ** -23 * (a.abs() @ b.abs().T) + (2.0 ** -8 if out_bf16 else 2.0 ** -22) * want.abs() + 1e-6
    assert ((got.double() - want).abs() <= room).all(), float(((got.double() - want).abs() / room).max())


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(129, 24, 64), (161, 36, 1024), (300, 1000, 2048), (257, 255, 2176), (385, 512, 136), (1030, 272, 4096), (2048, 2064, 128), (1285, 2560, 256)])
@pytest.mark.parametrize("shift,pad", [(0, 0), (8, 24), (0, 4), (3, 7)])
@pytest.mark.parametrize("epi", ["store", "relu2", "acc", "f32", "bias"])
def test_rows_and_columns_that_end_anywhere(M, N, K, shift, pad, epi):
    from fellm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N + K + shift)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    bias = torch.randn(N, generator=g, device=DEV) if epi in ("bias", "acc") else None
    dt = torch.float32 if epi in ("acc", "f32") else torch.bfloat16
    held = torch.randn(shift + (M + 1) * (N + pad), generator=g, device=DEV).to(dt)
    before = held.clone()
    view = lambda t: t[shift:shift + M * (N + pad)].view(M, N + pad)[:, :N]  # noqa: E731
    ops.gemm_bf16(x, w, bias, out=view(held), accumulate=epi == "acc", act="relu2" if epi == "relu2" else None)
    ops.check_umma_status(DEV)
    a, b = x.double(), w.double()
    want = a @ b.T + (bias.double() if bias is not None else 0.0)
    if epi == "acc":
        want = want + view(before).double()
    if epi == "relu2":
        scale = want.abs().max()
        want = want.clamp(min=0) ** 2
        _near(view(held), a * 2 * (1 + scale), b, want, True)
    else:
        _near(view(held), a, b, want, dt == torch.bfloat16)
    view(held).copy_(view(before))
    assert torch.equal(held, before), "something beside the product's rows was written"


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(129, 16, 64), (300, 1008, 1024), (600, 4624, 2048), (1030, 528, 256)])
def test_gated_columns_that_end_anywhere(M, N, K):
    from fellm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    wg, wu = ((torch.randn(N // 2, K, generator=g, device=DEV) * K ** -0.5).bfloat16() for _ in range(2))
    held = torch.full((M + 1, N // 2 + 8), 3.0, device=DEV, dtype=torch.bfloat16)
    ops.gemm_bf16(x, ops.interleave_gate_up(wg, wu), out=held[:M, :N // 2], swiglu=True)
    ops.check_umma_status(DEV)
    a = x.double()
    gate, up = a @ wg.double().T, a @ wu.double().T
    want = torch.nn.functional.silu(gate) * up
    sums = 4 * K * 2.0 ** -23 * torch.maximum(a.abs() @ wg.double().abs().T, a.abs() @ wu.double().abs().T)
    room = 1.1 * sums * (gate.abs() + up.abs() + 1) + 2.0 ** -7 * want.abs() + 1e-6          # (|silu'| <= 1.1; the exponential's own 2^-21)
    assert ((held[:M, :N // 2].double() - want).abs() <= room).all()
    assert (held[M:] == 3).all() and (held[:, N // 2:] == 3).all()


@pytest.mark.gpu
@pytest.mark.parametrize("K", [512, 584, 1024, 1976, 2048])
@pytest.mark.parametrize("M,N", [(129, 1000), (600, 1024), (1100, 1024), (300, 96)])
@pytest.mark.parametrize("epi", ["f32", "acc", "store"])
def test_few_tiles_add_two_halves_of_k(M, N, K, epi):
    """Products of few tiles: two sums over half of K each, added with rounding, whether one CTA or two make them (an MMA that adds into
    its accumulator truncates: one sum over all of K is less exact).  The halves' own sums: the same rows in a product of so many tiles that
    none is halved."""
    from fellm_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    dt = torch.bfloat16 if epi == "store" else torch.float32
    out = torch.randn(M, N, generator=g, device=DEV).to(dt)
    held = out.clone()
    ops.gemm_bf16(x, w, out=out, accumulate=epi == "acc")
    cut = 64 * (-(-K // 64) // 2)
    many = -(-148 * 128 // M) + 1
    parts = [ops.gemm_bf16(x[:, at].repeat(many, 1), w[:, at].contiguous(), out_dtype=torch.float32)[:M] for at in (slice(0, cut), slice(cut, K))]
    ops.check_umma_status(DEV)
    want = parts[0] + parts[1]
    if epi == "acc":
        want = want + held
    assert torch.equal(out, want.to(dt))
    x, w = x.double(), w.double()
    exact = x @ w.T + (held.double() if epi == "acc" else 0.0)
    whole = ops.gemm_bf16(x.bfloat16().repeat(many, 1), w.bfloat16(), out_dtype=torch.float32)[:M].double()
    if epi == "f32":
        assert float((out.double() - exact).norm()) < float((whole - exact).norm())
