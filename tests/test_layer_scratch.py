"""Forms of a layer that trade scratch for speed: how much they may take, and what is kept of their weights."""
from __future__ import annotations

import pytest
import torch

from fellm_b200 import ops
from fellm_b200.parts.base import build_part
from fellm_b200.parts.spec import PartSpec


def test_latents_per_head_have_a_limit():
    """A step's latents, rotated parts, keys and values per head stay within the limit, whatever the heads and the requests."""
    def rows(H, n_items, longest, T):
        return ops.latent_expand_key_rows(H, 128, 64, 128, 512, 1024, 64, T, n_items, longest)
    assert rows(16, 1, 2048, 2048) == 3136                           # a prompt's portion: 29 MB
    for H in (16, 64, 128):
        for n_items in range(1, 61):
            for T in (512, 2048, 4096, 8192):
                longest = -(-T // n_items)
                n = rows(H, n_items, longest, T)
                assert n_items * n * (512 + 64 + H * 256) * 2 <= ops.LAYER_SCRATCH_MAX_BYTES
    assert rows(16, 53, 78, 4096) == 0 and rows(64, 4, 1024, 4096) > 0


def test_value_projections_are_held_once():
    spec = PartSpec.make("latent_attention", size=256, heads=2, dim=128, rot_dim=64, v_dim=128, q_rank=64, kv_rank=128, scale=0.1, norm_eps=1e-5,
                         window=64, position=PartSpec.make("rope", rot_dim=64, theta=10000.0, pairing="adjacent"))
    part = build_part("mixer", spec, "bfloat16")
    g = torch.Generator().manual_seed(1)
    w = {n: torch.randn(d.shape, generator=g).to(torch.bfloat16 if len(d.shape) > 1 else torch.float32) for n, d in part.param_decls().items()}
    uv = w["uv.weight"].clone()
    part.bind(dict(w))
    kv, got = part.w["kv.weight"], part.w["uv.weight"]
    assert got.untyped_storage().data_ptr() == kv.untyped_storage().data_ptr()
    assert torch.equal(got.reshape(256, 128), uv)


def test_short_steps_keep_the_scan():
    bf, rule = torch.bfloat16, ops.recurrent_chunk_rows
    assert rule(torch.float32, 2048, 1, 2048, 128) == 0
    for key_dim, rows in ((64, 121), (128, 91)):
        assert rule(bf, rows, 1, rows, key_dim) == rule(bf, 4 * 32, 4, 32, key_dim) == ops.RECURRENT_CHUNK_MIN_ROWS
        assert rule(bf, rows - 1, 1, rows - 1, key_dim) == rule(bf, 64, 1, 64, key_dim) == 0
        assert rule(bf, 200 + 15, 16, 200, key_dim) == 0             # one portion among single tokens
        assert rule(bf, 256 + 15, 16, 256, key_dim) > 0


@pytest.mark.gpu
def test_recurrences_beyond_the_limit_keep_the_scan(monkeypatch):
    from test_recurrent_chunk_gpu import MODES, Step
    for mode in MODES:
        s = Step(mode, (70, 40), 2, 2, 64, 64, seed=3)
        scan, _ = s.run(0)
        assert not torch.equal(s.run(32)[0], scan)
        with monkeypatch.context() as m:
            m.setattr(ops, "LAYER_SCRATCH_MAX_BYTES", 1 << 16)
            assert torch.equal(s.run(32)[0], scan)
