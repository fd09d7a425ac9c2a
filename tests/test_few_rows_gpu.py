"""Decode steps of few rows that are filled up to a count the tcgen05 products take (engine/step.py): the logits of the rows
asked for, whatever was filled in, and no trace of the filling in the requests' caches."""
from __future__ import annotations

import types

import pytest
import torch


def test_which_models_are_filled_up():
    from fellm_b200.engine.step import few_rows_pad_from

    def model(width, mixer="shortconv", ffn="swiglu", dtype=torch.bfloat16):
        block = types.SimpleNamespace(mixer=types.SimpleNamespace(kind=mixer), ffn=types.SimpleNamespace(kind=ffn))
        return types.SimpleNamespace(blocks=[block], spec=types.SimpleNamespace(hidden_size=width), act_dtype=dtype)
    assert [few_rows_pad_from(model(w)) for w in (512, 768, 1024, 1152, 1280, 1536, 1792, 2048, 2304, 3072)] == [17, 17, 17, 17, 17, 2, 2, 9, 9, 2]
    assert few_rows_pad_from(model(1536, ffn="moe")) == few_rows_pad_from(model(1536, mixer="gated_delta")) == 17
    assert few_rows_pad_from(model(1536, dtype=torch.float32)) == 17


def test_which_feed_forwards_are_filled_up():
    """Gate and up within the few-rows product's columns (up to width 2048), and large enough for two rows to gain; LFM2's own parts only."""
    from fellm_b200.engine.step import few_rows_pad_from

    def pad(width, ff, general=False):
        block = types.SimpleNamespace(mixer=types.SimpleNamespace(kind="attention", general=general), ffn=types.SimpleNamespace(kind="swiglu", ff=ff))
        return few_rows_pad_from(types.SimpleNamespace(blocks=[block], spec=types.SimpleNamespace(hidden_size=width), act_dtype=torch.bfloat16))
    assert [pad(1536, ff) for ff in (4608, 6144, 7168, 8192, 9216)] == [9, 2, 2, 2, 17]
    assert [pad(2048, ff) for ff in (8192, 9728, 10240)] == [9, 17, 17]
    assert pad(1792, 8192) == 2 and pad(2304, 10752) == pad(2560, 12288) == 9 and pad(3072, 14336) == 2
    assert pad(1536, 7168, general=True) == 17


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 7, 16])
def test_filled_up_steps_give_the_rows_own_logits(n):
    from fellm_b200.config import EngineOptions
    from fellm_b200.engine import Engine, StepItem
    cfg = dict(architectures=["Lfm2ForCausalLM"], vocab_size=640, hidden_size=1536, num_hidden_layers=3, num_attention_heads=24,
               num_key_value_heads=8, head_dim=64, full_attn_idxs=[1], block_ff_dim=512, block_auto_adjust_ff_dim=False,
               rope_theta=10000.0, rope_pairing="split_half", conv_L_cache=3, conv_bias=False, norm_eps=1e-5, tie_word_embeddings=True,
               max_position_embeddings=512)
    engines = [Engine.random(cfg, 7, EngineOptions(n_ctx=256, max_requests=16, max_tokens=16 * 128, cuda_graphs=g)) for g in (True, False)]
    g = torch.Generator().manual_seed(n)
    prompts = [torch.randint(0, 640, (3 + 5 * r,), generator=g).tolist() for r in range(n)]
    follow = torch.randint(0, 640, (n, 5), generator=g).tolist()
    got = []
    for e in engines:
        for r in range(n):
            e.add_request(r)
            e.step([StepItem(r, prompts[r], [])])
        out = [e.step([StepItem(r, [follow[r][t]], [0]) for r in range(n)]).double().cpu() for t in range(4)]
        # behind the filled-up steps, some rows alone and without logits: what the filling left must not show
        e.step([StepItem(r, [follow[r][4]], []) for r in range(n)])
        out.append(e.step([StepItem(0, [1], [0])]).double().cpu())
        e.check_status()
        e.cache.audit()
        got.append(out)
    for a, b in zip(*got):
        assert a.shape == b.shape and torch.isfinite(a).all()
        # two kernels of the same bfloat16 operands: other orders of float32 sums, then roundings of activations
        assert float((a - b).norm() / b.norm()) < 2e-2


@pytest.mark.gpu
@pytest.mark.parametrize("width,n", [(1536, 2), (1536, 16), (2048, 9), (2048, 16)])
def test_filled_up_steps_plan_for_the_requests_rows(width, n, monkeypatch):
    """Contexts beyond 1,024 keys: attention's key ranges are those of the requests' rows, the logits those of a step as it is, and
    greedy steps pick their tokens without the logits, as such a step does."""
    from fellm_b200 import ops
    from fellm_b200.config import EngineOptions
    from fellm_b200.engine import Engine, StepItem
    cfg = dict(architectures=["Lfm2ForCausalLM"], vocab_size=640, hidden_size=width, num_hidden_layers=3, num_attention_heads=width // 64,
               num_key_value_heads=8, head_dim=64, full_attn_idxs=[1], block_ff_dim=6144 if width == 1536 else 512, block_auto_adjust_ff_dim=False,
               rope_theta=10000.0, rope_pairing="split_half", conv_L_cache=3, conv_bias=False, norm_eps=1e-5, tie_word_embeddings=True,
               max_position_embeddings=4096)
    options = dict(n_ctx=2048, max_requests=16, max_tokens=16 * 1280, n_batch=2048)
    engines = [Engine.random(cfg, 7, EngineOptions(cuda_graphs=g, **options)) for g in (True, False)]
    g = torch.Generator().manual_seed(n)
    prompts = [torch.randint(0, 640, (1025 + 7 * r,), generator=g).tolist() for r in range(n)]
    follow = torch.randint(0, 640, (n, 4), generator=g).tolist()
    assert n >= engines[0].stepper.pad_from
    planned, picked = [], []
    split, argmax = ops.decode_split, ops.gemm_bf16_argmax
    monkeypatch.setattr(ops, "decode_split", lambda max_len, rows, *a, **k: planned.append(rows) or split(max_len, rows, *a, **k))
    monkeypatch.setattr(ops, "gemm_bf16_argmax", lambda x, *a, **k: picked.append(x.shape[0]) or argmax(x, *a, **k))
    got = []
    for e in engines:
        for r in range(n):
            e.add_request(r)
            e.step([StepItem(r, prompts[r], [])])
        out = [e.step([StepItem(r, [follow[r][t]], [0]) for r in range(n)]).double().cpu() for t in range(3)]
        items = [StepItem(r, [follow[r][3]], [0]) for r in range(n)]
        if e is engines[0]:
            tokens = torch.full((n,), -1, dtype=torch.int32, device="cuda")
            assert e.stepper.step(items, greedy_tokens=tokens) is None and picked == [n]
        else:
            out.append(e.step(items).double().cpu())
        e.check_status()
        e.cache.audit()
        got.append(out)
    assert planned and set(planned) == {n}
    for a, b in zip(*got):
        assert a.shape == b.shape and torch.isfinite(a).all()
        assert float((a - b).norm() / b.norm()) < 2e-2                     # as above
    near_best(got[1][3], tokens.cpu())


def near_best(logits, tokens):
    """Every token is its row's best, up to what two kernels' roundings of the logits may turn: 2e-2 of their size, twice."""
    slack = 0.08 * logits.pow(2).mean(-1).sqrt()
    assert bool((logits.gather(1, tokens.long()[:, None])[:, 0] >= logits.max(-1).values - slack).all())


@pytest.mark.gpu
def test_greedy_generation_of_a_filled_up_batch(monkeypatch):
    """Engine.generate_batch where steps are filled up: tokens picked for the requests' rows, each its own context's best."""
    from fellm_b200 import ops
    from fellm_b200.config import EngineOptions
    from fellm_b200.engine import Engine, GenParams, StepItem
    cfg = dict(architectures=["Lfm2ForCausalLM"], vocab_size=640, hidden_size=1536, num_hidden_layers=3, num_attention_heads=24,
               num_key_value_heads=8, head_dim=64, full_attn_idxs=[1], block_ff_dim=6144, block_auto_adjust_ff_dim=False,
               rope_theta=10000.0, rope_pairing="split_half", conv_L_cache=3, conv_bias=False, norm_eps=1e-5, tie_word_embeddings=True,
               max_position_embeddings=512)
    e = Engine.random(cfg, 7, EngineOptions(n_ctx=256, max_requests=16, max_tokens=16 * 128, cuda_graphs=True))
    assert e.stepper.pad_from <= 5
    prompts = [torch.randint(0, 640, (3 + 5 * r,), generator=torch.Generator().manual_seed(r)).tolist() for r in range(5)]
    picked, argmax = [], ops.gemm_bf16_argmax
    monkeypatch.setattr(ops, "gemm_bf16_argmax", lambda x, *a, **k: picked.append(x.shape[0]) or argmax(x, *a, **k))
    streams, _ = e.generate_batch(prompts, GenParams.greedy(6))
    assert 5 in picked and max(picked) <= 16
    for r, (p, t) in enumerate(zip(prompts, streams)):
        assert len(t) == 6
        e.add_request(("check", r))
        logits = e.step([StepItem(("check", r), p + t[:-1], list(range(len(p) - 1, len(p) + 5)))]).double().cpu()
        e.release(("check", r))
        near_best(logits, torch.tensor(t))
