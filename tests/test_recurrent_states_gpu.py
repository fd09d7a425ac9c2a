"""Recurrences in chunks, in both forms: one walk over the chunks, or the states in front of the chunks first and the outputs beside one
another behind them.  More chunks than are read ahead, last chunks of one to five tokens, value columns that end inside a block's 64 or
pass the keys' number."""
from __future__ import annotations

import pytest
import torch

import test_recurrent_chunk_gpu
from test_recurrent_chunk_gpu import MODES, Step, near

pytestmark = pytest.mark.gpu


def choose(monkeypatch, apart):
    """Every portion in one walk (False) or apart (True), whatever its length; -> the list of the forms that the launches take."""
    from fellm_b200 import ops
    monkeypatch.setattr(ops, "RECURRENT_APART_ROWS", 1 if apart else 1 << 30)
    monkeypatch.setattr(ops, "RECURRENT_APART_ROWS_FULL", 1 if apart else 1 << 30)
    taken, fn = [], ops._fn

    def watched(module, name, *args, **kw):
        f = fn(module, name, *args, **kw)
        if name != "fellm_recurrent_chunk":
            return f
        return lambda *a: (taken.append(bool(a[-2])), f(*a))[1]
    monkeypatch.setattr(ops, "_fn", watched)
    return taken


@pytest.fixture(params=[False, True], ids=["walk", "apart"])
def form(request, monkeypatch):
    taken = choose(monkeypatch, request.param)
    yield
    assert taken and set(taken) == {request.param}


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens,H,G,dk,dv", [((289,), 2, 1, 64, 80), ((33, 34, 35, 36, 37), 2, 2, 64, 144), ((258, 160), 2, 2, 128, 144),
                                            ((131, 32), 1, 1, 128, 16), ((64, 1, 355), 2, 1, 128, 256), ((1030,), 13, 13, 128, 128)])
def test_states_and_outputs_are_the_walk(form, mode, lens, H, G, dk, dv):
    if mode == "decay_bonus":
        dv = dk
    if not mode.endswith("delta"):
        G = H
    for zero in (False, True):
        s = Step(mode, lens, H, G, dk, dv, seed=sum(lens), decay_zero=zero)
        o, st = s.run(32)
        want, want_state = s.oracle()
        assert near(o, want) and near(st, want_state)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens,H,G,dk,dv", [((289,), 2, 1, 64, 80), ((33, 34, 35, 36, 37), 2, 2, 64, 144), ((64, 1, 355), 2, 1, 128, 256), ((700, 330), 3, 3, 128, 16)])
def test_both_forms_have_the_same_bits(monkeypatch, mode, lens, H, G, dk, dv):
    """What else is in a step chooses the form: it must not be in a portion's bits."""
    if mode == "decay_bonus":
        dv = dk
    if not mode.endswith("delta"):
        G = H
    got = []
    for apart in (False, True):
        with monkeypatch.context() as m:
            taken = choose(m, apart)
            got.append(Step(mode, lens, H, G, dk, dv, seed=sum(lens), decay_zero=True).run(32))
            assert taken == [apart]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("mode", MODES)
def test_short_items_keep_the_scan(form, mode):
    test_recurrent_chunk_gpu.test_short_items_keep_the_scan(mode)


@pytest.mark.parametrize("mode", MODES)
def test_a_later_token_leaves_earlier_ones_alone(form, mode):
    test_recurrent_chunk_gpu.test_a_later_token_leaves_earlier_ones_alone(mode)


@pytest.mark.parametrize("alike", [False, True])
@pytest.mark.parametrize("mode", MODES)
def test_chunks_are_no_less_exact_than_the_walk(form, mode, alike):
    test_recurrent_chunk_gpu.test_chunks_are_no_less_exact_than_the_walk(mode, alike)


@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("mode", MODES)
def test_states_anywhere(form, mode, dk):
    """States are read and written element by element: a slot may start anywhere and be any number of floats behind the one before."""
    from fellm_b200 import ops
    s = Step(mode, (70, 33), 2, 2, dk, dk, seed=dk)
    o, st = s.run(32)
    keep, args = [], ops._state_args

    def shifted(state):
        wide = torch.full((state.shape[0], state[0].numel() + 5), 7.0, device=state.device)
        wide[:, 3:-2] = state.view(state.shape[0], -1)
        keep.append((state, wide))
        return args(wide[:, 3:-2])
    with pytest.MonkeyPatch.context() as m:
        m.setattr(ops, "_state_args", shifted)
        o2, _ = s.run(32)
    state, wide = keep[0]
    assert torch.equal(o, o2) and torch.equal(wide[:, 3:-2].double().cpu().view(st.shape), st)
    assert (wide[:, :3] == 7).all() and (wide[:, -2:] == 7).all()


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens", [(40, 40), (32, 33, 34), (60, 31), (96, 33, 32), (96, 64, 1)])
def test_the_scan_behind_the_chunks_is_left_out_for_nobody(mode, lens):
    """Steps whose portions are all of 32 rows or more, by their sum or only in fact, and steps with one that is not."""
    from fellm_b200 import ops
    assert ops._no_item_below(32, sum(lens), len(lens), max(lens)) == (sum(lens) - (len(lens) - 1) * max(lens) >= 32)
    s = Step(mode, lens, 2, 2, 64, 64, seed=sum(lens))
    o, st = s.run(32)
    want, want_state = s.oracle()
    assert near(o, want) and near(st, want_state)


@pytest.mark.parametrize("mode", ["decay_bonus", "gated_write"])
def test_rows_in_front_of_the_first_item_are_nobodys(form, mode):
    from fellm_b200 import ops
    H, dk, front, n = 2, 64, 70, 75
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    z, decay, bonus = rnd(front + n, 3 * H * dk), torch.rand(front + n, H * dk, generator=g, device="cuda"), rnd(H, dk)
    lower, bias = torch.rand(H * dk, generator=g, device="cuda"), rnd(H * dk)

    def run(first):
        m, w, state = z[front - first:].contiguous(), decay[front - first:].contiguous(), torch.zeros(1, H, dk, dk, device="cuda")
        out = torch.full((first + n, H * dk), 3.0, device="cuda")
        at = dict(item_start=torch.tensor([first, first + n], dtype=torch.int32, device="cuda"), item_slot=torch.zeros(1, dtype=torch.int32, device="cuda"))
        if mode == "decay_bonus":
            ops.decay_bonus_scan(m[:, :H * dk], m[:, H * dk:2 * H * dk], m[:, 2 * H * dk:], w, bonus, state, n_items=1, H=H, dk=dk, out=out,
                                 max_item_rows=n, chunk_rows=32, **at)
        else:
            ops.gated_write_scan(m, H * dk, 2 * H * dk, lower, bias, state, n_items=1, H=H, dk=dk, dv=dk, out=out, max_item_rows=n, chunk_rows=32, **at)
        return out, state
    (out, state), (alone, alone_state) = run(front), run(0)
    assert (out[:front] == 3).all() and torch.equal(out[front:], alone) and torch.equal(state, alone_state)
