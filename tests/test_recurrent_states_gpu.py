"""Recurrences in chunks, the states in front of the chunks and the outputs made beside one another: more chunks than are read ahead, last
chunks of one to five tokens (the last ones' terms are added by themselves), value columns that end inside a block's 64 or pass the
keys' number."""
from __future__ import annotations

import pytest

from test_recurrent_chunk_gpu import MODES, Step, near

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("lens,H,G,dk,dv", [((289,), 2, 1, 64, 80), ((33, 34, 35, 36, 37), 2, 2, 64, 144), ((258, 160), 2, 2, 128, 144),
                                            ((131, 32), 1, 1, 128, 16), ((64, 1, 355), 2, 1, 128, 256), ((1030,), 13, 13, 128, 128)])
def test_states_and_outputs_are_the_walk(mode, lens, H, G, dk, dv):
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
@pytest.mark.parametrize("lens", [(40, 40), (32, 33, 34), (60, 31), (96, 33, 32), (96, 64, 1)])
def test_the_scan_behind_the_chunks_is_left_out_for_nobody(mode, lens):
    """Steps whose portions are all of 32 rows or more, by their sum or only in fact, and steps with one that is not."""
    from fellm_b200 import ops
    assert ops._no_item_below(32, sum(lens), len(lens), max(lens)) == (sum(lens) - (len(lens) - 1) * max(lens) >= 32)
    s = Step(mode, lens, 2, 2, 64, 64, seed=sum(lens))
    o, st = s.run(32)
    want, want_state = s.oracle()
    assert near(o, want) and near(st, want_state)
