"""A wait that ran out inside a kernel reaches the engine's caller (the count is a stand-in: no kernel is made to wait)."""
import types

import pytest
import torch

from lia_b200 import Engine, ops
from lia_b200._lib import LiaError


class _Model:
    config, device = types.SimpleNamespace(vocab=50), torch.device("cpu")

    def new_state(self, slots, tokens):
        from lia_b200.seq_state import SlotState
        return SlotState(slots, tokens, "cpu")

    def forward_rows(self, ids, batch, want, slots, trace=None):
        return None if want is None else torch.zeros(want.numel(), 50)


def test_the_step_after_a_timeout_raises_once(monkeypatch):
    count = [3]                                            # what happened before this engine is not its business
    monkeypatch.setattr(ops, "moe_timeouts_seen", lambda: count[0])
    e = Engine(_Model(), max_tokens=64)
    entry = [{"id": 0, "tokens": [1, 2], "want": [1]}]
    assert e.step(entry).shape == (1, 50)
    count[0] = 5
    with pytest.raises(LiaError, match="2 blocks"):
        e.step(entry)
    assert e.step(entry).shape == (1, 50)
    count[0] = 6
    with pytest.raises(LiaError):
        e.check()
    e.check()


def test_generate_asks_after_each_step(monkeypatch):
    count, steps = [0], [0]
    monkeypatch.setattr(ops, "moe_timeouts_seen", lambda: count[0])

    def argmax(logits, suppress_id=-1):
        steps[0] += 1
        count[0] = int(steps[0] >= 3)                      # the third step's kernels gave up
        return logits.argmax(-1)
    monkeypatch.setattr(ops, "argmax_f32", argmax)
    with pytest.raises(LiaError):
        Engine(_Model(), max_tokens=64).generate([[1, 2, 3]], 8)
    assert steps[0] == 3


def test_nothing_is_counted_where_nothing_ran():
    assert ops.moe_timeouts_seen() >= 0
