"""The matrix-memory recurrence where a head has more blocks than the chip holds at a time: every block of a head starts from the same normaliser and
stabiliser, also when the head's first block is long done; and through the entry without a workspace."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import _lib, ops

pytestmark = pytest.mark.gpu
F32 = torch.float32


def _inputs(seqs, tokens, H, d, e):
    g = torch.Generator(device="cuda").manual_seed(seqs)
    M = seqs * tokens
    y = torch.randn(M, 2 * H * d + H * e, generator=g, device="cuda")
    gates = torch.randn(M, 2 * H, generator=g, device="cuda")
    gates[:, H:] = -gates[:, H:].abs()
    state = [torch.randn(seqs, H, *s, generator=g, device="cuda") for s in ((e, d), (d,), ())]
    return y, gates, state, torch.tensor([(s, 3, s * tokens, tokens) for s in range(seqs)], dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("seqs,tokens", [(64, 1), (40, 9)])
def test_many_heads_at_once(seqs, tokens):
    H, d, e = 4, 256, 512
    y, gates, state, segs = _inputs(seqs, tokens, H, d, e)
    want, alone = torch.empty(seqs * tokens, H * e, dtype=F32, device="cuda"), [t.clone() for t in state]
    part = lambda t: (t[:, :H * d], t[:, H * d:2 * H * d], t[:, 2 * H * d:])
    for s in range(seqs):                                     # each sequence by itself: all its blocks are resident
        rows = slice(s * tokens, (s + 1) * tokens)
        one = torch.tensor([(s, 3, 0, tokens)], dtype=torch.int32, device="cuda")
        ops.mlstm_scan(*part(y[rows]), gates[rows], *alone, one, H, d, e, d ** -0.5, 1e-6, want[rows])
    for entry in ("ops", "plain"):
        st, o = [t.clone() for t in state], torch.empty_like(want)
        if entry == "ops":
            ops.mlstm_scan(*part(y), gates, *st, segs, H, d, e, d ** -0.5, 1e-6, o)
        else:
            q, k, v = (t.data_ptr() for t in part(y))
            rc = _lib.load().lia_mlstm_scan(q, k, v, 1, y.stride(0), gates.data_ptr(), *(t.data_ptr() for t in st), segs.data_ptr(), seqs, H, d, e, d ** -0.5, 1e-6,
                                            o.data_ptr(), torch.cuda.current_stream().cuda_stream)
            assert rc == 0
        assert torch.equal(o, want) and all(torch.equal(a, b) for a, b in zip(st, alone))
