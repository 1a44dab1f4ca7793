"""Decode attention around the edges of its stream of row loads: a CTA's four warps keep ten rows a lane on their way, two or four where those are all, K's and
then V's, so that histories just below, at and above whole batches (16, 32 and 80 rows of 128 values, 32, 64 and 160 of 64) take every mixture of
"the next row is K's", "is V's" and "is not there"."""
import pytest
import torch

from test_gpu_kernels import attn_ref, close_bf16, ops, rnd  # noqa: F401  (ops is the fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,T,splits", [(128, t, 1) for t in (1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 79, 80, 81, 160, 161)] +
                         [(64, t, 1) for t in (1, 15, 17, 31, 32, 33, 63, 64, 65, 159, 160, 161, 321)] +
                         [(128, 167, 2), (64, 331, 3), (128, 64, 2), (128, 31, 2), (64, 130, 2)])
def test_histories_around_whole_batches(ops, d, T, splits):  # noqa: F811
    B, H, Bc, b0 = 2, 3, 4, 1
    q = rnd(B, H, d, std=0.3, seed=4)
    kc, vc = (rnd(T + 2, Bc, H, d, seed=s) for s in (5, 6))
    kc[T:], vc[T:] = float("nan"), float("nan")              # rows that no token has written yet
    ws = ops.attn_decode_workspace(B, H, d, "cuda")
    out = ops.attn_decode(q.view(B, H * d), kc, vc, B, T, b0, splits=splits, workspace=ws)
    ref = attn_ref(q.view(B, H, 1, d), kc[:T, b0:b0 + B].permute(1, 2, 0, 3), vc[:T, b0:b0 + B].permute(1, 2, 0, 3), False).reshape(B, H * d)
    # a score or a probability may round to the neighbouring bf16 value, and so may the sum: two steps of the row's largest
    # value, four where the parts of a split history are joined in 32 bits without the probabilities' rounding
    close_bf16(out, ref, ulps=2.01 if splits == 1 else 4.01, what=f"decode attention T={T} d={d}", scale=ref.abs().amax(-1, keepdim=True))
