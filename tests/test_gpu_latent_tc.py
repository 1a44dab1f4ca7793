"""Latent portions over expanded keys on tcgen05 (csrc/latent_attn_sm100.cu) against a float64 softmax: portions of 1 to 300 rows beside each other behind 0 to 500 positions (blocks of 32 keys to
the third turn of the ring, tiles of 128 rows, a portion's last block beside the next portion's rows), windows, sinks, gates, scales of either sign and near 0, both outputs, and a workspace
that holds a group of heads; and the expansion (csrc/latent_expand_sm100.cu) of latents of 64 to 512 numbers, beside those it leaves to mma.sync."""
import math

import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DIM, ROT, RANK = 128, 64, 64
PORTIONS = [(1, 0, 0, 300), (0, 500, 300, 129), (2, 31, 429, 1), (3, 0, 430, 33)]        # slot, first position, first row, rows
# scores of size 5 carry about 5 * 2^-23 * sqrt(192) of relative error through exp: below 1e-5 of the largest value with room to spare
TOL = 1e-5


def reference(q, qr, lat, w, H, scale, window, sink, gate):
    out = torch.zeros(q.shape[0], H, DIM, dtype=F64, device="cuda")
    for slot, p0, r0, n in PORTIONS:
        c, pos, j = lat[slot, :p0 + n].to(F64), torch.arange(p0, p0 + n, device="cuda")[:, None], torch.arange(p0 + n, device="cuda")[None, :]
        seen = (j <= pos) & ((pos - j < window) if window else True)
        for h in range(H):
            k, v = (c[:, :RANK] @ w[(t * H + h) * DIM:(t * H + h + 1) * DIM].to(F64).T for t in (0, 1))
            s = (q[r0:r0 + n].view(n, H, DIM + ROT)[:, h, :DIM].to(F64) @ k.T + qr[r0:r0 + n, h].to(F64) @ c[:, RANK:].T) * scale
            s = s.masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].to(F64).expand(n, 1)], 1)
            out[r0:r0 + n, h] = torch.softmax(s, -1)[:, :p0 + n] @ v
    return (out * gate[:, :, None].to(F64) if gate is not None else out).reshape(q.shape[0], -1)


@pytest.mark.parametrize("H,window,scale,sink,gate", [(2, 0, 0.1, False, False), (5, 40, 0.1, True, True), (3, 200, -0.1, False, True), (1, 0, 0.0, True, False), (2, 33, 1e-9, False, False)])
def test_portions(H, window, scale, sink, gate):
    g = torch.Generator().manual_seed(H)
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    M = PORTIONS[-1][2] + PORTIONS[-1][3]
    q, qr = rnd(M, H * (DIM + ROT)).to(BF16).cuda(), rnd(M, H, ROT).cuda()
    lat, w = rnd(4, 640, RANK + ROT).to(BF16).cuda(), (rnd(2 * H * DIM, RANK) * RANK ** -0.5).to(BF16).cuda()
    for slot, p0, _, n in PORTIONS:
        lat[slot, p0 + n:] = float("nan")                           # what lies behind a sequence's last position is never read
    sk, gt = (rnd(H).cuda() if sink else None), (torch.rand(M, H, generator=g).cuda() if gate else None)
    want = reference(q, qr, lat, w, H, scale, window, sk, gt)

    def run(dtype, portions=PORTIONS, **kw):
        out = torch.full((M, H * DIM), 7.0, dtype=dtype, device="cuda")
        return ops.latent_attn_expanded(q, qr, lat, portions, w, gt, out, H, DIM, ROT, RANK, scale, window=window, sink=sk, **kw)
    out = run(F32)
    assert float((out.to(F64) - want).abs().max() / want.abs().max()) < TOL
    assert float((run(BF16).to(F64) - want).abs().max() / want.abs().max()) < 2.0 ** -8
    assert torch.equal(run(F32, room=700), out)                     # heads in turn: the same sums
    for slot, p0, r0, n in PORTIONS:                                # a portion does not depend on its company
        assert torch.equal(run(F32, [(slot, p0, r0, n)])[r0:r0 + n], out[r0:r0 + n])


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("rank", [64, 128, 192, 448, 512, 576, 72])
def test_expansion(dim, rank):
    """One row that sees one latent gives back its value, the sum of its three parts."""
    H, slots, cap = 3, 2, 140
    g = torch.Generator().manual_seed(rank)
    lat = torch.randn(slots, cap, rank + ROT, generator=g).to(BF16).cuda()
    w = (torch.randn(2 * H * dim, rank, generator=g) * rank ** -0.5).to(BF16).cuda()
    q, qr = torch.zeros(cap, H * (dim + ROT), dtype=BF16, device="cuda"), torch.zeros(cap, H, ROT, device="cuda")
    out = torch.empty(cap, H * dim, dtype=F32, device="cuda")
    ops.latent_attn_expanded(q, qr, lat, [(1, 0, 0, cap)], w, None, out, H, dim, ROT, rank, 1.0, window=1)
    want = lat[1, :, :rank].to(F64) @ w[H * dim:].to(F64).T
    assert float((out.to(F64) - want).abs().max()) < 2.0 ** -20      # sums of size up to 5: a few last places of 2^-21


def test_weights_below_the_smallest_normal_number():
    """A weight of exp(-88.5) = 2^-127.7, as three parts of which the first has five bits left, times a value of 2^127."""
    H = 2
    q, qr, lat, w = (torch.zeros(*s, device="cuda") for s in ((2, H * (DIM + ROT)), (2, H, ROT), (1, 2, RANK + ROT), (2 * H * DIM, RANK)))
    qr[:, :, 3], lat[0, 1, RANK + 3], lat[0, 1, 7], w[H * DIM + 5, 7] = 1.0, -88.5, 2.0 ** 100, 2.0 ** 27
    out = torch.empty(2, H * DIM, device="cuda")
    ops.latent_attn_expanded(q.to(BF16), qr, lat.to(BF16), [(0, 0, 0, 2)], w.to(BF16), None, out, H, DIM, ROT, RANK, 1.0)
    assert abs(float(out[1, 5]) / (math.exp(-88.5) * 2.0 ** 127) - 1) < 2.0 ** -5 and float(out.abs().sum() - out[1, 5].abs()) == 0.0
