"""The tensor-core kernels behind ``linear_plain`` (csrc/linear_mma.cu) and latent attention of long portions (csrc/latent_attn_mma.cu) against
float64, at the edges of their tiles."""
import math

import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops
from lia_b200.seq_layers import LatentAttentionMixer, StepBatch
from lia_b200.seq_state import SlotState

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DEV = "cuda"


@pytest.mark.parametrize("a_dt,w_dt,c_dt", [(BF16, BF16, F32), (BF16, BF16, BF16), (F32, BF16, F32), (F32, BF16, BF16), (F32, F32, F32), (F32, F32, BF16), (BF16, F32, F32)])
@pytest.mark.parametrize("M,N,K,batch", [(65, 64, 8, 1), (127, 61, 40, 3), (128, 128, 64, 2), (129, 130, 96, 1), (300, 7, 520, 1), (200, 257, 1000, 2)])
def test_linear_plain(a_dt, w_dt, c_dt, M, N, K, batch):
    g = torch.Generator().manual_seed(M + N)
    a = torch.randn(M, batch * K + 8, generator=g).to(a_dt)[:, 8:]                        # batches side by side in a wider buffer
    a[1, 0], a[M - 1, 0] = 1e30, -1e-30
    a = torch.cat([torch.zeros(M, 8, dtype=a_dt), a], 1).to(DEV)[:, 8:]
    w = torch.randn(batch, N, K, generator=g).to(w_dt).to(DEV)
    out = torch.full((M, batch * N + 3), 7.0, dtype=c_dt, device=DEV)
    ops.linear_plain(a, w, out, scale=0.5, batch=batch, a_batch_stride=K, w_batch_stride=N * K, out_batch_stride=N, n=N, k=K)
    A, W = a.cpu().to(F64).reshape(M, batch, K), w.cpu().to(F64)
    want, size = 0.5 * torch.einsum("mbk,bnk->mbn", A, W).reshape(M, -1), 0.5 * torch.einsum("mbk,bnk->mbn", A.abs(), W.abs()).reshape(M, -1)
    got = out.cpu().to(F64)
    # tensor cores: fp32 sums over stages of 32 channels, each within 2^-24 of the partial sum, and parts left out 2^-24 below; bf16 x fp32 stays
    # on the CUDA cores: one chain of K fused multiply-adds, each within 2^-24 of a partial sum that `size` bounds
    bound = size * (K * 2.0 ** -24 if a_dt == BF16 and w_dt == F32 else 2.0 ** -22) + (want.abs() * 2.0 ** -8 if c_dt == BF16 else 0.0)
    assert bool(((got[:, :batch * N] - want).abs() <= bound + 1e-37).all())
    assert bool((got[:, batch * N:] == 7.0).all())


def mixer(H, dim, rank, gate, sink, window, seed):
    g = torch.Generator().manual_seed(seed)
    W = 64

    def r(*s):
        return (torch.randn(*s, generator=g) * s[-1] ** -0.5).to(BF16).float()
    w = {"q": r(H * (dim + 64), W) * 4, "dkv": r(rank + 64, W), "dkv.norm": torch.ones(rank), "uk": r(H * dim, rank), "uv": r(H * dim, rank), "o": r(W, H * dim)}
    if gate:
        w["g"] = r(H if gate == "head" else H * dim, W)
    if sink:
        w["sink"] = torch.linspace(-1.0, 1.0, H)
    return LatentAttentionMixer(w, H, dim, 64, dim, rank, 32, 10000.0, 0.2, 1e-6, BF16, DEV, gate=gate, window=window, sink=sink), torch.randn(400, W, generator=g).to(BF16).to(DEV)


def step(m, state, h, portions):
    segs, meta, row = [], [], 0
    for slot, p0, n in portions:
        segs.append((slot, p0, row, n))
        meta += [(slot, p0 + i) for i in range(n)]
        row += n
    i32 = dict(dtype=torch.int32, device=DEV)
    return m(h[:row], StepBatch(row, torch.tensor(segs, **i32), torch.tensor(meta, **i32), max(p + n for _, p, n in portions), portions=segs), state)


@pytest.mark.parametrize("dim,rank,gate,sink,window", [(128, 512, "head", False, 0), (64, 72, None, True, 40), (128, 64, "channel", True, 100), (64, 256, "head", False, 33)])
def test_latent_portions(dim, rank, gate, sink, window, monkeypatch):
    """Portions of one step in both orders of the projections, against each other: the results may differ by the rounding of the output alone."""
    H = 3
    m, h = mixer(H, dim, rank, gate, sink, window, 5)
    assert m.w_ukv is not None
    many = [(i, 3 * i, 16 + i % 3) for i in range(18)]           # more than one launch holds
    for portions in ([(0, 0, 32)], [(0, 0, 1), (2, 70, 64), (1, 5, 65), (3, 0, 7), (4, 129, 130)], [(1, 200, 33), (0, 0, 200)], many):
        got = []
        for rows in (1 << 30, LatentAttentionMixer.EXPAND_ROWS_EXACT):
            monkeypatch.setattr(LatentAttentionMixer, "EXPAND_ROWS_EXACT", rows)
            slots = SlotState(18, 280, DEV)
            state = m.new_state(slots)
            state[0].copy_(torch.randn(state[0].shape, generator=torch.Generator().manual_seed(1)).to(BF16))
            for slot, p0, n in portions:
                state[0][slot, p0 + n:] = float("nan")          # what lies behind the last position is never read
            got.append(step(m, state, h, portions).double())
            monkeypatch.undo()
        assert float((got[0] - got[1]).norm() / got[0].norm()) < 2e-3 and float((got[0] - got[1]).abs().max() / got[0].abs().max()) < 2.0 ** -7


@pytest.mark.parametrize("dim,rank,n,past,window,sink", [(128, 512, 64, 0, 0, False), (64, 128, 33, 31, 0, True), (128, 64, 130, 70, 50, True), (64, 64, 65, 300, 0, False)])
def test_latent_expanded_exactness(dim, rank, n, past, window, sink):
    """fp32 output against float64 on the numbers that the kernel reads."""
    H, ctx, g = 2, past + n, torch.Generator().manual_seed(n)
    q = torch.randn(n, H * (dim + 64), generator=g).to(BF16)
    qr, lat = torch.randn(n, H, 64, generator=g), torch.randn(ctx, rank + 64, generator=g).to(BF16)
    w = (torch.randn(2 * H * dim, rank, generator=g) * rank ** -0.5).to(BF16)
    s = torch.linspace(-2.0, 2.0, H) if sink else None
    out = torch.empty(n, H * dim, dtype=F32, device=DEV)
    ops.latent_attn_expanded(q.to(DEV), qr.to(DEV), lat.to(DEV).unsqueeze(0), [(0, past, 0, n)], w.to(DEV), None, out, H, dim, 64, rank, 0.1, window=window,
                             sink=s.to(DEV) if sink else None)
    kv = (lat[:, :rank].to(F64) @ w.to(F64).T).view(ctx, 2, H, dim)
    sc = (torch.einsum("nhd,shd->hns", q.to(F64).view(n, H, dim + 64)[..., :dim], kv[:, 0]) + torch.einsum("nhd,sd->hns", qr.to(F64), lat[:, rank:].to(F64))) * 0.1
    i, j = torch.arange(past, ctx)[:, None], torch.arange(ctx)[None, :]
    sc = sc.masked_fill(~((j <= i) & ((i - j < window) if window else True)), -math.inf)
    if sink:
        sc = torch.cat([sc, s.to(F64)[:, None, None].expand(H, n, 1)], 2)
    want = torch.einsum("hns,shd->nhd", torch.softmax(sc, -1)[..., :ctx], kv[:, 1]).reshape(n, -1)
    # scores of size 3 within a few 2^-24 of their size, weights and values as exact: a few 1e-7 of the result
    assert float((out.cpu().to(F64) - want).norm() / want.norm()) < 2e-6


@pytest.mark.parametrize("w_dt", [BF16, F32])
@pytest.mark.parametrize("M,N,K", [(65, 24, 40), (130, 65, 520)])
def test_linear_plain_with_numbers_that_are_not_finite(w_dt, M, N, K):
    """An infinity times a finite weight is one, whatever the weight's low bits; largest finite numbers do not become one; a NaN stays in its row or column."""
    g = torch.Generator().manual_seed(K)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g).to(w_dt)
    inf = float("inf")
    w[1, 7] = 1.0                                               # no lower parts: 0 beside the infinity
    a[3, 7], a[4, 0], a[5, K - 1] = inf, -inf, float("nan")
    a[6, 2:4] = torch.tensor([inf, -inf])
    a[7], a[8] = 0.0, 0.0
    a[7, 1], w[:, 1] = 3.4e38, 0.5                              # the nearest bf16 number would be an infinity
    a[8, 9], w[2, 9] = 1.0, inf
    out = torch.empty(M, N, dtype=F32, device=DEV)
    ops.linear_plain(a.to(DEV), w.to(DEV), out)
    want = a.to(F64) @ w.to(F64).T                              # (float64 holds the finite sums; none of them overflows fp32)
    got = out.cpu().to(F64)
    fin = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[~fin & ~torch.isnan(want)], want[~fin & ~torch.isnan(want)])
    bound = torch.nan_to_num(a.to(F64).abs() @ w.to(F64).abs().T, nan=inf) * K * 2.0 ** -24
    assert bool(((got - want).abs()[fin] <= bound[fin]).all())
    assert not bool(fin[3].any()) and bool((~torch.isnan(want[3])).all()) and bool(fin[7, :2].all())


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("dim", [64, 128])
def test_latent_workspace_of_any_size(window, dim):
    """Portions in as many launches as the workspace asks for, a large one by groups of heads: the same bits."""
    H, rank, rot = 5, 72, 64
    portions = [(0, 0, 0, 30), (2, 100, 30, 65), (1, 31, 95, 40), (3, 250, 135, 16)] + [(4 + i, i, 151 + i, 1) for i in range(17)]
    portions.insert(2, (21, 20, 168, 256))                        # of many rows, among those of few
    M, g = 424, torch.Generator().manual_seed(dim)
    q, qr = torch.randn(M, H * (dim + rot), generator=g).to(BF16).to(DEV), torch.randn(M, H, rot, generator=g).to(DEV)
    lat = torch.randn(22, 280, rank + rot, generator=g).to(BF16).to(DEV)
    w = (torch.randn(2 * H * dim, rank, generator=g) * rank ** -0.5).to(BF16).to(DEV)
    gate, sink = torch.rand(M, H, generator=g).to(DEV), torch.linspace(-1.0, 1.0, H, device=DEV)
    want = None
    for room in (1 << 20, 3000, 1100, 400, 1):                  # everything; some portions; one at a time; 2 heads; one head
        out = torch.full((M, H * dim), float("nan"), dtype=F32, device=DEV)
        ops.latent_attn_expanded(q, qr, lat, portions, w, gate, out, H, dim, rot, rank, 0.1, window=window, sink=sink, room=room)
        assert bool(torch.isfinite(out).all())
        want = out if want is None else want
        assert torch.equal(out, want)


@pytest.mark.parametrize("H,n,past", [(4, 16, 100), (4, 33, 300), (16, 20, 200), (16, 64, 100), (4, 255, 0), (16, 256, 300)])
def test_latent_portions_are_as_close_to_64_bits_as_in_the_latent_space(H, n, past):
    """Mean over inputs of the two forms' errors: a measured 0.60 to 0.95."""
    dim, rank, rot, ctx, ratio = 128, 512, 64, past + n, []
    i32 = dict(dtype=torch.int32, device=DEV)
    meta = torch.tensor([(0, past + i) for i in range(n)], **i32)
    for seed in range(4):
        g = torch.Generator().manual_seed(seed)
        q = torch.randn(n, H * (dim + rot), generator=g).to(BF16).to(DEV)
        lat, qr = torch.randn(1, ctx, rank + rot, generator=g).to(BF16).to(DEV), torch.randn(n, H, rot, generator=g).to(DEV)
        w = (torch.randn(2 * H * dim, rank, generator=g) * rank ** -0.5).to(BF16).to(DEV)
        scale, D = (dim + rot) ** -0.5, rank + rot
        new = torch.empty(n, H * dim, dtype=F32, device=DEV)
        ops.latent_attn_expanded(q, qr, lat, [(0, past, 0, n)], w, None, new, H, dim, rot, rank, scale)
        wk, wv = w.view(2, H, dim, rank)
        qa, oa, old = torch.empty(n, H * D, dtype=F32, device=DEV), torch.empty(n, H * rank, dtype=F32, device=DEV), torch.empty(n, H * dim, dtype=F32, device=DEV)
        ops.linear_plain(q, wk.transpose(1, 2).contiguous(), qa, batch=H, a_batch_stride=dim + rot, w_batch_stride=rank * dim, out_batch_stride=D, n=rank, k=dim)
        qa.view(n, H, D)[:, :, rank:] = qr
        ops.latent_attn(qa, lat, meta, None, oa, H, rank, rot, scale, max_ctx=ctx)
        ops.linear_plain(oa, wv, old, batch=H, a_batch_stride=rank, w_batch_stride=dim * rank, out_batch_stride=dim, n=dim, k=rank)
        kv = (lat[0, :, :rank].to(F64) @ w.to(F64).T).view(ctx, 2, H, dim)
        sc = (torch.einsum("nhd,shd->hns", q.to(F64).view(n, H, dim + rot)[..., :dim], kv[:, 0]) + torch.einsum("nhd,sd->hns", qr.to(F64), lat[0, :, rank:].to(F64))) * scale
        sc = sc.masked_fill(torch.arange(ctx, device=DEV)[None, :] > torch.arange(past, ctx, device=DEV)[:, None], -math.inf)
        want = torch.einsum("hns,shd->nhd", torch.softmax(sc, -1), kv[:, 1]).reshape(n, -1)
        ratio.append(float((new.to(F64) - want).norm() / (old.to(F64) - want).norm()))
    assert sum(ratio) / len(ratio) <= 1.0, ratio
