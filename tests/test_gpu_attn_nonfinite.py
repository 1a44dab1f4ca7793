"""Numbers that are not finite in the keys and values of the tensor-core attention kernels (csrc/window_attn_mma.cu and csrc/window_attn_sm100.cu, csrc/latent_attn_mma.cu and
csrc/latent_attn_sm100.cu): a row that sees them says so, and no other row does."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32
DEV = "cuda"
TOL = 2.0 ** -19        # rows beside a bad key are summed in another order: a few 2^-24 of numbers of size 1, through exp of scores of a few units


def randn(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(BF16).to(DEV)


@pytest.mark.parametrize("max_ctx", [0, 700])                     # one key range, and several
@pytest.mark.parametrize("at", [0, 333, 639, 699])
def test_single_token_sees_a_nan_key(max_ctx, at):
    H, G, d, ctx = 4, 2, 128, 700
    q, kc, vc = randn(2, H * d, seed=1), randn(2, ctx, G * d, seed=2), randn(2, ctx, G * d, seed=3)
    kc[0, at, 5] = float("nan")                                   # of key head 0: query heads 0 and 1 of the first row
    meta = torch.tensor([(0, ctx - 1), (1, ctx - 1)], dtype=torch.int32, device=DEV)
    out = torch.empty(2, H * d, dtype=F32, device=DEV)
    ops.window_attn(q, kc, vc, meta, None, out, H, G, d, d, 0, 0.1, 0.0, max_ctx=max_ctx)
    bad = torch.zeros(2, H, dtype=torch.bool)
    bad[0, :2] = True
    assert torch.equal(torch.isnan(out).view(2, H, d).all(-1).cpu(), bad) and torch.equal(torch.isnan(out).view(2, H, d).any(-1).cpu(), bad)


def one_portion(kc, vc, q, n, past, H, G, d, **kw):
    i32 = dict(dtype=torch.int32, device=DEV)
    meta = torch.tensor([(0, past + i) for i in range(n)], **i32)
    out = torch.empty(n, H * d, dtype=F32, device=DEV)
    return ops.window_attn(q, kc, vc, meta, None, out, H, G, d, d, kw.get("window", 0), 0.1, kw.get("softcap", 0.0), nseg=1, max_ctx=past + n,
                           segs=torch.tensor([(0, past, 0, n)], **i32), chunk=kw.get("chunk", 0))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("q_dt", [BF16, F32])
@pytest.mark.parametrize("kw", [dict(), dict(window=40), dict(chunk=48, softcap=20.0)])
@pytest.mark.parametrize("at", [3, 70, 129])
def test_prompt_rows_that_see_a_bad_key_and_those_that_do_not(d, q_dt, kw, at):
    H, G, n, past = 2, 1, 130, 20
    q, kc, vc = randn(n, H * d, seed=1).to(q_dt), randn(1, past + n, G * d, seed=2), randn(1, past + n, G * d, seed=3)
    clean = one_portion(kc, vc, q, n, past, H, G, d, **kw).view(n, H, d)
    pos, key = torch.arange(past, past + n), past + at
    sees = ((pos >= key) & (pos - key < kw.get("window", 1 << 30)) & ((pos // kw["chunk"] == key // kw["chunk"]) if "chunk" in kw else True)).to(DEV)
    others = [c for c in range(d) if c != 9]
    for bad in (float("inf"), float("nan")):
        v = vc.clone()
        v[0, key, 9] = bad
        out = one_portion(kc, v, q, n, past, H, G, d, **kw).view(n, H, d)
        assert float((out[~sees] - clean[~sees]).abs().max()) < TOL if bool((~sees).any()) else True
        assert bool((out[sees][..., 9] == bad).all() if bad == bad else torch.isnan(out[sees][..., 9]).all())        # an infinity, weighed, is one
        assert float((out[sees][..., others] - clean[sees][..., others]).abs().max()) < TOL
    k = kc.clone()
    k[0, key, 9] = float("nan")
    out = one_portion(k, vc, q, n, past, H, G, d, **kw).view(n, H, d)
    assert (float((out[~sees] - clean[~sees]).abs().max()) < TOL if bool((~sees).any()) else True) and bool(torch.isnan(out[sees]).all())


@pytest.mark.parametrize("max_ctx", [0, 700])
@pytest.mark.parametrize("H", [2, 16])
def test_single_token_weighs_an_infinite_value(max_ctx, H):
    G, d, ctx = 2, 128, 700
    q, kc, vc = randn(1, H * d, seed=1), randn(1, ctx, G * d, seed=2), randn(1, ctx, G * d, seed=3)
    meta = torch.tensor([(0, ctx - 1)], dtype=torch.int32, device=DEV)
    got = []
    for at in (None, 5, ctx - 1):                                 # (the last key also stands in for those behind it)
        v = vc.clone()
        if at is not None:
            v[0, at, 9] = float("-inf")
        got.append(torch.empty(1, H * d, dtype=F32, device=DEV))
        ops.window_attn(q, kc, v, meta, None, got[-1], H, G, d, d, 0, 0.1, 0.0, max_ctx=max_ctx)
    for out in got[1:]:
        o, c = out.view(H, d), got[0].view(H, d)
        assert bool((o[:H // 2, 9] == float("-inf")).all())
        o, c = o.clone(), c.clone()
        o[:H // 2, 9] = c[:H // 2, 9] = 0.0
        assert float((o - c).abs().max()) < TOL


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("at", [3, 70, 129])
def test_latent_rows_that_see_a_bad_key_and_those_that_do_not(dim, window, at):
    H, n, past, rank, rot = 2, 130, 20, 64, 64
    q, qr, lat = randn(n, H * (dim + rot), seed=1), randn(n, H, rot, seed=2).float(), randn(1, past + n, rank + rot, seed=3)
    w = (randn(2 * H * dim, rank, seed=4).float() * rank ** -0.5).to(BF16)
    sink = torch.linspace(-1.0, 1.0, H, device=DEV)

    def run(lat):
        out = torch.empty(n, H * dim, dtype=F32, device=DEV)
        return ops.latent_attn_expanded(q, qr, lat, [(0, past, 0, n)], w, None, out, H, dim, rot, rank, 0.1, window=window, sink=sink)
    clean, pos, key = run(lat), torch.arange(past, past + n), past + at
    sees = ((pos >= key) & (pos - key < (window or 1 << 30))).to(DEV)
    for c, bad in ((5, float("inf")), (5, float("nan")), (rank + 5, float("nan"))):         # in the latent, in the rotated part of the key
        x = lat.clone()
        x[0, key, c] = bad
        out = run(x)
        assert (float((out[~sees] - clean[~sees]).abs().max()) < TOL if bool((~sees).any()) else True) and bool((~torch.isfinite(out[sees])).all())
