"""Tensor-core window attention (csrc/window_attn_mma.cu) against a float64 softmax, at the edges of its tiles: portions of 1, 63, 64, 65 rows
beside each other, key counts around a stage, 1 to 16 query heads per key head, every option of the scores and the output, and
single tokens with one and several key ranges; and which inputs it leaves to the general kernel."""
import math

import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import _lib, ops

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DEV = "cuda"


def reference(q, kc, vc, segs, H, G, dim, vdim, scale, window=0, chunk=0, softcap=0.0, temp=None, slopes=None, sink=None, v_div=1):
    """float64 [rows, H, vdim] on the CPU; caches [slots, capacity, ...] and q as the kernel reads them."""
    q, kc, vc = q.cpu().to(F64), kc.cpu().to(F64), vc.cpu().to(F64)
    out = torch.zeros(q.shape[0], H, vdim, dtype=F64)
    for slot, p0, r0, n in segs:
        k = kc[slot, :p0 + n].view(p0 + n, G, dim)
        v = vc[slot, :p0 + n].view(p0 + n, G // v_div, vdim)
        pos, j = torch.arange(p0, p0 + n)[:, None], torch.arange(p0 + n)[None, :]
        seen = (j <= pos) & ((pos - j < window) if window else True) & ((j >= pos - pos % chunk) if chunk else True)
        for h in range(H):
            g = h // (H // G)
            s = (q[r0:r0 + n].view(n, H, dim)[:, h] @ k[:, g].T) * scale * (float(temp[h]) if temp is not None else 1.0)
            s = softcap * torch.tanh(s / softcap) if softcap else s
            s = (s - float(slopes[h]) * (pos - j) if slopes is not None else s).masked_fill(~seen, -math.inf)
            s = torch.cat([s, torch.full((n, 1), float(sink[h]), dtype=F64)], 1) if sink is not None else s
            out[r0:r0 + n, h] = torch.softmax(s, -1)[:, :p0 + n] @ v[:, g // v_div]
    return out


def inputs(portions, H, G, dim, vdim, q_f32, seed, v_div=1, cap=None):
    g = torch.Generator().manual_seed(seed)
    slots = max(p[0] for p in portions) + 1
    cap = cap or max(p[1] + p[2] for p in portions) + 3
    segs, row = [], 0
    for slot, p0, n in portions:
        segs.append((slot, p0, row, n))
        row += n
    meta = [(s, p + i) for s, p, _, n in segs for i in range(n)]
    q = torch.randn(row, H * dim, generator=g)
    kc = torch.randn(slots, cap, G * dim, generator=g).to(BF16).to(DEV)
    vc = torch.randn(slots, cap, G // v_div * vdim, generator=g).to(BF16).to(DEV)
    for slot in range(slots):                                   # what lies behind a sequence's last position is never read
        end = max([p0 + n for s, p0, n in portions if s == slot], default=0)
        kc[slot, end:], vc[slot, end:] = float("nan"), float("nan")
    return q.to(F32 if q_f32 else BF16).to(DEV), kc, vc, segs, torch.tensor(segs, dtype=torch.int32, device=DEV), torch.tensor(meta, dtype=torch.int32, device=DEV)


OPTIONS = [dict(), dict(window=70, softcap=20.0, temp=True), dict(sink=True, slopes=True), dict(chunk=48)]
# scores of size 5 carry about 5 * 2^-23 * sqrt(dim) of relative error through exp: below 1e-5 of the largest value with room to spare
TOL = 1e-5


@pytest.mark.parametrize("q_f32", [False, True])
@pytest.mark.parametrize("H,G,dim,vdim,v_div", [(4, 2, 128, 128, 1), (3, 3, 64, 64, 1), (4, 4, 128, 256, 2), (2, 1, 64, 128, 1), (16, 1, 128, 64, 1), (2, 2, 64, 256, 1)])
@pytest.mark.parametrize("opt", range(len(OPTIONS)))
def test_portions(q_f32, H, G, dim, vdim, v_div, opt):
    o = dict(OPTIONS[opt])
    portions = [(2, 0, 64), (0, 5, 1), (3, 31, 65), (1, 64, 63), (4, 127, 2), (5, 0, 130)]
    q, kc, vc, segs, d_segs, meta = inputs(portions, H, G, dim, vdim, q_f32, 7 + opt, v_div)
    g = torch.Generator().manual_seed(1)
    for n in ("temp", "sink", "slopes"):
        if o.get(n):
            o[n] = 0.5 + torch.rand(H, generator=g)
    want = reference(q, kc, vc, segs, H, G, dim, vdim, 0.1, v_div=v_div, **o)
    dev = {n: o[n].to(DEV) if o.get(n) is not None else None for n in ("temp", "sink", "slopes")}
    out = torch.empty(q.shape[0], H * vdim, dtype=F32, device=DEV)
    ops.window_attn(q, kc, vc, meta, dev["temp"], out, H, G, dim, vdim, o.get("window", 0), 0.1, o.get("softcap", 0.0), nseg=len(segs), segs=d_segs,
                    max_ctx=140, slopes=dev["slopes"], sink=dev["sink"], chunk=o.get("chunk", 0), v_div=v_div)
    assert float((out.cpu().to(F64) - want.reshape(out.shape)).abs().max() / want.abs().max()) < TOL
    # the same rows one by one (single tokens), with as many key ranges as the rule takes, in bf16 behind a gate
    gate = torch.randn(q.shape[0], H * vdim + 8, generator=g).to(BF16).to(DEV)[:, 8:]
    one = torch.empty(q.shape[0], H * vdim, dtype=BF16, device=DEV)
    ops.window_attn(q, kc, vc, meta, dev["temp"], one, H, G, dim, vdim, o.get("window", 0), 0.1, o.get("softcap", 0.0), slopes=dev["slopes"], sink=dev["sink"],
                    chunk=o.get("chunk", 0), v_div=v_div, max_ctx=140, gate=gate)
    want = want.reshape(out.shape) * torch.sigmoid(gate.cpu().to(F64))
    assert float((one.cpu().to(F64) - want).abs().max() / want.abs().max()) < 2.0 ** -8


@pytest.mark.parametrize("rep", [1, 2, 3, 8, 12, 16])
@pytest.mark.parametrize("ctx", [1, 15, 16, 17, 64, 700, 4000])
def test_single_tokens(rep, ctx):
    G, dim, vdim = 2, 128, 128
    H = rep * G
    portions = [(0, ctx - 1, 1), (2, max(ctx - 9, 0), 1)]
    q, kc, vc, segs, _, meta = inputs(portions, H, G, dim, vdim, rep % 2 == 1, ctx)
    sink = torch.linspace(-1, 1, H)
    want = reference(q, kc, vc, segs, H, G, dim, vdim, 0.1, sink=sink)
    for max_ctx in (0, ctx):                                    # one range, and the rule's
        out = torch.empty(2, H * vdim, dtype=F32, device=DEV)
        ops.window_attn(q, kc, vc, meta, None, out, H, G, dim, vdim, 0, 0.1, 0.0, max_ctx=max_ctx, sink=sink.to(DEV))
        assert float((out.cpu().to(F64) - want.reshape(out.shape)).abs().max() / want.abs().max()) < TOL


def test_what_the_general_kernel_keeps():
    lib = _lib.load()
    q, kc, vc, segs, d_segs, meta = inputs([(0, 0, 70)], 2, 2, 128, 128, False, 3)
    out = torch.empty(70, 256, dtype=BF16, device=DEV)

    def takes(ldq=256, q=q, dim=128, vdim=128, kss=None):
        return lib.lia_window_attn_mma_takes(q.data_ptr(), ldq, 0, kc.data_ptr(), kss or kc.stride(0), vc.data_ptr(), vc.stride(0), out.data_ptr(), 2, 2, 1, dim, vdim)
    assert takes() == 1
    assert takes(ldq=260) == 0 and takes(q=q.view(-1)[4:]) == 0 and takes(dim=96) == 0 and takes(vdim=80) == 0 and takes(kss=kc.stride(0) + 4) == 0
    want = reference(q, kc, vc, segs, 2, 2, 128, 128, 0.1)
    wide = torch.empty(70, 260, dtype=BF16, device=DEV)         # rows of 260 numbers: the queries' rows start between 16-byte boundaries
    wide[:, 4:] = q
    ops.window_attn(wide[:, 4:], kc, vc, meta, None, out, 2, 2, 128, 128, 0, 0.1, 0.0, nseg=1, max_ctx=70)
    assert float((out.cpu().to(F64) - want.reshape(out.shape)).abs().max() / want.abs().max()) < 2.0 ** -8


@pytest.mark.parametrize("q_f32", [False, True])
@pytest.mark.parametrize("at", [[(0, 5), (1, 69)], [(0, 69), (0, 68), (0, 0)], None])
@pytest.mark.parametrize("d", [64, 128])                            # heads of 128: csrc/window_attn_sm100.cu
def test_one_portion_announced_whose_rows_are_others(q_f32, at, d):
    """Without segments `nseg` is advice: a row's slot and position come from meta alone, up to the caches' last rows."""
    H, G, cap, M = 4, 2, 70, 130
    g = torch.Generator().manual_seed(4)
    q = torch.randn(M, H * d, generator=g).to(F32 if q_f32 else BF16).to(DEV)
    kc, vc = (torch.randn(2, cap, G * d, generator=g).to(BF16).to(DEV) for _ in range(2))
    rows = [(at * M)[i] if at else (i % 2, (7 * i) % cap) for i in range(M)]
    out = torch.empty(M, H * d, dtype=F32, device=DEV)
    ops.window_attn(q, kc, vc, torch.tensor(rows, dtype=torch.int32, device=DEV), None, out, H, G, d, d, 33, 0.1, 0.0, nseg=1, max_ctx=cap)
    want = reference(q, kc, vc, [(s, p, r, 1) for r, (s, p) in enumerate(rows)], H, G, d, d, 0.1, window=33)
    assert float((out.cpu().to(F64) - want.reshape(out.shape)).abs().max() / want.abs().max()) < TOL
