"""Prompts through window attention on tcgen05 (csrc/window_attn_sm100.cu) against a float64 softmax, where its tiles can go wrong: portions of 1 to 300 rows behind 0 to 700
positions (blocks of 64 keys to the second turn of the ring, tiles of 128 rows), windows and chunks that hide whole blocks from some warps, scores beyond and below the soft cap's short form,
gates whose rows are whole vectors and not, bf16 and fp32 outputs."""
import math

import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops
from test_gpu_attn_mma import BF16, DEV, F32, F64, TOL, inputs, reference

pytestmark = pytest.mark.gpu
PORTIONS = [(0, 0, 300), (1, 700, 129), (2, 255, 1), (3, 63, 128), (4, 0, 2), (5, 129, 191)]


@pytest.mark.parametrize("q_f32", [False, True])
@pytest.mark.parametrize("H,G,v_div", [(4, 2, 1), (3, 3, 3), (8, 1, 1)])
@pytest.mark.parametrize("opt", [dict(), dict(window=33), dict(window=200, softcap=30.0, temp=True), dict(softcap=1.5), dict(chunk=100, sink=True, slopes=True)], ids=str)
def test_portions(q_f32, H, G, v_div, opt):
    opt, d = dict(opt), 128
    q, kc, vc, segs, d_segs, meta = inputs(PORTIONS, H, G, d, d, q_f32, 3, v_div)
    g = torch.Generator().manual_seed(1)
    for n in ("temp", "sink", "slopes"):
        if opt.get(n):
            opt[n] = 0.5 + torch.rand(H, generator=g)
    want = reference(q, kc, vc, segs, H, G, d, d, 0.1, v_div=v_div, **opt).reshape(q.shape[0], -1)
    dev = {n: opt[n].to(DEV) if opt.get(n) is not None else None for n in ("temp", "sink", "slopes")}

    def run(dtype, gate=None):
        out = torch.full((q.shape[0], H * d), 7.0, dtype=dtype, device=DEV)
        ops.window_attn(q, kc, vc, meta, dev["temp"], out, H, G, d, d, opt.get("window", 0), 0.1, opt.get("softcap", 0.0), nseg=len(segs), segs=d_segs, max_ctx=830,
                        slopes=dev["slopes"], sink=dev["sink"], chunk=opt.get("chunk", 0), v_div=v_div, gate=gate)
        return out
    out = run(F32)
    assert float((out.cpu().to(F64) - want).abs().max() / want.abs().max()) < TOL
    for i, (slot, p0, r0, n) in enumerate(segs):                    # a portion does not depend on its company
        alone = torch.empty(n, H * d, dtype=F32, device=DEV)
        ops.window_attn(q[r0:r0 + n].contiguous(), kc, vc, meta[r0:r0 + n].contiguous(), dev["temp"], alone, H, G, d, d, opt.get("window", 0), 0.1, opt.get("softcap", 0.0), nseg=1,
                        segs=torch.tensor([(slot, p0, 0, n)], dtype=torch.int32, device=DEV), max_ctx=p0 + n, slopes=dev["slopes"], sink=dev["sink"], chunk=opt.get("chunk", 0), v_div=v_div)
        assert n == 1 or torch.equal(alone, out[r0:r0 + n])
    for first, pad in ((8, 0), (8, 4), (8, 1), (1, 7)):             # rows of whole 16 and 8 bytes, rows and a first one at 2; one rounding to bf16 of numbers up to the largest
        wide = torch.randn(q.shape[0], first + H * d + pad, generator=g).to(BF16).to(DEV)
        gate = wide[:, first:first + H * d]
        assert (gate.data_ptr() | 2 * gate.stride(0)) % 8 == (0 if first == 8 and pad != 1 else 2)
        got = want * torch.sigmoid(gate.cpu().to(F64))
        assert float((run(BF16, gate).cpu().to(F64) - got).abs().max() / got.abs().max()) < 2.0 ** -8


@pytest.mark.parametrize("spec,form", [([(0, 40)] * 40, 3), ([(0, 16), (0, 17), (40, 5), (0, 64)], 3), ([(0, 200)] + [(30, 1)] * 40, 4), ([(300, 90)] + [(100, 16)] * 70 + [(0, 97)], 5),
                                       ([(0, 96), (33, 64)] * 100, 6), ([(0, 130)] * 20, 2), ([(0, 60), (10, 60)], 2)], ids=str)
@pytest.mark.parametrize("q_f32,opt", [(False, dict()), (True, dict(window=24, sink=True))], ids=str)
def test_short_portions(spec, form, q_f32, opt):
    """Steps whose portions go to mma.sync, to tcgen05 or to both (on 148 SMs): every row is written once, known or not on the host, and a long portion's bits are those it has alone."""
    H, G, d = 8, 4, 128
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the forms are those of 148 SMs")
    portions = [(i, p, n) for i, (p, n) in enumerate(spec)]
    q, kc, vc, segs, d_segs, meta = inputs(portions, H, G, d, d, q_f32, 5, 1)
    sink = torch.full((H,), 0.5) if opt.get("sink") else None
    want = reference(q, kc, vc, segs, H, G, d, d, 0.1, window=opt.get("window", 0), sink=sink).reshape(q.shape[0], -1)
    sink = sink.to(DEV) if sink is not None else None

    def run(segs, d_segs, rows, form):
        out = torch.full((len(rows), H * d), 7.0, dtype=F32, device=DEV)
        return ops.window_attn(q[rows].contiguous(), kc, vc, meta[rows].contiguous(), None, out, H, G, d, d, opt.get("window", 0), 0.1, 0.0, nseg=len(segs), segs=d_segs, max_ctx=400, sink=sink,
                               form=form)
    known = ops.window_prompt_form(segs, len(segs), q.shape[0], H, opt.get("window", 0))
    assert known == form or (opt and form != 2)                     # a window leaves fewer keys to see: more portions are short ones
    rows = list(range(q.shape[0]))
    for f in (known, None, 2, 3):
        assert float((run(segs, d_segs, rows, f).cpu().to(F64) - want).abs().max() / want.abs().max()) < TOL
    out = run(segs, d_segs, rows, known)
    for slot, p0, r0, n in segs:
        if n > 96 and known != 3:
            alone = torch.tensor([(slot, p0, 0, n)], dtype=torch.int32, device=DEV)
            assert torch.equal(run([(slot, p0, 0, n)], alone, list(range(r0, r0 + n)), None), out[r0:r0 + n])


STEPS = {"40 of 40 rows": ([(0, 40)] * 40, 3), "few tiles": ([(0, 16), (0, 17), (40, 5), (0, 64)], 3), "a prompt and 40 tokens": ([(0, 200)] + [(30, 1)] * 40, 4),
         "two prompts and 70 of 16 rows": ([(300, 190)] + [(100, 16)] * 70 + [(0, 129)], 4), "200 of 64 and 96 rows": ([(0, 96), (33, 64)] * 100, 3), "20 of 130 rows": ([(0, 130)] * 20, 2)}


@pytest.mark.parametrize("step", STEPS)
@pytest.mark.parametrize("q_f32,opt", [(False, dict()), (True, dict(window=24, sink=True))], ids=str)
def test_short_portions(step, q_f32, opt):
    """Steps whose portions go to mma.sync, to tcgen05 or to both (on 148 SMs): every row is written, known or not on the host, and a long portion's bits are those it has alone."""
    H, G, d = 8, 4, 128
    spec, kernels = STEPS[step]
    q, kc, vc, segs, d_segs, meta = inputs([(i, p, n) for i, (p, n) in enumerate(spec)], H, G, d, d, q_f32, 5, 1)
    sink = torch.full((H,), 0.5) if opt.get("sink") else None
    want = reference(q, kc, vc, segs, H, G, d, d, 0.1, window=opt.get("window", 0), sink=sink).reshape(q.shape[0], -1)
    sink = sink.to(DEV) if sink is not None else None

    def run(segs, rows, form):
        out = torch.full((rows.stop - rows.start, H * d), float("nan"), dtype=F32, device=DEV)
        return ops.window_attn(q[rows].contiguous(), kc, vc, meta[rows].contiguous(), None, out, H, G, d, d, opt.get("window", 0), 0.1, 0.0, nseg=len(segs), max_ctx=600, sink=sink, form=form,
                               segs=torch.tensor(segs, dtype=torch.int32, device=DEV))
    form = ops.window_prompt_form(segs, len(segs), q.shape[0], H, opt.get("window", 0))
    assert form & 7 == kernels or torch.cuda.get_device_properties(0).multi_processor_count != 148
    whole = slice(0, q.shape[0])
    for f in (form, 4, None, 2, 3):
        assert float((run(segs, whole, f).cpu().to(F64) - want).abs().max() / want.abs().max()) < TOL
    for slot, p0, r0, n in segs:
        if n > 128:
            assert torch.equal(run([(slot, p0, 0, n)], slice(r0, r0 + n), None), run(segs, whole, form)[r0:r0 + n])


@pytest.mark.parametrize("q_f32", [False, True])
def test_weights_below_the_smallest_normal_number(q_f32):
    """A weight of exp(-88.5) = 2^-127.7, as three parts of which the first has five bits left, times a value of 2^127."""
    H, d = 2, 128
    q, kc, vc = torch.zeros(2, H * d, device=DEV), torch.zeros(1, 2, H * d, device=DEV), torch.zeros(1, 2, H * d, device=DEV)
    q[:, ::d], kc[0, 1, ::d], vc[0, 1, 5] = 1.0, -88.5, 2.0 ** 127
    out = torch.empty(2, H * d, device=DEV)
    ops.window_attn(q if q_f32 else q.to(BF16), kc.to(BF16), vc.to(BF16), torch.tensor([(0, 0), (0, 1)], dtype=torch.int32, device=DEV), None, out, H, H, d, d, 0, 1.0, 0.0, nseg=1, form=2)
    want = math.exp(-88.5) * 2.0 ** 127
    assert abs(float(out[1, 5]) / want - 1) < 2.0 ** -5 and float(out.abs().sum() - out[1, 5].abs()) == 0.0
