"""The vectorised forms of the row kernels against float64 and against the general forms, at the edges of their ranges (rows of one vector, of a block's
1024 numbers and around it, of more than stay in registers) and where alignment sends a call to the general form."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DEV = "cuda"
TOL = {F32: 2e-6, BF16: 2.0 ** -8}          # a few roundings of 2^-24 of a row's largest number; one rounding to bf16


def close(got, want, dt):
    return float((got.cpu().to(F64) - want).abs().max() / want.abs().max().clamp_min(1e-30)) < TOL[dt]


@pytest.mark.parametrize("W", [4, 30, 1020, 1024, 1028, 2048, 3000, 4096, 4100])
@pytest.mark.parametrize("y_dt,h_dt", [(F32, F32), (F32, BF16), (BF16, F32), (BF16, BF16)])
def test_ln_add_norm(W, y_dt, h_dt):
    g = torch.Generator().manual_seed(W)
    x, y, e = torch.randn(3, W, generator=g) + 3, torch.randn(3, W, generator=g).to(y_dt), torch.randn(3, W, generator=g)
    post, pre = [(torch.randn(W, generator=g), torch.randn(W, generator=g)) for _ in range(2)]

    def ln(v, p):
        return torch.nn.functional.layer_norm(v, (W,), p[0].to(F64), p[1].to(F64), 1e-5)
    dev = lambda p: tuple(t.to(DEV) for t in p)  # noqa: E731
    for with_y, extra, with_h in ((True, True, True), (True, False, False), (False, True, True), (False, False, True)):
        gx, h = x.clone().to(DEV), torch.empty(3, W, dtype=h_dt, device=DEV)
        ops.ln_add_norm(gx, y.to(DEV) if with_y else None, dev(post) if with_y else None, 0.5, dev(pre) if with_h else None, h if with_h else None, 1e-5,
                        extra=e.to(DEV) if extra else None)
        want = x.to(F64) + (0.5 * ln(y.to(F64), post) if with_y else 0.0) + (e.to(F64) if extra else 0.0)
        assert close(gx, want, F32)
        if with_h:
            assert float((h.cpu().to(F64) - ln(want, pre)).abs().max()) < (2e-5 if h_dt == F32 else 0.03)


@pytest.mark.parametrize("H,vdim", [(3, 4), (2, 128), (1, 512), (1, 516), (2, 1024), (1, 4100), (3, 30), (2, 132), (1, 256), (2, 260), (1, 1028), (1, 2048), (1, 2052)])
@pytest.mark.parametrize("dt", [F32, BF16])
def test_headnorm_gate(H, vdim, dt):
    g = torch.Generator().manual_seed(vdim)
    M, n = 9, H * vdim
    o, w = torch.randn(M, n, generator=g), torch.randn(n, generator=g)
    buf = torch.randn(M, n + 8, generator=g).to(dt).to(DEV)
    for off, silu in ((8, False), (8, True), (3, True), (None, False)):                      # a gate between vectors takes the general form
        gate = buf[:, off:off + n] if off is not None else None
        out = torch.empty(M, n, dtype=dt, device=DEV)
        ops.headnorm_gate(o.to(DEV), w.to(DEV), gate, out, H, vdim, 1e-5, gate_silu=silu)
        v = o.to(F64).view(M, H, vdim)
        want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5)).view(M, n) * w.to(F64)
        if gate is not None:
            z = gate.cpu().to(F64)
            want = want * torch.sigmoid(z) * (z if silu else 1.0)
        assert close(out, want, dt)


@pytest.mark.parametrize("F,up", [(4, 8), (4, -1), (30, 32), (264, 264), (264, 266)])
@pytest.mark.parametrize("dt", [F32, BF16])
def test_gated_act(F, up, dt):
    g = torch.Generator().manual_seed(F)
    a = torch.randn(7, 2 * F + 8, generator=g).to(dt)
    perm, wt = torch.tensor([3, -1, 0, 5, 1, -1, 2], dtype=torch.int32), torch.rand(6, generator=g)
    for weighed in (False, True):
        out = torch.empty(7, F, dtype=dt, device=DEV)
        ops.gated_act(a.to(DEV), F, out, ops.ACT_SILU, up_off=up, perm=perm.to(DEV) if weighed else None, wt=wt.to(DEV))
        s = torch.where(perm >= 0, wt[perm.clamp_min(0).long()], torch.zeros(7))[:, None].to(F64) if weighed else 1.0
        z = a.to(F64)[:, :F] * s
        want = z * torch.sigmoid(z) * (a.to(F64)[:, up:up + F] * s if up >= 0 else 1.0)
        assert close(out, want, dt)


@pytest.mark.parametrize("M", [1, 5, 1183, 1184, 1187])
@pytest.mark.parametrize("N,K", [(1, 8), (8, 1000), (17, 129)])
@pytest.mark.parametrize("a_dt,w_dt", [(BF16, BF16), (F32, F32), (F32, BF16)])
def test_linear_small(M, N, K, a_dt, w_dt):
    g = torch.Generator().manual_seed(M + N)
    a, w, b = torch.randn(M, K, generator=g).to(a_dt), torch.randn(N, K, generator=g).to(w_dt), torch.randn(N, generator=g)
    out = torch.empty(M, N, device=DEV)
    ops.linear_small(a.to(DEV), w.to(DEV), b.to(DEV), out, ops.GATE_SIGMOID)
    assert float((out.cpu().to(F64) - torch.sigmoid(a.to(F64) @ w.to(F64).T + b.to(F64))).abs().max()) < 2e-5


@pytest.mark.parametrize("F,groups", [(64, 1), (128, 1), (132, 1), (512, 1), (1536, 3), (2000, 5)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_a_row_of_a_gated_norm_does_not_depend_on_how_many_there_are(F, groups, dt):
    g = torch.Generator(device=DEV).manual_seed(F)
    M = 2200
    o, z, w = torch.randn(M, F, generator=g, device=DEV), torch.randn(M, F, generator=g, device=DEV).to(dt), torch.randn(F, generator=g, device=DEV)
    whole = torch.empty(M, F, dtype=dt, device=DEV)
    ops.silu_gate_norm(o, z, w, whole, groups, 1e-6)
    for m in (1, 7, 2047 // groups, -(-2048 // groups)):
        out = torch.empty(m, F, dtype=dt, device=DEV)
        ops.silu_gate_norm(o[:m], z[:m], w, out, groups, 1e-6)
        assert torch.equal(out, whole[:m]), m
    u = (o.double() * z.double() * torch.sigmoid(z.double())).view(M, groups, -1)
    want = (u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-6)).view(M, F) * w.double()
    assert float((whole.double() - want).abs().max() / want.abs().max()) < (2.0 ** -20 if dt == torch.float32 else 2.0 ** -8)


@pytest.mark.parametrize("lens", [[65], [72, 1, 7], [300], [2] * 40, [1] * 70 + [9]])
@pytest.mark.parametrize("taps,act", [(4, ops.ACT_SILU), (3, ops.ACT_NONE), (1, ops.ACT_NONE)])
@pytest.mark.parametrize("dt", [F32, BF16])
def test_convolution_by_pairs_of_channels(lens, taps, act, dt):
    """Two channels a thread and one, chosen by the output's row stride, give the same bits, wherever portions begin."""
    from lia_b200.seq_layers import StepBatch
    C, M, n = 512, sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(M + taps)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    y, w, bias, in_bias, state = r(M, C + 8).to(dt), r(C, taps), r(C), r(C), r(n, max(taps - 1, 1), C)
    segs, meta, row = [], [], 0
    for i, k in enumerate(lens):
        segs.append((i, 2 * (i % 3), row, k))
        meta += [(i, 2 * (i % 3) + j) for j in range(k)]
        row += k
    batch = StepBatch(M, torch.tensor(segs, dtype=torch.int32, device=DEV), torch.tensor(meta, dtype=torch.int32, device=DEV), portions=segs)
    got = []
    for ld in (C + 2, C + 1):
        out, st = torch.zeros(M, ld, device=DEV)[:, :C], state.clone()
        ops.conv_act(y, 4, w, out, batch, state=st if taps > 1 else None, in_bias=in_bias, bias=bias, act=act)
        got.append((out.clone(), st))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("G,H,dim,taps", [(1, 1, 32, 4), (2, 4, 64, 4), (2, 4, 64, 7), (1, 2, 128, 1)])
@pytest.mark.parametrize("dt", [F32, BF16])
def test_a_row_of_the_delta_rules_convolution_does_not_depend_on_how_many_there_are(G, H, dim, taps, dt):
    g = torch.Generator(device=DEV).manual_seed(taps + dim)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    M, C = 70, (2 * G + H) * dim
    y, w, state, gates = r(M, C + 8).to(dt), r(C, taps), r(1, max(taps - 1, 1), C), r(M, 2 * H)
    a_log, dt_bias = r(H), r(H)
    meta = torch.tensor([(0, 3 + i) for i in range(M)], dtype=torch.int32, device=DEV)

    def run(m):
        ga, qk, v = gates[:m].clone(), torch.empty(m, 2 * G * dim, device=DEV), torch.empty(m, H * dim, device=DEV)
        ops.conv_prep(y[:m], (0, G * dim, 2 * G * dim), w, state, meta[:m], ga, a_log, dt_bias, qk, v, G, H, dim, dim, taps, 0.25)
        return qk, v, ga

    whole = run(M)
    for m in (1, 33, 64, 65):
        assert all(torch.equal(a, b[:m]) for a, b in zip(run(m), whole)), m
