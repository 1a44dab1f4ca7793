"""The matrix-state recurrences in chunks of tokens on the tensor cores (fixed decay; gated with a normaliser) against the token loop in 64 bits, beside the kernel that
goes token by token: portions that end around the chunks and blocks of 16, columns that do not fill a slice, shared keys, states carried in, values that are not finite."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
F32, BF16, F64 = torch.float32, torch.bfloat16, torch.float64
LENS = [[32], [47, 49, 16], [31, 32, 33], [63, 64, 65, 1], [200, 129, 1, 96]]


def _step(lens, H, G, dim, vdim, seed=0, pad=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(lens) + vdim)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    M = sum(lens)
    y = r(M, 2 * G * dim + H * vdim + pad).to(BF16)
    slots = [(5 * i + 2) % len(lens) if len(lens) % 5 else i for i in range(len(lens))]
    segs, row = [], 0
    for s, n in zip(slots, lens):
        segs.append((s, 0, row, n))
        row += n
    return y[:, :G * dim], y[:, G * dim:2 * G * dim], y[:, 2 * G * dim:2 * G * dim + H * vdim], segs, torch.tensor(segs, dtype=torch.int32, device="cuda"), r


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def _close(new, old, want):
    """Both kernels sum the same products in fp32, in another order: errors of the same size, a few roundings of 2^-24 either way."""
    assert _rel(new, want) <= 2 * _rel(old, want) + 2.0 ** -22


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("H,G,vdim", [(2, 2, 128), (4, 2, 72), (3, 1, 8)])
def test_fixed_decay(lens, H, G, vdim):
    dim = 128
    q, k, v, segs, dsegs, r = _step(lens, H, G, dim, vdim)
    S0, d = r(len(lens), H, vdim, dim), torch.tensor([0.999, 0.5, 0.0, 1.0][:H], device="cuda")
    got = {}
    for name, lengths in (("old", (1, 1)), ("new", None if len(lens) == 3 else (min(lens), max(lens)))):
        S, o = S0.clone(), torch.empty(sum(lens), H * vdim, device="cuda")
        ops.linear_scan(q, k, v, S, dsegs, H, G, dim, vdim, o, decay=d, lengths=lengths)
        got[name] = (o, S)
    want, state = torch.empty(sum(lens), H, vdim, dtype=F64, device="cuda"), S0.double()
    for slot, _, row, n in segs:
        S = state[slot]
        for t in range(row, row + n):
            qt, kt = (x[t].double().view(G, dim).repeat_interleave(H // G, 0) for x in (q, k))
            S.mul_(d.double()[:, None, None]).add_(v[t].double().view(H, vdim, 1) * kt[:, None, :])
            want[t] = (S @ qt[:, :, None])[..., 0]
    _close(got["new"][0], got["old"][0], want.view(-1, H * vdim))
    _close(got["new"][1], got["old"][1], state)


@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("dim,vdim", [(256, 512), (128, 40), (256, 32)])
def test_gated_with_normaliser(lens, dim, vdim):
    H = 2
    q, k, v, segs, dsegs, r = _step(lens, H, H, dim, vdim)
    gates = torch.cat([r(sum(lens), H), torch.nn.functional.logsigmoid(r(sum(lens), H) + 2)], 1).contiguous()
    start, scale = (r(len(lens), H, vdim, dim), r(len(lens), H, dim), r(len(lens), H)), dim ** -0.5
    got = {}
    for name, lengths in (("old", (1, 1)), ("new", None if len(lens) == 3 else (min(lens), max(lens)))):
        st, o = [t.clone() for t in start], torch.empty(sum(lens), H * vdim, device="cuda")
        ops.mlstm_scan(q, k, v, gates, *st, dsegs, H, dim, vdim, scale, 1e-6, o, lengths=lengths)
        got[name] = (o, *st)
    want, state = torch.empty(sum(lens), H, vdim, dtype=F64, device="cuda"), [t.double() for t in start]
    for slot, _, row, n in segs:
        S, nn, m = (t[slot] for t in state)
        for t in range(row, row + n):
            i, f = gates[t].double().view(2, H)
            new = torch.maximum(f + m, i)
            a, b = torch.exp(f + m - new), torch.exp(i - new)
            kt, qt = k[t].double().view(H, dim), q[t].double().view(H, dim) * scale
            S.mul_(a[:, None, None]).add_(b[:, None, None] * v[t].double().view(H, vdim, 1) * kt[:, None, :])
            nn.mul_(a[:, None]).add_(b[:, None] * kt)
            m.copy_(new)
            want[t] = (S @ qt[:, :, None])[..., 0] / (torch.maximum((nn * qt).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
    for new, old, w in zip(got["new"], got["old"], (want.view(-1, H * vdim), *state)):
        _close(new, old, w)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 21, 70])
def test_values_that_are_not_finite_stay_in_their_column_and_after_their_token(bad, at):
    H, dim, vdim, n = 1, 128, 64, 100
    q, k, v, segs, dsegs, r = _step([n], H, H, dim, vdim)
    d, clean = torch.tensor([0.9], device="cuda"), torch.empty(n, vdim, device="cuda")
    ops.linear_scan(q, k, v, torch.zeros(1, H, vdim, dim, device="cuda"), dsegs, H, H, dim, vdim, clean, decay=d, lengths=(n, n))
    v[at, 5] = bad
    S, o = torch.zeros(1, H, vdim, dim, device="cuda"), torch.empty_like(clean)
    ops.linear_scan(q, k, v, S, dsegs, H, H, dim, vdim, o, decay=d, lengths=(n, n))
    other = [c for c in range(vdim) if c != 5]
    assert torch.equal(o[:, other], clean[:, other]) and torch.equal(o[:at, 5], clean[:at, 5])
    assert not torch.isfinite(o[at:, 5]).any() and not torch.isfinite(S[0, 0, 5]).any() and bool(torch.isfinite(S[0, 0, other]).all())


def test_rows_that_are_not_whole_vectors_go_token_by_token():
    H, dim, vdim, lens = 2, 128, 16, [80]
    q, k, v, segs, dsegs, r = _step(lens, H, H, dim, vdim, pad=4)
    outs = []
    for lengths in ((1, 1), (80, 80)):
        S, o = torch.zeros(1, H, vdim, dim, device="cuda"), torch.empty(80, H * vdim, device="cuda")
        ops.linear_scan(q, k, v, S, dsegs, H, H, dim, vdim, o, decay=torch.tensor([0.9, 0.8], device="cuda"), lengths=lengths)
        outs.append((o, S))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("gated", [False, True])
def test_a_portion_does_not_depend_on_its_company(gated):
    H, dim, vdim, lens = 2, 128, 64, [70, 1, 40, 31, 1]
    q, k, v, segs, dsegs, r = _step(lens, H, H, dim, vdim)
    M = sum(lens)
    gates, d = torch.cat([r(M, H), -r(M, H).abs()], 1).contiguous(), torch.tensor([0.99, 0.7], device="cuda")
    start = (r(len(lens), H, vdim, dim), r(len(lens), H, dim), r(len(lens), H))

    def run(rows, segs_, lengths):
        st, o = [t.clone() for t in start], torch.empty(q[rows].shape[0], H * vdim, device="cuda")
        dsegs_ = torch.tensor(segs_, dtype=torch.int32, device="cuda")
        if gated:
            ops.mlstm_scan(q[rows], k[rows], v[rows], gates[rows], *st, dsegs_, H, dim, vdim, 0.1, 1e-6, o, lengths=lengths)
        else:
            ops.linear_scan(q[rows], k[rows], v[rows], st[0], dsegs_, H, H, dim, vdim, o, decay=d, lengths=lengths)
        return o, st

    together = run(slice(0, M), segs, (min(lens), max(lens)))
    assert all(torch.equal(x, y) for x, y in zip([together[0]] + together[1], (lambda o, st: [o] + st)(*run(slice(0, M), segs, None))))
    for slot, p0, row, n in segs:
        o, st = run(slice(row, row + n), [(slot, p0, 0, n)], (n, n))
        assert torch.equal(o, together[0][row:row + n]) and all(torch.equal(a[slot], b[slot]) for a, b in zip(st, together[1]))


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("lens", [[20], [70], [31]])
def test_portions_of_unknown_lengths_in_a_larger_buffer(gated, lens):
    """What the segments say counts, not how many rows the buffers have."""
    H, dim, vdim, M, n = 2, 128, 64, 100, len(lens)
    q, k, v, _, _, r = _step([M], H, H, dim, vdim)
    segs = [(i, 0, 0, x) for i, x in enumerate(lens)]
    dsegs = torch.tensor(segs, dtype=torch.int32, device="cuda")
    gates, d = torch.cat([r(M, H), -r(M, H).abs()], 1).contiguous(), torch.tensor([0.99, 0.7], device="cuda")
    start, got = (r(n, H, vdim, dim), r(n, H, dim), r(n, H)), []
    for rows, lengths in ((M, None), (lens[0], (min(lens), max(lens)))):
        st, o = [t.clone() for t in start], torch.full((rows, H * vdim), 7.0, device="cuda")
        if gated:
            ops.mlstm_scan(q[:rows], k[:rows], v[:rows], gates[:rows], *st, dsegs, H, dim, vdim, 0.1, 1e-6, o, lengths=lengths)
        else:
            ops.linear_scan(q[:rows], k[:rows], v[:rows], st[0], dsegs, H, H, dim, vdim, o, decay=d, lengths=lengths)
        got.append((o, *st))
    assert torch.equal(got[0][0][:lens[0]], got[1][0]) and bool((got[0][0][lens[0]:] == 7.0).all())
    assert all(torch.equal(a, b) for a, b in zip(got[0][1:], got[1][1:])) and not torch.equal(got[0][1], start[0])


@pytest.mark.parametrize("gated,n", [(False, 32), (False, 63), (False, 64), (False, 100), (True, 32), (True, 65)])
def test_outputs_are_as_close_to_64_bits_as_token_by_token(gated, n):
    """Mean over inputs: the error in chunks is no larger than that of the token loop (a measured 0.72 to 0.98 times)."""
    H, dim, vdim, ratio = 4, 128, 128, []
    for seed in range(6):
        q, k, v, _, dsegs, r = _step([n], H, H, dim, vdim, seed)
        q, k = (x if gated else torch.nn.functional.silu(x.float()).to(BF16) for x in (q, k))
        q, k, v = torch.cat([q, k, v], 1).split([H * dim, H * dim, H * vdim], 1)
        gates, d = torch.cat([r(n, H), torch.nn.functional.logsigmoid(r(n, H) + 2)], 1).contiguous(), torch.tensor([0.5, 0.9, 0.98, 0.996], device="cuda")
        start, scale, err = (r(1, H, vdim, dim), r(1, H, dim), r(1, H)), dim ** -0.5, []
        S, nn, m = (t[0].double() for t in start)
        want = torch.empty(n, H, vdim, dtype=F64, device="cuda")
        for t in range(n):
            kt, qt, vt = k[t].double().view(H, dim), q[t].double().view(H, dim), v[t].double().view(H, vdim)
            if gated:
                i, f = gates[t].double().view(2, H)
                new = torch.maximum(f + m, i)
                a, b, m = torch.exp(f + m - new), torch.exp(i - new), new
                nn = nn * a[:, None] + b[:, None] * kt
            else:
                a, b = d.double(), torch.ones_like(d, dtype=F64)
            S = S * a[:, None, None] + b[:, None, None] * vt[:, :, None] * kt[:, None, :]
            want[t] = (S @ qt[:, :, None])[..., 0]
            if gated:
                want[t] *= scale / (torch.maximum((nn * qt).sum(-1).abs() * scale, torch.exp(-m)) + 1e-6)[:, None]
        for lengths in ((1, 1), (n, n)):
            st, o = [t.clone() for t in start], torch.empty(n, H * vdim, device="cuda")
            if gated:
                ops.mlstm_scan(q, k, v, gates, *st, dsegs, H, dim, vdim, scale, 1e-6, o, lengths=lengths)
            else:
                ops.linear_scan(q, k, v, st[0], dsegs, H, H, dim, vdim, o, decay=d, lengths=lengths)
            e = ((o.double() - want.view(n, -1)).abs() / want.view(n, -1).abs().clamp_min(1e-30)).flatten().median() if gated else _rel(o, want.view(n, -1))
            err.append(float(e))
        ratio.append(err[1] / err[0])
    assert sum(ratio) / len(ratio) <= 1.01, ratio
