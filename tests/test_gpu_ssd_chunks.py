"""The state-space recurrence in chunks of tokens (csrc/ssd_chunk_sm100.cu) against the token loop in 64 bits, beside the kernel that goes token by token: portions that end
around the chunks, heads of one and two slices, groups of more heads than a CTA takes, a workspace that holds some of the chunks, values that are not finite or too large."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import _lib, ops

pytestmark = pytest.mark.gpu
F32, F64 = torch.float32, torch.float64
N = 128


class Step:
    def __init__(self, lens, H, G, vdim, rate=1.0, pad=0, seed=0):
        g = torch.Generator(device="cuda").manual_seed(seed + sum(lens) + H)
        r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
        self.shape, self.lens, M = (H, G, N, vdim), lens, sum(lens)
        self.inner = H * vdim
        self.xbc = torch.nn.functional.silu(r(M, self.inner + 2 * G * N + pad))[:, :self.inner + 2 * G * N]
        dt = torch.nn.functional.softplus(r(M, H) - 2)
        self.gates = torch.cat([dt, torch.exp(-torch.exp(r(H) * 0.7) * rate * dt)], 1).contiguous()
        self.D, self.S0 = r(H), r(len(lens) + 1, H, vdim, N)
        self.slots = [(3 * i + 1) % (len(lens) + 1) if (len(lens) + 1) % 3 else i for i in range(len(lens))]
        self.segs, row = [], 0
        for s, n in zip(self.slots, lens):
            self.segs.append((s, 0, row, n))
            row += n

    def run(self, by_tokens=False, segs=None):
        S, o = self.S0.clone(), torch.full((self.xbc.shape[0], self.inner), 7.0, device="cuda")
        d, (H, G, _, vdim) = torch.tensor(segs or self.segs, dtype=torch.int32, device="cuda"), self.shape
        if by_tokens:
            x, p = self.xbc, ops._p
            ops.check(_lib.load().lia_ssd_scan(p(x[:, self.inner:]), p(x[:, self.inner + G * N:]), p(x), x.stride(0), p(self.gates), p(self.D), p(S), p(d), d.shape[0], x.shape[0],
                                               H, G, N, vdim, p(o), ops._stream()), "lia_ssd_scan")
        else:
            ops.ssd_scan(self.xbc, self.gates, self.D, S, d, H, G, N, vdim, o)
        return o, S

    def exact(self):
        (H, G, _, vdim), M = self.shape, self.xbc.shape[0]
        x, B, C = torch.split(self.xbc.double(), [self.inner, G * N, G * N], -1)
        x, (B, C) = x.view(M, H, vdim), (t.reshape(M, G, N).repeat_interleave(H // G, 1) for t in (B, C))
        dt, a = self.gates.double().split(H, 1)
        u, o, state = dt[:, :, None] * x, torch.empty(M, H, vdim, dtype=F64, device="cuda"), self.S0.double()
        for slot, _, row, n in self.segs:
            S = state[slot]
            for t in range(row, row + n):
                S.mul_(a[t][:, None, None]).add_(u[t][:, :, None] * B[t][:, None, :])
                o[t] = (S @ C[t][:, :, None])[..., 0]
        return (o + self.D.double()[:, None] * x).view(M, -1), state


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def _chunked(step):
    H, G, _, vdim = step.shape
    return _lib.load().lia_ssd_workspace(step.xbc.shape[0], len(step.segs), H, G, N, vdim, 1) > 0


@pytest.mark.parametrize("lens,H,G,vdim,rate,pad", [([256], 2, 1, 64, 1.0, 0), ([257, 40, 300], 4, 4, 64, 1.0, 4), ([511, 1], 18, 2, 64, 1.0, 0), ([512], 4, 2, 128, 0.02, 8),
                                                   ([385, 255, 640], 3, 1, 64, 20.0, 0), ([900], 8, 8, 192, 0.3, 0),
                                                   ([448], 2, 1, 64, 1.0, 0), ([449, 40, 500], 4, 4, 64, 1.0, 4), ([447, 513], 18, 2, 64, 1.0, 0)])
def test_against_the_token_loop(lens, H, G, vdim, rate, pad):
    """Either kernel's numbers are fp32 sums of the same products in another order: this one's error is at most the other's, up to a rounding of 2^-25."""
    step = Step(lens, H, G, vdim, rate, pad)
    assert _chunked(step)
    want = step.exact()
    for new, old, w in zip(step.run(), step.run(by_tokens=True), want):
        assert _rel(new, w) <= _rel(old, w) + 2.0 ** -25


def test_a_workspace_for_some_of_the_chunks_changes_no_bit(monkeypatch):
    step = Step([1000, 300], 4, 2, 64)
    whole = step.run()
    for size in (1, 1 << 21):
        monkeypatch.setattr(ops, "SSD_WORKSPACE", size)
        assert all(torch.equal(a, b) for a, b in zip(whole, step.run()))


@pytest.mark.parametrize("lens,H", [([700, 200, 129, 255, 447, 1], 4), ([500] + [200] * 15, 128)])
def test_short_portions_beside_some_of_the_chunks(lens, H, monkeypatch):
    """Portions that go token by token are done whole, however few chunks of the others are taken at a time."""
    step = Step(lens, H, 2, 64)
    old = step.run(by_tokens=True)
    for size in (ops.SSD_WORKSPACE, 1):
        monkeypatch.setattr(ops, "SSD_WORKSPACE", size)
        o, S = step.run()
        for slot, _, row, n in step.segs:
            if n < 448:
                assert torch.equal(o[row:row + n], old[0][row:row + n]) and torch.equal(S[slot], old[1][slot]), n


def test_an_empty_portion_takes_no_token_from_the_others(monkeypatch):
    step = Step([0, 513, 0], 4, 2, 64)
    whole = Step([513], 4, 2, 64)
    whole.xbc, whole.gates, whole.D, whole.S0, whole.segs = step.xbc, step.gates, step.D, step.S0, step.segs[1:2]
    want = whole.run()
    for size in (ops.SSD_WORKSPACE, 1):
        monkeypatch.setattr(ops, "SSD_WORKSPACE", size)
        assert all(torch.equal(a, b) for a, b in zip(step.run(), want))


@pytest.mark.parametrize("at", [40, 140, 299, 600])
def test_heads_go_token_by_token_for_some_of_the_chunks(at, monkeypatch):
    """A value out of range leaves its head to the token loop for the chunks that are taken together, and these begin with the state that the ones before them left."""
    H, G, vdim = 4, 2, 64
    step = Step([700, 130], H, G, vdim)
    step.xbc[at, 2 * vdim + 5] = 3e30                            # of head 2
    whole, old = step.run(), step.run(by_tokens=True)
    monkeypatch.setattr(ops, "SSD_WORKSPACE", 1)
    o, S = step.run()
    first = at // 128 * 128                                      # the tokens that are taken with it
    assert torch.equal(o.view(-1, H, vdim)[:, [0, 1, 3]], whole[0].view(-1, H, vdim)[:, [0, 1, 3]]) and torch.equal(S[:, [0, 1, 3]], whole[1][:, [0, 1, 3]])
    want = step.exact()
    rows = lambda t: t.view(-1, H, vdim)[:first, 2]  # noqa: E731
    if first:
        assert _rel(rows(o), rows(want[0])) <= _rel(rows(old[0]), rows(want[0])) + 2.0 ** -25
    assert _rel(o.view(-1, H, vdim)[first:, 2], want[0].view(-1, H, vdim)[first:, 2]) <= 2.0 ** -20 and _rel(S[:, 2], want[1][:, 2]) <= 2.0 ** -20


@pytest.mark.parametrize("lens", [[300, 1, 256, 255, 700], [500, 1, 448, 447, 700]])
def test_a_portion_does_not_depend_on_its_company(lens):
    step = Step(lens, 8, 2, 64)
    o, S = step.run()
    for slot, p0, row, n in step.segs:
        alone, state = step.run(segs=[(slot, p0, row, n)])
        assert torch.equal(alone[row:row + n], o[row:row + n]) and torch.equal(state[slot], S[slot])
    short = step.run(by_tokens=True)
    for slot, _, row, n in step.segs:
        if n < 448:
            assert torch.equal(o[row:row + n], short[0][row:row + n]) and torch.equal(S[slot], short[1][slot])


@pytest.mark.parametrize("what,value", [("x", float("nan")), ("x", float("inf")), ("x", 3e38), ("B", float("-inf")), ("C", float("nan")), ("C", 1e30), ("dt", float("inf")), ("g", float("nan")),
                                        ("g", 1.5), ("S", float("inf")), ("S", 1e35)])
@pytest.mark.parametrize("at", [0, 131, 299])
@pytest.mark.parametrize("tokens", [300, 460])
def test_values_out_of_range_go_token_by_token(what, value, at, tokens):
    H, G, vdim = 4, 2, 64
    step = Step([tokens], H, G, vdim)
    clean = step.run()
    if what in ("x", "B", "C"):
        col = {"x": 2 * vdim + 5, "B": step.inner + N + 9, "C": step.inner + G * N + N + 9}[what]
        step.xbc[at, col] = value
        heads = [2] if what == "x" else [2, 3]
    elif what == "S":
        step.S0[step.slots[0], 2, 7, at % N] = value
        heads = [2]
    else:
        step.gates[at, 2 + (H if what == "g" else 0)] = value
        heads = [2]
    got, old = step.run(), step.run(by_tokens=True)
    for h in range(H):
        o, p, q = (t[0].view(-1, H, vdim)[:, h] for t in (got, old, clean))
        S, T, U = (t[1][:, h] for t in (got, old, clean))
        same, like = (p, T) if h in heads else (q, U), (o, S)
        assert all(torch.equal(a.nan_to_num(nan=123.0), b.nan_to_num(nan=123.0)) for a, b in zip(same, like)), h


@pytest.mark.parametrize("what", ["x", "column", "B", "C", "channels", "x and dt", "S"])
@pytest.mark.parametrize("size", [300.0, 3e3, 1e5])
@pytest.mark.parametrize("at", [5, 60, 127, 200])
def test_small_numbers_beside_large_ones(what, size, at):
    """Tokens before and after a large number, and the state, are no further from 64 bits than the token loop's, up to one more rounding of 2^-24; and each number by
    itself is off by no more than 2^-20 of the sum of its terms' magnitudes (at most a dozen roundings and cut sums of 2^-24 lie between the inputs and a term)."""
    H, G, vdim = 2, 1, 64
    step = Step([450], H, G, vdim, seed=int(size) + at)
    x, B, C = step.xbc[:, :step.inner], step.xbc[:, step.inner:step.inner + N], step.xbc[:, step.inner + N:]
    if what in ("x", "x and dt"):
        x[at] *= size
        step.gates[at, :H] /= size if what == "x and dt" else 1.0
    elif what == "column":
        x[at, 7::vdim] *= size
    elif what in ("B", "C"):
        (B if what == "B" else C)[at] *= size
    elif what == "channels":                                      # each of the two large where the other is as ever
        B[:, 9] *= size
        C[:, 7] *= size
    else:
        step.S0[:, :, :, at % N] *= size
    new, old, want = step.run(), step.run(by_tokens=True), step.exact()
    part = slice(7, None, vdim) if what == "column" else slice(None)
    for rows in (slice(0, at), slice(at + 1, None), slice(at // 128 * 128, at)):       # (the row itself is one weight's rounding many times over: by the second bound)
        n, o, w = (t[0][rows, part] for t in (new, old, want))
        assert _rel(n, w) <= _rel(o, w) + 2.0 ** -24, (rows, _rel(n, w), _rel(o, w))
    for t in (step.xbc, step.D, step.S0):
        t.abs_()
    assert all(bool(((n - w).abs() <= 2.0 ** -20 * m).all()) for n, w, m in zip(new, want, step.exact()))
    slot = step.slots[0]
    assert _rel(new[1][slot], want[1][slot]) <= _rel(old[1][slot], want[1][slot]) + 2.0 ** -24


def test_the_skip_term_is_of_x_as_it_is():
    """Without a state the outputs are D x and C B x dt: where that vanishes, D x rounded once."""
    step = Step([450], 2, 1, 64)
    step.gates[:, :2] = 0.0
    step.S0.zero_()
    step.xbc[131, :step.inner] *= 3e4
    o, _ = step.run()
    assert torch.equal(o, (step.D[:, None] * step.xbc[:, :step.inner].view(450, 2, 64)).reshape(450, -1))


@pytest.mark.parametrize("lens,H,known,unknown", [([128] * 16, 8, 1, 4), ([100] * 4, 8, 1, 4), ([1] * 300, 8, 1, 4), ([2048] + [1] * 63, 64, 4, 4), ([500] + [1] * 256, 64, 4, 4),
                                                  ([500, 1, 600] + [7] * 40, 4, 4, 4)])
def test_passes_by_the_portions(lens, H, known, unknown):
    """The form is chosen from the portions and the passes from the long ones among them: single tokens beside a prompt add neither passes nor workspace."""
    step = Step(lens, H, 2, 64)
    S, o, d = step.S0.clone(), torch.empty(step.xbc.shape[0], step.inner, device="cuda"), torch.tensor(step.segs, dtype=torch.int32, device="cuda")
    before = _lib.launch_count
    ops.ssd_scan(step.xbc, step.gates, step.D, S, d, H, 2, N, 64, o, portions=step.segs, lengths=(min(lens), max(lens)))
    mid = _lib.launch_count
    other = step.run()
    assert mid - before == known and _lib.launch_count - mid <= unknown
    assert torch.equal(o, other[0]) and torch.equal(S, other[1])
    want = step.exact() if sum(lens) < 1000 else step.run(by_tokens=True)
    for a, w in zip((o, S), want):
        assert _rel(a, w.double()) <= 2.0 ** -21                 # (the sums of either side are tested above)
    long = [n for n in lens if n >= _lib.load().lia_ssd_chunk_rows()]
    if long:
        few, whole = (_lib.load().lia_ssd_workspace(m, n, H, 2, N, 64, -(-max(long) // 128)) for m, n in ((sum(long), len(long)), (sum(lens), len(lens))))
        assert few <= whole <= 2 * few


def test_rows_that_are_not_whole_vectors_and_other_shapes_go_token_by_token():
    for step in (Step([300], 2, 1, 64, pad=1), Step([300], 2, 1, 40), Step([255, 200], 2, 1, 64), Step([500], 2, 1, 64, pad=1), Step([500], 2, 1, 40), Step([447, 200], 2, 1, 64)):
        assert all(torch.equal(a, b) for a, b in zip(step.run(), step.run(by_tokens=True)))
