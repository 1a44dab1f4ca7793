"""Projections of few rows or to few columns on mma.sync (csrc/linear_rows_mma.cu): around the lines of its forms, strided and batched, and as gates."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def _rand(*s, seed=0, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(s))
    return (torch.randn(*s, generator=g, device="cuda") * std).to(BF16)


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 128])
@pytest.mark.parametrize("N,K", [(8, 8), (24, 40), (1000, 264), (2376, 2080), (4096, 3072)])
def test_projections(M, N, K):
    """Sums rounded once to bf16; one that lies next to a rounding's middle may go the other way: one step of 2^-8 of sums up to 8."""
    a, w = _rand(M, K), _rand(N, K, std=K ** -0.5)
    out, y = ops.linear(a, w), (a.double() @ w.double().T).to(BF16).double()
    assert float((out.double() - y).abs().max()) <= 0.0325 and float((out.double() != y).double().mean()) < 2e-3
    assert torch.equal(ops.linear(a[:1], w), out[:1])


@pytest.mark.parametrize("N,K", [(2048, 520), (1184, 1032), (2368, 264), (2376, 264), (4096, 136), (64, 8192), (1184, 8192), (2048, 5632), (2560, 3272)])
def test_a_row_does_not_depend_on_how_many_there_are(N, K):
    """Blocks of 8, 16, 24 and 32 rows and of 16 and 32 columns give the same bits, at the edges of the weights that are taken and of the SMs."""
    a, w = _rand(128, K), _rand(N, K, std=K ** -0.5)
    whole = ops.linear(a, w)
    y = (a.double() @ w.double().T).to(BF16).double()
    assert float((whole.double() - y).abs().max()) <= 0.0325 and float((whole.double() != y).double().mean()) < 2e-3
    for M in (1, 7, 8, 9, 15, 16, 17, 24, 25, 33, 40, 48, 49, 64, 65, 72, 73, 96, 97, 127):
        assert torch.equal(ops.linear(a[:M], w), whole[:M]), M


@pytest.mark.parametrize("N,K", [(8, 1024), (16, 2056), (34, 136), (128, 520)])
def test_a_row_of_gates_does_not_depend_on_how_many_there_are(N, K):
    a, w = _rand(5000, K), _rand(N, K, std=K ** -0.5)
    whole = torch.empty(5000, N, device="cuda")
    ops.linear_small(a, w, None, whole)
    assert float((whole.double() - a.double() @ w.double().T).abs().max()) < 3e-6
    for M in (1, 8, 9, 16, 17, 148, 149, 300, 1184, 1185, 2368, 2369, 4736, 4737):
        out = torch.empty(M, N, device="cuda")
        ops.linear_small(a[:M], w, None, out)
        assert torch.equal(out, whole[:M]), M


@pytest.mark.parametrize("M,N,K,batch", [(1, 5, 8, 3), (7, 16, 136, 2), (16, 33, 2088, 1), (40, 130, 512, 4), (64, 4800, 96, 1), (33, 2400, 128, 1)])
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_plain(M, N, K, batch, dtype):
    """A sum of 16 products is cut off at the 24th bit and what the sums of these round off is kept: at most 2^-23 of the sum of the magnitudes."""
    a, w = _rand(M, batch * K + 8), _rand(batch, N, K + 8, std=K ** -0.5)
    out = torch.full((M, batch * N + 3), 9.0, device="cuda").to(dtype)
    ops.linear_plain(a, w[0], out, scale=0.5, batch=batch, a_batch_stride=K, w_batch_stride=w.stride(0), out_batch_stride=N, n=N, k=K)
    for b in range(batch):
        x, y = a[:, b * K:(b + 1) * K].double(), w[b, :, :K].double()
        want, size = 0.5 * x @ y.T, 0.5 * x.abs() @ y.abs().T
        err = (out[:, b * N:(b + 1) * N].double() - want).abs()
        assert bool((err <= 2.0 ** -23 * size + (2.0 ** -8 * want.abs() if dtype == BF16 else 0.0)).all())
    assert bool((out[:, batch * N:] == 9.0).all())


@pytest.mark.parametrize("M", [1, 9, 40, 300])
@pytest.mark.parametrize("N,K", [(2, 64), (16, 2048), (34, 136)])
@pytest.mark.parametrize("mode", [ops.GATE_NONE, ops.GATE_LOG_INPUT_FORGET, ops.GATE_SIGMOID])
def test_gates(M, N, K, mode):
    a, w, bias = _rand(M, K + 8)[:, :K], _rand(N, K, std=K ** -0.5), _rand(N).float()
    out = torch.empty(M, N, device="cuda")
    ops.linear_small(a, w, bias, out, mode, 15.0)
    z = a.double() @ w.double().T + bias.double()
    if mode == ops.GATE_LOG_INPUT_FORGET:
        z = 15.0 * torch.tanh(z / 15.0)
        z[:, N // 2:] = torch.nn.functional.logsigmoid(z[:, N // 2:])
    elif mode == ops.GATE_SIGMOID:
        z = torch.sigmoid(z)
    assert float((out.double() - z).abs().max()) < 3e-6        # sums up to 8 rounded at 2^-24 of their terms, then functions of slope 1 at most
    few = torch.empty(1, N, device="cuda")
    ops.linear_small(a[:1], w, bias, few, mode, 15.0)
    assert torch.equal(few, out[:1])


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_bad_number_stays_in_its_row(bad):
    a, w = _rand(20, 256), _rand(48, 256, std=0.06)
    clean, out = torch.empty(20, 48, device="cuda"), torch.empty(20, 48, device="cuda")
    ops.linear_plain(a, w, clean)
    a[5, 77] = bad
    ops.linear_plain(a, w, out)
    rest = [r for r in range(20) if r != 5]
    assert torch.equal(out[rest], clean[rest]) and torch.equal(out[5].isnan(), (a[5:6].float() @ w.float().T)[0].isnan())


@pytest.mark.parametrize("between", [0, 1, 2])
def test_a_second_operand_that_the_launches_before_wrote(between):
    """Plain projections and gates read both operands after the work before them has ended, unless told that ``w`` is resident."""
    K, x, a = 1024, _rand(64, 2048), _rand(7, 1024, seed=1)
    makers = [_rand(K, 2048, seed=2 + i, std=2048 ** -0.5) for i in range(2)]
    w, other = torch.zeros(64, K, device="cuda", dtype=BF16), torch.zeros(64, K, device="cuda", dtype=BF16)
    want = []
    for maker in makers:
        ops.linear_plain(x, maker, w)
        torch.cuda.synchronize()
        out = [torch.empty(7, 64, device="cuda") for _ in range(2)]
        ops.linear_plain(a, w, out[0]), ops.linear_small(a, w, None, out[1])
        want.append(out)
    assert not torch.equal(want[0][0], want[1][0])
    got = [[torch.empty(7, 64, device="cuda") for _ in range(2)] for _ in range(60)]
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        for f, o in zip((lambda o: ops.linear_plain(a, w, o), lambda o: ops.linear_small(a, w, None, o)), out):
            ops.linear_plain(x, makers[1 - i % 2], w)            # the other number first, so that an old one shows
            ops.linear_plain(x, makers[i % 2], w)
            for _ in range(between):
                ops.linear_plain(x[:8], makers[0], other[:8])
            f(o)
    torch.cuda.synchronize()
    assert all(torch.equal(g, t) for i, out in enumerate(got) for g, t in zip(out, want[i % 2]))


def test_a_resident_second_operand_gives_the_same_bits():
    a, w, bias = _rand(20, 264), _rand(40, 264, std=0.06), _rand(40).float()
    out = [torch.empty(20, 40, device="cuda") for _ in range(4)]
    for i in range(2):
        ops.linear_plain(a, w, out[i], resident=bool(i)), ops.linear_small(a, w, bias, out[2 + i], ops.GATE_SIGMOID, resident=bool(i))
    assert torch.equal(out[0], out[1]) and torch.equal(out[2], out[3])
