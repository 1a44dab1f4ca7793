"""Prompt projections with 64-, 128- and 256-wide tiles: the same bits whatever the width (every tile runs the whole of K), in every epilogue, at ragged
sizes and where the widths' tiles end differently; and the width the rule takes is one of them."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("M", [129, 255, 257, 640])
@pytest.mark.parametrize("N,K", [(8, 64), (72, 200), (192, 1000), (264, 72), (2048, 136), (2568, 256)])
@pytest.mark.parametrize("epilogue", [ops.EPI_BIAS, ops.EPI_BIAS_RELU, ops.EPI_BIAS_RESIDUAL])
def test_same_bits(M, N, K, epilogue, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, w = torch.randn(M, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    bias, res = torch.randn(N, generator=g, device="cuda").to(BF16), torch.randn(M, N, generator=g, device="cuda").to(BF16)
    r = res if epilogue == ops.EPI_BIAS_RESIDUAL else None
    outs = []
    for width in ("64", "128", "256", None):
        monkeypatch.setenv("LIA_GEMM_BN", width) if width else monkeypatch.delenv("LIA_GEMM_BN")
        outs.append(ops.gemm(a, w, bias, epilogue=epilogue, residual=r))
    assert all(torch.equal(outs[0], o) for o in outs)
    # the reference's rounding points: bf16 after the sums, the bias and the last step; sums of K terms of size K^-1/2 differ by less than one such rounding
    y = ((a.float() @ w.float().T).to(BF16).float() + bias.float()).to(BF16).float()
    y = torch.relu(y) if epilogue == ops.EPI_BIAS_RELU else (y + res.float()).to(BF16).float() if r is not None else y
    assert float((outs[0].float() - y).abs().max()) < 0.07


def test_qkv_scatter(monkeypatch):
    B, S, H, d = 3, 77, 4, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    a, w = torch.randn(B * S, 256, generator=g, device="cuda").to(BF16), (torch.randn(3 * H * d, 256, generator=g, device="cuda") / 16).to(BF16)
    got = []
    for width in ("64", "128", "256"):
        monkeypatch.setenv("LIA_GEMM_BN", width)
        q, k, v = torch.zeros(B * S, H * d, dtype=BF16, device="cuda"), *(torch.zeros(S + 2, B, H, d, dtype=BF16, device="cuda") for _ in range(2))
        ops.gemm(a, w, None, epilogue=ops.EPI_QKV, qkv=ops.qkv_args(q, k, v, S, 1, 0, 0.125))
        got.append((q, k, v))
    for other in got[1:]:
        assert all(torch.equal(x, y) for x, y in zip(got[0], other))
    assert bool((got[0][1][0] == 0).all()) and bool((got[0][1][1] != 0).any())


@pytest.mark.parametrize("N,K", [(8, 64), (136, 1024), (1024, 1032), (512, 1920), (2176, 1920), (2176, 1912), (2560, 2560), (7552, 640), (7560, 1280), (1024, 12288), (1024, 12296)])
def test_few_rows_at_the_lines_between_tiles_parts_and_spans(N, K):
    """Whole tiles, equal parts of tiles and spans: a row's result is right and does not depend on the rows beside it."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w = torch.randn(100, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    y = ops.gemm(a, w, None)
    assert float((y.float() - a.float() @ w.float().T).abs().max()) < 0.035            # sums of size up to 5, rounded once to bf16
    for M in (1, 16, 17, 33, 65):
        assert torch.equal(ops.gemm(a[:M].contiguous(), w, None), y[:M])
