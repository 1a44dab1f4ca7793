"""Projections whose tiles' K is shared by the CTAs of a cluster: every number of parts and both widths against the projection by whole tiles, at ragged
sizes, in every epilogue; and sizes at which the rule takes parts by itself."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
# fp32 sums of the same products in another order, of size 1 with magnitudes up to 6: apart by far less than one rounding to bf16 (2^-6 at 4 to 8), which may fall the
# other way once per rounding point (sum, bias, residual)
TOL = 3 * 2.0 ** -6


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g, device="cuda").to(BF16), (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF16)
    return a, w, torch.randn(N, generator=g, device="cuda").to(BF16), torch.randn(M, N, generator=g, device="cuda").to(BF16)


@pytest.mark.parametrize("parts,width", [(2, 128), (3, 128), (4, 128), (6, 128), (8, 128), (2, 256), (3, 256), (4, 256)])
@pytest.mark.parametrize("M,N,K", [(129, 8, 512), (255, 264, 1096), (257, 136, 2048), (300, 768, 4104)])
def test_parts(parts, width, M, N, K, monkeypatch):
    a, w, bias, res = operands(M, N, K)
    for epilogue in (ops.EPI_BIAS, ops.EPI_BIAS_RELU, ops.EPI_BIAS_RESIDUAL):
        r = res if epilogue == ops.EPI_BIAS_RESIDUAL else None
        monkeypatch.setenv("LIA_GEMM_SPLIT", "1")
        whole = ops.gemm(a, w, bias, epilogue=epilogue, residual=r)
        monkeypatch.setenv("LIA_GEMM_SPLIT", str(parts))
        monkeypatch.setenv("LIA_GEMM_BN", str(width))
        got = [ops.gemm(a, w, bias, epilogue=epilogue, residual=r) for _ in range(2)]
        monkeypatch.delenv("LIA_GEMM_BN")
        assert torch.equal(got[0], got[1])
        assert float((got[0].float() - whole.float()).abs().max()) <= TOL


@pytest.mark.parametrize("M,N,K", [(129, 768, 3072), (231, 2560, 10240), (384, 2048, 8192), (512, 2560, 10240)])
def test_taken_by_the_rule(M, N, K, monkeypatch):
    a, w, bias, res = operands(M, N, K)
    y = ops.gemm(a, w, bias, epilogue=ops.EPI_BIAS_RESIDUAL, residual=res)
    ref = ((a.float() @ w.float().T).to(BF16).float() + bias.float()).to(BF16).float() + res.float()
    assert float((y.float() - ref).abs().max()) <= TOL
    monkeypatch.setenv("LIA_GEMM_SPLIT", "1")
    assert not torch.equal(y, ops.gemm(a, w, bias, epilogue=ops.EPI_BIAS_RESIDUAL, residual=res))       # other sums: the parts were taken


def test_qkv_scatter(monkeypatch):
    B, S, H, d = 3, 77, 4, 64
    g = torch.Generator(device="cuda").manual_seed(0)
    a, w = torch.randn(B * S, 2048, generator=g, device="cuda").to(BF16), (torch.randn(3 * H * d, 2048, generator=g, device="cuda") * 2048 ** -0.5).to(BF16)
    got = []
    for parts in ("1", "4"):
        monkeypatch.setenv("LIA_GEMM_SPLIT", parts)
        q, k, v = torch.zeros(B * S, H * d, dtype=BF16, device="cuda"), *(torch.zeros(S + 2, B, H, d, dtype=BF16, device="cuda") for _ in range(2))
        ops.gemm(a, w, None, epilogue=ops.EPI_QKV, qkv=ops.qkv_args(q, k, v, S, 1, 0, 0.125))
        got.append((q, k, v))
    assert all(float((x.float() - y.float()).abs().max()) <= TOL for x, y in zip(*got))
    assert bool((got[1][1][0] == 0).all()) and bool((got[1][1][1] != 0).any())
