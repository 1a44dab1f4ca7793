"""Numbers that are not finite in the keys and values of the tensor-core attention kernels (csrc/window_attn_mma.cu, csrc/latent_attn_mma.cu): a row that
sees them says so, and no other row does."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import ops

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32
DEV = "cuda"


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
