"""Waits that run out in the attention kernels on tcgen05 (csrc/window_attn_sm100.cu, csrc/latent_attn_sm100.cu, csrc/latent_expand_sm100.cu): built with a limit of 0, so that every bounded wait
gives up at once and no barrier is touched, a launch ends, leaves NaN in every row it owns and nothing elsewhere, and counts its CTAs; the next launch of the usual build is right."""
import ctypes
import os
import subprocess

import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import _lib, ops

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32
D = 128


@pytest.fixture(scope="module")
def nowait():
    _lib.load()                                                     # first, so that its own calls stay its own
    csrc = os.path.join(os.path.dirname(_lib.__file__), "csrc")
    subprocess.run(["make", "-C", csrc, "-j", str(os.cpu_count() or 4), "nowait"], check=True, capture_output=True, timeout=900)
    lib = ctypes.CDLL(os.path.join(csrc, "build", "nowait", "libliab200_nowait.so"))
    for name, (res, args) in _lib._PROTOTYPES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    return lib


def given_up(lib, monkeypatch, call):
    """``call`` with the kernels that give up; how many CTAs did."""
    with monkeypatch.context() as m:
        m.setattr(_lib, "_lib", lib)
        before = lib.lia_moe_timeouts()
        call()
        return lib.lia_moe_timeouts() - before


@pytest.mark.parametrize("q_f32", [False, True])
def test_window_attention(nowait, monkeypatch, q_f32):
    H, G, portions = 4, 2, [(0, 0, 0, 300), (1, 70, 300, 129), (2, 5, 431, 33)]         # rows 429 and 430 are nobody's
    g = torch.Generator(device="cuda").manual_seed(0)
    M, cap = 464, 400
    q = torch.randn(M, H * D, generator=g, device="cuda")
    q = q if q_f32 else q.to(BF16)
    kc, vc = (torch.randn(3, cap, G * D, generator=g, device="cuda").to(BF16) for _ in range(2))
    segs = torch.tensor(portions, dtype=torch.int32, device="cuda")
    meta = torch.zeros(M, 2, dtype=torch.int32, device="cuda")
    out = torch.full((M, H * D), 7.0, device="cuda")

    def call():
        ops.window_attn(q, kc, vc, meta, None, out, H, G, D, D, 0, 0.1, 0.0, nseg=3, segs=segs, form=2)
    assert given_up(nowait, monkeypatch, call) == H * (3 + 2 + 1)
    assert torch.isnan(out[:429]).all() and torch.isnan(out[431:]).all() and (out[429:431] == 7.0).all()
    call()
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("rank", [64, 192, 512])
def test_latent_attention_and_expansion(nowait, monkeypatch, rank):
    H, rot, portions = 24, 64, [(1, 0, 0, 300), (0, 40, 302, 33)]                       # 300 and 73 latents: last tiles with lanes and warps without a row; 5 or 6 tiles of columns a CTA
    g = torch.Generator(device="cuda").manual_seed(0)
    M = 335
    q, qr = torch.randn(M, H * (D + rot), generator=g, device="cuda").to(BF16), torch.randn(M, H, rot, generator=g, device="cuda")
    lat = torch.randn(2, 320, rank + rot, generator=g, device="cuda").to(BF16)
    w = (torch.randn(2 * H * D, rank, generator=g, device="cuda") * rank ** -0.5).to(BF16)
    out = torch.full((M, H * D), 7.0, device="cuda")

    def call():
        ops.latent_attn_expanded(q, qr, lat, portions, w, None, out, H, D, rot, rank, 0.1)
    tiles = 3 + 1
    groups = min(2 * H * D // 32, torch.cuda.get_device_properties(0).multi_processor_count // tiles)
    assert given_up(nowait, monkeypatch, call) == tiles * groups + H * tiles
    assert torch.isnan(out[:300]).all() and torch.isnan(out[302:]).all() and (out[300:302] == 7.0).all()
    call()
    assert torch.isfinite(out).all()
