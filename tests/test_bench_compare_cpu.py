"""The per-kernel tables of the comparison benchmark: every operator a layer calls is in them, with the work it does and the unit that does it."""
import inspect
import re

import torch

from lia_b200 import bench_compare, ops, seq_layers
from lia_b200 import modeling_bebulorn, modeling_bizetar, modeling_davasun, modeling_pazivik, modeling_sekenex, modeling_zatusun

BF16, F32 = torch.bfloat16, torch.float32
# what launches nothing, or asks
HOST = {"count_launches", "GemmWorkspace", "moe_tiles", "moe_timeouts_seen", "latent_attn_splits", "latent_attn_split_class", "window_attn_split_class", "window_decode_splits"}


def test_every_operator_of_the_layers_is_instrumented():
    named = set()
    for m in (seq_layers, modeling_bebulorn, modeling_bizetar, modeling_davasun, modeling_pazivik, modeling_sekenex, modeling_zatusun):
        named |= set(re.findall(r"\bops\.([a-z]\w*)\(", inspect.getsource(m)))
    assert {"moe_gemm_tc", "latent_attn_expanded", "mlstm_scan"} <= named and all(callable(getattr(ops, n)) for n in named)
    assert named - HOST <= set(bench_compare.Instrument.NAMES), sorted(named - HOST - set(bench_compare.Instrument.NAMES))
    assert all(callable(getattr(ops, n)) for n in bench_compare.Instrument.NAMES)


def test_costs_of_the_tensor_core_forms():
    e = lambda *s, dt=BF16: torch.empty(*s, dtype=dt)  # noqa: E731
    M, H, dim, rot, rank = 100, 4, 128, 64, 512
    portions, cache, out = [(0, 20, 0, 60), (1, 0, 60, 40)], e(2, 80, rank + rot), e(M, H * dim)
    keys, latents = sum(range(21, 81)) + sum(range(1, 41)), 80 + 40
    fl, by, kind = bench_compare._cost("latent_attn_expanded", (e(M, H * 192), e(M, H, rot, dt=F32), cache, portions, e(2 * H * dim, rank), None, out, H, dim, rot, rank, 0.1), {})
    assert kind == "tc" and fl == 2 * keys * H * (2 * dim + rot) + 2 * latents * 2 * H * dim * rank
    assert by == M * (H * 192 * 2 + H * rot * 4 + H * dim * 2) + latents * (rank + rot) * 2 + 2 * H * dim * rank * 2
    fl, _, _ = bench_compare._cost("latent_attn_expanded", (e(M, H * 192), e(M, H, rot, dt=F32), cache, portions, e(2 * H * dim, rank), None, out, H, dim, rot, rank, 0.1), {"window": 8})
    assert fl == 2 * (60 * 8 + sum(min(8, i) for i in range(1, 41))) * H * (2 * dim + rot) + 2 * (60 + 7 + 40) * 2 * H * dim * rank
    pairs, E, N, K = 300, 16, 256, 128
    args = (e(2048, K), e(E, 2 * N, K), e(2048, N), None, None, e(150, 2, dt=F32), True)
    fl, by, kind = bench_compare._cost("moe_gemm_tc", args, {"gated": True})
    assert kind == "tc" and fl == 2 * pairs * 2 * N * K and by == pairs * (K * 2 + N * 2) + E * 2 * N * K * 2
    scan = lambda q, **kw: bench_compare._cost("linear_scan", (q, q, q, None, e(1, 4, dt=torch.int32), 4, 4, 128, 128, e(q.shape[0], 512, dt=F32)), kw)[2]  # noqa: E731
    d = e(4, dt=F32)
    assert scan(e(64, 512), decay=d, lengths=(64, 64)) == "tc" and scan(e(64, 512), decay=d, lengths=(1, 31)) == "f32"
    assert scan(e(64, 512), gates=d, lengths=(64, 64)) == "f32" and scan(e(64, 512, dt=F32), decay=d, lengths=(64, 64)) == "f32"
    plain = lambda x, w: bench_compare._cost("linear_plain", (x, w, e(x.shape[0], w.shape[0], dt=F32)), {})[2]  # noqa: E731
    assert plain(e(65, 64), e(8, 64)) == "tc" and plain(e(64, 64), e(8, 64)) == "tc" and plain(e(65, 64), e(8, 64, dt=F32)) == "f32" and plain(e(65, 60), e(8, 60)) == "f32"
    assert plain(e(64, 64, dt=F32), e(8, 64)) == "f32" and plain(e(65, 64, dt=F32), e(8, 64)) == "tc" and plain(e(64, 60), e(8, 60)) == "f32"
    ssd = lambda M, N, vdim, **kw: bench_compare._cost("ssd_scan", (e(M, 4 * vdim + 2 * N, dt=F32), e(M, 8, dt=F32), None, None, e(1, 4, dt=torch.int32), 4, 1, N, vdim,  # noqa: E731
                                                                    e(M, 4 * vdim, dt=F32)), kw)[2]
    assert ssd(448, 128, 64) == "tc" and ssd(447, 128, 64) == "f32" and ssd(600, 128, 64, lengths=(1, 300)) == "f32" and ssd(600, 64, 64) == "f32" and ssd(600, 128, 40) == "f32"
