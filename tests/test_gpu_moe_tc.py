"""The experts' projections in one tensor-core launch (csrc/moe_sm100.cu) against float64, at the edges of its tiles: experts with 0, 1, 127, 128, 129 and
more rows, widths around 64, 128 and 256 columns, every form of the projections, pairs of experts without weights; and the vectorised gather
and combination around them."""
import pytest
import torch

import lia_b200  # noqa: F401
from lia_b200 import _lib, ops

pytestmark = pytest.mark.gpu
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
DEV = "cuda"


def act64(z, act):
    if act == ops.ACT_SILU:
        return z * torch.sigmoid(z)
    return torch.relu(z) ** 2 if act == ops.ACT_RELU_SQUARED else z


@pytest.mark.parametrize("counts,top", [([128, 0, 1, 127], 1), ([129, 300, 64], 2), ([5], 1), ([60, 3, 0, 9, 30], 3), ([1] * 149, 1)])            # (149 row tiles: more than SMs, wide and narrow column tiles)
@pytest.mark.parametrize("W,ff", [(64, 8), (72, 136), (264, 128), (136, 264)])
@pytest.mark.parametrize("form", ["plain", "gated", "clamped", "gated weigh in"])
def test_projections(counts, top, W, ff, form):
    g = torch.Generator().manual_seed(W + ff + len(counts))
    E, gated, weigh_in = len(counts) - (1 if len(counts) == 5 else 0), form != "plain", form == "gated weigh in"     # the last expert of five has no weights
    act = {"plain": ops.ACT_RELU_SQUARED, "clamped": ops.ACT_CLAMPED_SWISH}.get(form, ops.ACT_SILU)
    experts = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)])
    pairs = len(experts) // top * top
    idx = experts[torch.randperm(len(experts), generator=g)][:pairs].to(torch.int32).view(-1, top).contiguous()
    M = idx.shape[0]
    wt = torch.rand(M, top, generator=g) + 0.1
    h = torch.randn(M, W, generator=g).to(BF16)
    w_up = (torch.randn(E, (2 if gated else 1) * ff, W, generator=g) * W ** -0.5).to(BF16)
    w_down = (torch.randn(E, W, ff, generator=g) * ff ** -0.5).to(BF16)
    R = len(counts)
    n_tiles, tm = ops.moe_tiles(pairs, R, tensor_core=True)
    i32 = dict(dtype=torch.int32, device=DEV)
    perm, tile_expert, pos_of = torch.empty(n_tiles * tm, **i32), torch.empty(n_tiles, **i32), torch.empty(pairs, **i32)
    ops.moe_plan(idx.to(DEV), R, perm, tile_expert, pos_of)
    xs = torch.empty(n_tiles * tm, W, dtype=BF16, device=DEV)
    ops.moe_gather(h.to(DEV), perm, xs, top)
    at = pos_of.cpu().long()
    assert torch.equal(xs.cpu()[at], h.repeat_interleave(top, 0)) and bool((xs.cpu()[perm.cpu() < 0] == 0).all())
    mid = torch.empty(n_tiles * tm, ff, dtype=BF16, device=DEV)
    dwt = wt.to(DEV)
    ops.moe_gemm_tc(xs, w_up.to(DEV), mid, perm, tile_expert, dwt, True, act, gated=gated, act_params=(1.5, 1.7), weigh_in=weigh_in)
    # every pair in float64, from the bf16 numbers that the projections read
    e = idx.reshape(-1).long()
    real = e < E
    x = h.to(F64).repeat_interleave(top, 0)
    z = torch.stack([w_up.to(F64)[min(int(k), E - 1)] @ v for k, v in zip(e, x)]) * (wt.reshape(-1, 1).to(F64) if weigh_in else 1.0)
    if form == "clamped":
        a, u = z[:, :ff].clamp(max=1.5), z[:, ff:].clamp(-1.5, 1.5)
        want = a * torch.sigmoid(1.7 * a) * (u + 1.0)
    else:
        want = act64(z[:, :ff], act) * (z[:, ff:] if gated else 1.0)
    got = mid.cpu()[at][real].to(F64)
    assert float(((got - want[real]).abs() - want[real].abs() * 2.0 ** -8).max()) < 1e-5        # one rounding of a result made in fp32
    m64 = mid.cpu()[at].to(F64)
    down = torch.stack([w_down.to(F64)[min(int(k), E - 1)] @ v for k, v in zip(e, m64)])
    ys = torch.empty(n_tiles * tm, W, dtype=BF16, device=DEV)
    ops.moe_gemm_tc(mid, w_down.to(DEV), ys, perm, tile_expert, dwt, False)
    assert float(((ys.cpu()[at][real].to(F64) - down[real]).abs() - down[real].abs() * 2.0 ** -8).max()) < 1e-5
    yp = torch.full((pairs, W), 3.0, device=DEV)
    ops.moe_gemm_tc(mid, w_down.to(DEV), yp, perm, tile_expert, dwt, False, weigh_in=weigh_in)
    weighed = down * (1.0 if weigh_in else wt.reshape(-1, 1).to(F64))
    assert float((yp.cpu().to(F64)[real] - weighed[real]).abs().max()) < 1e-5 and bool((yp.cpu()[~real] == 3.0).all())
    # both ways through the combination, beside a gated shared expert and experts that hand the token back
    shared, gate = torch.randn(M, W, generator=g).to(BF16), torch.randn(M, 3, generator=g)
    ident = (idx.to(DEV), E, h.to(DEV), dwt) if E < R else None
    terms = torch.where(real[:, None], weighed, wt.reshape(-1, 1).to(F64) * x)
    total = terms.view(M, top, W).sum(1) + shared.to(F64) * torch.sigmoid(gate[:, 1:2].to(F64))
    for plan in (False, True):
        y = torch.empty(M, W, device=DEV)
        if plan:
            ops.moe_combine(ys, shared.to(DEV), y, top, pos_of=pos_of, wt=None if weigh_in else dwt, identity=ident, weighted=weigh_in, shared_gate=gate.to(DEV)[:, 1:2])
        else:
            ops.moe_combine(yp, shared.to(DEV), y, top, identity=ident, shared_gate=gate.to(DEV)[:, 1:2])
        # the plan's outputs are rounded to bf16 before they are weighted: half a unit of 2^-8 of each term
        bound = 1e-5 + (terms.abs().view(M, top, W).sum(1) * 2.0 ** -8 if plan else 0.0)
        assert bool(((y.cpu().to(F64) - total).abs() <= bound).all())
    assert _lib.load().lia_moe_timeouts() == 0


def test_a_plan_in_a_larger_buffer():
    """The rows of a tile do not follow from how much room a caller has left behind the plan."""
    E, idx = 3, torch.tensor([0, 2, 2, 0, 1] * 30, dtype=torch.int32, device=DEV)
    n_tiles, tm = ops.moe_tiles(idx.numel(), E)
    i32 = dict(dtype=torch.int32, device=DEV)
    plans = []
    for room in (0, 1, 36 * n_tiles):
        perm, tile_expert, pos_of = torch.full((n_tiles * tm + room,), 7, **i32), torch.empty(n_tiles, **i32), torch.empty(idx.numel(), **i32)
        ops.moe_plan(idx, E, perm, tile_expert, pos_of)
        place = perm[:n_tiles * tm].view(n_tiles, tm)
        assert all(bool((idx[p[p >= 0].long()] == e).all()) for p, e in zip(place, tile_expert.tolist())) and bool((perm[n_tiles * tm:] == 7).all())
        assert torch.equal(perm[pos_of.long()], torch.arange(idx.numel(), **i32))
        plans.append(tile_expert)
    assert torch.equal(plans[0], plans[1]) and torch.equal(plans[0], plans[2])
    with pytest.raises(_lib.LiaError):
        ops.moe_plan(idx, E, torch.empty(n_tiles * tm - 1, **i32), torch.empty(n_tiles, **i32), torch.empty(idx.numel(), **i32))


def test_captured_steps_keep_the_experts_outputs_in_fp32(monkeypatch):
    """However many pairs a captured (decoding) step has: the form that fewer pairs take, bit for bit."""
    from lia_b200.seq_layers import MoEFeedForward
    g = torch.Generator().manual_seed(2)
    E, top, W, ff, M = 4, 2, 64, 72, 300

    def r(*s):
        return torch.randn(*s, generator=g) * s[-1] ** -0.5
    experts = [{"gate": r(ff, W), "up": r(ff, W), "down": r(W, ff)} for _ in range(E)]
    m, h = MoEFeedForward(r(E, W), experts, top, ff, ops.ACT_SILU, None, BF16, DEV), torch.randn(M, W, generator=g).to(BF16).to(DEV)
    assert M * top >= MoEFeedForward.TENSOR_CORE_PAIRS
    m(h)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = m(h)
    graph.replay()
    eager = m(h)
    monkeypatch.setattr(MoEFeedForward, "TENSOR_CORE_PAIRS", 1 << 30)
    want = m(h)
    assert torch.equal(got, want) and not torch.equal(eager, want)


def test_expert_gemms_of_the_published_interface():
    """lia_moe_expert_gemms, a GEMM per expert for callers who know the rows per expert on the host: the feed-forward itself takes one launch for all."""
    g = torch.Generator().manual_seed(1)
    E, N, K, counts, tm = 3, 72, 64, [1, 0, 3], 64
    rows = sum(counts) * tm
    a, w = torch.randn(rows, K, generator=g).to(BF16), (torch.randn(E, N, K, generator=g) * K ** -0.5).to(BF16)
    out = torch.empty(rows, N, dtype=BF16, device=DEV)
    ops.moe_expert_gemms(a.to(DEV), w.to(DEV), out, counts, tm, ops.GemmWorkspace(ops.GemmWorkspace.bytes_for([(n * tm, N, K) for n in counts if n]), DEV))
    want, at = torch.empty(rows, N, dtype=F64), 0
    for e, n in enumerate(counts):
        want[at:at + n * tm] = a[at:at + n * tm].to(F64) @ w[e].to(F64).T
        at += n * tm
    assert bool(((out.cpu().to(F64) - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all())        # one rounding of a result made in fp32
