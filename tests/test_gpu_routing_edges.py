"""GPU: the one-block permute plan and the one-pass routing at the edges of their ranges."""

import pytest
import torch

from oracle import moe_oracle as O
from tests.util import make_layer

pytestmark = pytest.mark.gpu


def _router_only(E, k, H=256, gating=O.GATE_SOFTMAX_GREEDY, n_group=1, topk_group=1):
    spec = O.LayerSpec(H, 128, E, k, 0, n_group, topk_group, gating, True, 1.0, O.WEIGHT_BF16, O.COMBINE_FP32)
    g = torch.Generator().manual_seed(3)
    bias = torch.randn(E, generator=g) * 0.01 if gating == O.GATE_SIGMOID_NOAUX_TC else None
    return spec, make_layer(spec, O.LayerWeights((torch.randn(E, H, generator=g) * 0.02).to(torch.bfloat16), bias))


@pytest.mark.parametrize("E,k", [(8, 2), (64, 6), (512, 16)])
@pytest.mark.parametrize("T", [1, 31, 32, 33, 256, 1023, 1024, 1025])
def test_permute_plan_at_the_one_block_limit(built_lib, T, E, k):
    _, layer = _router_only(E, k)
    idx = torch.rand(T, E, generator=torch.Generator().manual_seed(T)).topk(k, dim=1).indices
    counts, offsets, pad, dst = layer.permute_plan(idx.int().cuda())
    rc, roff, order, _ = O.permute_plan(idx, E)
    assert torch.equal(counts.cpu().long(), rc) and torch.equal(offsets.cpu().long(), roff)
    padc = pad.cpu().long()
    assert torch.equal(padc[1:] - padc[:-1], (rc + 127) // 128 * 128)
    rank = torch.arange(T * k) - roff[:-1].repeat_interleave(rc)
    want = torch.empty(T * k, dtype=torch.int64)
    want[order] = padc[:-1].repeat_interleave(rc) + rank
    assert torch.equal(dst.cpu().long().view(-1), want)


@pytest.mark.parametrize("gating", [O.GATE_SOFTMAX_GREEDY, O.GATE_SOFTMAX_TOPK_RENORM])
@pytest.mark.parametrize("E", [36, 40, 100, 160, 252])
def test_router_product_in_narrow_tiles_equals_the_wide_ones(built_lib, E, gating):
    """32-column tiles while they fit one wave, at expert counts that are no multiple of 32: the same bits as rows of a
    batch too large for them, fp32 and bf16-rounded logits, at the edges of the row tiles and of the rule."""
    _, layer = _router_only(E, 4, gating=gating)
    tiles = torch.cuda.get_device_properties(0).multi_processor_count // ((E + 31) // 32)       # row tiles of one wave
    x = torch.randn(128 * tiles + 1, 256, generator=torch.Generator().manual_seed(E)).to(torch.bfloat16).cuda()
    wide = layer.gate_logits(x)
    exact = x.double() @ layer.gate_w.double().t()
    # fp32 sums of 256 products in any order; bf16 logits round once more
    bound = 256 * 2.0 ** -24 * (x.double().abs() @ layer.gate_w.double().abs().t())
    if gating == O.GATE_SOFTMAX_TOPK_RENORM:
        bound = bound + 2.0 ** -8 * exact.abs()
    assert bool(((wide.double() - exact).abs() <= bound).all())
    for T in (1, 127, 128, 129, 128 * tiles - 1, 128 * tiles):
        assert torch.equal(layer.gate_logits(x[:T].contiguous()), wide[:T]), T


@pytest.mark.parametrize("lo,n", [(0, 24), (5, 13)])
@pytest.mark.parametrize("T", [1, 40, 256, 257, 700, 1024])
def test_one_block_plan_of_repeated_and_foreign_picks_equals_the_general_plan(built_lib, T, lo, n):
    """Picks that name an expert twice count twice and foreign picks not at all, in one block as in the four
    kernels of larger batches; those run here on the same picks followed by tokens without a pick."""
    _, layer = _router_only(24, 6)
    idx = torch.randint(0, 24, (T, 6), generator=torch.Generator().manual_seed(T), dtype=torch.int32)
    idx[::7, 5] = idx[::7, 0]
    idx[::5, 2] = -1
    got = layer.permute_plan(idx.cuda(), lo, n)
    padded = torch.cat([idx, torch.full((1100, 6), -1, dtype=torch.int32)])
    want = layer.permute_plan(padded.cuda(), lo, n)
    assert torch.equal(got[0].cpu().long(), torch.bincount(idx[(idx >= lo) & (idx < lo + n)].long() - lo, minlength=n))
    for a, b in zip(got[:3], want[:3]):
        assert torch.equal(a, b)
    assert torch.equal(got[3], want[3][:T])


@pytest.mark.parametrize("gating,E,k,n_group,topk_group", [
    (O.GATE_SOFTMAX_GREEDY, 64, 6, 1, 1), (O.GATE_SOFTMAX_GROUP_MAX, 160, 6, 8, 3),
    (O.GATE_SIGMOID_NOAUX_TC, 256, 8, 8, 4), (O.GATE_SOFTMAX_GROUP_MAX, 96, 4, 3, 2)])
@pytest.mark.parametrize("T", [1, 8, 9, 700])
def test_forward_routes_as_the_staged_call(built_lib, gating, E, k, n_group, topk_group, T):
    """The forward's picks, weights and logits are those of the staged call, bit for bit; every configuration's groups are
    runs of lanes (8 in the last one).  Tokens that tie: the next test."""
    spec = O.LayerSpec(512, 128, E, k, 0, n_group, topk_group, gating, True, 1.0, O.WEIGHT_BF16, O.COMBINE_FP32)
    _, W = O.make_inputs(spec, 1, 7)
    layer = make_layer(spec, W)
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, 512, generator=g, device="cuda").to(torch.bfloat16)
    x[T // 2:] = x[0]                                   # repeated tokens, and rows of a single column
    x[::3, 1:] = 0
    idx, w, logits, _ = layer.gate_route(x)
    layer.forward(x)
    torch.cuda.synchronize()

    def view(which, shape, dtype):
        off = layer.workspace_view(which, T) - layer._ws.data_ptr()
        n = torch.Size(shape).numel() * 4
        return layer._ws[off:off + n].view(dtype).view(shape)
    assert torch.equal(view(1, (T, k), torch.int32), idx)
    assert torch.equal(view(2, (T, k), torch.float32), w)
    assert torch.equal(view(0, (T, E), torch.float32), logits)


def _workspace(layer, which, T, shape, dtype):
    off = layer.workspace_view(which, T) - layer._ws.data_ptr()
    n = torch.Size(shape).numel() * 4
    return layer._ws[off:off + n].view(dtype).view(shape)


@pytest.mark.parametrize("gating,E,k,n_group,topk_group,lane_runs", [
    (O.GATE_SOFTMAX_GREEDY, 64, 6, 1, 1, True), (O.GATE_SOFTMAX_GROUP_MAX, 160, 6, 8, 3, True),
    (O.GATE_SIGMOID_NOAUX_TC, 256, 8, 8, 4, True), (O.GATE_SOFTMAX_GROUP_MAX, 96, 4, 4, 2, False)])
@pytest.mark.parametrize("T", [1, 7, 8, 9, 296, 297, 592, 593, 1184, 1185, 2500])
def test_rows_with_many_logits_in_play_are_routed_by_the_exact_logits(built_lib, gating, E, k, n_group, topk_group,
                                                                      lane_runs, T):
    """Rows of zeros (all, a few, the last half), tiny rows and rows with a few close logits among ordinary ones, alone and in runs, at the edges of
    the cluster sizes: picks as from the correctly rounded logits.  Where the listing kernels' list of pairs holds, the
    logits and weights are theirs bit for bit; where it overflows they recompute whole rows, and a logit out of play may
    be off by the bound e of the router product, a weight by 2 e of itself (softmax; the sigmoid moves by e / 4, and its
    share of the sum by twice that).  Groups of six lanes take the listing kernels either way."""
    H = 1024
    spec = O.LayerSpec(H, 128, E, k, 0, n_group, topk_group, gating, True, 1.0, O.WEIGHT_BF16, O.COMBINE_FP32)
    g = torch.Generator().manual_seed(T)
    gw = (torch.randn(E, H, generator=g) * 0.02).to(torch.bfloat16)
    bias = torch.zeros(E) if gating == O.GATE_SIGMOID_NOAUX_TC else None
    layer = make_layer(spec, O.LayerWeights(gw, bias))
    base = torch.randn(T, H, generator=g).to(torch.bfloat16)
    for name in ("ordinary", "zeros", "few", "tail", "tiny", "scattered"):
        x = base.clone()
        if name == "zeros":
            x[:] = 0
        elif name == "few":
            x[::97] = 0
        elif name == "tail":
            x[T // 2:] = 0
        elif name == "tiny":
            x *= torch.tensor(2.0 ** -11, dtype=torch.bfloat16)
        elif name == "scattered":
            x[::5] = 0
            x[1::5] *= torch.tensor(2.0 ** -9, dtype=torch.bfloat16)
        x = x.cuda()
        idx, w, logits, fix = layer.gate_route(x)
        layer.forward(x)
        torch.cuda.synchronize()
        assert layer.device_status() == (0, 0)
        got_idx, got_w = _workspace(layer, 1, T, (T, k), torch.int32), _workspace(layer, 2, T, (T, k), torch.float32)
        exact = (x.double() @ gw.cuda().double().t()).float()
        want = layer.route_topk(exact)[0]
        assert torch.equal(got_idx.sort(1).values, want.sort(1).values), (name, T)
        assert torch.equal(got_idx.sort(1).values, idx.sort(1).values), (name, T)
        n_fix, n_rows, n_pairs = (int(v) for v in fix[:3])
        if name == "zeros":                              # every token ties, with all its logits (or groups) in play
            assert n_fix == T and (n_pairs > 0 if lane_runs else n_rows == T), (n_fix, n_rows, n_pairs)
        if name == "few":                                # the list holds them: compared bit for bit below
            assert n_fix > 0 and (0 < n_pairs <= 8 * T + 64 or T < 296 or not lane_runs), (n_fix, n_pairs)
        if n_pairs <= 8 * T + 64 or not lane_runs:
            assert torch.equal(got_w, w) and torch.equal(_workspace(layer, 0, T, (T, E), torch.float32), logits), name
        else:
            assert n_rows > 0
            bound = 2 * (6.0e-9 * H + 4.0e-6) * max(1.0, float(exact.abs().max())) + 8 * 2.0 ** -24
            order, ref = got_idx.argsort(1), idx.argsort(1)
            a, b = got_w.gather(1, order), w.gather(1, ref)
            assert float(((a - b).abs() / b.abs()).max()) <= bound, name
