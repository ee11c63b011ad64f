"""GPU: the expert GEMMs with the weights on the accumulator's lanes (gemm_wl.cu), at the edges of their jobs: no row, one
row, multiples of 32 tokens and the rows around them, accumulators that share columns with the next job's and that do not,
one job and several per expert and per SM pair, jobs handed out by the counter and in fixed turns.  Rows between the
segments hold NaN, which must not reach a live row.  The shared expert runs the kernel with the tokens on the lanes
(gemm.cu) at the same edges."""
import pytest
import torch
import torch.nn.functional as F

from oracle import moe_oracle as O
from tests.util import make_layer

pytestmark = pytest.mark.gpu


def _close(got, ref, mag, what):
    """bf16 rounding of the result (2^-9, doubled for a value at a rounding edge) plus fp32 sums in any order:
    n additions of terms of total magnitude `mag` err by less than n 2^-24 mag, here with n <= 512."""
    err = (got.double() - ref).abs()
    bound = 2.0 ** -8 * ref.abs() + 512 * 2.0 ** -24 * mag
    assert torch.isfinite(got.float()).all(), what
    assert bool((err <= bound).all()), (what, float((err / bound.clamp_min(1e-30)).max()))


def _reference(x, wg, wu, wd, h_got):
    """h and its magnitude from x; out and its magnitude from the h the kernel produced."""
    x, wg, wu, wd = (t.double() for t in (x, wg, wu, wd))
    g, u = F.linear(x, wg), F.linear(x, wu)
    gm, um = F.linear(x.abs(), wg.abs()), F.linear(x.abs(), wu.abs())
    h = F.silu(g) * u
    # |d silu| <= 1.1: errors of g and u reach h times the other factor; __expf and the fast division add 4 ulp
    h_mag = 1.1 * gm * u.abs() + F.silu(g).abs() * um
    hq = h_got.double()
    return h, h_mag, F.linear(hq, wd), F.linear(hq.abs(), wd.abs())


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("counts", [
    [0, 1, 0, 31, 32, 33, 0, 2],
    [63, 64, 65, 127, 128, 129, 0, 0],
    [191, 192, 193, 255, 256, 257, 1, 0],
    [383, 384, 385, 0, 767, 769, 32, 16],
    [3100, 0, 1, 5, 0, 0, 40, 400],
    [0, 0, 0, 0, 0, 0, 0, 1],
])
def test_expert_products_at_job_edges(built_lib, counts, fp8):
    spec = O.LayerSpec(512, 384, 8, 2, 0, 1, 1, O.GATE_SOFTMAX_GREEDY, False, 1.0,
                       O.WEIGHT_FP8_BLOCK128 if fp8 else O.WEIGHT_BF16, O.COMBINE_FP32)
    _, W = O.make_inputs(spec, 4, 11)
    layer = make_layer(spec, W)
    cnt = torch.tensor(counts)
    pad = torch.zeros(9, dtype=torch.int64)
    pad[1:] = ((cnt + 127) // 128 * 128).cumsum(0)
    rows = int(pad[-1]) + 256
    x = torch.full((rows, 512), float("nan"), dtype=torch.bfloat16, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    for e, c in enumerate(counts):
        x[pad[e]:pad[e] + c] = torch.randn(c, 512, generator=g, device="cuda").to(torch.bfloat16)
    h, out = layer.expert_ffn(x, pad.int().cuda(), cnt.int().cuda())
    torch.cuda.synchronize()
    assert layer.device_status()[0] == 0
    for e, c in enumerate(counts):
        s = slice(int(pad[e]), int(pad[e]) + c)
        w = [m[e].cuda() for m in (W.w_gate, W.w_up, W.w_down)]
        rh, mh, ro, mo = _reference(x[s], *w, h[s])
        _close(h[s], rh, mh, ("h", e, c))
        _close(out[s], ro, mo, ("out", e, c))


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("counts", [
    [7, 8, 9, 15, 16, 17, 23, 24],         # jobs of 32 tokens leave out groups of eight without a live row
    [25, 1, 0, 41, 8, 392, 16, 400],
    [258, 287, 288, 289, 319, 320, 321, 0],     # jobs of 288, 320, 352 and 384 tokens are two MMAs per K step
    [351, 352, 353, 290, 0, 383, 700, 2],
])
def test_expert_products_at_the_edges_of_token_groups(built_lib, counts, fp8):
    test_expert_products_at_job_edges(built_lib, counts, fp8)


@pytest.mark.parametrize("T", [1, 31, 32, 33, 256, 257, 384, 385, 1000, 3500])
def test_shared_expert_at_job_edges(built_lib, T):
    spec = O.LayerSpec(512, 128, 8, 2, 384, 1, 1, O.GATE_SOFTMAX_GREEDY, False, 1.0, O.WEIGHT_BF16, O.COMBINE_FP32)
    x, W = O.make_inputs(spec, T, 12)
    layer = make_layer(spec, W)
    x = x.cuda()
    out = layer.shared_ffn(x)
    torch.cuda.synchronize()
    assert layer.device_status()[0] == 0
    xd, (wg, wu, wd) = x.double(), (m.cuda().double() for m in W.shared)
    h = F.silu(F.linear(xd, wg)) * F.linear(xd, wu)
    # the kernel rounds h to bf16 on the way: 2^-9 of it, carried through the second product
    hm = F.linear(h.abs(), wd.abs())
    err = (out.double() - F.linear(h, wd)).abs()
    assert bool((err <= 2.0 ** -8 * F.linear(h, wd).abs() + 2.0 ** -8 * hm).all())


@pytest.mark.parametrize("form", [0, 1, 2])
def test_inner_size_beyond_the_scale_row_is_refused_in_every_form(built_lib, form):
    """FP8 weights converted in the kernel take K up to 16384, whichever form converts them."""
    from moe_gen_b200 import MoELayer
    from moe_gen_b200 import lib as L
    layer = MoELayer(hidden=256, inter=16512, n_experts=4, top_k=2, weight_format=L.WEIGHT_FP8_BLOCK128, device="cuda:0")
    layer.set_router(torch.zeros(4, 256))
    layer.set_option(L.OPT_FP8_M256, form)
    with pytest.raises(L.MoeGenError, match="K a multiple of 128 up to 16384") as e:
        layer.forward(torch.zeros(3, 256, dtype=torch.bfloat16, device="cuda"))
    assert e.value.code == -2
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)


def _random_fp8_layer(hidden, inter, n_experts, seed):
    """A layer whose expert weights are random e4m3 values of every exponent below 2^5, drawn on the GPU."""
    from moe_gen_b200 import MoELayer
    from moe_gen_b200 import lib as L
    layer = MoELayer(hidden=hidden, inter=inter, n_experts=n_experts, top_k=2, weight_format=L.WEIGHT_FP8_BLOCK128,
                     device="cuda:0")
    layer.set_router(torch.zeros(n_experts, hidden))
    g = torch.Generator(device="cuda").manual_seed(seed)
    for e in range(n_experts):
        mats, scales = [], []
        for m, n in ((inter, hidden), (inter, hidden), (hidden, inter)):
            byte = torch.randint(0, 0x60, (m, n), generator=g, device="cuda", dtype=torch.uint8)
            sign = torch.randint(0, 2, (m, n), generator=g, device="cuda", dtype=torch.uint8)
            mats.append((byte | (sign << 7)).view(torch.float8_e4m3fn))
            scales.append(torch.rand(m // 128, n // 128, generator=g, device="cuda") * 0.01 + 0.001)
        layer.load_expert(e, *mats, tuple(scales))
    return layer


# every pattern repeats over the experts: narrow jobs (up to 192 tokens, one accumulator half), jobs of one and of two
# MMAs (up to 256 tokens, up to 384) and experts of several jobs next to one another
PATTERNS = {
    "mixed": [1, 384, 32, 193, 0, 256, 257, 192, 769, 64, 385, 5],
    "narrow": [1, 33, 192, 0, 96, 31, 160, 8],
    "wide_after_narrow": [7, 384, 7, 300, 7, 7, 224, 7],
}


@pytest.mark.parametrize("hidden,inter,n_experts", [(2304, 2176, 24), (512, 384, 256)])
@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_several_jobs_per_sm_pair_equal_the_other_forms(built_lib, pattern, hidden, inter, n_experts):
    """Rings, accumulator halves and scales carried from job to job: every SM pair gets several jobs of different
    lengths, K passes the 16 scale columns a converter loads at a time and ends inside a group of them (18 and 17
    columns).  Every live row has the same bits as with the tokens on the lanes and as with weights converted first."""
    layer = _random_fp8_layer(hidden, inter, n_experts, 3)
    counts = (PATTERNS[pattern] * n_experts)[:n_experts]
    tiles = sum((c + 383) // 384 for c in counts)
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert tiles * (2 * inter // 256) > 3 * pairs or tiles * (hidden // 256) > 3 * pairs
    cnt = torch.tensor(counts)
    pad = torch.zeros(n_experts + 1, dtype=torch.int64)
    pad[1:] = ((cnt + 127) // 128 * 128).cumsum(0)
    rows = int(pad[-1]) + 128
    x = torch.full((rows, hidden), float("nan"), dtype=torch.bfloat16, device="cuda")
    live = torch.zeros(rows, dtype=torch.bool, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    for e, c in enumerate(counts):
        live[pad[e]:pad[e] + c] = True
    x[live] = (torch.randn(int(live.sum()), hidden, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    pad_d, cnt_d = pad.int().cuda(), cnt.int().cuda()
    got = layer.expert_ffn(x, pad_d, cnt_d)
    again = layer.expert_ffn(x, pad_d, cnt_d)
    first = layer.expert_ffn(x, pad_d, cnt_d, predequant=True)
    layer.set_option(4, 0)
    tokens_on_lanes = layer.expert_ffn(x, pad_d, cnt_d)
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    for which, out in enumerate(got):
        assert bool(torch.isfinite(out[live].float()).all()) and bool((out[live] != 0).any())
        for other in (again, first, tokens_on_lanes):
            assert torch.equal(out[live].view(torch.int16), other[which][live].view(torch.int16)), which


@pytest.mark.parametrize("hidden,inter,n_experts", [(2304, 2176, 24), (512, 384, 256)])
@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_bf16_jobs_equal_the_form_with_tokens_on_the_lanes(built_lib, pattern, hidden, inter, n_experts):
    """bf16 weights: the same job patterns; every live row has the same bits as from 256 x 256 tiles with the tokens on the
    lanes.  K ends inside a stage that packs several steps for few tokens (34 and 6 steps)."""
    from moe_gen_b200 import MoELayer
    from moe_gen_b200 import lib as L
    layer = MoELayer(hidden=hidden, inter=inter, n_experts=n_experts, top_k=2, device="cuda:0")
    layer.set_router(torch.zeros(n_experts, hidden))
    g = torch.Generator(device="cuda").manual_seed(4)
    for e in range(n_experts):
        layer.load_expert(e, *((torch.randn(*shape, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
                               for shape in ((inter, hidden), (inter, hidden), (hidden, inter))))
    counts = (PATTERNS[pattern] * n_experts)[:n_experts]
    cnt = torch.tensor(counts)
    pad = torch.zeros(n_experts + 1, dtype=torch.int64)
    pad[1:] = ((cnt + 127) // 128 * 128).cumsum(0)
    x = torch.full((int(pad[-1]) + 128, hidden), float("nan"), dtype=torch.bfloat16, device="cuda")
    live = torch.zeros(x.shape[0], dtype=torch.bool, device="cuda")
    for e, c in enumerate(counts):
        live[pad[e]:pad[e] + c] = True
    x[live] = torch.randn(int(live.sum()), hidden, generator=g, device="cuda").to(torch.bfloat16)
    pad_d, cnt_d = pad.int().cuda(), cnt.int().cuda()
    got = layer.expert_ffn(x, pad_d, cnt_d)
    again = layer.expert_ffn(x, pad_d, cnt_d)
    layer.set_option(L.OPT_PAIR_GEMM, 1)
    tokens_on_lanes = layer.expert_ffn(x, pad_d, cnt_d)
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    for which, out in enumerate(got):
        assert bool(torch.isfinite(out[live].float()).all()) and bool((out[live] != 0).any())
        for other in (again, tokens_on_lanes):
            assert torch.equal(out[live].view(torch.int16), other[which][live].view(torch.int16)), which


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("T", [1, 40, 1024, 1025, 6000])
def test_jobs_handed_out_by_the_counter_equal_fixed_turns(built_lib, T, fp8):
    """The whole layer hands the jobs out by a counter that the plan kernels reset (one kernel up to 1024 tokens, another
    above); the stages by themselves give every pair its turns.  Same bits, forward after forward and on graph replay."""
    spec = O.LayerSpec(1024, 768, 32, 4, 256, 1, 1, O.GATE_SOFTMAX_GREEDY, False, 1.0,
                       O.WEIGHT_FP8_BLOCK128 if fp8 else O.WEIGHT_BF16, O.COMBINE_FP32)
    x, W = O.make_inputs(spec, T, 90 + T)
    x[:, 0] = 3.0                                # a skewed load: the router's column 0 decides
    layer = make_layer(spec, W)
    x = x.cuda()
    idx, w = layer.gate_route(x)[:2]
    counts, offsets, pad, dst = layer.permute_plan(idx)
    perm = layer.permute_rows(x, dst, layer.padded_rows(T * spec.top_k))
    want = layer.combine(layer.expert_ffn(perm, pad, counts)[1], dst, idx, w, layer.shared_ffn(x))
    for _ in range(3):
        assert torch.equal(layer.forward(x).view(torch.int16), want.view(torch.int16))
    out, s = torch.empty_like(x), torch.cuda.Stream()
    with torch.cuda.stream(s):
        layer.forward(x, out=out)
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            layer.forward(x, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert layer.device_status() == (0, 0)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_stage_call_by_counters_equals_fixed_turns(built_lib, pattern, fp8):
    """mg_expert_ffn with the caller's job counters, whose words hold anything before: the bits of fixed turns, also
    with FP8 weights converted first (a counter per part and product)."""
    from moe_gen_b200 import MoELayer
    from moe_gen_b200 import lib as L
    hidden, inter, n_experts = 2304, 2176, 24
    if fp8:
        layer = _random_fp8_layer(hidden, inter, n_experts, 6)
    else:
        layer = MoELayer(hidden=hidden, inter=inter, n_experts=n_experts, top_k=2, device="cuda:0")
        layer.set_router(torch.zeros(n_experts, hidden))
        g = torch.Generator(device="cuda").manual_seed(6)
        for e in range(n_experts):
            layer.load_expert(e, *((torch.randn(*shape, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
                                   for shape in ((inter, hidden), (inter, hidden), (hidden, inter))))
    cnt = torch.tensor((PATTERNS[pattern] * n_experts)[:n_experts])
    pad = torch.zeros(n_experts + 1, dtype=torch.int64)
    pad[1:] = ((cnt + 127) // 128 * 128).cumsum(0)
    g = torch.Generator(device="cuda").manual_seed(7)
    x = (torch.randn(int(pad[-1]), hidden, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    live = torch.zeros(x.shape[0], dtype=torch.bool, device="cuda")
    for e, c in enumerate(cnt.tolist()):
        live[pad[e]:pad[e] + c] = True
    pad_d, cnt_d = pad.int().cuda(), cnt.int().cuda()
    want = layer.expert_ffn(x, pad_d, cnt_d)
    buf = torch.full((L.JOB_COUNTERS + 1,), 12345, dtype=torch.int32, device="cuda")
    with layer.job_counters(buf[:L.JOB_COUNTERS]):
        got = [layer.expert_ffn(x, pad_d, cnt_d) for _ in range(3)]
        if fp8:
            got.append(layer.expert_ffn(x, pad_d, cnt_d, predequant=True))
    used = buf.clone()
    got.append(layer.expert_ffn(x, pad_d, cnt_d))
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    assert int(used[L.JOB_COUNTERS]) == 12345 and bool((used[:L.JOB_COUNTERS] != 12345).all())
    assert torch.equal(used, buf)                          # not touched once they are no longer set
    for out in got:
        for a, b in zip(out, want):
            assert torch.equal(a[live].view(torch.int16), b[live].view(torch.int16))


def test_auto_converts_first_where_the_kernels_that_convert_refuse(built_lib):
    """Inner sizes beyond 16384: MG_FP8_AUTO de-quantises first from 1024 rows per expert of the call on, or of the batch
    the caller says it belongs to; below, the call is refused."""
    from moe_gen_b200 import lib as L
    layer = _random_fp8_layer(256, 16512, 4, 9)
    g = torch.Generator(device="cuda").manual_seed(10)
    layer.set_router(torch.randn(4, 256, generator=g, device="cuda") * 0.05)
    x = (torch.randn(2048, 256, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    got = layer.forward(x)
    with pytest.raises(L.MoeGenError, match="K a multiple of 128 up to 16384"):
        layer.forward(x[:2047])
    layer.set_option(L.OPT_BATCH_TOKENS, 2048)
    part = layer.forward(x[:3])
    layer.set_option(L.OPT_BATCH_TOKENS, 0)
    layer.set_option(L.OPT_FP8_MODE, L.FP8_PREDEQUANT)
    want, want_part = layer.forward(x), layer.forward(x[:3])
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    assert bool(torch.isfinite(want.float()).all()) and bool((want != 0).any())
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.equal(part.view(torch.int16), want_part.view(torch.int16))
