"""GPU: kernels whose split of the work depends on how few tokens there are: the scatter's slices of a row, the plan and the
scatter in one launch, and the router product of few experts in narrow tiles."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _sm_count():
    return torch.cuda.get_device_properties(0).multi_processor_count


def _layer(hidden, n_experts, top_k, gating=0):
    from moe_gen_b200 import MoELayer
    return MoELayer(hidden=hidden, inter=128, n_experts=n_experts, top_k=top_k, gating=gating, device="cuda:0")


@pytest.mark.parametrize("hidden", [256, 1024, 1280, 2304, 7168])       # 32 to 896 vectors, slices of 128 with and without a rest
@pytest.mark.parametrize("per_sm,T", [(0, 1), (0, 2), (0, 7), (0, 64), (0, 333), (16, -1), (16, 1)])     # 16 warps per SM: one slice from there on
def test_scatter_copies_whole_rows(built_lib, hidden, per_sm, T):
    k, T = 3, T + per_sm * _sm_count()
    layer = _layer(hidden, 16, k)
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, hidden, generator=g, device="cuda").to(torch.bfloat16)
    dst = torch.randperm(T * k + 5, generator=g, device="cuda")[:T * k].view(T, k).int()
    dst[T // 2, 1] = -1                                                   # a pick that goes nowhere
    rows = T * k + 128
    got = layer.permute_rows(x, dst, rows)
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    for j in range(k):
        live = dst[:, j] >= 0
        assert torch.equal(got[dst[live, j].long()].view(torch.int16), x[live].view(torch.int16))


@pytest.mark.parametrize("n_experts", [4, 8, 16, 20, 32, 36])
@pytest.mark.parametrize("T", [1, 127, 129, 2048])
@pytest.mark.parametrize("gating", [0, 3])
def test_router_product_of_few_experts(built_lib, n_experts, T, gating):
    """The same bits whatever the tile: those of a call of so many tokens that no wave of narrow tiles takes them.  And within
    fp32 sums of H products (truncated partial sums: H / 16 steps of 2^-23 of the terms' magnitude), or one bf16 rounding."""
    H, many = 512, _sm_count() * 128 + 1
    layer = _layer(H, n_experts, 2, gating)
    g = torch.Generator(device="cuda").manual_seed(n_experts)
    w = (torch.randn(n_experts, H, generator=g, device="cuda") * 0.05).to(torch.bfloat16).float()
    layer.set_router(w)
    x = torch.randn(many, H, generator=g, device="cuda").to(torch.bfloat16)
    got, want = layer.gate_logits(x[:T]), layer.gate_logits(x)[:T]
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    assert torch.equal(got, want)
    ref, mag = F.linear(x[:T].double(), w.double()), F.linear(x[:T].double().abs(), w.double().abs())
    err = H / 16 * 2.0 ** -23 * mag
    if gating == 3:
        err = err + 2.0 ** -8 * (ref.abs() + err)
    assert bool(((got.double() - ref).abs() <= err).all())


@pytest.mark.parametrize("hidden", [1280, 2304, 4096])                   # 160, 288 and 512 vectors
@pytest.mark.parametrize("T", [1, 2, 3, 4, 31, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("n_experts", [8, 260])
def test_plan_and_scatter_in_one_launch(built_lib, hidden, T, n_experts):
    """Up to 128 tokens, from 4096 elements on, the forward plans and scatters in one launch: its tables, its rows and its
    result are those of the stages.  Twice in one workspace: first over bytes that are no tables, then over the tables of
    other picks."""
    k = 3
    layer = _layer(hidden, n_experts, k)
    g = torch.Generator(device="cuda").manual_seed(T)
    layer.set_router(torch.randn(n_experts, hidden, generator=g, device="cuda") * 0.02)
    for e in range(n_experts):
        layer.load_expert(e, *((torch.randn(*s, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
                               for s in ((128, hidden), (128, hidden), (hidden, 128))))
    ws = layer._workspace(T)
    ws.fill_(0xff)

    def section(which, like):
        p = C.c_void_p()
        assert layer.lib.mg_workspace_ptr(layer._h, ws.data_ptr(), T, 0, which, C.byref(p)) == 0
        at = p.value - ws.data_ptr()
        return ws[at:at + like.numel() * like.element_size()].view(like.dtype).view(like.shape)

    for _ in range(2):
        x = torch.randn(T, hidden, generator=g, device="cuda").to(torch.bfloat16)
        logits = torch.randn(T, n_experts, generator=g, device="cuda")
        idx, w = layer.route_topk(logits)
        plan = layer.permute_plan(idx)
        counts, offsets, pad, dst = plan
        rows = layer.permute_rows(x, dst, layer.padded_rows(T * k))
        want = layer.combine(layer.expert_ffn(rows, pad, counts)[1], dst, idx, w, None)
        got = layer.forward_from_logits(x, logits)
        torch.cuda.synchronize()
        assert layer.device_status() == (0, 0)
        # top-k, plan, scatter, two products, combine
        assert layer.last_launch_count() == (5 if T <= 128 and T * hidden >= 4096 else 6)
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
        for which, t in zip((3, 4, 5, 6), plan):
            assert torch.equal(section(which, t), t), which
        live = dst.flatten().long()
        assert torch.equal(section(7, rows)[live].view(torch.int16), rows[live].view(torch.int16))
