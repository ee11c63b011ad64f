"""GPU: kernels whose split of the work depends on how few tokens there are: the scatter's slices of a row, and the router
product of few experts in narrow tiles."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _layer(hidden, n_experts, top_k, gating=0):
    from moe_gen_b200 import MoELayer
    return MoELayer(hidden=hidden, inter=128, n_experts=n_experts, top_k=top_k, gating=gating, device="cuda:0")


@pytest.mark.parametrize("hidden", [256, 1024, 1280, 2304, 7168])       # 32 to 896 vectors, slices of 128 with and without a rest
@pytest.mark.parametrize("T", [1, 2, 7, 64, 333, 2367, 2369])           # 2368 = 16 warps on each of 148 SMs: one slice from there on
def test_scatter_copies_whole_rows(built_lib, hidden, T):
    k = 3
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
    H, many = 512, 148 * 128 + 1
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
