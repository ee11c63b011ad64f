"""GPU: the kernels of a forward overlap by programmatic dependence.  Forwards of different inputs, back to back without a
wait, give the bits of forwards whose kernels are launched one after the other (stage times are recorded then)."""
import pytest
import torch

from oracle import moe_oracle as O
from tests.util import make_layer

pytestmark = pytest.mark.gpu

SPECS = {
    "bf16_shared": O.LayerSpec(1024, 512, 32, 4, 512, 1, 1, O.GATE_SOFTMAX_GREEDY, False, 1.0, O.WEIGHT_BF16, O.COMBINE_BF16_PROD),
    "bf16_renorm": O.LayerSpec(1024, 512, 8, 2, 0, 1, 1, O.GATE_SOFTMAX_TOPK_RENORM, True, 1.0, O.WEIGHT_BF16, O.COMBINE_BF16_SEQ),
    "fp8_groups": O.LayerSpec(1024, 512, 64, 6, 256, 8, 4, O.GATE_SIGMOID_NOAUX_TC, True, 2.5, O.WEIGHT_FP8_BLOCK128, O.COMBINE_FP32),
}


@pytest.mark.parametrize("T", [1, 60, 1024, 1100, 5000, 16500])
@pytest.mark.parametrize("name", sorted(SPECS))
def test_back_to_back_forwards_equal_single_launches(built_lib, name, T):
    """Up to 128 tokens plan and scatter are one kernel, up to 1024 the plan, above it is four; the shared expert joins from
    its own stream up to 16384 tokens and follows in the same stream above, where every kernel behind the first is chained."""
    x, W = O.make_inputs(SPECS[name], T, 70 + T)
    layer = make_layer(SPECS[name], W)
    xs = [x.cuda(), x.flip(0).contiguous().cuda(), (x * 0.5).cuda()]
    norm = torch.ones(x.shape[1], dtype=torch.bfloat16, device="cuda")
    layer.set_stage_timing(True)
    want = [layer.forward(v).clone() for v in xs]
    want_block = [layer.block_forward(v, norm).clone() for v in xs]
    torch.cuda.synchronize()
    layer.set_stage_timing(False)
    got = [layer.forward(xs[i % 3]) for i in range(12)]
    got_block = [layer.block_forward(xs[i % 3], norm) for i in range(6)]
    torch.cuda.synchronize()
    assert layer.device_status() == (0, 0)
    for i, y in enumerate(got):
        assert torch.equal(y.view(torch.int16), want[i % 3].view(torch.int16)), i
    for i, y in enumerate(got_block):
        assert torch.equal(y.view(torch.int16), want_block[i % 3].view(torch.int16)), i


def test_workspace_sections_that_may_be_asked_for(built_lib):
    """The section behind the last of them, the job counters, is the library's own."""
    import ctypes as C
    from moe_gen_b200 import lib as L
    layer = make_layer(SPECS["bf16_renorm"], O.make_inputs(SPECS["bf16_renorm"], 1, 3)[1])
    ws = layer._workspace(64)
    p, got = C.c_void_p(), []
    for which in range(-1, 18):
        got.append(layer.lib.mg_workspace_ptr(layer._h, ws.data_ptr(), 64, 0, which, C.byref(p)))
    assert got == [-2] + [0] * 15 + [-2] * 3


@pytest.mark.parametrize("fill", [0, 0x7f, 0xff])
@pytest.mark.parametrize("T", [3, 200, 1500])
@pytest.mark.parametrize("name", sorted(SPECS))
def test_what_a_workspace_held_before_does_not_matter(built_lib, name, T, fill):
    """The expert GEMMs peek at the workspace's counts before the plan is known to be there; the peek may show anything,
    such as zeros, large numbers or negative ones, and decides nothing."""
    x, W = O.make_inputs(SPECS[name], T, 80 + T)
    layer = make_layer(SPECS[name], W)
    x = x.cuda()
    layer.set_stage_timing(True)
    want = layer.forward(x).clone()
    torch.cuda.synchronize()
    layer.set_stage_timing(False)
    for _ in range(3):
        layer._ws.fill_(fill)
        assert torch.equal(layer.forward(x).view(torch.int16), want.view(torch.int16))
    assert layer.device_status() == (0, 0)
