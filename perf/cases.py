"""Cases that time the MoE layer through its public entry points (MoELayer.forward, .block_forward and
.forward_host), over the layer shapes and token counts the benchmark and the tests name.

A case is a dict: "shape" (a key of SHAPES), "tokens", "entry" ("forward": device tensors; "block": the
decoder layer's second half, norm + layer + residual; "host": pinned host buffers in and out) and "zipf"
(exponent of the router's load skew, 0 for a balanced load).  Weights are N(0, 0.02) and hidden states
N(0, 1), all drawn from the seed on the GPU.
"""
import math

import torch
import torch.nn.functional as F

SOFTMAX_GREEDY, SOFTMAX_GROUP_MAX, SIGMOID_NOAUX_TC, SOFTMAX_TOPK_RENORM = 0, 1, 2, 3     # MoELayer(gating=...)

# hidden, inter, experts, top_k, inter_shared, n_group, topk_group, gating, norm_topk_prob, routed_scale,
# fp8 (W8A16: e4m3 expert weights, one fp32 scale per 128x128 block), combine mode, most tokens of one call
SHAPES = {
    "v2lite": (2048, 1408, 64, 6, 2816, 1, 1, SOFTMAX_GREEDY, False, 1.0, False, 1, 16384),
    "mixtral8x7b": (4096, 14336, 8, 2, 0, 1, 1, SOFTMAX_TOPK_RENORM, True, 1.0, False, 2, 16384),
    "v2_236b": (5120, 1536, 160, 6, 3072, 8, 3, SOFTMAX_GROUP_MAX, False, 16.0, False, 1, 32768),
    "v3": (7168, 2048, 256, 8, 2048, 8, 4, SIGMOID_NOAUX_TC, True, 2.5, True, 0, 65536),
}
EPS = 1e-6
HOST_CHUNK = 4096


def _case(name, shape, tokens, entry="forward", zipf=0.0):
    return {"name": name, "shape": shape, "tokens": tokens, "entry": entry, "zipf": zipf}


def listed():
    return [
        # a handful of sequences decoding on the small model: launches and latency
        _case("v2lite_decode_8", "v2lite", 8),
        # the small model's prefill micro-batch (the shape the reference can run on a CPU)
        _case("v2lite_prefill_2048", "v2lite", 2048),
        # decoding with few, very large experts: every weight read for a few rows, odd batch
        _case("mixtral_decode_61", "mixtral8x7b", 61),
        # 32 sequences of 512 tokens, dense contraction, no shared expert
        _case("mixtral_prefill_16384", "mixtral8x7b", 16384),
        # decode batch of the 160-expert bf16 model: 19 rows per expert on average
        _case("v2_236b_decode_512", "v2_236b", 512),
        # its prefill, called as the decoder layer calls it (norm, layer, residual)
        _case("v2_236b_block_prefill_32768", "v2_236b", 32768, entry="block"),
        # W8A16 decode of a small batch: two rows per expert
        _case("v3_decode_64", "v3", 64),
        # W8A16 decode of an odd batch under the skewed load of real routers, as a decoder layer
        _case("v3_block_decode_333_zipf", "v3", 333, entry="block", zipf=1.2),
        # a middle batch under skew: experts from a few rows to thousands
        _case("v3_4096_zipf", "v3", 4096, zipf=1.2),
        # W8A16 prefill of one micro-batch from and to host memory, ragged length
        _case("v3_host_prefill_10007", "v3", 10007, entry="host"),
        # a decode batch as module-based batching builds it (512 rows per expert)
        _case("v3_decode_16384", "v3", 16384),
        # the headline batch
        _case("v3_prefill_65536", "v3", 65536),
    ]


def draw(rng):
    shape = rng.choice(["v2lite", "mixtral8x7b", "v2_236b", "v3", "v3"])
    most = SHAPES[shape][12]
    tokens = min(most, int(round(math.exp(rng.uniform(0.0, math.log(most))))))
    entry = rng.choice(["forward", "forward", "forward", "block", "host"])
    zipf = rng.choice([0.0, 0.0, 1.2, round(rng.uniform(0.3, 1.2), 2)])
    return {"shape": shape, "tokens": max(1, tokens), "entry": entry, "zipf": zipf}


# ------------------------------------------------------------------ inputs, from the seed alone
def _gen(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + what) % (1 << 62))
    return g


def _router(case, seed):
    H, E, gating = (SHAPES[case["shape"]][i] for i in (0, 2, 7))
    g = _gen(seed, 1)
    w = (torch.randn(E, H, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    bias = torch.randn(E, generator=g, device="cuda") * 0.01 if gating == SIGMOID_NOAUX_TC else None
    if case["zipf"] > 0:
        # a constant per expert, the log of a Zipf law over a random order, added through hidden column 0
        order = torch.randperm(E, generator=g, device="cuda")
        law = (torch.arange(1, E + 1, dtype=torch.float64, device="cuda") ** -case["zipf"]).log()
        col = torch.empty(E, device="cuda")
        col[order] = (law - law.mean()).float()
        w[:, 0] = col.to(torch.bfloat16)
    return w, bias


def _quantise(w):
    m, n = w.shape
    v = w.view(m // 128, 128, n // 128, 128)
    amax = v.abs().amax(dim=(1, 3), keepdim=True).float().clamp(1e-4)
    q = (v * (448.0 / amax)).to(torch.float8_e4m3fn).view(m, n)
    return q, (amax / 448.0).view(m // 128, n // 128)


def _expert(case, seed, e):
    """gate [I,H], up [I,H], down [H,I] of expert e (-1: the shared one), and their scales or None."""
    H, I, Is, fp8 = (SHAPES[case["shape"]][i] for i in (0, 1, 4, 10))
    n = Is if e < 0 else I
    flat = torch.randn(3 * n * H, generator=_gen(seed, 1000 + e), device="cuda", dtype=torch.bfloat16).mul_(0.02)
    mats = [flat[i * n * H:(i + 1) * n * H].view(*shp) for i, shp in enumerate(((n, H), (n, H), (H, n)))]
    if not fp8 or e < 0:
        return mats, None
    q = [_quantise(m) for m in mats]
    return [a for a, _ in q], tuple(b for _, b in q)


def _hidden(case, seed):
    H = SHAPES[case["shape"]][0]
    x = torch.randn(case["tokens"], H, generator=_gen(seed, 2), device="cuda").to(torch.bfloat16)
    if case["zipf"] > 0:
        x[:, 0] = 1.0
    norm = torch.ones(H, device="cuda")
    if case["entry"] == "block":
        norm = 1.0 + 0.05 * torch.randn(H, generator=_gen(seed, 3), device="cuda")
    return x, norm.to(torch.bfloat16)


def prepare(case, seed):
    from moe_gen_b200 import MoELayer
    H, I, E, k, Is, G, keep, gating, norm_prob, scale, fp8, combine, _ = SHAPES[case["shape"]]
    layer = MoELayer(hidden=H, inter=I, n_experts=E, top_k=k, inter_shared=Is, n_group=G, topk_group=keep,
                     gating=gating, norm_topk_prob=norm_prob, routed_scale=scale, weight_format=int(fp8),
                     combine_mode=combine, device="cuda:0")
    layer.set_router(*_router(case, seed))
    for e in range(E):
        mats, scales = _expert(case, seed, e)
        layer.load_expert(e, *mats, scales)
    if Is:
        layer.load_shared(*_expert(case, seed, -1)[0])
    x, norm = _hidden(case, seed)
    state = {"entry": case["entry"], "layer": layer, "x": x, "norm": norm}
    if case["entry"] == "host":
        state["x"] = x.cpu().pin_memory()
        state["y"] = torch.empty_like(state["x"], pin_memory=True)
    return state


def run(state):
    layer, x = state["layer"], state["x"]
    if state["entry"] == "block":
        return layer.block_forward(x, state["norm"], EPS)
    if state["entry"] == "host":
        return layer.forward_host(x, state["y"], chunk_tokens=HOST_CHUNK)
    return layer.forward(x)


# ------------------------------------------------------------------ what a pass cannot do without
def _experts_hit(E, k, T, zipf):
    """Expected number of experts with at least one row."""
    p = [float(i + 1) ** -zipf for i in range(E)]
    s = sum(p)
    return sum(1.0 - max(0.0, 1.0 - min(1.0, k * v / s)) ** T for v in p)


def work(case):
    H, I, E, k, Is, _, _, _, _, _, fp8, _, _ = SHAPES[case["shape"]]
    T = case["tokens"]
    expert = 3 * I * H * (1 + 4 / 16384 if fp8 else 2)
    weights = _experts_hit(E, k, T, case["zipf"]) * expert + 3 * Is * H * 2 + E * H * 2
    return {"bytes": weights + 2 * T * H * 2, "flops": 2.0 * T * H * (3 * (k * I + Is) + E)}


def tolerance(case):
    # bf16 rows, hidden activations and outputs, fp32 sums: 0.0029 to 0.0041 off the 64-bit result over the
    # listed cases.  No bound on single values: a token whose last pick is a tie at fp32 may go either way.
    return {"rel": 1.2e-2}


# ------------------------------------------------------------------ the same in 64 bits
def _route64(case, logits):
    """Picks [T,k] and weights from logits already rounded as the model defines them.  Scores are rounded
    to fp32 for the selection; equal scores go to the lower expert."""
    H, I, E, k, Is, G, keep, gating, norm_prob, scale, fp8, combine, _ = SHAPES[case["shape"]]
    logits, bias = logits
    T = logits.shape[0]

    def best(v, n):
        return v.sort(dim=-1, descending=True, stable=True).indices[:, :n]

    s = logits.double().sigmoid() if gating == SIGMOID_NOAUX_TC else logits.double().softmax(dim=-1)
    c = s.float()
    if gating == SIGMOID_NOAUX_TC:
        c = c + bias
    if gating in (SIGMOID_NOAUX_TC, SOFTMAX_GROUP_MAX):
        by_group = c.view(T, G, E // G)
        if gating == SIGMOID_NOAUX_TC:
            score = by_group.topk(2, dim=-1).values.sum(-1)
        else:
            score = by_group.max(dim=-1).values
        mask = torch.zeros(T, G, device=c.device).scatter_(1, best(score, keep), 1.0).bool()
        c = by_group.masked_fill(~mask.unsqueeze(-1), 0.0).view(T, E)
    idx = best(c, k)
    w = s.gather(1, idx)
    if norm_prob:
        w = w / (w.sum(-1, keepdim=True) + (0.0 if gating == SOFTMAX_TOPK_RENORM else 1e-20))
    if gating == SIGMOID_NOAUX_TC or not norm_prob:
        w = w * scale
    return idx, w


def _mlp64(x, mats, scales, step=8192):
    if scales is not None:
        # the weights of a W8A16 layer are bf16(float(q) * scale)
        mats = [(q.view(q.shape[0] // 128, 128, -1, 128).float() * s[:, None, :, None]).to(torch.bfloat16).view(q.shape)
                for q, s in zip(mats, scales)]
    g, u, d = (m.double() for m in mats)
    return torch.cat([F.linear(F.silu(F.linear(p, g)) * F.linear(p, u), d) for p in x.split(step)])


def exact(case, seed):
    H, I, E, k, Is, G, keep, gating, norm_prob, scale, fp8, combine, _ = SHAPES[case["shape"]]
    gate_w, bias = _router(case, seed)
    hidden, norm = _hidden(case, seed)
    x = hidden
    if case["entry"] == "block":
        # the layer's input is a bf16 tensor: rounded after the norm and after its weight
        h = hidden.double()
        h = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + EPS)).to(torch.bfloat16)
        x = (norm.double() * h.double()).to(torch.bfloat16)
    logits = torch.cat([F.linear(p.double(), gate_w.double()) for p in x.split(8192)])
    logits = logits.to(torch.bfloat16) if gating == SOFTMAX_TOPK_RENORM else logits.float()
    idx, w = _route64(case, (logits.float(), bias))
    y = torch.zeros(case["tokens"], H, dtype=torch.float64, device="cuda")
    for e in range(E):
        token, slot = (idx == e).nonzero(as_tuple=True)
        if token.numel():
            mats, scales = _expert(case, seed, e)
            y.index_add_(0, token, _mlp64(x[token].double(), mats, scales) * w[token, slot].unsqueeze(1))
    if Is:
        shared = _expert(case, seed, -1)[0]
        for i in range(0, case["tokens"], 8192):
            y[i:i + 8192] += _mlp64(x[i:i + 8192].double(), shared, None)
    if case["entry"] == "block":
        y += hidden.double()
    return y.cpu() if case["entry"] == "host" else y
