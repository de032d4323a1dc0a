"""The work a user of the fused MoE layer has it do, as measurable cases.

A case is one pass of one of these operations through ``b12x_b200.moe.fused_moe``:

* ``layer``  -- router logits in hand: ``route_topk`` -> ``bind`` -> ``run`` (what a model's MoE block calls);
* ``sparse`` -- hidden states and a gate matrix in hand: ``bind_sparse`` -> ``run_sparse``;
* ``route``  -- hidden states and a gate matrix in hand, the selection alone: ``bind_route`` -> ``route``.

``graph`` is the serving form of a decode step: the pass is captured once in a CUDA graph over static buffers and
replayed.  Activations are N(0, 1), weights N(0, 0.02) quantised to the recipe's 4-bit format, router logits N(0, 1)
(with a Zipf load bias where ``zipf`` is set), all made on the GPU from the seed.
"""

from __future__ import annotations

import math

import torch

from b12x_b200.moe import fused_moe

# Model-shaped layers.  max_tokens: the largest batch a case or a draw takes.
FAMILIES = {
    # DeepSeek-V3-shaped experts: many small experts, sigmoid router with a route scale
    "dsv3": dict(recipe="nvfp4", activation="silu", hidden=7168, inter=2048, experts=256, topk=8, router="sigmoid",
                 route_scale=2.5, zipf=0.0, max_tokens=4096),
    # Mixtral-shaped experts: few large experts, skewed load
    "mixtral": dict(recipe="nvfp4", activation="silu", hidden=4096, inter=14336, experts=8, topk=2, router="softmax",
                    route_scale=1.0, zipf=1.2, max_tokens=8192),
    # Qwen3-235B-shaped experts with 16-bit activations; `inter` is 768 / 384 / 192 under tensor parallelism
    "qwen3": dict(recipe="w4a16", activation="silu", hidden=4096, inter=1536, experts=128, topk=8, router="softmax",
                  route_scale=1.0, zipf=0.0, max_tokens=4096),
    # GPT-OSS-shaped experts: MXFP4 weights, MXFP8 activations, SwiGLU-OAI
    "gptoss": dict(recipe="w4a8_mx", activation="swigluoai", hidden=2880, inter=2880, experts=128, topk=4,
                   router="softmax", route_scale=1.0, zipf=0.0, max_tokens=16384),
}

ACT_API = {"silu": "silu", "swigluoai": "swigluoai_uninterleave"}
SOURCE = {"nvfp4": "modelopt_nvfp4", "w4a16": "modelopt_nvfp4", "w4a8_mx": "fp4_e8m0_k32"}


def _case(name, op, family, tokens, graph=False, **over):
    shape = {k: v for k, v in FAMILIES[family].items() if k != "max_tokens"}
    case = dict(name=name, op=op, tokens=tokens, graph=graph, **{**shape, **over})
    if name is None:
        del case["name"]
    return case


def listed():
    return [
        # one user's next token: latency, eight experts' weights
        _case("decode_nvfp4_t1", "layer", "dsv3", 1, graph=True),
        # a full decode batch: nearly every expert's weights are read for a handful of rows each
        _case("decode_nvfp4_t64", "layer", "dsv3", 64, graph=True),
        # decode tokens and a piece of a prompt in one ragged batch
        _case("mixed_nvfp4_t517", "layer", "dsv3", 517),
        # a large prompt batch on few, unevenly loaded experts
        _case("prefill_nvfp4_skew_t8192", "layer", "mixtral", 8192),
        # decode with 8-bit activations
        _case("decode_mx_t32", "layer", "gptoss", 32, graph=True),
        # one prefill chunk of the usual chunked-prefill size
        _case("chunk_mx_t2048", "layer", "gptoss", 2048),
        # the largest prompt batch
        _case("prefill_mx_t16384", "layer", "gptoss", 16384),
        # decode with 16-bit activations
        _case("decode_w4a16_t16", "layer", "qwen3", 16, graph=True),
        # a prompt batch with 16-bit activations
        _case("prefill_w4a16_t4096", "layer", "qwen3", 4096),
        # one rank's share of the same layer under 4-way tensor parallelism, a ragged batch
        _case("shard_w4a16_i384_t777", "layer", "qwen3", 777, inter=384),
        # the whole block from hidden states on, called without a graph at a small batch
        _case("sparse_mx_t8", "sparse", "gptoss", 8),
        # gate projection and selection of a prompt batch
        _case("route_t4096", "route", "dsv3", 4096),
    ]


def draw(rng):
    op = rng.choice(["layer"] * 8 + ["sparse", "route"])
    family = rng.choice(["dsv3", "mixtral", "qwen3", "gptoss"])
    most = FAMILIES[family]["max_tokens"]
    if op == "sparse":
        most = 64
    tokens = min(most, max(1, int(round(math.exp(rng.uniform(0.0, math.log(most)))))))
    shape = FAMILIES[family]
    # neighbouring models: hidden sizes down to two thirds, intermediate sizes down to a tensor-parallel share
    hidden = 64 * rng.randint(shape["hidden"] * 2 // 3 // 64, shape["hidden"] // 64)
    inter = shape["inter"] // rng.choice([1, 1, 2, 4])
    inter = max(192, 64 * rng.randint(inter * 3 // 4 // 64, inter // 64))
    graph = op == "layer" and tokens <= 256 and rng.random() < 0.75
    return _case(None, op, family, tokens, graph=graph, hidden=hidden, inter=inter)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _fp4_index(a):
    """Magnitudes -> index into (0, .5, 1, 1.5, 2, 3, 4, 6), round to nearest, ties to the even code."""
    q = torch.zeros_like(a, dtype=torch.uint8)
    for edge, closed in ((0.25, False), (0.75, True), (1.25, False), (1.75, True), (2.5, False), (3.5, True), (5.0, False)):
        q += (a >= edge) if closed else (a > edge)
    return q


def _fp4_pack(x):
    code = _fp4_index(x.abs())
    code |= ((x < 0) & (code > 0)).to(torch.uint8) << 3
    return code[..., 0::2] | (code[..., 1::2] << 4)


def _quantised_rows(gen, rows, cols, mx):
    """Rows of N(0, 0.02) weights -> (codes [rows, cols/2], plain block-scale bytes, global scale)."""
    w = torch.randn(rows, cols, generator=gen, device=gen.device) * 0.02
    if mx:
        blocks = w.view(rows, cols // 32, 32)
        exponent = torch.ceil(torch.log2(blocks.abs().amax(-1, keepdim=True) / 6.0)).clamp(-127, 127)
        codes = _fp4_pack((blocks / torch.exp2(exponent)).view(rows, cols))
        return codes, (exponent + 127).to(torch.uint8).squeeze(-1), 1.0
    g = 448.0 * 6.0 / float(w.abs().amax())
    blocks = w.view(rows, cols // 16, 16)
    sf = (g * blocks.abs().amax(-1, keepdim=True) / 6.0).to(torch.float8_e4m3fn)
    codes = _fp4_pack((blocks * (g / sf.float())).view(rows, cols))
    return codes, sf.view(torch.uint8).squeeze(-1), 1.0 / g


def _expert_weights(gen, experts, rows, cols, mx):
    """[experts, rows, cols/2] codes and plain block scales: every row drawn from a pool of quantised rows."""
    pool = min(4096, experts * rows)
    codes, sf, g = _quantised_rows(gen, pool, cols, mx)
    idx = torch.randint(pool, (experts * rows,), generator=gen, device=gen.device)
    w = codes.index_select(0, idx).view(experts, rows, cols // 2)
    s = sf.index_select(0, idx).view(experts, rows, -1)
    return w, s, g


def _inputs(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    t, k, i, e = case["tokens"], case["hidden"], case["inter"], case["experts"]
    d = {"x": torch.randn(t, k, generator=gen, device=dev).to(torch.bfloat16)}
    if case["op"] == "layer":
        logits = torch.randn(t, e, generator=gen, device=dev)
        if case["zipf"] > 0:
            # the logit bias under which the top-2 loads of eight experts fall about as rank ** -zipf
            logits += 0.9 * torch.arange(1, e + 1, device=dev).float().pow(-case["zipf"]).log()
        d["logits"] = logits
    else:
        d["gate"] = (torch.randn(e, k, generator=gen, device=dev) * 0.02).to(torch.bfloat16)
        d["gate_bias"] = torch.randn(e, generator=gen, device=dev).to(torch.bfloat16) * 0.1
        d["selection_bias"] = torch.randn(e, generator=gen, device=dev) * 0.02
    if case["op"] == "route":
        return d
    mx = case["recipe"] == "w4a8_mx"
    spread = lambda: torch.rand(e, generator=gen, device=dev) * 0.2 + 0.9
    d["w1"], d["s1"], g1 = _expert_weights(gen, e, 2 * i, k, mx)
    d["w2"], d["s2"], g2 = _expert_weights(gen, e, k, i, mx)
    d["g1"], d["g2"] = g1 * spread(), g2 * spread()
    # reciprocal input scales 448 * 6 / amax, amax as a calibration run would see it
    d["a1"] = 448.0 * 6.0 / (5.0 * spread())
    d["a2"] = 448.0 * 6.0 / ((4.0 * 0.02 * math.sqrt(k)) ** 2 * spread())
    return d


def _swizzled(grid):
    """[E, rows, cols] block-scale bytes -> the checkpoint's 128x4-swizzled storage."""
    e, rows, cols = grid.shape
    rp, cp = (rows + 127) // 128 * 128, (cols + 3) // 4 * 4
    padded = torch.zeros((e, rp, cp), dtype=torch.uint8, device=grid.device)
    padded[:, :rows, :cols] = grid
    return padded.view(e, rp // 128, 4, 32, cp // 4, 4).permute(0, 1, 4, 3, 2, 5).contiguous().view(e, rp, cp)


def _experts(case, d):
    wp = fused_moe.plan_weights(
        quant_modes=case["recipe"], source_format=SOURCE[case["recipe"]], activation=ACT_API[case["activation"]],
        params_dtype=torch.bfloat16, num_experts=case["experts"], hidden_size=case["hidden"],
        intermediate_size=case["inter"])
    kw = dict(plan=wp, params_dtype=torch.bfloat16, w1_fp4=d["w1"], w2_fp4=d["w2"])
    if case["recipe"] == "w4a8_mx":
        kw.update(w1_blockscale=d["s1"], w2_blockscale=d["s2"])
    else:
        kw.update(w1_blockscale=_swizzled(d["s1"]), w2_blockscale=_swizzled(d["s2"]), w1_global_scale=d["g1"],
                  w2_global_scale=d["g2"])
    if case["recipe"] == "nvfp4":
        kw.update(a1_gscale=d["a1"], a2_gscale=d["a2"])
    return fused_moe.prepare_weights(**kw)


def prepare(case, seed):
    d = _inputs(case, seed)
    dev, t, k = d["x"].device, case["tokens"], case["topk"]
    state = {"case": case, "x": d["x"]}
    if case["op"] == "layer":
        state["logits"] = d["logits"]
        state["topk"] = (torch.empty(t, k, device=dev), torch.empty(t, k, dtype=torch.int32, device=dev),
                         torch.empty(t, k, device=dev))
    else:
        state.update(gate=d["gate"], gate_bias=d["gate_bias"], selection_bias=d["selection_bias"])
    if case["op"] == "route":
        return state
    state["experts"] = ex = _experts(case, d)
    del d
    caps = fused_moe.Caps(max_tokens=t, num_topk=k, device=dev, weight_plan=ex.plan, quant_mode=case["recipe"],
                          route_num_experts=case["experts"] if case["op"] == "sparse" else None)
    state["workspace"] = fused_moe.Workspace.allocate(fused_moe.plan(caps))
    state["out"] = torch.empty(t, case["hidden"], dtype=torch.bfloat16, device=dev)
    if case["graph"]:
        _layer(state)                       # eager once, as every program does before it captures
        torch.cuda.synchronize()
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            _layer(state)
    return state


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _layer(state):
    case, (tl, ti, tw) = state["case"], state["topk"]
    if case["router"] == "sigmoid":
        fused_moe.route_topk(state["logits"], tl, ti, tw, renormalize=True, score_func="sigmoid",
                             route_scale=case["route_scale"])
    else:
        fused_moe.route_topk(state["logits"], tl, ti, tw, renormalize=True)
    ws = state["workspace"]
    binding = fused_moe.bind(ws.plan, scratch=ws.storage, a=state["x"], experts=state["experts"], topk_weights=tw,
                             topk_ids=ti, output=state["out"])
    return fused_moe.run(binding=binding)


def run(state):
    case = state["case"]
    if case["op"] == "layer":
        if case["graph"]:
            state["graph"].replay()
            out = state["out"]
        else:
            out = _layer(state)
        return {"out": out, "topk_ids": state["topk"][1], "topk_weights": state["topk"][2]}
    if case["op"] == "sparse":
        out, routing = fused_moe.run_sparse(binding=fused_moe.bind_sparse(
            scratch=state["workspace"], hidden_states=state["x"], experts=state["experts"], top_k=case["topk"],
            gate_weight=state["gate"], gate_bias=state["gate_bias"], output=state["out"], return_routing=True,
            **_scoring(case, state)))
        return {"out": out, "logits": routing.router_logits, "topk_ids": routing.topk_ids,
                "topk_weights": routing.topk_weights}
    routing = fused_moe.route(binding=fused_moe.bind_route(
        hidden_states=state["x"], top_k=case["topk"], gate_weight=state["gate"], gate_bias=state["gate_bias"],
        **_scoring(case, state)))
    return {"logits": routing.router_logits, "topk_ids": routing.topk_ids, "topk_weights": routing.topk_weights}


def _scoring(case, state):
    if case["router"] == "sigmoid":
        return dict(score_func="sigmoid", selection_bias=state["selection_bias"], route_scale=case["route_scale"])
    return {}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without, and how far another correct one may be off
# ---------------------------------------------------------------------------------------------
def work(case):
    t, k, i, e, top = case["tokens"], case["hidden"], case["inter"], case["experts"], case["topk"]
    nbytes, flops = t * k * 2 + t * top * 8, 0
    if case["op"] == "layer":
        nbytes += t * e * 4
    else:
        nbytes += e * k * 2 + t * e * 2
        flops += 2 * t * e * k
    if case["op"] != "route":
        # experts that receive rows when tokens pick `top` of `e` independently
        active = e * (1.0 - (1.0 - top / e) ** t)
        group = 32 if case["recipe"] == "w4a8_mx" else 16
        nbytes += active * 3 * k * i * (0.5 + 1.0 / group) + t * k * 2
        flops += t * top * 6 * k * i
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Measured against :func:`exact`: a layer's outputs are 1.7e-3 off (one bf16 rounding); behind a gate projection,
    whose logits are rounded to bf16 before the selection, weights and outputs are up to 7e-3 off.  Selections are
    compared as whole values: where two bf16 logits tie or nearly tie, another order of the sums may swap them."""
    if case["op"] == "layer":
        return {"rel": 7e-3}
    return {"rel": 2.5e-2, "differ": 0.002}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
_FP4 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _dequantised(codes, sf, mx):
    lut = torch.tensor(_FP4, dtype=torch.float64, device=codes.device)
    v = torch.stack([lut[(codes & 15).long()], lut[(codes >> 4).long()]], dim=-1).view(codes.shape[0], -1)
    s = torch.exp2(sf.double() - 127.0) if mx else sf.view(torch.float8_e4m3fn).double()
    g = 32 if mx else 16
    return (v.view(v.shape[0], -1, g) * s.unsqueeze(-1)).view(v.shape[0], -1)


def _nvfp4_values(x, gs):
    """The values NVFP4 quantisation with reciprocal scale ``gs`` leaves of ``x`` (the format's own fp32 rule), times gs."""
    r, c = x.shape
    b = x.float().view(r, c // 16, 16)
    sf = (b.abs().amax(-1, keepdim=True) * gs / 6.0).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    scaled = b / (sf / gs).clamp(min=1e-30)
    mag = torch.tensor(_FP4[:8], dtype=torch.float64, device=x.device)[_fp4_index(scaled.abs()).long()]
    return (mag * torch.sign(scaled).double() * sf.double()).view(r, c)


def _mxfp8_values(x):
    r, c = x.shape
    b = x.float().view(r, c // 32, 32)
    need = b.abs().amax(-1, keepdim=True) * (1.0 / 448.0)
    mant, exp = torch.frexp(need)                      # need = mant * 2^exp, mant in [0.5, 1)
    scale = torch.exp2((exp - (mant == 0.5).int()).float())
    scale = torch.where(need > 0, scale, torch.ones_like(scale))
    return ((b / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double() * scale.double()).view(r, c)


def _selection(case, logits, bias):
    """Top-k in slot order and the weights, ties to the larger expert index."""
    lg = logits.float()
    score = torch.sigmoid(lg) if case["router"] == "sigmoid" else lg
    select = score + bias if bias is not None else score
    ids = torch.sort(select.flip(1), dim=1, descending=True, stable=True).indices[:, : case["topk"]]
    ids = lg.shape[1] - 1 - ids
    v = logits.double().gather(1, ids)
    if case["router"] == "sigmoid":
        w = torch.sigmoid(v)
        w = w / w.sum(1, keepdim=True) * case["route_scale"]
    else:
        w = torch.softmax(v, dim=1)
    return ids, w


def exact(case, seed):
    d = _inputs(case, seed)
    x = d["x"]
    res = {}
    if case["op"] == "layer":
        ids, w = _selection(case, d["logits"], None)
    else:
        full = x.double() @ d["gate"].double().T + d["gate_bias"].double()
        res["logits"] = full
        ids, w = _selection(case, full.to(torch.bfloat16), d["selection_bias"] if case["router"] == "sigmoid" else None)
    res.update(topk_ids=ids.int(), topk_weights=w)
    if case["op"] == "route":
        return res
    i, mx, recipe = case["inter"], case["recipe"] == "w4a8_mx", case["recipe"]
    out = torch.zeros(x.shape, dtype=torch.float64, device=x.device)
    for e in range(case["experts"]):
        tok, slot = (ids == e).nonzero(as_tuple=True)
        if tok.numel() == 0:
            continue
        a = x[tok]
        al1 = al2 = 1.0
        if recipe == "nvfp4":
            al1, al2 = (d["g1"][e].double() / d["a1"][e].double()), (d["g2"][e].double() / d["a2"][e].double())
            a = _nvfp4_values(a, d["a1"][e])
        elif mx:
            a = _mxfp8_values(a)
        else:
            al1, al2 = d["g1"][e].double(), d["g2"][e].double()
            a = a.double()
        f = (a @ _dequantised(d["w1"][e], d["s1"][e], mx).T) * al1
        if case["activation"] == "swigluoai":            # gate rows first, clamped at 7
            gate, up = f[:, :i].clamp(max=7.0), f[:, i:].clamp(-7.0, 7.0)
            h = gate * torch.sigmoid(1.702 * gate) * (up + 1.0)
        else:
            up, gate = f[:, :i], f[:, i:]
            h = gate * torch.sigmoid(gate) * up
        if recipe == "nvfp4":
            h = _nvfp4_values(h.to(torch.bfloat16), d["a2"][e])
        elif mx:
            h = _mxfp8_values(h)
        else:
            h = h.to(torch.bfloat16).double()
        y = (h @ _dequantised(d["w2"][e], d["s2"][e], mx).T) * al2
        out.index_add_(0, tok, y * w[tok, slot].unsqueeze(1))
    res["out"] = out
    return res
