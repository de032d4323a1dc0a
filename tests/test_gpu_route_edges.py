"""-m gpu: the router at the edges of its per-lane tables (1 .. 32 values a lane), on masked, tied and NaN
logits, and the split gate kernel at the edges of its split rule."""

import pytest
import torch

from b12x_b200.moe import fused_moe
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _route(lg, k, **kw):
    n = lg.shape[0]
    tl, tw = torch.empty(n, k, device=DEV), torch.empty(n, k, device=DEV)
    ti = torch.empty(n, k, dtype=torch.int32, device=DEV)
    fused_moe.route_topk(lg.to(DEV), tl, ti, tw, renormalize=True, **kw)
    return tl.cpu(), ti.cpu(), tw.cpu()


@pytest.mark.parametrize("experts,topk", [(1, 1), (31, 31), (32, 32), (33, 5), (64, 8), (65, 8), (128, 4), (129, 32),
                                          (256, 8), (257, 8), (512, 6), (513, 6), (1024, 32)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_tables_match_the_oracle(experts, topk, dtype):
    gen = torch.Generator().manual_seed(experts + topk)
    lg = torch.randn(9, experts, generator=gen)
    lg[1] = 0.0                                   # every expert ties
    lg[2, ::2] = -0.0                             # signed zeros are one value
    lg[2, 1::2] = 0.0
    lg[3] = torch.finfo(torch.bfloat16).min       # masked with the type's lowest value ...
    lg[3, experts // 2] = 1.0
    lg[4] = float("-inf")                         # ... and with -infinity, fewer finite values than slots
    lg[4, experts // 3] = -2.0
    lg[5] = lg[5].round()                         # many ties
    lg[6, 0] = float("inf")
    lg = lg.to(dtype)
    tl, ids, w = _route(lg, topk)
    rl, rids, rw = O.route_topk(lg.float(), topk)
    assert torch.equal(ids, rids)
    keep = [0, 1, 2, 3, 4, 5, 7, 8]               # row 6: inf - inf
    assert torch.equal(tl[keep], rl[keep])
    torch.testing.assert_close(w[keep], rw[keep], rtol=2e-6, atol=1e-7)   # one expf and one sum of <= 32 terms
    bias = torch.randn(experts, generator=gen) * 0.1
    _, ids, w = _route(lg[[0, 1, 2, 7, 8]], topk, score_func="sigmoid", selection_bias=bias.to(DEV), route_scale=2.5)
    _, rids, rw = O.route_topk(lg[[0, 1, 2, 7, 8]].float(), topk, mode="sigmoid", bias=bias, route_scale=2.5)
    same = (ids == rids).all(dim=1)               # two sigmoids an ulp apart may swap on the way through the bias
    assert int(same.sum()) >= 4
    torch.testing.assert_close(w[same], rw[same], rtol=4e-6, atol=1e-7)


def test_router_never_selects_nan_before_a_number():
    lg = torch.full((3, 40), float("nan"))
    lg[0, 3:9] = torch.arange(6.0)
    lg[1, 39], lg[1, 0] = float("-inf"), 7.0
    tl, ids, _ = _route(lg, 2)
    assert ids[0].tolist() == [8, 7] and ids[1].tolist() == [0, 39]
    assert ids[2].tolist() == [0, 0] and bool((tl[2] == float("-inf")).all())


@pytest.mark.parametrize("tokens,hidden,experts,topk", [
    (1, 64, 16, 1),          # one k-block: a single part
    (5, 136, 48, 3),         # three k-blocks (the last one ragged): two parts
    (127, 1096, 256, 8),     # eight parts, rows short of a tile
    (2432, 320, 256, 8),     # 19 token tiles: five k-blocks in four uneven parts
    (4737, 128, 32, 2),      # 38 token tiles: two parts
    (9601, 192, 128, 4),     # 76 token tiles: one part
])
def test_split_gate_kernel(tokens, hidden, experts, topk):
    gen = torch.Generator().manual_seed(tokens)
    hs = torch.randn(tokens, hidden, generator=gen).to(torch.bfloat16)
    gw = (torch.randn(experts, hidden, generator=gen) * 0.05).to(torch.bfloat16)
    gb = torch.randn(experts, generator=gen).to(torch.bfloat16)
    r = fused_moe.route(binding=fused_moe.bind_route(hidden_states=hs.to(DEV), top_k=topk, gate_weight=gw.to(DEV),
                                                     gate_bias=gb.to(DEV)))
    prod = torch.nn.functional.linear(hs.float(), gw.float())
    ref = prod + gb.float()
    got = r.router_logits.float().cpu()
    # two bf16 roundings (the product, then the biased sum), half an ulp each of the larger magnitude, and the
    # fp32 sums' error
    ulp = torch.exp2(torch.floor(torch.log2(torch.maximum(prod.abs(), ref.abs()).clamp(min=1e-30))) - 7)
    assert bool(((got - ref).abs() <= 1.02 * ulp + 3e-5 * ref.abs() + 3e-4).all()), (got - ref).abs().max()
    _, ids, w = O.route_topk(got, topk)
    assert torch.equal(r.topk_ids.cpu(), ids)
    torch.testing.assert_close(r.topk_weights.cpu(), w, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("hidden,experts", [(1096, 256), (2048, 32), (320, 64)])     # 18, 32 and 5 k-blocks
def test_logits_do_not_depend_on_the_batch(hidden, experts):
    """K is cut and summed alike for every number of tokens, whatever the number of CTAs that share a tile."""
    gen = torch.Generator().manual_seed(hidden)
    hs = torch.randn(9700, hidden, generator=gen).to(torch.bfloat16).to(DEV)
    gw = (torch.randn(experts, hidden, generator=gen) * 0.05).to(torch.bfloat16).to(DEV)

    def logits(n):
        return fused_moe.route(binding=fused_moe.bind_route(hidden_states=hs[:n], top_k=2, gate_weight=gw,
                                                            gate_kernel="tc")).router_logits

    whole = logits(9700)
    for n in (1, 100, 2304, 2433, 4736, 4737):
        assert torch.equal(logits(n), whole[:n]), n
