"""-m gpu: the w4a8_mx small-batch kernel at the edges of its token tiles (multiples of 16 up to 80 columns, then
tiles of 64 = halves of the plan's 128-row tiles), and the left-over row tiles of CTA-pair plans on both sides of
the 80 rows that decide which kernel takes them."""

import pytest
import torch

from b12x_b200 import synth
from oracle import moe_oracle as O
from tests.gpu_utils import run_layer
from tests.helpers import atoms_to_rows
from tests.test_gpu_parity import FLIP_TOL, _check_mx_layer, _mx

pytestmark = pytest.mark.gpu


def _run(tokens, experts, hidden, inter, act):
    """Every token on one expert: the plan's average decides the kernel, the expert's rows the tiles."""
    shp = _mx(tokens=tokens, experts=experts, topk=1, hidden=hidden, intermediate=inter, activation=act)
    ids = torch.full((tokens, 1), experts - 1, dtype=torch.int32)
    _check_mx_layer(run_layer(synth.make_inputs(shp, seed=tokens + inter), topk_ids=ids, topk_weights=torch.ones(tokens, 1)))


@pytest.mark.parametrize("tokens", [1, 15, 17, 32, 33, 48, 63, 65, 79, 80, 81, 128, 129, 192, 200])
@pytest.mark.parametrize("hidden,inter,act", [
    (320, 192, "swigluoai"),      # half a k-block and half a weight tile left over
    (128, 64, "silu"),            # one k-block, one half weight tile
])
def test_token_tiles(tokens, hidden, inter, act):
    _run(tokens, 4, hidden, inter, act)


@pytest.mark.parametrize("tokens", [257, 300, 335, 336, 337, 384, 600, 640])
def test_left_over_row_tiles(tokens):
    _run(tokens, 1, 256, 192, "swigluoai")


@pytest.mark.parametrize("tokens,planned", [(24, 1200), (300, 1200), (560, 1200)])   # 12, 150 and 280 rows per expert
def test_small_calls_through_a_large_plan(tokens, planned):
    """The call's rows choose the kernel; the plan's capacity does not change a bit of the result."""
    shp = _mx(tokens=tokens, experts=2, topk=1, hidden=320, intermediate=192, activation="swigluoai")
    inp = synth.make_inputs(shp, seed=tokens)
    run = run_layer(inp, max_tokens=planned)
    _check_mx_layer(run)
    assert torch.equal(run.out_f32, run_layer(inp).out_f32)


@pytest.mark.parametrize("tokens", [17, 80, 150])
@pytest.mark.parametrize("limit,act", [(0.5, "silu"), (None, "situ")])
def test_other_gated_epilogues(tokens, limit, act):
    """SwiGLU with a clamp that cuts many values, and SiTU: FC1's stored MXFP8 rows against the tap's activation."""
    shp = _mx(tokens=tokens, experts=4, topk=1, hidden=320, intermediate=192, activation=act)
    inp = synth.make_inputs(shp, seed=tokens)
    run = run_layer(inp, topk_ids=torch.full((tokens, 1), 2, dtype=torch.int32), topk_weights=torch.ones(tokens, 1),
                    swiglu_limit=limit)
    b = run.binding
    f = run.fc1[:tokens]
    if limit is not None:
        assert float((f.abs() > limit).float().mean()) > 0.05
    codes, scales, _ = O.quantize_mxfp8_rows(O.gated_activation(f[:, 192:], f[:, :192], act, limit, 1.0, 0.0))
    # the kernel's exponential and reciprocal are an ulp or two off torch's: codes at a rounding boundary may flip
    assert float((b.materialized_intermediate.cpu()[:tokens] != codes).float().mean()) <= FLIP_TOL
    sf = b.intermediate_scale.cpu()
    for mt in range((tokens + 127) // 128):
        rows = slice(128 * mt, min(tokens, 128 * mt + 128))
        assert torch.equal(atoms_to_rows(sf, mt, 2, rows.stop - rows.start, 6), scales[rows])
