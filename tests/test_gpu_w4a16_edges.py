"""-m gpu: the W4A16 kernels at the edges of their token tiles (16-column steps on one CTA, at most 64; 32-column
steps on a CTA pair, at most 64 or 160), of their stages (two and four k-blocks of 64) and of their weight tiles, and the
per-row power-of-two scaling of the FP16 token rows over the range of BF16."""

import ctypes as C
import os
import subprocess
import sys
from dataclasses import replace
from pathlib import Path

import pytest
import torch

from b12x_b200 import synth
from b12x_b200._lib import ext
from tests.gpu_utils import oracle_layer, run_layer
from tests.test_gpu_parity import _check_w4a16_layer, _w16

pytestmark = pytest.mark.gpu


def _one_expert(tokens, experts, hidden, inter, act="silu"):
    """Every token on one expert of ``experts``: the plan's average decides the kernel, the expert's rows the tiles."""
    shp = _w16(tokens=tokens, experts=experts, topk=1, hidden=hidden, intermediate=inter, activation=act)
    ids = torch.full((tokens, 1), experts // 2, dtype=torch.int32)
    return synth.make_inputs(shp, seed=tokens + hidden), ids, torch.full((tokens, 1), 0.75)


@pytest.mark.parametrize("tokens", [1, 15, 16, 17, 32, 33, 63, 64, 65, 127, 130])
@pytest.mark.parametrize("hidden,inter", [(64, 64), (320, 192)])      # one k-block; five and three
def test_single_cta_token_tiles(tokens, hidden, inter):
    inp, ids, w = _one_expert(tokens, 16, hidden, inter)
    _check_w4a16_layer(run_layer(inp, topk_ids=ids, topk_weights=w))


@pytest.mark.parametrize("tokens", [18, 32, 33, 57, 80, 115, 128, 150])
@pytest.mark.parametrize("hidden,inter", [(64, 64), (320, 192), (256, 128)])
def test_narrow_pair_token_tiles(tokens, hidden, inter):
    """Plans of 18 to 57 rows per expert (four experts above that many rows, all on one of them)."""
    inp, ids, w = _one_expert(tokens, 1 if tokens < 58 else 4, hidden, inter)
    _check_w4a16_layer(run_layer(inp, topk_ids=ids, topk_weights=w))


@pytest.mark.parametrize("tokens", [58, 160, 161, 320, 321, 500])
@pytest.mark.parametrize("hidden,inter,act", [(64, 64, "silu"), (448, 320, "silu"), (192, 192, "relu2")])
def test_cta_pair_token_tiles(tokens, hidden, inter, act):
    inp, ids, w = _one_expert(tokens, 1, hidden, inter, act)
    _check_w4a16_layer(run_layer(inp, topk_ids=ids, topk_weights=w))


def test_more_work_items_than_a_cta_lists_ahead():
    """1024 experts x 40 weight tiles: more than 256 items on each of 148 SMs."""
    shp = _w16(tokens=1024, experts=1024, topk=1, hidden=64, intermediate=2560)
    ids = torch.randperm(1024, generator=torch.Generator().manual_seed(1)).to(torch.int32).reshape(-1, 1)
    _check_w4a16_layer(run_layer(synth.make_inputs(shp, seed=3), topk_ids=ids, topk_weights=torch.ones(1024, 1)))


def test_row_scaling_over_the_bf16_range():
    shp = _w16(tokens=48, experts=2, topk=1, hidden=256, intermediate=128)
    inp = synth.make_inputs(shp, seed=8)
    gen = torch.Generator().manual_seed(9)
    x = inp.x.float()
    x[8:16] *= 2.0 ** 50
    x[16:24] *= 2.0 ** -40
    x[24:32] *= torch.exp2(torch.randint(-24, 1, (8, 256), generator=gen).float())   # a row over 24 binades
    x[32] = 0.0
    x[33, 1:] = 0.0
    inp = replace(inp, x=x.to(torch.bfloat16))
    ids = (torch.arange(48) % 2).to(torch.int32).reshape(-1, 1)
    w = torch.ones(48, 1)
    run = run_layer(inp, topk_ids=ids, topk_weights=w)
    _, taps = oracle_layer(inp, ids, w)
    # row by row, since their sizes lie 2^180 apart: 1e-2 x the row's RMS
    err = (run.out_f32 - taps.out_f32).abs().amax(dim=1)
    rms = taps.out_f32.double().square().mean(dim=1).sqrt().float()
    assert bool((err <= 1e-2 * rms).all()), (err / rms.clamp(min=1e-38)).max()
    # an infinity or a NaN stays in its own row
    bad = x.clone()
    bad[5, 7], bad[40, 3] = float("inf"), float("nan")
    again = run_layer(replace(inp, x=bad.to(torch.bfloat16)), topk_ids=ids, topk_weights=w)
    keep = [i for i in range(48) if i not in (5, 40)]
    assert torch.equal(again.out_f32[keep], run.out_f32[keep])
    assert not bool(torch.isfinite(again.out_f32[5]).any()) and bool(torch.isnan(again.out_f32[40]).all())


@pytest.mark.parametrize("tokens,hidden,inter", [(40, 256, 128), (150, 192, 448)])      # wider and narrower than I
def test_token_rows_are_readable_after_a_run(tokens, hidden, inter):
    """``packed_input`` holds the sorted BF16 rows after the whole layer, and the calibration maxima taken after FC2
    equal those of the BF16 rows; there are no activation scales to read."""
    shp = _w16(tokens=tokens, experts=5, topk=2, hidden=hidden, intermediate=inter)
    run = run_layer(synth.make_inputs(shp, seed=tokens))
    b, rows = run.binding, tokens * 2
    x = run.inp.x.cpu()[(b.packed_route_indices.cpu() // 2).long()]
    assert torch.equal(b.packed_input.cpu()[:rows].view(torch.bfloat16), x)
    assert b.packed_input_scale.numel() == 0 and b.intermediate_scale.numel() == 0
    amax = torch.zeros(1, 5, 2, device="cuda")
    args = ext.AmaxArgs(b.kernel_workspace.data_ptr(), C.pointer(b.core_layout), amax.data_ptr(), rows, 5, hidden, inter, 0,
                        ext.RECIPES["w4a16"])
    ext.check(ext.load().b200moe_activation_amax(C.byref(args), torch.cuda.current_stream().cuda_stream), "amax")
    mid = b.materialized_intermediate.cpu()[:rows].view(torch.bfloat16).float()
    offs = b.expert_offsets.cpu().tolist()
    for e in range(5):
        for which, v in enumerate((x.float(), mid)):
            part = v[offs[e]:offs[e + 1]].abs()
            assert amax[0, e, which].item() == (part.max().item() if part.numel() else 0.0)


def _rowwise(got, ref, tol):
    """Row by row, since the rows' sizes lie far apart: max-abs error <= tol x the row's RMS."""
    err = (got - ref).abs().amax(dim=1)
    rms = ref.double().square().mean(dim=1).sqrt().float()
    assert bool((rms > 0).all()) and bool((err <= tol * rms).all()), (err / rms).max()


@pytest.mark.parametrize("tokens,experts,act", [(40, 4, "silu"), (40, 2, "silu"), (140, 2, "silu"), (40, 4, "relu2"),
                                                (140, 2, "relu2")])
def test_rows_wider_than_fp16(tokens, experts, act):
    """Rows whose largest element lies 20 to 60 binades above the others and meets a zero weight, so that the small
    elements are the whole sum: up to 32 binades on FP16 operands (expert 0), beyond on BF16 operands."""
    shp = _w16(tokens=tokens, experts=experts, topk=1, hidden=320, intermediate=192, activation=act)
    inp = synth.make_inputs(shp, seed=tokens)
    gap = 20 + torch.arange(tokens) * 41 // tokens
    gen = torch.Generator().manual_seed(3)
    x = (torch.rand(tokens, 320, generator=gen) * 1.5 + 0.5) * (torch.randint(0, 2, (tokens, 320), generator=gen) * 2 - 1)
    x *= torch.exp2(17.0 - gap)[:, None]
    x[:, 0] = 2.0 ** 17                                 # 2 ** (gap + 1) above the smallest
    w1 = inp.w1_fp4.clone()
    w1[..., 0] &= 0xF0                                  # the weights of element 0
    inp = replace(inp, x=x.to(torch.bfloat16), w1_fp4=w1)
    ids = (gap > 30).to(torch.int32).reshape(-1, 1)
    run = run_layer(inp, topk_ids=ids, topk_weights=torch.ones(tokens, 1))
    _, taps = oracle_layer(inp, ids, torch.ones(tokens, 1))
    _rowwise(run.fc1[:tokens], taps.fc1, 1e-4)          # fp32 sums of 320 terms in another order


def test_one_row_wider_than_fp16_among_others():
    """One row of one of two experts puts that expert on BF16 operands: the other rows keep their bits."""
    shp = _w16(tokens=400, experts=2, topk=1, hidden=320, intermediate=192)
    inp = synth.make_inputs(shp, seed=2)
    w1 = inp.w1_fp4.clone()
    w1[..., 0] &= 0xF0
    x = inp.x.float().cpu()
    ids, w = (torch.arange(400) >= 100).to(torch.int32).reshape(-1, 1), torch.ones(400, 1)
    plain = run_layer(replace(inp, w1_fp4=w1), topk_ids=ids, topk_weights=w)
    x[200] = 2.0 ** -36
    x[200, 0] = 16.0
    run = run_layer(replace(inp, x=x.to(torch.bfloat16), w1_fp4=w1), topk_ids=ids, topk_weights=w)
    keep = [i for i in range(400) if i != 200]
    assert torch.equal(run.fc1[keep], plain.fc1[keep]) and torch.equal(run.out_f32[keep], plain.out_f32[keep])
    _, taps = oracle_layer(run.inp, ids, w)
    _rowwise(run.fc1[200:201], taps.fc1[200:201], 1e-4)


@pytest.mark.parametrize("tokens,experts", [(30, 4), (40, 2), (140, 2)])
def test_intermediate_rows_wider_than_fp16(tokens, experts):
    """The same for FC2: 16 intermediate columns 2 ** 36 above the others, with zero weights in FC2."""
    shp = _w16(tokens=tokens, experts=experts, topk=1, hidden=64, intermediate=192)
    inp = synth.make_inputs(shp, seed=tokens)
    gen = torch.Generator().manual_seed(4)
    x = (torch.rand(tokens, 64, generator=gen) * 0.5 + 0.5).to(torch.bfloat16)
    codes = torch.randint(1, 8, (experts, 384, 64), generator=gen).to(torch.uint8)          # positive weights
    scale = torch.full((384, 4), 0x01, dtype=torch.uint8)                                   # 2 ** -9 ...
    scale[:16] = scale[192:208] = 0x7E                                                      # ... and 448
    w2 = inp.w2_fp4.clone()
    w2[..., :8] = 0
    inp = replace(inp, x=x, w1_fp4=codes[..., 0::2] | codes[..., 1::2] << 4, w2_fp4=w2,
                  w1_blockscale=synth.swizzle_block_scale(scale).expand(experts, -1, -1).contiguous().view(inp.w1_blockscale.dtype),
                  w1_global_scale=torch.ones_like(inp.w1_global_scale))
    ids = torch.ones(tokens, 1, dtype=torch.int32)
    run = run_layer(inp, topk_ids=ids, topk_weights=torch.ones(tokens, 1))
    _, taps = oracle_layer(inp, ids, torch.ones(tokens, 1))
    mid = taps.mid.abs()
    assert (mid.amax(dim=1) / mid.amin(dim=1)).min() > 2.0 ** 34
    _rowwise(run.out_f32, taps.out_f32, 1e-2)           # BF16 roundings of the intermediate that fall the other way


@pytest.mark.parametrize("tokens,planned", [(20, 1200), (60, 1200), (200, 1200)])    # 10, 30 and 100 rows per expert
def test_small_calls_through_a_large_plan(tokens, planned):
    """The call's rows choose the form; the plan's capacity does not change a bit of the result."""
    inp = synth.make_inputs(_w16(tokens=tokens, experts=2, topk=1, hidden=320, intermediate=192), seed=tokens)
    run = run_layer(inp, max_tokens=planned)
    _check_w4a16_layer(run)
    assert torch.equal(run.out_f32, run_layer(inp).out_f32)


@pytest.mark.timeout(300)
def test_grid_of_one_cta():
    """A persistent grid limited to one CTA cannot hold a pair: batches of every size run on the one-CTA form."""
    if os.environ.get("B200MOE_NUM_SMS"):
        pytest.skip("already the child run")
    here = Path(__file__).resolve()
    r = subprocess.run([sys.executable, "-m", "pytest", str(here), "-m", "gpu", "-q", "-p", "no:cacheprovider",
                        "-k", "narrow_pair_token_tiles or cta_pair_token_tiles"],
                       env=dict(os.environ, B200MOE_NUM_SMS="1"), capture_output=True, text=True, timeout=280,
                       cwd=str(here.parent.parent))
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
