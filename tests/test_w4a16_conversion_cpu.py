"""CPU checks of the arithmetic claims behind the W4A16 kernels (csrc/grouped_gemm_w4a16.cu).  For every E2M1
code and every finite E4M3 block scale the product is exactly representable in FP16 and in BF16, so "convert
to FP16, multiply in FP16" (and "re-encode as BF16") equals the oracle's "dequantise, hold in BF16"
(tests/_reference/w4a16_reference.py:288-338 of the reference).  And the rule by which a row of BF16 values
may go into the MMA as FP16 times a power of two loses no bit of it."""

import torch

from oracle import moe_oracle


def _all_scales():
    b = torch.arange(256, dtype=torch.uint8)
    s = b.view(torch.float8_e4m3fn).float()
    return s[torch.isfinite(s)]


def test_code_times_e4m3_scale_is_exact_in_fp16_and_bf16():
    codes = moe_oracle.fp4_lut()                                           # 16 entries, sign in bit 3
    assert codes.numel() == 16 and torch.equal(codes[:8], torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]))
    assert torch.equal(codes[8:], -codes[:8])
    prod = codes[:, None].double() * _all_scales()[None, :].double()       # exact in f64
    assert torch.equal(prod.half().double(), prod), "FP16 would round a product"
    assert torch.equal(prod.bfloat16().double(), prod), "BF16 would round a product"
    nz = prod[prod != 0].abs()
    assert nz.min().item() >= 2.0 ** -14 and nz.max().item() <= 65504.0     # normal FP16 range
    # the FP16 multiply of the two FP16 factors gives the same value
    got = codes[:, None].half() * _all_scales()[None, :].half()
    assert torch.equal(got.double(), prod)


def test_rows_that_pass_the_rule_are_exact_in_fp16():
    """Exhaustive: every exponent of a row's largest magnitude x every magnitude not above it.  ``sh`` and the rule
    restate permute_rows_f16_kernel."""
    mag = torch.arange(1, 0x7F80, dtype=torch.int32)                        # nonzero finite magnitudes
    x = mag.to(torch.int16).view(torch.bfloat16).double()
    field = (mag >> 7).clamp(min=1)
    loses_outside = 0
    for top in range(1, 255):                                               # exponent field (subnormal maxima: 1)
        sh = min(142 - top, 126)
        row = field <= top
        scaled = x[row] * 2.0 ** sh
        exact = scaled.float().half().double() == scaled                    # the kernel multiplies in fp32
        ok = field[row] + sh >= 110
        assert bool(exact[ok].all()) and scaled.abs().max() <= 65504.0
        loses_outside += int((~exact[~ok]).sum())
        assert int(field[row][ok].min()) == max(1, top - 32)
    assert loses_outside > 0
