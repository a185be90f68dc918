"""The fused SiLU-mul quantiser against the separate activation kernel, which divides with the IEEE routine."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("group_size", [128, 16])
def test_every_gate_value_has_the_bits_of_the_division(dtype, group_size):
    from sglang_b200._lib import check, dtype_code, lib
    from sglang_b200.sgl_kernel import silu_and_mul

    rows, hidden = 1024 + 3, 128  # two rounds over all 65536 gates, and a last block that is not full
    gate = torch.arange(rows * hidden, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype).view(rows, hidden)
    torch.manual_seed(0)
    up = torch.randn(rows, hidden, device="cuda").to(dtype)
    up[:512] = 1
    x = torch.cat([gate, up], dim=1).contiguous()
    want = silu_and_mul(x)
    act = torch.empty_like(want)
    codes = torch.empty(rows, hidden, dtype=torch.uint8, device="cuda")
    scales = torch.empty(rows, hidden // group_size, device="cuda")
    check(lib().sglb200_silu_mul_group_quant_fp8(
        x.data_ptr(), dtype_code(dtype), codes.data_ptr(), scales.data_ptr(), act.data_ptr(), rows, hidden, group_size, 1e-10,
        -448.0, 448.0, 0, hidden // group_size, 1, torch.cuda.current_stream().cuda_stream), "silu_mul_group_quant_fp8")
    assert torch.equal(act.isnan(), want.isnan())
    keep = ~want.isnan()
    assert torch.equal(act.view(torch.int16)[keep], want.view(torch.int16)[keep])
    plain = torch.empty_like(codes)
    plain_s = torch.empty_like(scales)
    check(lib().sglb200_per_token_group_quant_fp8(
        want.data_ptr(), dtype_code(dtype), plain.data_ptr(), plain_s.data_ptr(), rows, hidden, group_size, 1e-10, -448.0, 448.0,
        0, hidden // group_size, 1, torch.cuda.current_stream().cuda_stream), "per_token_group_quant_fp8")
    assert torch.equal(codes[keep], plain[keep]) and torch.equal(scales.view(torch.int32), plain_s.view(torch.int32))
