"""The one-call expert layer against the same layer put together from the single ops, bit for bit: every shape crosses an edge
of the routing, scatter or combine kernels (one token, slots beyond eight, ids of no expert, a scale word that is not full)."""

import pytest
import torch

import oracle
from helpers import make_activations

pytestmark = pytest.mark.gpu


def _layer(E, H, I, ue8m0, seed):
    g = torch.Generator().manual_seed(seed)
    w1 = [oracle.block_quant_weight(torch.randn(2 * I, H, generator=g) * 0.05, scale_ue8m0=ue8m0) for _ in range(E)]
    w2 = [oracle.block_quant_weight(torch.randn(H, I, generator=g) * 0.05, scale_ue8m0=ue8m0) for _ in range(E)]
    return [torch.stack([w[j] for w in ws]).cuda() for ws in (w1, w2) for j in (0, 1)]


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("M,E,topk,H,I,dtype", [(1, 4, 2, 256, 128, torch.bfloat16), (33, 7, 3, 640, 384, torch.float16),
                                                (300, 16, 9, 384, 256, torch.bfloat16), (70, 40, 17, 4224, 128, torch.bfloat16)])
def test_one_call_layer_equals_the_single_steps(M, E, topk, H, I, dtype, ue8m0):
    from sglang_b200._lib import lib
    from sglang_b200.layers.moe import (_grouped_mm, _grouped_mm_ue8m0, fused_experts_block_fp8,
                                        fused_experts_block_fp8_ue8m0)
    from sglang_b200.layers.quantization.fp8_kernel import pack_ue8m0_scales, sglang_per_token_group_quant_fp8
    from sglang_b200.sgl_kernel import apply_shuffle_mul_sum, prepare_moe_input, shuffle_rows
    w1, s1, w2, s2 = _layer(E, H, I, ue8m0, seed=M)
    if ue8m0:
        s1, s2 = (pack_ue8m0_scales(s.view(-1, s.shape[2])).view(E, s.shape[1], -1) for s in (s1, s2))
    x = make_activations(M, H, seed=M + 1).to(dtype).cuda()
    g = torch.Generator().manual_seed(M + 2)
    weights, ids = torch.topk(torch.softmax(torch.randn(M, E, generator=g), -1), topk)
    weights, ids = weights.cuda(), ids.to(torch.int32)
    if M > 1:
        ids[3, 1], ids[M - 1, 0] = -1, E + 5
    ids = torch.cat([torch.zeros(1, dtype=torch.int32), ids.flatten()]).cuda()[1:].view(M, topk)  # not 16-byte aligned
    layer = fused_experts_block_fp8_ue8m0 if ue8m0 else fused_experts_block_fp8
    got = layer(x, w1, w2, s1, s2, weights, ids, 2.5)

    rows, i32 = M * topk, {"dtype": torch.int32, "device": "cuda"}
    offs, ps1, ps2 = torch.empty(E + 1, **i32), torch.empty(E, 3, **i32), torch.empty(E, 3, **i32)
    a_map, c_map = torch.empty(rows, **i32), torch.empty(rows, **i32)
    prepare_moe_input(ids.clone(), offs, ps1, ps2, a_map, c_map, E, I, H)
    q, s = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=ue8m0, scale_tma_aligned=ue8m0, scale_ue8m0=ue8m0)
    mm = _grouped_mm_ue8m0 if ue8m0 else _grouped_mm
    c1 = torch.zeros(rows, 2 * I, dtype=dtype, device="cuda")
    mm(shuffle_rows(q, a_map, (rows, H)), shuffle_rows(s.contiguous(), a_map, (rows, s.shape[1])), w1, s1, c1, offs)
    q2, sc2 = sglang_per_token_group_quant_fp8(c1, 128, column_major_scales=ue8m0, scale_tma_aligned=ue8m0, scale_ue8m0=ue8m0,
                                               fuse_silu_and_mul=True)
    c2 = torch.zeros(rows, H, dtype=dtype, device="cuda")
    mm(q2, sc2, w2, s2, c2, offs)
    want = torch.empty(M, H, dtype=dtype, device="cuda")
    apply_shuffle_mul_sum(c2, want, c_map, (weights * 2.5).to(dtype).flatten(), round_products=True)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
