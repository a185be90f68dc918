"""The CTA-pair GEMM (tcgen05 cta_group::2, 256 x 256 tiles) through its C-ABI entry against the CPU
oracle, and bit for bit against the single-CTA kernel (both add the k-blocks of a row in the same order)."""

import pytest
import torch

import oracle
from helpers import assert_gemm_close, bits, last_gemm, make_activations, make_weight

pytestmark = pytest.mark.gpu
PAIRS, TILES, FEW_ROWS = "fp8_block_gemm_pair_kernel", "fp8_block_gemm_kernel", "fp8_block_gemm_smallm_kernel"


def _pair(aq, a_s, wq, ws, tile_n, out_dtype=torch.bfloat16):
    from sglang_b200._lib import check, dtype_code, lib
    M, K = aq.shape
    N = wq.shape[0]
    out = torch.empty(M, N, dtype=out_dtype, device="cuda")
    check(lib().sglb200_fp8_blockwise_scaled_mm_pair(
        aq.data_ptr(), wq.data_ptr(), a_s.data_ptr(), ws.data_ptr(), out.data_ptr(), M, N, K, aq.stride(0), wq.stride(0),
        out.stride(0), a_s.stride(0), a_s.stride(1), ws.stride(0), ws.stride(1), dtype_code(out_dtype), tile_n,
        torch.cuda.current_stream().cuda_stream), "fp8_blockwise_scaled_mm_pair")
    return out


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (129, 576, 1024), (300, 1536, 384), (2100, 2368, 512),
                                   (512, 4096, 4096)])
def test_pair_gemm_matches_oracle_and_single_cta_kernel(M, N, K):
    from sglang_b200._lib import check, lib
    a = make_activations(M, K, seed=M + N)
    aq, a_s = oracle.per_token_group_quant_fp8(a, 128)
    wq, ws = make_weight(N, K, seed=K + N)
    ref = oracle.w8a8_block_fp8_matmul(aq, wq, a_s, ws)
    aq_d, as_d, wq_d, ws_d = aq.cuda(), a_s.cuda(), wq.cuda(), ws.cuda()
    out = _pair(aq_d, _m_major(a_s), wq_d, ws_d, 256)
    assert last_gemm() == PAIRS
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert_gemm_close(out, ref, f"pair M={M} N={N} K={K}")
    if M > 64:  # with row-major scales the plain entry runs the 128 x 128 kernel, and without scratch it leaves K whole
        plain = torch.empty_like(out)
        check(lib().sglb200_fp8_blockwise_scaled_mm(
            aq_d.data_ptr(), wq_d.data_ptr(), as_d.data_ptr(), ws_d.data_ptr(), plain.data_ptr(), M, N, K, K, K, N,
            as_d.stride(0), as_d.stride(1), ws_d.stride(0), ws_d.stride(1), 0, torch.cuda.current_stream().cuda_stream),
            "mm")
        assert last_gemm() == TILES
        torch.cuda.synchronize()
        assert torch.equal(bits(out), bits(plain))


def test_pair_gemm_full_size_rows_sample_and_f16():
    M, N, K = 4096, 7168, 16384
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    from sglang_b200.layers.quantization import block_quant_weight_fp8, sglang_per_token_group_quant_fp8
    wq, ws = block_quant_weight_fp8(torch.randn(N, K, generator=g, device="cuda") * 0.02)
    q, s = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True)
    rows = torch.randperm(M, generator=torch.Generator().manual_seed(1))[:48].sort().values.cuda()
    ref = oracle.w8a8_block_fp8_matmul(q[rows].cpu(), wq.cpu(), s[rows].cpu().contiguous(), ws.cpu(),
                                       output_dtype=torch.float16)
    for tile_n in (128, 256):
        out = _pair(q, s, wq, ws, tile_n, out_dtype=torch.float16)
        assert last_gemm() == PAIRS
        torch.cuda.synchronize()
        assert_gemm_close(out[rows], ref, f"pair tile_n={tile_n} full size")


def _m_major(scales):
    """The scales as the quantiser's TMA-aligned layout: M-major, each group's row padded to four."""
    m, k = scales.shape
    buf = torch.full((k, (m + 3) // 4 * 4), float("nan"))
    buf[:, :m] = scales.t()
    return buf.cuda().t()[:m]


@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 8, 128), (127, 136, 272), (129, 576, 640), (256, 256, 4224), (257, 264, 1408), (770, 1000, 1024),
                                   (2500, 5120, 384), (2304, 12288, 128)])
def test_pair_gemm_edges_of_tiles_bit_for_bit(M, N, K, out_dtype):
    # tiles cut off in either direction, one to 33 k-blocks (the shuffle of the weight scales wraps at 32), a K tail, more tiles than
    # pairs, and a dozen tiles of one k-block for every CTA of the other kernel (its ring of tile notes has eight); rows behind the
    # output stay untouched.  Row-major scales send the plain entry to the kernels that the pairs are compared with.
    from sglang_b200._lib import check, dtype_code, lib
    kg = (K + 127) // 128
    a = make_activations(M, kg * 128, seed=M + N)
    aq, a_s = oracle.per_token_group_quant_fp8(a, 128)
    wq, ws = make_weight(N, kg * 128, seed=K + N)
    aq[:, K:] = 0
    ref = oracle.w8a8_block_fp8_matmul(aq, wq, a_s, ws * 0.01, output_dtype=out_dtype)
    aq_d, wq_d, ws_d = aq.cuda()[:, :K], wq.cuda()[:, :K], (ws * 0.01).cuda()
    out, plain = (torch.full((M + 3, N), 7.0, dtype=out_dtype, device="cuda") for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream
    sm, sr = _m_major(a_s), a_s.cuda()
    check(lib().sglb200_fp8_blockwise_scaled_mm_pair(
        aq_d.data_ptr(), wq_d.data_ptr(), sm.data_ptr(), ws_d.data_ptr(), out.data_ptr(), M, N, K, kg * 128, kg * 128, N, sm.stride(0),
        sm.stride(1), ws_d.stride(0), ws_d.stride(1), dtype_code(out_dtype), 256, st), "pair")
    assert last_gemm() == PAIRS
    check(lib().sglb200_fp8_blockwise_scaled_mm(
        aq_d.data_ptr(), wq_d.data_ptr(), sr.data_ptr(), ws_d.data_ptr(), plain.data_ptr(), M, N, K, kg * 128, kg * 128, N, sr.stride(0),
        sr.stride(1), ws_d.stride(0), ws_d.stride(1), dtype_code(out_dtype), st), "mm")
    assert last_gemm() == (FEW_ROWS if M <= 64 else TILES)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    # one unit in the last place: the tensor core sums a k-block in another order than the oracle, and among 28 million results
    # some lie within such a difference (2^-24 of a sum) of a rounding boundary
    assert_gemm_close(out[:M], ref, f"pair M={M} N={N} K={K}", allow_one_ulp=True)
    assert torch.equal(bits(out), bits(plain))  # the three rows behind the output included


@pytest.mark.parametrize("M,N,K", [(1, 576, 7168), (16, 7168, 16384), (64, 1024, 8192), (100, 2112, 7168), (128, 5120, 2560)])
def test_other_scale_layouts_give_the_pairs_bits_at_few_rows(M, N, K):
    # sizes at which the plain entry adds K in ranges (clusters of the few-rows kernel): scales that the pairs do not take, and a limit
    # of one SM, send the call to the 128 x 128 tiles, which add it in the pairs' order
    from sglang_b200._lib import check, lib
    from sglang_b200.layers.quantization import block_quant_weight_fp8, sglang_per_token_group_quant_fp8
    g = torch.Generator(device="cuda").manual_seed(M)
    q, s = sglang_per_token_group_quant_fp8(torch.randn(M, K, generator=g, device="cuda").bfloat16(), 128, column_major_scales=True,
                                            scale_tma_aligned=True)
    wq, ws = block_quant_weight_fp8(torch.randn(N, K, generator=g, device="cuda") * 0.02)
    want = _pair(q, s, wq, ws, 256)
    assert last_gemm() == PAIRS
    ld = (M + 3) // 4 * 4
    odd = torch.empty(1 + K // 128 * ld, device="cuda").as_strided((M, K // 128), (1, ld), 1)
    odd.copy_(s)  # M-major, off the 16-byte boundary
    got = [_pair(q, scales, wq, ws, 256) for scales in (s.contiguous(), odd)]
    assert last_gemm() == TILES
    check(lib().sglb200_set_num_sms(1), "set_num_sms")
    try:
        got.append(_pair(q, s, wq, ws, 256))
    finally:
        lib().sglb200_set_num_sms(0)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    ref = oracle.w8a8_block_fp8_matmul(q.cpu(), wq[:256].cpu(), s.cpu().contiguous(), ws[:2].cpu())
    assert_gemm_close(want[:, :256], ref, f"pair M={M} N={N} K={K}")
    assert all(torch.equal(bits(o), bits(want)) for o in got)


@pytest.mark.parametrize("step", [4, 8, 128])
def test_scales_whose_columns_overlap_stay_on_the_tiles(step):
    # M-major scales with a column stride below M, which a tensor map's strides do not describe: the same bits as from a copy of them
    M, N, K = 132, 256, 1024
    aq, _ = oracle.per_token_group_quant_fp8(make_activations(M, K, seed=1), 128)
    wq, ws = make_weight(N, K, seed=2)
    buf = torch.rand(M + 7 * step, generator=torch.Generator().manual_seed(3)).cuda() * 0.1
    s = buf.as_strided((M, 8), (1, step))
    aq_d, wq_d, ws_d = aq.cuda(), wq.cuda(), ws.cuda()
    out = _pair(aq_d, s, wq_d, ws_d, 256)
    assert last_gemm() == TILES
    want = _pair(aq_d, s.contiguous(), wq_d, ws_d, 256)
    torch.cuda.synchronize()
    assert torch.equal(bits(out), bits(want))
    assert_gemm_close(out, oracle.w8a8_block_fp8_matmul(aq, wq, s.cpu().contiguous(), ws), f"step={step}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_linear_layer_on_pairs_adds_its_bias(dtype):
    # 3072 x 4096 x 4096 is a size the plain entry gives to the pairs; through row-major scales it stays on the 128 x 128 tiles
    from sglang_b200.layers.quantization import block_quant_weight_fp8, sglang_per_token_group_quant_fp8, w8a8_block_fp8_matmul
    from sglang_b200.layers.quantization.fp8 import Fp8Config, Fp8LinearMethod
    M, N, K = 3072, 4096, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    layer, method = torch.nn.Module(), Fp8LinearMethod(Fp8Config())
    method.create_weights(layer, K, [N], K, N, dtype, device="cuda")
    codes, scales = block_quant_weight_fp8(torch.randn(N, K, generator=g, device="cuda") * 0.02)
    layer.weight.data.copy_(codes)
    layer.weight_scale_inv.data.copy_(scales)
    method.process_weights_after_loading(layer)
    bias = torch.randn(N, generator=g, device="cuda").to(dtype)
    out = method.apply(layer, x, bias)
    assert last_gemm() == PAIRS
    q, s = sglang_per_token_group_quant_fp8(x, 128)
    want = w8a8_block_fp8_matmul(q, codes, s, scales, [128, 128], dtype) + bias
    assert last_gemm() == TILES
    torch.cuda.synchronize()
    assert torch.equal(bits(out), bits(want))


@pytest.mark.parametrize("limit", [1, 2, 3, 17, 132, 147])
def test_pairs_under_an_sm_limit(limit):
    # even and odd limits, from one tile after the other on a single pair to all but one SM; under 1 no pair is left and under 3 the
    # 128 x 128 tiles are the better choice.  Plain entries and the pair entry, fp32 and UE8M0 scales: the bits of an unlimited call
    from sglang_b200._lib import check, lib
    from sglang_b200.layers.quantization import (block_quant_weight_fp8, pack_ue8m0_scales, per_block_cast_to_fp8,
                                                 sglang_per_token_group_quant_fp8, w8a8_block_fp8_matmul, w8a8_block_fp8_matmul_ue8m0)
    M, N, K = 1024, 2368, 2048
    g = torch.Generator(device="cuda").manual_seed(limit)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    w = torch.randn(N, K, generator=g, device="cuda") * 0.02
    (wq, ws), (uq, us) = block_quant_weight_fp8(w), per_block_cast_to_fp8(w)
    up = pack_ue8m0_scales(us)
    q, s = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True)
    uxq, uxs = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=True)
    calls = [lambda: w8a8_block_fp8_matmul(q, wq, s, ws, [128, 128], torch.bfloat16), lambda: _pair(q, s, wq, ws, 256),
             lambda: w8a8_block_fp8_matmul_ue8m0(uxq, uq, uxs, up, torch.bfloat16)]
    want = [f() for f in calls]
    check(lib().sglb200_set_num_sms(limit), "set_num_sms")
    try:
        got, ran = [], []
        for f in calls:
            got.append(f())
            ran.append(last_gemm())
    finally:
        lib().sglb200_set_num_sms(0)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    pairs = limit not in (1, 3)
    assert ran == [PAIRS if pairs else TILES, PAIRS if limit > 1 else TILES,
                   "fp8_ue8m0_gemm_pair_kernel" if pairs else "fp8_ue8m0_gemm_kernel"]
    assert all(torch.equal(bits(a), bits(b)) for a, b in zip(got, want))


def test_pair_gemm_refuses_bad_arguments():
    from sglang_b200._lib import lib
    L = lib()
    assert L.sglb200_fp8_blockwise_scaled_mm_pair(None, None, None, None, None, 128, 128, 128, 128, 128, 128, 1, 1, 1, 1, 0,
                                                  192, None) == -1
    assert L.sglb200_fp8_blockwise_scaled_mm_pair(None, None, None, None, None, 128, 128, 128, 128, 128, 128, 1, 1, 1, 1, 0,
                                                  128, None) == -6
