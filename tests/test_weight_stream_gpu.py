"""The weight-streaming kernel at the edges of its token tiles (16 / 32 / 64 / 128 columns, chunks of uneven rows) and the
masked layout with an expected row count, which picks the kernel and must not change the result."""

import pytest
import torch

import oracle
from helpers import assert_gemm_close, last_gemm, make_activations, make_weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 15, 17, 33, 63, 65, 80, 127, 128])
@pytest.mark.parametrize("N,K,dtype", [(264, 640, torch.bfloat16), (1160, 2048, torch.float16)])
def test_token_tile_edges(M, N, K, dtype):
    from sglang_b200._lib import lib
    from sglang_b200.layers.quantization import w8a8_block_fp8_matmul
    a, a_s = oracle.per_token_group_quant_fp8(make_activations(M, K, seed=M), 128)
    w, w_s = make_weight(N, K, seed=N)
    got = w8a8_block_fp8_matmul(a.cuda(), w.cuda(), a_s.cuda(), w_s.cuda(), [128, 128], dtype)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert_gemm_close(got, oracle.w8a8_block_fp8_matmul(a, w, a_s, w_s, output_dtype=dtype), f"M={M}")


@pytest.mark.parametrize("expected", [0, 1, 9, 24, 48, 100])
def test_masked_layout_with_expected_rows(expected):
    from sglang_b200.layers.deep_gemm_wrapper import grouped_gemm_nt_f8f8bf16_masked
    G, max_m, N, K = 5, 100, 384, 640
    masked = torch.tensor([100, 0, 1, 37, 65], dtype=torch.int32)
    q, s = oracle.per_token_group_quant_fp8(make_activations(G * max_m, K, seed=7), 128)
    ws = [make_weight(N, K, seed=20 + g) for g in range(G)]
    out = torch.full((G, max_m, N), 7.0, dtype=torch.bfloat16, device="cuda")
    grouped_gemm_nt_f8f8bf16_masked((q.view(G, max_m, K).cuda(), s.view(G, max_m, -1).cuda()),
                                    (torch.stack([w[0] for w in ws]).cuda(), torch.stack([w[1] for w in ws]).cuda()), out,
                                    masked.cuda(), expected)
    out = out.cpu()
    for g in range(G):
        m = int(masked[g])
        assert (out[g, m:] == 7.0).all(), f"group {g}: rows past masked_m were written"
        if m:
            ref = oracle.w8a8_block_fp8_matmul(q.view(G, max_m, K)[g, :m], ws[g][0], s.view(G, max_m, -1)[g, :m], ws[g][1])
            assert_gemm_close(out[g, :m], ref, f"group {g}")


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 576, 7168), (5, 8, 128), (16, 7168, 2048), (33, 1000, 1024), (64, 10240, 1536),
                                   (113, 2112, 7168), (128, 136, 4096), (129, 576, 2048), (300, 392, 1024), (200, 264, 2176), (385, 1000, 4480)])
def test_linear_layer_with_bias(M, N, K, ue8m0):
    """The one-call linear layer against its parts: quantiser, GEMM entry, then the bias in the output type.  The shapes
    put K on one CTA, on a few and on all of them, and cross the row limits of the kernels."""
    from sglang_b200._lib import lib
    from sglang_b200.layers.quantization.fp8 import Fp8Config, Fp8LinearMethod
    dtype = torch.float16 if N % 16 else torch.bfloat16
    layer, method = torch.nn.Module(), Fp8LinearMethod(Fp8Config())
    method.create_weights(layer, K, [N], K, N, dtype, device="cuda")
    w, w_s = oracle.block_quant_weight(torch.randn(N, K, generator=torch.Generator().manual_seed(N)) * 0.02, scale_ue8m0=ue8m0)
    layer.weight.data.copy_(w)
    layer.weight_scale_inv.data.copy_(w_s)
    method.process_weights_after_loading(layer)
    assert (layer.weight_scale_ue8m0 is not None) == ue8m0
    x = make_activations(M, K, seed=M).to(dtype)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(3)).to(dtype)
    q, s = oracle.per_token_group_quant_fp8(x, 128, scale_ue8m0=ue8m0)
    ref = oracle.w8a8_block_fp8_matmul(q, w, s, w_s, output_dtype=dtype)
    xd, bd = x.cuda(), bias.cuda()
    plain, again, biased = method.apply(layer, xd), method.apply(layer, xd), method.apply(layer, xd, bd)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert torch.equal(plain, again), "the sum over the SMs depends on their order"
    assert torch.equal(biased, plain + bd)
    assert_gemm_close(plain, ref, f"{M}x{N}x{K}", allow_one_ulp=True)


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("M,N,K,dtype", [(1, 576, 7168, torch.bfloat16), (2, 136, 640, torch.float16), (1, 24576, 1152, torch.bfloat16),
                                         (2, 20000, 896, torch.float16), (3, 7168, 2048, torch.bfloat16)])
def test_rows_quantised_by_the_gemm_itself(M, N, K, dtype, ue8m0):
    """Up to two rows the GEMM quantises its activations: the bits of the separate quantiser and the same GEMM.  The shapes put K on
    one CTA and on clusters, several tiles on a CTA, and end K inside a group of four k-blocks."""
    from sglang_b200._lib import lib
    from sglang_b200.layers.quantization import w8a8_block_fp8_matmul
    from sglang_b200.layers.quantization.fp8_kernel import sglang_per_token_group_quant_fp8
    from sglang_b200.layers.quantization.fp8 import Fp8Config, Fp8LinearMethod
    layer, method = torch.nn.Module(), Fp8LinearMethod(Fp8Config())
    method.create_weights(layer, K, [N], K, N, dtype, device="cuda")
    w, w_s = oracle.block_quant_weight(torch.randn(N, K, generator=torch.Generator().manual_seed(N)) * 0.02, scale_ue8m0=ue8m0)
    layer.weight.data.copy_(w)
    layer.weight_scale_inv.data.copy_(w_s)
    method.process_weights_after_loading(layer)
    x = make_activations(M, K, seed=M).to(dtype)
    if not ue8m0:
        x[0, :128] = 0  # a group without a maximum
    x[M - 1, -1] = -0.0
    x = x.cuda()
    got = method.apply(layer, x)
    if ue8m0:
        q, s = oracle.per_token_group_quant_fp8(x.cpu(), 128, scale_ue8m0=True)
    else:
        q, s = sglang_per_token_group_quant_fp8(x, 128)
    want = w8a8_block_fp8_matmul(q.cuda(), w.cuda(), s.cuda(), w_s.cuda(), [128, 128], dtype)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert torch.equal(got, want)


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16])
@pytest.mark.parametrize("N,K,dtype", [(576, 7168, torch.bfloat16), (136, 640, torch.float16), (20000, 1408, torch.bfloat16),
                                       (3072, 1536, torch.float16), (1000, 128, torch.bfloat16), (37888, 256, torch.bfloat16),
                                       (37896, 256, torch.bfloat16)])
def test_up_to_eight_rows_quantised_by_the_gemm(N, K, dtype, M, ue8m0):
    """One and two passes of four rows, full and ragged, from one k-block to several rings on a CTA, and from nine rows on, or
    three where a CTA has more than two tiles, the quantiser kernel: the bits of that kernel and the same GEMM.  A group of
    zeros, and a row beyond the range of the branch-free division (scale above 2^100)."""
    from sglang_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + K)
    x = torch.randn(M, K, generator=g, device="cuda")
    x = (x * torch.pow(10.0, torch.rand(M, 1, generator=g, device="cuda") * 4 - 2)).to(dtype)
    x[M // 2, :128] = 0
    if dtype == torch.bfloat16:
        x[M - 1, -128:] *= 1e35
    w = (torch.randn(N, K, generator=g, device="cuda") * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    words = (K // 128 + 3) // 4
    if ue8m0:
        ws = torch.randint(120, 130, (-(-N // 128), words * 4), generator=g, device="cuda", dtype=torch.uint8).view(torch.int32)
    else:
        ws = torch.rand(-(-N // 128), K // 128, generator=g, device="cuda") + 0.5
    kind = 0 if dtype == torch.bfloat16 else 1
    L, stream = lib(), torch.cuda.current_stream().cuda_stream
    bytes_ = L.sglb200_fp8_block_linear_scratch_bytes(M, N, K, int(ue8m0))
    scratch = torch.full((max(bytes_, 1),), 0x5a, dtype=torch.uint8, device="cuda")
    got = torch.full((M, N), 7.0, dtype=dtype, device="cuda")

    def linear(rows, out):
        check(L.sglb200_fp8_block_linear(rows.data_ptr(), w.data_ptr(), ws.data_ptr(), None, out.data_ptr(), M, N, K, ws.stride(0),
                                         ws.stride(1), int(ue8m0), 1e-10, kind, scratch.data_ptr(), bytes_, stream), "fp8_block_linear")

    linear(x, got)
    torch.cuda.synchronize()
    assert last_gemm() == "fp8_block_gemm_smallm_kernel"
    tiles, sms = -(-N // 128), torch.cuda.get_device_properties(0).multi_processor_count
    assert bool((scratch == 0x5a).all()) == (M <= 2 or (M <= 8 and tiles <= 2 * sms)), "which kernel quantised"
    # the quantiser kernel, then the same GEMM on its codes
    q = torch.empty(M, K, dtype=torch.float8_e4m3fn, device="cuda")
    ld = (M + 3) // 4 * 4
    s = torch.zeros(words if ue8m0 else K // 128, ld, dtype=torch.int32 if ue8m0 else torch.float32, device="cuda")
    check(L.sglb200_per_token_group_quant_fp8(x.data_ptr(), kind, q.data_ptr(), s.data_ptr(), M, K, 128, 1e-10, -448.0, 448.0,
                                              int(ue8m0), 1, ld, stream), "per_token_group_quant_fp8")
    want = torch.empty_like(got)
    if ue8m0:
        check(L.sglb200_fp8_ue8m0_scaled_mm(q.data_ptr(), w.data_ptr(), s.data_ptr(), ws.data_ptr(), want.data_ptr(), M, N, K, K, K, N,
                                            ld, ws.stride(0), ws.stride(1), kind, stream), "fp8_ue8m0_scaled_mm")
    else:
        check(L.sglb200_fp8_blockwise_scaled_mm(q.data_ptr(), w.data_ptr(), s.data_ptr(), ws.data_ptr(), want.data_ptr(), M, N, K, K, K,
                                                N, 1, ld, ws.stride(0), ws.stride(1), kind, stream), "fp8_blockwise_scaled_mm")
    torch.cuda.synchronize()
    assert L.sglb200_read_device_status() == 0
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    if N <= K:  # an output on top of the input: quantised before anything is stored; one or two rows need scratch for it
        three = L.sglb200_fp8_block_linear_scratch_bytes(max(M, 3), N, K, int(ue8m0))
        more = torch.empty(three, dtype=torch.uint8, device="cuda")
        both = x.clone()
        on_top = both.view(-1)[:M * N].view(M, N)

        def in_place(room, size):
            return L.sglb200_fp8_block_linear(both.data_ptr(), w.data_ptr(), ws.data_ptr(), None, on_top.data_ptr(), M, N, K, ws.stride(0),
                                              ws.stride(1), int(ue8m0), 1e-10, kind, room, size, stream)

        assert in_place(None, 0) != 0 and torch.equal(both, x)
        check(in_place(more.data_ptr(), three), "fp8_block_linear")
        torch.cuda.synchronize()
        assert torch.equal(on_top.view(torch.int16), want.view(torch.int16))


def _linear(x, w, ws, ue8m0, eps, in_parts):
    """The C linear layer, or the quantiser kernel followed by the GEMM entry."""
    from sglang_b200._lib import check, lib
    L, (M, K), N, kind = lib(), x.shape, w.shape[0], 0 if x.dtype == torch.bfloat16 else 1
    stream = torch.cuda.current_stream().cuda_stream
    out = torch.full((M, N), 7.0, dtype=x.dtype, device="cuda")
    if not in_parts:
        scratch = torch.empty(L.sglb200_fp8_block_linear_scratch_bytes(M, N, K, int(ue8m0)) + 256, dtype=torch.uint8, device="cuda")
        check(L.sglb200_fp8_block_linear(x.data_ptr(), w.data_ptr(), ws.data_ptr(), None, out.data_ptr(), M, N, K, ws.stride(0), ws.stride(1),
                                         int(ue8m0), eps, kind, scratch.data_ptr(), scratch.numel(), stream), "fp8_block_linear")
        return out
    ld = (M + 3) // 4 * 4
    q = torch.empty(M, K, dtype=torch.float8_e4m3fn, device="cuda")
    s = torch.zeros(-(-K // 512) if ue8m0 else K // 128, ld, dtype=torch.int32 if ue8m0 else torch.float32, device="cuda")
    check(L.sglb200_per_token_group_quant_fp8(x.data_ptr(), kind, q.data_ptr(), s.data_ptr(), M, K, 128, eps, -448.0, 448.0, int(ue8m0), 1,
                                              ld, stream), "per_token_group_quant_fp8")
    if ue8m0:
        check(L.sglb200_fp8_ue8m0_scaled_mm(q.data_ptr(), w.data_ptr(), s.data_ptr(), ws.data_ptr(), out.data_ptr(), M, N, K, K, K, N, ld,
                                            ws.stride(0), ws.stride(1), kind, stream), "fp8_ue8m0_scaled_mm")
    else:
        check(L.sglb200_fp8_blockwise_scaled_mm(q.data_ptr(), w.data_ptr(), s.data_ptr(), ws.data_ptr(), out.data_ptr(), M, N, K, K, K, N, 1,
                                                ld, ws.stride(0), ws.stride(1), kind, stream), "fp8_blockwise_scaled_mm")
    return out


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 2, 4, 7, 8])
def test_odd_values_quantised_by_the_gemm(M, dtype, ue8m0):
    """NaN, infinities, denormals and groups of zeros with no floor, rows that begin on 16 bytes and no more, a limit on the SMs and
    a captured graph: what the quantiser kernel and the GEMM give, bit for bit (a NaN for a NaN)."""
    from sglang_b200._lib import lib
    N, K, L = 1160, 1408, lib()
    g = torch.Generator(device="cuda").manual_seed(M)
    room = torch.randn(M * K + 8, generator=g, device="cuda").to(dtype)
    x = room[8:].view(M, K)  # 16 bytes past the allocation's alignment
    assert x.data_ptr() % 32 == 16
    w = (torch.randn(N, K, generator=g, device="cuda") * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    if ue8m0:
        ws = torch.randint(120, 130, (-(-N // 128), 12), generator=g, device="cuda", dtype=torch.uint8).view(torch.int32)
    else:
        ws = torch.rand(-(-N // 128), K // 128, generator=g, device="cuda") + 0.5
    tiny = torch.finfo(dtype).smallest_normal

    def same(got, want):
        nan = want.isnan()
        return torch.equal(got.isnan(), nan) and torch.equal(got[~nan].view(torch.int16), want[~nan].view(torch.int16))

    odd = {"plain": lambda: None, "nan": lambda: x[M // 2, 130:133].fill_(float("nan")),
           "nan group": lambda: x[M - 1, 256:384].fill_(float("nan")), "inf": lambda: x[0, 5].fill_(float("-inf")),
           "zeros": lambda: x[M // 2, 512:640].zero_(), "denormals": lambda: x[M - 1, 640:768].fill_(tiny / 4),
           "minus zero": lambda: x[0, 768:800].fill_(-0.0)}
    for name, put in odd.items():
        x.copy_(torch.randn(M, K, generator=g, device="cuda"))
        put()
        for eps in (1e-10, 0.0):
            got, want = _linear(x, w, ws, ue8m0, eps, False), _linear(x, w, ws, ue8m0, eps, True)
            assert same(got, want), f"{name}, eps {eps}"
    x.copy_(torch.randn(M, K, generator=g, device="cuda"))
    want = _linear(x, w, ws, ue8m0, 1e-10, True)
    try:
        assert L.sglb200_set_num_sms(5) == 0  # ten tiles at most: two each
        assert same(_linear(x, w, ws, ue8m0, 1e-10, False), _linear(x, w, ws, ue8m0, 1e-10, True))
    finally:
        assert L.sglb200_set_num_sms(0) == 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = _linear(x, w, ws, ue8m0, 1e-10, False)
    keep = x.clone()
    x.zero_()
    graph.replay()
    assert (out == 0).all()
    x.copy_(keep)
    graph.replay()
    torch.cuda.synchronize()
    assert same(out, want) and L.sglb200_read_device_status() == 0


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("M", [1, 7, 9, 16, 17, 31, 33, 64, 65, 100, 121, 128])
@pytest.mark.parametrize("N,K,dtype", [(1000, 7168, torch.bfloat16), (4072, 4096, torch.float16), (7112, 7168, torch.bfloat16)])
def test_shares_of_a_tile_in_clusters(N, K, dtype, M, ue8m0):
    """Clusters of eight, four and two add up a tile's sums, a share each: rows that give every CTA a full share, an uneven one or
    none, a ragged last tile, a bias, and nothing written past the last row."""
    from sglang_b200._lib import check, lib
    w, w_s = make_weight(N, K, seed=N) if not ue8m0 else oracle.block_quant_weight(
        torch.randn(N, K, generator=torch.Generator().manual_seed(N)) * 0.02, scale_ue8m0=True)
    x = make_activations(M, K, seed=M).to(dtype)
    a, a_s = oracle.per_token_group_quant_fp8(x, 128, scale_ue8m0=ue8m0)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(3)).to(dtype).cuda()
    ref = oracle.w8a8_block_fp8_matmul(a, w, a_s, w_s, output_dtype=dtype)
    L, kind = lib(), 0 if dtype == torch.bfloat16 else 1
    xd, wd = x.cuda(), w.cuda()
    if ue8m0:
        from sglang_b200.layers.quantization.fp8_kernel import pack_ue8m0_scales
        ws = pack_ue8m0_scales(w_s.cuda())
    else:
        ws = w_s.cuda()
    bytes_ = L.sglb200_fp8_block_linear_scratch_bytes(M, N, K, int(ue8m0))
    scratch = torch.empty(max(bytes_, 1), dtype=torch.uint8, device="cuda")
    outs = []
    for b in (None, bias):
        out = torch.full((M + 1, N), 7.0, dtype=dtype, device="cuda")
        check(L.sglb200_fp8_block_linear(xd.data_ptr(), wd.data_ptr(), ws.data_ptr(), None if b is None else b.data_ptr(), out.data_ptr(),
                                         M, N, K, ws.stride(0), ws.stride(1), int(ue8m0), 1e-10, kind, scratch.data_ptr(), bytes_,
                                         torch.cuda.current_stream().cuda_stream), "fp8_block_linear")
        assert last_gemm() == "fp8_block_gemm_smallm_kernel"
        outs.append(out)
    torch.cuda.synchronize()
    assert L.sglb200_read_device_status() == 0
    assert (outs[0][M] == 7.0).all() and (outs[1][M] == 7.0).all(), "a row past the last one was written"
    assert torch.equal(outs[1][:M], outs[0][:M] + bias)
    assert_gemm_close(outs[0][:M], ref, f"{M}x{N}x{K}", allow_one_ulp=True)


@pytest.mark.parametrize("M,N,K,kernel", [(129, 576, 7168, "fp8_block_gemm_smallm_kernel"), (177, 1000, 4096, "fp8_block_gemm_smallm_kernel"),
                                          (255, 520, 7168, "fp8_block_gemm_smallm_kernel"), (256, 576, 7168, "fp8_block_gemm_smallm_kernel"),
                                          (257, 576, 7168, "fp8_block_gemm_kernel"), (200, 4096, 4096, "fp8_block_gemm_kernel")])
def test_two_chunks_of_rows_in_clusters(M, N, K, kernel):
    """129 to 256 rows where clusters share K: two chunks of rows, even and uneven, and the sizes beyond, which keep the 128 x 128
    tiles with K cut through scratch.  A bias, nothing written past the last row, the same result twice."""
    from sglang_b200._lib import check, lib
    w, w_s = make_weight(N, K, seed=N)
    x = make_activations(M, K, seed=M)
    a, a_s = oracle.per_token_group_quant_fp8(x, 128)
    bias = torch.randn(N, generator=torch.Generator().manual_seed(3)).bfloat16().cuda()
    L, xd, wd, ws = lib(), x.cuda(), w.cuda(), w_s.cuda()
    bytes_ = L.sglb200_fp8_block_linear_scratch_bytes(M, N, K, 0)
    scratch = torch.empty(bytes_, dtype=torch.uint8, device="cuda")
    outs = []
    for b in (None, bias, None):
        out = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
        check(L.sglb200_fp8_block_linear(xd.data_ptr(), wd.data_ptr(), ws.data_ptr(), None if b is None else b.data_ptr(), out.data_ptr(),
                                         M, N, K, ws.stride(0), ws.stride(1), 0, 1e-10, 0, scratch.data_ptr(), bytes_,
                                         torch.cuda.current_stream().cuda_stream), "fp8_block_linear")
        assert last_gemm() == kernel
        outs.append(out)
    torch.cuda.synchronize()
    assert L.sglb200_read_device_status() == 0
    assert all((out[M] == 7.0).all() for out in outs), "a row past the last one was written"
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1][:M], outs[0][:M] + bias)
    assert_gemm_close(outs[0][:M], oracle.w8a8_block_fp8_matmul(a, w, a_s, w_s), f"{M}x{N}x{K}")


@pytest.mark.parametrize("M", [1, 16, 128])
def test_weights_written_by_the_kernel_before(M):
    """The quantiser writes the codes that the next call takes as weights, into the same memory every time: the
    weight-streaming kernel, which reads weight tiles ahead of its other operands, must see the new ones."""
    from sglang_b200.layers.quantization import w8a8_block_fp8_matmul
    from sglang_b200.sgl_kernel import sgl_per_token_group_quant_8bit
    N, K = 24576, 1536
    a, a_s = oracle.per_token_group_quant_fp8(make_activations(M, K, seed=M), 128)
    a, a_s = a.cuda(), a_s.cuda()
    y = [torch.randn(N, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)).bfloat16() for i in range(3)]
    w, w_s = torch.empty(N, K, dtype=torch.float8_e4m3fn, device="cuda"), torch.empty(N, K // 128, device="cuda")
    blocks = torch.ones(N // 128, K // 128, device="cuda")

    def product(i, wait):
        sgl_per_token_group_quant_8bit(y[i], w, w_s, 128, 1e-10, -448.0, 448.0)
        if wait:
            torch.cuda.synchronize()
        return w8a8_block_fp8_matmul(a, w, a_s, blocks, [128, 128], torch.bfloat16)

    want = [product(i, True) for i in range(3)]
    got = [product(i % 3, False) for i in range(9)]
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 3]), f"call {i} saw other weights"


@pytest.mark.parametrize("M", [129, 200, 256])
def test_weights_written_by_a_kernel_that_releases_early(M):
    """Above 128 rows the weights may come from a kernel that releases its dependents before it has ended, as the SiLU quantiser
    does: the few-rows kernel, which takes these sizes too, must not read them ahead of it."""
    from sglang_b200._lib import check, lib
    from sglang_b200.layers.quantization import w8a8_block_fp8_matmul
    N, K = 576, 7168
    a, a_s = oracle.per_token_group_quant_fp8(make_activations(M, K, seed=M), 128)
    a, a_s = a.cuda(), a_s.cuda()
    y = [torch.randn(N, 2 * K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(i)).bfloat16() for i in range(3)]
    w, w_s = torch.empty(N, K, dtype=torch.float8_e4m3fn, device="cuda"), torch.empty(N, K // 128, device="cuda")
    blocks = torch.ones(-(-N // 128), K // 128, device="cuda")

    def product(i, wait):
        check(lib().sglb200_silu_mul_group_quant_fp8(y[i].data_ptr(), 0, w.data_ptr(), w_s.data_ptr(), None, N, K, 128, 1e-10, -448.0, 448.0,
                                                     0, K // 128, 1, torch.cuda.current_stream().cuda_stream), "silu_mul_group_quant_fp8")
        if wait:
            torch.cuda.synchronize()
        out = w8a8_block_fp8_matmul(a, w, a_s, blocks, [128, 128], torch.bfloat16)
        assert last_gemm() == "fp8_block_gemm_smallm_kernel"
        return out

    want = [product(i, True) for i in range(3)]
    assert not torch.equal(want[0], want[1])
    got = [product(i % 3, False) for i in range(9)]
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 3]), f"call {i} saw other weights"


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("k_blocks", [1, 2, 5, 11, 12, 23])
def test_rings_over_several_tiles(M, k_blocks):
    """Barriers, tensor-memory stages and scale slots go round in rings of different lengths, over the end of a tile too: up to
    three tiles on a CTA, K from one k-block to more than twice the longest ring, an odd end of K.  No cluster shares K here, so
    the bits are those of the 128 x 128 tiles (row-major scales keep the explicit entry on them)."""
    from sglang_b200._lib import check, lib
    from sglang_b200.layers.quantization import w8a8_block_fp8_matmul
    N, K = 128 * 300 + 8, 128 * k_blocks - (96 if k_blocks > 1 else 0)
    g = torch.Generator(device="cuda").manual_seed(M * 100 + k_blocks)
    a = (torch.randn(M, K, generator=g, device="cuda") * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    w = (torch.randn(N, K, generator=g, device="cuda") * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    a_s = torch.rand(M, k_blocks, generator=g, device="cuda") + 0.5
    w_s = torch.rand(-(-N // 128), k_blocks, generator=g, device="cuda") + 0.5
    got = w8a8_block_fp8_matmul(a, w, a_s, w_s, [128, 128], torch.bfloat16)
    assert last_gemm() == "fp8_block_gemm_smallm_kernel"
    want = torch.empty_like(got)
    check(lib().sglb200_fp8_blockwise_scaled_mm_pair(
        a.data_ptr(), w.data_ptr(), a_s.data_ptr(), w_s.data_ptr(), want.data_ptr(), M, N, K, K, K, N, a_s.stride(0), a_s.stride(1),
        w_s.stride(0), w_s.stride(1), 0, 256, torch.cuda.current_stream().cuda_stream), "fp8_blockwise_scaled_mm_pair")
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    if M > 1:  # a single row's scales pass for M-major ones, which the pair kernel takes (the same bits again)
        assert last_gemm() == "fp8_block_gemm_kernel"
    assert torch.equal(got, want)


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("M", [33, 47, 48, 49, 64])
@pytest.mark.parametrize("N,K", [(576, 7168), (2112, 1536), (1000, 1024)])
def test_two_promotion_sets_in_clusters(M, N, K, ue8m0):
    """33 to 64 rows where clusters share K: two sets of 32 columns, the second one full, ragged and down to a single column."""
    from sglang_b200._lib import lib
    from sglang_b200.layers.quantization import w8a8_block_fp8_matmul
    x = make_activations(M, K, seed=M)
    w, w_s = oracle.block_quant_weight(torch.randn(N, K, generator=torch.Generator().manual_seed(N)) * 0.02, scale_ue8m0=ue8m0)
    a, a_s = oracle.per_token_group_quant_fp8(x, 128, scale_ue8m0=ue8m0)
    got = w8a8_block_fp8_matmul(a.cuda(), w.cuda(), a_s.cuda(), w_s.cuda(), [128, 128], torch.bfloat16)
    assert last_gemm() == "fp8_block_gemm_smallm_kernel"
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert_gemm_close(got, oracle.w8a8_block_fp8_matmul(a, w, a_s, w_s), f"{M}x{N}x{K}")
