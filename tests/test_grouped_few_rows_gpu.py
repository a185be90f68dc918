"""The grouped GEMM on few rows per expert (the decode case of a mixture-of-experts layer): the weight-streaming kernel
with swapped operands against the oracle run expert by expert, and bit for bit against the 128 x 128 grouped kernel on
the same inputs.  The reference checks its grouped kernel against a per-expert loop of the torch-native block matmul the
same way (sgl-kernel/tests/test_fp8_blockwise_moe.py:122-221)."""

import contextlib

import numpy as np
import pytest
import torch

import oracle
from helpers import assert_gemm_close, make_activations

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def few_rows_limit(limit):
    from sglang_b200._lib import lib
    L = lib()
    before = L.sglb200_get_grouped_few_rows()
    assert L.sglb200_set_grouped_few_rows(limit) == 0
    try:
        yield
    finally:
        assert L.sglb200_set_grouped_few_rows(before) == 0


def _weights(E, N, K, seed, ue8m0=False):
    g = torch.Generator().manual_seed(seed)
    ws = [oracle.block_quant_weight(torch.randn(N, K, generator=g) * 0.05, scale_ue8m0=ue8m0) for _ in range(E)]
    return torch.stack([w[0] for w in ws]), torch.stack([w[1] for w in ws])


def _run_sorted(aq, a_s, wq, wsc, counts, out_dtype=torch.bfloat16, pad_rows=3):
    from sglang_b200.sgl_kernel import fp8_blockwise_scaled_grouped_mm
    E, N, K = wq.shape
    rows = sum(counts)
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    ps = torch.tensor([[c, N, K] for c in counts], dtype=torch.int32)
    out = torch.full((rows + pad_rows, N), 7.0, dtype=out_dtype, device="cuda")
    d = torch.empty(0, device="cuda")
    fp8_blockwise_scaled_grouped_mm(out[:rows], d, d, d, d, d, aq.cuda(), wq.cuda().transpose(1, 2), a_s.cuda(),
                                    wsc.cuda().transpose(1, 2), d, d, d, d, d, ps.cuda(),
                                    torch.from_numpy(offs[:-1].copy()).cuda(), d)
    torch.cuda.synchronize()
    from sglang_b200._lib import lib
    assert lib().sglb200_read_device_status() == 0
    return out.cpu(), offs


@pytest.mark.parametrize("counts,N,K", [
    ([3, 0, 17, 1, 9, 0, 40, 2], 384, 512),      # 16-row chunks; experts with 2 and 3 chunks; empty experts
    ([0, 0, 7], 256, 128),                       # one k-block, leading empty experts
    ([20] * 12, 256, 1024),                      # 32-row chunks
    ([33, 40, 1, 64, 50], 512, 640),             # 64-row chunks, one exactly full
    ([1] * 64, 128, 7168),                       # one row each, a long K
    ([16, 16, 16, 16], 2048, 256),               # full 16-row chunks
])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16])
def test_few_rows_grouped_matches_oracle_and_tile_kernel(counts, N, K, out_dtype):
    E, rows = len(counts), sum(counts)
    a = make_activations(rows, K, seed=rows + N)
    aq, a_s = oracle.per_token_group_quant_fp8(a, 128)
    wq, wsc = _weights(E, N, K, seed=K)
    with few_rows_limit(64):
        got, offs = _run_sorted(aq, a_s, wq, wsc, counts, out_dtype)
    with few_rows_limit(0):
        tiled, _ = _run_sorted(aq, a_s, wq, wsc, counts, out_dtype)
    assert (got[rows:] == 7.0).all(), "rows past the last expert were written"
    assert torch.equal(got.view(torch.int16), tiled.view(torch.int16)), "few-rows kernel and 128 x 128 kernel differ"
    ref = torch.cat([oracle.w8a8_block_fp8_matmul(aq[offs[e]:offs[e + 1]], wq[e], a_s[offs[e]:offs[e + 1]], wsc[e],
                                                  output_dtype=out_dtype) for e in range(E) if counts[e]])
    assert_gemm_close(got[:rows], ref, f"few rows {counts}")


def test_few_rows_grouped_offsets_without_problem_sizes():
    """The C entry point with expert_offsets [E + 1] alone (no problem-size table), as the fused MoE calls it."""
    from sglang_b200.layers.moe import _grouped_mm
    counts, N, K = [2, 0, 11, 5, 0, 0, 30, 1], 200, 384  # a ragged last weight tile
    E, rows = len(counts), sum(counts)
    a = make_activations(rows, K, seed=5)
    aq, a_s = oracle.per_token_group_quant_fp8(a, 128)
    wq, wsc = _weights(E, N, K, seed=6)
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32)
    outs = []
    for limit in (64, 0):
        out = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device="cuda")
        with few_rows_limit(limit):
            _grouped_mm(aq.cuda(), a_s.cuda(), wq.cuda(), wsc.cuda(), out, offs.cuda())
        torch.cuda.synchronize()
        outs.append(out.cpu())
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    ref = torch.cat([oracle.w8a8_block_fp8_matmul(aq[offs[e]:offs[e + 1]], wq[e], a_s[offs[e]:offs[e + 1]], wsc[e])
                     for e in range(E) if counts[e]])
    assert_gemm_close(outs[0], ref, "offsets only")


@pytest.mark.parametrize("G,max_m", [(6, 16), (5, 24), (4, 64)])
def test_few_rows_masked_layout(G, max_m):
    from sglang_b200.layers.deep_gemm_wrapper import grouped_gemm_nt_f8f8bf16_masked
    N, K = 384, 512
    masked = torch.randint(0, max_m + 1, (G,), generator=torch.Generator().manual_seed(G), dtype=torch.int32)
    masked[0], masked[1] = max_m, 0
    x = make_activations(G * max_m, K, seed=max_m, outliers=False)
    q, s = oracle.per_token_group_quant_fp8(x, 128)
    wq, ws = _weights(G, N, K, seed=3)
    outs = []
    for limit in (64, 0):
        out = torch.full((G, max_m, N), 7.0, dtype=torch.bfloat16, device="cuda")
        with few_rows_limit(limit):
            grouped_gemm_nt_f8f8bf16_masked((q.view(G, max_m, K).cuda(), s.view(G, max_m, -1).cuda()),
                                            (wq.cuda(), ws.cuda()), out, masked.cuda(), max_m)
        torch.cuda.synchronize()
        outs.append(out.cpu())
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    for g in range(G):
        m = int(masked[g])
        assert (outs[0][g, m:] == 7.0).all(), f"group {g}: rows past masked_m were written"
        if m:
            ref = oracle.w8a8_block_fp8_matmul(q.view(G, max_m, K)[g, :m], wq[g], s.view(G, max_m, -1)[g, :m], ws[g])
            assert_gemm_close(outs[0][g, :m], ref, f"group {g}")


@pytest.mark.parametrize("counts,N,K", [([3, 0, 17, 1, 9, 0, 40, 2], 448, 512), ([20] * 6, 256, 1152), ([1] * 32, 128, 7168)])
def test_few_rows_grouped_ue8m0(counts, N, K):
    """Power-of-two scales: the few-rows kernel decodes the packed exponent words and applies the scales after each
    k-block, exactly; within the output rounding of the oracle, and within one unit in the last place of the block-scaled
    tensor-core kernel (which applies the scales inside the MMA, before its fp32 accumulation)."""
    from sglang_b200.layers.moe import _grouped_mm_ue8m0
    from sglang_b200.layers.quantization import pack_ue8m0_scales
    E, rows = len(counts), sum(counts)
    x = make_activations(rows, K, seed=rows + N, outliers=False)
    q, s = oracle.per_token_group_quant_fp8(x, 128, scale_ue8m0=True)
    wq, wsc = _weights(E, N, K, seed=N, ue8m0=True)
    wp = torch.stack([pack_ue8m0_scales(t) for t in wsc])
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32)
    outs = []
    for limit in (64, 0):
        out = torch.full((rows, N), 7.0, dtype=torch.bfloat16, device="cuda")
        with few_rows_limit(limit):
            _grouped_mm_ue8m0(q.cuda(), pack_ue8m0_scales(s).cuda(), wq.cuda(), wp.cuda(), out, offs.cuda())
        torch.cuda.synchronize()
        from sglang_b200._lib import lib
        assert lib().sglb200_read_device_status() == 0
        outs.append(out.cpu())
    for e in range(E):
        r0, r1 = int(offs[e]), int(offs[e + 1])
        if r1 > r0:
            ref = oracle.w8a8_block_fp8_matmul(q[r0:r1], wq[e], s[r0:r1], wsc[e])
            assert_gemm_close(outs[0][r0:r1], ref, f"expert {e}, few-rows kernel")
            assert_gemm_close(outs[1][r0:r1], ref, f"expert {e}, tile kernel", allow_one_ulp=True)
            assert_gemm_close(outs[0][r0:r1], outs[1][r0:r1], f"expert {e}, kernels against each other", allow_one_ulp=True)


def test_few_rows_limit_setter_rejects_bad_values():
    from sglang_b200._lib import lib
    L = lib()
    before = L.sglb200_get_grouped_few_rows()
    assert L.sglb200_set_grouped_few_rows(-1) != 0
    assert L.sglb200_set_grouped_few_rows(65) != 0
    assert L.sglb200_get_grouped_few_rows() == before


@pytest.mark.parametrize("tokens", [4, 48])
def test_fused_experts_decode_sizes_same_bits_on_both_kernels(tokens):
    """A whole fused-expert layer at decode sizes (few tokens, many experts) takes the few-rows grouped kernel for both
    GEMMs; its output equals the 128 x 128 path's bit for bit and the oracle's within the output-rounding bar."""
    from sglang_b200.layers.moe import fused_experts_block_fp8
    E, topk, H, I = 32, 4, 512, 256
    g = torch.Generator().manual_seed(tokens)
    x = make_activations(tokens, H, seed=tokens, outliers=False)
    w13, w13s = _weights(E, 2 * I, H, seed=11)
    w2, w2s = _weights(E, H, I, seed=12)
    scores = torch.randn(tokens, E, generator=g)
    tw, ti = torch.topk(torch.softmax(scores, -1), topk)
    tw = (tw / tw.sum(-1, keepdim=True)).float()
    outs = []
    for limit in (64, 0):
        with few_rows_limit(limit):
            y = fused_experts_block_fp8(x.cuda(), w13.cuda(), w2.cuda(), w13s.cuda(), w2s.cuda(), tw.cuda(),
                                        ti.int().cuda())
        torch.cuda.synchronize()
        outs.append(y.cpu())
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    ref = oracle.fused_experts_block_fp8(x, w13, w2, w13s, w2s, tw, ti)
    assert_gemm_close(outs[0], ref, f"fused experts, {tokens} tokens")


ROW_ENDS = [1, 16, 17, 31, 0, 32, 33, 64, 95, 96, 97, 112, 113, 127, 128, 129, 224, 225, 5]  # both sides of the boxes of 16 and 32 rows


def test_tile_kernel_at_the_ends_of_experts():
    """A tile that an expert's end cuts loads its rows in boxes and zeros behind them, and stores blocks of 32 rows whole
    or by the row.  fp32 scales: bit for bit what the few-rows kernel gives, and the oracle's."""
    N, K, rows = 384, 896, sum(ROW_ENDS)
    aq, a_s = oracle.per_token_group_quant_fp8(make_activations(rows, K, seed=1), 128)
    wq, wsc = _weights(len(ROW_ENDS), N, K, seed=2)
    with few_rows_limit(0):
        tiled, offs = _run_sorted(aq, a_s, wq, wsc, ROW_ENDS)
    with few_rows_limit(64):  # 85 rows an expert on average: above its limit, so expert by expert
        for e, n in enumerate(ROW_ENDS):
            if 0 < n <= 64:
                one, _ = _run_sorted(aq[offs[e]:offs[e + 1]], a_s[offs[e]:offs[e + 1]], wq[e:e + 1], wsc[e:e + 1], [n])
                assert torch.equal(one[:n].view(torch.int16), tiled[offs[e]:offs[e + 1]].view(torch.int16)), n
    assert (tiled[rows:] == 7.0).all()
    ref = torch.cat([oracle.w8a8_block_fp8_matmul(aq[offs[e]:offs[e + 1]], wq[e], a_s[offs[e]:offs[e + 1]], wsc[e])
                     for e in range(len(ROW_ENDS)) if ROW_ENDS[e]])
    assert_gemm_close(tiled[:rows], ref, "ends of experts", allow_one_ulp=True)


def test_ue8m0_tile_kernel_at_the_ends_of_experts():
    from sglang_b200._lib import check, lib
    from sglang_b200.layers.quantization import pack_ue8m0_scales
    N, K, rows, E = 264, 896, sum(ROW_ENDS), len(ROW_ENDS)
    aq, a_s = oracle.per_token_group_quant_fp8(make_activations(rows, K, seed=1), 128, scale_ue8m0=True)
    wq, wsc = _weights(E, N, K, seed=2, ue8m0=True)
    offs = np.concatenate([[0], np.cumsum(ROW_ENDS)]).astype(np.int32)
    a, w, sa = aq.cuda(), wq.cuda(), pack_ue8m0_scales(a_s).cuda()
    sw = pack_ue8m0_scales(wsc.view(-1, wsc.shape[2]).cuda()).view(E, wsc.shape[1], -1)
    out, o = torch.full((rows + 3, N), 7.0, dtype=torch.bfloat16, device="cuda"), torch.from_numpy(offs).cuda()
    with few_rows_limit(0):
        check(lib().sglb200_fp8_ue8m0_scaled_grouped_mm(a.data_ptr(), w.data_ptr(), sa.data_ptr(), sw.data_ptr(), out.data_ptr(), o.data_ptr(),
                                                        rows, E, N, K, K, K, N * K, N, sa.stride(0), sa.stride(1), sw.stride(0), sw.stride(1),
                                                        sw.stride(2), 0, torch.cuda.current_stream().cuda_stream), "grouped mm")
        torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert (out[rows:] == 7.0).all()
    ref = torch.cat([oracle.w8a8_block_fp8_matmul(aq[offs[e]:offs[e + 1]], wq[e], a_s[offs[e]:offs[e + 1]], wsc[e])
                     for e in range(E) if ROW_ENDS[e]])
    assert_gemm_close(out[:rows], ref, "ends of experts, UE8M0", allow_one_ulp=True)


@pytest.mark.parametrize("ue8m0", [False, True])
@pytest.mark.parametrize("rows", [5, 20, 60])
@pytest.mark.parametrize("K", [128, 256, 896, 1024, 1280, 1408])
def test_few_rows_many_short_items(K, rows, ue8m0):
    """Several items on every CTA, K from one k-block to past the ring: below its length two warps load the scales in turn, from there
    one.  Experts without rows in between (runs of more than a warp's 32 too) and the masked layout; the bits of the tile kernel."""
    from sglang_b200.layers.deep_gemm_wrapper import grouped_gemm_nt_f8f8bf16_masked
    from sglang_b200.layers.moe import _grouped_mm
    from sglang_b200._lib import lib
    E, N = 120, 1160
    g = torch.Generator(device="cuda").manual_seed(K + rows)
    counts = torch.randint(0, 2 * rows + 1, (E,), generator=g, device="cuda").clamp(max=64)
    counts[3:40] = 0
    counts[E - 1] = 0
    w = (torch.randn(E, N, K, generator=g, device="cuda") * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    ws = torch.rand(E, -(-N // 128), K // 128, generator=g, device="cuda") + 0.5
    total = int(counts.sum())
    a = (torch.randn(total, K, generator=g, device="cuda") * 50).clamp(-448, 448).to(torch.float8_e4m3fn)
    a_s = torch.rand(total, K // 128, generator=g, device="cuda") + 0.5
    offs = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), counts.cumsum(0)]).int()
    if ue8m0:  # the masked layout has fp32 scales only: powers of two in both forms of the sorted one
        from sglang_b200.layers.quantization import pack_ue8m0_scales
        a_s, ws = torch.exp2(torch.floor(torch.log2(a_s))), torch.exp2(torch.floor(torch.log2(ws)))
        pa, pw = pack_ue8m0_scales(a_s), pack_ue8m0_scales(ws.view(-1, K // 128)).view(E, -(-N // 128), -1)
        outs = []
        for limit in (64, 0):
            out = torch.full((total + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
            with few_rows_limit(limit):
                from sglang_b200._lib import check
                check(lib().sglb200_fp8_ue8m0_scaled_grouped_mm(
                    a.data_ptr(), w.data_ptr(), pa.data_ptr(), pw.data_ptr(), out.data_ptr(), offs.data_ptr(), total, E, N, K, K, K, N * K, N,
                    pa.stride(0), pa.stride(1), pw.stride(0), pw.stride(1), pw.stride(2), 0, torch.cuda.current_stream().cuda_stream), "mm")
            outs.append(out)
        torch.cuda.synchronize()
        assert lib().sglb200_read_device_status() == 0 and (outs[0][total] == 7.0).all()
        err = (outs[0][:total].float() - outs[1][:total].float()).norm() / outs[1][:total].float().norm()
        assert err < 2e-3, "another order of the same fp32 sums: a bf16 rounding apart at most"
        return
    outs, masked = [], []
    for limit in (64, 0):
        out = torch.full((total + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
        rows_out = torch.full((E, 64, N), 7.0, dtype=torch.bfloat16, device="cuda")
        am, sm = torch.zeros(E, 64, K, device="cuda").to(a.dtype), torch.ones(E, 64, K // 128, device="cuda")
        for e in range(E):
            n, o = int(counts[e]), int(offs[e])
            am[e, :n], sm[e, :n] = a[o:o + n], a_s[o:o + n]
        with few_rows_limit(limit):
            _grouped_mm(a, a_s, w, ws, out[:total], offs)
            grouped_gemm_nt_f8f8bf16_masked((am, sm), (w, ws), rows_out, counts.int(), rows)
        outs.append(out)
        masked.append(rows_out)
    torch.cuda.synchronize()
    assert lib().sglb200_read_device_status() == 0
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    assert torch.equal(masked[0].view(torch.int16), masked[1].view(torch.int16))
    assert (outs[0][total] == 7.0).all()
