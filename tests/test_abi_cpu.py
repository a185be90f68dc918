"""CPU-side checks: the C-ABI library loads without a GPU and exports every symbol the header
declares; host-side validation raises before anything could launch; the quantiser's FMA division
is checked against the IEEE division on a sample of the exhaustive host test."""

import os
import re
import subprocess
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "sglb200.h")


@pytest.fixture(scope="module")
def built_lib():
    from sglang_b200 import build
    path = build.build()
    assert os.path.exists(path)
    return path


def _declared_symbols():
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(sglb200_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol(built_lib):
    from sglang_b200._lib import SIGNATURES, lib
    handle = lib()
    declared = _declared_symbols()
    assert len(declared) >= 12
    for name in declared:
        assert hasattr(handle, name), f"{name} is declared in include/sglb200.h but not exported"
    assert sorted(SIGNATURES) == declared, "ctypes signatures and header are out of step"
    assert handle.sglb200_version().decode() == "0.2"
    assert handle.sglb200_status_string(0).decode() == "ok"
    assert "alignment" in handle.sglb200_status_string(-2).decode()


def test_header_cites_the_reference_for_each_kernel_entry():
    text = open(HEADER).read()
    for name in ["per_token_group_quant_8bit.cu", "fp8_blockwise_gemm_kernel.cu", "fp8_blockwise_moe_kernel.cu",
                 "prepare_moe_input.cu", "activation.cu", "common_extension.cc"]:
        assert name in text


def test_host_validation_without_gpu(built_lib):
    """Shape / dtype / null checks come first, so they are reachable on a machine with no GPU."""
    from sglang_b200._lib import check, lib
    L = lib()
    assert L.sglb200_per_token_group_quant_fp8(None, 0, None, None, 4, 200, 128, 1e-10, -448.0, 448.0, 0, 2, 1, None) == -1
    assert "multiple of group_size" in L.sglb200_last_error_detail().decode()
    assert L.sglb200_per_token_group_quant_fp8(None, 0, None, None, 4, 256, 8, 1e-10, -448.0, 448.0, 0, 2, 1, None) == -1
    assert L.sglb200_per_token_group_quant_fp8(None, 7, None, None, 4, 256, 128, 1e-10, -448.0, 448.0, 0, 2, 1, None) == -5
    assert L.sglb200_per_token_group_quant_fp8(None, 0, None, None, 4, 256, 128, 1e-10, -448.0, 448.0, 0, 2, 1, None) == -6
    assert L.sglb200_per_token_group_quant_fp8(None, 0, None, None, 0, 256, 128, 1e-10, -448.0, 448.0, 0, 2, 1, None) == 0
    assert L.sglb200_fp8_blockwise_scaled_mm(None, None, None, None, None, 4, 128, 100, 100, 100, 128, 1, 4, 1, 1, 0, None) == -1
    assert L.sglb200_fp8_blockwise_scaled_mm(None, None, None, None, None, 4, 128, 128, 128, 128, 128, 1, 4, 1, 1, 2, None) == -5
    assert L.sglb200_fp8_blockwise_scaled_mm(None, None, None, None, None, 0, 128, 128, 128, 128, 128, 1, 4, 1, 1, 0, None) == 0
    assert L.sglb200_shuffle_rows(None, None, None, 4, 6, None) == -1
    assert L.sglb200_prepare_moe_input(None, None, None, None, None, None, 4, 2, 5000, 1, 1, None) == -1
    with pytest.raises(RuntimeError, match="bad shape"):
        check(-1, "op")


def test_ops_refuse_cpu_tensors(built_lib):
    from sglang_b200.sgl_kernel import fp8_blockwise_scaled_mm, silu_and_mul
    a = torch.zeros(4, 128, dtype=torch.float8_e4m3fn)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        fp8_blockwise_scaled_mm(a, a.t(), torch.ones(4, 1), torch.ones(1, 1), torch.bfloat16)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        silu_and_mul(torch.zeros(4, 16, dtype=torch.bfloat16))


def test_missing_library_fails_loudly(monkeypatch):
    import sglang_b200._lib as L
    monkeypatch.setattr(L, "_lib", None)
    monkeypatch.setattr(L, "LIB_PATH", "/nonexistent/libsglb200.so")
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        L.lib()


@pytest.mark.parametrize("fmt", ["bf16", "f16"])
def test_fma_division_matches_ieee_on_a_sample(tmp_path, fmt):
    """tests/csrc/check_quant_math.cpp with stride 97 (the full run, stride 1, takes ~15 s per format)."""
    exe = str(tmp_path / "check_quant_math")
    subprocess.check_call(["g++", "-O2", "-fopenmp", "-x", "c++", "-o", exe,
                           os.path.join(ROOT, "tests", "csrc", "check_quant_math.cpp"),
                           "-L/usr/lib/gcc/x86_64-linux-gnu/13", "-lgomp"])
    out = subprocess.run([exe, fmt, "97"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    assert "code_mismatch=0" in out.stdout and "scale_mismatch=0" in out.stdout


def test_linear_method_create_weights_checks():
    from sglang_b200.layers.quantization import Fp8Config, Fp8LinearMethod
    cfg = Fp8Config.from_config({"quant_method": "fp8", "activation_scheme": "dynamic", "weight_block_size": [128, 128]})
    layer = torch.nn.Module()
    Fp8LinearMethod(cfg, tp_size=1).create_weights(layer, 7168, [576], 7168, 576, torch.bfloat16)
    assert layer.weight.shape == (576, 7168) and layer.weight.dtype == torch.float8_e4m3fn
    assert layer.weight_scale_inv.shape == (5, 56) and layer.input_scale is None
    with pytest.raises(ValueError, match="block_k"):
        Fp8LinearMethod(cfg, tp_size=8).create_weights(torch.nn.Module(), 200, [512], 1600, 512, torch.bfloat16)
    with pytest.raises(ValueError, match="block_n"):
        Fp8LinearMethod(cfg, tp_size=1).create_weights(torch.nn.Module(), 1024, [192, 192], 1024, 384, torch.bfloat16)
    with pytest.raises(ValueError):
        Fp8Config(weight_block_size=[64, 64])
    with pytest.raises(ValueError):
        Fp8Config(activation_scheme="static")


def test_scale_allocator_layouts():
    from sglang_b200.layers.quantization import create_per_token_group_quant_fp8_output_scale as alloc
    assert alloc((6, 640), "cpu", 128, False, False, False).stride() == (5, 1)
    assert alloc((6, 640), "cpu", 128, True, False, False).stride() == (1, 6)
    t = alloc((6, 640), "cpu", 128, True, True, False)
    assert t.shape == (6, 5) and t.stride() == (1, 8)
    u = alloc((6, 640), "cpu", 128, True, True, True)
    assert u.dtype == torch.int32 and u.shape == (6, 2) and u.stride() == (1, 8)


def test_host_validation_of_routing_and_exchange_entries(built_lib):
    """The routing, masked-layout and peer-exchange entry points check their arguments before touching a device too."""
    import ctypes
    from sglang_b200._lib import lib
    L = lib()
    detail = lambda: L.sglb200_last_error_detail().decode()
    assert L.sglb200_topk_softmax(None, 2, None, None, 4, 2048, 2, 0, None) == -1 and "num_experts" in detail()
    assert L.sglb200_topk_softmax(None, 2, None, None, 4, 8, 9, 0, None) == -1 and "topk" in detail()
    assert L.sglb200_topk_softmax(None, 2, None, None, 0, 8, 2, 0, None) == 0
    assert L.sglb200_moe_fused_gate(None, None, 2, None, None, 4, 256, 7, 4, 8, 0, 2.5, 0, None) == -1
    assert "num_expert_group" in detail()
    assert L.sglb200_moe_fused_gate(None, None, 2, None, None, 4, 256, 8, 4, 8, 2, 0.0, 0, None) == -1
    assert "routed_scaling_factor" in detail()
    assert L.sglb200_moe_align_block_size(None, 1 << 25, 9, 16, None, None, None, None, 0, None) == -1
    assert L.sglb200_moe_sum_reduce(None, None, 4, 2, 100, 0, 1.0, None) == -1 and "multiple of 8" in detail()
    assert L.sglb200_moe_sum_reduce(None, None, 0, 2, 128, 0, 1.0, None) == 0
    assert L.sglb200_fp8_blockwise_scaled_masked_grouped_mm(None, None, None, None, None, None, 4, 64, 128, 128, 128, 128,
                                                            128 * 128, 128, 64, 1, 1, 1, 1, 1, 0, None) == -6
    assert "masked_m" in detail()
    assert L.sglb200_group_quant_fp8_batched(None, 2, None, None, 4, 16, 256, 128, 1e-10, -448.0, 448.0, 0, 0, None, 32, 2,
                                             1, None) == -1 and "16-bit" in detail()
    ptrs = (ctypes.c_void_p * 2)(None, None)
    assert L.sglb200_fp8_blockwise_scaled_mm_push(None, None, None, None, 64, 512, 256, 256, 256, 2, 1, 2, 1, 0, ptrs, ptrs,
                                                  0, 2, 1024, None, 0, None) == -7 and "receive slot" in detail()
    assert L.sglb200_fp8_blockwise_scaled_mm_push(None, None, None, None, 64, 512, 256, 256, 256, 2, 1, 2, 1, 0, ptrs, ptrs,
                                                  3, 2, 64 * 512, None, 0, None) == -1 and "rank" in detail()
    assert L.sglb200_peer_reduce(None, None, None, 64, 500, 512, 0, 2, 64 * 512, 0, None) == -1
    assert L.sglb200_fp8_blockwise_scaled_mm_push_scatter(None, None, None, None, 64, 128, 256, 256, 256, 2, 1, 2, 1, 0,
                                                          ptrs, ptrs, 0, 2, 64 * 128, None) == -1
    assert "fewer output tiles than ranks" in detail()
    assert L.sglb200_peer_reduce_scatter(ptrs, ptrs, None, 256, 512, 512, 0, 0, 2, 1024, 0, None) == -7
    assert L.sglb200_peer_gather(None, None, None, 256, 512, 512, 0, 0, 2, 256 * 512, 0, None) == -6
    assert L.sglb200_ep_dispatch(None, None, 2, 1, None, None, 4, 200, 2, 4, ptrs, 0, 2, 16, 16, None) == -1
    assert "multiple of 128" in detail()
    assert L.sglb200_ep_dispatch(None, None, 2, 1, None, None, 40, 256, 2, 4, ptrs, 0, 2, 16, 16, None) == -6
    assert L.sglb200_ep_dispatch_quant(None, 2, 256, None, None, 4, 256, 2, 4, ptrs, 0, 2, 16, 16, 1e-10, None) == -5
    assert L.sglb200_ep_dispatch_quant(None, 0, 100, None, None, 4, 256, 2, 4, ptrs, 0, 2, 16, 16, 1e-10, None) == -1
    assert "ldx" in detail()
    assert L.sglb200_ep_combine_reduce(ptrs, 0, 9, None, None, 0, 4, 256, 2, 4, 16, 16, 0, None) == -1
    assert L.sglb200_ep_buffer_bytes(16, 256, 2, 2, 16) > 16 * 256 and L.sglb200_ep_buffer_bytes(0, 256, 2, 2, 16) == 0
    assert L.sglb200_peer_flag_bytes() > 0 and L.sglb200_peer_recv_bytes(1024) == 2 * 8 * 1024 * 2
    assert L.sglb200_fp8_blockwise_scaled_mm_push_workspace_bytes(129, 7168, 8192) == 0
    h = (ctypes.c_ubyte * 64)()
    assert L.sglb200_peer_alloc(0, None, h) == -6 and L.sglb200_peer_open(None, None) == -6
    assert L.sglb200_peer_close(None) == 0 and L.sglb200_peer_free(None) == 0


def test_peer_ep_exchange_refuses_a_receive_buffer_that_could_overflow():
    """capacity < world * m_max is refused before anything is allocated (no GPU needed to see the refusal)."""
    from sglang_b200.distributed.peer_ep import PeerEpExchange
    with pytest.raises(ValueError, match="capacity"):
        PeerEpExchange(capacity=10, hidden=256, topk=2, m_max=11, device="cpu")


def test_num_sms_limit_round_trip(built_lib):
    """The SM bound is plain host state: settable and readable without a GPU; a negative value is refused."""
    from sglang_b200._lib import lib
    L = lib()
    assert L.sglb200_set_num_sms(-1) == -1
    assert L.sglb200_set_num_sms(132) == 0
    assert L.sglb200_get_num_sms() == 132
    assert L.sglb200_set_num_sms(0) == 0
    assert L.sglb200_get_num_sms() != 132


def test_symm_mem_communicator_is_disabled_without_a_gpu():
    """The reference's wrapper stays disabled and declines when a prerequisite is missing
    (``device_communicators/symm_mem.py:46-47,113-123``); so does this one, and the row-parallel layer then takes the
    collective library's all-reduce."""
    import torch
    from sglang_b200.distributed import SymmMemCommunicator
    comm = SymmMemCommunicator(None, "cpu")
    assert comm.disabled and comm.all_reduce(torch.zeros(8, dtype=torch.bfloat16)) is None
    assert not comm.should_symm_mem_allreduce(torch.zeros(8, dtype=torch.bfloat16))
    with pytest.raises(RuntimeError):
        comm.view((8,))
    comm.close()


def test_host_validation_of_the_multicast_and_few_rows_entries(built_lib):
    """The multicast all-reduce, the GEMM with the all-reduce in its launch and the kernel-selection setters refuse bad
    arguments on the host, before any device is touched."""
    import ctypes
    from sglang_b200._lib import lib
    L = lib()
    detail = lambda: L.sglb200_last_error_detail().decode()
    flags = (ctypes.c_uint64 * 8)(*([4096] * 8))
    assert L.sglb200_nvls_flag_bytes() == (2 * 8 * 128 + 128) * 4
    assert L.sglb200_nvls_all_reduce(4096, flags, 0, 1, 64, 0, 0, None) == -1 and "world" in detail()
    assert L.sglb200_nvls_all_reduce(4096, flags, 2, 2, 64, 0, 0, None) == -1 and "rank" in detail()
    assert L.sglb200_nvls_all_reduce(4096, flags, 0, 2, 60, 0, 0, None) == -1 and "multiple of 8" in detail()
    assert L.sglb200_nvls_all_reduce(4096, flags, 0, 2, 64, 2, 0, None) == -5          # fp32 is not a dtype it adds
    assert L.sglb200_nvls_all_reduce(4096, flags, 0, 2, 64, 0, 129, None) == -1 and "blocks" in detail()
    assert L.sglb200_nvls_all_reduce(4096, flags, 0, 2, 0, 0, 0, None) == 0             # nothing to add
    assert L.sglb200_nvls_all_reduce(0, flags, 0, 2, 64, 0, 0, None) == -6
    assert L.sglb200_nvls_all_reduce(4104, flags, 0, 2, 64, 0, 0, None) == -2           # not 16-byte aligned
    mm = L.sglb200_fp8_blockwise_scaled_mm_allreduce
    args = lambda **kw: [kw.get(k, v) for k, v in dict(a=None, b=None, sa=None, sb=None, out=None, mc=4096, flags=flags,
                                                       done=None, rank=0, world=2, ctas=16, M=256, N=512, K=1024, lda=1024,
                                                       ldb=1024, sam=1, sak=256, sbn=8, sbk=1, dt=0, st=None).items()]
    assert mm(*args(world=9)) == -1 and "ranks" in detail()
    assert mm(*args(ctas=0)) == -1 and "comm_ctas" in detail()
    assert mm(*args(ctas=65)) == -1
    assert mm(*args(K=1000)) == -1 and "multiple of 16" in detail()
    assert mm(*args(dt=2)) == -5
    assert mm(*args(M=0)) == 0
    assert mm(*args(M=64 * 16 * 128 + 1)) == -1 and "row blocks" in detail()
    assert mm(*args()) == -6                                                          # NULL operands
    before = L.sglb200_get_grouped_few_rows()
    assert L.sglb200_set_grouped_few_rows(65) == -1 and L.sglb200_set_grouped_few_rows(-1) == -1
    assert L.sglb200_set_grouped_few_rows(0) == 0 and L.sglb200_get_grouped_few_rows() == 0
    assert L.sglb200_set_grouped_few_rows(before) == 0 and L.sglb200_get_grouped_few_rows() == before == 20


@pytest.mark.parametrize("M,N,K,served", [
    (65, 8192, 8192, True), (128, 8192, 8192, True), (74, 7168, 16384, True), (117, 7168, 18432, True),
    (103, 5120, 2560, True), (128, 576, 7168, True), (118, 7168, 16384, False), (128, 7168, 16384, False),
    (240, 5888, 18432, True), (684, 2048, 28672, True), (2978, 512, 28672, True)])
def test_shapes_the_no_allocation_entry_takes(built_lib, M, N, K, served):
    """The refusal comes before any pointer is looked at: a served shape gets past it and fails on the NULL operands (or,
    with scratch, on the missing device).  The sizes lie on both sides of 16 MiB of partial sums, and above 128 rows where
    a split would be larger than that but the tiles alone occupy the SMs (the answers are those for 148 SMs, which the
    library assumes without a device)."""
    from sglang_b200._lib import lib
    L = lib()
    if L.sglb200_get_num_sms() not in (0, 148):
        pytest.skip("sizes chosen for 148 SMs")
    rc = L.sglb200_fp8_blockwise_scaled_mm_noalloc(None, None, None, None, None, M, N, K, K, K, N, 1, M, K // 128, 1, 0, None)
    assert (rc != -7) == served and rc != 0
    if M <= 128:
        assert (L.sglb200_fp8_blockwise_scaled_mm_workspace_bytes(M, N, K) <= 16 << 20) == served


def test_few_rows_limit_of_twenty_itself(built_lib):
    """20 stands for the library's rule; with the mark it is the limit itself, and what the getter answers restores either."""
    import ctypes
    from sglang_b200._lib import lib
    L, exact = lib(), 0x100
    chunk = L.sglb200_debug_grouped_chunk
    chunk.argtypes, chunk.restype = [ctypes.c_int64] * 6 + [ctypes.c_int], ctypes.c_int
    average = lambda rows, k=2048, ue8m0=0: chunk(rows * 64, 64, 0, 0, 7168, k, ue8m0)
    before = L.sglb200_get_grouped_few_rows()
    try:
        assert before == 20 and [average(r) for r in (20, 21, 48, 49)] == [32, 32, 64, 0]
        assert average(20, ue8m0=1) == 32 and average(21, ue8m0=1) == 0
        assert L.sglb200_set_grouped_few_rows(20 | exact) == 0
        assert [average(r) for r in (20, 21, 48)] == [32, 0, 0] and average(20, 512, 1) == 32
        mark = L.sglb200_get_grouped_few_rows()
        assert L.sglb200_set_grouped_few_rows(30 | exact) == 0 and L.sglb200_get_grouped_few_rows() == 30
        assert average(30) == 64 and average(31) == 0
        assert L.sglb200_set_grouped_few_rows(mark) == 0 and average(21) == 0
        assert L.sglb200_set_grouped_few_rows(65 | exact) == -1 and L.sglb200_set_grouped_few_rows(0x200 | 20) == -1
        assert L.sglb200_set_grouped_few_rows(0) == 0 and average(1) == 0
    finally:
        assert L.sglb200_set_grouped_few_rows(before) == 0
    assert average(48) == 64


@pytest.mark.parametrize("rows,experts,n,k,chunk", [
    (64, 64, 2048, 256, 16), (1280, 64, 2048, 512, 32), (32, 32, 7168, 512, 16), (128, 32, 7168, 128, 0),
    (256, 256, 7168, 256, 0), (5120, 256, 7168, 512, 0), (256, 256, 7168, 640, 16), (5120, 256, 7168, 2048, 32), (1, 256, 7168, 128, 16)])
def test_short_k_leaves_the_few_rows_kernel_only_in_large_layers(built_lib, rows, experts, n, k, chunk):
    """UE8M0 grouped GEMM with K of at most 512: small layers stay with the few-rows kernel, on both sides of the bound."""
    import ctypes
    from sglang_b200._lib import lib
    fn = lib().sglb200_debug_grouped_chunk
    fn.argtypes, fn.restype = [ctypes.c_int64] * 6 + [ctypes.c_int], ctypes.c_int
    assert fn(rows, experts, 0, 0, n, k, 1) == chunk


@pytest.mark.parametrize("M,N,K,ranges", [(1, 576, 7168, 0), (128, 576, 7168, 0), (128, 7168, 16384, 0), (129, 576, 7168, 8),
                                          (4096, 7168, 16384, 0)])
def test_scratch_that_a_dense_call_uses(built_lib, M, N, K, ranges):
    """What the wrappers allocate: nothing where K is added up on the chip or not cut, else one fp32 output per range.  The
    linear layer's scratch holds the same."""
    from sglang_b200._lib import lib
    L = lib()
    used = L.sglb200_fp8_blockwise_scaled_mm_scratch_bytes(M, N, K)
    assert used == ranges * M * N * 4 and used <= L.sglb200_fp8_blockwise_scaled_mm_workspace_bytes(M, N, K)
    if M > 2:
        rest = (K // 128) * (-(-M // 4) * 4) * 4 + M * K
        assert used + rest <= L.sglb200_fp8_block_linear_scratch_bytes(M, N, K, 0) <= used + rest + 1024


@pytest.mark.parametrize("M", [1, 2])
def test_one_or_two_rows_under_their_own_output_are_refused_without_scratch(built_lib, M):
    """At one or two rows the GEMM reads x while it stores: an output that overlaps x is refused before anything else happens, one
    that only touches it is not (the pointers are never read here)."""
    from sglang_b200._lib import lib
    L, N, K, x = lib(), 512, 1024, 1 << 20
    call = lambda out: L.sglb200_fp8_block_linear(x, 1 << 24, 1 << 25, None, out, M, N, K, 8, 1, 0, 1e-10, 0, None, 0, None)
    assert [call(out) for out in (x, x + 16, x + M * K * 2 - 16, x - M * N * 2 + 16)] == [-7] * 4
    assert "overlaps" in L.sglb200_last_error_detail().decode()
    if not torch.cuda.is_available():
        assert all(call(out) not in (0, -7) for out in (x + M * K * 2, x - M * N * 2))  # no device here


def test_host_path_reports_integers_out_of_range(built_lib):
    """An integer argument that does not fit is an OverflowError, raised before anything is launched, and leaves no pending
    exception behind."""
    from sglang_b200._lib import host
    t = torch.zeros(2, 4)
    with pytest.raises(OverflowError):
        host().topk_softmax(t, 1 << 80, True)
    with pytest.raises(OverflowError):
        host().grouped_masked(t, t, t, t, t, t, 1 << 80)
    assert host().topk_softmax(t, 1, True) is None  # a CPU tensor: left to the Python route


def test_linear_method_takes_a_layer_that_is_no_module(built_lib):
    """Only ``weight`` and ``weight_scale_inv`` are asked of the layer; CPU tensors are then refused by the op itself."""
    from types import SimpleNamespace
    from sglang_b200.layers.quantization.fp8 import Fp8Config, Fp8LinearMethod
    layer = SimpleNamespace(weight=torch.zeros(128, 128).to(torch.float8_e4m3fn), weight_scale_inv=torch.ones(1, 1))
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        Fp8LinearMethod(Fp8Config()).apply(layer, torch.zeros(2, 128, dtype=torch.bfloat16))


def test_host_path_leaves_tensors_without_plain_memory_alone(built_lib):
    """Traced tensors (static and symbolic sizes) and sparse ones that claim to be on a GPU: every function of the host path
    answers None and the process lives.  In a child process, which an exception escaping from C++ would end."""
    code = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.symbolic_shapes import ShapeEnv
from sglang_b200._lib import host
mode = FakeTensorMode(shape_env=ShapeEnv())
with mode:
    n = mode.shape_env.create_unbacked_symint()
    w = torch.empty(128, 128, dtype=torch.float8_e4m3fn, device="cuda")
    s = torch.empty(1, 1, device="cuda")
    xs = [torch.empty(r, 128, dtype=torch.bfloat16, device="cuda") for r in (4, n)]
    xs.append(torch.sparse_coo_tensor(torch.zeros(2, 1, dtype=torch.int64, device="cuda"),
                                      torch.ones(1, dtype=torch.bfloat16, device="cuda"), (4, 128)))
h = host()
for x in xs:
    assert x.is_cuda
    assert h.block_linear(x, w, s, None, False) is None and h.block_linear(x, w, s, x, True) is None
    assert h.quant(x, 128, 1e-10, -448.0, 448.0, False, False, False, False, None) is None
    assert h.topk_softmax(x, 2, True) is None
    assert h.fused_experts(x, x, x, x, x, x, x, 1.0, None, False) is None
    assert h.grouped_masked(x, x, x, x, x, x, 1) is None
print("alive")
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "alive", r.stderr[-2000:]
