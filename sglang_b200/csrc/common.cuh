// Shared host/device plumbing: status codes, argument checks, launch error capture.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/sglb200.h"

namespace sglb {

// Thread-local text of the last failed host-side check.
char* error_buffer();
int fail(int code, const char* fmt, ...);
// Name of the GEMM kernel that this thread launched last (sglb200_last_gemm_kernel); a string literal.
void note_gemm(const char* kernel);

// Number of SMs and compute capability of the current device, cached per device.
struct DeviceInfo {
  int sm_count;
  int cc_major;
  int cc_minor;
  int max_smem_optin;
};
int device_info(DeviceInfo* out);  // returns SGLB200_OK or an error code

// Tensor map of a rank-2 or rank-3 byte tensor with innermost extent dims[0] (K), 128-byte-swizzled boxes of
// [box_rows x 128 bytes].  Defined in gemm.cu.
int make_map_sw128(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                   uint32_t box_rows, CUtensorMapL2promotion promo);

// Tensor map of an fp32 [rows][cols] tensor (scales), boxes of box_cols x 1.  Defined in gemm.cu.
int make_map_f32(CUtensorMap* map, const void* base, uint64_t cols, uint64_t rows, uint64_t stride_bytes, uint32_t box_cols);

// Tensor map of a [rows][cols] tensor of 16-bit results for TMA stores.  Defined in gemm.cu.
int make_map_out16(CUtensorMap* map, void* base, uint64_t cols, uint64_t rows, uint64_t stride_bytes, uint32_t box_cols, uint32_t box_rows);

// The few-rows (M <= smallm_max_rows()) weight-streaming GEMM, gemm_smallm.cu
int smallm_max_rows();
constexpr int kMaxCluster = 8;
int smallm_cluster(int64_t M, int64_t N, int64_t K, int sm_count, bool ue8m0);  // CTAs that share a tile's K, 1..kMaxCluster
int64_t tile_cost(int64_t M, int64_t N, int64_t K, int sm_count);  // what the tile kernel is expected to take, ns, K cut or not
bool takes_few_rows(int64_t M, int64_t N, int64_t K, int sm_count, bool ue8m0);  // a dense call of either scale kind runs on it
int smallm_splits(int64_t N, int64_t K, int sm_count);  // K ranges of a split through memory: sizes scratch, see there
// Rows that are not quantised yet: `a` of smallm_gemm is [M, K] of the output type, contiguous, K in whole groups of 128, and the
// kernel quantises them itself with this floor; M <= kMaxQuantRows, `sa` and `partial` unused
struct RawRows {
  float eps;
};
int smallm_quant_rows();
constexpr int kMaxQuantRows = 8;
bool smallm_quantises(int64_t M, int64_t N, int sm_count);
int smallm_gemm(const void* a, const void* b, const float* sa, const float* sb, void* out, int64_t M, int64_t N, int64_t K,
                int64_t lda, int64_t ldb, int64_t ldc, int64_t sa_stride_m, int64_t sa_stride_k, int64_t sb_stride_n,
                int64_t sb_stride_k, int out_dtype, const void* bias, float* partial, int64_t partial_floats, int sm_count,
                void* stream, int* splits_used, bool ue8m0, const RawRows* raw = nullptr);
void launch_splitk_reduce(const float* partial, void* out, const void* bias, int64_t M, int64_t N, int64_t ldc, int splits,
                          int out_dtype, int sm_count, void* stream);  // gemm.cu
// Per-token-group quantisation (groups of 128) of the linear layer's rows, quant.cu: the GEMM after it may start beside it
int quant_rows(const void* input, int in_dtype, void* out_q, void* out_s, int64_t rows, int64_t hidden, float eps, bool ue8m0,
               int64_t s_stride_row, int64_t s_stride_group, void* stream);
// The UE8M0 GEMM of the linear layer, gemm_ue8m0.cu
int ue8m0_linear_gemm(const void* a, const void* b, const int32_t* sfa, const int32_t* sfb, const void* bias, void* out, int64_t M,
                      int64_t N, int64_t K, int64_t sfa_ld, int64_t sfb_stride_n, int64_t sfb_stride_k, int out_dtype,
                      void* stream, float* workspace, int64_t workspace_floats);
int ue8m0_splits(int64_t M, int64_t N, int64_t K, int sm_count);  // with `workspace` of that many [M][N] fp32 sums
// The same GEMM on CTA pairs (256 x 224 tiles), gemm_ue8m0_pair.cu
int64_t ue8m0_pair_cost(int64_t M, int64_t N, int64_t K, int sm_count);
int ue8m0_pair_gemm(const void* a, const void* b, const int32_t* sfa, const int32_t* sfb, const void* bias, void* out, int64_t M, int64_t N,
                    int64_t K, int64_t lda, int64_t ldb, int64_t ldc, int64_t sfa_ld, int64_t sfb_stride_n, int64_t sfb_stride_k,
                    int out_dtype, int sm_count, void* stream);
int smallm_take_device_status();
int nvls_take_device_status();  // nvls.cu
constexpr int kGroupedFewRowsDefault = 20;  // stands for the library's rule; the limit 20 itself carries SGLB200_FEW_ROWS_EXACT
extern int g_grouped_few_rows_max;  // common.cu; as given to sglb200_set_grouped_few_rows
// The grouped form of the few-rows kernel (one weight matrix per expert, few rows per expert); chunk 0 = do not use it
int smallm_grouped_chunk(int64_t total_rows, int64_t num_experts, int64_t rows_per_expert, int64_t expected_rows, int64_t N, int64_t K,
                         bool ue8m0);
int smallm_grouped_gemm(int chunk, const void* a, const void* b, const float* sa, const float* sb, void* out,
                        const int32_t* expert_offsets, const int32_t* problem_sizes, int count_stride, int64_t total_rows,
                        int64_t num_experts, int64_t rows_per_expert, int64_t N, int64_t K, int64_t lda, int64_t ldb,
                        int64_t ldb_e, int64_t ldc, int64_t sa_stride_e, int64_t sa_stride_m, int64_t sa_stride_k,
                        int64_t sb_stride_e, int64_t sb_stride_n, int64_t sb_stride_k, int out_dtype, int sm_count,
                        void* stream, bool ue8m0);

// Dense GEMM on CTA pairs (256 x 256 tiles), gemm_pair.cu
int pair_gemm(const void* a, const void* b, const float* sa, const float* sb, void* out, int64_t M, int64_t N, int64_t K,
              int64_t lda, int64_t ldb, int64_t ldc, int64_t sa_stride_m, int64_t sa_stride_k, int64_t sb_stride_n,
              int64_t sb_stride_k, int out_dtype, const void* bias, int sm_count, void* stream);

bool pair_takes_scales(const float* sa, int64_t M, int64_t sa_stride_m, int64_t sa_stride_k);
// The dense GEMM on 128 x 128 tiles at any size, K uncut, gemm.cu: the pair entry's way out for other scale layouts
int tile_gemm(const void* a, const void* b, const float* sa, const float* sb, void* out, int64_t M, int64_t N, int64_t K, int64_t lda,
              int64_t ldb, int64_t ldc, int64_t sa_stride_m, int64_t sa_stride_k, int64_t sb_stride_n, int64_t sb_stride_k,
              int out_dtype, void* stream);

// Launch with programmatic stream serialization allowed: the kernel may begin before the previous kernel of the stream
// has finished and must call ptx::grid_dep_wait() before it touches anything that kernel writes or reads.  With cluster > 1
// in clusters of that many CTAs.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                      int cluster, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  return launch_pdl_cluster(kernel, grid, block, smem, stream, 1, args...);
}

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

#define SGLB_CHECK_LAUNCH(what)                                                                   \
  do {                                                                                            \
    cudaError_t e__ = cudaGetLastError();                                                         \
    if (e__ != cudaSuccess) return ::sglb::fail(SGLB200_ERR_LAUNCH, "%s: %s", what, cudaGetErrorString(e__)); \
  } while (0)

#define SGLB_REQUIRE(cond, code, ...)                       \
  do {                                                      \
    if (!(cond)) return ::sglb::fail(code, __VA_ARGS__);    \
  } while (0)

}  // namespace sglb
