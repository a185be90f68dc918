// Integer routing tables and the HBM-bound row movers around the grouped GEMMs:
// prepare_moe_input (stable counting sort by expert), shuffle_rows (row gather),
// apply_shuffle_mul_sum (weighted top-k combine) and silu_and_mul.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"
#include "quant_math.cuh"
#include "quant_vec.cuh"

namespace sglb {
namespace {

// ------------------------------------------------------------------------------------------
// prepare_moe_input: one block per expert, no exchange between blocks.  Every block reads all ids (from L2): the ids below
// its expert give the expert's first row, its own ids, taken in order, the rows, so rows of one expert stay in ascending slot
// order (a stable sort).  Warp w owns a contiguous slice of the ids and 128 of them per step.  Reading the ids once per expert is
// far cheaper than walking them once: one block with __match_any_sync took 73 us for 32768 ids and 256 experts.
// ------------------------------------------------------------------------------------------
constexpr int kPrepThreads = 512;
constexpr int kPrepWarps = kPrepThreads / 32;

template <bool VEC>
__device__ __forceinline__ int4 load_ids4(const int32_t* __restrict__ ids, int32_t i, int32_t end) {
  if (VEC && i + 3 < end) return __ldg(reinterpret_cast<const int4*>(ids + i));
  return make_int4(i < end ? __ldg(ids + i) : -1, i + 1 < end ? __ldg(ids + i + 1) : -1, i + 2 < end ? __ldg(ids + i + 2) : -1,
                   i + 3 < end ? __ldg(ids + i + 3) : -1);
}

template <bool VEC>
__global__ void __launch_bounds__(kPrepThreads)
prepare_moe_input_kernel(const int32_t* __restrict__ topk_ids, int32_t* __restrict__ expert_offsets,
                         int32_t* __restrict__ ps1, int32_t* __restrict__ ps2, int32_t* __restrict__ a_map,
                         int32_t* __restrict__ c_map, int32_t len, int32_t topk, int32_t E, int32_t n, int32_t k) {
  __shared__ int32_t s_eq[kPrepWarps], s_less[kPrepWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t e = blockIdx.x;
  const int32_t chunk = ((len + kPrepWarps - 1) / kPrepWarps + 127) / 128 * 128;
  const int32_t c0 = min(warp * chunk, len), c1 = min(c0 + chunk, len);
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();  // the ids come from the router

  int32_t eq = 0, less = 0;
#pragma unroll 4
  for (int32_t i = c0 + lane * 4; i < c1; i += 128) {
    const int4 v = load_ids4<VEC>(topk_ids, i, c1);
    eq += ((uint32_t)v.x == e) + ((uint32_t)v.y == e) + ((uint32_t)v.z == e) + ((uint32_t)v.w == e);
    less += ((uint32_t)v.x < e) + ((uint32_t)v.y < e) + ((uint32_t)v.z < e) + ((uint32_t)v.w < e);
  }
  eq = __reduce_add_sync(0xffffffffu, eq);
  less = __reduce_add_sync(0xffffffffu, less);
  if (lane == 0) {
    s_eq[warp] = eq;
    s_less[warp] = less;
  }
  __syncthreads();
  int32_t start = 0, total = 0, base = 0;
#pragma unroll
  for (int w = 0; w < kPrepWarps; ++w) {
    start += s_less[w];
    if (w < warp) base += s_eq[w];
    total += s_eq[w];
  }
  base += start;
  if (threadIdx.x == 0) {
    if (e == 0) expert_offsets[0] = 0;
    expert_offsets[e + 1] = start + total;
    if (ps1) { ps1[e * 3] = total; ps1[e * 3 + 1] = 2 * n; ps1[e * 3 + 2] = k; }
    if (ps2) { ps2[e * 3] = total; ps2[e * 3 + 1] = k; ps2[e * 3 + 2] = n; }
  }
  const uint32_t before = (1u << lane) - 1u;
  for (int32_t i0 = c0; i0 < c1; i0 += 128) {
    const int32_t i = i0 + lane * 4;
    const int4 v4 = load_ids4<VEC>(topk_ids, i, c1);
    const int32_t v[4] = {v4.x, v4.y, v4.z, v4.w};
    uint32_t hit[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) hit[j] = __ballot_sync(0xffffffffu, (uint32_t)v[j] == e);
    if (hit[0] | hit[1] | hit[2] | hit[3]) {  // uniform
      int32_t pos = base + __popc(hit[0] & before) + __popc(hit[1] & before) + __popc(hit[2] & before) + __popc(hit[3] & before);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if ((uint32_t)v[j] == e) {
          a_map[pos] = (i + j) / topk;
          c_map[i + j] = pos;
          ++pos;
        }
        base += __popc(hit[j]);
      }
    }
    if (e == 0) {  // ids of no expert here
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (i + j < c1 && (uint32_t)v[j] >= (uint32_t)E) c_map[i + j] = -1;
    }
  }
  // rows past the last routed one (only when some ids were out of range)
  if (e + 1 == (uint32_t)E)
    for (int32_t i = start + total + (int32_t)threadIdx.x; i < len; i += kPrepThreads) a_map[i] = 0;
}

// ------------------------------------------------------------------------------------------
// The activations of the expert layer, quantised once per token and written to every row the token has in expert order: one
// pass instead of quantiser, row gather and scale gather.  One block per token; a group of 128 is eight lanes of 16 elements.
// ------------------------------------------------------------------------------------------
constexpr int kScatterThreads = 256;
constexpr int kScatterMaxTopk = 32;

template <typename T, bool UE8M0>
__global__ void __launch_bounds__(kScatterThreads)
quant_scatter_kernel(const T* __restrict__ x, const int32_t* __restrict__ c_map, uint8_t* __restrict__ out_q,
                     void* __restrict__ out_s, int32_t H, int32_t topk, float eps) {
  __shared__ int32_t s_row[kScatterMaxTopk];
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int64_t t = blockIdx.x;
  if ((int)threadIdx.x < topk) s_row[threadIdx.x] = __ldg(c_map + t * topk + threadIdx.x);
  __syncthreads();
  const int32_t G = H / 128;
  const int sub = threadIdx.x & 7;
  const float inv_max = __frcp_rn(448.0f);
  const uint4* row = reinterpret_cast<const uint4*>(x + t * H);
  for (int32_t g0 = 0; g0 < G; g0 += kScatterThreads / 8) {
    const int32_t g = g0 + (threadIdx.x >> 3);
    const bool live = g < G;
    uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
    if (live) {
      v0 = __ldg(row + g * 16 + sub * 2);
      v1 = __ldg(row + g * 16 + sub * 2 + 1);
    }
    float amax = fmaxf(eps, fmaxf(Elem<T>::vec_absmax(v0), Elem<T>::vec_absmax(v1)));
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
    const float s = group_scale_fast(amax, 448.0f, inv_max, UE8M0);
    if (!live) continue;
    const uint4 codes = encode16_e4m3<T>(v0, v1, s);
    for (int32_t j = 0; j < topk; ++j) {
      const int64_t r = s_row[j];
      if (r < 0) continue;
      reinterpret_cast<uint4*>(out_q + r * H)[g * 8 + sub] = codes;
      if (sub == 0) {
        if constexpr (UE8M0) {
          const int32_t words = (G + 3) / 4;
          uint8_t* wp = static_cast<uint8_t*>(out_s) + 4 * (r * words + (g >> 2));
          wp[g & 3] = (uint8_t)(__float_as_uint(s) >> 23);
          if (g + 1 == G)
            for (int z = (g & 3) + 1; z < 4; ++z) wp[z] = 0;  // bytes of the word past the last group
        } else {
          static_cast<float*>(out_s)[r * G + g] = s;
        }
      }
    }
  }
}

// ------------------------------------------------------------------------------------------
// shuffle_rows: one warp per destination row, 16-byte (or 4-byte) pieces
// ------------------------------------------------------------------------------------------
template <typename V>
__global__ void __launch_bounds__(256)
shuffle_rows_kernel(const V* __restrict__ in, const int32_t* __restrict__ map, V* __restrict__ out, int64_t n_dst,
                    int64_t row_vecs) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * 8;
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < n_dst; r += warps) {
    const V* src = in + (int64_t)map[r] * row_vecs;
    V* dst = out + r * row_vecs;
    for (int64_t c = lane; c < row_vecs; c += 32) dst[c] = __ldg(src + c);
  }
}

// ------------------------------------------------------------------------------------------
// apply_shuffle_mul_sum and silu_and_mul
// ------------------------------------------------------------------------------------------
template <typename T>
struct Cvt;
template <>
struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float f(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 t(float x) { return __float2bfloat16_rn(x); }
};
template <>
struct Cvt<__half> {
  static __device__ __forceinline__ float f(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half t(float x) { return __float2half_rn(x); }
};

// ROUND: each product is rounded to T before it is added (the torch-native expert-MLP reference sums
// bf16 products); otherwise products stay in fp32 (the reference's CUDA combine kernel).  The factor of a slot is
// factors[slot], or T(weights[slot] * scale) from the router's fp32 weights, or 1.  The rows and factors of eight slots are read
// first and their pieces of the row requested together, so that the sum waits for HBM once per eight slots and not once per
// slot.
constexpr int kCombineMax = 512, kCombineSlots = 8;

template <typename T, bool ROUND>
__global__ void __launch_bounds__(kCombineMax)
combine_kernel(const T* __restrict__ in, T* __restrict__ out, const int32_t* __restrict__ perm, const T* __restrict__ factors,
               const float* __restrict__ weights, float scale, int32_t topk, int32_t hidden) {
  __shared__ int32_t s_src[kCombineSlots];
  __shared__ float s_w[kCombineSlots];
  ptx::grid_dep_launch();
  ptx::grid_dep_wait();
  const int64_t i = blockIdx.x;
  const int32_t vecs = hidden / 8;
  const bool small = vecs * 8 != hidden;  // rows of fewer than eight elements
  for (int32_t c0 = 0; c0 < (small ? 1 : vecs); c0 += blockDim.x) {
    const int32_t c = c0 + threadIdx.x;
    float2 acc[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[x] = make_float2(0.f, 0.f);
    for (int32_t j0 = 0; j0 < topk; j0 += kCombineSlots) {
      if (c0 == 0 || topk > kCombineSlots) {  // otherwise the slots of the first pass are still there
        __syncthreads();
        if ((int)threadIdx.x < kCombineSlots) {
          const int32_t j = j0 + threadIdx.x;
          s_src[threadIdx.x] = j < topk ? __ldg(perm + i * topk + j) : -1;
          s_w[threadIdx.x] = j >= topk ? 0.f
                             : factors ? Cvt<T>::f(factors[i * topk + j])
                             : weights ? Cvt<T>::f(Cvt<T>::t(__fmul_rn(__ldg(weights + i * topk + j), scale)))
                                       : 1.f;
        }
        __syncthreads();
      }
      if (small) {
        if ((int)threadIdx.x < hidden)
          for (int j = 0; j < kCombineSlots; ++j)
            if (s_src[j] >= 0) {
              const float v = Cvt<T>::f(in[(int64_t)s_src[j] * hidden + threadIdx.x]);
              if constexpr (ROUND) acc[0].x += Cvt<T>::f(Cvt<T>::t(s_w[j] * v));
              else acc[0].x = fmaf(s_w[j], v, acc[0].x);
            }
        continue;
      }
      if (c >= vecs) continue;
      uint4 u[kCombineSlots];
#pragma unroll
      for (int j = 0; j < kCombineSlots; ++j)
        if (s_src[j] >= 0) u[j] = __ldcs(reinterpret_cast<const uint4*>(in + (int64_t)s_src[j] * hidden) + c);
#pragma unroll
      for (int j = 0; j < kCombineSlots; ++j) {
        if (s_src[j] < 0) continue;
        const float w = s_w[j];
        const uint32_t* h = reinterpret_cast<const uint32_t*>(&u[j]);
        // the factor is a T, so with ROUND the packed product has the bits of the rounded fp32 one; the sums stay fp32
        const uint32_t ww = Elem<T>::pack(w, w);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          if constexpr (ROUND) acc[x] = __fadd2_rn(acc[x], Elem<T>::pair(Elem<T>::mul2(ww, h[x])));
          else acc[x] = __ffma2_rn(make_float2(w, w), Elem<T>::pair(h[x]), acc[x]);
        }
      }
    }
    if (small) {
      if ((int)threadIdx.x < hidden) out[i * hidden + threadIdx.x] = Cvt<T>::t(acc[0].x);
    } else if (c < vecs) {
      reinterpret_cast<uint4*>(out + i * hidden)[c] =
          make_uint4(Elem<T>::pack(acc[0].x, acc[0].y), Elem<T>::pack(acc[1].x, acc[1].y), Elem<T>::pack(acc[2].x, acc[2].y),
                     Elem<T>::pack(acc[3].x, acc[3].y));
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
silu_and_mul_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t rows, int32_t hidden) {
  const int32_t vecs = hidden / 8;
  const int64_t total = rows * vecs;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / vecs;
    const int32_t c = (int32_t)(idx - r * vecs);
    const uint4 g = __ldg(reinterpret_cast<const uint4*>(in + r * 2 * hidden) + c);
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(in + r * 2 * hidden + hidden) + c);
    const T* gh = reinterpret_cast<const T*>(&g);
    const T* uh = reinterpret_cast<const T*>(&u);
    uint4 o;
    T* oh = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float gv = Cvt<T>::f(gh[x]);
      const T s = Cvt<T>::t(__fdiv_rn(gv, 1.0f + expf(-gv)));
      oh[x] = Cvt<T>::t(Cvt<T>::f(s) * Cvt<T>::f(uh[x]));
    }
    reinterpret_cast<uint4*>(out + r * hidden)[c] = o;
  }
}

int check_arch() {
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  SGLB_REQUIRE(di.cc_major == 10, SGLB200_ERR_ARCH, "compute capability %d.%d: this library is built for sm_100a only",
               di.cc_major, di.cc_minor);
  return SGLB200_OK;
}

int combine(const void* input, void* output, const int32_t* perm, const void* factors, const float* weights, float scale, int64_t m,
            int64_t topk, int64_t hidden, int dtype, bool round_products, cudaStream_t st) {
  // as few passes over the row as 512 threads allow, and no idle warp in the last one
  const int64_t vecs = hidden / 8, passes = vecs > 0 ? (vecs + kCombineMax - 1) / kCombineMax : 1;
  const int64_t per = (vecs + passes - 1) / passes;
  const int threads = per < 32 ? 32 : (int)((per + 31) / 32 * 32);
#define SGLB_COMBINE(T, R)                                                                                                  \
  launch_pdl(combine_kernel<T, R>, dim3((unsigned)m), dim3(threads), 0, st, static_cast<const T*>(input), static_cast<T*>(output), \
             perm, static_cast<const T*>(factors), weights, scale, (int32_t)topk, (int32_t)hidden)
  if (dtype == SGLB200_BF16) {
    if (round_products) SGLB_COMBINE(__nv_bfloat16, true); else SGLB_COMBINE(__nv_bfloat16, false);
  } else {
    if (round_products) SGLB_COMBINE(__half, true); else SGLB_COMBINE(__half, false);
  }
#undef SGLB_COMBINE
  SGLB_CHECK_LAUNCH("combine_kernel");
  return SGLB200_OK;
}

int prepare(const int32_t* topk_ids, int32_t* expert_offsets, int32_t* ps1, int32_t* ps2, int32_t* a_map, int32_t* c_map, int64_t len,
            int64_t topk, int64_t E, int64_t n, int64_t k, cudaStream_t st) {
  auto kernel = aligned(topk_ids, 16) ? prepare_moe_input_kernel<true> : prepare_moe_input_kernel<false>;
  launch_pdl(kernel, dim3((unsigned)E), dim3(kPrepThreads), 0, st, topk_ids, expert_offsets, ps1, ps2, a_map, c_map, (int32_t)len,
             (int32_t)topk, (int32_t)E, (int32_t)n, (int32_t)k);
  SGLB_CHECK_LAUNCH("prepare_moe_input_kernel");
  return SGLB200_OK;
}

}  // namespace
}  // namespace sglb

using namespace sglb;

extern "C" int sglb200_prepare_moe_input(const int32_t* topk_ids, int32_t* expert_offsets, int32_t* problem_sizes1,
                                         int32_t* problem_sizes2, int32_t* a_map, int32_t* c_map, int64_t num_tokens,
                                         int64_t topk, int64_t num_experts, int64_t n, int64_t k, void* stream) {
  SGLB_REQUIRE(num_tokens >= 0 && topk >= 1, SGLB200_ERR_SHAPE, "num_tokens=%lld topk=%lld", (long long)num_tokens,
               (long long)topk);
  SGLB_REQUIRE(num_experts >= 1 && num_experts <= 1024, SGLB200_ERR_SHAPE, "num_experts=%lld: 1..1024",
               (long long)num_experts);
  SGLB_REQUIRE(num_tokens * topk <= (1 << 24), SGLB200_ERR_SHAPE, "num_tokens*topk=%lld exceeds 2^24",
               (long long)(num_tokens * topk));
  SGLB_REQUIRE(expert_offsets && a_map && c_map && (topk_ids || num_tokens == 0), SGLB200_ERR_NULL,
               "topk_ids/expert_offsets/a_map/c_map must not be NULL");
  if (int rc = check_arch()) return rc;
  return prepare(topk_ids, expert_offsets, problem_sizes1, problem_sizes2, a_map, c_map, num_tokens * topk, topk, num_experts, n, k,
                 static_cast<cudaStream_t>(stream));
}

extern "C" int sglb200_shuffle_rows(const void* input, const int32_t* dst2src, void* output, int64_t num_dst_rows,
                                    int64_t row_bytes, void* stream) {
  SGLB_REQUIRE(num_dst_rows >= 0 && row_bytes >= 0 && row_bytes % 4 == 0, SGLB200_ERR_SHAPE,
               "num_dst_rows=%lld row_bytes=%lld (must be a multiple of 4)", (long long)num_dst_rows,
               (long long)row_bytes);
  if (num_dst_rows == 0 || row_bytes == 0) return SGLB200_OK;
  SGLB_REQUIRE(input && dst2src && output, SGLB200_ERR_NULL, "input/dst2src/output must not be NULL");
  if (int rc = check_arch()) return rc;
  DeviceInfo di;
  device_info(&di);
  int64_t blocks = (num_dst_rows + 7) / 8;
  const int64_t cap = (int64_t)di.sm_count * 32;
  if (blocks > cap) blocks = cap;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (row_bytes % 16 == 0 && aligned(input, 16) && aligned(output, 16)) {
    shuffle_rows_kernel<uint4><<<(int)blocks, 256, 0, st>>>(static_cast<const uint4*>(input), dst2src,
                                                            static_cast<uint4*>(output), num_dst_rows, row_bytes / 16);
  } else {
    SGLB_REQUIRE(aligned(input, 4) && aligned(output, 4), SGLB200_ERR_ALIGN, "input/output must be 4-byte aligned");
    shuffle_rows_kernel<uint32_t><<<(int)blocks, 256, 0, st>>>(static_cast<const uint32_t*>(input), dst2src,
                                                               static_cast<uint32_t*>(output), num_dst_rows,
                                                               row_bytes / 4);
  }
  SGLB_CHECK_LAUNCH("shuffle_rows_kernel");
  return SGLB200_OK;
}

extern "C" int sglb200_apply_shuffle_mul_sum(const void* input, void* output, const int32_t* perm, const void* factors,
                                             int64_t m, int64_t topk, int64_t hidden, int dtype, int round_products,
                                             void* stream) {
  SGLB_REQUIRE(m >= 0 && topk >= 1 && hidden >= 0, SGLB200_ERR_SHAPE, "m=%lld topk=%lld hidden=%lld", (long long)m,
               (long long)topk, (long long)hidden);
  SGLB_REQUIRE(dtype == SGLB200_BF16 || dtype == SGLB200_F16, SGLB200_ERR_DTYPE, "dtype=%d", dtype);
  if (m == 0 || hidden == 0) return SGLB200_OK;
  SGLB_REQUIRE(input && output && perm, SGLB200_ERR_NULL, "input/output/perm must not be NULL");
  SGLB_REQUIRE(hidden % 8 == 0 ? (aligned(input, 16) && aligned(output, 16)) : true, SGLB200_ERR_ALIGN,
               "input/output must be 16-byte aligned");
  SGLB_REQUIRE(hidden % 8 == 0 || hidden < 8, SGLB200_ERR_SHAPE,
               "hidden=%lld: rows must be a multiple of 8 elements (16-byte rows)", (long long)hidden);
  SGLB_REQUIRE(m < ((int64_t)1 << 31), SGLB200_ERR_SHAPE, "m too large");
  if (int rc = check_arch()) return rc;
  return combine(input, output, perm, factors, nullptr, 1.f, m, topk, hidden, dtype, round_products != 0,
                 static_cast<cudaStream_t>(stream));
}

extern "C" int sglb200_silu_and_mul(const void* input, void* output, int64_t num_rows, int64_t hidden, int dtype,
                                    void* stream) {
  SGLB_REQUIRE(num_rows >= 0 && hidden >= 0, SGLB200_ERR_SHAPE, "num_rows=%lld hidden=%lld", (long long)num_rows,
               (long long)hidden);
  SGLB_REQUIRE(dtype == SGLB200_BF16 || dtype == SGLB200_F16, SGLB200_ERR_DTYPE, "dtype=%d", dtype);
  SGLB_REQUIRE(hidden % 8 == 0, SGLB200_ERR_SHAPE, "hidden=%lld must be a multiple of 8", (long long)hidden);
  if (num_rows == 0 || hidden == 0) return SGLB200_OK;
  SGLB_REQUIRE(input && output, SGLB200_ERR_NULL, "input/output must not be NULL");
  SGLB_REQUIRE(aligned(input, 16) && aligned(output, 16), SGLB200_ERR_ALIGN, "input/output must be 16-byte aligned");
  if (int rc = check_arch()) return rc;
  DeviceInfo di;
  device_info(&di);
  const int64_t total = num_rows * (hidden / 8);
  int64_t blocks = (total + 255) / 256;
  const int64_t cap = (int64_t)di.sm_count * 16;
  if (blocks > cap) blocks = cap;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == SGLB200_BF16) {
    silu_and_mul_kernel<__nv_bfloat16><<<(int)blocks, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(input),
                                                                   static_cast<__nv_bfloat16*>(output), num_rows,
                                                                   (int32_t)hidden);
  } else {
    silu_and_mul_kernel<__half><<<(int)blocks, 256, 0, st>>>(static_cast<const __half*>(input),
                                                            static_cast<__half*>(output), num_rows, (int32_t)hidden);
  }
  SGLB_CHECK_LAUNCH("silu_and_mul_kernel");
  return SGLB200_OK;
}

// ------------------------------------------------------------------------------------------
// The expert layer in one call: routing tables -> quantise + scatter -> grouped GEMM (gate_up) -> SiLU-mul + requantise ->
// grouped GEMM (down) -> weighted sum over the slots.  Six launches, no copy of the bf16 activations in expert order.
// Scratch: tables, then one region used twice (rows in expert order and gate_up output; later the down output), then the
// requantised rows.
// ------------------------------------------------------------------------------------------
namespace sglb {
namespace {
struct ExpertScratch {
  int64_t offsets, a_map, c_map, rep_s, q2_s, rep_q, c1, c2, q2, bytes;
};
ExpertScratch expert_scratch(int64_t M, int64_t H, int64_t I, int64_t E, int64_t topk, bool ue) {
  auto up = [](int64_t x) { return (x + 511) / 512 * 512; };
  const int64_t rows = M * topk, ld = (rows + 3) / 4 * 4;
  ExpertScratch l;
  l.offsets = 0;
  l.a_map = up((E + 1) * 4);
  l.c_map = l.a_map + up(rows * 4);
  l.rep_s = l.c_map + up(rows * 4);
  l.q2_s = l.rep_s + up(rows * (ue ? (H / 128 + 3) / 4 : H / 128) * 4);
  l.rep_q = l.c2 = l.q2_s + up(ld * (ue ? (I / 128 + 3) / 4 : I / 128) * 4);
  l.c1 = l.rep_q + up(rows * H);
  const int64_t first = up(rows * H) + up(rows * 2 * I * 2), second = up(rows * H * 2);
  l.q2 = l.rep_q + (first > second ? first : second);
  l.bytes = l.q2 + up(rows * I);
  return l;
}
}  // namespace
}  // namespace sglb

extern "C" int64_t sglb200_fused_experts_scratch_bytes(int64_t M, int64_t H, int64_t I, int64_t E, int64_t topk, int scale_ue8m0) {
  if (M <= 0 || H <= 0 || I <= 0 || E <= 0 || topk <= 0) return 0;
  return expert_scratch(M, H, I, E, topk, scale_ue8m0 != 0).bytes;
}

extern "C" int sglb200_fused_experts(const void* x, int dtype, const void* w1, const void* w2, const void* w1_scale,
                                     const void* w2_scale, const int64_t* w1_scale_strides, const int64_t* w2_scale_strides,
                                     const float* topk_weights, const int32_t* topk_ids, float weight_factor, void* out, int64_t M,
                                     int64_t H, int64_t I, int64_t E, int64_t topk, int scale_ue8m0, float eps, void* scratch,
                                     int64_t scratch_bytes, void* stream) {
  SGLB_REQUIRE(dtype == SGLB200_BF16 || dtype == SGLB200_F16, SGLB200_ERR_DTYPE, "dtype=%d: only bf16 (0) and f16 (1)", dtype);
  SGLB_REQUIRE(M >= 0 && H > 0 && I > 0 && H % 128 == 0 && I % 128 == 0, SGLB200_ERR_SHAPE,
               "M=%lld H=%lld I=%lld: hidden and intermediate sizes in whole groups of 128", (long long)M, (long long)H, (long long)I);
  SGLB_REQUIRE(E >= 1 && E <= 1024 && topk >= 1 && topk <= kScatterMaxTopk && M * topk <= (1 << 24), SGLB200_ERR_SHAPE,
               "experts=%lld topk=%lld M*topk=%lld: at most 1024, %d and 2^24", (long long)E, (long long)topk, (long long)(M * topk),
               kScatterMaxTopk);
  if (M == 0) return SGLB200_OK;
  SGLB_REQUIRE(x && w1 && w2 && w1_scale && w2_scale && w1_scale_strides && w2_scale_strides && topk_weights && topk_ids && out,
               SGLB200_ERR_NULL, "pointers must not be NULL");
  SGLB_REQUIRE(aligned(x, 16) && aligned(out, 16) && scratch && aligned(scratch, 256), SGLB200_ERR_ALIGN,
               "x and out must be 16-byte, scratch 256-byte aligned");
  if (int rc = check_arch()) return rc;
  const bool ue = scale_ue8m0 != 0;
  const ExpertScratch l = expert_scratch(M, H, I, E, topk, ue);
  SGLB_REQUIRE(scratch_bytes >= l.bytes, SGLB200_ERR_WORKSPACE, "scratch_bytes=%lld: %lld needed", (long long)scratch_bytes,
               (long long)l.bytes);
  char* base = static_cast<char*>(scratch);
  int32_t *offsets = reinterpret_cast<int32_t*>(base + l.offsets), *a_map = reinterpret_cast<int32_t*>(base + l.a_map),
          *c_map = reinterpret_cast<int32_t*>(base + l.c_map);
  void *rep_q = base + l.rep_q, *rep_s = base + l.rep_s, *c1 = base + l.c1, *c2 = base + l.c2, *q2 = base + l.q2, *q2_s = base + l.q2_s;
  const int64_t rows = M * topk, ld = (rows + 3) / 4 * 4, kg1 = (H / 128 + 3) / 4;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (int rc = prepare(topk_ids, offsets, nullptr, nullptr, a_map, c_map, rows, topk, E, I, H, st)) return rc;
#define SGLB_SCATTER(T, U)                                                                                            \
  launch_pdl(quant_scatter_kernel<T, U>, dim3((unsigned)M), dim3(kScatterThreads), 0, st, static_cast<const T*>(x),     \
             static_cast<const int32_t*>(c_map), static_cast<uint8_t*>(rep_q), rep_s, (int32_t)H, (int32_t)topk, eps)
  if (dtype == SGLB200_BF16) {
    if (ue) SGLB_SCATTER(__nv_bfloat16, true); else SGLB_SCATTER(__nv_bfloat16, false);
  } else {
    if (ue) SGLB_SCATTER(__half, true); else SGLB_SCATTER(__half, false);
  }
#undef SGLB_SCATTER
  SGLB_CHECK_LAUNCH("quant_scatter_kernel");
  const int64_t *p1 = w1_scale_strides, *p2 = w2_scale_strides;
  int rc;
  if (ue) {
    rc = sglb200_fp8_ue8m0_scaled_grouped_mm(rep_q, w1, static_cast<const int32_t*>(rep_s), static_cast<const int32_t*>(w1_scale), c1,
                                             offsets, rows, E, 2 * I, H, H, H, 2 * I * H, 2 * I, kg1, 1, p1[0], p1[1], p1[2], dtype,
                                             stream);
  } else {
    rc = sglb200_fp8_blockwise_scaled_grouped_mm(rep_q, w1, static_cast<const float*>(rep_s), static_cast<const float*>(w1_scale), c1,
                                                 offsets, nullptr, rows, E, 2 * I, H, H, H, 2 * I * H, 2 * I, H / 128, 1, p1[0], p1[1],
                                                 p1[2], dtype, stream);
  }
  if (rc) return rc;
  // the scales of the requantised rows are column-major: the GEMM reads a column of 128 rows at a time
  rc = sglb200_silu_mul_group_quant_fp8(c1, dtype, q2, q2_s, nullptr, rows, I, 128, eps, -448.f, 448.f, ue, 1, ld, stream);
  if (rc) return rc;
  if (ue) {
    rc = sglb200_fp8_ue8m0_scaled_grouped_mm(q2, w2, static_cast<const int32_t*>(q2_s), static_cast<const int32_t*>(w2_scale), c2,
                                             offsets, rows, E, H, I, I, I, H * I, H, 1, ld, p2[0], p2[1], p2[2], dtype, stream);
  } else {
    rc = sglb200_fp8_blockwise_scaled_grouped_mm(q2, w2, static_cast<const float*>(q2_s), static_cast<const float*>(w2_scale), c2,
                                                 offsets, nullptr, rows, E, H, I, I, I, H * I, H, 1, ld, p2[0], p2[1], p2[2], dtype,
                                                 stream);
  }
  if (rc) return rc;
  return combine(c2, out, c_map, nullptr, topk_weights, weight_factor, M, topk, H, dtype, true, st);
}
