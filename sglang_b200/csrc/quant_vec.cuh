// Vector arithmetic of the per-token-group quantiser that more than one kernel uses: the element traits of the
// input types, the packed quotient step and the e4m3 pair conversion (device only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>

#include "quant_math.cuh"

namespace sglb {

// ---- element traits: E = elements per 16-byte vector -----------------------------------------
template <typename T>
struct Elem;

template <>
struct Elem<__nv_bfloat16> {
  static constexpr int E = 8;
  // |.| maximum over the 8 packed values of a vector, as fp32
  static __device__ __forceinline__ float vec_absmax(const uint4& u) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
    __nv_bfloat162 m = __hmax2(__habs2(h[0]), __habs2(h[1]));
    m = __hmax2(m, __hmax2(__habs2(h[2]), __habs2(h[3])));
    const float2 f = __bfloat1622float2(m);
    return fmaxf(f.x, f.y);
  }
  static __device__ __forceinline__ float2 pair(uint32_t w) {  // two bf16 -> two fp32 (exact)
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  static __device__ __forceinline__ uint32_t sign_bytes(uint32_t w0, uint32_t w1) {  // bytes 1,3 of each word
    return __byte_perm(w0, w1, 0x7531);
  }
  static __device__ __forceinline__ float round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {  // products of the pairs, rounded to T
    const __nv_bfloat162 h = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&h);
  }
};

template <>
struct Elem<__half> {
  static constexpr int E = 8;
  static __device__ __forceinline__ float vec_absmax(const uint4& u) {
    const __half2* h = reinterpret_cast<const __half2*>(&u);
    __half2 m = __hmax2(__habs2(h[0]), __habs2(h[1]));
    m = __hmax2(m, __hmax2(__habs2(h[2]), __habs2(h[3])));
    const float2 f = __half22float2(m);
    return fmaxf(f.x, f.y);
  }
  static __device__ __forceinline__ float2 pair(uint32_t w) {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
  static __device__ __forceinline__ uint32_t sign_bytes(uint32_t w0, uint32_t w1) {
    return __byte_perm(w0, w1, 0x7531);
  }
  static __device__ __forceinline__ float round(float x) { return __half2float(__float2half_rn(x)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {  // products of the pairs, rounded to T
    const __half2 h = __hmul2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&h);
  }
};

template <>
struct Elem<float> {
  static constexpr int E = 4;
  static __device__ __forceinline__ float vec_absmax(const uint4& u) {
    return fmaxf(fmaxf(fabsf(__uint_as_float(u.x)), fabsf(__uint_as_float(u.y))),
                 fmaxf(fabsf(__uint_as_float(u.z)), fabsf(__uint_as_float(u.w))));
  }
  static __device__ __forceinline__ float round(float x) { return x; }
};

__device__ __forceinline__ float silu_f32(float x) { return __fdiv_rn(x, 1.0f + expf(-x)); }

// Two quotients x / s with the shared reciprocal r = RN(1/s): packed Markstein step.
__device__ __forceinline__ float2 quotient2(float2 x, float2 rr, float2 neg_ss) {
  const float2 q0 = __fmul2_rn(x, rr);
  const float2 rem = __ffma2_rn(q0, neg_ss, x);
  return __ffma2_rn(rem, rr, q0);
}

// x / (1 + exp(-x)) rounded to T, times u, rounded to T, on eight packed pairs.  The quotient is the approximate reciprocal
// (one ulp) and one Markstein correction q0 + (x - q0 t) r, whose error is 2^-46 before its single rounding; for |x| <= 80
// nothing in it under- or overflows and it agrees with the IEEE division for every bf16 and every fp16 x (all of them are
// tested).  The division routine is a call with special cases per element: the fused quantiser spent 104 us on 32768 x 2048
// with it (issue-bound, half the copy rate of HBM), 68 without.
template <typename T>
__device__ __forceinline__ uint4 silu_mul8(const uint4& g, const uint4& u) {
  const uint32_t* gw = reinterpret_cast<const uint32_t*>(&g);
  const uint32_t* uw = reinterpret_cast<const uint32_t*>(&u);
  uint4 out;
  uint32_t* ow = reinterpret_cast<uint32_t*>(&out);
  const bool fast = Elem<T>::vec_absmax(g) <= 80.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = Elem<T>::pair(gw[j]);
    const float2 t = make_float2(1.0f + expf(-x.x), 1.0f + expf(-x.y));
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(t.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(t.y));
    const float2 q0 = __fmul2_rn(x, r);
    const float2 rem = __ffma2_rn(q0, make_float2(-t.x, -t.y), x);
    const float2 q = __ffma2_rn(rem, r, q0);
    // the sign comes from x: the FMA chain gives +0 for x = -0
    ow[j] = Elem<T>::mul2((Elem<T>::pack(q.x, q.y) & 0x7fff7fffu) | (gw[j] & 0x80008000u), uw[j]);
  }
  if (!fast) {
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const uint32_t a = j == 0 ? g.x : j == 1 ? g.y : j == 2 ? g.z : g.w;
      const uint32_t b = j == 0 ? u.x : j == 1 ? u.y : j == 2 ? u.z : u.w;
      const float2 x = Elem<T>::pair(a);
      const uint32_t o = Elem<T>::mul2(Elem<T>::pack(silu_f32(x.x), silu_f32(x.y)), b);
      if (j == 0) out.x = o;
      else if (j == 1) out.y = o;
      else if (j == 2) out.z = o;
      else out.w = o;
    }
  }
  return out;
}

__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {
  return (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}

// Sixteen consecutive 16-bit inputs (two 16-byte vectors) divided by the group's scale and converted to e4m3 with the
// e4m3 limits (the saturating conversion clamps): the same operations, in the same order, as group_quant16_kernel.
// r = RN(1 / s); kNormal: the caller knows that the scale lies between the limits below.
template <typename T, bool kNormal = false>
__device__ __forceinline__ uint4 encode16_e4m3(const uint4& v0, const uint4& v1, float s, float r) {
  const bool fast = kNormal || (s >= 7.888609e-31f) && (s <= 1.2676506e30f);
  const float2 rr = make_float2(r, r), nss = make_float2(-s, -s);
  uint32_t packed[4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(h == 0 ? &v0 : &v1);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float2 qa, qb;
      const float2 xa = Elem<T>::pair(w[2 * j]), xb = Elem<T>::pair(w[2 * j + 1]);
      if (fast) {
        qa = quotient2(xa, rr, nss);
        qb = quotient2(xb, rr, nss);
      } else {
        qa = make_float2(__fdiv_rn(xa.x, s), __fdiv_rn(xa.y, s));
        qb = make_float2(__fdiv_rn(xb.x, s), __fdiv_rn(xb.y, s));
      }
      const uint32_t codes = cvt_e4m3x2(qa.x, qa.y) | (cvt_e4m3x2(qb.x, qb.y) << 16);
      const uint32_t signs = Elem<T>::sign_bytes(w[2 * j], w[2 * j + 1]);
      packed[2 * h + j] = (codes & 0x7f7f7f7fu) | (signs & 0x80808080u);
    }
  }
  return make_uint4(packed[0], packed[1], packed[2], packed[3]);
}
template <typename T>
__device__ __forceinline__ uint4 encode16_e4m3(const uint4& v0, const uint4& v1, float s) {
  return encode16_e4m3<T>(v0, v1, s, __frcp_rn(s));
}

}  // namespace sglb
