// Block-scaled FP8 GEMM on CTA pairs (tcgen05 cta_group::2), dense: the kernel for many rows.
//
//   out[m, n] = cast( sum_kb ( sum_{k in kb} a[m,k] * b[n,k] ) * sa[m,kb] * sb[n/128,kb] )
//
// Two CTAs of a cluster (two SMs of one TPC) work on one 256 x 256 output tile: each CTA loads its own 128 rows of A and HALF of
// the B rows with its own TMA copies, and one tcgen05.mma.cta_group::2 issued by the even CTA reads both halves from both
// shared memories.  No load is broadcast; only mbarrier arrivals cross between the two CTAs.
//
// Why pairs: the 128 x 128 tiles of gemm.cu need 32 KB of operands per SM and k-block, 15.8 TB/s out of L2 at the rate they reach,
// which is what bounds them at high clocks, and the energy of that traffic is part of what bounds them under the power cap.
// Here it is 16 KB per 128 x 128 x 128 of work.  Measured (B200, this / the tile kernel): a second of load at the 1000 W cap
// 8192 x 36864 x 7168 2112 us / 2450, 8192 x 24576 x 1536 366 / 420; one burst 4096 x 7168 x 7168 187 / 212.
//
// Per CTA, 384 threads, warp-specialised:
//   warp 0      TMA producer: per k-block A [128 x 128 B], two boxes of B [64 x 128 B] and the 128 activation scales into a 5-stage
//               ring.  The bytes of BOTH CTAs are counted on the even CTA's `full` barrier.
//   warp 1      idle (registers move in whole warpgroups).
//   warps 2-3   MMA issuers, active in the even CTA only, one per HALF (128 columns) of the tile: four tcgen05.mma
//               (256 x 128 x 32) per k-block that overwrite one of the half's two 128-column TMEM stages in both CTAs.
//   warps 4-11  promotion + epilogue for the CTA's own 128 rows: four warps (one per TMEM lane quarter) per half, 128
//               columns each.  acc += partial * scale in fp32 registers (packed FMAs); the TMEM stage is handed back by an arrival
//               on the even CTA's `acc_empty` barrier; results leave through swizzled shared memory and TMA stores.
// What bounds it: the two TMEM stages a half has, times the time a stage is away (about 1100 cycles from the issue of its MMAs
// to the promotion warps' seeing them, the other half's MMAs among them, then reading and 150 of hand-back): 767 cycles per
// k-block against 512 of MMA at 2048 x 36864 x 7168 (70 % tensor pipe; 900 to 950 with loads of 32 columns in turn).  Sixteen promotion warps of 64 columns, one 256-column stage for both halves, and 256 x 128
// tiles with four stages are level or slower (549, 542 and 587 ns per 256 x 256 x 128 against 535 at the time).
// Scales: a warp that wrote the products sa * sb into a ring of its own, with two more barriers, cost 150 ns of 620 per k-block in
// shared-memory and barrier latency of the promotion warps; the TMA copy shares the operands' barrier, and sb (one value per
// half and k-block) comes out of a register by shuffle.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"

namespace sglb {

__device__ int g_pair_status = 0;

int pair_take_device_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_pair_status, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  if (v != 0) {
    int z = 0;
    cudaMemcpyToSymbol(g_pair_status, &z, sizeof(int));
  }
  return v;
}

namespace {

constexpr int BK = 128, BN = 256;
constexpr int kThreads = 384;
constexpr int kFirstMmaWarp = 2, kFirstPromoWarp = 4, kHalfWarps = 4;
constexpr int kStages = 5, kAcc = 2;  // kAcc: TMEM stages of 128 columns per half
// Slots of 128 activation scales.  A copy into the slot of k-block j + kStages is issued when the MMAs of j are done; those were
// issued after the promotion warps had handed back j - kAcc and so read its scales: kStages + kAcc slots would do.
constexpr int kScaleSlots = 2 * kStages;
constexpr uint32_t kSlotBytes = 128 * sizeof(float);
constexpr int kGroupM = 8;  // 256-row tiles per raster group
constexpr uint32_t kTileBytes = 128 * BK, kStageBytes = 2 * kTileBytes;
constexpr uint32_t kPatchBytes = 32 * 128;  // a warp's staging: 32 rows x 64 columns of the output, 128-byte-swizzled
constexpr size_t kPatchOffset = (size_t)kStages * kStageBytes;
constexpr size_t kScaleOffset = kPatchOffset + 2 * kHalfWarps * kPatchBytes;  // [slot][row]
constexpr size_t kCtlOffset = kScaleOffset + (size_t)kScaleSlots * kSlotBytes;
constexpr uint32_t kCtlBytes = 512;
constexpr size_t kSmem = 1024 + kCtlOffset + kCtlBytes;
static_assert(kSmem <= 227 * 1024, "shared memory of one CTA");
constexpr int kAuxRegs = 40, kPromoRegs = 232;

struct PairParams {
  const float* sb;
  const void* bias;  // optional: [N] of the output type, added to the rounded result
  int32_t M, N;
  int32_t m2_tiles, n2_tiles, k_tiles, sb_blocks;
  int64_t sb_stride_n, sb_stride_k;
  int32_t out_dtype;
};

struct Ctl {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full[2][kAcc];
  uint64_t acc_empty[2][kAcc];
  uint32_t tmem_base;
  volatile int32_t abort_flag;
};
static_assert(sizeof(Ctl) <= kCtlBytes, "control block");

__device__ __forceinline__ void timeout(Ctl* ctl, int code) {
  ctl->abort_flag = 1;
  atomicCAS(&g_pair_status, 0, code);
}

__device__ __forceinline__ uint32_t pack16(float a, float b, int out_dtype) {
  if (out_dtype == SGLB200_BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ void fma64(float2* acc, const uint32_t (&v)[64], float2 scale2) {
#pragma unroll
  for (int j = 0; j < 32; ++j)
    acc[j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), scale2, acc[j]);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
fp8_block_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                           const __grid_constant__ CUtensorMap map_sa,
                           const __grid_constant__ CUtensorMap map_out, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + kCtlOffset);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();  // 0: issues the MMAs; 1: partner
  const int32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int32_t total = p.m2_tiles * p.n2_tiles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&ctl->full[i], 1);
      ptx::mbar_init(&ctl->empty[i], 2);  // both issuers
    }
    for (int i = 0; i < 2 * kAcc; ++i) {
      ptx::mbar_init(&ctl->acc_full[0][i], 1);
      ptx::mbar_init(&ctl->acc_empty[0][i], 2 * kHalfWarps);  // one arrival per promotion warp of the half in both CTAs
    }
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
  }
  if (warp == kFirstMmaWarp) {
    ptx::tmem_alloc_pair(&ctl->tmem_base, 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // both CTAs' barriers are initialised before either signals the other
  ptx::tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  const uint32_t full0 = ptx::smem_u32(&ctl->full[0]), empty0 = ptx::smem_u32(&ctl->empty[0]);
  const uint32_t stage0 = ptx::smem_u32(smem);
  const bool leader = ptx::elect_one();  // the lane that issues TMA and tcgen05 instructions

  auto tile_of = [&](int32_t t, int32_t& row0, int32_t& n0) {
    const int32_t per_group = kGroupM * p.n2_tiles, gid = t / per_group, first_m = gid * kGroupM;
    const int32_t gm = min(p.m2_tiles - first_m, kGroupM), local = t - gid * per_group, nt = local / gm;
    row0 = (first_m + (local - nt * gm)) * 256 + (int32_t)rank * 128;
    n0 = nt * BN;
  };

  // No call may sit behind a changed register limit, hence the inlined waits.
  if (warp >= kFirstPromoWarp) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPromoRegs));
    // ===== promotion + epilogue; TMEM lane quarter = warp % 4
    const int q = warp & 3, wi = warp - kFirstPromoWarp, half = wi >> 2;
    const uint32_t acc_full0 = ptx::smem_u32(&ctl->acc_full[half][0]);
    const uint32_t lead_acc_empty0 = ptx::mapa_shared(ptx::smem_u32(&ctl->acc_empty[half][0]), 0);  // the even CTA's
    const uint32_t tlane = tmem_base + ((uint32_t)(q * 32) << 16) + half * 256;
    const uint32_t sc0 = stage0 + (uint32_t)kScaleOffset + (q * 32 + lane) * 4;
    uint32_t acc_stage = 0, acc_phase = 0, slot = 0;
    const uint32_t patch = stage0 + (uint32_t)kPatchOffset + wi * kPatchBytes;
    bool ready = false;
    float2 acc[64];
    for (int32_t t = pair; t < total; t += pairs) {
      int32_t row0, n0;
      tile_of(t, row0, n0);
      const float* sb = p.sb + (int64_t)min(n0 / 128 + half, p.sb_blocks - 1) * p.sb_stride_n;
      float sb_now = __ldg(sb + (int64_t)min(lane, p.k_tiles - 1) * p.sb_stride_k);  // of 32 k-blocks, one a lane
      float b = __shfl_sync(0xffffffffu, sb_now, 0);
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = make_float2(0.f, 0.f);
      bool ok = true;
#pragma unroll 1
      for (int32_t kb = 0; kb < p.k_tiles; ++kb) {
        if (!ready && !ptx::mbar_wait_inl_a(acc_full0 + acc_stage * 8, acc_phase)) {
          timeout(ctl, 34);
          ok = false;
          break;
        }
        ptx::tc_fence_after();
        const uint32_t taddr = tlane + acc_stage * 128;
        uint32_t v[64];
        ptx::tmem_ld_32x64(taddr, v);
        const float scale = ptx::ld_shared_f32(sc0 + slot) * b;
        const float2 s2 = make_float2(scale, scale);
        ptx::tmem_ld_wait(v);
        fma64(acc, v, s2);
        ptx::tmem_ld_32x64_reuse(taddr + 64, v);
        ptx::tmem_ld_wait(v);
        ptx::tc_fence_before();
        __syncwarp();
        ptx::mbar_arrive_cluster_if(lead_acc_empty0 + acc_stage * 8, leader);
        acc_stage ^= 1;
        acc_phase ^= acc_stage ^ 1;
        // Asked early, answered while the sums are added.  test_wait: try_wait would hold the warp, and at the very end, where no
        // further stage comes, for 4 us.
        ready = ptx::mbar_test_wait_a(acc_full0 + acc_stage * 8, acc_phase);
        if (((kb + 1) & 31) == 0) sb_now = __ldg(sb + (int64_t)min(kb + 1 + lane, p.k_tiles - 1) * p.sb_stride_k);
        b = __shfl_sync(0xffffffffu, sb_now, (kb + 1) & 31);
        slot = slot == (kScaleSlots - 1) * kSlotBytes ? 0 : slot + kSlotBytes;
        fma64(acc + 32, v, s2);
      }
      if (!ok || ctl->abort_flag) break;
      // 64 columns per pass: a lane's row of 128 bytes into the warp's swizzled staging, from there one TMA store (which leaves out
      // what lies past M and N)
      const int32_t n_first = n0 + half * 128, row_base = row0 + q * 32;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int32_t c0 = n_first + 64 * h;
        if (c0 >= p.N || row_base >= p.M) break;  // uniform over the warp
        if (leader) ptx::bulk_wait_read();  // the store before has read the staging
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2* v = acc + 32 * h + 4 * i;
          uint4 u = make_uint4(pack16(v[0].x, v[0].y, p.out_dtype), pack16(v[1].x, v[1].y, p.out_dtype),
                               pack16(v[2].x, v[2].y, p.out_dtype), pack16(v[3].x, v[3].y, p.out_dtype));
          if (p.bias != nullptr && c0 + 8 * i < p.N)
            u = ptx::add_bias8(u, __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.bias) + c0 + 8 * i)), p.out_dtype);
          ptx::st_shared_v4(patch + lane * 128 + ((i ^ (lane & 7)) << 4), u);
        }
        ptx::fence_proxy_async();
        __syncwarp();
        if (leader) ptx::tma_store_2d(&map_out, patch, c0, row_base);
      }
    }
    if (leader) ptx::bulk_wait_read();  // the staging must outlive its stores
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kAuxRegs));
    if (warp == 0) {
      // ===== TMA producer
      const uint32_t lead_full0 = ptx::mapa_shared(full0, 0);
      uint32_t stage = 0, phase = 0, slot = 0;
      uint32_t armed = 0, armed_phase = 0;  // bit i: stage i was armed / the phase bit of its last arming
      for (int32_t t = pair; t < total; t += pairs) {
        int32_t row0, n0;
        tile_of(t, row0, n0);
        n0 += (int32_t)rank * 64;  // of either half's 128 columns this CTA holds 64
        bool ok = true;
        for (int32_t kb = 0; kb < p.k_tiles; ++kb) {
          if (!ptx::mbar_wait_inl_a(empty0 + stage * 8, phase ^ 1)) {
            timeout(ctl, 31);
            ok = false;
            break;
          }
          armed |= 1u << stage;
          armed_phase = (armed_phase & ~(1u << stage)) | (phase << stage);
          if (leader) {
            const uint32_t dst = stage0 + stage * kStageBytes;
            if (rank == 0) ptx::mbar_arrive_expect_tx_a(full0 + stage * 8, 2 * (kStageBytes + kSlotBytes));  // both CTAs' bytes
            ptx::tma_load_2d_pair(dst, &map_a, lead_full0 + stage * 8, kb * BK, row0);
            ptx::tma_load_2d_pair(stage0 + (uint32_t)kScaleOffset + slot, &map_sa, lead_full0 + stage * 8, row0, kb);
            ptx::tma_load_2d_pair(dst + kTileBytes, &map_b, lead_full0 + stage * 8, kb * BK, n0);
            ptx::tma_load_2d_pair(dst + kTileBytes + kTileBytes / 2, &map_b, lead_full0 + stage * 8, kb * BK, n0 + 128);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
          slot = slot == (kScaleSlots - 1) * kSlotBytes ? 0 : slot + kSlotBytes;
        }
        if (!ok || ctl->abort_flag) break;
      }
      if (ctl->abort_flag) {
        // After a time-out: no CTA may exit while bulk copies into its shared memory are in flight.  Both CTAs' copies are
        // counted on the even CTA's `full` barriers, so the even CTA waits (20 ms at most per stage) for the stages it
        // announced; the cluster barrier at the exit then holds the partner until that is done.
        if (rank == 0)
          for (uint32_t i = 0; i < (uint32_t)kStages; ++i)
            if (armed & (1u << i)) ptx::mbar_wait_inl_a(full0 + i * 8, (armed_phase >> i) & 1u, 20000000ull);
      } else {
        // the last arrivals on `empty` come from asynchronous commits: take every stage once more before leaving
        for (int i = 0; i < kStages; ++i) {
          if (!ptx::mbar_wait_inl_a(empty0 + stage * 8, phase ^ 1)) { timeout(ctl, 35); break; }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    } else if (rank == 0 && warp >= kFirstMmaWarp) {
      // ===== MMA issuers, one per half of the tile's columns
      const uint32_t half = warp - kFirstMmaWarp;
      constexpr uint32_t idesc = ptx::make_idesc_e4m3_f32(256, 128);
      const uint32_t acc_full0 = ptx::smem_u32(&ctl->acc_full[half][0]), acc_empty0 = ptx::smem_u32(&ctl->acc_empty[half][0]);
      const uint64_t desc0 = ptx::make_kmajor_sw128_desc(stage0);
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      for (int32_t t = pair; t < total; t += pairs) {
        bool ok = true;
        for (int32_t kb = 0; kb < p.k_tiles; ++kb) {
          if (!ptx::mbar_wait_inl_a(full0 + stage * 8, phase)) { timeout(ctl, 33); ok = false; break; }
          if (!ptx::mbar_wait_inl_a(acc_empty0 + acc * 8, acc_phase ^ 1)) { timeout(ctl, 32); ok = false; break; }
          ptx::tc_fence_after();
          if (leader) {
            const uint64_t a_desc = desc0 + (uint64_t)(stage * (kStageBytes >> 4));
            const uint64_t b_desc = a_desc + ((kTileBytes + half * (kTileBytes / 2)) >> 4);
            const uint32_t d_tmem = tmem_base + half * 256 + acc * 128;
            ptx::mma_f8f6f4_pair(d_tmem, a_desc, b_desc, idesc, 0);
#pragma unroll
            for (uint32_t k = 1; k < BK / 32; ++k) ptx::mma_f8f6f4_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, 1);
            ptx::mma_commit_pair_a(acc_full0 + acc * 8);
            ptx::mma_commit_pair_a(empty0 + stage * 8);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
          acc ^= 1;
          acc_phase ^= acc ^ 1;
        }
        if (!ok || ctl->abort_flag) break;
      }
    }
  }

  // ---------------------------------------------------------------- tear-down
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers or read its tiles
  if (warp == kFirstMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

// Activation scales that the kernel's TMA copies can fetch: M-major, whole 16-byte units, columns that do not overlap (a tensor map's
// strides are not smaller than its rows).
bool pair_takes_scales(const float* sa, int64_t M, int64_t sa_stride_m, int64_t sa_stride_k) {
  return sa_stride_m == 1 && sa_stride_k >= M && sa_stride_k % 4 == 0 && aligned(sa, 16);
}

// Dense GEMM on CTA pairs; arguments as gemm_common's dense case (checked there), scales as above.
int pair_gemm(const void* a, const void* b, const float* sa, const float* sb, void* out, int64_t M, int64_t N, int64_t K,
              int64_t lda, int64_t ldb, int64_t ldc, int64_t sa_stride_m, int64_t sa_stride_k, int64_t sb_stride_n,
              int64_t sb_stride_k, int out_dtype, const void* bias, int sm_count, void* stream) {
  static bool attr_done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(fp8_block_gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return fail(SGLB200_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    // setmaxnreg.inc draws on the registers the block was launched with and waits for good if they do not suffice: a build
    // whose register count is too low for the split must not be launched
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, fp8_block_gemm_pair_kernel);
    if (e != cudaSuccess || fa.numRegs * kThreads < 128 * kAuxRegs + 256 * kPromoRegs)
      return fail(SGLB200_ERR_LAUNCH, "fp8_block_gemm_pair_kernel: %d registers a thread are too few for its register split",
                  e == cudaSuccess ? fa.numRegs : 0);
    attr_done[dev] = true;
  }
  alignas(64) CUtensorMap map_a, map_b;
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t str[1] = {(uint64_t)lda};
    if (int rc = make_map_sw128(&map_a, a, 2, dims, str, 128, CU_TENSOR_MAP_L2_PROMOTION_L2_128B)) return rc;
  }
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)N};
    const uint64_t str[1] = {(uint64_t)ldb};
    if (int rc = make_map_sw128(&map_b, b, 2, dims, str, 64, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) return rc;
  }
  alignas(64) CUtensorMap map_sa;
  if (int rc = make_map_f32(&map_sa, sa, (uint64_t)M, (uint64_t)((K + BK - 1) / BK), (uint64_t)sa_stride_k * 4, 128)) return rc;
  alignas(64) CUtensorMap map_out;
  if (int rc = make_map_out16(&map_out, out, (uint64_t)N, (uint64_t)M, (uint64_t)ldc * 2, 64, 32)) return rc;
  PairParams p;
  p.sb = sb;
  p.bias = bias;
  p.M = (int32_t)M;
  p.N = (int32_t)N;
  p.m2_tiles = (int32_t)((M + 255) / 256);
  p.n2_tiles = (int32_t)((N + BN - 1) / BN);
  p.k_tiles = (int32_t)((K + BK - 1) / BK);
  p.sb_blocks = (int32_t)((N + 127) / 128);
  p.sb_stride_n = sb_stride_n;
  p.sb_stride_k = sb_stride_k;
  p.out_dtype = out_dtype;
  const int64_t tiles = (int64_t)p.m2_tiles * p.n2_tiles;
  int64_t pairs = sm_count / 2;
  if (tiles < pairs) pairs = tiles;
  fp8_block_gemm_pair_kernel<<<(unsigned)(2 * pairs), kThreads, kSmem, static_cast<cudaStream_t>(stream)>>>(map_a, map_b, map_sa, map_out, p);
  SGLB_CHECK_LAUNCH("fp8_block_gemm_pair_kernel");
  note_gemm("fp8_block_gemm_pair_kernel");
  return SGLB200_OK;
}

}  // namespace sglb

extern "C" int sglb200_fp8_blockwise_scaled_mm_pair(const void* a, const void* b, const float* sa, const float* sb,
                                                    void* out, int64_t M, int64_t N, int64_t K, int64_t lda,
                                                    int64_t ldb, int64_t ldc, int64_t sa_stride_m, int64_t sa_stride_k,
                                                    int64_t sb_stride_n, int64_t sb_stride_k, int out_dtype,
                                                    int tile_n, void* stream) {
  using namespace sglb;
  SGLB_REQUIRE(tile_n == 128 || tile_n == 256, SGLB200_ERR_SHAPE, "tile_n=%d: 128 or 256", tile_n);
  SGLB_REQUIRE(M >= 0 && N >= 0 && K > 0, SGLB200_ERR_SHAPE, "M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
  SGLB_REQUIRE(M < ((int64_t)1 << 31) - 512 && N < ((int64_t)1 << 31) - 512 && K < ((int64_t)1 << 31) - 512,
               SGLB200_ERR_SHAPE, "a dimension exceeds 2^31");
  SGLB_REQUIRE(out_dtype == SGLB200_BF16 || out_dtype == SGLB200_F16, SGLB200_ERR_DTYPE,
               "out_dtype=%d: only bf16 (0) and f16 (1)", out_dtype);
  SGLB_REQUIRE(K % 16 == 0 && N % 8 == 0, SGLB200_ERR_SHAPE, "K=%lld must be a multiple of 16, N=%lld of 8", (long long)K,
               (long long)N);
  if (M == 0 || N == 0) return SGLB200_OK;
  SGLB_REQUIRE(a && b && sa && sb && out, SGLB200_ERR_NULL, "a/b/sa/sb/out must not be NULL");
  SGLB_REQUIRE(lda >= K && lda % 16 == 0 && ldb >= K && ldb % 16 == 0 && ldc >= N && ldc % 8 == 0, SGLB200_ERR_ALIGN,
               "lda=%lld ldb=%lld (>= K, multiples of 16) ldc=%lld (>= N, multiple of 8)", (long long)lda, (long long)ldb,
               (long long)ldc);
  SGLB_REQUIRE(aligned(a, 16) && aligned(b, 16) && aligned(out, 16) && aligned(sa, 4) && aligned(sb, 4), SGLB200_ERR_ALIGN,
               "a, b and out must be 16-byte aligned, the scales 4-byte aligned");
  DeviceInfo di;
  if (int rc = device_info(&di)) return rc;
  SGLB_REQUIRE(di.cc_major == 10, SGLB200_ERR_ARCH, "compute capability %d.%d: this library is built for sm_100a only",
               di.cc_major, di.cc_minor);
  // The same bits from the 128 x 128 tiles, which add K in the same order at every size.  Not the plain entry's choice: for few rows
  // that is the few-rows kernel, whose clusters add ranges of K (16 x 7168 x 16384: 14 of 114688 results one rounding apart).
  if (di.sm_count < 2 || !pair_takes_scales(sa, M, sa_stride_m, sa_stride_k))
    return tile_gemm(a, b, sa, sb, out, M, N, K, lda, ldb, ldc, sa_stride_m, sa_stride_k, sb_stride_n, sb_stride_k, out_dtype, stream);
  return pair_gemm(a, b, sa, sb, out, M, N, K, lda, ldb, ldc, sa_stride_m, sa_stride_k, sb_stride_n, sb_stride_k,
                   out_dtype, nullptr, di.sm_count, stream);
}
