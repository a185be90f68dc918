// UE8M0 GEMM (hardware block scaling, see gemm_ue8m0.cu) on CTA pairs, dense: the form for many rows.
//
// Two CTAs of a cluster work on one 256 x 224 output tile: each loads its own 128 rows of A and HALF (112) of the B rows with its
// own TMA copies, and one tcgen05.mma.cta_group::2 (kind::mxf8f6f4.block_scale, 256 x 224 x 32) issued by the even CTA reads both
// halves from both shared memories.  Scale factors of A for the CTA's own rows and of ALL B rows lie in the TMEM of each CTA
// (tcgen05.cp.cta_group::2 copies from both CTAs' shared memory at once).  No load is broadcast.
//
// Why pairs: the single-CTA kernel moves 45 KB of operands per SM and k-block, 14.4 TB/s out of L2 at the rate it reaches, and has
// shared memory for four stages of that; here it is 30 KB and six stages.  Measured in bursts, single-CTA kernel / this: 4096 x
// 7168 x 18432 426 / 368 us (2942 TFLOP/s), 8192 x 24576 x 1536 421 / 237 (that one's epilogue stores 32 rows an instruction).
// What bounds it: the tensor pipe, 484 cycles per k-block of which 448 are MMA at 2048 x 36864 x 7168 (97 % of active cycles; the
// single-CTA kernel 634), and the power cap.
//
// Per CTA, 384 threads: warp 0 TMA producer; warps 1 and 3 scale loaders (per group of four k-blocks the packed exponent words of 128 A rows
// and 224 B rows, in the arrangement of tcgen05.cp.32x128b.warpx4); warp 2 MMA issuer (even CTA only; one thread issues copies,
// MMAs and commits, which is what orders them); warps 4-11 epilogue: two warps per TMEM lane quarter, 128 and 96
// columns, 32 at a time through swizzled shared memory and TMA stores.  Two 224-column accumulators: the epilogue of a tile
// overlaps the next tile's MMAs.  Every wait is bounded (about two seconds).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"

namespace sglb {

__device__ int g_ue8m0_pair_status = 0;

int ue8m0_pair_take_device_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_ue8m0_pair_status, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  if (v != 0) {
    const int z = 0;
    cudaMemcpyToSymbol(g_ue8m0_pair_status, &z, sizeof(int));
  }
  return v;
}

namespace {

constexpr int BN = 224, BK = 128;
constexpr int kStages = 6, kSfBufs = 4;
constexpr int kThreads = 384;
constexpr int kMmaWarp = 2, kEpiWarp0 = 4, kEpiWarps = 8;
constexpr int kGroupM = 8;  // 256-row tiles per raster group
constexpr uint32_t kTileABytes = 128 * BK, kTileBBytes = BN / 2 * BK, kStageBytes = kTileABytes + kTileBBytes;
constexpr uint32_t kSfABytes = 512, kSfBBytes = 1024, kSfBufBytes = kSfABytes + kSfBBytes;
constexpr uint32_t kSfTmemBase = 2 * BN, kSfTmemPerSet = 12;  // scale columns behind the two accumulators: 4 for A, 8 for B, two sets
constexpr uint32_t kBoxBytes = 32 * 64;                       // 32 rows x 32 columns of the output, 64-byte-swizzled
constexpr size_t kBoxOffset = (size_t)kStages * kStageBytes;
constexpr size_t kSfOffset = kBoxOffset + kEpiWarps * kBoxBytes;
constexpr size_t kCtlOffset = kSfOffset + (size_t)kSfBufs * kSfBufBytes;
constexpr size_t kSmem = 1024 + kCtlOffset + 256;
static_assert(kStageBytes % 1024 == 0 && kSmem <= 227 * 1024, "shared memory of one CTA");

struct PairParams {
  const int32_t* sfa;  // packed exponents of A: word (m, kg) at sfa[kg * sfa_ld + m]
  const int32_t* sfb;  // of B: word (nb, kg) at sfb[nb * sfb_stride_n + kg * sfb_stride_k]
  const void* bias;    // optional: [N] of the output type, added to the rounded result
  int32_t M, N;
  int32_t m2_tiles, n_tiles, k_tiles, k_groups;
  int64_t sfa_ld, sfb_stride_n, sfb_stride_k;
  int32_t out_dtype;
};

struct Ctl {
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t sf_full[kSfBufs];
  uint64_t sf_empty[kSfBufs];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  volatile int32_t abort_flag;
};
static_assert(sizeof(Ctl) <= 256, "control block");

__device__ __forceinline__ void timeout(Ctl* ctl, int code) {
  ctl->abort_flag = 1;
  atomicCAS(&g_ue8m0_pair_status, 0, code);
}

template <typename OutT>
__device__ __forceinline__ uint32_t pack_pair(uint32_t a, uint32_t b);
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(uint32_t a, uint32_t b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
  return *reinterpret_cast<uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(uint32_t a, uint32_t b) {
  __half2 h = __floats2half2_rn(__uint_as_float(a), __uint_as_float(b));
  return *reinterpret_cast<uint32_t*>(&h);
}

// a lane's row of 32 columns into the warp's box
template <typename OutT>
__device__ __forceinline__ void fill_box(const uint32_t (&v)[32], const void* bias, uint32_t box, int32_t c0, int32_t N, int lane, int out_dtype) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 u = make_uint4(pack_pair<OutT>(v[8 * i], v[8 * i + 1]), pack_pair<OutT>(v[8 * i + 2], v[8 * i + 3]),
                         pack_pair<OutT>(v[8 * i + 4], v[8 * i + 5]), pack_pair<OutT>(v[8 * i + 6], v[8 * i + 7]));
    if (bias != nullptr && c0 + 8 * i < N)  // N % 8 == 0
      u = ptx::add_bias8(u, __ldg(reinterpret_cast<const uint4*>(static_cast<const OutT*>(bias) + c0 + 8 * i)), out_dtype);
    ptx::st_shared_v4(box + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4), u);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
fp8_ue8m0_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                           const __grid_constant__ CUtensorMap map_out, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sf_smem = smem + kSfOffset;
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + kCtlOffset);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();  // 0: issues the MMAs; 1: partner
  const int32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int32_t total = p.m2_tiles * p.n_tiles;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      ptx::mbar_init(&ctl->full[i], 1);
      ptx::mbar_init(&ctl->empty[i], 1);
    }
    for (int i = 0; i < kSfBufs; ++i) {
      ptx::mbar_init(&ctl->sf_full[i], 2);  // the scale loaders of both CTAs
      ptx::mbar_init(&ctl->sf_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&ctl->acc_full[i], 1);
      ptx::mbar_init(&ctl->acc_empty[i], 2 * kEpiWarps);
    }
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
    ptx::prefetch_tensormap(&map_a);
    ptx::prefetch_tensormap(&map_b);
    ptx::prefetch_tensormap(&map_out);
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc_pair(&ctl->tmem_base, 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // both CTAs' barriers are initialised before either signals the other
  ptx::tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  const uint32_t full0 = ptx::smem_u32(&ctl->full[0]), empty0 = ptx::smem_u32(&ctl->empty[0]);
  const uint32_t sf_full0 = ptx::smem_u32(&ctl->sf_full[0]), sf_empty0 = ptx::smem_u32(&ctl->sf_empty[0]);
  const uint32_t acc_full0 = ptx::smem_u32(&ctl->acc_full[0]), acc_empty0 = ptx::smem_u32(&ctl->acc_empty[0]);
  const uint32_t stage0 = ptx::smem_u32(smem);
  const bool leader = ptx::elect_one();  // the lane that issues TMA and tcgen05 instructions

  auto tile_of = [&](int32_t t, int32_t& row0, int32_t& n0) {
    const int32_t per_group = kGroupM * p.n_tiles, gid = t / per_group, first_m = gid * kGroupM;
    const int32_t gm = min(p.m2_tiles - first_m, kGroupM), local = t - gid * per_group, nt = local / gm;
    row0 = (first_m + (local - nt * gm)) * 256 + (int32_t)rank * 128;
    n0 = nt * BN;
  };

  if (warp == 0) {
    // ===== TMA producer
    const uint32_t lead_full0 = ptx::mapa_shared(full0, 0);
    uint32_t stage = 0, phase = 0;
    uint32_t armed = 0, armed_phase = 0;  // bit i: stage i was armed / the phase bit of its last arming
    for (int32_t t = pair; t < total; t += pairs) {
      int32_t row0, n0;
      tile_of(t, row0, n0);
      n0 += (int32_t)rank * (BN / 2);
      bool ok = true;
      for (int32_t kb = 0; kb < p.k_tiles; ++kb) {
        if (!ptx::mbar_wait_a(empty0 + stage * 8, phase ^ 1)) {
          timeout(ctl, 51);
          ok = false;
          break;
        }
        armed |= 1u << stage;
        armed_phase = (armed_phase & ~(1u << stage)) | (phase << stage);
        if (leader) {
          const uint32_t dst = stage0 + stage * kStageBytes;
          if (rank == 0) ptx::mbar_arrive_expect_tx_a(full0 + stage * 8, 2 * kStageBytes);  // both CTAs' bytes
          ptx::tma_load_2d_pair(dst, &map_a, lead_full0 + stage * 8, kb * BK, row0);
          ptx::tma_load_2d_pair(dst + kTileABytes, &map_b, lead_full0 + stage * 8, kb * BK, n0);
        }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
      if (!ok || ctl->abort_flag) break;
    }
    if (ctl->abort_flag) {
      // After a time-out: no CTA may exit while bulk copies into its shared memory are in flight.  Both CTAs' copies are counted on
      // the even CTA's `full` barriers, so the even CTA waits (20 ms at most per stage) for the stages it announced; the
      // cluster barrier at the exit then holds the partner until that is done.
      if (rank == 0)
        for (uint32_t i = 0; i < (uint32_t)kStages; ++i)
          if (armed & (1u << i)) ptx::mbar_wait_a(full0 + i * 8, (armed_phase >> i) & 1u, 20000000ull);
    } else {
      // the last arrivals on `empty` come from asynchronous commits: take every stage once more before leaving
      for (int i = 0; i < kStages; ++i) {
        if (!ptx::mbar_wait_a(empty0 + stage * 8, phase ^ 1)) { timeout(ctl, 55); break; }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1 || warp == 3) {
    // ===== scale loaders: groups alternate between the two warps, the words of a warp's next group are on their way while it
    // writes this one's.  One warp alone, loads and all one after the other, held the kernel at 890 cycles a k-block (4096 x 7168 x 18432 487 us, not 368).
    const uint32_t lead_sf_full0 = ptx::mapa_shared(sf_full0, 0), me = warp >> 1;
    const int32_t nb_last = (p.N + 127) / 128 - 1;
    uint32_t a[4], b[8], q = me;
    int32_t t = pair, kg = me;  // the group after the one in registers
    auto fetch = [&] {
      while (kg >= p.k_groups && t < total) {
        kg -= p.k_groups;
        t += pairs;
      }
      if (t >= total) return false;
      int32_t row0, n0;
      tile_of(t, row0, n0);
      const int32_t* a_col = p.sfa + (int64_t)kg * p.sfa_ld;
      const int32_t* b_col = p.sfb + (int64_t)kg * p.sfb_stride_k;
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] = (uint32_t)__ldg(a_col + min(row0 + 32 * j + lane, p.M - 1));
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] = (uint32_t)__ldg(b_col + (int64_t)min((n0 + 32 * j + lane) / 128, nb_last) * p.sfb_stride_n);
      kg += 2;
      return true;
    };
    bool have = fetch();
    while (have) {
      const uint32_t buf = q % kSfBufs;
      if (!ptx::mbar_wait_a(sf_empty0 + buf * 8, ((q / kSfBufs) & 1) ^ 1)) {
        timeout(ctl, 56);
        break;
      }
      uint4* dst = reinterpret_cast<uint4*>(sf_smem + (size_t)buf * kSfBufBytes) + lane;
      dst[0] = make_uint4(a[0], a[1], a[2], a[3]);
      dst[32] = make_uint4(b[0], b[1], b[2], b[3]);
      dst[64] = make_uint4(b[4], b[5], b[6], b[7]);
      ptx::fence_proxy_async();  // the tensor core reads this block through the async proxy
      have = fetch();
      __syncwarp();
      if (lane == 0) {
        // the odd CTA's write is published to the thread of the even CTA that has the tensor core read it
        if (rank == 0) ptx::mbar_arrive_a(sf_full0 + buf * 8);
        else ptx::mbar_arrive_release_cluster(lead_sf_full0 + buf * 8);
      }
      q += 2;
      if (ctl->abort_flag) break;
    }
    // Tail, as for the producer: the commits on this warp's scale buffers must have arrived.
    if (!ctl->abort_flag) {
      for (int i = 0; i < kSfBufs / 2; ++i, q += 2) {
        if (!ptx::mbar_wait_a(sf_empty0 + (q % kSfBufs) * 8, ((q / kSfBufs) & 1) ^ 1)) { timeout(ctl, 58); break; }
      }
    }
  } else if (warp == kMmaWarp) {
    if (rank == 0) {
      // ===== MMA issuer
      const uint64_t desc0 = ptx::make_kmajor_sw128_desc(stage0);
      const uint32_t sf0 = ptx::smem_u32(sf_smem);
      uint32_t stage = 0, phase = 0, q = 0, tile_i = 0;
      for (int32_t t = pair; t < total; t += pairs, ++tile_i) {
        const uint32_t as = tile_i & 1;  // accumulator of this tile
        bool ok = ptx::mbar_wait_a(acc_empty0 + as * 8, ((tile_i >> 1) & 1) ^ 1);
        if (!ok) timeout(ctl, 52);
        const uint32_t d_tmem = tmem_base + as * BN;
        for (int32_t kg = 0; kg < p.k_groups && ok; ++kg, ++q) {
          const uint32_t buf = q % kSfBufs;
          if (!ptx::mbar_wait_a(sf_full0 + buf * 8, (q / kSfBufs) & 1)) {
            timeout(ctl, 53);
            ok = false;
            break;
          }
          ptx::tc_fence_after();
          const uint32_t sf_col = tmem_base + kSfTmemBase + (q & 1) * kSfTmemPerSet;
          if (leader) {
            const uint32_t src = sf0 + buf * kSfBufBytes;
            ptx::tmem_cp_32x128b_warpx4_pair(sf_col, ptx::make_sf_desc(src));
            ptx::tmem_cp_32x128b_warpx4_pair(sf_col + 4, ptx::make_sf_desc(src + kSfABytes));
            ptx::tmem_cp_32x128b_warpx4_pair(sf_col + 8, ptx::make_sf_desc(src + kSfABytes + 512));
            ptx::mma_commit_pair_a(sf_empty0 + buf * 8);
          }
          const int32_t kb_end = min(kg * 4 + 4, p.k_tiles);
          for (int32_t kb = kg * 4; kb < kb_end; ++kb) {
            if (!ptx::mbar_wait_a(full0 + stage * 8, phase)) {
              timeout(ctl, 54);
              ok = false;
              break;
            }
            ptx::tc_fence_after();
            if (leader) {
              const uint64_t a_desc = desc0 + (uint64_t)(stage * (kStageBytes >> 4));
              const uint64_t b_desc = a_desc + (kTileABytes >> 4);
              const uint32_t idesc = ptx::make_idesc_mxf8(256, BN, (uint32_t)(kb & 3));
              ptx::mma_mxf8_block_scaled_pair(d_tmem, a_desc, b_desc, idesc, sf_col, sf_col + 4, kb > 0 ? 1u : 0u);
#pragma unroll
              for (uint32_t k = 1; k < BK / 32; ++k)
                ptx::mma_mxf8_block_scaled_pair(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, sf_col, sf_col + 4, 1u);
              ptx::mma_commit_pair_a(empty0 + stage * 8);
            }
            if (++stage == kStages) { stage = 0; phase ^= 1; }
          }
        }
        if (!ok || ctl->abort_flag) break;
        if (leader) ptx::mma_commit_pair_a(acc_full0 + as * 8);  // the tile is complete when everything issued so far is
      }
    }
  } else if (warp >= kEpiWarp0) {
    // ===== epilogue: TMEM lane quarter = warp % 4; the quarter's seven boxes of 32 columns go 4 : 3 to its two warps
    const int qd = warp & 3, half = (warp - kEpiWarp0) >> 2;
    const uint32_t lead_acc_empty0 = ptx::mapa_shared(acc_empty0, 0);
    const uint32_t box = stage0 + (uint32_t)kBoxOffset + (warp - kEpiWarp0) * kBoxBytes;
    uint32_t tile_i = 0;
    for (int32_t t = pair; t < total; t += pairs, ++tile_i) {
      int32_t row0, n0;
      tile_of(t, row0, n0);
      const uint32_t as = tile_i & 1;
      if (!ptx::mbar_wait_a(acc_full0 + as * 8, (tile_i >> 1) & 1)) {
        timeout(ctl, 57);
        break;
      }
      ptx::tc_fence_after();
      const uint32_t tlane = tmem_base + ((uint32_t)(qd * 32) << 16) + as * BN + half * 128;
      const int32_t row_base = row0 + qd * 32, boxes = 4 - half;
#pragma unroll 1
      for (int i = 0; i < boxes; ++i) {
        uint32_t v[32];
        ptx::tmem_ld_32x32(tlane + i * 32, v);
        ptx::tmem_ld_wait(v);
        if (i == boxes - 1) {
          // all TMEM reads of this tile have landed: the issuer may overwrite this accumulator
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(lead_acc_empty0 + as * 8);
        }
        const int32_t c0 = n0 + half * 128 + i * 32;
        if (c0 < p.N && row_base < p.M) {  // uniform over the warp
          if (leader) ptx::bulk_wait_read();  // the store before has read the box
          __syncwarp();
          if (p.out_dtype == SGLB200_BF16) fill_box<__nv_bfloat16>(v, p.bias, box, c0, p.N, lane, SGLB200_BF16);
          else fill_box<__half>(v, p.bias, box, c0, p.N, lane, SGLB200_F16);
          ptx::fence_proxy_async();
          __syncwarp();
          if (leader) ptx::tma_store_2d(&map_out, box, c0, row_base);
        }
      }
      if (ctl->abort_flag) break;
    }
    if (leader) ptx::bulk_wait_read();  // the boxes must outlive their stores
  }

  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();  // neither CTA leaves while the other may still signal its barriers or read its tiles
  if (warp == kMmaWarp) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace

// Nanoseconds that this kernel takes for a dense problem, about; for ue8m0_common's choice, fitted to runs of one call at a time (11
// layers of N = 576 to 36864, K = 1024 to 16384, 160 to 4096 rows).  Above 128 rows the pairs are 5 to 38 % ahead of the single
// CTAs, except where those need fewer waves (384 x 10240 x 8192 41 against 30 us) or K is a few k-blocks and their later start
// counts (K = 1024 8.2 against 7.2).
int64_t ue8m0_pair_cost(int64_t M, int64_t N, int64_t K, int sm_count) {
  const int64_t pairs = sm_count / 2;
  if (pairs == 0) return INT64_MAX;
  return 1500 + (((M + 255) / 256) * ((N + BN - 1) / BN) + pairs - 1) / pairs * ((K + BK - 1) / BK * 300 + 600);
}

// Dense UE8M0 GEMM on CTA pairs; arguments checked by the caller (ue8m0_common).
int ue8m0_pair_gemm(const void* a, const void* b, const int32_t* sfa, const int32_t* sfb, const void* bias, void* out, int64_t M, int64_t N,
                    int64_t K, int64_t lda, int64_t ldb, int64_t ldc, int64_t sfa_ld, int64_t sfb_stride_n, int64_t sfb_stride_k,
                    int out_dtype, int sm_count, void* stream) {
  static bool attr_done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(fp8_ue8m0_gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return fail(SGLB200_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    attr_done[dev] = true;
  }
  alignas(64) CUtensorMap map_a, map_b, map_out;
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t str[1] = {(uint64_t)lda};
    if (int rc = make_map_sw128(&map_a, a, 2, dims, str, 128, CU_TENSOR_MAP_L2_PROMOTION_L2_128B)) return rc;
  }
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)N};
    const uint64_t str[1] = {(uint64_t)ldb};
    if (int rc = make_map_sw128(&map_b, b, 2, dims, str, BN / 2, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) return rc;
  }
  if (int rc = make_map_out16(&map_out, out, (uint64_t)N, (uint64_t)M, (uint64_t)ldc * 2, 32, 32)) return rc;
  PairParams p;
  p.sfa = sfa;
  p.sfb = sfb;
  p.bias = bias;
  p.M = (int32_t)M;
  p.N = (int32_t)N;
  p.m2_tiles = (int32_t)((M + 255) / 256);
  p.n_tiles = (int32_t)((N + BN - 1) / BN);
  p.k_tiles = (int32_t)((K + BK - 1) / BK);
  p.k_groups = (p.k_tiles + 3) / 4;
  p.sfa_ld = sfa_ld;
  p.sfb_stride_n = sfb_stride_n;
  p.sfb_stride_k = sfb_stride_k;
  p.out_dtype = out_dtype;
  const int64_t tiles = (int64_t)p.m2_tiles * p.n_tiles;
  int64_t pairs = sm_count / 2;
  if (tiles < pairs) pairs = tiles;
  fp8_ue8m0_gemm_pair_kernel<<<(unsigned)(2 * pairs), kThreads, kSmem, static_cast<cudaStream_t>(stream)>>>(map_a, map_b, map_out, p);
  SGLB_CHECK_LAUNCH("fp8_ue8m0_gemm_pair_kernel");
  note_gemm("fp8_ue8m0_gemm_pair_kernel");
  return SGLB200_OK;
}

}  // namespace sglb
