// Block-scaled FP8 GEMM for few rows of activations (up to 64, or 256 where clusters share K: the decode case), weight-streaming bound.
//
// The roles of the operands are swapped: the tensor core computes C^T = W * A^T, a tile being 128 WEIGHT rows (the MMA's
// M) by MT token columns (the MMA's N, MT = 16 / 32 / 64 / 128, and as few of them as the item has rows).  An accumulator
// stage is then only MT TMEM columns wide, so 4 to 11 k-blocks are in flight between the MMA warp and the promotion warps, and
// a shared-memory stage is 16 KB of weights plus MT x 128 bytes of activations, 6 to 11 of them: 64 KB of weights in flight
// per SM already bring a plain stream of such tiles to 90 % of the HBM rate, 128 KB to all of it.  When N / 128 tiles alone cannot
// occupy the SMs, the CTAs of a cluster cut a tile's K among themselves and add their sums up out of each other's shared memory, each
// a share of the tile (smallm_cluster, add_up_share).  Against fp32 partial sums in memory and a kernel that adds them, quantiser
// included, N=576 K=7168 M=1 / 48 went 9.6 / 14.1 -> 6.8 / 11.1 us, N=7168 K=16384 M=48 32.3 -> 27.1, N=10240 K=8192 M=48 27.0 -> 22.1
// with rank 0 adding everything; 4.7 / 7.8, 26.6 and 20.9 are calls of the present kernel.
// Where clusters share K eight promotion warps share every accumulator stage from 33 rows on; from 65 to 128 rows without (partial
// sums for the peer exchange, the only such calls left) sixteen do.
//
// One barrier each way per k-block.  `full` counts the producer's bytes, the scale loader and the promotion warps, who arrive for the
// k-block that gets the TMEM stage they have just read; `done` is one commit, on which the producer, the scale loader and the
// promotion warps wait.  A wait on a barrier that is ready costs its warp about 120 cycles and a commit 60: with a barrier per ring
// (two waits, two commits) a k-block took the one issuing warp 500 cycles with everything ready, so 337, and issued under a
// predicate instead of a branch 256 at 128 columns, which is what the MMAs take.  The scales have no barrier of their own: the
// promotion warps, who wait for `done` alone, ask `full` too, which is complete by then, so that they acquire what the loader
// released there.  These warps are what is left: they ask
// for the next k-block before they add, step through the rings by offsets and take four k-blocks a turn (a turn each: 4 to 10 % slower).  Two
// waits and two commits -> this, GEMM alone, weights from HBM, us: 48 x 10240 x 8192 21.8 -> 18.6, 64 x 7168 x 16384 27.5 -> 24.6, 32 x
// 10240 x 8192 18.0 -> 16.7, 48 x 24576 x 1536 13.2 -> 11.4, 96 x 7168 x 16384 31.4 -> 30.5, 16 x 7168 x 16384 22.2 -> 21.5.
// Measured against scales that every promotion warp fetched and spread by shuffles, weights from HBM (B200):
// N=36864 K=7168 M=32 / 64 / 128: 46.6 / 54.8 / 75.0 -> 41.8 / 43.3 / 55.1 us (6.1 TB/s at 64 rows);
// N=24576 K=1536 M=16 / 64 / 128: 8.4 / 15.4 / 21.8 -> 7.7 / 9.8 / 13.9 us.
//
// GROUPED variant (one weight matrix per expert, few rows per expert: the decode case of a mixture-of-experts layer): a
// work item is (expert, 128 weight rows, chunk of MT of the expert's rows).  The row ranges come from the same device
// tables as in the 128 x 128 grouped kernel; an expert with more than MT rows gets several chunks (its weight tile is
// then re-read, from L2), an expert without rows gets no item, so only the weights of routed experts are streamed.
//
// warp 0: TMA producer; warp 1: TMEM owner + MMA issuer; warp 2: scale loader (sa[token] * sb into a slot per k-block), or
// up to eight rows warps 2, 3 and 8..15: quantisers (QUANT); warps 4..7
// (..11, ..19): promotion (tcgen05.ld, acc += p * scale) and the transposed store.  All waits are bounded.
//
// The kernel is launched with programmatic stream serialization: it may start while the kernel before it (the
// activation quantiser, or the previous layer's reduce kernel) is still running.  Its set-up and the WEIGHT tiles of the
// first ring of stages are issued at once (up to 128 rows), ahead of griddepcontrol.wait; the activation tiles, all scales and
// every store come after it.  The kernel starts when all blocks of the one before have ended, or have released it early: of this
// library's kernels that write e4m3 codes only those for activations do that (quant.cu), and callers' own kernels that write weights
// must not.  At decode sizes the fixed cost of a call (launch, set-up, first TMA round trip) is of the order of the streaming time
// itself, and this hides most of it.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"
#include "quant_math.cuh"
#include "quant_vec.cuh"

namespace sglb {

// device status word of this translation unit (0 = no bounded wait ran out); collected by sglb200_read_device_status
__device__ int g_smallm_status = 0;

int smallm_take_device_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_smallm_status, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  if (v != 0) {
    const int z = 0;
    cudaMemcpyToSymbol(g_smallm_status, &z, sizeof(int));
  }
  return v;
}

namespace {

constexpr int BN = 128, BK = 128;  // weight rows per tile, K per block
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kWBytes = BN * BK;
constexpr int kScaleGroup = 4;   // k-blocks whose scales the loader fetches at once
constexpr uint32_t kCtlBytes = 256;
constexpr uint32_t kPatchRow = 80, kPatchBytes = 16 * kPatchRow;  // epilogue patch of a warp: 16 tokens x 64 bytes, padded

constexpr int kAuxRegs = 96, kPromoRegs = 200;  // register split of the NSUB = 2 form (four and eight warps)

constexpr int kMaxExperts = 1024;

// NSUB > 1: the MMA covers up to MT * NSUB activation rows and every set of four promotion warps takes its MT of every accumulator
// stage's columns.  Two sets of 32 from 33 to 64 rows in a cluster (launch_cluster); at 65 to 128 rows two sets of 64 there (call, two
// sets / four, us: 113 x 7168 x 16384 35.1 / 36.0, 128 x 576 x 7168 10.8 / 11.7, 113 x 2048 x 2048 8.8 / 9.4), and four of 32 alone on a
// tile, where 16 warps hide each other's chain of wait, load, hand-back and FMA (measured when such calls came here: N=10240 K=8192 M=113
// 31.3 -> 30.1 us, N=24576 K=1536 18.7 -> 17.6, N=36864 K=7168 65 -> 59 against two sets of 64).
template <int MT, int NSUB = 1>
struct Cfg {
  static constexpr int kTile = MT * NSUB;  // most activation rows per work item = TMEM columns per stage
  static constexpr int kStages = kTile == 128 ? 6 : (kTile == 64 ? 8 : (kTile == 32 ? 10 : 11));
  static constexpr int kAcc = (512 / kTile) < kStages ? (512 / kTile) : kStages;
  static constexpr int kThreads = 128 + 128 * NSUB;
  static constexpr uint32_t kABytes = kTile * BK;
  static constexpr uint32_t kStageBytes = kWBytes + kABytes;
  // Slots of kTile scale products, one per k-block.  Slot j + kStages is written when the MMAs of j are done; those were issued
  // after every promotion warp had read the sums of j - kAcc, and its scales before them.
  static constexpr int kScaleSlots = 2 * kStages;
  static constexpr uint32_t kSlotBytes = kTile * sizeof(float), kScaleBytes = kScaleSlots * kSlotBytes;
  static constexpr size_t kPatchOffset = (size_t)kStages * kStageBytes + kScaleBytes;
  static constexpr size_t kSmem = 1024 + kPatchOffset + 4 * NSUB * kPatchBytes + kCtlBytes;
  // grouped: the tables of rows and of first work items per expert follow the control block
  static constexpr size_t smem_grouped(size_t experts) { return kSmem + experts * sizeof(int2) + (experts + 1) * sizeof(int32_t) + 12; }
  static_assert((kTile > 64 ? kSmem : kSmem + kMaxExperts * 12 + 16) <= 227 * 1024, "shared memory of one CTA");  // grouped: chunks of up to 64 rows
};

struct SmallParams {
  const float* sa;  // UE8M0 variant: int32 words, four exponent bytes (k-blocks 4g .. 4g + 3) per word
  const float* sb;
  void* out;
  const void* bias;  // [N] of the output type, or NULL: added to the rounded result
  float* partial;    // fp32 sums [splits][M][N] instead of `out`
  int32_t cluster;   // > 1: the CTAs of a cluster share one tile's K and add their sums up (k_splits == cluster)
  int32_t chunks, chunk_rows;  // cluster form: M rows in `chunks` of chunk_rows, one work item each
  int32_t M, N, K;
  int32_t n_tiles, k_tiles, k_splits, kb_per_split;
  int64_t ldc;
  int64_t sa_stride_m, sa_stride_k, sb_stride_n, sb_stride_k;
  int32_t out_dtype;
  // grouped only
  const int32_t* expert_offsets;  // [E + 1] first row of every expert, or NULL in the masked layout
  const int32_t* problem_sizes;   // optional: rows of expert e = problem_sizes[count_stride * e]
  int32_t count_stride, rows_per_expert, num_experts;
  int64_t sa_stride_e, sb_stride_e;
  // QUANT form: rows not quantised yet, [M, K] of the output type, and the quantiser's floor
  const void* x;
  float eps;
};

// one unit of work: rows [row0, row0 + rows) of the activations against weight rows [nt * 128, +128) of expert e,
// k-blocks [kb0, kb1)
struct Item {
  int32_t e, nt, row0, rows, kb0, kb1, split;
};

__device__ __forceinline__ void expert_rows(const SmallParams& p, int32_t e, int32_t* r0, int32_t* cnt) {
  if (p.rows_per_expert > 0) {
    *r0 = e * p.rows_per_expert;
    *cnt = max(0, min(__ldg(p.problem_sizes + p.count_stride * e), p.rows_per_expert));
  } else {
    *r0 = __ldg(p.expert_offsets + e);
    *cnt = max(0, p.problem_sizes ? __ldg(p.problem_sizes + p.count_stride * e) : __ldg(p.expert_offsets + e + 1) - *r0);
  }
}

// Work item t.  Grouped: `e` is the expert of an earlier item of this warp (0 at first), from which its 32 lanes look for that of t side
// by side; the rows come from shared memory.
template <int TILE, bool GROUPED, bool CLUSTER>
__device__ __forceinline__ Item get_item(const SmallParams& p, const int2* expert, const int32_t* item_start, int32_t t, int32_t& e) {
  Item it;
  if constexpr (!GROUPED) {
    it.row0 = 0;
    it.rows = p.M;
    if constexpr (CLUSTER) {
      it.nt = t / p.cluster;
      it.split = t - it.nt * p.cluster;
      if (p.chunks > 1) {  // chunks of one weight tile side by side: it comes from HBM once
        const int32_t tile = it.nt;
        it.nt = tile / p.chunks;
        it.row0 = (tile - it.nt * p.chunks) * p.chunk_rows;
        it.rows = min(p.chunk_rows, p.M - it.row0);
      }
    } else {
      it.split = t / p.n_tiles;
      it.nt = t - it.split * p.n_tiles;
    }
    it.kb0 = it.split * p.kb_per_split;
    it.kb1 = min(it.kb0 + p.kb_per_split, p.k_tiles);
    it.e = 0;
  } else {
    const int32_t lane = threadIdx.x & 31;
    for (;;) {  // last e with item_start[e] <= t
      const int32_t n = e + 1 + lane;
      const int32_t k = __popc(__ballot_sync(0xffffffffu, n < p.num_experts && item_start[n] <= t));
      e += k;
      if (k < 32) break;
    }
    const int32_t r0 = expert[e].x, cnt = expert[e].y;
    const int32_t chunks = (cnt + TILE - 1) / TILE;
    const int32_t local = t - item_start[e];
    it.e = e;
    it.nt = local / chunks;
    const int32_t ch = local - it.nt * chunks;
    const int32_t per = (cnt + chunks - 1) / chunks;  // chunks of even size: the MMA is as wide as the chunk
    it.row0 = r0 + ch * per;
    it.rows = min(per, cnt - ch * per);
    it.kb0 = 0;
    it.kb1 = p.k_tiles;
    it.split = 0;
  }
  return it;
}

struct Ctl {
  uint64_t full[12];  // k-block g may be multiplied: operands and scales have arrived, its TMEM stage has been read out
  uint64_t done[12];  // k-block g has been multiplied: its operands may be overwritten, its sums be read
  uint32_t tmem_base;
  volatile int32_t abort_flag;
  int32_t total;
};
static_assert(sizeof(Ctl) <= kCtlBytes, "control block");

__device__ __forceinline__ void timeout(Ctl* ctl, int code) {
  ctl->abort_flag = 1;
  atomicCAS(&g_smallm_status, 0, code);
}

// 16 lanes x 8 * G fp32 columns in the accumulator-fragment arrangement: registers 4g + {0, 1} of thread t hold lane t / 4,
// columns 8g + 2 * (t % 4) + {0, 1}; registers 4g + {2, 3} the same columns of lane t / 4 + 8.
template <int G>
__device__ __forceinline__ void tmem_ld_16x256(uint32_t taddr, uint32_t* r);
template <>
__device__ __forceinline__ void tmem_ld_16x256<2>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x2.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_16x256<4>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld_16x256<8>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// wait for this thread's outstanding tcgen05.ld; the registers are tied to the statement so that their first use
// cannot move above it
template <int N>
__device__ __forceinline__ void tmem_ld_fence(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i])::"memory");
}

// The 32 bits that hold the scale of k-block kc: fp32 at base[kc * stride_k], or the packed word at base[(kc / 4) * stride_k], whose
// byte kc % 4 stands for 2^(byte - 127).  Loads that are to stay in flight are decoded where they are used, not here.
template <bool UE>
__device__ __forceinline__ float load_scale_bits(const float* base, int32_t kc, int64_t stride_k) {
  return __ldg(base + (int64_t)(UE ? kc >> 2 : kc) * stride_k);
}
template <bool UE>
__device__ __forceinline__ float scale_of(float bits, int32_t kc) {
  return UE ? __uint_as_float(((__float_as_uint(bits) >> (8 * (kc & 3))) & 0xffu) << 23) : bits;
}
template <bool UE>
__device__ __forceinline__ float load_scale(const float* base, int32_t kc, int64_t stride_k) {
  return scale_of<UE>(load_scale_bits<UE>(base, kc, stride_k), kc);
}

// Four 8 x 8 matrices of 16-bit values in fragment arrangement, stored transposed: lane l passes the address of row l % 8 of
// matrix l / 8.
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c),
               "r"(d)
               : "memory");
}
// two of them: lanes 0 to 15 pass the addresses
__device__ __forceinline__ void stmatrix_x2_trans(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("stmatrix.sync.aligned.m8n8.x2.trans.shared.b16 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ uint32_t pack16(float a, float b, int out_dtype) {
  if (out_dtype == SGLB200_BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Ten warps (2, 3 and 8 to 15) of the QUANT form, up to eight rows: the activations come as they are, and these warps quantise them
// on their way into the ring, with the arithmetic of the separate quantiser.  Each takes every tenth k-block whole, four rows a pass,
// with the rows of its next k-block in flight while it waits for its stage.  Every CTA does so for all k-blocks it multiplies, which
// is less work than the weights take to arrive, and saves a kernel and the hand-over from it.
//
// Eight rows are the limit (smallm_quantises) because of what these loads take where the rows have just been written by another kernel:
// by the times of calls about 2 us beside the weight stream, against the 2.8 us in which 112 CTAs go through ten k-blocks.  With one or two passes of
// conversion that fits in, with three or four it does not, and every k-block waits.  With registers for four passes the block also left
// no room on its SM for another kernel's (94 a thread now, 127 then).  Graph of calls, quantiser kernel / this, us, at 4 / 8 rows:
// 576 x 7168 6.2 / 6.4 -> 4.8 / 5.1, 24576 x 1536 10.4 / 10.3 -> 8.6 / 8.7, 7168 x 16384 23.6 / 24.1 -> 21.7 / 21.9, 36864 x 7168 42.3 / 42.2 ->
// 40.5 / 40.6.  The same with rms_norm before each call and a bf16 matmul, softmax and top-k behind it, this less the kernel, at 4 / 8 rows:
// -0.7 / -1.0, 0.0 / -0.2, -0.9 / -1.0, -0.6 / -0.2; with three and four passes, at 9 / 16 rows: +0.3 / +0.8, +1.1 / +2.5, +3.2 / +5.1, +3.1 /
// +4.7, which a graph of nothing but such calls did not show (24.7 -> 23.1 at 16 x 7168 x 16384).  Five projections of a layer in
// turn: 140 -> 138 / 139, and 153 / 161 at 9 / 16 rows.  Rows asked for into the L2 ahead: level where they were not there, 1 us
// slower where they were.
//
// A warp's wait for a stage looks at one parity, which is right only if the stage's k-block before last is known to be done; the
// warp's wait for its own k-block before this one says so if that one is at most a ring back (commits arrive in order).
constexpr int kQuantRows = 2;  // rows that a call may pass without scratch
constexpr int kQuantWarps = 10;
static_assert(kQuantWarps <= Cfg<16>::kStages, "see above");

template <typename T, int PASSES, bool UE, bool CLUSTER>
__device__ __forceinline__ void quantise_rows(const SmallParams& p, Ctl* ctl, uint8_t* smem, float* scale_ring, uint32_t me, int lane,
                                              int32_t total) {
  using C = Cfg<16>;
  static_assert(kMaxQuantRows == 8 && (PASSES == 1 || PASSES == 2), "four rows a pass");
  const uint32_t full0 = ptx::smem_u32(&ctl->full[0]), done0 = ptx::smem_u32(&ctl->done[0]);
  const int rows = p.M, sub = lane & 7, r0 = lane >> 3;  // eight lanes, sixteen elements each, take a row of a pass
  const uint4* row[PASSES];
#pragma unroll
  for (int u = 0; u < PASSES; ++u)  // rows past the last one are read as the last one, and not stored
    row[u] = reinterpret_cast<const uint4*>(static_cast<const T*>(p.x) + (int64_t)min(4 * u + r0, rows - 1) * p.K) + 2 * sub;
  const float inv_max = __frcp_rn(448.0f);
  const int scale_row = sub + r0;  // the row whose scale this lane has, if it is lane 0 or 4 of the eight
  const bool has_scale = (sub & 3) == 0 && scale_row < rows;
  uint32_t stage = me, phase = 0, slot = me;
  int32_t i = (int32_t)me;  // this warp's next k-block, counted from the item's first
  for (int32_t t = blockIdx.x; t < total; t += gridDim.x) {
    int32_t none = 0;
    const Item it = get_item<C::kTile, false, CLUSTER>(p, nullptr, nullptr, t, none);
    const float* sb_blk = p.sb + (int64_t)it.nt * p.sb_stride_n;
    uint4 v[PASSES][2];
    float b = 0.f;
    auto fetch = [&](int32_t kb) {
      b = load_scale<UE>(sb_blk, kb, p.sb_stride_k);
#pragma unroll
      for (int u = 0; u < PASSES; ++u) {
        v[u][0] = __ldg(row[u] + (int64_t)kb * (BK / 8));
        v[u][1] = __ldg(row[u] + (int64_t)kb * (BK / 8) + 1);
      }
    };
    const int32_t n = it.kb1 - it.kb0;
    if (i < n) fetch(it.kb0 + i);
    for (; i < n; i += kQuantWarps) {
      // Maxima of both passes at once: lanes 0 to 3 of a row's eight end up with that of the first pass, 4 to 7 with the second's
      float amax = fmaxf(Elem<T>::vec_absmax(v[0][0]), Elem<T>::vec_absmax(v[0][1]));
      float other = amax;  // what the lane four away is to have
      if constexpr (PASSES == 2) {
        const float second = fmaxf(Elem<T>::vec_absmax(v[1][0]), Elem<T>::vec_absmax(v[1][1]));
        if (sub & 4) amax = second;
        else other = second;
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, other, 4));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      amax = fmaxf(p.eps, fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1)));
      uint4 codes[PASSES];
      float s;
      // no branch inside the passes where every scale is an ordinary number, so that they run side by side
      if (__all_sync(0xffffffffu, amax >= 1e-27f && amax <= 1e30f)) {
        s = group_scale_fast(amax, 448.0f, inv_max, UE, true);
        const float r = __frcp_rn(s);
#pragma unroll
        for (int u = 0; u < PASSES; ++u)
          codes[u] = encode16_e4m3<T, true>(v[u][0], v[u][1], __shfl_sync(0xffffffffu, s, 4 * u, 8), __shfl_sync(0xffffffffu, r, 4 * u, 8));
      } else {
        s = group_scale_fast(amax, 448.0f, inv_max, UE);
#pragma unroll
        for (int u = 0; u < PASSES; ++u) codes[u] = encode16_e4m3<T>(v[u][0], v[u][1], __shfl_sync(0xffffffffu, s, 4 * u, 8));
      }
      const float prod = s * b;
      if (i + kQuantWarps < n) fetch(it.kb0 + i + kQuantWarps);
      if (!ptx::mbar_wait_inl_a(done0 + stage * 8, phase ^ 1)) { timeout(ctl, 11); return; }
      (void)ptx::mbar_test_wait_a(full0 + stage * 8, phase ^ 1);  // the promotion warps have read this slot: see there
      uint8_t* dst = smem + (size_t)stage * C::kStageBytes + kWBytes;
#pragma unroll
      for (int u = 0; u < PASSES; ++u) {
        const int r = 4 * u + r0;
        if (r < rows) *reinterpret_cast<uint4*>(dst + r * 128 + ((sub ^ r) << 4)) = codes[u];  // 128-byte swizzle
      }
      if (has_scale) scale_ring[slot * C::kTile + scale_row] = prod;
      ptx::fence_proxy_async();  // the MMA reads shared memory through the asynchronous proxy
      __syncwarp();
      ptx::mbar_arrive_if(full0 + stage * 8, lane == 0);
      stage += kQuantWarps;
      if (stage >= (uint32_t)C::kStages) { stage -= C::kStages; phase ^= 1; }
      slot += kQuantWarps;
      if (slot >= (uint32_t)C::kScaleSlots) slot -= C::kScaleSlots;
    }
    i -= n;
    if (ctl->abort_flag) return;
  }
}

template <typename T, bool UE, bool CLUSTER>
__device__ __forceinline__ void quantise_rows(const SmallParams& p, Ctl* ctl, uint8_t* smem, float* scale_ring, uint32_t me, int lane,
                                              int32_t total) {
  if (p.M <= 4) quantise_rows<T, 1, UE, CLUSTER>(p, ctl, smem, scale_ring, me, lane, total);
  else quantise_rows<T, 2, UE, CLUSTER>(p, ctl, smem, scale_ring, me, lane, total);
}

// One CTA's share of a tile whose K a cluster of RANKS cuts.  A piece is 16 weight rows x 8 tokens of a warp's 32 x MT sums, 16 bytes a
// lane, piece 2g + h for token group g and half h of the rows; the CTAs take equal runs of the pieces that have rows, and add them in
// the order of K.  All loads of a turn (eight) are in flight at once: a round trip through another CTA's shared memory is what
// bounds this.  Rank 0 adding up everything, rank after rank, took
// seven round trips in clusters of eight, each over the whole tile.  Calls, weights from HBM, us, that -> this, M = 1 / 16 / 64 / 128: 576 x 7168
// 5.6 / 7.1 / 11.3 / 18.7 -> 4.8 / 5.9 / 7.9 / 10.8, 1536 x 7168 6.2 / 7.8 / 12.3 / 20.3 -> 5.5 / 6.6 / 8.8 / 11.8, 4096 x 4096 (four) 6.6 / 8.1 /
// 11.4 / 16.8 -> 6.3 / 7.7 / 9.4 / 12.6, 7168 x 16384 (two) 26.7 -> 26.4 at 64.  With 16 loads a turn the kernel spilled in its main loop and
// took twice as long.
template <int RANKS>
__device__ __forceinline__ void add_up_share(const SmallParams& p, uint32_t local, uint8_t* patch, int32_t rank, int32_t row0, int32_t rows,
                                             int32_t n_warp, int lane) {
  constexpr int kTurn = RANKS == 2 ? 4 : (RANKS == 4 ? 2 : 1);  // pieces a turn
  const int32_t pieces = 2 * ((rows + 7) >> 3), per = (pieces + RANKS - 1) / RANKS;
  const int32_t first = rank * per, last = min(first + per, pieces);
  char* out = static_cast<char*>(p.out) + ((int64_t)row0 * p.ldc + n_warp) * 2;
  const char* bias = static_cast<const char*>(p.bias);
  const uint32_t st_addr = ptx::smem_u32(patch) + (uint32_t)(lane & 7) * kPatchRow + (uint32_t)((lane >> 3) & 1) * 16;
#pragma unroll 1
  for (int32_t e0 = first; e0 < last; e0 += kTurn) {
    float4 v[kTurn][RANKS];
#pragma unroll
    for (int k = 0; k < kTurn; ++k)
#pragma unroll
      for (int r = 0; r < RANKS; ++r)  // past the last piece: that one again, not stored
        v[k][r] = ptx::ld_cluster_f4(ptx::mapa_shared(local + (uint32_t)min(e0 + k, last - 1) * 32 * (uint32_t)sizeof(float4), (uint32_t)r));
    __syncwarp();  // the patch has been read out
#pragma unroll
    for (int k = 0; k < kTurn; ++k) {
      float4 sum = v[k][0];
#pragma unroll
      for (int r = 1; r < RANKS; ++r) {
        sum.x += v[k][r].x;
        sum.y += v[k][r].y;
        sum.z += v[k][r].z;
        sum.w += v[k][r].w;
      }
      stmatrix_x2_trans(st_addr + (k >> 1) * 8 * kPatchRow + (k & 1) * 32, pack16(sum.x, sum.y, p.out_dtype),
                        pack16(sum.z, sum.w, p.out_dtype));
    }
    __syncwarp();
    // 16 bytes a lane: eight tokens x two halves of a piece's 16 columns, as many pieces as the warp has lanes for
#pragma unroll
    for (int i = 0; i < (kTurn + 1) / 2; ++i) {
      const int32_t k = 2 * i + (lane >> 4), e = e0 + k, tok = 8 * (e >> 1) + (lane & 7), part = (lane >> 3) & 1;
      const int32_t c = (e & 1) * 16 + part * 8;
      if (k < kTurn && e < last && tok < rows && n_warp + c < p.N) {  // N % 8 == 0
        uint4 val = *reinterpret_cast<const uint4*>(patch + (i * 8 + (lane & 7)) * kPatchRow + (lane >> 4) * 32 + part * 16);
        if (bias != nullptr)
          val = ptx::add_bias8(val, __ldg(reinterpret_cast<const uint4*>(bias + (int64_t)(n_warp + c) * 2)), p.out_dtype);
        *reinterpret_cast<uint4*>(out + ((int64_t)tok * p.ldc + c) * 2) = val;
      }
    }
  }
}

// CLUSTER is a template parameter because the mere presence of the adding-up code cost the main loop of the other form up to
// 18 % (N=36864 K=7168 M=113: 57 -> 68 us) through its register allocation.
// QUANT: see quantise_rows.
template <int MT, bool UE, bool GROUPED, int NSUB, bool CLUSTER, bool QUANT>
// NSUB = 1 has 256 threads of at most 166 registers (QUANT: 512 of 94), so that a block of the quantiser or of another small kernel
// (256 threads of 48) fits beside it and programmatic dependent launch really overlaps the two.
__global__ void __launch_bounds__(QUANT ? 192 + 32 * kQuantWarps : (NSUB == 1 ? 320 : 128 + 128 * NSUB), 1)
fp8_block_gemm_smallm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                             const SmallParams p) {
  using C = Cfg<MT, NSUB>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* scale_ring = reinterpret_cast<float*>(smem + (size_t)C::kStages * C::kStageBytes);  // [slot][token]
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + C::kPatchOffset + 4 * NSUB * kPatchBytes);
  int2* expert = reinterpret_cast<int2*>(reinterpret_cast<uint8_t*>(ctl) + kCtlBytes);  // grouped: first row and rows
  int32_t* item_start = reinterpret_cast<int32_t*>(expert + p.num_experts);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::kStages; ++i) {
      // the producer (and its bytes), the scale loader or (QUANT) the warp that wrote codes and scales, every promotion warp
      ptx::mbar_init(&ctl->full[i], 2 + 4 * NSUB);
      ptx::mbar_init(&ctl->done[i], 1);
    }
    ctl->abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async();
    ptx::prefetch_tensormap(&map_w);
    if constexpr (!QUANT) ptx::prefetch_tensormap(&map_a);
  }
  if (warp == 1) {
    ptx::tmem_alloc(&ctl->tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  if constexpr (GROUPED) {
    // The row tables are written by kernels earlier in the stream: nothing of the work list is known before they end.
    ptx::grid_dep_wait();
    if (warp == 2) {  // exclusive prefix sum of work items per expert
      int32_t running = 0;
      for (int32_t base = 0; base < p.num_experts; base += 32) {
        const int32_t e = base + lane;
        int32_t v = 0;
        if (e < p.num_experts) {
          int32_t r0, cnt;
          expert_rows(p, e, &r0, &cnt);
          expert[e] = make_int2(r0, cnt);
          v = ((cnt + C::kTile - 1) / C::kTile) * p.n_tiles;
        }
        int32_t incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int32_t o = __shfl_up_sync(0xffffffffu, incl, d);
          if (lane >= d) incl += o;
        }
        if (e < p.num_experts) item_start[e] = running + incl - v;
        running += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) {
        item_start[p.num_experts] = running;
        ctl->total = running;
      }
    }
  } else {
    if (threadIdx.x == 0) ctl->total = p.n_tiles * p.chunks * p.k_splits;
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  const int32_t total = ctl->total;
  const uint32_t full0 = ptx::smem_u32(&ctl->full[0]), done0 = ptx::smem_u32(&ctl->done[0]);
  const uint32_t stage0 = ptx::smem_u32(smem);

  if (threadIdx.x == 0) ptx::grid_dep_launch();  // the next kernel of the stream may begin its own set-up

  const bool leader = ptx::elect_one();  // the lane that issues TMA and tcgen05 instructions
  // Register split (NSUB = 2): eight promotion warps with 64 accumulators, 64 loaded sums and the scales in flight want more
  // than the 168 registers that 384 threads start with; the other four warps need few: 128 * 96 + 256 * 200 = 63488 <=
  // 384 * 168.  No call may sit in a region with a changed limit, hence the inlined waits.
  if (warp >= 4 && (!QUANT || warp < 8)) {
    if constexpr (NSUB == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPromoRegs));
    // ===== promotion + transposed store; TMEM lane quarter = warp % 4.  A warp owns 32 weight rows (columns of the output)
    // and MT tokens.  The sums are loaded in fragment arrangement (tmem_ld_16x256), in which a thread meets only MT / 4
    // tokens: with one weight row per thread (32x32b loads) every thread needs every token's scale, and the 64 KB of
    // broadcast scale reads per k-block of 128 tokens kept the shared memory busier than the loads and the MMAs.
    // (16x256b loads are slower, 125 against 74 cycles per k-block of 128 x 128, and still far from the bound.)
    // Every TMEM stage is free, which waits for no other kernel: after the wait below it held the first MMA up (512 x 256 at one to
    // nine rows 0.04 us of 2.6 to 4)
    for (uint32_t i = 0; i < C::kAcc; ++i) ptx::mbar_arrive_if(full0 + i * 8, leader);
    if constexpr (!GROUPED) ptx::grid_dep_wait();  // the kernel before this one may still read `out` / `partial`
    constexpr int G = MT / 8;  // groups of eight tokens
    const int q = warp & 3;
    const int sub = NSUB == 1 ? 0 : (warp - 4) >> 2;  // which sub-tile of the item this warp promotes
    const int tr = lane >> 2, tc = 2 * (lane & 3);    // this thread's row inside 8 weight rows / column inside 8 tokens
    uint8_t* patch = reinterpret_cast<uint8_t*>(smem) + C::kPatchOffset + (size_t)(warp - 4) * kPatchBytes;
    const uint32_t sc_row = ptx::smem_u32(scale_ring + sub * MT + tc), tlane = tmem_base + ((uint32_t)(q * 32) << 16);
    // The next k-block's place in the rings, as offsets that are added to: `done` barrier, the `full` barrier kAcc k-blocks on, TMEM
    // columns, scales.
    uint32_t done_at = 0, phase = 0, full_at = C::kAcc % C::kStages * 8, column = sub * MT, slot = 0;
    bool ready = false;  // the next k-block's sums are known to be there
    [[maybe_unused]] bool met = false;  // this warp has passed the cluster's first barrier
    int32_t e_last = 0;
    float2 acc[2][G][2];  // [lanes 0-15 / 16-31][token group][rows tr / tr + 8]: two neighbouring tokens
    for (int32_t t = blockIdx.x; t < total; t += gridDim.x) {
      const Item it = get_item<C::kTile, GROUPED, CLUSTER>(p, expert, item_start, t, e_last);
      const int32_t kb0 = it.kb0, kb1 = it.kb1;
      const int32_t row0 = it.row0 + sub * MT, rows = max(0, min(MT, it.rows - sub * MT));
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int g = 0; g < G; ++g) acc[h][g][0] = acc[h][g][1] = make_float2(0.f, 0.f);
      bool ok = true;
#pragma unroll 4
      for (int32_t kb = kb0; kb < kb1; ++kb) {
        if (!ready && !ptx::mbar_wait_inl_a(done0 + done_at, phase)) {
          timeout(ctl, 14);
          ok = false;
          break;
        }
        // The scales come from another warp's ordinary stores, released through `full`; the commit on `done` says nothing of them, nor,
        // to the warp that writes the slot again, of these reads.  `full` of a k-block is complete when `done` is (the MMAs were issued
        // after) and cannot go on before this warp has read the sums, nor before the scales of the stage's next k-block are there.  So
        // the answer needs no look: it is asked for its acquire, and nothing waits for it (0 to 1.6 % of a call).
        (void)ptx::mbar_test_wait_a(full0 + done_at, phase);
        ptx::tc_fence_after();
        const uint32_t taddr = tlane + column;
        const bool mine = NSUB == 1 || rows > 0;  // uniform over the warp
        uint32_t v[2 * 4 * G];
        float2 s[G];
        // The loads and the wait for them stand in one block: with a wait in a block of its own, behind the same condition, the
        // registers pass the point where the two join before they have been filled, where nothing keeps the compiler from copying them.
        if (mine) {
          tmem_ld_16x256<G>(taddr, v);
          tmem_ld_16x256<G>(taddr + (16u << 16), v + 4 * G);
#pragma unroll
          for (int g = 0; g < G; ++g) s[g] = ptx::ld_shared_f32x2(sc_row + slot + 32 * g);
          tmem_ld_fence<8 * G>(v);
        }
        column = column >= (C::kAcc - 1) * C::kTile ? sub * MT : column + C::kTile;
        phase ^= done_at == (C::kStages - 1) * 8;
        done_at = done_at == (C::kStages - 1) * 8 ? 0 : done_at + 8;
        slot = slot == (C::kScaleSlots - 1) * C::kSlotBytes ? 0 : slot + C::kSlotBytes;
        // this TMEM stage and these scales have been read: the k-block kAcc further on may have the stage
        ptx::tc_fence_before();
        __syncwarp();
        ptx::mbar_arrive_if(full0 + full_at, leader);
        full_at = full_at == (C::kStages - 1) * 8 ? 0 : full_at + 8;
        ready = ptx::mbar_test_wait_a(done0 + done_at, phase);  // answered while the sums are added
        if (mine) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const int i = (h * G + g) * 4 + 2 * r;
                acc[h][g][r] = __ffma2_rn(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), s[g], acc[h][g][r]);
              }
        }
      }
      if (!ok || ctl->abort_flag) break;
      const int32_t n_warp = it.nt * BN + q * 32;  // first of the warp's 32 output columns
      if constexpr (CLUSTER) {
        // One tile per cluster, K cut into as many ranges.  Every CTA leaves its sums, fragment order, in its own shared memory (the
        // ring of stages: all of its loads and MMAs are done), and adds up and stores its share of the tile.
        constexpr int kWarps = 4 * NSUB;
        static_assert((size_t)kWarps * 2 * G * 32 * sizeof(float4) <= (size_t)C::kStages * C::kStageBytes, "sums of a tile");
        float4* mine = reinterpret_cast<float4*>(smem) + (size_t)(warp - 4) * 2 * G * 32 + lane;
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (8 * g < rows) mine[(2 * g + h) * 32] = make_float4(acc[h][g][0].x, acc[h][g][0].y, acc[h][g][1].x, acc[h][g][1].y);
        met = true;
        ptx::cluster_arrive_release();
        ptx::cluster_wait_acquire();
        const uint32_t local = ptx::smem_u32(mine);
        switch (p.cluster) {
          case 2: add_up_share<2>(p, local, patch, it.split, row0, rows, n_warp, lane); break;
          case 4: add_up_share<4>(p, local, patch, it.split, row0, rows, n_warp, lane); break;
          default: add_up_share<8>(p, local, patch, it.split, row0, rows, n_warp, lane); break;
        }
        continue;
      }
      if (p.partial != nullptr) {
        float* dst = p.partial + ((int64_t)it.split * p.M + row0) * p.N + n_warp;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int32_t c = h * 16 + r * 8 + tr;
            if (n_warp + c < p.N) {
#pragma unroll
              for (int g = 0; g < G; ++g) {
                const int32_t tok = 8 * g + tc;
                if (tok < rows) dst[(int64_t)tok * p.N + c] = acc[h][g][r].x;
                if (tok + 1 < rows) dst[(int64_t)(tok + 1) * p.N + c] = acc[h][g][r].y;
              }
            }
          }
      } else {
        // 16 tokens per pass through the warp's patch: transposed there by stmatrix, read back as 64 bytes of a token's row
        const uint32_t st_addr = ptx::smem_u32(patch) + (uint32_t)(lane & 7) * kPatchRow + (uint32_t)(lane >> 3) * 16;
        char* out = static_cast<char*>(p.out) + ((int64_t)row0 * p.ldc + n_warp) * 2;
        auto store = [&](auto with_bias) {
          const char* bias = static_cast<const char*>(p.bias);
#pragma unroll
          for (int g = 0; g < G; g += 2) {
            if (8 * g >= rows) break;
            __syncwarp();  // the previous pass has been read out
#pragma unroll
            for (int i = 0; i < 2; ++i)
              stmatrix_x4_trans(st_addr + i * 8 * kPatchRow, pack16(acc[0][g + i][0].x, acc[0][g + i][0].y, p.out_dtype),
                                pack16(acc[0][g + i][1].x, acc[0][g + i][1].y, p.out_dtype),
                                pack16(acc[1][g + i][0].x, acc[1][g + i][0].y, p.out_dtype),
                                pack16(acc[1][g + i][1].x, acc[1][g + i][1].y, p.out_dtype));
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int32_t tl = i * 8 + (lane >> 2), tok = 8 * g + tl, c = (lane & 3) * 8;
              uint4 val = *reinterpret_cast<const uint4*>(patch + tl * kPatchRow + c * 2);
              if (tok < rows && n_warp + c < p.N) {  // N % 8 == 0
                if constexpr (decltype(with_bias)::value)
                  val = ptx::add_bias8(val, __ldg(reinterpret_cast<const uint4*>(bias + (int64_t)(n_warp + c) * 2)), p.out_dtype);
                *reinterpret_cast<uint4*>(out + ((int64_t)tok * p.ldc + c) * 2) = val;
              }
            }
          }
        };
        if constexpr (GROUPED) {
          store(std::false_type{});
        } else {
          if (p.bias == nullptr) store(std::false_type{});
          else store(std::true_type{});
        }
      }
    }
    if constexpr (CLUSTER) {
      if (!met) {  // after a time-out: the other CTAs of the cluster still wait for this warp
        ptx::cluster_arrive_release();
        ptx::cluster_wait_acquire();
      }
    }
  } else {
    if constexpr (NSUB == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kAuxRegs));
    if (warp == 0) {
      // ===== TMA producer.  Pass 0 runs before griddepcontrol.wait: the weight tiles of the first k-blocks (at most one
      // ring of stages, whose barriers are fresh) are requested; pass 1 adds their activation tiles and then continues
      // with whole stages.  Above 128 rows (two chunks) nothing is requested early: a caller may have those weights written by a
      // kernel that releases its dependents before it has ended.
      const uint32_t early = CLUSTER && p.chunks > 1 ? 0 : C::kStages;
      uint32_t pre = 0;
      uint32_t armed = 0, armed_phase = 0;  // bit i: stage i was armed / the phase bit of its last arming
      for (int pass = GROUPED ? 1 : 0; pass < 2; ++pass) {
        uint32_t stage = 0, phase = 0, idx = 0;
        int32_t e_last = 0;
        bool ok = true;
        for (int32_t t = blockIdx.x; t < total && ok; t += gridDim.x) {
          const Item it = get_item<C::kTile, GROUPED, CLUSTER>(p, expert, item_start, t, e_last);
          const int32_t nt = it.nt;
          for (int32_t kb = it.kb0; kb < it.kb1; ++kb, ++idx) {
            const uint32_t dst = stage0 + stage * C::kStageBytes;
            if (pass == 0) {
              if (idx >= early) { ok = false; break; }
              if (leader) {
                ptx::mbar_arrive_expect_tx_a(full0 + stage * 8, QUANT ? kWBytes : C::kStageBytes);
                ptx::tma_load_3d_a(dst, &map_w, full0 + stage * 8, kb * BK, nt * BN, 0);
              }
              armed |= 1u << stage;
              armed_phase = (armed_phase & ~(1u << stage)) | (phase << stage);
              pre = idx + 1;
            } else if (idx < pre) {
              if constexpr (!QUANT)
                if (leader) ptx::tma_load_2d_a(dst + kWBytes, &map_a, full0 + stage * 8, kb * BK, it.row0);
            } else {
              if (!ptx::mbar_wait_inl_a(done0 + stage * 8, phase ^ 1)) {
                timeout(ctl, 11);
                ok = false;
                break;
              }
              if (leader) {
                ptx::mbar_arrive_expect_tx_a(full0 + stage * 8, QUANT ? kWBytes : C::kStageBytes);
                ptx::tma_load_3d_a(dst, &map_w, full0 + stage * 8, kb * BK, nt * BN, it.e);
                if constexpr (!QUANT) ptx::tma_load_2d_a(dst + kWBytes, &map_a, full0 + stage * 8, kb * BK, it.row0);
              }
              armed |= 1u << stage;
              armed_phase = (armed_phase & ~(1u << stage)) | (phase << stage);
            }
            if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          }
          if (ctl->abort_flag) ok = false;
        }
        if (pass == 0) {
          ptx::grid_dep_wait();  // the activations are written by the kernel before this one
        } else if (ctl->abort_flag) {
          // bulk copies must not be in flight when the CTA exits: wait for every stage that may still be armed (20 ms, in which the
          // copies land; the stage's other arrivals may never come)
          for (int i = 0; i < C::kStages; ++i)
            if (armed & (1u << i)) ptx::mbar_wait_inl_a(full0 + i * 8, (armed_phase >> i) & 1u, 20000000ull);
        } else {
          // the last tcgen05.commit arrivals on `done` must have landed before the CTA's shared memory is reused
          for (int i = 0; i < C::kStages; ++i) {
            if (!ptx::mbar_wait_inl_a(done0 + stage * 8, phase ^ 1)) { timeout(ctl, 15); break; }
            if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          }
        }
      }
    } else if (warp == 1) {
      // ===== MMA issuer: D[128 weight rows][tokens] (+)= W_tile * A_tile^T, one TMEM stage per k-block; the instruction is
      // as wide as the item's rows (in steps of 16), so a ragged chunk costs neither time nor power for its padding
      const uint64_t desc0 = ptx::make_kmajor_sw128_desc(stage0);
      uint32_t stage = 0, phase = 0, acc = 0;
      int32_t e_last = 0;
      for (int32_t t = blockIdx.x; t < total; t += gridDim.x) {
        const Item it = get_item<C::kTile, GROUPED, CLUSTER>(p, expert, item_start, t, e_last);
        const int32_t kb0 = it.kb0, kb1 = it.kb1;
        const uint32_t idesc = ptx::make_idesc_e4m3_f32(BN, (uint32_t)(it.rows + 15) / 16 * 16);
        bool ok = true;
        for (int32_t kb = kb0; kb < kb1; ++kb) {
          if (!ptx::mbar_wait_inl_a(full0 + stage * 8, phase)) { timeout(ctl, 13); ok = false; break; }
          ptx::tc_fence_after();
          const uint64_t w_desc = desc0 + (uint64_t)(stage * (C::kStageBytes >> 4));
          ptx::mma_f8f6f4_x4_if(tmem_base + acc * C::kTile, w_desc, w_desc + (kWBytes >> 4), idesc, leader);
          ptx::mma_commit_if(done0 + stage * 8, leader);
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          if (++acc == C::kAcc) acc = 0;
        }
        if (!ok || ctl->abort_flag) break;
      }
    } else if constexpr (QUANT) {
      // ===== quantisers (warps 2, 3 and 8 to 15)
      ptx::grid_dep_wait();  // the rows come from the kernel before this one
      const uint32_t me = warp < 4 ? warp - 2 : warp - 6;
      if (p.out_dtype == SGLB200_BF16) quantise_rows<__nv_bfloat16, UE, CLUSTER>(p, ctl, smem, scale_ring, me, lane, total);
      else quantise_rows<__half, UE, CLUSTER>(p, ctl, smem, scale_ring, me, lane, total);
    } else if (warp == 2 || (GROUPED && p.k_tiles < C::kStages)) {
      // ===== scale loader: per group of four k-blocks the products sa[token, kb] * sb[nt, kb], 0 for tokens past the item's
      // rows (the accumulator columns there hold leftovers and are not stored).  The loads of the next group, the next item's
      // too, are in flight while this group waits for its place in the ring.  Grouped items of fewer k-blocks than the ring has
      // stages (quantise_rows says why not more) come to warps 2 and 3 in turn: a short item is mostly these loads' way to
      // memory and back.  One loader, which looked for its item and its rows in global memory before each fetch -> this, expert layer
      // of 256 x (7168, 256), eight a token, at 4 / 16 / 64 / 128 / 512 tokens: 67 / 146 / 272 / 306 / 347 us -> 62 / 123 / 224 / 252 / 292
      // Exponent words are decoded where the products are formed.  Decoded at the load they had to arrive before the group ahead of them
      // was handed over, a way to memory and back in every call and, at K = 2560, 7 % of it: UE8M0, 24 / 64 x 5120 x 2560 7.5 / 8.85 ->
      // 7.05 / 8.4 us, 32 x 1000 x 1024 5.9 -> 5.6, 24 x 576 x 7168 6.8 -> 6.5, 48 x 10240 x 8192 21.6 -> 20.7, 48 x 36864 x 7168 level.
      if constexpr (!GROUPED) ptx::grid_dep_wait();  // the activation scales come from the kernel before this one
      constexpr int kPerLane = C::kTile / 32 > 0 ? C::kTile / 32 : 1;
      const uint32_t loaders = GROUPED && p.k_tiles < C::kStages ? 2 : 1, skip = loaders == 2 ? p.k_tiles : 0;
      uint32_t stage = 0, phase = 0, slot = 0;
      auto pass_over = [&](uint32_t n) {  // n k-blocks, fewer than the ring has stages
        stage += n;
        if (stage >= (uint32_t)C::kStages) { stage -= C::kStages; phase ^= 1; }
        slot += n;
        if (slot >= (uint32_t)C::kScaleSlots) slot -= C::kScaleSlots;
      };
      if (warp == 3) pass_over(skip);
      int32_t e_last = 0, t = blockIdx.x + (warp - 2) * gridDim.x;
      const int32_t step = loaders * gridDim.x;
      float a[kPerLane][kScaleGroup], b[kScaleGroup];
      const float *sb_blk = nullptr, *sa_base = nullptr;
      int32_t rows = 0, kb = 0, kb1 = 0;  // of the group to be fetched
      auto next_item = [&] {
        const Item it = get_item<C::kTile, GROUPED, CLUSTER>(p, expert, item_start, t, e_last);
        sb_blk = p.sb + (int64_t)it.nt * p.sb_stride_n;
        sa_base = p.sa + (int64_t)it.row0 * p.sa_stride_m;
        if constexpr (GROUPED) {
          sb_blk += (int64_t)it.e * p.sb_stride_e;
          if (p.rows_per_expert > 0)
            sa_base = p.sa + (int64_t)it.e * p.sa_stride_e + (int64_t)(it.row0 - it.e * p.rows_per_expert) * p.sa_stride_m;
        }
        rows = it.rows;
        kb = it.kb0;
        kb1 = it.kb1;
      };
      auto fetch = [&] {
#pragma unroll
        for (int u = 0; u < kScaleGroup; ++u) {
          const int32_t k = min(kb + u, kb1 - 1);
          b[u] = load_scale_bits<UE>(sb_blk, k, p.sb_stride_k);
#pragma unroll
          for (int h = 0; h < kPerLane; ++h) {
            const int32_t tok = lane + 32 * h;
            a[h][u] = tok < rows ? load_scale_bits<UE>(sa_base + (int64_t)tok * p.sa_stride_m, k, p.sa_stride_k) : 0.f;
          }
        }
      };
      bool ok = true;
      if (t < total) {
        next_item();
        fetch();
      }
      while (t < total && ok) {
        float v[kPerLane][kScaleGroup];
#pragma unroll
        for (int h = 0; h < kPerLane; ++h)
#pragma unroll
          for (int u = 0; u < kScaleGroup; ++u) v[h][u] = scale_of<UE>(a[h][u], kb + u) * scale_of<UE>(b[u], kb + u);
        const int32_t n = min(kScaleGroup, kb1 - kb);
        kb += kScaleGroup;
        const bool last = kb >= kb1;
        if (last) {
          t += step;
          if (t < total) next_item();
        }
        if (t < total) fetch();
#pragma unroll
        for (int u = 0; u < kScaleGroup; ++u) {
          if (u >= n) break;
          if (!ptx::mbar_wait_inl_a(done0 + stage * 8, phase ^ 1)) { timeout(ctl, 16); ok = false; break; }
          (void)ptx::mbar_test_wait_a(full0 + stage * 8, phase ^ 1);  // the promotion warps have read this slot: see there
#pragma unroll
          for (int h = 0; h < kPerLane; ++h)
            if (C::kTile >= 32 || lane < C::kTile) scale_ring[slot * C::kTile + lane + 32 * h] = v[h][u];
          __syncwarp();
          ptx::mbar_arrive_if(full0 + stage * 8, leader);
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          if (++slot == C::kScaleSlots) slot = 0;
        }
        if (last) pass_over(skip);
        if (ctl->abort_flag) break;
      }
    }
    if constexpr (CLUSTER) {  // the barrier at which the promotion warps meet those of the other CTAs counts every thread
      ptx::cluster_arrive_release();
      ptx::cluster_wait_acquire();
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if constexpr (CLUSTER) {  // no CTA leaves, and no shared memory goes, before all have read the sums
    ptx::cluster_arrive_release();
    ptx::cluster_wait_acquire();
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int MT, bool UE, bool GROUPED, int NSUB = 1, bool CLUSTER = false, bool QUANT = false>
int launch(const CUtensorMap& map_w, const CUtensorMap& map_a, const SmallParams& p, int sm_count, cudaStream_t st,
           int64_t max_items, int cluster = 1) {
  using C = Cfg<MT, NSUB>;
  // the tables as long as there are experts: what is left of an SM's memory is its L1, which holds the scales' sectors
  const size_t smem = GROUPED ? C::smem_grouped((size_t)p.num_experts) : C::kSmem;
  constexpr int kThreads = QUANT ? 192 + 32 * kQuantWarps : Cfg<MT, NSUB>::kThreads;
  static bool done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(fp8_block_gemm_smallm_kernel<MT, UE, GROUPED, NSUB, CLUSTER, QUANT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(GROUPED ? C::smem_grouped(kMaxExperts) : smem));
    if (e != cudaSuccess) return fail(SGLB200_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (NSUB == 2) {
      // setmaxnreg.inc draws on the registers the block was launched with and waits for good if they do not suffice: a
      // build whose register count is too low for the split must not be launched
      cudaFuncAttributes fa;
      e = cudaFuncGetAttributes(&fa, fp8_block_gemm_smallm_kernel<MT, UE, GROUPED, NSUB, CLUSTER, QUANT>);
      if (e != cudaSuccess || fa.numRegs * kThreads < 128 * kAuxRegs + 256 * kPromoRegs)
        return fail(SGLB200_ERR_LAUNCH, "fp8_block_gemm_smallm_kernel: %d registers a thread are too few for its register split",
                    e == cudaSuccess ? fa.numRegs : 0);
    }
    done[dev] = true;
  }
  const int grid = (int)(max_items < sm_count ? max_items : sm_count);
  const cudaError_t le = launch_pdl_cluster(fp8_block_gemm_smallm_kernel<MT, UE, GROUPED, NSUB, CLUSTER, QUANT>, dim3(grid), dim3(kThreads), smem, st,
                                            cluster, map_w, map_a, p);
  if (le != cudaSuccess) {
    cudaGetLastError();
    return fail(SGLB200_ERR_LAUNCH, "fp8_block_gemm_smallm_kernel: %s", cudaGetErrorString(le));
  }
  note_gemm("fp8_block_gemm_smallm_kernel");
  return SGLB200_OK;
}

// one tile per cluster, as many clusters as tiles
template <bool UE>
int launch_cluster(int MT, bool two, const CUtensorMap& map_w, const CUtensorMap& map_a, const SmallParams& p, cudaStream_t st,
                   int64_t items) {
  const int grid = (int)items, c = p.cluster;
  if (two) return launch<64, UE, false, 2, true>(map_w, map_a, p, grid, st, items, c);
  switch (MT) {
    case 16: return launch<16, UE, false, 1, true>(map_w, map_a, p, grid, st, items, c);
    case 32: return launch<32, UE, false, 1, true>(map_w, map_a, p, grid, st, items, c);
    default: return launch<32, UE, false, 2, true>(map_w, map_a, p, grid, st, items, c);  // two sets: 64 x 7168 x 16384 24.9 -> 24.6 us, 40 x 2112 x 7168 9.4 -> 8.9
  }
}

// rows that the GEMM itself quantises
int launch_quant(const CUtensorMap& map_w, const SmallParams& p, bool ue8m0, int sm_count, cudaStream_t st, int64_t items) {
  if (p.cluster > 1)
    return ue8m0 ? launch<16, true, false, 1, true, true>(map_w, map_w, p, (int)items, st, items, p.cluster)
                 : launch<16, false, false, 1, true, true>(map_w, map_w, p, (int)items, st, items, p.cluster);
  return ue8m0 ? launch<16, true, false, 1, false, true>(map_w, map_w, p, sm_count, st, items)
               : launch<16, false, false, 1, false, true>(map_w, map_w, p, sm_count, st, items);
}

}  // namespace

// Row limit of this kernel, and of the scratch sizes that callers know (smallm_splits)
int smallm_max_rows() { return 128; }
constexpr int kMaxChunkedRows = 256;  // two chunks, fp32 scales: see takes_few_rows

int smallm_quant_rows() { return kQuantRows; }

// Whether the GEMM quantises M rows itself rather than after the quantiser kernel: up to eight (see quantise_rows), and where no CTA has
// more than two tiles, each with all of its k-blocks to convert again: 4 / 8 x 57344 x 8192 among other kernels 99.5 / 100.5 -> 101.3 /
// 102.1 us, 36864 x 7168 (two tiles) 67.5 / 67.6 -> 67.0 / 67.4.  One and two rows have no scratch for the kernel.
bool smallm_quantises(int64_t M, int64_t N, int sm_count) {
  return M <= kQuantRows || (M <= kMaxQuantRows && (N + BN - 1) / BN <= 2 * (int64_t)sm_count);
}

// From 65 rows up a k-block takes this kernel 390 ns where clusters share K, 360 alone, and the 128 x 128 kernel 250: where every CTA works alone,
// that one takes the call (GEMM alone in a replayed graph, this / the tile kernel, us: 113 x 10240 x 8192 27.5/20.3, 65 x 36864 x 7168
// 48.6/46.6, 128 x 57344 x 8192 108/94, 128 x 24576 x 1536 16.9/12.3), and so it does where the cost model has a cluster behind it.  Up to 128
// rows, where no cluster shares K, both add k-blocks in the same order, so that the bits are the few-rows kernel's either way.
// From 129 to 256 rows (fp32 scales) clusters work on two even chunks, as long as all of them fit the chip at once, where the tile kernel, which
// would cut K through memory and add the sums up in a kernel of its own, is expected to be slower.  Calls, tile kernel / this, us, 129 / 192 / 256 rows:
// 576 x 7168 14.0 / 14.0 / 14.2 -> 10.2 / 11.0 / 12.3, 1536 x 7168 16.1 / 16.1 / 16.4 -> 16.1 (not taken) / 14.4 / 14.9; three and more chunks
// are level.  UE8M0 calls there keep the block-scaled kernels, whose sums the entry with a workspace shares.
bool takes_few_rows(int64_t M, int64_t N, int64_t K, int sm_count, bool ue8m0) {
  return M <= 64 || smallm_cluster(M, N, K, sm_count, ue8m0) > 1;
}

// CTAs per cluster that share one tile's K (1, 2, 4 or 8) for a dense problem.  Cost model in nanoseconds: a k-block takes one CTA
// `step` (the MMA issuer at 16 columns, the promotion above), or longer once the CTAs together ask for more than HBM delivers (16 KB
// of weights each at 6.5 TB/s); adding up over the cluster costs a barrier and a round trip or two (add_up_share).  From 65 rows a CTA
// that works alone is the tile kernel's (takes_few_rows).  Fitted to calls of thirteen layers, K = 512 to 16384, at every cluster
// size, 2 to 128 rows; the choice is the best one or within 3 % of it, where the constants of rank 0 adding up alone were up to 19 % off: 24 x
// 3072 x 1536 6.6 -> 6.0 us, 32 x 7168 x 2048 7.85 -> 7.3, 16 x 6144 x 1536 6.3 -> 5.8, 128 x 6144 x 1536 10.2 -> 8.5, 128 x 7168 x 2048 11.3 ->
// 9.8, 128 x 9216 x 4096 16.2 -> 14.1, 128 x 1000 x 1024 (UE8M0) 9.4 -> 7.7.  Larger clusters leave SMs of a GPC unused.
int smallm_cluster(int64_t M, int64_t N, int64_t K, int sm_count, bool ue8m0) {
  const int64_t k_tiles = (K + BK - 1) / BK, chunks = M <= smallm_max_rows() ? 1 : (M + 127) / 128;
  const int64_t n_tiles = (N + BN - 1) / BN * chunks;
  if (M > kMaxChunkedRows || (ue8m0 && chunks > 1) || (M > 64 && n_tiles > sm_count)) return 1;
  const int64_t step = M <= 16 ? 195 : (M <= 32 ? 215 : (M <= 64 ? 240 : 390));
  const int64_t base = M <= 16 ? 800 : (M <= 64 ? 1000 : 2400);
  const int64_t rank = M <= 16 ? 60 : (M <= 32 ? 100 : (M <= 64 ? 130 : 150));
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int c = 1; c <= kMaxCluster; c *= 2) {
    if (c > 1 && k_tiles < 2 * c) break;
    const int64_t kb = (k_tiles + c - 1) / c;
    if ((k_tiles + kb - 1) / kb != c) continue;  // every CTA of the cluster must get k-blocks
    // CTAs resident at once, about; a cluster takes one tile, so more tiles than fit are left to CTAs that walk the list
    const int64_t ctas = n_tiles * c, fit = c <= 2 ? sm_count : sm_count - 4 * c;
    if (c > 1 && ctas > fit) break;
    const int64_t waves = (ctas + fit - 1) / fit, hbm = (ctas < fit ? ctas : fit) * 16384 * 10 / 65000;
    int64_t cost = waves * kb * (step > hbm ? step : hbm);
    if (c == 1 && M > 64) cost = waves * (ue8m0 ? kb * 340 + 1700 : kb * 250 + 500);
    if (c == 1 && chunks > 1) cost = tile_cost(M, N, K, sm_count);
    if (c > 1) cost += base + (int64_t)(c - 1) * rank;
    if (cost < best_cost) {
      best_cost = cost;
      best = c;
    }
  }
  return best;
}

// K ranges that fp32 partial sums in memory would be cut into, in units of one k-block of one work item: an item costs its
// k-blocks plus 3 (fill, store), the kernel that adds the sums 8.  The kernels here add up on the chip and write no such sums; this is
// what sglb200_fp8_blockwise_scaled_mm_workspace_bytes answers up to smallm_max_rows() and what the built-in buffer's limit is held
// against.  Callers sized buffers by it and know from it which shapes the no-allocation entry takes, so it stays as it is.
int smallm_splits(int64_t N, int64_t K, int sm_count) {
  const int64_t n_tiles = (N + BN - 1) / BN, k_tiles = (K + BK - 1) / BK;
  constexpr int64_t kItemCost = 3, kReduceCost = 8;
  int best = 1;
  int64_t best_cost = ((n_tiles + sm_count - 1) / sm_count) * (k_tiles + kItemCost);
  for (int64_t s = 2; s <= 32 && s * 2 <= k_tiles; ++s) {
    const int64_t kb = (k_tiles + s - 1) / s;
    if ((k_tiles + kb - 1) / kb != s) continue;  // every range must get k-blocks
    const int64_t cost = ((n_tiles * s + sm_count - 1) / sm_count) * (kb + kItemCost) + kReduceCost;
    if (cost < best_cost) {
      best_cost = cost;
      best = (int)s;
    }
  }
  return best;
}

// Launches the small-M kernel (arguments already validated by the caller).  `partial` != NULL: the fp32 sums [splits][M][N]
// go there, *splits_used of them, and the caller converts and moves them itself.
// With ue8m0 the scale pointers are packed exponent words (sa: word (m, kg) at m * sa_stride_m + kg * sa_stride_k; sb
// likewise per 128 weight rows) and the scales are the exact powers of two they encode.
int smallm_gemm(const void* a, const void* b, const float* sa, const float* sb, void* out, int64_t M, int64_t N, int64_t K,
                int64_t lda, int64_t ldb, int64_t ldc, int64_t sa_stride_m, int64_t sa_stride_k, int64_t sb_stride_n,
                int64_t sb_stride_k, int out_dtype, const void* bias, float* partial, int64_t partial_floats, int sm_count,
                void* stream, int* splits_used, bool ue8m0, const RawRows* raw) {
  const int MT = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
  const bool two = M > 64;  // up to 128 activation rows per work item, several sets of promotion warps
  alignas(64) CUtensorMap map_w, map_a;
  {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, 1};
    const uint64_t str[2] = {(uint64_t)ldb, (uint64_t)ldb * (uint64_t)N};
    if (int rc = make_map_sw128(&map_w, b, 3, dims, str, BN, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) return rc;
  }
  if (raw == nullptr) {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t str[1] = {(uint64_t)lda};
    if (int rc = make_map_sw128(&map_a, a, 2, dims, str, (uint32_t)(M > 64 ? 128 : MT), CU_TENSOR_MAP_L2_PROMOTION_L2_128B))
      return rc;
  }
  SmallParams p = {};
  p.sa = sa;
  p.sb = sb;
  p.out = out;
  p.bias = bias;
  p.M = (int32_t)M;
  p.N = (int32_t)N;
  p.K = (int32_t)K;
  p.n_tiles = (int32_t)((N + BN - 1) / BN);
  p.k_tiles = (int32_t)((K + BK - 1) / BK);
  p.ldc = ldc;
  p.sa_stride_m = sa_stride_m;
  p.sa_stride_k = sa_stride_k;
  p.sb_stride_n = sb_stride_n;
  p.sb_stride_k = sb_stride_k;
  p.out_dtype = out_dtype;
  p.count_stride = 1;
  p.num_experts = 1;
  p.cluster = 1;
  int splits = 1;
  if (partial != nullptr) {
    p.partial = partial;
    splits = smallm_cluster(M, N, K, sm_count, ue8m0);  // the same ranges, added in the same order: the same bits as `out`
    if ((int64_t)splits * M * N > partial_floats) splits = 1;
  } else {
    splits = p.cluster = smallm_cluster(M, N, K, sm_count, ue8m0);
  }
  p.kb_per_split = (p.k_tiles + splits - 1) / splits;
  p.k_splits = (p.k_tiles + p.kb_per_split - 1) / p.kb_per_split;
  if (splits_used) *splits_used = p.k_splits;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  p.chunks = M <= 128 ? 1 : (int32_t)((M + 127) / 128);
  p.chunk_rows = (int32_t)((M + p.chunks - 1) / p.chunks);
  p.chunks = (int32_t)((M + p.chunk_rows - 1) / p.chunk_rows);
  const int64_t items = (int64_t)p.n_tiles * p.chunks * p.k_splits;
  if (raw != nullptr) {
    p.x = a;
    p.eps = raw->eps;
    return launch_quant(map_w, p, ue8m0, sm_count, st, items);
  }
  if (p.cluster > 1)
    return ue8m0 ? launch_cluster<true>(MT, two, map_w, map_a, p, st, items) : launch_cluster<false>(MT, two, map_w, map_a, p, st, items);
  if (M > smallm_max_rows()) return fail(SGLB200_ERR_SHAPE, "%lld rows: at most %d unless K is shared", (long long)M, smallm_max_rows());
  if (two) {
    if (ue8m0) return fail(SGLB200_ERR_SHAPE, "UE8M0 scales: at most 64 rows unless K is shared, not %lld", (long long)M);
    return launch<32, false, false, 4>(map_w, map_a, p, sm_count, st, items);
  }
  if (ue8m0) {
    switch (MT) {
      case 16: return launch<16, true, false>(map_w, map_a, p, sm_count, st, items);
      case 32: return launch<32, true, false>(map_w, map_a, p, sm_count, st, items);
      default: return launch<64, true, false>(map_w, map_a, p, sm_count, st, items);
    }
  }
  switch (MT) {
    case 16: return launch<16, false, false>(map_w, map_a, p, sm_count, st, items);
    case 32: return launch<32, false, false>(map_w, map_a, p, sm_count, st, items);
    default: return launch<64, false, false>(map_w, map_a, p, sm_count, st, items);
  }
}

// Above this average the 128 x 128 tile kernel is level with or ahead of chunks of up to 128 rows (256 experts, N=7168 K=2048:
// 896 against 920 us at 64 rows, 1327 against 1410 at 128); at 32 rows the chunks win (875 against 689 us).  The UE8M0 tile
// kernel has no promotion to pay for and draws level much earlier (whole layer at 32 rows: 1940 us it, 1990 the chunks).
// With a K of a few k-blocks an item is mostly start and store, of which the UE8M0 tile kernel has less (its epilogue overlaps the
// next tile), once there are enough items for that to outweigh its later start (it is launched without programmatic overlap).
// Measured when the line was drawn, on 11 layers of 8 to 256 experts and 2048 to 7168 columns, K = 128 to 512, 0.5 to 20 rows per
// expert: with up to 1400 items (128 weight rows of an expert that has rows) the chunks took 0.67 to 1.05 of the tile kernel's time
// (64 x 2048 x 256 at 4 rows: 12.3 against 14.4 us), with more 0.95 to 1.48; K = 1024 gave 1.0 to 1.12 there and K = 2048 0.94 to 1.02.
// Since short items look for their scales ahead, with two loaders, the line is behind the kernel: with more than 1400 items the chunks
// take 0.62 to 0.98 of the tile kernel's time up to K = 384 and 24 rows per expert (256 x 7168 x 256 at 1 / 4 / 16 rows: 57 / 82 / 97 against
// 79 / 113 / 117 us), and 0.90 to 1.05 at K = 512.  It stays where it is until it is fitted again.
// The fp32 tile kernel gains nothing from a short K (256 x 7168 x 256 at 4 rows: 151 against 82 us).
constexpr int64_t kWideRowsMax = 48, kWideRowsMaxUe8m0 = 20, kShortKUe8m0 = 512;
constexpr double kShortKItems = 1400.;

// Work items of one chunk per expert that `rows` rows routed evenly at random make.
double routed_items(int64_t rows, int64_t num_experts, int64_t N) {
  return -std::expm1(-(double)rows / (double)num_experts) * (double)num_experts * (double)((N + BN - 1) / BN);
}

// Rows per chunk of the grouped few-rows kernel for `total_rows` rows spread over `num_experts` experts (or
// rows_per_expert rows at most per expert in the masked layout); 0 = the 128 x 128 grouped kernel is the better choice.
int smallm_grouped_chunk(int64_t total_rows, int64_t num_experts, int64_t rows_per_expert, int64_t expected_rows, int64_t N, int64_t K,
                         bool ue8m0) {
  const int setting = g_grouped_few_rows_max, limit = setting & ~SGLB200_FEW_ROWS_EXACT;
  if (limit == 0) return 0;
  int64_t avg = (total_rows + num_experts - 1) / num_experts;
  if (rows_per_expert > 0) {  // masked layout: the row bound is known, the rows in use only if the caller expects a number
    if (expected_rows <= 0 || expected_rows > rows_per_expert) {
      if (rows_per_expert > limit) return 0;
      return rows_per_expert <= 16 ? 16 : (rows_per_expert <= 32 ? 32 : 64);
    }
    avg = expected_rows;
  }
  // the setter's default stands for the rule above; a caller who sets another limit gets exactly that
  const bool short_k = ue8m0 && K <= kShortKUe8m0 && routed_items(total_rows, num_experts, N) > kShortKItems;
  const int64_t rule = !ue8m0 ? kWideRowsMax : (short_k ? 0 : kWideRowsMaxUe8m0);
  if (avg > (setting == kGroupedFewRowsDefault ? rule : limit)) return 0;
  return avg <= 8 ? 16 : (avg <= 24 ? 32 : 64);
}

// Grouped few-rows GEMM (arguments already validated by the caller): chunk = smallm_grouped_chunk(...) != 0.
int smallm_grouped_gemm(int chunk, const void* a, const void* b, const float* sa, const float* sb, void* out,
                        const int32_t* expert_offsets, const int32_t* problem_sizes, int count_stride, int64_t total_rows,
                        int64_t num_experts, int64_t rows_per_expert, int64_t N, int64_t K, int64_t lda, int64_t ldb,
                        int64_t ldb_e, int64_t ldc, int64_t sa_stride_e, int64_t sa_stride_m, int64_t sa_stride_k,
                        int64_t sb_stride_e, int64_t sb_stride_n, int64_t sb_stride_k, int out_dtype, int sm_count,
                        void* stream, bool ue8m0) {
  if (num_experts > kMaxExperts) return fail(SGLB200_ERR_SHAPE, "num_experts=%lld: at most %d", (long long)num_experts, kMaxExperts);
  alignas(64) CUtensorMap map_w, map_a;
  {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, (uint64_t)num_experts};
    const uint64_t str[2] = {(uint64_t)ldb, (uint64_t)ldb_e};
    if (int rc = make_map_sw128(&map_w, b, 3, dims, str, BN, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) return rc;
  }
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)total_rows};
    const uint64_t str[1] = {(uint64_t)lda};
    if (int rc = make_map_sw128(&map_a, a, 2, dims, str, (uint32_t)chunk, CU_TENSOR_MAP_L2_PROMOTION_L2_128B)) return rc;
  }
  SmallParams p = {};
  p.sa = sa;
  p.sb = sb;
  p.out = out;
  p.M = (int32_t)total_rows;
  p.N = (int32_t)N;
  p.K = (int32_t)K;
  p.n_tiles = (int32_t)((N + BN - 1) / BN);
  p.k_tiles = (int32_t)((K + BK - 1) / BK);
  p.k_splits = 1;
  p.kb_per_split = p.k_tiles;
  p.ldc = ldc;
  p.sa_stride_m = sa_stride_m;
  p.sa_stride_k = sa_stride_k;
  p.sb_stride_n = sb_stride_n;
  p.sb_stride_k = sb_stride_k;
  p.out_dtype = out_dtype;
  p.expert_offsets = expert_offsets;
  p.problem_sizes = problem_sizes;
  p.count_stride = count_stride;
  p.rows_per_expert = (int32_t)rows_per_expert;
  p.num_experts = (int32_t)num_experts;
  p.sa_stride_e = sa_stride_e;
  p.sb_stride_e = sb_stride_e;
  // an upper bound on the work items without reading the device: every expert can add one ragged chunk
  const int64_t items = ((total_rows + chunk - 1) / chunk + num_experts) * p.n_tiles;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (ue8m0) {
    switch (chunk) {
      case 16: return launch<16, true, true>(map_w, map_a, p, sm_count, st, items);
      case 32: return launch<32, true, true>(map_w, map_a, p, sm_count, st, items);
      default: return launch<64, true, true>(map_w, map_a, p, sm_count, st, items);
    }
  }
  switch (chunk) {
    case 16: return launch<16, false, true>(map_w, map_a, p, sm_count, st, items);
    case 32: return launch<32, false, true>(map_w, map_a, p, sm_count, st, items);
    default: return launch<64, false, true>(map_w, map_a, p, sm_count, st, items);
  }
}

}  // namespace sglb

// Test hook (not in the public header): the grouped kernel's choice for a call without touching a device.
extern "C" int sglb200_debug_grouped_chunk(int64_t total_rows, int64_t num_experts, int64_t rows_per_expert, int64_t expected_rows,
                                           int64_t N, int64_t K, int ue8m0) {
  return sglb::smallm_grouped_chunk(total_rows, num_experts, rows_per_expert, expected_rows, N, K, ue8m0 != 0);
}
