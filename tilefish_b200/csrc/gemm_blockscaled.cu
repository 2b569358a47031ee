// Block-scaled GEMM for sm_100a: out[M,N] = bf16( sum_k deq(a)[m,k] * deq(b)[n,k] ), f32 accumulation in tensor memory.
//
// One persistent CTA per SM walks output tiles of 128 x BLOCK_N. Three warp roles:
//   warp 0   operand loads: TMA tiled loads of the A and B code tiles (128-byte swizzle) into a ring of shared-memory stages,
//            signalled through mbarriers (complete_tx). ONE instruction per stage: lane 0 loads the A tile, lanes 1-2 the
//            128-row halves of the B tile (issuing a TMA copy costs the issuing thread 40-90 clocks; six copies issued one
//            after another by one thread made that thread, not the memory system, the limit of the whole kernel)
//   warp 6   scale loads: bulk copies of the pre-swizzled scale tiles of the same stage, again one instruction (lane 0 the A
//            scales, lanes 1-2 the B scales); both load warps arrive on the stage's "full" barrier with their own byte counts
//   warp 1   MMA issuer: copies the scale tiles shared -> tensor memory (tcgen05.cp) and issues
//            tcgen05.mma.kind::{mxf8f6f4, mxf4, mxf4nvf4}.block_scale, 4 per stage (32 bytes of K each); tcgen05.commit frees
//            the stage and, after the last one, hands the accumulator to the epilogue
//   warps 2-5 and 7-10   epilogue, two groups of four warps: a warp reads its 32 lanes of the accumulator (tcgen05.ld), the groups
//            share the columns (even / odd 32-column chunks); scale, fused epilogue (none / SiLU gate / residual add), bf16
//            stores. With short K (10-20 stages per tile) one group of four could not drain a tile as fast as the MMAs fill one
// The accumulator is double-buffered in tensor memory (overlapped for 256-column tiles, see TileCfg), so a tile's epilogue
// runs while the next tile's MMAs are issued.
// Further forms, chosen by launch_plan and use_pair_kernel: a pair of CTAs per 256 x 256 tile, K ranges over a cluster of CTAs or over
// planes of a workspace. No TMA multicast. Every mbarrier wait is bounded (about one second): on a timeout the kernel records
// TF_ERR_DEVICE_TIMEOUT in a device status word, every role leaves its loop, tensor memory is freed and the kernel returns.
//
// Scale layout consumed: the 512-byte 128x4 tiles described in the header; one tile feeds 4 tensor-memory columns through
// tcgen05.cp.32x128b.warpx4, byte k of a column being the scale of K-block k (selected by the SF-id field of the instruction
// descriptor for the MX formats; NVFP4 uses all four bytes per MMA).
#include <cuda.h>

#include <atomic>
#include <cstdlib>

#include "ask_once.h"
#include "async_copy.cuh"
#include "quant_core.cuh"

namespace tf {

__device__ int g_device_status[2];  // [0] status, [1] detail

constexpr int kBlockM = 128;
constexpr int kStageKBytes = 128;  // bytes of K per row per stage: one 128-byte swizzle atom
constexpr int kAStageBytes = kBlockM * kStageKBytes;
constexpr int kGemmThreads = 352;  // 11 warps: operand loads, MMA issue, epilogue group 0 (4), scale loads, epilogue group 1 (4)
constexpr int kSmemLimit = 227 * 1024;
constexpr unsigned long long kWaitLimitNs = 1000000000ull;

template <int FMT>
struct FmtTraits;
template <>
struct FmtTraits<TF_FMT_MXFP8> {
  static constexpr int kSfTiles = 1;  // 512-byte scale tiles per operand row-tile per stage
  static constexpr uint32_t kElemFormat = 0, kScaleIsE8 = 1;
};
template <>
struct FmtTraits<TF_FMT_MXFP4> {
  static constexpr int kSfTiles = 2;
  static constexpr uint32_t kElemFormat = 1, kScaleIsE8 = 1;
};
template <>
struct FmtTraits<TF_FMT_NVFP4> {
  static constexpr int kSfTiles = 4;
  static constexpr uint32_t kElemFormat = 1, kScaleIsE8 = 0;
};

template <int FMT, int BLOCK_N>
struct TileCfg {
  static constexpr int kNB = BLOCK_N / 128;  // 128-row halves of the B tile
  static constexpr int kST = FmtTraits<FMT>::kSfTiles;
  static constexpr int kBStageBytes = BLOCK_N * kStageKBytes;
  static constexpr int kSfaStageBytes = kST * 512;
  static constexpr int kSfbStageBytes = kST * 512 * kNB;
  static constexpr int kStageBytes = kAStageBytes + kBStageBytes + kSfaStageBytes + kSfbStageBytes;
  static constexpr int kBarrierBytes = 256;
  static constexpr int kStagesRaw = (kSmemLimit - 1024 - kBarrierBytes) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  static constexpr int kSmemBytes = kStages * kStageBytes + kBarrierBytes + 1024;
  // Tensor memory (512 columns): two accumulators used by alternate tiles, so that the epilogue of one tile runs under the
  // MMAs of the next, then two scale buffers used by alternate stages. Two 256-column accumulators plus 96 scale columns do
  // not fit, so with BLOCK_N = 256 the accumulators OVERLAP: accumulator 1 starts at column 160 and shares columns
  // [160, 256) with accumulator 0. The epilogue first moves the shared columns of its tile into registers, then releases
  // the next tile's MMAs, then drains the rest. With BLOCK_N = 128 the accumulators are disjoint.
  static constexpr int kAccStride = BLOCK_N == 256 ? 160 : BLOCK_N;  // first column of accumulator 1
  static constexpr int kOverlapChunks = BLOCK_N == 256 ? 3 : 0;      // 32-column chunks both accumulators cover
  static constexpr int kTmemSfSet = kST * 4 * (1 + kNB);             // columns of one scale buffer: A scales then B scales
  static constexpr int kTmemSfBase = kAccStride + BLOCK_N;           // 416 or 256
  static constexpr int kTmemSfa = kTmemSfBase;                       // first column of the A scales of buffer 0
  static constexpr int kTmemSfb = kTmemSfBase + kST * 4;             // first column of the B scales of buffer 0
  static constexpr int kTmemUsed = kTmemSfBase + 2 * kTmemSfSet;
  static constexpr int kTmemCols = 512;
  static_assert(kTmemUsed <= 512, "tensor memory budget");
};

struct GemmParams {
  int m, n, n_rows_b, k_bytes;
  int num_k_stages, sf_col_tiles;  // K stages per tile; 512-byte tiles per scale row-tile
  int m_blocks, n_blocks, num_tiles;
  int sfb_row_tiles;
  const uint8_t* sfa;
  const uint8_t* sfb;
  const float* a_gs;
  const float* b_gs;
  uint16_t* out;
  int64_t ldo;
  float* residual;
  unsigned int* out_amax;
  int splits, k_stages_per_split;  // split-K: every (tile, split) accumulates a K range into the f32 workspace
  float* ws;
  uint8_t* q_codes;   // optional MX-quantized copy of the output (same format as the operands), swizzled scales
  uint8_t* q_scales;
  int q_pad;      // the scales have padding that this launch zeroes (by the epilogue warps, while they wait for the first tile)
  int a_gs_rows;  // 0: a has one global scale; else a_gs[row / a_gs_rows] (row blocks quantized separately, e.g. gathered from ranks)
  int a_box_bytes;  // bytes one A load brings per stage: 128 bytes x the rows of its box (fewer than 128 rows when M is small)
  int early_stages;  // K stages of B that a CTA asks into L2 while it waits for the kernel in front (0: none), see prefetch_b_stage
  // Scattered output (tf_gemm_blockscaled_scatter): rows [i * scatter_rows, (i + 1) * scatter_rows) go to scatter_out[i], a
  // [scatter_rows, n] matrix with leading dimension ldo that may live in another GPU's memory (plain stores over NVLink).
  // scatter_rows is a multiple of 128, so a tile has one destination. 0: everything goes to `out`.
  int scatter_rows;
  uint16_t* scatter_out[8];
};

// The address of output row `row`: in `out`, or in the row block's own destination.
__device__ __forceinline__ uint16_t* out_row_ptr(const GemmParams& p, int row) {
  if (p.scatter_rows == 0) return p.out + (int64_t)row * p.ldo;
  const int owner = row / p.scatter_rows;
  uint16_t* base = p.scatter_out[0];
#pragma unroll
  for (int i = 1; i < 8; ++i)
    if (i == owner) base = p.scatter_out[i];
  return base + (int64_t)(row - owner * p.scatter_rows) * p.ldo;
}

// ---- PTX wrappers ----------------------------------------------------------------------------------------------------------
// ---- thread-block-cluster helpers (the 2-CTA kernel) ----
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The shared::cluster address of `addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// The aligned form needs whole warps, which branches in front of it (lanes without data in the cluster's reduction) need not leave converged.
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// tcgen05.commit of a CTA pair: arrives on the barrier at the same offset in both CTAs (a barrier signal, not a data multicast).
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask) : "memory");
}
// TMA load issued by either CTA of a pair: the destination is this CTA's shared memory, the mbarrier may be the peer's
// (cta_group::2 lifts the same-CTA rule). No multicast.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(bar_cluster)
               : "memory");
}
__device__ __forceinline__ void tc_cp_sf_pair(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
template <int FMT>
__device__ __forceinline__ void tc_mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
  if (FMT == TF_FMT_MXFP8) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
  } else if (FMT == TF_FMT_MXFP4) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
  }
}

// Bounded wait. Returns false when the limit ran out here or another role already gave up (abort flag).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int where,
                                          unsigned long long limit_ns = kWaitLimitNs) {
  return mbar_wait_bounded(bar, parity, abort_flag, g_device_status, where, limit_ns);
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map),
               "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// TMA store of a shared-memory box (box row 0 = matrix row y), tracked by this thread's bulk groups.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void sts_128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_cp_sf(uint32_t taddr, uint64_t desc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(desc) : "memory");
}
template <int FMT>
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
  if (FMT == TF_FMT_MXFP8) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
  } else if (FMT == TF_FMT_MXFP4) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
  } else {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%5], [%6], p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
        : "memory");
  }
}
// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets row (lane base + t), v[j] = column (base + j).
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
      "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
        "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
        "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
        "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile stored by TMA with the 128-byte swizzle: rows 128 bytes apart, 8-row
// groups 1024 bytes apart (stride byte offset), descriptor version 1, layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// Descriptor of one 512-byte scale tile for tcgen05.cp.32x128b: 32 rows of 16 bytes, no swizzle, 8-row groups 128 bytes apart.
__device__ __forceinline__ uint64_t desc_sf(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}

__device__ __forceinline__ uint64_t make_desc(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
// True in exactly one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.b32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}


// Self-test of the bounded wait: one thread waits on an mbarrier that nothing arrives at; the wait must give up after limit_ns,
// record TF_ERR_DEVICE_TIMEOUT (detail: wait 9) and return, leaving the context usable.
__global__ void bounded_wait_selftest_kernel(unsigned long long limit_ns) {
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    (void)mbar_wait(smem_u32(&bar), 0, &abort_flag, 9, limit_ns);
  }
}

// ---- epilogue helpers ------------------------------------------------------------------------------------------------------
// Stores 32 consecutive bf16 outputs of one row (packed two per word) and applies the residual / amax side effects.
// The 32 outputs a thread holds are exactly one MX block of its row: amax, scale byte and codes by the quantizer's rules
// (quant_core.cuh), written as the A operand of the next GEMM. FMT is the operands' (and the output's) format.
template <int FMT>
__device__ __forceinline__ void store_chunk_quantized(const GemmParams& p, const uint32_t (&packed)[16], int row, int col) {
  if (FMT == TF_FMT_NVFP4) return;
  const uint32_t k = 0x7FFF7FFFu;
  uint32_t t = 0;
#pragma unroll
  for (int j = 0; j < 16; j += 2) t = __vimax3_u16x2(t, packed[j] & k, packed[j + 1] & k);
  const uint32_t mx = max(t & 0xFFFFu, t >> 16);
  const int emax = (FMT == TF_FMT_MXFP8) ? 8 : 2;
  const int e = (int)(mx >> 7) - emax;
  const uint32_t scale = (mx == 0) ? 127u : (uint32_t)max(e, 0);
  const uint32_t inv1 = (254u - scale) << 7;
  const uint32_t inv2 = inv1 | (inv1 << 16);
  uint32_t q[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) q[j] = mul_bf16x2(packed[j], inv2);
  if (FMT == TF_FMT_MXFP8) {
    uint32_t c[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      c[j] = cvt_e4m3x4(bf16lo_to_f32(q[2 * j]), bf16hi_to_f32(q[2 * j]), bf16lo_to_f32(q[2 * j + 1]), bf16hi_to_f32(q[2 * j + 1]));
    uint4* dst = reinterpret_cast<uint4*>(p.q_codes + (int64_t)row * p.n + col);
    dst[0] = make_uint4(c[0], c[1], c[2], c[3]);
    dst[1] = make_uint4(c[4], c[5], c[6], c[7]);
  } else {
    uint32_t c[4];
#pragma unroll
    for (int h = 0; h < 4; ++h)
      c[h] = cvt_e2m1x8(bf16lo_to_f32(q[4 * h]), bf16hi_to_f32(q[4 * h]), bf16lo_to_f32(q[4 * h + 1]), bf16hi_to_f32(q[4 * h + 1]),
                        bf16lo_to_f32(q[4 * h + 2]), bf16hi_to_f32(q[4 * h + 2]), bf16lo_to_f32(q[4 * h + 3]), bf16hi_to_f32(q[4 * h + 3]));
    *reinterpret_cast<uint4*>(p.q_codes + (int64_t)row * (p.n >> 1) + (col >> 1)) = make_uint4(c[0], c[1], c[2], c[3]);
  }
  p.q_scales[swizzled_scale_offset(row, col >> 5, ((p.n >> 5) + 3) >> 2)] = (uint8_t)scale;
}

__device__ __forceinline__ void store_256(void* dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f, uint32_t g, uint32_t h) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(a), "r"(b), "r"(c), "r"(d), "r"(e), "r"(f), "r"(g), "r"(h) : "memory");
}

// Stores the chunk's bf16 outputs and adds them into the residual where STORE_OUT (the CTA-pair kernel stages them in shared memory
// instead: the TMA store and residual_add_box take them from there), and applies the quantized copy and the running amax.
template <int EPI, int FMT, bool STORE_OUT = true>
__device__ __forceinline__ void store_chunk(const GemmParams& p, const uint32_t (&packed)[16], int row, int col, uint32_t& amax2) {
  if (row >= p.m) return;
  if (p.q_codes && col + 32 <= p.n) store_chunk_quantized<FMT>(p, packed, row, col);
  if (!p.out) return;
  uint16_t* orow = STORE_OUT ? out_row_ptr(p, row) + col : nullptr;
  // 32-byte stores (whole L2 sectors, half as many store transactions per row) where the row's chunk is whole and 32-byte aligned
  const bool wide = STORE_OUT && col + 32 <= p.n && (reinterpret_cast<uintptr_t>(orow) & 31u) == 0;
  if (wide) {
    store_256(orow, packed[0], packed[1], packed[2], packed[3], packed[4], packed[5], packed[6], packed[7]);
    store_256(orow + 16, packed[8], packed[9], packed[10], packed[11], packed[12], packed[13], packed[14], packed[15]);
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    if (col + g * 8 + 8 <= p.n) {
      if (STORE_OUT && !wide) *reinterpret_cast<uint4*>(orow + g * 8) = make_uint4(packed[4 * g], packed[4 * g + 1], packed[4 * g + 2], packed[4 * g + 3]);
      if (p.out_amax) {
#pragma unroll
        for (int e = 0; e < 4; ++e) amax2 = __vmaxu2(amax2, packed[4 * g + e] & 0x7FFF7FFFu);
      }
      if (STORE_OUT && EPI == TF_EPI_RESIDUAL) {
        float4* rp = reinterpret_cast<float4*>(p.residual + (int64_t)row * p.n + col + g * 8);
        float4 r0 = rp[0], r1 = rp[1];
        r0.x = __fadd_rn(r0.x, bf16lo_to_f32(packed[4 * g]));
        r0.y = __fadd_rn(r0.y, bf16hi_to_f32(packed[4 * g]));
        r0.z = __fadd_rn(r0.z, bf16lo_to_f32(packed[4 * g + 1]));
        r0.w = __fadd_rn(r0.w, bf16hi_to_f32(packed[4 * g + 1]));
        r1.x = __fadd_rn(r1.x, bf16lo_to_f32(packed[4 * g + 2]));
        r1.y = __fadd_rn(r1.y, bf16hi_to_f32(packed[4 * g + 2]));
        r1.z = __fadd_rn(r1.z, bf16lo_to_f32(packed[4 * g + 3]));
        r1.w = __fadd_rn(r1.w, bf16hi_to_f32(packed[4 * g + 3]));
        rp[0] = r0;
        rp[1] = r1;
      }
    }
  }
}

// Which epilogue warps read chunk `c` (32 accumulator columns): the two groups of four warps (GRP 0 / 1) share the columns, alternating
// between the groups (with the SiLU gate: by the gate chunk; its up chunk goes with it).
template <int GRP, int EPI, int BLOCK_N>
__device__ __forceinline__ constexpr bool chunk_is_mine(int c) {
  // the unit a group owns is a PAIR of adjacent chunks where there are at least four (a thread then writes 128 contiguous bytes of its
  // output row, a whole line), else single chunks
  constexpr int kUnits = (EPI == TF_EPI_SILU_GATE) ? BLOCK_N / 64 : BLOCK_N / 32;
  const int u = (EPI == TF_EPI_SILU_GATE) ? (c % (BLOCK_N / 64)) : c;
  return ((kUnits >= 4 ? (u >> 1) : u) & 1) == GRP;
}

// residual += f32(staged bf16) for one warp's box of 32 rows x 64 columns, whose first row and column are row0 and col0. A half-warp
// takes one row's 64 columns, 256 contiguous bytes, and all 16 loads of a thread are in flight at once, 64 KB per SM: with four (16 KB per SM) a
// 256 x 256 tile whose residual is in HBM took 24000 clocks, twice its 20 K stages. Taken straight from the accumulator layout (a thread
// owns a row) every access of a warp would touch 32 lines.
constexpr int kResidualLoads = 16;
__device__ __forceinline__ void residual_add_box(const GemmParams& p, uint32_t box, int lane, int row0, int col0) {
  const int half = lane >> 4, c4 = lane & 15, col = col0 + c4 * 4;
  if (col >= p.n) return;  // n is a multiple of 8: the four columns are inside together
  float4* at = reinterpret_cast<float4*>(p.residual + (int64_t)(row0 + half) * p.n + col);
  const int step = p.n >> 1;  // float4 units of two rows
  const int rows = p.m - row0 - half;
  float4 r[kResidualLoads];
#pragma unroll
  for (int i = 0; i < kResidualLoads; ++i)
    if (i * 2 < rows) r[i] = at[(int64_t)i * step];
#pragma unroll
  for (int i = 0; i < kResidualLoads; ++i) {
    const int rr = i * 2 + half;
    if (i * 2 < rows) {
      uint32_t w0, w1;
      asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(w0), "=r"(w1) : "r"(box + rr * 128 + (((c4 >> 1) ^ (rr & 7)) << 4) + (c4 & 1) * 8));
      r[i].x = __fadd_rn(r[i].x, bf16lo_to_f32(w0));
      r[i].y = __fadd_rn(r[i].y, bf16hi_to_f32(w0));
      r[i].z = __fadd_rn(r[i].z, bf16lo_to_f32(w1));
      r[i].w = __fadd_rn(r[i].w, bf16hi_to_f32(w1));
      at[(int64_t)i * step] = r[i];
    }
  }
}

// One tile's epilogue for accumulator BUF (compile time, so that the chunks held in registers are indexed statically).
// t_acc: tensor-memory address of the accumulator for this warp's 32 lanes. Returns after the last store.
// PAIR (the CTA-pair kernel): the release goes to the leader's barrier, and the bf16 outputs leave through `stage_smem`, this warp's
// 4 KB staging box of 32 rows x 64 columns (128-byte swizzle), as one TMA store per pair of chunks.
template <int FMT, int BLOCK_N, int EPI, int BUF, int GRP, bool PAIR = false>
__device__ __forceinline__ void epilogue_tile(const GemmParams& p, uint32_t t_acc, uint32_t bar_release, int lane, int row, int col0, float alpha,
                                              uint32_t& amax2, const CUtensorMap* tma_out = nullptr, uint32_t stage_smem = 0) {
  using Cfg = TileCfg<FMT, BLOCK_N>;
  constexpr int kOutCols = (EPI == TF_EPI_SILU_GATE) ? BLOCK_N / 2 : BLOCK_N;
  constexpr int kOv = Cfg::kOverlapChunks;
  constexpr int kOvFirst = (BUF == 0) ? (BLOCK_N / 32 - kOv) : 0;  // first chunk (of this accumulator) the other accumulator also covers
  uint32_t ov[kOv > 0 ? kOv : 1][32];  // rows of chunks this warp does not read are never touched and cost no registers
  bool any_ov = false;
#pragma unroll
  for (int i = 0; i < kOv; ++i) {
    if (chunk_is_mine<GRP, EPI, BLOCK_N>(kOvFirst + i)) {
      tc_ld32(t_acc + (kOvFirst + i) * 32, ov[i]);
      any_ov = true;
    }
  }
  if (any_ov) tc_wait_ld();
  // With a residual the held columns become their bf16 outputs right away: half the registers, which the residual's loads need (2 x 34432 x 608 mxfp8 11.8 ->
  // 11.4 us; the plain epilogue has them to spare and is 1.5 % faster without).
  constexpr bool kHold = EPI == TF_EPI_RESIDUAL;
  // the columns shared with the other accumulator are in registers (or there are none): the next tile's MMAs may start
  tc_fence_before();
  __syncwarp();
  if (lane == 0) {
    if (PAIR) mbar_arrive_cluster(bar_release);
    else mbar_arrive(bar_release);
  }
  uint32_t held[kOv > 0 ? kOv : 1][16];
  if (kHold) {
#pragma unroll
    for (int i = 0; i < kOv; ++i) {
      if (chunk_is_mine<GRP, EPI, BLOCK_N>(kOvFirst + i)) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          held[i][j] = pack_bf16x2(__fmul_rn(__uint_as_float(ov[i][2 * j]), alpha), __fmul_rn(__uint_as_float(ov[i][2 * j + 1]), alpha));
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kOutCols / 32; ++c) {
    if (!chunk_is_mine<GRP, EPI, BLOCK_N>(c)) continue;
    uint32_t v[32], packed[16];
    const bool v_in_regs = kOv > 0 && c >= kOvFirst && c < kOvFirst + kOv;
    if (v_in_regs) {
      const int h = (c - kOvFirst) < 0 ? 0 : ((c - kOvFirst) >= kOv ? 0 : (c - kOvFirst));
      if (!kHold) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = ov[h][j];
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) packed[j] = held[h][j];
      }
    } else {
      tc_ld32(t_acc + c * 32, v);
    }
    if (EPI == TF_EPI_SILU_GATE) {
      uint32_t u[32];
      const int cu = BLOCK_N / 64 + c;  // the up chunk that pairs with gate chunk c
      const bool u_in_regs = kOv > 0 && cu >= kOvFirst && cu < kOvFirst + kOv;
      if (u_in_regs) {
#pragma unroll
        for (int j = 0; j < 32; ++j) u[j] = ov[(cu - kOvFirst) < 0 ? 0 : ((cu - kOvFirst) >= kOv ? 0 : (cu - kOvFirst))][j];
      } else {
        tc_ld32(t_acc + cu * 32, u);
      }
      if (!v_in_regs || !u_in_regs) tc_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        // the GEMM result is bf16 (one rounding); the gate then reads it back as f32, as the unfused graph does
        const uint32_t g2 = pack_bf16x2(__fmul_rn(__uint_as_float(v[2 * j]), alpha), __fmul_rn(__uint_as_float(v[2 * j + 1]), alpha));
        const uint32_t u2 = pack_bf16x2(__fmul_rn(__uint_as_float(u[2 * j]), alpha), __fmul_rn(__uint_as_float(u[2 * j + 1]), alpha));
        const float lo = __fmul_rn(silu_f32(bf16lo_to_f32(g2)), bf16lo_to_f32(u2));
        const float hi = __fmul_rn(silu_f32(bf16hi_to_f32(g2)), bf16hi_to_f32(u2));
        packed[j] = pack_bf16x2(lo, hi);
      }
    } else if (!v_in_regs || !kHold) {
      if (!v_in_regs) tc_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        packed[j] = pack_bf16x2(__fmul_rn(__uint_as_float(v[2 * j]), alpha), __fmul_rn(__uint_as_float(v[2 * j + 1]), alpha));
    }
    if (!PAIR) {
      store_chunk<EPI, FMT>(p, packed, row, col0 + c * 32, amax2);
      continue;
    }
    store_chunk<EPI, FMT, false>(p, packed, row, col0 + c * 32, amax2);
    if (!p.out) continue;
    if ((c & 1) == 0) {  // the box is free once the previous store has read it
      if (lane == 0) bulk_wait_read();
      __syncwarp();
    }
#pragma unroll
    for (int g = 0; g < 4; ++g)
      sts_128(stage_smem + (uint32_t)lane * 128u + ((uint32_t)(((c & 1) * 4 + g) ^ (lane & 7)) << 4), packed[4 * g], packed[4 * g + 1], packed[4 * g + 2],
              packed[4 * g + 3]);
    if (c & 1) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      // a box that starts inside the matrix is clipped at its edges; one that starts outside is not stored
      if (lane == 0 && row < p.m && col0 + (c - 1) * 32 < p.n) tma_store_2d(tma_out, stage_smem, col0 + (c - 1) * 32, row);
      if (lane == 0) bulk_commit();
    }
  }
}

// The pair kernel's epilogue one pair of chunks (64 columns) after the other: `count` pairs from chunk c0 on, c_step chunks apart; staged as bf16,
// stored, and (residual) added with nothing held in registers but the residual's loads. The accumulator is released behind pair `release_at`: the last
// one where tiles have accumulators of their own (192 columns), the first one with 256 columns. There the columns shared with the other accumulator (chunks 5-7 of accumulator 0, 0-2 of
// accumulator 1) lie in a group's first pair, so they need not be held either. Residual, four loads in flight and held columns -> this (graphs of 10):
// mxfp4 787 x 7536 x 1696 23.4 -> 19.8 us, 1000 x 3000 x 2720 16.6 -> 15.4; nvfp4 4096 x 4096 x 4096 56.5 -> 51.0, 8192 x 8192 x 1024 178.6 -> 163.6; mxfp8
// 8192 x 2560 x 3072 75.9 -> 70.5, 1024 x 4096 x 4096 22.0 -> 21.7. Both pairs staged at once in two boxes cost mxfp8 its fifth ring stage (78.6).
template <int FMT, int EPI>
__device__ __forceinline__ void epilogue_pairs(const GemmParams& p, uint32_t t_acc, int c0, int c_step, int count, int release_at, uint32_t bar_release, int lane,
                                               int row, int col0, float alpha, uint32_t& amax2, const CUtensorMap* tma_out, uint32_t stage_smem) {
#pragma unroll 1
  for (int i = 0; i < count; ++i, c0 += c_step) {
    if (lane == 0) bulk_wait_read();  // the box is free once the previous store has read it
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t v[32], packed[16];
      tc_ld32(t_acc + (c0 + h) * 32, v);
      tc_wait_ld();
      if (i == release_at && h == 1) {  // the accumulator (or what the next tile's shares of it) is read
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(bar_release);
      }
#pragma unroll
      for (int e = 0; e < 16; ++e)
        packed[e] = pack_bf16x2(__fmul_rn(__uint_as_float(v[2 * e]), alpha), __fmul_rn(__uint_as_float(v[2 * e + 1]), alpha));
      store_chunk<EPI, FMT, false>(p, packed, row, col0 + (c0 + h) * 32, amax2);
      if (p.out) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
          sts_128(stage_smem + (uint32_t)lane * 128u + ((uint32_t)((h * 4 + g) ^ (lane & 7)) << 4), packed[4 * g], packed[4 * g + 1], packed[4 * g + 2], packed[4 * g + 3]);
      }
    }
    if (!p.out) continue;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    // a box that starts inside the matrix is clipped at its edges; one that starts outside is not stored
    if (lane == 0 && row < p.m && col0 + c0 * 32 < p.n) tma_store_2d(tma_out, stage_smem, col0 + c0 * 32, row);
    if (lane == 0) bulk_commit();
    if (EPI == TF_EPI_RESIDUAL) {
      residual_add_box(p, stage_smem, lane, row - lane, col0 + c0 * 32);
      __syncwarp();  // every lane has read the box before the next pair is staged in it
    }
  }
}

// The one-CTA kernel's epilogue with a residual for 128-column tiles: a warp's pair of chunks is stored from the accumulator's layout as without
// one, staged in its box (the ring gives up a stage for the boxes), and added from there: rows of 256 contiguous bytes, sixteen loads in flight per thread.
// Before (each thread its own row, 32 lines per access) -> after: mxfp8 353 x 1104 x 1760 14.3 -> 10.2 us, 1024 x 2304 x 512 13.2 -> 8.0, 100 x 4000 x 1024
// 10.9 -> 7.5; nvfp4 769 x 1952 x 2592 17.0 -> 10.8, 16 x 8192 x 1024 7.0 -> 5.3; mxfp4 682 x 952 x 3808 16.4 -> 13.0, 200 x 2048 x 1024 11.1 -> 7.1.
template <int FMT>
__device__ __forceinline__ void epilogue_residual_128(const GemmParams& p, uint32_t t_acc, int grp, uint32_t bar_release, int lane, int row, int col0, float alpha,
                                                      uint32_t& amax2, uint32_t box) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = grp * 2 + h;
    uint32_t v[32], packed[16];
    tc_ld32(t_acc + c * 32, v);
    tc_wait_ld();
    if (h == 1) {  // the accumulator is read
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_release);
    }
#pragma unroll
    for (int e = 0; e < 16; ++e)
      packed[e] = pack_bf16x2(__fmul_rn(__uint_as_float(v[2 * e]), alpha), __fmul_rn(__uint_as_float(v[2 * e + 1]), alpha));
    store_chunk<TF_EPI_NONE, FMT>(p, packed, row, col0 + c * 32, amax2);
#pragma unroll
    for (int g = 0; g < 4; ++g)
      sts_128(box + (uint32_t)lane * 128u + ((uint32_t)((h * 4 + g) ^ (lane & 7)) << 4), packed[4 * g], packed[4 * g + 1], packed[4 * g + 2], packed[4 * g + 3]);
  }
  __syncwarp();
  residual_add_box(p, box, lane, row - lane, col0 + grp * 64);
  __syncwarp();  // every lane has read the box before the next tile is staged in it
}

// Split-K: dumps this (tile, split)'s raw f32 accumulator rows into the workspace [splits][M][acc columns].
template <int FMT, int BLOCK_N, int BUF, int GRP>
__device__ __forceinline__ void epilogue_partial(const GemmParams& p, uint32_t t_acc, uint32_t bar_release, int lane, int row, int col0,
                                                 float* __restrict__ ws_row) {
  using Cfg = TileCfg<FMT, BLOCK_N>;
  constexpr int kOv = Cfg::kOverlapChunks;
  constexpr int kOvFirst = (BUF == 0) ? (BLOCK_N / 32 - kOv) : 0;
  uint32_t ov[kOv > 0 ? kOv : 1][32];
  bool any_ov = false;
#pragma unroll
  for (int i = 0; i < kOv; ++i) {
    if (chunk_is_mine<GRP, TF_EPI_NONE, BLOCK_N>(kOvFirst + i)) {
      tc_ld32(t_acc + (kOvFirst + i) * 32, ov[i]);
      any_ov = true;
    }
  }
  if (any_ov) tc_wait_ld();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar_release);
#pragma unroll
  for (int c = 0; c < BLOCK_N / 32; ++c) {
    if (!chunk_is_mine<GRP, TF_EPI_NONE, BLOCK_N>(c)) continue;
    uint32_t v[32];
    const bool in_regs = kOv > 0 && c >= kOvFirst && c < kOvFirst + kOv;
    if (in_regs) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = ov[(c - kOvFirst) < 0 ? 0 : ((c - kOvFirst) >= kOv ? 0 : (c - kOvFirst))][j];
    } else {
      tc_ld32(t_acc + c * 32, v);
      tc_wait_ld();
    }
    if (row < p.m) {
      const int col = col0 + c * 32;
#pragma unroll
      for (int g = 0; g < 8; ++g)
        if (col + g * 4 + 4 <= p.n)
          *reinterpret_cast<uint4*>(ws_row + col + g * 4) = make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
    }
  }
}

// Split-K second pass: sums the partials in split order (deterministic), then the same epilogue arithmetic as the one-pass
// kernel. n_acc = accumulator columns (2 * n with the SiLU gate), one thread per 8 output columns. Bound by latency: four planes' loads
// are in flight at once (a loop over the planes waits for each: mxfp8 1 x 3072 x 2560 + gate 7.06 -> 6.65 us with three planes, mxfp4 5 x 288 x 28672 8.7 -> 7.95 with
// sixteen, README block at one row 18.2 -> 16.5).
constexpr int kReducePlanes = 4;
template <int EPI, int QFMT>  // QFMT: -1, or the MX format of a quantized copy of the output
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ ws, int splits, int m, int n, int n_acc, const float* a_gs,
                                                            const float* b_gs, uint16_t* __restrict__ out, int64_t ldo, float* __restrict__ residual,
                                                            unsigned int* __restrict__ out_amax, uint8_t* __restrict__ q_codes,
                                                            uint8_t* __restrict__ q_scales, int q_pad, int a_gs_rows) {
  griddep_launch_dependents();
  griddep_wait();
  if (QFMT >= 0 && q_pad)
    zero_scale_padding(q_scales, m, n >> 5, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
  const float alpha0 = (a_gs && b_gs) ? __fmul_rn(load_f32(a_gs), load_f32(b_gs)) : 1.0f;
  const int nvec = n >> 3;
  const int64_t total = (int64_t)m * nvec;
  const int64_t plane = (int64_t)m * n_acc;
  uint32_t amax2 = 0;
  // every thread runs the same number of rounds (the quantizer's shuffles need whole warps); n is a multiple of 32 when a
  // quantized copy is asked for, so the 4 lanes of one block have data together
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < total; i0 += stride) {
    const int64_t i = i0 + threadIdx.x;
    const bool live = i < total;
    if (!live && QFMT < 0) continue;
    const int row = live ? (int)(i / nvec) : 0, col = live ? (int)(i - (int64_t)row * nvec) * 8 : 0;
    float acc[8], up[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = up[j] = 0.0f;
    const float alpha = (a_gs && b_gs && a_gs_rows > 0) ? __fmul_rn(load_f32(a_gs + row / a_gs_rows), load_f32(b_gs)) : alpha0;
    const float* base = ws + (int64_t)row * n_acc + col;
    const int n_planes = live ? splits : 0;
    for (int sp = 0; sp < n_planes; sp += kReducePlanes) {
      float4 x[kReducePlanes][2], u[kReducePlanes][2];
#pragma unroll
      for (int j = 0; j < kReducePlanes; ++j) {
        if (sp + j < n_planes) {
          const float4* at = reinterpret_cast<const float4*>(base + (sp + j) * plane);
          x[j][0] = __ldcs(at);
          x[j][1] = __ldcs(at + 1);
          if (EPI == TF_EPI_SILU_GATE) {
            u[j][0] = __ldcs(at + (n >> 2));
            u[j][1] = __ldcs(at + (n >> 2) + 1);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kReducePlanes; ++j) {
        if (sp + j < n_planes) {
          const float4 x0 = x[j][0], x1 = x[j][1];
          acc[0] += x0.x; acc[1] += x0.y; acc[2] += x0.z; acc[3] += x0.w; acc[4] += x1.x; acc[5] += x1.y; acc[6] += x1.z; acc[7] += x1.w;
          if (EPI == TF_EPI_SILU_GATE) {
            const float4 u0 = u[j][0], u1 = u[j][1];
            up[0] += u0.x; up[1] += u0.y; up[2] += u0.z; up[3] += u0.w; up[4] += u1.x; up[5] += u1.y; up[6] += u1.z; up[7] += u1.w;
          }
        }
      }
    }
    uint32_t packed[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t g2 = pack_bf16x2(__fmul_rn(acc[2 * j], alpha), __fmul_rn(acc[2 * j + 1], alpha));
      if (EPI == TF_EPI_SILU_GATE) {
        const uint32_t u2 = pack_bf16x2(__fmul_rn(up[2 * j], alpha), __fmul_rn(up[2 * j + 1], alpha));
        packed[j] = pack_bf16x2(__fmul_rn(silu_f32(bf16lo_to_f32(g2)), bf16lo_to_f32(u2)), __fmul_rn(silu_f32(bf16hi_to_f32(g2)), bf16hi_to_f32(u2)));
      } else {
        packed[j] = g2;
      }
      amax2 = __vmaxu2(amax2, packed[j] & 0x7FFF7FFFu);
    }
    if (QFMT >= 0) {
      uint32_t c0, c1, sc;
      quantize_vec8<(QFMT < 0 ? 0 : QFMT)>(make_uint4(packed[0], packed[1], packed[2], packed[3]), 0.0f, 0.0f, c0, c1, sc);
      if (live) store_quantized<(QFMT < 0 ? 0 : QFMT)>(q_codes, q_scales, 1, row, col >> 3, n, c0, c1, sc);
    }
    if (!live) continue;
    if (out) *reinterpret_cast<uint4*>(out + (int64_t)row * ldo + col) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    if (EPI == TF_EPI_RESIDUAL) {
      float4* rp = reinterpret_cast<float4*>(residual + (int64_t)row * n + col);
      float4 r0 = rp[0], r1 = rp[1];
      r0.x = __fadd_rn(r0.x, bf16lo_to_f32(packed[0])); r0.y = __fadd_rn(r0.y, bf16hi_to_f32(packed[0]));
      r0.z = __fadd_rn(r0.z, bf16lo_to_f32(packed[1])); r0.w = __fadd_rn(r0.w, bf16hi_to_f32(packed[1]));
      r1.x = __fadd_rn(r1.x, bf16lo_to_f32(packed[2])); r1.y = __fadd_rn(r1.y, bf16hi_to_f32(packed[2]));
      r1.z = __fadd_rn(r1.z, bf16lo_to_f32(packed[3])); r1.w = __fadd_rn(r1.w, bf16hi_to_f32(packed[3]));
      rp[0] = r0;
      rp[1] = r1;
    }
  }
  if (out_amax) {
    uint32_t mx = max(amax2 & 0xFFFFu, amax2 >> 16);
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(out_amax, mx << 16);
  }
}

// ---- split-K inside a cluster -----------------------------------------------------------------------------------------------
// The CTAs of a cluster hold one K range each of the same output tile. Every CTA leaves its f32 accumulator rows in its own shared
// memory (the operand ring is free by then), the cluster meets, and each CTA sums its share of the tile over the ranges, read
// from its peers' shared memory, in split order: the arithmetic, and so the bytes, of epilogue_partial + splitk_reduce_kernel
// without the second launch and without the trip of the partial sums through the workspace.
template <int BLOCK_N>
struct DumpCfg {
  static constexpr int kPitch = (BLOCK_N + 4) * 4;  // bytes per row; the 16 bytes of padding spread a warp's rows over the banks
  static constexpr int kBytes = kBlockM * kPitch;
};

template <int FMT, int BLOCK_N, int GRP>
__device__ __forceinline__ void epilogue_dump(uint32_t t_acc, uint32_t smem_row) {
#pragma unroll
  for (int c = 0; c < BLOCK_N / 32; ++c) {
    if (!chunk_is_mine<GRP, TF_EPI_NONE, BLOCK_N>(c)) continue;
    uint32_t v[32];
    tc_ld32(t_acc + c * 32, v);
    tc_wait_ld();
#pragma unroll
    for (int g = 0; g < 8; ++g) sts_128(smem_row + c * 128 + g * 16, v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
  }
}

// All threads of the CTA; `dump` is the shared address of the dumped rows (the same in every CTA of the cluster).
template <int FMT, int BLOCK_N, int EPI>
__device__ __forceinline__ void cluster_reduce(const GemmParams& p, uint32_t dump, int rank, int m_blk, int n_blk) {
  constexpr int kOutCols = (EPI == TF_EPI_SILU_GATE) ? BLOCK_N / 2 : BLOCK_N;
  constexpr int kVecs = kOutCols / 8;
  const int rows = min(kBlockM, p.m - m_blk * kBlockM);
  const int total = rows * kVecs;
  const bool quantize = FMT != TF_FMT_NVFP4 && p.q_codes != nullptr;
  const float alpha0 = (FMT == TF_FMT_NVFP4) ? __fmul_rn(load_f32(p.a_gs), load_f32(p.b_gs)) : 1.0f;
  uint32_t amax2 = 0;
  // whole warps run every round (the quantizer's shuffles); the 4 lanes of one MX block always have data together
  for (int i0 = rank * kGemmThreads; i0 < total; i0 += p.splits * kGemmThreads) {
    const int i = i0 + (int)threadIdx.x;
    const int r = i / kVecs, cv = i - r * kVecs;
    const int row = m_blk * kBlockM + r, col = n_blk * kOutCols + cv * 8;
    const bool live = i < total && col < p.n;
    float acc[8], up[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = up[j] = 0.0f;
    const uint32_t local = dump + (uint32_t)(live ? r : 0) * DumpCfg<BLOCK_N>::kPitch + (uint32_t)(live ? cv : 0) * 32u;
    // four ranges' loads in flight (a remote read takes about 0.4 us); the second four lanes of every eight take their two halves in
    // the other order, so that the eight lanes a read serves together touch different banks
    const uint32_t swap = (threadIdx.x >> 2) & 1u;
    for (int sp = 0; sp < p.splits; sp += 4) {
      float4 x[4][2], u[4][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (sp + j < p.splits) {
          const uint32_t src = mapa_shared(local, (uint32_t)(sp + j));
          x[j][0] = ld_cluster_f4(src + 16 * swap);
          x[j][1] = ld_cluster_f4(src + 16 - 16 * swap);
          if (EPI == TF_EPI_SILU_GATE) {
            u[j][0] = ld_cluster_f4(src + BLOCK_N * 2 + 16 * swap);
            u[j][1] = ld_cluster_f4(src + BLOCK_N * 2 + 16 - 16 * swap);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (sp + j < p.splits) {
          const float4 x0 = swap ? x[j][1] : x[j][0], x1 = swap ? x[j][0] : x[j][1];
          acc[0] += x0.x; acc[1] += x0.y; acc[2] += x0.z; acc[3] += x0.w; acc[4] += x1.x; acc[5] += x1.y; acc[6] += x1.z; acc[7] += x1.w;
          if (EPI == TF_EPI_SILU_GATE) {
            const float4 u0 = swap ? u[j][1] : u[j][0], u1 = swap ? u[j][0] : u[j][1];
            up[0] += u0.x; up[1] += u0.y; up[2] += u0.z; up[3] += u0.w; up[4] += u1.x; up[5] += u1.y; up[6] += u1.z; up[7] += u1.w;
          }
        }
      }
    }
    const float alpha = (FMT == TF_FMT_NVFP4 && live && p.a_gs_rows > 0) ? __fmul_rn(load_f32(p.a_gs + row / p.a_gs_rows), load_f32(p.b_gs)) : alpha0;
    uint32_t packed[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t g2 = pack_bf16x2(__fmul_rn(acc[2 * j], alpha), __fmul_rn(acc[2 * j + 1], alpha));
      if (EPI == TF_EPI_SILU_GATE) {
        const uint32_t u2 = pack_bf16x2(__fmul_rn(up[2 * j], alpha), __fmul_rn(up[2 * j + 1], alpha));
        packed[j] = pack_bf16x2(__fmul_rn(silu_f32(bf16lo_to_f32(g2)), bf16lo_to_f32(u2)), __fmul_rn(silu_f32(bf16hi_to_f32(g2)), bf16hi_to_f32(u2)));
      } else {
        packed[j] = g2;
      }
    }
    if (quantize) {
      uint32_t c0, c1, sc;
      constexpr int kQ = FMT == TF_FMT_NVFP4 ? TF_FMT_MXFP8 : FMT;
      quantize_vec8<kQ>(make_uint4(packed[0], packed[1], packed[2], packed[3]), 0.0f, 0.0f, c0, c1, sc);
      if (live) store_quantized<kQ>(p.q_codes, p.q_scales, 1, row, col >> 3, p.n, c0, c1, sc);
    }
    if (!live) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) amax2 = __vmaxu2(amax2, packed[j] & 0x7FFF7FFFu);
    if (p.out) *reinterpret_cast<uint4*>(out_row_ptr(p, row) + col) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    if (EPI == TF_EPI_RESIDUAL) {
      float4* rp = reinterpret_cast<float4*>(p.residual + (int64_t)row * p.n + col);
      float4 r0 = rp[0], r1 = rp[1];
      r0.x = __fadd_rn(r0.x, bf16lo_to_f32(packed[0])); r0.y = __fadd_rn(r0.y, bf16hi_to_f32(packed[0]));
      r0.z = __fadd_rn(r0.z, bf16lo_to_f32(packed[1])); r0.w = __fadd_rn(r0.w, bf16hi_to_f32(packed[1]));
      r1.x = __fadd_rn(r1.x, bf16lo_to_f32(packed[2])); r1.y = __fadd_rn(r1.y, bf16hi_to_f32(packed[2]));
      r1.z = __fadd_rn(r1.z, bf16lo_to_f32(packed[3])); r1.w = __fadd_rn(r1.w, bf16hi_to_f32(packed[3]));
      rp[0] = r0;
      rp[1] = r1;
    }
  }
  if (p.out_amax) {
    uint32_t mx = max(amax2 & 0xFFFFu, amax2 >> 16);
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(p.out_amax, mx << 16);
  }
}

// ---- L2 prefetch of the weights ---------------------------------------------------------------------------------------------
// A dependent of at most 128 rows streams its weights once, and HBM is idle while it waits: the row kernels between two GEMMs of a decode
// step touch a few MB. So a waiting CTA asks its first stages of B and their scales into L2. Nothing is read here: the lines are coherent
// with what the kernel in front may still write (it may be the one that quantizes these weights), and the loads behind griddep_wait()
// read them as they would without. Captured stacks, us per step, dependents without -> with this: 70B-shaped NVFP4 blocks 64 rows, 4 layers 382.7 ->
// 378.6, 128 rows, 2 layers 209.0 -> 207.8; MXFP8 64 x 4096 x 8192, 4 layers 146.5 -> 142.5, 8 x 2560 x 3072, 6 layers 105.8 -> 100.7; MXFP4 1 x 4096 x 14336,
// 3 layers 103.3 -> 101.4. Eight stages give the first 376.2 and the fourth 99.4, but behind a GEMM that streams weights of its own they take
// HBM from its last CTAs: nvfp4 8 x 26240 x 5984 back to back over cold weights 19.4 without, 19.5 with four, 20.4 with eight, mxfp4 3 x 20096 x 4096
// 13.1 / 13.1 / 13.6 (mxfp8 2 x 34432 x 608 9.5 / 8.9 / 8.9). The SM's copy engine serves the prefetch before the loads (about 2.7
// clocks per 128-byte row), so prefetching ahead inside the main loop or for other CTAs' tiles loses too (64 x 28672 x 8192 + gate 50.6 -> 53.4 us;
// 2 to 3 us per layer). It stands in the epilogue's branch: in front of the roles the same code cost every launch 0.2 us.
constexpr int kEarlyStages = 4;
constexpr unsigned kEarlyStageNs = 300;  // pause between two stages: 36 KB per SM and pause is more than HBM brings
__device__ __forceinline__ void l2_prefetch_2d(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void l2_prefetch_bulk(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
template <int FMT, int BLOCK_N, int EPI>
__device__ __forceinline__ void prefetch_b_stage(const GemmParams& p, const CUtensorMap* tma_b, int n_blk, int ks) {
  constexpr int kST = TileCfg<FMT, BLOCK_N>::kST;
  const int sf_tiles = min(p.sf_col_tiles - ks * kST, kST);
#pragma unroll
  for (int nb = 0; nb < TileCfg<FMT, BLOCK_N>::kNB; ++nb) {
    const int row = (EPI == TF_EPI_SILU_GATE) ? nb * p.n + n_blk * 128 : n_blk * BLOCK_N + nb * 128;
    if (row < p.n_rows_b) {
      l2_prefetch_2d(tma_b, ks * kStageKBytes, row);
      l2_prefetch_bulk(p.sfb + ((int64_t)(row >> 7) * p.sf_col_tiles + ks * kST) * 512, (uint32_t)sf_tiles * 512u);
    }
  }
}

// ---- the kernel ------------------------------------------------------------------------------------------------------------
// SPLITK: kSplitNone; kSplitPlanes: every (tile, K range) is a unit of its own and leaves its accumulator in the workspace;
// kSplitCluster: a cluster of `splits` CTAs per tile, launched with exactly one tile per cluster.
constexpr int kSplitNone = 0, kSplitPlanes = 1, kSplitCluster = 2;
constexpr int kFormPair = 3;  // what tf_gemm_launch_form calls the CTA pair
constexpr int kMaxClusterSplits = 8;  // the portable cluster size
// BOXES (128-column tiles with a residual): a 4 KB staging box per epilogue warp in place of a ring stage, see epilogue_residual_128.
template <int FMT, int BLOCK_N, int EPI, int SPLITK, bool BOXES = false>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_blockscaled_kernel(const __grid_constant__ CUtensorMap tma_a,
                                                                            const __grid_constant__ CUtensorMap tma_b, const GemmParams p) {
  using Cfg = TileCfg<FMT, BLOCK_N>;
  static_assert(!BOXES || (EPI == TF_EPI_RESIDUAL && SPLITK == kSplitNone && BLOCK_N == 128), "staging boxes");
  constexpr int kBoxBytes = BOXES ? 8 * 4096 : 0;
  constexpr int kStages = Cfg::kStages - (BOXES ? 1 : 0);
  static_assert(kBoxBytes <= (Cfg::kStages - kStages) * Cfg::kStageBytes, "the boxes take a stage's place");
  constexpr int kNB = Cfg::kNB;
  constexpr int kST = Cfg::kST;
  constexpr int kOutCols = (EPI == TF_EPI_SILU_GATE) ? BLOCK_N / 2 : BLOCK_N;  // output columns per tile
  constexpr bool kCluster = SPLITK == kSplitCluster;
  static_assert(!kCluster || DumpCfg<BLOCK_N>::kBytes <= kStages * Cfg::kStageBytes, "the dumped accumulator must fit in the operand ring");
  static_assert(EPI != TF_EPI_SILU_GATE || BLOCK_N == 256, "the SiLU-gate epilogue pairs a 128-column gate tile with its up tile");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_a = smem_base;
  const uint32_t smem_b = smem_a + kStages * kAStageBytes;
  const uint32_t smem_boxes = smem_b + kStages * Cfg::kBStageBytes;
  const uint32_t smem_sfa = smem_boxes + kBoxBytes;
  const uint32_t smem_sfb = smem_sfa + kStages * Cfg::kSfaStageBytes;
  const uint32_t bars = smem_sfb + kStages * Cfg::kSfbStageBytes;  // 8-byte aligned
  const uint32_t bar_full = bars, bar_empty = bars + 8 * kStages, bar_tmem_full = bars + 16 * kStages, bar_tmem_empty = bar_tmem_full + 8;
  const uint32_t tmem_slot = bar_tmem_empty + 8;
  const uint32_t abort_slot = tmem_slot + 4;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - smem_base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + (abort_slot - smem_base));
  volatile int* started_flag = abort_flag + 1;  // the kernel in front has completed

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  griddep_launch_dependents();  // the next kernel on the stream may be scheduled; it waits for this one before touching memory

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full + 8 * s, 2);  // the operand-load warp and the scale-load warp
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_tmem_full, 1);
    mbar_init(bar_tmem_empty, 8);  // every epilogue warp, once it holds its share of the columns both accumulators cover
    *abort_flag = 0;
    *started_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // whole warp: allocate tensor memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"((uint32_t)Cfg::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // barriers and tensor memory are set up; every role waits (griddep_wait) before it reads or writes global memory

  if (warp == 0 || warp == 6) {
    // ---------------- load warps: warp 0 the operand tiles (TMA), warp 6 the scale tiles (bulk copies) ----------------
    // The whole warp runs the loops; lane 0 serves the A side, lane 1 + nb the 128-row half nb of the B tile, so that one
    // instruction per stage issues all of the warp's copies.
    griddep_wait();
    const bool scales = warp == 6;
    if (!scales && lane == 0) *started_flag = 1;
    const int nb = lane - 1;
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
      const int split = SPLITK == kSplitPlanes ? tile / (p.m_blocks * p.n_blocks) : kCluster ? tile % p.splits : 0;
      const int rest = SPLITK == kSplitPlanes ? tile % (p.m_blocks * p.n_blocks) : kCluster ? tile / p.splits : tile;
      const int m_blk = rest % p.m_blocks, n_blk = rest / p.m_blocks;
      const int ks_begin = split * p.k_stages_per_split;
      const int ks_end = min(ks_begin + p.k_stages_per_split, p.num_k_stages);
      int n_b_ok = 0;  // B halves that lie inside the matrix (uniform)
#pragma unroll
      for (int i = 0; i < kNB; ++i)
        n_b_ok += (((EPI == TF_EPI_SILU_GATE) ? i * p.n + n_blk * 128 : n_blk * BLOCK_N + i * 128) < p.n_rows_b) ? 1 : 0;
      // this lane's copy: source row (operands) or scale row-tile, destination inside a stage
      const int my_row = lane == 0 ? m_blk * kBlockM : ((EPI == TF_EPI_SILU_GATE) ? nb * p.n + n_blk * 128 : n_blk * BLOCK_N + nb * 128);
      const bool mine = lane == 0 || (lane <= kNB && my_row < p.n_rows_b);
      const CUtensorMap* my_map = lane == 0 ? &tma_a : &tma_b;
      const uint32_t my_dst = scales ? (lane == 0 ? smem_sfa : smem_sfb + (uint32_t)(nb < 0 ? 0 : nb) * kST * 512)
                                     : (lane == 0 ? smem_a : smem_b + (uint32_t)(nb < 0 ? 0 : nb) * 128 * kStageKBytes);
      const uint32_t my_stage_bytes = scales ? (lane == 0 ? Cfg::kSfaStageBytes : Cfg::kSfbStageBytes) : (lane == 0 ? kAStageBytes : Cfg::kBStageBytes);
      const uint8_t* my_sf = (lane == 0 ? p.sfa : p.sfb) + (int64_t)((lane == 0 ? my_row : (my_row < 0 ? 0 : my_row)) >> 7) * p.sf_col_tiles * 512;
      for (int ks = ks_begin; ks < ks_end; ++ks) {
        ok = mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, 1);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        const uint32_t full = bar_full + 8 * stage;
        if (scales) {
          int sf_tiles = p.sf_col_tiles - ks * kST;
          sf_tiles = sf_tiles > kST ? kST : sf_tiles;
          const uint32_t sf_bytes = (uint32_t)sf_tiles * 512u;
          if (lane == 0) mbar_expect_tx(full, sf_bytes * (uint32_t)(1 + n_b_ok));
          __syncwarp();
          if (mine) bulk_load(my_dst + stage * my_stage_bytes, my_sf + (int64_t)ks * kST * 512, sf_bytes, full);
        } else {
          if (lane == 0) mbar_expect_tx(full, (uint32_t)p.a_box_bytes + (uint32_t)n_b_ok * (128u * kStageKBytes));
          __syncwarp();
          if (mine) tma_load_2d(my_dst + stage * my_stage_bytes, my_map, ks * kStageKBytes, my_row, full);
        }
        __syncwarp();
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok && lane == 0) {
      // give copies already in flight time to land before shared memory is released
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    griddep_wait();
    // ---------------- MMA issuer ----------------
    // The whole warp runs the loops (so every value below is warp-uniform and lives in the uniform datapath); one elected lane
    // issues the tcgen05 instructions. A full stage is straight-line code: its descriptors differ from the stage's base by
    // compile-time constants added to the low word (the 14-bit address field cannot carry out for addresses below 256 KB).
    constexpr uint32_t idesc_base = (FmtTraits<FMT>::kElemFormat << 7) | (FmtTraits<FMT>::kElemFormat << 10) | ((uint32_t)(BLOCK_N >> 3) << 17) |
                                    (FmtTraits<FMT>::kScaleIsE8 << 23) | ((uint32_t)(kBlockM >> 4) << 24);
    constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024 B, version 1, SWIZZLE_128B
    constexpr uint32_t kDescHiSf = (128u >> 4) | (1u << 14);                   // SBO 128 B, version 1, no swizzle
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0, tile_phase = 0, sf_buf = 0, acc_buf = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < p.num_tiles && ok; tile += gridDim.x) {
      ok = mbar_wait(bar_tmem_empty, tile_phase ^ 1, abort_flag, 2);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t tmem_acc = tmem_base + acc_buf * Cfg::kAccStride;
      acc_buf ^= 1;
      const int split = SPLITK == kSplitPlanes ? tile / (p.m_blocks * p.n_blocks) : kCluster ? tile % p.splits : 0;
      const int n_blk = (SPLITK == kSplitPlanes ? tile % (p.m_blocks * p.n_blocks) : kCluster ? tile / p.splits : tile) / p.m_blocks;
      const int ks_begin = split * p.k_stages_per_split;
      const int ks_end = min(ks_begin + p.k_stages_per_split, p.num_k_stages);
      bool all_b = true;
      bool b_ok[kNB];
#pragma unroll
      for (int nb = 0; nb < kNB; ++nb) {
        b_ok[nb] = ((EPI == TF_EPI_SILU_GATE) ? nb * p.n + n_blk * 128 : n_blk * BLOCK_N + nb * 128) < p.n_rows_b;
        all_b = all_b && b_ok[nb];
      }
      for (int ks = ks_begin; ks < ks_end; ++ks) {
        ok = mbar_wait(bar_full + 8 * stage, phase, abort_flag, 3);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tmem_sfa = tmem_base + Cfg::kTmemSfa + sf_buf * Cfg::kTmemSfSet;
        const uint32_t tmem_sfb = tmem_base + Cfg::kTmemSfb + sf_buf * Cfg::kTmemSfSet;
        sf_buf ^= 1;
        const uint32_t sfa_lo = ((smem_sfa + stage * Cfg::kSfaStageBytes) & 0x3FFFFu) >> 4;
        const uint32_t sfb_lo = ((smem_sfb + stage * Cfg::kSfbStageBytes) & 0x3FFFFu) >> 4;
        const uint32_t a_lo = (((smem_a + stage * kAStageBytes) & 0x3FFFFu) >> 4) | (1u << 16);
        const uint32_t b_lo = (((smem_b + stage * Cfg::kBStageBytes) & 0x3FFFFu) >> 4) | (1u << 16);
        const int sf_left = p.sf_col_tiles - ks * kST;
        const int k_left = p.k_bytes - ks * kStageKBytes;
        const uint32_t first = (ks > ks_begin) ? 1u : 0u;
        if (elected) {
          if (sf_left >= kST && k_left >= kStageKBytes && all_b) {
#pragma unroll
            for (int t = 0; t < kST; ++t) {
              tc_cp_sf(tmem_sfa + t * 4, make_desc(sfa_lo + t * 32, kDescHiSf));
#pragma unroll
              for (int nb = 0; nb < kNB; ++nb) tc_cp_sf(tmem_sfb + (t * kNB + nb) * 4, make_desc(sfb_lo + (nb * kST + t) * 32, kDescHiSf));
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              constexpr int kDummy = 0;
              (void)kDummy;
              const int t = (FMT == TF_FMT_MXFP8) ? 0 : (FMT == TF_FMT_MXFP4) ? (j >> 1) : j;
              const uint32_t sf_id = (FMT == TF_FMT_MXFP8) ? (uint32_t)j : (FMT == TF_FMT_MXFP4) ? (uint32_t)((j & 1) * 2) : 0u;
              tc_mma<FMT>(tmem_acc, make_desc(a_lo + j * 2, kDescHiSw128), make_desc(b_lo + j * 2, kDescHiSw128),
                          idesc_base | (sf_id << 4) | (sf_id << 29), tmem_sfa + t * 4, tmem_sfb + t * kNB * 4, j > 0 ? 1u : first);
            }
          } else {  // ragged stage: fewer scale tiles, fewer MMAs or a B half that lies outside the matrix
            const int sf_tiles = sf_left > kST ? kST : sf_left;
            for (int t = 0; t < sf_tiles; ++t) {
              tc_cp_sf(tmem_sfa + t * 4, make_desc(sfa_lo + t * 32, kDescHiSf));
#pragma unroll
              for (int nb = 0; nb < kNB; ++nb)
                if (b_ok[nb]) tc_cp_sf(tmem_sfb + (t * kNB + nb) * 4, make_desc(sfb_lo + (nb * kST + t) * 32, kDescHiSf));
            }
            const int n_mma = k_left >= kStageKBytes ? 4 : (k_left + 31) >> 5;
            for (int j = 0; j < n_mma; ++j) {
              const int t = (FMT == TF_FMT_MXFP8) ? 0 : (FMT == TF_FMT_MXFP4) ? (j >> 1) : j;
              const uint32_t sf_id = (FMT == TF_FMT_MXFP8) ? (uint32_t)j : (FMT == TF_FMT_MXFP4) ? (uint32_t)((j & 1) * 2) : 0u;
              tc_mma<FMT>(tmem_acc, make_desc(a_lo + j * 2, kDescHiSw128), make_desc(b_lo + j * 2, kDescHiSw128),
                          idesc_base | (sf_id << 4) | (sf_id << 29), tmem_sfa + t * 4, tmem_sfb + t * kNB * 4, j > 0 ? 1u : first);
            }
          }
          tc_commit(bar_empty + 8 * stage);  // the stage is free once these MMAs have read it
        }
        __syncwarp();
        if (++stage == kStages) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      if (elected) tc_commit(bar_tmem_full);  // accumulator complete
      __syncwarp();
      tile_phase ^= 1;
    }
  } else {
    // ---------------- epilogue (warps 2..5 = group 0, warps 7..10 = group 1; warp w reads lanes 32*(w%4) .. +31) ----------------
    if (p.early_stages > 0 && warp == 10) {
      // stage by stage until warp 0 is through its wait (not by a load warp, which must not be late for its own wait)
      int left = p.early_stages;
      for (int tile = blockIdx.x; tile < p.num_tiles && left > 0; tile += gridDim.x) {
        const int split = SPLITK == kSplitPlanes ? tile / (p.m_blocks * p.n_blocks) : kCluster ? tile % p.splits : 0;
        const int n_blk = (SPLITK == kSplitPlanes ? tile % (p.m_blocks * p.n_blocks) : kCluster ? tile / p.splits : tile) / p.m_blocks;
        const int ks_end = min((split + 1) * p.k_stages_per_split, p.num_k_stages);
        for (int ks = split * p.k_stages_per_split; ks < ks_end && left > 0; ++ks, --left) {
          if (__any_sync(0xFFFFFFFFu, *started_flag)) left = 0;  // one answer for the warp: warp 0 may be storing it just now
          if (left > 0 && lane == 0) prefetch_b_stage<FMT, BLOCK_N, EPI>(p, &tma_b, n_blk, ks);
          __syncwarp();
          if (left > 0) __nanosleep(kEarlyStageNs);
        }
      }
    }
    __syncwarp();
    griddep_wait();
    const int q = warp & 3;
    const int grp = warp >= 7 ? 1 : 0;
    const float alpha = (FMT == TF_FMT_NVFP4 && SPLITK == kSplitNone) ? __fmul_rn(load_f32(p.a_gs), load_f32(p.b_gs)) : 1.0f;
    uint32_t tile_phase = 0, acc_buf = 0;
    uint32_t amax2 = 0;  // running max of |out| as two packed bf16 magnitudes
    if (FMT != TF_FMT_NVFP4 && p.q_codes && p.q_pad)
      zero_scale_padding(p.q_scales, p.m, p.n >> 5, (int64_t)blockIdx.x * 256 + (grp * 4 + q) * 32 + lane, (int64_t)gridDim.x * 256);
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x) {
      const int split = SPLITK == kSplitPlanes ? tile / (p.m_blocks * p.n_blocks) : kCluster ? tile % p.splits : 0;
      const int rest = SPLITK == kSplitPlanes ? tile % (p.m_blocks * p.n_blocks) : kCluster ? tile / p.splits : tile;
      const int m_blk = rest % p.m_blocks, n_blk = rest / p.m_blocks;
      bool ok = mbar_wait(bar_tmem_full, tile_phase, abort_flag, 4);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after();
      const int row = m_blk * kBlockM + q * 32 + lane;
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
      const int col0 = n_blk * kOutCols;
      const float alpha_t = (FMT == TF_FMT_NVFP4 && SPLITK == kSplitNone && p.a_gs_rows > 0) ? __fmul_rn(load_f32(p.a_gs + min(row, p.m - 1) / p.a_gs_rows), load_f32(p.b_gs)) : alpha;
      if (kCluster) {
        if (m_blk * kBlockM + q * 32 < p.m) {
          const uint32_t smem_row = smem_a + (uint32_t)(q * 32 + lane) * DumpCfg<BLOCK_N>::kPitch;
          if (grp == 0) epilogue_dump<FMT, BLOCK_N, 0>(t_row, smem_row);
          else epilogue_dump<FMT, BLOCK_N, 1>(t_row, smem_row);
        }
      } else if (SPLITK == kSplitPlanes) {
        float* ws_row = p.ws + ((int64_t)split * p.m + row) * p.n;
        if (acc_buf == 0) {
          if (grp == 0) epilogue_partial<FMT, BLOCK_N, 0, 0>(p, t_row, bar_tmem_empty, lane, row, col0, ws_row);
          else epilogue_partial<FMT, BLOCK_N, 0, 1>(p, t_row, bar_tmem_empty, lane, row, col0, ws_row);
        } else {
          if (grp == 0) epilogue_partial<FMT, BLOCK_N, 1, 0>(p, t_row + Cfg::kAccStride, bar_tmem_empty, lane, row, col0, ws_row);
          else epilogue_partial<FMT, BLOCK_N, 1, 1>(p, t_row + Cfg::kAccStride, bar_tmem_empty, lane, row, col0, ws_row);
        }
      } else if (BOXES) {
        epilogue_residual_128<FMT>(p, t_row + acc_buf * Cfg::kAccStride, grp, bar_tmem_empty, lane, row, col0, alpha_t, amax2, smem_boxes + (uint32_t)(grp * 4 + q) * 4096u);
      } else if (acc_buf == 0) {
        if (grp == 0) epilogue_tile<FMT, BLOCK_N, EPI, 0, 0>(p, t_row, bar_tmem_empty, lane, row, col0, alpha_t, amax2);
        else epilogue_tile<FMT, BLOCK_N, EPI, 0, 1>(p, t_row, bar_tmem_empty, lane, row, col0, alpha_t, amax2);
      } else {
        if (grp == 0) epilogue_tile<FMT, BLOCK_N, EPI, 1, 0>(p, t_row + Cfg::kAccStride, bar_tmem_empty, lane, row, col0, alpha_t, amax2);
        else epilogue_tile<FMT, BLOCK_N, EPI, 1, 1>(p, t_row + Cfg::kAccStride, bar_tmem_empty, lane, row, col0, alpha_t, amax2);
      }
      acc_buf ^= 1;
      tile_phase ^= 1;
    }
    if (SPLITK == kSplitNone && p.out_amax) {  // one atomic per warp
      uint32_t mx = max(amax2 & 0xFFFFu, amax2 >> 16);
      for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
      if (lane == 0 && mx) atomicMax(p.out_amax, mx << 16);
    }
  }

  // ---------------- teardown: every thread arrives, then the allocating warp frees tensor memory ----------------
  tc_fence_before();
  __syncthreads();
  if (kCluster) {
    cluster_sync_all();  // every CTA's rows are dumped
    const int rest = (int)blockIdx.x / p.splits;
    cluster_reduce<FMT, BLOCK_N, EPI>(p, smem_a, (int)blockIdx.x % p.splits, rest % p.m_blocks, rest / p.m_blocks);
    cluster_sync_all();  // nobody leaves while a peer may still read this CTA's shared memory
  }
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)Cfg::kTmemCols) : "memory");
  }
}

// ---- the 2-CTA kernel ------------------------------------------------------------------------------------------------------
// Two CTAs of a cluster (a pair of SMs) compute one 256 x 256 tile (or 256 x 192, see pair_width) with tcgen05.mma.cta_group::2: CTA r of the pair holds
// rows [128 r, 128 r + 128) of the A tile and half r of the B tile in its own shared memory and the accumulator of its 128 rows in its own
// tensor memory. Per stage each SM fills 256 operand rows instead of the 384 that bound the one-CTA kernel (38 KB instead of 54
// for nvfp4). Each CTA loads its own halves with plain (non-multicast) TMA; the scale tiles of all 256 B rows are loaded by
// both CTAs (4 KB per stage). The warp roles are the one-CTA kernel's: operand loads (warp 0) and scale loads (warp 6), one
// multi-lane instruction per stage each; the MMA issuer (warp 1, leader CTA only: it issues the scale copies and MMAs for both);
// two groups of four epilogue warps. Barriers that both CTAs wait on are signalled with tcgen05.commit's multicast arrive; the
// peer's load and epilogue warps signal the leader through cluster-mapped mbarrier addresses. The bf16 outputs are staged in
// shared memory (a 4 KB box per epilogue warp) and leave as TMA stores: whole 128-byte lines instead of 32 partial lines per
// warp instruction. Same bounded waits and teardown as the one-CTA kernel, plus a cluster barrier at both ends.
template <int FMT, int BLOCK_N>
struct PairCfg {
  static_assert(BLOCK_N == 256 || BLOCK_N == 192, "tile widths of the pair");
  static constexpr int kST = FmtTraits<FMT>::kSfTiles;
  static constexpr int kBHalfBytes = BLOCK_N / 2 * kStageKBytes;
  static constexpr int kSfaStageBytes = kST * 512;
  static constexpr int kSfbStageBytes = kST * 512 * 2;
  static constexpr int kStageBytes = kAStageBytes + kBHalfBytes + kSfaStageBytes + kSfbStageBytes;
  static constexpr int kBarrierBytes = 256;
  static constexpr int kOutBoxBytes = 32 * 128;            // one epilogue warp's staging box
  static constexpr int kOutStageBytes = 8 * kOutBoxBytes;
  static constexpr int kStagesRaw = (kSmemLimit - 1024 - kBarrierBytes - kOutStageBytes) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  // Tensor memory of each CTA (128 lanes): 256 columns as the one-CTA kernel's; two accumulators of 192 and the scales fit without overlap
  static constexpr int kAccStride = BLOCK_N == 256 ? TileCfg<FMT, 256>::kAccStride : BLOCK_N;
  static constexpr int kAccBars = BLOCK_N == 256 ? 1 : 2;  // full and empty barriers: one pair for both accumulators, or one each
  static constexpr int kTmemSfSet = kST * 12;              // the A scales and those of two 128-row tiles of B
  static constexpr int kTmemSfa = kAccStride + BLOCK_N, kTmemSfb = kTmemSfa + kST * 4;
  static_assert(kTmemSfa + 2 * kTmemSfSet <= 512, "tensor memory budget");
  static constexpr int kSmemBytes = kStages * kStageBytes + kOutStageBytes + kBarrierBytes + 1024;
};

// TURNS: each load warp loads all of every second stage, instead of warp 0 the operands and warp 6 the scales of every stage (see pair_turns).
template <int FMT, int EPI, int BLOCK_N, bool TURNS>
__global__ void __launch_bounds__(kGemmThreads, 1) gemm_blockscaled_pair_kernel(const __grid_constant__ CUtensorMap tma_a,
                                                                                 const __grid_constant__ CUtensorMap tma_b,
                                                                                 const __grid_constant__ CUtensorMap tma_sfa,
                                                                                 const __grid_constant__ CUtensorMap tma_sfb,
                                                                                 const __grid_constant__ CUtensorMap tma_out, const GemmParams p) {
  static_assert(EPI != TF_EPI_SILU_GATE || BLOCK_N == 256, "the SiLU-gate epilogue pairs a 128-column gate tile with its up tile");
  using PC = PairCfg<FMT, BLOCK_N>;
  constexpr int kStages = PC::kStages;
  constexpr int kST = PC::kST;
  constexpr int kNB = 2;
  constexpr int kOutCols = (EPI == TF_EPI_SILU_GATE) ? BLOCK_N / 2 : BLOCK_N;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_a = smem_base;
  const uint32_t smem_b = smem_a + kStages * kAStageBytes;
  const uint32_t smem_out = smem_b + kStages * PC::kBHalfBytes;  // 1024-byte aligned like the operand stages (the store's swizzle atom)
  const uint32_t smem_sfa = smem_out + PC::kOutStageBytes;
  const uint32_t smem_sfb = smem_sfa + kStages * PC::kSfaStageBytes;
  const uint32_t bars = smem_sfb + kStages * PC::kSfbStageBytes;
  const uint32_t bar_full = bars, bar_empty = bars + 8 * kStages, bar_tmem_full = bars + 16 * kStages,
                 bar_tmem_empty = bar_tmem_full + 8 * PC::kAccBars;
  const uint32_t tmem_slot = bar_tmem_empty + 8 * PC::kAccBars;
  const uint32_t abort_slot = tmem_slot + 4;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - smem_base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + (abort_slot - smem_base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  griddep_launch_dependents();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full + 8 * s, TURNS ? 2 : 4);  // an arrive.expect_tx of each load warp that serves the stage, from both CTAs (used in the leader only)
      mbar_init(bar_empty + 8 * s, 1);  // the leader's commit arrives in both CTAs
    }
    for (int i = 0; i < PC::kAccBars; ++i) {
      mbar_init(bar_tmem_full + 8 * i, 1);
      mbar_init(bar_tmem_empty + 8 * i, 16);  // 8 epilogue warps of each CTA (used in the leader only)
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // the same warp of both CTAs allocates the pair's tensor memory
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are initialised before anything crosses
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  griddep_wait();

  if (warp == 0 || warp == 6) {
    // ---------------- load warps (each CTA loads its own halves; completion is counted on the leader's barrier) ----------------
    // Role 0 loads the A rows, role 1 the B rows of this CTA, role 2 the A scales, roles 3-4 the scales of the two B halves: lanes 0-4 of both
    // warps with TURNS, else lanes 0-1 of warp 0 and 0-2 of warp 6 (on lanes 2-4 the scales came 1 to 2 % later for short K: mxfp8
    // 6933 x 128 x 736 + gate 9.03 -> 9.17 us). The scales go through tensor maps too ([tiles, 512 bytes] as 128 x u32 rows; a box is
    // always kST tiles, rows past the end read as zero), because only the tensor form of the copy may signal the peer's barrier.
    constexpr int kStep = TURNS ? 2 : 1;
    const int turn = TURNS && warp == 6 ? 1 : 0;
    const int role = TURNS || warp == 0 ? lane : lane + 2;
    const bool sf = role >= 2;
    const int half = role < 2 ? (int)rank : (role == 4 ? 1 : 0);  // the B half of a role that serves B
    const bool serves_a = role == 0 || role == 2;
    const CUtensorMap* my_map = role == 0 ? &tma_a : role == 1 ? &tma_b : role == 2 ? &tma_sfa : &tma_sfb;
    const uint32_t my_dst = role == 0 ? smem_a : role == 1 ? smem_b : role == 2 ? smem_sfa : smem_sfb + (uint32_t)half * kST * 512;
    const uint32_t my_stage_bytes = role == 0 ? kAStageBytes : role == 1 ? PC::kBHalfBytes : role == 2 ? PC::kSfaStageBytes : PC::kSfbStageBytes;
    int stage = turn, ks0 = turn;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = pair; tile < p.num_tiles && ok; tile += num_pairs) {
      const int m_blk = tile % p.m_blocks, n_blk = tile / p.m_blocks;
      const int a_row = m_blk * 256 + (int)rank * 128;
      // first B row of the lane's half, or (scales) of its 128-row tile: a 192-column tile starts in the middle of one or at its edge
      const int b_row = (EPI == TF_EPI_SILU_GATE) ? half * p.n + n_blk * 128
                        : BLOCK_N == 256 || !sf   ? n_blk * BLOCK_N + half * (BLOCK_N / 2)
                                                  : ((n_blk * BLOCK_N) & ~127) + half * 128;
      const int my_row = serves_a ? a_row : b_row;
      const bool mine = role < (TURNS || warp == 6 ? 5 : 2) && (serves_a ? a_row < p.m : b_row < p.n_rows_b);
      const uint32_t copies = __ballot_sync(0xFFFFFFFFu, mine) << (TURNS || warp == 0 ? 0 : 2);  // a bit per role
      const uint32_t tx = (copies & 1u) * kAStageBytes + (copies >> 1 & 1u) * PC::kBHalfBytes + (uint32_t)__popc(copies >> 2) * (kST * 512u);
      const int y_base = sf ? (my_row >> 7) * p.sf_col_tiles : my_row;
      int ks = ks0;
      for (; ks < p.num_k_stages; ks += kStep) {
        ok = mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, 1);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        const uint32_t full = mapa_shared(bar_full + 8 * stage, 0);  // the leader's barrier
        if (lane == 0) mbar_expect_tx_cluster(full, tx);
        __syncwarp();
        if (mine) tma_load_2d_pair(my_dst + stage * my_stage_bytes, my_map, sf ? 0 : ks * kStageKBytes, sf ? y_base + ks * kST : y_base, full);
        __syncwarp();
        stage += kStep;
        if (stage >= kStages) {
          stage -= kStages;
          phase ^= 1;
        }
      }
      ks0 = ks - p.num_k_stages;
    }
    if (!ok && lane == 0) {
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (rank == 0) {
      constexpr uint32_t idesc_base = (FmtTraits<FMT>::kElemFormat << 7) | (FmtTraits<FMT>::kElemFormat << 10) | ((uint32_t)(BLOCK_N >> 3) << 17) |
                                      (FmtTraits<FMT>::kScaleIsE8 << 23) | ((uint32_t)(256 >> 4) << 24);
      constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
      constexpr uint32_t kDescHiSf = (128u >> 4) | (1u << 14);
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0, tile_phase = 0, sf_buf = 0, acc_buf = 0;
      bool ok = true;
      for (int tile = pair; tile < p.num_tiles && ok; tile += num_pairs) {
        const uint32_t acc_bar = PC::kAccBars == 1 ? 0u : 8 * acc_buf;
        ok = mbar_wait(bar_tmem_empty + acc_bar, tile_phase ^ 1, abort_flag, 2);
        ok = __all_sync(0xFFFFFFFFu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t tmem_acc = tmem_base + acc_buf * PC::kAccStride;
        const uint32_t sfb_shift = BLOCK_N == 256 ? 0u : (uint32_t)(tile / p.m_blocks & 1) * 2u;  // odd 192-column tiles start 64 rows into their scales
        for (int ks = 0; ks < p.num_k_stages; ++ks) {
          ok = mbar_wait(bar_full + 8 * stage, phase, abort_flag, 3);
          ok = __all_sync(0xFFFFFFFFu, ok);
          if (!ok) break;
          tc_fence_after();
          const uint32_t tmem_sfa = tmem_base + PC::kTmemSfa + sf_buf * PC::kTmemSfSet;
          const uint32_t tmem_sfb = tmem_base + PC::kTmemSfb + sf_buf * PC::kTmemSfSet;
          sf_buf ^= 1;
          const uint32_t sfa_lo = ((smem_sfa + stage * PC::kSfaStageBytes) & 0x3FFFFu) >> 4;
          const uint32_t sfb_lo = ((smem_sfb + stage * PC::kSfbStageBytes) & 0x3FFFFu) >> 4;
          const uint32_t a_lo = (((smem_a + stage * kAStageBytes) & 0x3FFFFu) >> 4) | (1u << 16);
          const uint32_t b_lo = (((smem_b + stage * PC::kBHalfBytes) & 0x3FFFFu) >> 4) | (1u << 16);
          const int sf_left = p.sf_col_tiles - ks * kST;
          const int k_left = p.k_bytes - ks * kStageKBytes;
          const uint32_t first = ks > 0 ? 1u : 0u;
          if (elected) {
            if (sf_left >= kST && k_left >= kStageKBytes) {
#pragma unroll
              for (int t = 0; t < kST; ++t) {
                tc_cp_sf_pair(tmem_sfa + t * 4, make_desc(sfa_lo + t * 32, kDescHiSf));
#pragma unroll
                for (int nb = 0; nb < kNB; ++nb) tc_cp_sf_pair(tmem_sfb + (t * kNB + nb) * 4, make_desc(sfb_lo + (nb * kST + t) * 32, kDescHiSf));
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int t = (FMT == TF_FMT_MXFP8) ? 0 : (FMT == TF_FMT_MXFP4) ? (j >> 1) : j;
                const uint32_t sf_id = (FMT == TF_FMT_MXFP8) ? (uint32_t)j : (FMT == TF_FMT_MXFP4) ? (uint32_t)((j & 1) * 2) : 0u;
                tc_mma_pair<FMT>(tmem_acc, make_desc(a_lo + j * 2, kDescHiSw128), make_desc(b_lo + j * 2, kDescHiSw128),
                                 idesc_base | (sf_id << 4) | (sf_id << 29), tmem_sfa + t * 4, tmem_sfb + t * kNB * 4 + sfb_shift, j > 0 ? 1u : first);
              }
            } else {  // last, ragged stage: fewer scale tiles, fewer MMAs
              const int sf_tiles = sf_left > kST ? kST : sf_left;
              for (int t = 0; t < sf_tiles; ++t) {
                tc_cp_sf_pair(tmem_sfa + t * 4, make_desc(sfa_lo + t * 32, kDescHiSf));
#pragma unroll
                for (int nb = 0; nb < kNB; ++nb) tc_cp_sf_pair(tmem_sfb + (t * kNB + nb) * 4, make_desc(sfb_lo + (nb * kST + t) * 32, kDescHiSf));
              }
              const int n_mma = k_left >= kStageKBytes ? 4 : (k_left + 31) >> 5;
              for (int j = 0; j < n_mma; ++j) {
                const int t = (FMT == TF_FMT_MXFP8) ? 0 : (FMT == TF_FMT_MXFP4) ? (j >> 1) : j;
                const uint32_t sf_id = (FMT == TF_FMT_MXFP8) ? (uint32_t)j : (FMT == TF_FMT_MXFP4) ? (uint32_t)((j & 1) * 2) : 0u;
                tc_mma_pair<FMT>(tmem_acc, make_desc(a_lo + j * 2, kDescHiSw128), make_desc(b_lo + j * 2, kDescHiSw128),
                                 idesc_base | (sf_id << 4) | (sf_id << 29), tmem_sfa + t * 4, tmem_sfb + t * kNB * 4 + sfb_shift, j > 0 ? 1u : first);
              }
            }
            tc_commit_pair(bar_empty + 8 * stage);  // frees the stage in both CTAs
          }
          __syncwarp();
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (elected) tc_commit_pair(bar_tmem_full + acc_bar);  // both CTAs' epilogues may read their accumulator halves
        __syncwarp();
        if (PC::kAccBars == 1 || acc_buf) tile_phase ^= 1;
        acc_buf ^= 1;
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: each CTA drains its own 128 rows; the release goes to the leader's barrier ----------------
    const int q = warp & 3;
    const int grp = warp >= 7 ? 1 : 0;
    const float alpha = (FMT == TF_FMT_NVFP4) ? __fmul_rn(load_f32(p.a_gs), load_f32(p.b_gs)) : 1.0f;
    const uint32_t release = mapa_shared(bar_tmem_empty, 0);
    const uint32_t stage_smem = smem_out + (uint32_t)(grp * 4 + q) * PC::kOutBoxBytes;
    uint32_t tile_phase = 0, acc_buf = 0;
    uint32_t amax2 = 0;
    if (FMT != TF_FMT_NVFP4 && p.q_codes && p.q_pad)
      zero_scale_padding(p.q_scales, p.m, p.n >> 5, (int64_t)blockIdx.x * 256 + (grp * 4 + q) * 32 + lane, (int64_t)gridDim.x * 256);
    for (int tile = pair; tile < p.num_tiles; tile += num_pairs) {
      const int m_blk = tile % p.m_blocks, n_blk = tile / p.m_blocks;
      const uint32_t acc_bar = PC::kAccBars == 1 ? 0u : 8 * acc_buf;
      bool ok = mbar_wait(bar_tmem_full + acc_bar, tile_phase, abort_flag, 4);
      ok = __all_sync(0xFFFFFFFFu, ok);
      if (!ok) break;
      tc_fence_after();
      const int row = m_blk * 256 + (int)rank * 128 + q * 32 + lane;
      const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16);
      const int col0 = n_blk * kOutCols;
      const float alpha_t = (FMT == TF_FMT_NVFP4 && p.a_gs_rows > 0) ? __fmul_rn(load_f32(p.a_gs + min(row, p.m - 1) / p.a_gs_rows), load_f32(p.b_gs)) : alpha;
      const uint32_t t_acc = t_row + acc_buf * PC::kAccStride;
      if (BLOCK_N == 192) {  // three pairs: a group takes one and two of them in turn
        const int first = grp == 0 ? 0 : acc_buf == 0 ? 2 : 1, count = (int)acc_buf == grp ? 2 : 1;
        epilogue_pairs<FMT, EPI>(p, t_acc, first * 2, 2, count, count - 1, release + acc_bar, lane, row, col0, alpha_t, amax2, &tma_out, stage_smem);
      } else if (EPI == TF_EPI_RESIDUAL) {
        epilogue_pairs<FMT, EPI>(p, t_acc, grp * 2 + (acc_buf == 0 ? 4 : 0), acc_buf == 0 ? -4 : 4, 2, 0, release, lane, row, col0, alpha_t, amax2, &tma_out, stage_smem);
      } else if (acc_buf == 0) {
        if (grp == 0) epilogue_tile<FMT, 256, EPI, 0, 0, true>(p, t_row, release, lane, row, col0, alpha_t, amax2, &tma_out, stage_smem);
        else epilogue_tile<FMT, 256, EPI, 0, 1, true>(p, t_row, release, lane, row, col0, alpha_t, amax2, &tma_out, stage_smem);
      } else {
        if (grp == 0) epilogue_tile<FMT, 256, EPI, 1, 0, true>(p, t_acc, release, lane, row, col0, alpha_t, amax2, &tma_out, stage_smem);
        else epilogue_tile<FMT, 256, EPI, 1, 1, true>(p, t_acc, release, lane, row, col0, alpha_t, amax2, &tma_out, stage_smem);
      }
      if (PC::kAccBars == 1 || acc_buf) tile_phase ^= 1;
      acc_buf ^= 1;
    }
    if (lane == 0) bulk_wait_all();  // the stores have read their boxes and are written
    __syncwarp();
    if (p.out_amax) {
      uint32_t mx = max(amax2 & 0xFFFFu, amax2 >> 16);
      for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
      if (lane == 0 && mx) atomicMax(p.out_amax, mx << 16);
    }
  }

  // ---------------- teardown: nobody leaves while the peer may still touch this CTA's shared or tensor memory ----------------
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// ---- host side -------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// A [rows, k_bytes] byte matrix, boxes of 128 rows x 128 bytes, 128-byte swizzle, out-of-range bytes read as zero.
static tf_status make_operand_map(CUtensorMap* map, const void* base, int64_t rows, int64_t k_bytes, int box_rows = 128) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(TF_ERR_CUDA, "tf_gemm_blockscaled: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {(cuuint64_t)k_bytes, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)k_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)kStageKBytes, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TF_ERR_CUDA, "tf_gemm_blockscaled: cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return TF_OK;
}

// SMs the persistent GEMM leaves free (for a collective running beside it in another stream).
static std::atomic<int> g_sm_margin{0};  // process-wide (tf_set_sm_margin); atomic so that a concurrent reader sees the old or the new value
int sm_margin() { return g_sm_margin.load(std::memory_order_relaxed); }
static int gemm_sms() {
  const int n = sm_count() - sm_margin();
  return n < 2 ? 2 : n;
}

// Split-K plan of a problem: how many K ranges each output tile is cut into, so that small-M problems (few tiles, long K: the
// weight-streaming regime) still occupy every SM. Depends only on the sizes and the SM count: the workspace query and the launch
// agree by construction.
struct SplitPlan {
  int block_n, splits, k_stages_per_split;
};

// Small M (at most two row blocks): the GEMM streams the weights once and is bound by how evenly that stream is spread over
// the SMs. Measured on B200: one CTA's TMA pipeline draws about one 128-byte row segment per 4 clocks from HBM (about
// 60 GB/s), so the time of a launch is the largest number of row segments any CTA fetches. The plan minimises
//   waves * (K stages per unit + 3 stages of fill and drain) * (rows of B + rows of A per stage)  +  cost of the reduction pass
// over tile width {256, 128} and 1..16 K ranges, in units of one row segment (about 2.4 ns).
static SplitPlan split_plan(int64_t m, int64_t n, int64_t k_bytes, int epilogue) {
  SplitPlan sp;
  const int sms = sm_count();
  const int64_t m_blocks = (m + kBlockM - 1) / kBlockM;
  const int64_t n_acc = epilogue == TF_EPI_SILU_GATE ? 2 * n : n;
  const int64_t stages = (k_bytes + kStageKBytes - 1) / kStageKBytes;
  sp.block_n = 256;
  sp.splits = 1;
  sp.k_stages_per_split = (int)stages;
  if (n <= 128 && epilogue != TF_EPI_SILU_GATE) sp.block_n = 128;
  if (m > 256) return sp;
  const int64_t a_rows = m < kBlockM ? m : kBlockM;
  double best = 1e30;
  for (int bn = 256; bn >= 128; bn -= 128) {
    const int64_t tiles = m_blocks * ((n_acc + bn - 1) / bn);
    for (int64_t want = 1; want <= 16; ++want) {
      if (want > 1 && stages / want < 4) break;  // a K range shorter than the pipeline is all fill and drain
      const int64_t kps = (stages + want - 1) / want;
      const int64_t splits = (stages + kps - 1) / kps;
      if (bn == 128 && splits == 1 && epilogue == TF_EPI_SILU_GATE) continue;  // the fused SiLU gate pairs two 128-column halves
      const int64_t units = tiles * splits;
      const int64_t waves = (units + sms - 1) / sms;
      double cost = (double)waves * (double)(kps + 3) * (double)(bn + a_rows);
      if (splits > 1) cost += 1200.0 + 2.0 * (double)splits * (double)m * (double)n_acc * 4.0 / 7200.0;
      if (cost < best) {
        best = cost;
        sp.block_n = bn;
        sp.splits = (int)splits;
        sp.k_stages_per_split = (int)kps;
      }
    }
  }
  return sp;
}

template <int FMT, int BLOCK_N, int EPI, int SPLITK, bool BOXES = false>
static tf_status launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, GemmParams p, cudaStream_t stream) {
  using Cfg = TileCfg<FMT, BLOCK_N>;
  auto kernel = gemm_blockscaled_kernel<FMT, BLOCK_N, EPI, SPLITK, BOXES>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  TF_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    configured_dev = dev;
  }
  constexpr int out_cols = (EPI == TF_EPI_SILU_GATE) ? BLOCK_N / 2 : BLOCK_N;
  p.n_blocks = (p.n + out_cols - 1) / out_cols;
  p.num_tiles = p.m_blocks * p.n_blocks * p.splits;
  const int grid = SPLITK == kSplitCluster || p.num_tiles < gemm_sms() ? p.num_tiles : gemm_sms();
  const bool dependent = dependent_launch(chain_gemm_launch(p.m, p.num_tiles <= grid, GemmKind::kOneCta));
  if (dependent && p.m <= kBlockM) p.early_stages = kEarlyStages;
  if (SPLITK == kSplitCluster) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 2 : 1;
    TF_CUDA(cudaLaunchKernelEx(&cfg, kernel, ta, tb, p));
    return TF_OK;
  }
  TF_CUDA(launch_dependent(dependent, kernel, dim3(grid), dim3(kGemmThreads), (size_t)Cfg::kSmemBytes, stream, ta, tb, p));
  return TF_OK;
}

// The swizzled scale buffer as a [tiles, 128 x u32] matrix: a box is kST consecutive 512-byte tiles, no swizzle.
static tf_status make_scale_map(CUtensorMap* map, const void* base, int64_t tiles, int box_tiles) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(TF_ERR_CUDA, "tf_gemm_blockscaled: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {128u, (cuuint64_t)tiles};
  const cuuint64_t strides[1] = {512u};
  const cuuint32_t box[2] = {128u, (cuuint32_t)box_tiles};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TF_ERR_CUDA, "tf_gemm_blockscaled: cuTensorMapEncodeTiled (scales) failed with CUresult %d", (int)r);
  return TF_OK;
}

// The bf16 output as [m, n] with leading dimension ldo: boxes of 32 rows x 64 columns (128 bytes), 128-byte swizzle.
static tf_status make_output_map(CUtensorMap* map, const GemmParams& p) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(TF_ERR_CUDA, "tf_gemm_blockscaled: cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {(cuuint64_t)p.n, (cuuint64_t)p.m};
  const cuuint64_t strides[1] = {(cuuint64_t)p.ldo * 2u};
  const cuuint32_t box[2] = {64u, 32u};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.out, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(TF_ERR_CUDA, "tf_gemm_blockscaled: cuTensorMapEncodeTiled (output) failed with CUresult %d", (int)r);
  return TF_OK;
}

template <int FMT, int EPI, int BLOCK_N, bool TURNS = false>
static tf_status launch_gemm_pair(const CUtensorMap& ta, const CUtensorMap& tb, GemmParams p, cudaStream_t stream) {
  using PC = PairCfg<FMT, BLOCK_N>;
  CUtensorMap tsa, tsb, to = {};
  if (p.out) {
    const tf_status so = make_output_map(&to, p);
    if (so != TF_OK) return so;
  }
  tf_status st = make_scale_map(&tsa, p.sfa, (int64_t)((p.m + 127) / 128) * p.sf_col_tiles, PC::kST);
  if (st != TF_OK) return st;
  st = make_scale_map(&tsb, p.sfb, (int64_t)p.sfb_row_tiles * p.sf_col_tiles, PC::kST);
  if (st != TF_OK) return st;
  auto kernel = gemm_blockscaled_pair_kernel<FMT, EPI, BLOCK_N, TURNS>;
  static thread_local int configured_dev = -1;
  int dev = 0;
  TF_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PC::kSmemBytes));
    configured_dev = dev;
  }
  constexpr int out_cols = (EPI == TF_EPI_SILU_GATE) ? 128 : BLOCK_N;
  p.m_blocks = (p.m + 255) / 256;
  p.n_blocks = (p.n + out_cols - 1) / out_cols;
  p.num_tiles = p.m_blocks * p.n_blocks;
  int pairs = gemm_sms() / 2;
  if (p.num_tiles < pairs) pairs = p.num_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = PC::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent_launch(chain_gemm_launch(p.m, p.num_tiles <= pairs, EPI == TF_EPI_SILU_GATE ? GemmKind::kGatedPair : GemmKind::kPair)) ? 2 : 1;
  TF_CUDA(cudaLaunchKernelEx(&cfg, kernel, ta, tb, tsa, tsb, to, p));
  return TF_OK;
}

// How one call is launched: the form of the split along K (kSplit...), the tile width, the K ranges and the stages of each.
struct LaunchPlan {
  int form, block_n, splits, k_stages_per_split;
};

static int two_cta_forced() {
  static const int forced = getenv("TF_GEMM_TWO_CTA") ? atoi(getenv("TF_GEMM_TWO_CTA")) : -1;
  return forced;
}

// Whether the 2-CTA kernel serves this problem (TF_GEMM_TWO_CTA in the environment: 0 never, 1 wherever it can, unset this rule).
// Per wave of tiles the pair is 6-9 % faster than the one-CTA kernel (B200 after a second of load, one-CTA -> pair: nvfp4 4096 x 8192 x 28672
// 434 -> 400 us, 4096 x 28672 x 8192 + gate 836 -> 779, 4096 x 6144 x 2560 41.2 -> 37.9; mxfp8 8192 x 6144 x 2560 125.4 -> 117.7; problems of one wave 0-8 %,
// 14 of 15, mxfp8 512 x 3072 x 2560 + gate 14.1 -> 14.5), but its row blocks are 256 high: it is left where that costs a tenth more waves.
// Beside a margin it is left too: a pair needs two SMs of one TPC, and the kernel that the margin is for need not leave them whole. CTAs
// of 200 KB that start beside a quantizer split 4 to 12 pairs; with 16 pairs split, nvfp4 2048 x 14336 x 8192 + gate takes 303 us on pairs and 199 on
// single CTAs at margin 16 (342 and 217 at 32), since tiles are dealt out statically. With none split it is 184 and 203.
static bool use_pair_kernel(int64_t m, int64_t n, int epilogue, const LaunchPlan& lp) {
  const int forced = two_cta_forced();
  const bool gate = epilogue == TF_EPI_SILU_GATE;
  if (forced == 0 || lp.form != kSplitNone || lp.block_n != 256 || m <= kBlockM || (gate ? 2 * n : n) < 256) return false;
  if (forced == 1) return true;
  if (sm_margin() > 0) return false;
  const int64_t sms = sm_count(), pairs = sms / 2, n_blocks = gate ? (n + 127) / 128 : (n + 255) / 256;
  const int64_t waves = ((m + kBlockM - 1) / kBlockM * n_blocks + sms - 1) / sms, pair_waves = ((m + 255) / 256 * n_blocks + pairs - 1) / pairs;
  return 10 * pair_waves <= 11 * waves;
}

// The tile width of a pair. 192 columns take 0.79 of the time of 256 per K stage, not 0.75 (shared memory: 256 rows of operands are read for fewer
// columns), and lose 5 to 9 % over many waves (mxfp8 8192 x 6144 x 2560 96 -> 101 us), but fill a wave that 256 leave part empty: one wave either way
// mxfp8 512 x 6144 x 2560 13.4 -> 12.3, mxfp4 1000 x 3000 x 2720 residual 15.3 -> 14.3; six waves or seven nvfp4 4096 x 6144 x 2560 33.8 -> 33.8. Microseconds
// fitted to those; the gate pairs 128 + 128 columns.
static int pair_width(int64_t m, int64_t n, int64_t stages, int epilogue) {
  if (epilogue == TF_EPI_SILU_GATE) return 256;
  const int64_t pairs = gemm_sms() / 2, m_blocks = (m + 255) / 256;
  auto waves = [&](int64_t bn) { return (double)((m_blocks * ((n + bn - 1) / bn) + pairs - 1) / pairs); };
  return waves(192) * (0.33 * (double)stages + 0.95) < 0.97 * waves(256) * (0.414 * (double)stages + 0.85) ? 192 : 256;
}

// Whether the load warps of a gated pair take the stages in turn. The gate's arithmetic, which runs beside the next tile's stages, competes with them for
// issue slots: in turn they have two stages' time for five copies instead of one for two or three. It needs a next tile, and a tile's first
// stage comes later for it. Split by kind -> in turn, cold, us: mxfp8 8192 x 3072 with K 512 / 1024 / 1536 / 2560 / 4096 60.2 / 65.4 / 69.1 / 98.2 / 145.1
// -> 60.7 / 65.6 / 68.9 / 96.0 / 142.7; mxfp4 4096 x 4096 with K 1024 / 3072 / 5120 / 8192 38.7 / 47.4 / 66.9 / 96.1 -> 39.3 / 48.1 / 65.4 / 94.1; nvfp4 2048 x
// 8192 with K 2048 / 5120 42.7 / 67.9 -> 43.3 / 66.8; one tile per pair mxfp8 1024 x 2304 x 2560 14.7 -> 14.9, 512 x 3072 x 2560 14.3 -> 14.6. Without
// the gate it costs (mxfp4 300 x 8192 x 4096 12.3 -> 12.55, mxfp8 1024 x 4096 x 4096 residual 22.0 -> 22.65).
static bool pair_turns(const GemmParams& p) {
  const int64_t tiles = (int64_t)((p.m + 255) / 256) * ((p.n + 127) / 128);
  return p.num_k_stages >= 16 && tiles > gemm_sms() / 2;
}

// How many clusters of `splits` GEMM CTAs (one CTA fills an SM) the current device runs at once: a cluster lives inside one GPC, so
// this is less than SMs / splits (measured on B200: 47 clusters of 3 or fewer, where 48 would need 144 of the 148 SMs).
static int cluster_capacity(int splits) {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices][kMaxClusterSplits + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  return ask_once(cached[dev][splits], [splits]() -> int {
    using Cfg = TileCfg<TF_FMT_MXFP8, 128>;
    auto kernel = gemm_blockscaled_kernel<TF_FMT_MXFP8, 128, TF_EPI_NONE, kSplitCluster>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)splits);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return -1;
    }
    return n;
  });
}

// The launch plan: `sp` as it stands, or 128-column tiles, or (kSplitCluster) each tile cut over a cluster of CTAs, whichever the model
// below says is shortest. Microseconds beyond a launch's fixed 4.4, fitted to B200 measurements of graphs of 24 launches:
//   a K stage takes 0.235 with 128-column tiles and 0.38 with 256 (bound by shared-memory reads and fills), a tile's epilogue 0.5 / 1.0;
//   planes and a reduction launch 2.0 + 8 bytes per partial sum at 3 TB/s; a cluster 1.6 + its remote reads at 26.6 GB/s per SM.
// One form for all -> the plan: mxfp8 512 x 2560 x 3072 13.7 -> 10.9 us (128-column tiles), 128 x 2560 x 3072 12.3 -> 9.8 (4 ranges), 1 x 2560 x 3072
// 7.8 -> 5.9 (6), 700 x 1024 x 16384 51.6 -> 23.8 (2), mxfp4 300 x 1024 x 8192 residual 27.7 -> 12.7 (5).
// A problem with a planes plan keeps that plan's K ranges in every form, so that its result is the sum of the planes bit for bit.
// The plan is made for the whole device, whatever margin is set (tf_set_sm_margin): K ranges are part of a result, so they may not depend on
// it. Beside a margin a cluster launch takes the SMs it was planned for; the tile width, which no sum depends on, follows the free SMs.
// The SiLU gate pairs 128 + 128 columns, so its tiles stay 256 wide; with planes available (m <= 256) those measured faster (9.2 against
// 9.5 us at 1 x 3072 x 2560), so a cluster takes it only above that.
static LaunchPlan launch_plan(int64_t m, int64_t n, int64_t k_bytes, int epilogue, const SplitPlan& sp) {
  LaunchPlan best = {sp.splits > 1 ? kSplitPlanes : kSplitNone, sp.block_n, sp.splits, sp.k_stages_per_split};
  if (two_cta_forced() == 1) return best;
  const bool gate = epilogue == TF_EPI_SILU_GATE;
  const int64_t sms = sm_count(), m_blocks = (m + kBlockM - 1) / kBlockM, n_acc = gate ? 2 * n : n;
  const int64_t stages = (k_bytes + kStageKBytes - 1) / kStageKBytes, rows = m < kBlockM ? m : kBlockM;
  auto tiles = [&](int bn) { return m_blocks * ((n_acc + bn - 1) / bn); };
  auto stage_us = [](int bn) { return bn == 128 ? 0.235 : 0.38; };
  auto tile_us = [&](int bn, int64_t kps) { return (double)kps * stage_us(bn) + (bn == 128 ? 0.5 : 1.0); };
  if (tiles(128) > 2 * sms) return best;  // at least one full wave of 256-column tiles
  double cost = (double)((tiles(sp.block_n) * sp.splits + sms - 1) / sms) * tile_us(sp.block_n, sp.k_stages_per_split);
  if (sp.splits > 1) cost += 2.0 + (double)sp.splits * (double)m * (double)n_acc * 8.0 / 3.0e6;
  if (!gate && sp.splits == 1 && tiles(128) <= sms && tile_us(128, stages) < cost) {
    cost = tile_us(128, stages);
    best = {kSplitNone, 128, 1, (int)stages};
  }
  if (gate && m <= 256) return best;
  const int bn = gate ? 256 : 128;
  for (int64_t want = 2; want <= kMaxClusterSplits && stages / want >= 2; ++want) {
    const int64_t kps = (stages + want - 1) / want, splits = (stages + kps - 1) / kps;
    if (splits < 2 || tiles(bn) * splits > sms || tiles(bn) > cluster_capacity((int)splits)) continue;
    if (sp.splits > 1 && (splits != sp.splits || kps != sp.k_stages_per_split)) continue;  // the sums tf_gemm_blockscaled_partials leaves
    const double c = tile_us(bn, kps) + 1.6 + (double)rows * bn * 4.0 * (double)(splits - 1) / (double)splits / 26600.0;
    if (c < cost) {
      cost = c;
      best = {kSplitCluster, bn, (int)splits, (int)kps};
    }
  }
  if (best.form == kSplitNone && best.block_n != sp.block_n && tiles(best.block_n) > gemm_sms()) best.block_n = sp.block_n;
  return best;
}

template <int FMT>
static tf_status dispatch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, GemmParams p, int epilogue, const LaunchPlan& lp, int pair_n, cudaStream_t stream,
                               bool partials_only = false) {
  if (lp.form == kSplitCluster) {
    if (epilogue == TF_EPI_SILU_GATE) return launch_gemm<FMT, 256, TF_EPI_SILU_GATE, kSplitCluster>(ta, tb, p, stream);
    if (epilogue == TF_EPI_RESIDUAL) return launch_gemm<FMT, 128, TF_EPI_RESIDUAL, kSplitCluster>(ta, tb, p, stream);
    return launch_gemm<FMT, 128, TF_EPI_NONE, kSplitCluster>(ta, tb, p, stream);
  }
  if (lp.form == kSplitPlanes) {
    // first pass: plain accumulation over all accumulator columns into the workspace; second pass: reduce + epilogue
    const int n_out = p.n;
    float* residual = p.residual;
    unsigned int* amax = p.out_amax;
    p.n = p.n_rows_b;
    p.out_amax = nullptr;
    uint8_t* qc = p.q_codes;
    p.q_codes = nullptr;  // the quantized copy is produced by the second pass
    tf_status st = lp.block_n == 128 ? launch_gemm<FMT, 128, TF_EPI_NONE, kSplitPlanes>(ta, tb, p, stream) : launch_gemm<FMT, 256, TF_EPI_NONE, kSplitPlanes>(ta, tb, p, stream);
    if (st != TF_OK) return st;
    if (partials_only) return TF_OK;  // the caller's next kernel sums the planes (tf_gemm_blockscaled_partials)
    p.q_codes = qc;
    const int64_t total = (int64_t)p.m * (n_out >> 3);
    const int64_t need = (total + 255) / 256, cap = (int64_t)sm_count() * 8;
    unsigned grid = (unsigned)(need < cap ? need : cap);
    if (qc && p.q_pad && grid < kPadBlocks) grid = kPadBlocks;
    const float* ags = FMT == TF_FMT_NVFP4 ? p.a_gs : nullptr;
    const float* bgs = FMT == TF_FMT_NVFP4 ? p.b_gs : nullptr;
#define TF_REDUCE(EPI_, Q_) \
  launch_dependent(chain_rows_launch(p.m), splitk_reduce_kernel<EPI_, Q_>, dim3(grid), dim3(256), 0, stream, (const float*)p.ws, (int)lp.splits, (int)p.m, (int)n_out, (int)p.n_rows_b, ags, bgs, \
                   p.out, p.ldo, residual, amax, p.q_codes, p.q_scales, (int)p.q_pad, (int)p.a_gs_rows)
    const int qf = p.q_codes ? FMT : -1;
    if (epilogue == TF_EPI_SILU_GATE) {
      if (qf == TF_FMT_MXFP8) TF_REDUCE(TF_EPI_SILU_GATE, TF_FMT_MXFP8);
      else if (qf == TF_FMT_MXFP4) TF_REDUCE(TF_EPI_SILU_GATE, TF_FMT_MXFP4);
      else TF_REDUCE(TF_EPI_SILU_GATE, -1);
    } else if (epilogue == TF_EPI_RESIDUAL) {
      TF_REDUCE(TF_EPI_RESIDUAL, -1);
    } else {
      if (qf == TF_FMT_MXFP8) TF_REDUCE(TF_EPI_NONE, TF_FMT_MXFP8);
      else if (qf == TF_FMT_MXFP4) TF_REDUCE(TF_EPI_NONE, TF_FMT_MXFP4);
      else TF_REDUCE(TF_EPI_NONE, -1);
    }
#undef TF_REDUCE
    TF_LAUNCH_CHECK();
    return TF_OK;
  }
  if (pair_n == 192)
    return epilogue == TF_EPI_RESIDUAL ? launch_gemm_pair<FMT, TF_EPI_RESIDUAL, 192>(ta, tb, p, stream) : launch_gemm_pair<FMT, TF_EPI_NONE, 192>(ta, tb, p, stream);
  if (pair_n == 256) {
    if (epilogue == TF_EPI_SILU_GATE)
      return pair_turns(p) ? launch_gemm_pair<FMT, TF_EPI_SILU_GATE, 256, true>(ta, tb, p, stream) : launch_gemm_pair<FMT, TF_EPI_SILU_GATE, 256>(ta, tb, p, stream);
    if (epilogue == TF_EPI_RESIDUAL) return launch_gemm_pair<FMT, TF_EPI_RESIDUAL, 256>(ta, tb, p, stream);
    return launch_gemm_pair<FMT, TF_EPI_NONE, 256>(ta, tb, p, stream);
  }
  if (epilogue == TF_EPI_SILU_GATE) return launch_gemm<FMT, 256, TF_EPI_SILU_GATE, kSplitNone>(ta, tb, p, stream);
  if (epilogue == TF_EPI_RESIDUAL) {
    if (lp.block_n == 256) return launch_gemm<FMT, 256, TF_EPI_RESIDUAL, kSplitNone>(ta, tb, p, stream);
    // Up to 24 columns a staged row is 6 lanes of 16, and the ring keeps its stage: staged -> from the accumulator, mxfp8 33507 x 8 x 14112 129.7 -> 120.4 us,
    // x 24 84.7 -> 82.9, 64959 x 16 x 2048 42.3 -> 40.2, nvfp4 11355 x 8 x 1696 8.4 -> 7.8; at 32 columns 42.3 -> 43.9 and 8.7 -> 9.9.
    return p.n > 24 ? launch_gemm<FMT, 128, TF_EPI_RESIDUAL, kSplitNone, true>(ta, tb, p, stream) : launch_gemm<FMT, 128, TF_EPI_RESIDUAL, kSplitNone>(ta, tb, p, stream);
  }
  return lp.block_n == 256 ? launch_gemm<FMT, 256, TF_EPI_NONE, kSplitNone>(ta, tb, p, stream) : launch_gemm<FMT, 128, TF_EPI_NONE, kSplitNone>(ta, tb, p, stream);
}

// Scratch of tf_gemm_blockscaled_static: lives in the library's device image, one copy per GPU that loads the library,
// from load to process exit. Host code may not use this name as a pointer: it is a host-side stand-in for the symbol.
constexpr int64_t kStaticScratchBytes = 8ll << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

int* device_status_words() {
  constexpr int kMaxDevices = 64;
  static int* cached[kMaxDevices] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  if (!cached[dev]) {
    void* ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_device_status) != cudaSuccess) return nullptr;
    cached[dev] = static_cast<int*>(ptr);
  }
  return cached[dev];
}

}  // namespace tf

using namespace tf;

extern "C" {

tf_status tf_device_status(int32_t* status, int32_t* detail) {
  clear_error();
  TF_CHECK_ARG(status != nullptr, "%s: null pointer", __func__);
  int host[2] = {0, 0};
  TF_CUDA(cudaDeviceSynchronize());
  TF_CUDA(cudaMemcpyFromSymbol(host, g_device_status, sizeof(host)));
  if (host[0] != 0) {
    const int zero[2] = {0, 0};
    TF_CUDA(cudaMemcpyToSymbol(g_device_status, zero, sizeof(zero)));
  }
  *status = host[0];
  if (detail) *detail = host[1];
  return TF_OK;
}

tf_status tf_set_sm_margin(int32_t sms) {
  clear_error();
  TF_CHECK_ARG(sms >= 0 && sms <= 64, "%s: the margin must be in 0..64", __func__);
  g_sm_margin.store(sms, std::memory_order_relaxed);
  return TF_OK;
}

tf_status tf_selftest_bounded_wait(int32_t limit_ms, void* stream) {
  clear_error();
  TF_CHECK_ARG(limit_ms > 0 && limit_ms <= 2000, "%s: limit_ms must be in 1..2000", __func__);
  bounded_wait_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((unsigned long long)limit_ms * 1000000ull);
  TF_LAUNCH_CHECK();
  return TF_OK;
}

int64_t tf_gemm_workspace_bytes(int64_t m, int64_t n, int64_t k, int32_t format, int32_t epilogue) {
  if (m <= 0 || n <= 0 || k <= 0 || format < TF_FMT_MXFP8 || format > TF_FMT_NVFP4 || epilogue < TF_EPI_NONE || epilogue > TF_EPI_RESIDUAL) return 0;
  const int64_t k_bytes = format == TF_FMT_MXFP8 ? k : k / 2;
  const SplitPlan sp = split_plan(m, n, k_bytes, epilogue);
  if (sp.splits <= 1) return 0;
  const int64_t n_acc = epilogue == TF_EPI_SILU_GATE ? 2 * n : n;
  return (int64_t)sp.splits * m * n_acc * 4;
}

static tf_status static_scratch_address(void** out) {
  // The device address of g_static_scratch, looked up once per device (with that device current) and cached.
  constexpr int kMaxDevices = 64;
  static void* cached[kMaxDevices] = {nullptr};
  int dev = 0;
  TF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(TF_ERR_UNSUPPORTED, "tf_gemm_blockscaled_static: device ordinal %d is beyond %d", dev, kMaxDevices);
  if (!cached[dev]) {
    void* ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || !ptr)
      return fail(TF_ERR_CUDA, "tf_gemm_blockscaled_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
    cached[dev] = ptr;
  }
  *out = cached[dev];
  return TF_OK;
}

int32_t tf_gemm_splits(int64_t m, int64_t n, int64_t k, int32_t format, int32_t epilogue) {
  if (m <= 0 || n <= 0 || k <= 0 || format < TF_FMT_MXFP8 || format > TF_FMT_NVFP4 || epilogue < TF_EPI_NONE || epilogue > TF_EPI_RESIDUAL) return 0;
  return split_plan(m, n, format == TF_FMT_MXFP8 ? k : k / 2, epilogue).splits;
}

tf_status tf_gemm_launch_form(int64_t m, int64_t n, int64_t k, int32_t format, int32_t epilogue, int32_t* form) {
  clear_error();
  TF_CHECK_ARG(form != nullptr, "%s: null pointer", __func__);
  TF_CHECK_ARG(m > 0 && n > 0 && k > 0 && format >= TF_FMT_MXFP8 && format <= TF_FMT_NVFP4 && epilogue >= TF_EPI_NONE && epilogue <= TF_EPI_RESIDUAL,
               "%s: bad argument", __func__);
  const int64_t k_bytes = format == TF_FMT_MXFP8 ? k : k / 2;
  const LaunchPlan lp = launch_plan(m, n, k_bytes, epilogue, split_plan(m, n, k_bytes, epilogue));
  const bool gate = epilogue == TF_EPI_SILU_GATE;
  const int64_t n_acc = gate ? 2 * n : n;
  form[0] = use_pair_kernel(m, n, epilogue, lp) ? kFormPair : lp.form;
  form[1] = form[0] == kFormPair ? pair_width(m, n, (k_bytes + kStageKBytes - 1) / kStageKBytes, epilogue) : lp.block_n;
  form[2] = lp.splits;
  const bool pair = form[0] == kFormPair;
  const int64_t tiles = (m + (pair ? 255 : 127)) / (pair ? 256 : 128) * ((n_acc + form[1] - 1) / form[1]) * lp.splits;
  form[3] = dependent_launch(chain_gemm_launch(m, form[0] == kSplitCluster || tiles <= gemm_sms() / (pair ? 2 : 1),
                                               !pair ? GemmKind::kOneCta : gate ? GemmKind::kGatedPair : GemmKind::kPair));
  return TF_OK;
}

int64_t tf_gemm_static_scratch_bytes(void) { return kStaticScratchBytes; }

tf_status tf_gemm_blockscaled_static(const void* a_codes, const void* a_scales, const float* a_global_scale, const void* b_codes,
                                     const void* b_scales, const float* b_global_scale, void* out, int64_t ldo, int64_t m, int64_t n, int64_t k,
                                     int32_t format, int32_t epilogue, void* epilogue_arg, float* out_amax, void* stream) {
  clear_error();
  const int64_t need = tf_gemm_workspace_bytes(m, n, k, format, epilogue);
  if (need > kStaticScratchBytes)
    return fail(TF_ERR_WORKSPACE,
                "tf_gemm_blockscaled_static: this problem needs %lld bytes of scratch, the built-in scratch holds %lld; use tf_gemm_blockscaled "
                "with a caller-provided workspace",
                (long long)need, (long long)kStaticScratchBytes);
  void* scratch = nullptr;
  if (need > 0) {
    const tf_status st = static_scratch_address(&scratch);
    if (st != TF_OK) return st;
  }
  return tf_gemm_blockscaled(a_codes, a_scales, a_global_scale, b_codes, b_scales, b_global_scale, out, ldo, m, n, k, format, epilogue, epilogue_arg,
                             out_amax, nullptr, nullptr, 0, scratch, need > 0 ? kStaticScratchBytes : 0, stream);
}

}  // extern "C"

// The GEMM entry points. `scatter_ptrs` (null for tf_gemm_blockscaled): the destinations of the row blocks, see GemmParams.
// `partial_splits` (non-null for tf_gemm_blockscaled_partials): only the first pass of a split-K problem runs; receives the number of planes.
static tf_status gemm_entry(const char* fn, const void* a_codes, const void* a_scales, const float* a_global_scale, const void* b_codes,
                            const void* b_scales, const float* b_global_scale, void* out, int64_t ldo, int64_t m, int64_t n, int64_t k, int32_t format,
                            int32_t epilogue, void* epilogue_arg, float* out_amax, void* q_codes, void* q_scales, int64_t a_global_scale_rows,
                            void* workspace, int64_t workspace_bytes, const uint64_t* scatter_ptrs, int32_t owners, int64_t rows_per_owner,
                            void* stream_, int32_t* partial_splits = nullptr, bool check_only = false) {
  cudaStream_t stream = (cudaStream_t)stream_;
  TF_CHECK_ARG(format >= TF_FMT_MXFP8 && format <= TF_FMT_NVFP4, "%s: unknown format %d", fn, format);
  TF_CHECK_ARG(epilogue >= TF_EPI_NONE && epilogue <= TF_EPI_RESIDUAL, "%s: unknown epilogue %d", fn, epilogue);
  TF_CHECK_ARG(m >= 0 && n > 0 && k > 0, "%s: bad shape m=%lld n=%lld k=%lld", fn, (long long)m, (long long)n, (long long)k);
  if (m == 0) return TF_OK;
  TF_CHECK_ARG(a_codes && a_scales && b_codes && b_scales && (out || q_codes || partial_splits), "%s: null pointer", fn);
  TF_CHECK_ARG((q_codes == nullptr) == (q_scales == nullptr), "%s: q_codes and q_scales go together", fn);
  if (q_codes) {
    if (format == TF_FMT_NVFP4)
      return fail(TF_ERR_UNSUPPORTED, "%s: a quantized output needs the tensor's global scale first; nvfp4 outputs are quantized by tf_quantize_nvfp4_from_amax", fn);
    if (epilogue == TF_EPI_RESIDUAL) return fail(TF_ERR_UNSUPPORTED, "%s: the residual epilogue has no quantized output", fn);
    if (n % 32 != 0) return fail(TF_ERR_UNSUPPORTED, "%s: a quantized output needs n %% 32 == 0", fn);
    TF_CHECK_ALIGNED(q_codes, 16, "q_codes");
  }
  TF_CHECK_ARG(epilogue != TF_EPI_RESIDUAL || out, "%s: the residual epilogue needs out", fn);
  TF_CHECK_ARG(a_global_scale_rows >= 0 && a_global_scale_rows % 128 == 0, "%s: a_global_scale_rows must be 0 or a multiple of 128", fn);
  TF_CHECK_ARG(format != TF_FMT_NVFP4 || (a_global_scale && b_global_scale), "%s: nvfp4 needs both global scales", fn);
  TF_CHECK_ARG(epilogue != TF_EPI_RESIDUAL || epilogue_arg, "%s: the residual epilogue needs its f32 residual", fn);
  if (k % 32 != 0) return fail(TF_ERR_UNSUPPORTED, "%s: k=%lld is not a multiple of 32", fn, (long long)k);
  if (n % 8 != 0 || ldo % 8 != 0 || ldo < n) return fail(TF_ERR_ALIGNMENT, "%s: n and ldo must be multiples of 8 with ldo >= n", fn);
  if (epilogue == TF_EPI_SILU_GATE && n % 128 != 0) return fail(TF_ERR_UNSUPPORTED, "%s: the SiLU-gate epilogue needs n %% 128 == 0", fn);
  if (m > (1 << 30) || n > (1 << 30) || k > (1 << 30)) return fail(TF_ERR_UNSUPPORTED, "%s: a dimension exceeds 2^30", fn);
  TF_CHECK_ALIGNED(a_codes, 16, "a_codes");
  TF_CHECK_ALIGNED(b_codes, 16, "b_codes");
  TF_CHECK_ALIGNED(a_scales, 16, "a_scales");
  TF_CHECK_ALIGNED(b_scales, 16, "b_scales");
  if (out) TF_CHECK_ALIGNED(out, 16, "out");
  if (epilogue == TF_EPI_RESIDUAL) TF_CHECK_ALIGNED(epilogue_arg, 16, "residual");
  if (check_only) return TF_OK;  // tf_gemm_bf16, which has sized the workspace itself

  const int64_t k_bytes = (format == TF_FMT_MXFP8) ? k : k / 2;
  const int64_t n_rows_b = (epilogue == TF_EPI_SILU_GATE) ? 2 * n : n;
  const int64_t block = (format == TF_FMT_NVFP4) ? 16 : 32;
  CUtensorMap ta, tb;
  // M < 128: the A box covers only the rows that exist (in steps of 16), so every stage asks TMA for fewer row segments (measured:
  // 10 % on the M = 1 decode step). The rows of the shared-memory tile beyond the box are never written; they feed accumulator
  // rows that are never stored.
  const int a_box_rows = m >= kBlockM ? kBlockM : (int)((m + 15) / 16 * 16);
  tf_status st = make_operand_map(&ta, a_codes, m, k_bytes, a_box_rows);
  if (st != TF_OK) return st;

  GemmParams p;
  p.m = (int)m;
  p.n = (int)n;
  p.n_rows_b = (int)n_rows_b;
  p.k_bytes = (int)k_bytes;
  p.num_k_stages = (int)((k_bytes + kStageKBytes - 1) / kStageKBytes);
  p.sf_col_tiles = (int)((k / block + 3) / 4);
  p.m_blocks = (int)((m + kBlockM - 1) / kBlockM);
  p.n_blocks = 0;
  p.num_tiles = 0;
  p.sfb_row_tiles = (int)((n_rows_b + 127) / 128);
  p.sfa = static_cast<const uint8_t*>(a_scales);
  p.sfb = static_cast<const uint8_t*>(b_scales);
  p.a_gs = a_global_scale;
  p.b_gs = b_global_scale;
  p.out = static_cast<uint16_t*>(out);
  p.ldo = ldo;
  p.residual = static_cast<float*>(epilogue_arg);
  p.out_amax = reinterpret_cast<unsigned int*>(out_amax);
  p.q_codes = static_cast<uint8_t*>(q_codes);
  p.q_scales = static_cast<uint8_t*>(q_scales);
  p.q_pad = 0;
  p.a_gs_rows = (int)a_global_scale_rows;
  p.a_box_bytes = a_box_rows * kStageKBytes;
  p.early_stages = 0;
  p.scatter_rows = 0;
  for (int i = 0; i < 8; ++i) p.scatter_out[i] = nullptr;
  const SplitPlan sp = split_plan(m, n, k_bytes, epilogue);
  LaunchPlan lp = {kSplitPlanes, sp.block_n, sp.splits, sp.k_stages_per_split};
  if (!partial_splits) lp = launch_plan(m, n, k_bytes, epilogue, sp);
  if (scatter_ptrs) {
    if (sp.splits > 1)
      return fail(TF_ERR_UNSUPPORTED, "%s: this shape is split along K (tf_gemm_workspace_bytes > 0), which has no scattered output", fn);
    p.scatter_rows = (int)rows_per_owner;
    for (int i = 0; i < owners; ++i) p.scatter_out[i] = reinterpret_cast<uint16_t*>(scatter_ptrs[i]);
  }
  if (partial_splits) {
    if (sp.splits <= 1) return fail(TF_ERR_UNSUPPORTED, "%s: this shape is not split along K (tf_gemm_splits == 1): there are no partial sums to leave", fn);
    *partial_splits = sp.splits;
  }
  const int pair_n = !scatter_ptrs && !partial_splits && use_pair_kernel(m, n, epilogue, lp) ? pair_width(m, n, p.num_k_stages, epilogue) : 0;
  st = make_operand_map(&tb, b_codes, n_rows_b, k_bytes, pair_n == 192 ? 96 : kBlockM);
  if (st != TF_OK) return st;
  p.splits = lp.splits;
  p.k_stages_per_split = lp.k_stages_per_split;
  p.ws = static_cast<float*>(workspace);
  if (sp.splits > 1) {
    const int64_t need = (int64_t)sp.splits * m * n_rows_b * 4;
    if (!workspace || workspace_bytes < need)
      return fail(TF_ERR_WORKSPACE, "%s: this problem is split %d ways along K and needs a %lld-byte workspace (tf_gemm_workspace_bytes)", fn,
                  sp.splits, (long long)need);
    TF_CHECK_ALIGNED(workspace, 256, "workspace");
  }
  if (q_codes) {  // after every refusal: the unaligned case enqueues a memset
    st = scale_padding(q_scales, format, m, n, TF_SCALES_SWIZZLED, stream, &p.q_pad);
    if (st != TF_OK) return st;
  }
  switch (format) {
    case TF_FMT_MXFP8: return dispatch_gemm<TF_FMT_MXFP8>(ta, tb, p, epilogue, lp, pair_n, stream, partial_splits != nullptr);
    case TF_FMT_MXFP4: return dispatch_gemm<TF_FMT_MXFP4>(ta, tb, p, epilogue, lp, pair_n, stream, partial_splits != nullptr);
    default: return dispatch_gemm<TF_FMT_NVFP4>(ta, tb, p, epilogue, lp, pair_n, stream, partial_splits != nullptr);
  }
}

extern "C" {

tf_status tf_gemm_blockscaled(const void* a_codes, const void* a_scales, const float* a_global_scale, const void* b_codes, const void* b_scales,
                              const float* b_global_scale, void* out, int64_t ldo, int64_t m, int64_t n, int64_t k, int32_t format,
                              int32_t epilogue, void* epilogue_arg, float* out_amax, void* q_codes, void* q_scales,
                              int64_t a_global_scale_rows, void* workspace, int64_t workspace_bytes, void* stream) {
  clear_error();
  return gemm_entry(__func__, a_codes, a_scales, a_global_scale, b_codes, b_scales, b_global_scale, out, ldo, m, n, k, format, epilogue, epilogue_arg,
                    out_amax, q_codes, q_scales, a_global_scale_rows, workspace, workspace_bytes, nullptr, 0, 0, stream);
}

namespace {
// The scratch of tf_gemm_bf16: byte offsets of the quantized activation's parts and of the split-K workspace.
struct Bf16Scratch {
  int64_t scales, global_scale, partials, workspace, total;
};
Bf16Scratch bf16_scratch(int64_t m, int64_t n, int64_t k, int32_t format, int32_t epilogue) {
  auto align = [](int64_t b) { return (b + 255) / 256 * 256; };
  Bf16Scratch s;
  s.scales = align(m * (format == TF_FMT_MXFP8 ? k : k / 2));
  s.global_scale = s.scales + align(tf_scale_bytes(format, m, k, TF_SCALES_SWIZZLED));
  s.partials = s.global_scale + (format == TF_FMT_NVFP4 ? 256 : 0);
  s.workspace = s.partials + (format == TF_FMT_NVFP4 ? align(tf_quantize_nvfp4_dynamic_scratch_bytes()) : 0);
  s.total = s.workspace + tf_gemm_workspace_bytes(m, n, k, format, epilogue);
  return s;
}
}  // namespace

int64_t tf_gemm_bf16_scratch_bytes(int64_t m, int64_t n, int64_t k, int32_t format, int32_t epilogue) {
  if (m <= 0 || n <= 0 || k <= 0 || k % 32 || format < TF_FMT_MXFP8 || format > TF_FMT_NVFP4 || epilogue < TF_EPI_NONE || epilogue > TF_EPI_RESIDUAL) return 0;
  return bf16_scratch(m, n, k, format, epilogue).total;
}

tf_status tf_gemm_bf16(const void* x, int64_t ldx, const float* x_global_scale, const float* x_amax, const void* b_codes, const void* b_scales,
                       const float* b_global_scale, void* out, int64_t ldo, int64_t m, int64_t n, int64_t k, int32_t format, int32_t epilogue,
                       void* epilogue_arg, float* out_amax, void* scratch, int64_t scratch_bytes, void* stream) {
  clear_error();
  TF_CHECK_ARG(m >= 0 && n > 0 && k > 0 && format >= TF_FMT_MXFP8 && format <= TF_FMT_NVFP4 && epilogue >= TF_EPI_NONE && epilogue <= TF_EPI_RESIDUAL, "%s: bad argument", __func__);
  if (m == 0) return TF_OK;
  if (k % 32 != 0) return fail(TF_ERR_UNSUPPORTED, "%s: k=%lld is not a multiple of 32", __func__, (long long)k);
  TF_CHECK_ARG(!(x_global_scale && x_amax), "%s: x_global_scale and x_amax exclude each other", __func__);
  const Bf16Scratch at = bf16_scratch(m, n, k, format, epilogue);
  if (!scratch || scratch_bytes < at.total) return fail(TF_ERR_WORKSPACE, "%s: needs %lld bytes of scratch (tf_gemm_bf16_scratch_bytes)", __func__, (long long)at.total);
  TF_CHECK_ALIGNED(scratch, 256, "scratch");
  uint8_t* base = static_cast<uint8_t*>(scratch);
  float* own_scale = reinterpret_cast<float*>(base + at.global_scale);
  const float* a_gs = format != TF_FMT_NVFP4 ? nullptr : x_global_scale ? x_global_scale : own_scale;
  tf_status st = TF_OK;
  for (int pass = 0; pass < 2; ++pass) {  // first what the multiplication refuses, then the quantization, then the multiplication
    st = gemm_entry(__func__, base, base + at.scales, a_gs, b_codes, b_scales, b_global_scale, out, ldo, m, n, k, format, epilogue, epilogue_arg, out_amax, nullptr, nullptr, 0,
                    base + at.workspace, at.total - at.workspace, nullptr, 0, 0, stream, nullptr, pass == 0);
    if (st != TF_OK || pass == 1) return st;
    switch (format) {
      case TF_FMT_MXFP8: st = tf_quantize_mxfp8(x, m, k, ldx, base, base + at.scales, TF_SCALES_SWIZZLED, stream); break;
      case TF_FMT_MXFP4: st = tf_quantize_mxfp4(x, m, k, ldx, base, base + at.scales, TF_SCALES_SWIZZLED, stream); break;
      default:
        st = x_global_scale ? tf_quantize_nvfp4(x, m, k, ldx, base, base + at.scales, TF_SCALES_SWIZZLED, x_global_scale, stream)
             : x_amax       ? tf_quantize_nvfp4_from_amax(x, m, k, ldx, base, base + at.scales, TF_SCALES_SWIZZLED, x_amax, own_scale, stream)
                            : tf_quantize_nvfp4_dynamic(x, m, k, ldx, base, base + at.scales, TF_SCALES_SWIZZLED, own_scale,
                                                        reinterpret_cast<float*>(base + at.partials), stream);
    }
    if (st != TF_OK) return st;
  }
  return st;
}

tf_status tf_gemm_blockscaled_partials(const void* a_codes, const void* a_scales, const float* a_global_scale, const void* b_codes, const void* b_scales,
                                       const float* b_global_scale, int64_t m, int64_t n, int64_t k, int32_t format, void* workspace,
                                       int64_t workspace_bytes, int32_t* splits, void* stream) {
  clear_error();
  TF_CHECK_ARG(splits != nullptr, "%s: null pointer", __func__);
  return gemm_entry(__func__, a_codes, a_scales, a_global_scale, b_codes, b_scales, b_global_scale, nullptr, n, m, n, k, format, TF_EPI_NONE, nullptr,
                    nullptr, nullptr, nullptr, 0, workspace, workspace_bytes, nullptr, 0, 0, stream, splits);
}

tf_status tf_gemm_blockscaled_scatter(const void* a_codes, const void* a_scales, const float* a_global_scale, const void* b_codes, const void* b_scales,
                                      const float* b_global_scale, const uint64_t* out_ptrs, int32_t owners, int64_t rows_per_owner, int64_t ldo,
                                      int64_t m, int64_t n, int64_t k, int32_t format, int64_t a_global_scale_rows, void* stream) {
  clear_error();
  TF_CHECK_ARG(out_ptrs != nullptr, "%s: null pointer", __func__);
  TF_CHECK_ARG(owners >= 1 && owners <= 8, "%s: owners must be in 1..8", __func__);
  TF_CHECK_ARG(rows_per_owner > 0 && rows_per_owner % 128 == 0 && rows_per_owner <= (1 << 24), "%s: rows_per_owner must be a positive multiple of 128",
               __func__);
  TF_CHECK_ARG(m == (int64_t)owners * rows_per_owner, "%s: m=%lld is not owners x rows_per_owner", __func__, (long long)m);
  for (int i = 0; i < owners; ++i)
    if (!out_ptrs[i] || out_ptrs[i] % 16) return fail(TF_ERR_ALIGNMENT, "%s: destination %d is null or not 16-byte aligned", __func__, i);
  return gemm_entry(__func__, a_codes, a_scales, a_global_scale, b_codes, b_scales, b_global_scale, reinterpret_cast<void*>(out_ptrs[0]), ldo, m, n, k,
                    format, TF_EPI_NONE, nullptr, nullptr, nullptr, nullptr, a_global_scale_rows, nullptr, 0, out_ptrs, owners, rows_per_owner, stream);
}

}  // extern "C"
