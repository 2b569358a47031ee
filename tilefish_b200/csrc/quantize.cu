// BlockScaled quantization row kernels (bf16 -> MXFP8 / MXFP4 / NVFP4) and the scale-layout helpers.
//
// HBM-bound: four 256-bit loads of 16 bf16 in flight per thread, block maxima combined with at most one warp shuffle, codes stored as 16 (e4m3)
// or 8 bytes (e2m1) per thread, scales as whole sectors. Algorithmic bytes per element: 2 + 1 + 1/32 (mxfp8), 2 + 0.5 + 1/32 (mxfp4),
// 2 + 0.5 + 1/16 (nvfp4).
#include "async_copy.cuh"
#include "quant_core.cuh"

namespace tf {

constexpr int kQuantThreads = 256;
constexpr int kQuantUnroll = 4;

__device__ __forceinline__ void load_256(const void* p, uint32_t (&w)[8]) {
  asm volatile("ld.global.L1::no_allocate.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(p));
}

// One round of a row: vectors base + threadIdx.x + j * blockDim.x, kQuantUnroll 256-bit loads in flight per thread. Threads without
// data (no such row, or past its end) get zeros.
__device__ __forceinline__ void load_round(const uint8_t* __restrict__ xr, bool row_ok, int base, int nvec, uint32_t (&v)[kQuantUnroll][8],
                                           bool (&has)[kQuantUnroll]) {
#pragma unroll
  for (int j = 0; j < kQuantUnroll; ++j) {
    const int vj = base + threadIdx.x + j * (int)blockDim.x;
    has[j] = row_ok && vj < nvec;
    if (has[j]) {
      load_256(xr + (int64_t)vj * 32, v[j]);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[j][e] = 0;
    }
  }
}

// gridDim.y cuts the rows into segments of whole rounds (few, long rows: more CTAs than row blocks). The segment of this block.
__device__ __forceinline__ void row_segment(int nvec, int& begin, int& end) {
  const int step = kQuantUnroll * (int)blockDim.x;
  const int rounds = (nvec + step - 1) / step;
  const int per_seg = (rounds + (int)gridDim.y - 1) / (int)gridDim.y;
  begin = (int)blockIdx.y * per_seg * step;
  end = min(nvec, begin + per_seg * step);
}

// gs_ptr holds the nvfp4 global scale, or (gs_out != nullptr) the tensor's amax from which it is derived here: one value, or the
// `n_partials` maxima that the blocks of an amax launch left (every block of a quantizer takes their maximum again: at most 1024 words).
// All `threads` threads of the block call it.
__device__ __forceinline__ float partials_max(const float* __restrict__ partials, int n, int tid, int threads) {
  uint32_t mx = 0;  // non-negative floats order like their bits
  for (int i = tid; i < n; i += threads) mx = max(mx, __float_as_uint(load_f32(partials + i)));
  __shared__ uint32_t warp_max[kQuantThreads / 32];
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  if ((tid & 31) == 0) warp_max[tid >> 5] = mx;
  __syncthreads();
  for (int i = 0; i < threads / 32; ++i) mx = max(mx, warp_max[i]);
  return __uint_as_float(mx);
}

// ---- the quantizer ------------------------------------------------------------------------------------------------------------
// HBM-bound. A 32-byte sector of the swizzled scales holds 4 scales each of the rows r, r + 32, r + 64, r + 96 and of the rows behind them.
// Where a warp walks along one row, every such sector is put together in L2 from eight 4-byte pieces of different warps, a store transaction
// each (as many as the codes take, for nvfp4). Here a warp takes these eight rows together: in one step 16 vectors (256 elements) of each, half
// a warp per row, four 256-bit loads in flight per thread. The scale bytes of a thread's four loads are one word; a 4 x 4 byte transpose
// over the lanes that share a scale word (two shuffles) leaves each word in a lane of its own, and one store writes whole sectors,
// the padding's zeros included. Rows of fewer than 256 columns get four lanes or two, and a warp more of them (quantize_lanes).
// One step per warp, so that the hardware deals the steps out: blocks that stay and walk keep every SM's loads and stores in phase. Graphs of 12,
// rows per block with a persistent grid -> this: 65536 x 4096 mxfp8 133.5 -> 118.2 us (6.9 TB/s), mxfp4 102.8 -> 95.9 (7.1), nvfp4 105.9 -> 101.4 (6.8;
// with its amax launch 195 -> 187); 4096 x 28672 59.2 -> 53.5, 48.4 -> 44.1, 50.9 -> 46.6; 8192 x 4096 18.5 -> 17.3, 16.4 -> 15.2, 17.5 -> 16.2; 1000 x 2720
// 3.7 -> 2.9, 3.8 -> 2.9, 4.0 -> 3.2; 64 x 28672 3.4 -> 2.7, 3.4 -> 2.6, 3.8 -> 2.9; 1 x 4096 2.6 -> 1.7, 2.6 -> 1.6, 3.1 -> 1.9. The same steps with a
// persistent grid took 137 us for the first (four rounds 121), 8-warp blocks 118 / 96 / 102.7.
// nvfp4 is bound by its instructions where x is in L2 (8192 x 4096: 169 per 16 elements, 65 % of the issue slots): each block keeps the reciprocals of all
// block scales in a table, multiplies pairs, and loads without branches. Without -> with: 65536 x 4096 103.5 -> 100.5 us, with the amax launch 188.9 -> 185.7; 8192 x 4096
// 16.3 -> 15.8, 31.0 -> 29.6; 4096 x 28672 47.7 -> 46.0; 4096 x 4096 in L2 7.8 -> 7.2.
constexpr int kTileWarps = 4;  // of a block

// Lane i of four (lanes `step` and 2 * step apart) holds bytes a_i[0..3]; returns a_0[i] | a_1[i] << 8 | a_2[i] << 16 | a_3[i] << 24.
__device__ __forceinline__ uint32_t transpose_bytes(uint32_t a, int step, int i) {
  uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, a, step);
  a = __byte_perm(a, o, (i & 1) ? 0x3715 : 0x6240);
  o = __shfl_xor_sync(0xFFFFFFFFu, a, 2 * step);
  return __byte_perm(a, o, (i & 2) ? 0x3276 : 0x5410);
}

// A step is LANES vectors of 128 / LANES rows (16 of eight); steps_per_unit = ceil(nvec / LANES) steps along a row, `total` steps in all.
// n_partials > 0: the kernel in front is this tensor's own amax launch. That one starts only when x is complete, so a warp's first step is
// loaded while it still runs; and the last rows come first, which the amax launch read last and left in L2.
template <int FMT, bool WORDS, int LANES>
__global__ void __launch_bounds__(kTileWarps * 32, 8) quantize_tiles_kernel(const uint8_t* __restrict__ x, int64_t m, int k, int64_t ldx, uint8_t* __restrict__ codes,
                                                                          uint8_t* __restrict__ scales, int layout, int steps_per_unit, int total,
                                                                          const float* __restrict__ gs_ptr, float* __restrict__ gs_out, int n_partials) {
  constexpr bool kNv = FMT == TF_FMT_NVFP4;
  constexpr int kCodeBytes = FMT == TF_FMT_MXFP8 ? 16 : 8;  // per vector
  const int nvec = k >> 4, cols = kNv ? nvec : nvec >> 1, n_ct = (cols + 3) >> 2;
  constexpr int kBlockLanes = kNv ? 1 : 2;                  // lanes that hold one block's elements
  const int lane = threadIdx.x & 31, h = lane / LANES, q = lane % LANES;
  __shared__ uint32_t inverses[kNv ? 128 : 1];
  griddep_launch_dependents();
  float gs = 0.0f, inv_t = 0.0f;
  if (!kNv || n_partials == 0) {
    griddep_wait();
    if (kNv) gs = load_f32(gs_ptr);  // used behind the first loads
  }
  bool first = kNv;  // the first round, which every warp of the block runs: the scale is formed in it
  for (int s0 = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));; s0 += (int)(gridDim.x * (blockDim.x >> 5))) {
    const bool live = s0 < total;
    if (!live && !first) break;
    const int s = !live ? 0 : n_partials > 0 ? total - 1 - s0 : s0;
    const int unit = s / steps_per_unit, c = s - unit * steps_per_unit;
    const int rr = unit % LANES * (32 / LANES) + h;  // these lanes' place in a group of 32 rows
    const int64_t row = (int64_t)(unit / LANES) * 128 + rr;
    const int vec = c * LANES + q;
    const uint8_t* xp = x + row * ldx * 2 + (int64_t)vec * 32;
    uint32_t v[4][8];
    bool has[4];  // j: row + 32 * j
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      has[j] = live && row + 32 * j < m && vec < nvec;
      load_256(has[j] ? xp + 64 * j * ldx : x, v[j]);  // a load without data is read from the tensor's start and not used
    }
    if (kNv && first) {
      if (n_partials > 0) {
        griddep_wait();
        gs = partials_max(gs_ptr, n_partials, threadIdx.x, blockDim.x);
      }
      if (gs_out != nullptr) {
        gs = __fdiv_rn(gs, 2688.0f);
        if (blockIdx.x == 0 && threadIdx.x == 0) gs_out[0] = gs;
      }
      inv_t = gs != 0.0f ? __frcp_rn(__fmul_rn(6.0f, gs)) : 0.0f;
      // a block's scale byte has the sign of gs, its other seven bits are the index
      for (int i = threadIdx.x; i < 128; i += blockDim.x) inverses[i] = nvfp4_inverse(gs < 0.0f ? i | 0x80 : i, gs);
      __syncthreads();
      first = false;
      if (!live) break;
    }
    uint8_t* cp = codes + (row * nvec + vec) * kCodeBytes;
    uint32_t word = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t cw[4], sc;
      quantize_vec16<FMT>(v[j], gs, inv_t, cw, sc, inverses);
      if (has[j]) {
        word |= sc << (8 * j);
        uint8_t* dst = cp + (int64_t)(32 * j) * nvec * kCodeBytes;
        if (FMT == TF_FMT_MXFP8) *reinterpret_cast<uint4*>(dst) = make_uint4(cw[0], cw[1], cw[2], cw[3]);
        else *reinterpret_cast<uint2*>(dst) = make_uint2(cw[0], cw[1]);
      }
    }
    if (LANES >= 4 * kBlockLanes) {
      // four scales of one row are four lanes (nvfp4) or four pairs of lanes; lane (pair) i of them gets the word of load i
      const int i = q / kBlockLanes & 3;
      word = transpose_bytes(word, kBlockLanes, i);
      const int ct = vec / (4 * kBlockLanes);
      if (ct < n_ct && q % kBlockLanes == 0) store_scale_word<WORDS>(scales, layout, row + 32 * i, ct * 4, cols, n_ct, row + 32 * i < m, word);
    } else {
      // two scales of a row (one with mx and two lanes), in the lower and upper lanes; lane i gets the pair of load i (and of load i + 2 where there
      // are two lanes). The last step's pair is a word with the zeros behind it, if it starts one.
      const uint32_t other = LANES > kBlockLanes ? __shfl_xor_sync(0xFFFFFFFFu, word, LANES / 2) : 0u;
      const bool upper = LANES > kBlockLanes && q >= LANES / 2;
      const uint32_t lo = upper ? other : word, hi = upper ? word : other;
      const bool pair = LANES == 4 && ((c & 1) || (c + 1) * LANES < nvec);
#pragma unroll
      for (int i = q; i < 4; i += LANES)
        store_scale_word<WORDS>(scales, layout, row + 32 * i, c * 2, cols, n_ct, row + 32 * i < m, (lo >> (8 * i) & 255u) | (hi >> (8 * i) & 255u) << 8, pair);
    }
  }
}

// ---- the amax pass of a dense tensor: one run of bytes staged through a shared-memory ring by bulk copies ------------------------
// The tensor is cut into 8 KB chunks that the CTAs take in turn. Every CTA owns a ring of chunk buffers; thread 0 keeps it full with
// cp.async.bulk (completion counted on an mbarrier), so the loads wait for neither registers nor arithmetic. 96 % of the copy rate at
// 65536 x 4096 (84.5 us). Chunks are cut across rows, so widths that are no multiple of a chunk cost nothing: against a ring of row
// chunks 16384 x 2080 24.9 -> 18.3 us with its two small launches, 4096 x 2560 11.8 -> 8.4. Waits are bounded (async_copy.cuh).
constexpr int kStreamThreads = 128;
constexpr int kStreamVpt = 2;
constexpr int kStreamChunkVecs = kStreamThreads * kStreamVpt;
constexpr int kStreamChunkBytes = kStreamChunkVecs * 32;
constexpr int kStreamStages = 4;
constexpr int kStreamCtasPerSm = 6;
constexpr size_t kStreamSmem = (size_t)kStreamStages * (kStreamChunkBytes + 8);
constexpr unsigned long long kWaitLimitNs = 1000000000ull;

__device__ __forceinline__ void lds_256(uint32_t addr, uint32_t (&w)[8]) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "r"(addr + 16));
}

// Two packed 16-bit maxima of the magnitudes of 16 bf16, joined with `acc`.
__device__ __forceinline__ uint32_t amax16(const uint32_t (&w)[8], uint32_t acc) {
  const uint32_t km = 0x7FFF7FFFu;
  uint32_t t0 = __vimax3_u16x2(w[0] & km, w[1] & km, w[2] & km);
  uint32_t t1 = __vimax3_u16x2(w[3] & km, w[4] & km, w[5] & km);
  t0 = __vimax3_u16x2(t0, w[6] & km, w[7] & km);
  return __vimax3_u16x2(acc, t0, t1);
}

// The block's maximum of two packed maxima per thread, in thread 0. Every thread of the block calls it.
template <int THREADS>
__device__ __forceinline__ uint32_t block_amax(uint32_t acc, int tid) {
  __shared__ uint32_t warp_max[THREADS / 32];
  uint32_t mx = max(acc & 0xFFFFu, acc >> 16);
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  if ((tid & 31) == 0) warp_max[tid >> 5] = mx;
  __syncthreads();
  if (tid == 0)
    for (int wi = 1; wi < THREADS / 32; ++wi) mx = max(mx, warp_max[wi]);
  return mx;
}

// Dynamic shared memory: kStreamStages chunk buffers, then one mbarrier per stage. total: 16-element vectors of the tensor.
// The maximum goes to *out_bits (an atomic max), or as this block's own word to partials[blockIdx.x].
__global__ void __launch_bounds__(kStreamThreads) stream_amax_kernel(const uint8_t* __restrict__ x, int64_t total, unsigned int* __restrict__ out_bits,
                                                                     unsigned int* __restrict__ partials, int* __restrict__ status) {
  griddep_launch_dependents();
  extern __shared__ __align__(128) uint8_t ring_smem[];
  __shared__ int abort_flag;
  const uint32_t ring = smem_u32(ring_smem);
  const uint32_t bars = ring + (uint32_t)kStreamStages * kStreamChunkBytes;
  const int t = threadIdx.x;
  if (t == 0) {
    for (int s = 0; s < kStreamStages; ++s) mbar_init(bars + 8 * s, 1);
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  // thread 0: one bulk copy per chunk, the last one possibly short
  const int64_t stride = (int64_t)gridDim.x * kStreamChunkVecs;
  auto issue = [&](int64_t base, int stage) {
    const uint32_t bytes = (uint32_t)min((int64_t)kStreamChunkVecs, total - base) * 32u;
    const uint32_t bar = bars + 8 * stage;
    mbar_expect_tx(bar, bytes);
    bulk_load(ring + (uint32_t)stage * kStreamChunkBytes, x + base * 32, bytes, bar);
  };
  int64_t base = (int64_t)blockIdx.x * kStreamChunkVecs;
  if (t == 0) {
    for (int s = 0; s < kStreamStages; ++s)
      if (base + s * stride < total) issue(base + s * stride, s);
  }
  uint32_t acc = 0;  // two packed 16-bit maxima
  int stage = 0;
  uint32_t phase = 0;
  for (; base < total; base += stride) {
    const bool ok = mbar_wait_bounded(bars + 8 * stage, phase, &abort_flag, status, 10, kWaitLimitNs);
#pragma unroll
    for (int j = 0; j < kStreamVpt; ++j) {
      if (ok && base + t + j * kStreamThreads < total) {
        uint32_t w[8];
        lds_256(ring + (uint32_t)stage * kStreamChunkBytes + (t + j * kStreamThreads) * 32, w);
        acc = amax16(w, acc);
      }
    }
    // every thread has read its bytes (or the wait ran out somewhere: then all leave together)
    if (!__syncthreads_and(ok)) break;
    if (t == 0 && base + kStreamStages * stride < total) issue(base + kStreamStages * stride, stage);
    if (++stage == kStreamStages) {
      stage = 0;
      phase ^= 1;
    }
  }
  const uint32_t mx = block_amax<kStreamThreads>(acc, t);
  if (t == 0 && partials) partials[blockIdx.x] = mx << 16;
  else if (t == 0 && mx) atomicMax(out_bits, mx << 16);  // the f32 bit pattern of a non-negative bf16 orders like the integer
  if (t == 0 && abort_flag) {  // a wait ran out: give copies still in flight time to land before shared memory is released
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
}

// The amax of a dense tensor too small for the ring: 256-bit loads, four in flight per thread. Result as stream_amax_kernel's.
__global__ void __launch_bounds__(256) amax_bits_kernel(const uint8_t* __restrict__ x, int64_t total, unsigned int* __restrict__ out_bits,
                                                        unsigned int* __restrict__ partials) {
  griddep_launch_dependents();
  uint32_t acc = 0;  // two packed 16-bit maxima
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < total; i0 += 4 * stride) {
    uint32_t v[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = i0 + j * stride;
      if (i < total) {
        load_256(x + i * 32, v[j]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[j][e] = 0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc = amax16(v[j], acc);
  }
  const uint32_t mx = block_amax<256>(acc, threadIdx.x);
  if (threadIdx.x == 0 && partials) partials[blockIdx.x] = mx << 16;
  else if (threadIdx.x == 0 && mx) atomicMax(out_bits, mx << 16);
}

// The amax of rows with a stride (column slices), bound by HBM: the quantizer's walk over the rows. A flat index over the vectors costs a 64-bit
// division for each. Flat index -> here, tf_nvfp4_global_scale of 65536 x 4096 out of rows of 8192 106.7 -> 82.8 us, 131072 x 1024 out of 2048 57.9 ->
// 45.0, 2048 x 28672 out of 57344 31.0 -> 24.6, 1000 x 2080 out of 4160 8.2 -> 6.9.
__global__ void __launch_bounds__(kQuantThreads) amax_rows_kernel(const uint8_t* __restrict__ x, int64_t m, int nvec, int64_t ldx,
                                                                  unsigned int* __restrict__ out_bits, unsigned int* __restrict__ partials) {
  griddep_launch_dependents();
  uint32_t acc = 0;  // two packed 16-bit maxima
  int begin, end;
  row_segment(nvec, begin, end);
  for (int64_t row0 = (int64_t)blockIdx.x * blockDim.y; row0 < m; row0 += (int64_t)gridDim.x * blockDim.y) {
    const int64_t row = row0 + threadIdx.y;
    const bool row_ok = row < m;
    const uint8_t* xr = x + (row_ok ? row : 0) * ldx * 2;
    for (int base = begin; base < end; base += kQuantUnroll * (int)blockDim.x) {
      uint32_t v[kQuantUnroll][8];
      bool has[kQuantUnroll];
      load_round(xr, row_ok, base, nvec, v, has);
#pragma unroll
      for (int j = 0; j < kQuantUnroll; ++j) acc = amax16(v[j], acc);
    }
  }
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  const uint32_t mx = block_amax<kQuantThreads>(acc, tid);
  if (tid == 0 && partials) partials[blockIdx.y * gridDim.x + blockIdx.x] = mx << 16;
  else if (tid == 0 && mx) atomicMax(out_bits, mx << 16);
}

static void rows_shape(int64_t m, int64_t k, int per_sm, dim3& grid, dim3& block);

// nvfp4 without a given scale is two launches: an amax launch whose blocks leave their maxima, and the quantizer, which derives the scale
// from them. Before: a memset, an amax launch with an atomic, a one-thread launch for the scale and the quantizer. Graphs of 12: 128 x
// 4096 10.5 -> 5.7 us, 4096 x 2560 20.6 -> 14.1, 8192 x 4096 35.1 -> 30.0, 65536 x 4096 212 -> 194. One cooperative launch with a grid
// barrier in place of the two took 10.5 us at 128 x 4096 and 201 at 65536 x 4096 (such launches start late).
constexpr int kMaxAmaxBlocks = 1024;  // blocks of an amax launch, and words of its partial maxima

// The amax launch: into *out_bits (zeroed by the caller), or a word per block into `partials`, whose number goes to *blocks.
static tf_status launch_amax(const char* fn, const void* x, int64_t m, int64_t k, int64_t ldx, unsigned int* out_bits, unsigned int* partials, int* blocks,
                             cudaStream_t stream) {
  const uint8_t* xb = static_cast<const uint8_t*>(x);
  const int64_t total = m * (k >> 4);
  if (ldx != k && m > 1) {
    const int per_sm = kMaxAmaxBlocks / sm_count();
    dim3 grid, block;
    rows_shape(m, k, per_sm < kStreamCtasPerSm ? per_sm : kStreamCtasPerSm, grid, block);
    *blocks = (int)(grid.x * grid.y);
    amax_rows_kernel<<<grid, block, 0, stream>>>(xb, m, (int)(k >> 4), ldx, out_bits, partials);
  } else if (total >= 2 * (int64_t)sm_count() * kStreamChunkVecs) {  // at least two chunks per SM
    int* status = device_status_words();
    if (!status) return fail(TF_ERR_CUDA, "%s: cannot locate the device status words", fn);
    static thread_local int configured_dev = -1;
    int dev = 0;
    TF_CUDA(cudaGetDevice(&dev));
    if (configured_dev != dev) {
      // the ring is all this kernel uses of the SM's memory: let the carve-out hold as many CTAs' rings as possible
      TF_CUDA(cudaFuncSetAttribute(stream_amax_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
      configured_dev = dev;
    }
    const int64_t chunks = (total + kStreamChunkVecs - 1) / kStreamChunkVecs;
    int64_t cap = (int64_t)sm_count() * kStreamCtasPerSm;
    if (cap > kMaxAmaxBlocks) cap = kMaxAmaxBlocks;
    *blocks = (int)(chunks < cap ? chunks : cap);
    stream_amax_kernel<<<*blocks, kStreamThreads, kStreamSmem, stream>>>(xb, total, out_bits, partials, status);
  } else {
    const int64_t need = (total + 1023) / 1024;
    *blocks = (int)(need < kMaxAmaxBlocks ? need : kMaxAmaxBlocks);
    amax_bits_kernel<<<*blocks, 256, 0, stream>>>(xb, total, out_bits, partials);
  }
  TF_LAUNCH_CHECK();
  return TF_OK;
}

__global__ void finalize_global_scale_kernel(float* gs) { gs[0] = __fdiv_rn(gs[0], 2688.0f); }

__global__ void __launch_bounds__(256) swizzle_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int64_t rows, int64_t cols,
                                                      int to_swizzled) {
  const int64_t n_ct = (cols + 3) >> 2;
  const int64_t total = rows * cols;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / cols, c = i - r * cols;
    const int64_t off = swizzled_scale_offset(r, c, n_ct);
    if (to_swizzled) dst[off] = src[i];
    else dst[i] = src[off];
  }
}

static int block_of(int format) { return format == TF_FMT_NVFP4 ? 16 : 32; }

tf_status scale_padding(void* scales, int32_t format, int64_t rows, int64_t k, int32_t layout, cudaStream_t stream, int* pad) {
  *pad = layout == TF_SCALES_SWIZZLED && ((rows & 127) || ((k / block_of(format)) & 3));
  if (*pad && reinterpret_cast<uintptr_t>(scales) % 16) {
    *pad = 0;
    TF_CUDA(cudaMemsetAsync(scales, 0, (size_t)tf_scale_bytes(format, rows, k, layout), stream));
  }
  return TF_OK;
}

static tf_status check_quant_args(const char* fn, const void* x, int64_t m, int64_t k, int64_t ldx, const void* codes, const void* scales,
                                  int layout) {
  if (!x || !codes || !scales) return fail(TF_ERR_INVALID_ARGUMENT, "%s: null pointer", fn);
  if (m < 0 || k <= 0) return fail(TF_ERR_INVALID_ARGUMENT, "%s: bad shape m=%lld k=%lld", fn, (long long)m, (long long)k);
  if (layout != TF_SCALES_PLAIN && layout != TF_SCALES_SWIZZLED) return fail(TF_ERR_INVALID_ARGUMENT, "%s: unknown scale layout %d", fn, layout);
  if (k % 32 != 0) return fail(TF_ERR_UNSUPPORTED, "%s: k=%lld is not a multiple of 32", fn, (long long)k);
  if (ldx < k || ldx % 8 != 0) return fail(TF_ERR_ALIGNMENT, "%s: ldx=%lld must be >= k and a multiple of 8", fn, (long long)ldx);
  if (k > (int64_t)1 << 30) return fail(TF_ERR_UNSUPPORTED, "%s: k too large", fn);
  if ((uintptr_t)x % 16 || (uintptr_t)codes % 16) return fail(TF_ERR_ALIGNMENT, "%s: x and codes must be 16-byte aligned", fn);
  if ((uintptr_t)x % 32 || ldx % 16) return fail(TF_ERR_ALIGNMENT, "%s: x must be 32-byte aligned with ldx a multiple of 16 (256-bit loads)", fn);
  return TF_OK;
}

// Block and grid of amax_rows_kernel: a power of two of threads along the row, at most `per_sm` blocks per SM.
static void rows_shape(int64_t m, int64_t k, int per_sm, dim3& grid, dim3& block) {
  int tpr = 2;
  while (tpr < kQuantThreads && tpr * kQuantUnroll < (k >> 4)) tpr <<= 1;
  const int rpb = kQuantThreads / tpr;
  const int64_t blocks_needed = (m + rpb - 1) / rpb, cap = (int64_t)sm_count() * per_sm;
  block = dim3(tpr, rpb);
  grid = dim3((unsigned)(blocks_needed < cap ? blocks_needed : cap));
  const int64_t rounds = ((k >> 4) + kQuantUnroll * tpr - 1) / (kQuantUnroll * tpr);
  if (blocks_needed < 2 * sm_count() && rounds > 1) {  // few long rows: cut them into segments so that every SM gets work
    int64_t want = (2 * sm_count() + blocks_needed - 1) / blocks_needed;
    if (want * blocks_needed > cap) want = cap / blocks_needed;
    grid.y = (unsigned)(want < 1 ? 1 : want < rounds ? want : rounds);
  }
}

// Lanes per row of the quantizer. A step is bound by its instructions and costs the same whatever its lanes hold: below 256 columns, rows of 16 lanes took
// up to four times as long as a walk with two threads per row. 16 lanes -> 4 (2 at 32 columns; the walk), us, mxfp8 / mxfp4 / nvfp4: 1048576 x 32
// 112.9 -> 17.6 (27.8) / 112.3 -> 15.3 (28.3) / 112.0 -> 15.4 (28.3); 524288 x 64 60.4 -> 17.7 (20.3) / 59.0 -> 15.3 (19.8) / 59.1 -> 15.6 (20.4);
// 200001 x 96 25.9 -> 12.7 (12.8) / 25.0 -> 11.5 (12.0) / 25.2 -> 12.4 (13.2); 65536 x 192 11.6 -> 8.1 (9.6) / 10.8 -> 6.2 (8.0) / 11.1 -> 7.3 (8.7);
// 65536 x 224 11.7 -> 9.8 (10.9) / 11.1 -> 8.0 (9.9) / 11.3 -> 8.9 (10.9). Eight lanes are no better at 128 columns and took 15.9 us for 200001 x 96 mxfp8. At 256
// columns and above 16 lanes beat the walk everywhere (65536 x 288 13.2 (13.9) / 12.4 (13.6) / 13.8 (14.4)).
static int quantize_lanes(int64_t nvec) { return nvec >= 16 ? 16 : nvec == 2 ? 2 : 4; }

template <int FMT, bool WORDS>
static auto tiles_kernel(int lanes) {
  return lanes == 16 ? quantize_tiles_kernel<FMT, WORDS, 16> : lanes == 4 ? quantize_tiles_kernel<FMT, WORDS, 4> : quantize_tiles_kernel<FMT, WORDS, 2>;
}

template <int FMT>
static tf_status launch_quantize(const char* fn, const void* x, int64_t m, int64_t k, int64_t ldx, void* codes, void* scales, int layout,
                                 const float* gs, cudaStream_t stream, float* gs_out = nullptr, int n_partials = 0) {
  tf_status st = check_quant_args(fn, x, m, k, ldx, codes, scales, layout);
  if (st != TF_OK) return st;
  if (FMT == TF_FMT_NVFP4 && !gs) return fail(TF_ERR_INVALID_ARGUMENT, "%s: nvfp4 needs a global scale", fn);
  if (m == 0) return TF_OK;
  const int lanes = quantize_lanes(k >> 4);
  const int64_t steps_per_unit = ((k >> 4) + lanes - 1) / lanes, total = (m + 127) / 128 * lanes * steps_per_unit;
  if (total > INT32_MAX) return fail(TF_ERR_UNSUPPORTED, "%s: m=%lld x k=%lld is too large", fn, (long long)m, (long long)k);
  int64_t warps = (total + sm_count() - 1) / sm_count();  // few steps: narrower blocks, so that every SM gets some
  if (warps > kTileWarps) warps = kTileWarps;
  // Behind an amax launch every block takes the maximum of its words: two steps for each (65536 x 4096 with the amax launch 195.5 -> 187 us).
  // Up to 16 M elements the blocks start as that launch's dependents (128 x 4096 4.5 -> 4.0 us, 2048 x 4096 9.6 -> 8.3); beyond that their
  // waiting costs the amax launch more (8192 x 4096 29.9 -> 33.0).
  const int64_t rounds = n_partials > 0 && total > 32 * (int64_t)sm_count() ? 2 : 1;
  const bool dependent = (n_partials > 0 && m * k <= (int64_t)1 << 24) || chain_rows_launch(m);
  auto kernel = scales_as_words(scales, layout) ? tiles_kernel<FMT, true>(lanes) : tiles_kernel<FMT, false>(lanes);
  TF_CUDA(launch_dependent(dependent, kernel, dim3((unsigned)((total + warps * rounds - 1) / (warps * rounds))), dim3((unsigned)warps * 32), 0, stream,
                           static_cast<const uint8_t*>(x), m, (int)k, ldx, static_cast<uint8_t*>(codes), static_cast<uint8_t*>(scales), layout,
                           (int)steps_per_unit, (int)total, gs, gs_out, n_partials));
  return TF_OK;
}

}  // namespace tf

using namespace tf;

extern "C" {

int64_t tf_scale_bytes(int32_t format, int64_t rows, int64_t k, int32_t layout) {
  if (format < TF_FMT_MXFP8 || format > TF_FMT_NVFP4 || rows < 0 || k < 0) return -1;
  const int64_t blk = block_of(format);
  if (k % blk) return -1;
  const int64_t cols = k / blk;
  if (layout == TF_SCALES_PLAIN) return rows * cols;
  if (layout == TF_SCALES_SWIZZLED) return ((rows + 127) / 128) * ((cols + 3) / 4) * 512;
  return -1;
}

tf_status tf_quantize_mxfp8(const void* x, int64_t m, int64_t k, int64_t ldx, void* codes, void* scales, int32_t layout, void* stream) {
  clear_error();
  return launch_quantize<TF_FMT_MXFP8>(__func__, x, m, k, ldx, codes, scales, layout, nullptr, (cudaStream_t)stream);
}
tf_status tf_quantize_mxfp4(const void* x, int64_t m, int64_t k, int64_t ldx, void* codes, void* scales, int32_t layout, void* stream) {
  clear_error();
  return launch_quantize<TF_FMT_MXFP4>(__func__, x, m, k, ldx, codes, scales, layout, nullptr, (cudaStream_t)stream);
}
tf_status tf_quantize_nvfp4(const void* x, int64_t m, int64_t k, int64_t ldx, void* codes, void* scales, int32_t layout,
                            const float* global_scale, void* stream) {
  clear_error();
  return launch_quantize<TF_FMT_NVFP4>(__func__, x, m, k, ldx, codes, scales, layout, global_scale, (cudaStream_t)stream);
}

tf_status tf_quantize_nvfp4_from_amax(const void* x, int64_t m, int64_t k, int64_t ldx, void* codes, void* scales, int32_t layout,
                                      const float* amax, float* global_scale_out, void* stream) {
  clear_error();
  TF_CHECK_ARG(amax && global_scale_out, "%s: null pointer", __func__);
  if (m == 0) {  // no kernel runs for an empty tensor: derive the scale with the one-thread kernel
    TF_CUDA(cudaMemcpyAsync(global_scale_out, amax, sizeof(float), cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
    finalize_global_scale_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(global_scale_out);
    TF_LAUNCH_CHECK();
    return TF_OK;
  }
  return launch_quantize<TF_FMT_NVFP4>(__func__, x, m, k, ldx, codes, scales, layout, amax, (cudaStream_t)stream, global_scale_out);
}

int64_t tf_quantize_nvfp4_dynamic_scratch_bytes(void) { return kMaxAmaxBlocks * (int64_t)sizeof(float); }

tf_status tf_quantize_nvfp4_dynamic(const void* x, int64_t m, int64_t k, int64_t ldx, void* codes, void* scales, int32_t layout,
                                    float* global_scale_out, float* scratch, void* stream_) {
  clear_error();
  cudaStream_t stream = (cudaStream_t)stream_;
  TF_CHECK_ARG(global_scale_out && scratch, "%s: null pointer", __func__);
  TF_CHECK_ALIGNED(global_scale_out, 4, "global_scale_out");
  TF_CHECK_ALIGNED(scratch, 4, "scratch");
  tf_status st = check_quant_args(__func__, x, m, k, ldx, codes, scales, layout);
  if (st != TF_OK) return st;
  if (m == 0) {
    TF_CUDA(cudaMemsetAsync(global_scale_out, 0, sizeof(float), stream));
    return TF_OK;
  }
  int blocks = 0;
  st = launch_amax(__func__, x, m, k, ldx, nullptr, reinterpret_cast<unsigned int*>(scratch), &blocks, stream);
  if (st != TF_OK) return st;
  return launch_quantize<TF_FMT_NVFP4>(__func__, x, m, k, ldx, codes, scales, layout, scratch, stream, global_scale_out, blocks);
}

tf_status tf_nvfp4_global_scale(const void* x, int64_t m, int64_t k, int64_t ldx, float* out, void* stream_) {
  clear_error();
  cudaStream_t stream = (cudaStream_t)stream_;
  TF_CHECK_ARG(x && out, "%s: null pointer", __func__);
  TF_CHECK_ARG(m >= 0 && k > 0 && k % 16 == 0 && ldx >= k && ldx % 16 == 0, "%s: bad shape (k and ldx must be multiples of 16)", __func__);
  TF_CHECK_ALIGNED(x, 32, "x");
  TF_CUDA(cudaMemsetAsync(out, 0, sizeof(float), stream));
  if (m > 0) {
    int blocks = 0;
    const tf_status st = launch_amax(__func__, x, m, k, ldx, reinterpret_cast<unsigned int*>(out), nullptr, &blocks, stream);
    if (st != TF_OK) return st;
  }
  finalize_global_scale_kernel<<<1, 1, 0, stream>>>(out);
  TF_LAUNCH_CHECK();
  return TF_OK;
}

static tf_status swizzle_impl(const char* fn, const void* src, void* dst, int64_t rows, int64_t cols, int to_swizzled, cudaStream_t stream) {
  if (!src || !dst) return fail(TF_ERR_INVALID_ARGUMENT, "%s: null pointer", fn);
  if (rows < 0 || cols < 0) return fail(TF_ERR_INVALID_ARGUMENT, "%s: bad shape", fn);
  if (to_swizzled) {
    const size_t bytes = (size_t)(((rows + 127) / 128) * ((cols + 3) / 4) * 512);
    if (bytes) TF_CUDA(cudaMemsetAsync(dst, 0, bytes, stream));
  }
  const int64_t total = rows * cols;
  if (total == 0) return TF_OK;
  const int64_t need = (total + 255) / 256, cap = (int64_t)sm_count() * 8;
  swizzle_kernel<<<(unsigned)(need < cap ? need : cap), 256, 0, stream>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), rows,
                                                                          cols, to_swizzled);
  TF_LAUNCH_CHECK();
  return TF_OK;
}

tf_status tf_swizzle_scales(const void* plain, int64_t rows, int64_t cols, void* swizzled, void* stream) {
  clear_error();
  return swizzle_impl(__func__, plain, swizzled, rows, cols, 1, (cudaStream_t)stream);
}
tf_status tf_unswizzle_scales(const void* swizzled, int64_t rows, int64_t cols, void* plain, void* stream) {
  clear_error();
  return swizzle_impl(__func__, swizzled, plain, rows, cols, 0, (cudaStream_t)stream);
}

}  // extern "C"
