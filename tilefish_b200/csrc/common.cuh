// Shared host/device helpers of the sm_100a backend.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>

#include "../../include/tilefish_b200.h"

namespace tf {

// ---- host: status + thread-local last error ------------------------------------------------------------------------
tf_status fail(tf_status code, const char* fmt, ...);
void clear_error();
int sm_count();

#define TF_CHECK_ARG(cond, ...)                                   \
  do {                                                            \
    if (!(cond)) return tf::fail(TF_ERR_INVALID_ARGUMENT, __VA_ARGS__); \
  } while (0)
#define TF_CHECK_ALIGNED(ptr, bytes, name)                                                                  \
  do {                                                                                                      \
    if ((reinterpret_cast<uintptr_t>(ptr) % (bytes)) != 0)                                                  \
      return tf::fail(TF_ERR_ALIGNMENT, "%s: %s must be %d-byte aligned", __func__, name, (int)(bytes));    \
  } while (0)
#define TF_CUDA(call)                                                                                       \
  do {                                                                                                      \
    cudaError_t e__ = (call);                                                                               \
    if (e__ != cudaSuccess) return tf::fail(TF_ERR_CUDA, "%s: %s failed: %s", __func__, #call, cudaGetErrorString(e__)); \
  } while (0)
// What a kernel that writes swizzled scales does about their padding: nothing (there is none, or the layout is plain) or zero it itself.
// A scale pointer that is not 16-byte aligned gets the memset instead (*pad = 0).
tf_status scale_padding(void* scales, int32_t format, int64_t rows, int64_t k, int32_t layout, cudaStream_t stream, int* pad);

#define TF_LAUNCH_CHECK() TF_CUDA(cudaGetLastError())

// Programmatic dependent launch (tf_set_programmatic_launch): a kernel launched through launch_dependent() may be scheduled
// while the kernel before it on the stream is still draining, so that its launch latency and set-up overlap that tail. Every
// thread of such a kernel executes griddep_wait() before it reads or writes anything that the kernel in front may write or read; the wait
// ends when that kernel has completed and its writes are visible. Two things happen before it: a GEMM asks weights into L2
// (prefetch_b_stage: nothing is read), and the nvfp4 quantizer loads the tensor that its own amax launch in front only reads
// (quantize_tiles_kernel: that launch is a plain one, so the tensor is complete).
// Three settings: never, always, or (until the caller says otherwise) for chains of short kernels only (`chain`, see chain_gemm_launch),
// and those only without an SM margin: a dependent GEMM's waiting CTAs would take the SMs that the margin leaves to the kernel beside it.
int sm_margin();
bool dependent_launch(bool chain);
void set_programmatic_launch(int setting);  // 0 never, 1 always, -1 the rule

#ifdef __CUDACC__
// The rule: GEMMs of at most 256 rows (above 128 and with one CTA per tile: of one wave), gated GEMMs of CTA pairs in one wave up to 1024
// rows, row kernels of at most four rows, and the nvfp4 quantizer behind its own amax launch up to 16 M elements (launch_quantize).
// A GEMM's CTAs take a whole SM each, so starting early only hides their set-up: 200 GEMMs back to back on a full queue, plain ->
// dependent: mxfp8 1 x 2560 x 3072 8.2 -> 5.9 us, 128 x 6144 x 2560 11.6 -> 9.0, nvfp4 64 x 8192 x 28672 36.7 -> 32.9; pairs in two
// waves mxfp4 256 x 16384 x 2048 + gate 20.5 -> 17.2, mxfp8 256 x 28672 x 2048 22.5 -> 20.6; one CTA per tile in two waves nvfp4
// 64 x 28672 x 8192 + gate 52.2 -> 52.1 back to back, where it gains behind a row kernel instead (prefetch_b_stage).
// A row kernel's CTAs are small: started early they all pile onto the few SMs that the GEMM in front leaves free and then share those
// (70B-shaped decode at 64 rows: its rmsnorm launch went from 9.8 to 14.7 us; two blocks at 16 rows 184.6 us without, 190.4 with).
// Above 256 rows the waiting CTAs take the registers that the rest of the row kernel in front needs (README block at 8192 rows
// 189.5 -> 196.2 us). Gated pairs of one wave stand behind a row kernel of at most 1024 rows, which fits beside them. Graphs of 12 chains,
// 15 shapes of 300 to 1024 rows, 1024 to 16384 columns and 2048 to 4608 gate columns in each format, plain -> dependent: behind rmsnorm
// (and a quantizer and second GEMM) mxfp8 512 x 2560 x 3072 33.1 -> 31.8 us, 700 x 2560 x 3072 40.6 -> 39.0, 1024 x 8192 x 2304 76.9 -> 75.8,
// nvfp4 1024 x 4096 x 2304 38.1 -> 36.5; behind a quantizer alone mxfp8 512 x 8192 x 4608 36.9 -> 35.5, mxfp4 1024 x 2560 x 2304 15.3 ->
// 14.2, nvfp4 300 x 4096 x 4096 16.4 -> 16.0. All between 0.93 and 1.01 of the time; 300 x 1024 x 2048 is the one that gains nothing. Only
// behind one another do 48 tiles of long K lose (512 x 3072 x 8192 mxfp8 30.3 -> 31.4, 1024 x 2304 x 8192 33.6 -> 32.5). The second GEMM
// of a block as a dependent too gives back half of the gain.
// Captured graphs, before -> after: README block at one row 20.5 -> 18.4 us, 70B-shaped decode at 64 rows 402 -> 389, two
// 4096 x 8192 blocks at 200 rows 93 -> 85.
enum class GemmKind { kOneCta, kPair, kGatedPair };
inline bool chain_gemm_launch(int64_t rows, bool one_wave, GemmKind kind) {
  if (rows <= 256) return rows <= 128 || one_wave || kind != GemmKind::kOneCta;
  return rows <= 1024 && one_wave && kind == GemmKind::kGatedPair;
}
inline bool chain_rows_launch(int64_t rows) { return rows <= 4; }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(bool chain, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent_launch(chain) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
#endif

// ---- device: bit-level conversions -----------------------------------------------------------------------------------
#ifdef __CUDACC__

// Wait for the previous kernel on the stream (returns at once in a plain launch); let the next one be scheduled early.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One f32 that a kernel in front may have written. A dependent can be resident while its predecessor still runs, so what that kernel may
// write is read with ordinary loads that stay behind griddep_wait(): the non-coherent path (__ldg, ld.global.nc) holds only for memory
// that nobody writes during the kernel's whole lifetime, and the compiler may move such loads. It is left to the norm weights.
__device__ __forceinline__ float load_f32(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ float bf16lo_to_f32(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16hi_to_f32(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// f32 -> bf16 word, round to nearest even, NaN -> 0x7FFF (what cvt.rn.bf16.f32 gives).
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float f) {
  uint16_t r;
  asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(r) : "f"(f));
  return r;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// two f32 -> two e4m3 bytes (lo in bits 0-7), RNE, saturating to +-448, NaN -> 0x7F.
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi) {
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
// eight f32 -> eight e2m1 nibbles in one word (element i in bits 4i .. 4i+3), RNE ties-to-even, saturating to +-6. The four bytes are
// packed as registers, without a shift and an OR for each.
__device__ __forceinline__ uint32_t cvt_e2m1x8(float a0, float a1, float a2, float a3, float a4, float a5, float a6, float a7) {
  uint32_t r;
  asm("{ .reg .b8 b0, b1, b2, b3;\n cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      " cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n mov.b32 %0, {b0, b1, b2, b3}; }"
      : "=r"(r)
      : "f"(a0), "f"(a1), "f"(a2), "f"(a3), "f"(a4), "f"(a5), "f"(a6), "f"(a7));
  return r;
}
// four f32 -> four e4m3 bytes in one word.
__device__ __forceinline__ uint32_t cvt_e4m3x4(float a0, float a1, float a2, float a3) {
  uint32_t r;
  asm("{ .reg .b16 h0, h1;\n cvt.rn.satfinite.e4m3x2.f32 h0, %2, %1;\n cvt.rn.satfinite.e4m3x2.f32 h1, %4, %3;\n mov.b32 %0, {h0, h1}; }"
      : "=r"(r)
      : "f"(a0), "f"(a1), "f"(a2), "f"(a3));
  return r;
}
// one e4m3 byte -> f32 (exact).
__device__ __forceinline__ float e4m3_to_f32(uint32_t code) {
  uint32_t h2;
  uint16_t c = (uint16_t)code;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(c));
  float f;
  asm("{ .reg .b16 lo, hi;\n mov.b32 {lo, hi}, %1;\n cvt.f32.f16 %0, lo; }" : "=f"(f) : "r"(h2));
  return f;
}

// silu(x) = x * (1 / (1 + exp(-x))) with the hardware's approximate exp2 and reciprocal (what the reference's own binaries use:
// ex2.approx and div.full). One definition for the stand-alone kernel and the GEMM epilogue, so both give the same bytes.
__device__ __forceinline__ float silu_f32(float g) { return __fmul_rn(g, __fdividef(1.0f, __fadd_rn(1.0f, __expf(-g)))); }

// Byte offset of scale entry (r, c) of a [rows, cols] scale tensor in the swizzled layout; n_ct = ceil(cols / 4).
__host__ __device__ __forceinline__ int64_t swizzled_scale_offset(int64_t r, int64_t c, int64_t n_ct) {
  int64_t tile = (r >> 7) * n_ct + (c >> 2);
  int rr = (int)(r & 127);
  return tile * 512 + (rr & 31) * 16 + (rr >> 5) * 4 + (int)(c & 3);
}

#endif  // __CUDACC__

}  // namespace tf
