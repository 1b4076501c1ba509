// Shared definitions of the delta-rule backward kernels (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/rewy_b200.h"

namespace rewy {

constexpr int C = 64;    // chunk rows
constexpr int DK = 128;  // key head dim
constexpr int DV = 128;  // value head dim

enum GateMode { GATE_NONE = 0, GATE_SCALAR = 1, GATE_VECTOR = 2 };

using bf16 = __nv_bfloat16;

// Span (max - min over the 64 tokens of a chunk, log2 units) of a per-channel cumulative gate, and the centred factors
// 2^(G - c), 2^(c - G), c its mid-point:
//   below VECTOR_SPAN_FREE  the factors stay inside 2^-40 .. 2^40 and need no care;
//   below VECTOR_SPAN_LIMIT they reach 2^-100 and 2^100.  A product of such operands is 2^-100 .. 2^100 of the result, so
//     the backward first scales the chunk's two gradient matrices by a power of two (2^-25 .. 2^25) that brings the largest
//     entry towards 1.  Measured at a span of 199 without it: dq off by 4.4e-6 down to gradients of 2^-30, by 1.3e-5 at
//     2^-35 and 2.1e-4 at 2^-40, infinite at 2^40; with it that lies 25 powers further out, so that 2^-55 .. 2^45 (output
//     gradient times value) is summed as well as a short span.  The forward's kept (causal) sums have their natural size;
//     entries above the diagonal may overflow and are selected away, never multiplied.  q and k must not add to the
//     factors: a chunk whose largest |q| or |k| lies outside 2^-20 .. 2^20 goes to the pairwise sums (inside, an operand's
//     BF16 lo part keeps its place above 2^-133);
//   from VECTOR_SPAN_LIMIT on the chunk is summed pair by pair on the CUDA cores, some thirty times as slow.
// A layer with decay rates up to 16 and time steps up to 0.1 averages up to 165 in its fastest channel.  At B=2 T=4096 H=16
// with such a gate: a limit of 80 sent 71 % of the chunks to the pairwise sums (3.65 ms of the backward, 0.55 ms of the
// forward), 160 a few (0.41 ms and 0.10 ms), 200 none.
constexpr float VECTOR_SPAN_FREE = 80.f;
constexpr float VECTOR_SPAN_LIMIT = 200.f;
// largest |x| of a chunk's q or k, as the bits of a BF16 (an infinity or NaN is out of range)
__device__ __forceinline__ bool centred_range(uint32_t bits) {
  constexpr uint32_t LOW = (127 - 20) << 7, HIGH = (127 + 20) << 7;
  return bits == 0 || (bits >= LOW && bits < HIGH);
}
// larger magnitudes of two pairs of BF16 (m: none negative; a NaN wins)
__device__ __forceinline__ uint32_t max_abs2(uint32_t m, uint32_t x) {
  const __nv_bfloat162 r = __hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&m), __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x)));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// A scalar gate needs no centred factors unless it rises (its pairwise factor is applied to the 64x64 matrices): limit of
// the chunks that do.
constexpr float SCALAR_SPAN_LIMIT = 80.f;

struct Dims {
  int B, T, H, NT;
};

// Host-side launchers (one per stage); each returns a cudaError_t from the launch.
cudaError_t launch_prepare(const RewyBwdArgs& a, const RewyStageBuffers& s, cudaStream_t st);                // warp-MMA kernel
cudaError_t launch_prepare_tc(const RewyBwdArgs& a, const RewyStageBuffers& s, int* err, cudaStream_t st);  // TMA + tcgen05
cudaError_t launch_fwd_scan(const RewyBwdArgs& a, const RewyStageBuffers& s, cudaStream_t st);
cudaError_t launch_bwd_scan(const RewyBwdArgs& a, const RewyStageBuffers& s, cudaStream_t st);      // warp-MMA kernel
// tcgen05 forward scan; final_state (optional) receives the state after the last chunk
cudaError_t launch_fwd_scan_tc(const RewyBwdArgs& a, const RewyStageBuffers& s, int* err, cudaStream_t st,
                               float* final_state = nullptr);
cudaError_t launch_bwd_scan_tc(const RewyBwdArgs& a, const RewyStageBuffers& s, int* err, cudaStream_t st);  // tcgen05
// chunk adjoint: tensor-core kernel (ctrl = device int[2 + chunks]: status word, wide-chunk count, indices)
// followed by the warp-MMA kernel on the listed wide-span chunks; or the warp-MMA kernel on every chunk.
cudaError_t launch_chunk_adjoint_tc(const RewyBwdArgs& a, const RewyStageBuffers& s, int* ctrl, cudaStream_t st);
cudaError_t launch_chunk_adjoint_warp(const RewyBwdArgs& a, const RewyStageBuffers& s, const int* list, cudaStream_t st);
cudaError_t launch_chunk_fwd_tc(const RewyFwdArgs& a, int* err, cudaStream_t st);     // forward, chunk-local stage
cudaError_t launch_chunk_output_tc(const RewyFwdArgs& a, int* err, cudaStream_t st);  // forward output, TMA + tcgen05
void count_launch(int n = 1);
int report_error(int code, const char* text);  // stores the text rewy_last_error() returns; gives back `code`
// shape envelope + presence and 16-byte alignment of every pointer of a chunk-stage call (REWY_OK or an error code)
int validate_chunk_stage(const RewyBwdArgs* a, const RewyStageBuffers* s, bool need_ctrl);

__host__ __device__ inline int gate_mode_of(int family) {
  return family == REWY_DELTA ? GATE_NONE : (family == REWY_GDN ? GATE_SCALAR : GATE_VECTOR);
}

// Opt a kernel in to `bytes` of dynamic shared memory once per device (the attribute sticks to the function in that
// device's context), so that a launch costs no extra runtime call afterwards.  Kern is the kernel itself (one guard per
// template instance).
template <auto Kern>
inline cudaError_t ensure_dynamic_smem(size_t bytes) {
  static unsigned long long done = 0;  // bit d: set on device d
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 64 && ((__atomic_load_n(&done, __ATOMIC_ACQUIRE) >> dev) & 1ull)) return cudaSuccess;
  e = cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && dev < 64) __atomic_fetch_or(&done, 1ull << dev, __ATOMIC_RELEASE);
  return e;
}

// ---- small device helpers -------------------------------------------------------------------
__device__ __forceinline__ float bf2f(bf16 x) { return __bfloat162float(x); }
__device__ __forceinline__ bf16 f2bf(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&p);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u) {
  __nv_bfloat162 p = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(p);
}

// Sum of four products in one fixed order: whichever kernel normalises a row, the bits are the same.
__device__ __forceinline__ float dot4(const float* a, const float* b) {
  return fmaf(a[3], b[3], fmaf(a[2], b[2], fmaf(a[1], b[1], __fmul_rn(a[0], b[0]))));
}

// Copy a [rows x cols] BF16 tile (cols multiple of 8) from global (row pitch g_ld elements) to
// shared (row pitch s_ld elements) with 16-byte accesses by the whole CTA.
template <int ROWS, int COLS>
__device__ __forceinline__ void load_tile_bf16(bf16* __restrict__ s, int s_ld, const bf16* __restrict__ g,
                                               size_t g_ld) {
  constexpr int V8 = COLS / 8;
  for (int i = threadIdx.x; i < ROWS * V8; i += blockDim.x) {
    int r = i / V8, c = (i % V8) * 8;
    *reinterpret_cast<uint4*>(s + r * s_ld + c) = *reinterpret_cast<const uint4*>(g + (size_t)r * g_ld + c);
  }
}
template <int ROWS, int COLS>
__device__ __forceinline__ void store_tile_bf16(bf16* __restrict__ g, size_t g_ld, const bf16* __restrict__ s,
                                                int s_ld) {
  constexpr int V8 = COLS / 8;
  for (int i = threadIdx.x; i < ROWS * V8; i += blockDim.x) {
    int r = i / V8, c = (i % V8) * 8;
    *reinterpret_cast<uint4*>(g + (size_t)r * g_ld + c) = *reinterpret_cast<const uint4*>(s + r * s_ld + c);
  }
}

}  // namespace rewy
