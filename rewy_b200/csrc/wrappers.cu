// Element-wise stages around the core backward: the transformations the reference's autograd wrappers apply before
// the forward and after the family backward (src/fast_delta_rule/_compat/kda.py:56-63,202-210; FLA l2norm_fwd /
// l2norm_bwd, fused_beta_sigmoid(_bwd), kda_gate_chunk_cumsum and kda_gate_bwd).  Each is one pass over its tensor,
// bound by HBM: 16-byte accesses, one warp per 128-wide row, grids sized in multiples of the SM count.
//   l2norm      y = x * rsqrt(sum x^2 + eps)                       dx = (dy - y * sum(dy*y)) * rstd, cast to BF16
//   beta        y = scale * sigmoid(x)                             dx = dy * scale * s * (1 - s)
//   KDA gate    g = -exp(A_log[h]) * softplus(x + dt_bias[h,k])    chunk-local cumulative sum in log2 units
//               dx = -exp(A_log[h]) * dg * sigmoid(x + bias);  dA_log[h] = sum dg * g;  ddt_bias[h,k] = sum dx
#include <cstdio>
#include <type_traits>
#include "common.cuh"

namespace rewy {
namespace {

constexpr float RCP_LN2 = 1.4426950408889634f;

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
  return x;
}

__device__ __forceinline__ void load4_bf16(const bf16* p, float (&x)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y);
  x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}
__device__ __forceinline__ void store4_bf16(bf16* p, const float (&x)[4]) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]));
}

// One warp per row of 128 BF16 values; lane l owns columns 4l .. 4l+3.  Both kernels sum in the order of the front kernels in
// rows.cu (dot4, then the butterfly), so that a row's result does not depend on which of them the call goes through.
__global__ void __launch_bounds__(256) l2norm_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y,
                                                          float* __restrict__ rstd, long long rows, float eps) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    float v[4];
    load4_bf16(x + r * 128 + 4 * lane, v);
    const float ss = warp_sum(dot4(v, v));
    const float rs = rsqrtf(ss + eps);
    float o[4] = {v[0] * rs, v[1] * rs, v[2] * rs, v[3] * rs};
    store4_bf16(y + r * 128 + 4 * lane, o);
    if (lane == 0) rstd[r] = rs;
  }
}

template <bool DY_F32>
__global__ void __launch_bounds__(256) l2norm_bwd_kernel(const bf16* __restrict__ y, const float* __restrict__ rstd,
                                                          const void* __restrict__ dy, bf16* __restrict__ dx,
                                                          long long rows) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += warps) {
    float yv[4], g[4];
    load4_bf16(y + r * 128 + 4 * lane, yv);
    if (DY_F32) {
      const float4 t = *reinterpret_cast<const float4*>(static_cast<const float*>(dy) + r * 128 + 4 * lane);
      g[0] = t.x; g[1] = t.y; g[2] = t.z; g[3] = t.w;
    } else {
      load4_bf16(static_cast<const bf16*>(dy) + r * 128 + 4 * lane, g);
    }
    const float s = warp_sum(dot4(g, yv));
    const float rs = rstd[r];
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = fmaf(-yv[i], s, g[i]) * rs;
    store4_bf16(dx + r * 128 + 4 * lane, o);
  }
}

__device__ __forceinline__ float sigmoidf(float x) { return 1.f / (1.f + __expf(-x)); }
__device__ __forceinline__ float rcp(float x) {  // 1 ulp
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// log(1 + e) for 0 <= e <= 1 as 2 atanh(s), s = e / (2 + e) <= 1/3: the series to s^13 leaves 1.4e-8 of the value
__device__ __forceinline__ float log1p01(float e) {
  const float s = e * rcp(2.f + e), z = s * s;
  float r = fmaf(z, 1.f / 13, 1.f / 11);
  r = fmaf(z, r, 1.f / 9);
  r = fmaf(z, r, 1.f / 7);
  r = fmaf(z, r, 1.f / 5);
  r = fmaf(z, r, 1.f / 3);
  r = fmaf(z, r, 1.f);
  return 2.f * s * r;
}
// softplus(x) = max(x, 0) + log(1 + e^-|x|) and sigmoid(x) from one exponential
__device__ __forceinline__ float softplus_and_sigmoid(float x, float& sig) {
  const float e = __expf(-fabsf(x)), r = rcp(1.f + e);
  sig = x >= 0.f ? r : e * r;
  return fmaxf(x, 0.f) + log1p01(e);
}
__device__ __forceinline__ float softplusf(float x) { return fmaxf(x, 0.f) + log1p01(__expf(-fabsf(x))); }

// x: raw beta logits (BF16 or FP32); y: FP32 (what the backward kernels read) and, optionally, BF16.
template <bool X_F32>
__global__ void __launch_bounds__(256) beta_sigmoid_fwd_kernel(const void* __restrict__ x, float* __restrict__ y32,
                                                                bf16* __restrict__ y16, long long n, float scale) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float xv = X_F32 ? static_cast<const float*>(x)[i] : bf2f(static_cast<const bf16*>(x)[i]);
    float y = scale * sigmoidf(xv);
    if (y16 != nullptr) {  // the forward's beta is rounded to the logits' dtype, as the reference's fused sigmoid returns it
      const bf16 yb = f2bf(y);
      y16[i] = yb;
      y = bf2f(yb);
    }
    if (y32 != nullptr) y32[i] = y;
  }
}
template <bool X_F32>
__global__ void __launch_bounds__(256) beta_sigmoid_bwd_kernel(const void* __restrict__ x, const float* __restrict__ dy,
                                                                float* __restrict__ dx, long long n, float scale) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float xv = X_F32 ? static_cast<const float*>(x)[i] : bf2f(static_cast<const bf16*>(x)[i]);
    const float s = sigmoidf(xv);
    dx[i] = dy[i] * scale * s * (1.f - s);
  }
}

// Both gate kernels: one CTA per (chunk, head) at a time, thread = (two adjacent channels, 16 consecutive tokens).  All of a
// thread's rows are requested before the first is used; with one thread per channel walking 64 tokens the loads of a chunk
// came in eight dependent batches.  Bound by instruction issue (softplus and sigmoid from one exponential and an own log(1 + e)).
// B=2 T=4096 H=16, BF16 input: forward 41 -> 23 us (floor at the HBM rate 15), backward 54 -> 39 us including the rounding of dx
// that was another pass of 9 us; with log1pf and a division per token 31 and 55 us.
constexpr int SEGS = 4, SEG = 64 / SEGS;  // token segments of a chunk

// Two adjacent values; VEC: in one access (every pointer 8-byte aligned), else one by one.
template <bool F32, bool VEC>
__device__ __forceinline__ float2 load2(const void* x, size_t at) {
  const float* f = static_cast<const float*>(x) + at;
  const bf16* b = static_cast<const bf16*>(x) + at;
  if (F32) return VEC ? *reinterpret_cast<const float2*>(f) : make_float2(f[0], f[1]);
  return VEC ? unpack_bf16(*reinterpret_cast<const uint32_t*>(b)) : make_float2(bf2f(b[0]), bf2f(b[1]));
}
template <bool F32, bool VEC>
__device__ __forceinline__ void store2(void* x, size_t at, float2 v) {
  float* f = static_cast<float*>(x) + at;
  bf16* b = static_cast<bf16*>(x) + at;
  if (F32 && VEC) *reinterpret_cast<float2*>(f) = v;
  else if (F32) { f[0] = v.x; f[1] = v.y; }
  else if (VEC) *reinterpret_cast<uint32_t*>(b) = pack_bf16(v.x, v.y);
  else { b[0] = f2bf(v.x); b[1] = f2bf(v.y); }
}

// Chunk-local inclusive cumulative sum of the per-step gate in log2 units, with the KDA gate activation optionally
// applied first.  ACT: g = -exp(A_log[h]) * softplus(x + dt_bias[h*128 + k]); otherwise x is the per-step natural-log gate.
template <bool ACT, bool X_F32, bool VEC>
__global__ void __launch_bounds__(256) gate_cumsum_fwd_kernel(const void* __restrict__ x, const float* __restrict__ A_log,
                                                               const float* __restrict__ dt_bias, float* __restrict__ out,
                                                               float* __restrict__ g_act, int T, int H, long long chunks_h) {
  __shared__ float2 total[SEGS][64];
  const int c = threadIdx.x & 63, seg = threadIdx.x >> 6;
  for (long long ch = blockIdx.x; ch < chunks_h; ch += gridDim.x) {   // ch = (b*NT + n)*H + h
    const int h = (int)(ch % H);
    const size_t ld = (size_t)H * 128, at = ((size_t)(ch / H) * 64 + seg * SEG) * ld + h * 128 + 2 * c;  // T is a multiple of 64
    const float a = ACT ? -__expf(A_log[h]) : 1.f;
    float2 bias = make_float2(0.f, 0.f), run = bias, g[SEG];
    if (ACT && dt_bias != nullptr) bias = make_float2(dt_bias[h * 128 + 2 * c], dt_bias[h * 128 + 2 * c + 1]);
#pragma unroll
    for (int t = 0; t < SEG; t++) g[t] = load2<X_F32, VEC>(x, at + t * ld);
#pragma unroll
    for (int t = 0; t < SEG; t++) {
      if (ACT) {
        g[t].x = a * softplusf(g[t].x + bias.x);
        g[t].y = a * softplusf(g[t].y + bias.y);
        if (g_act != nullptr) store2<true, VEC>(g_act, at + t * ld, g[t]);
      }
      run.x += g[t].x; run.y += g[t].y;
      g[t] = run;
    }
    total[seg][c] = run;
    __syncthreads();
    float2 off = make_float2(0.f, 0.f);
    for (int s = 0; s < seg; s++) { off.x += total[s][c].x; off.y += total[s][c].y; }
#pragma unroll
    for (int t = 0; t < SEG; t++)
      store2<true, VEC>(out, at + t * ld, make_float2((off.x + g[t].x) * RCP_LN2, (off.y + g[t].y) * RCP_LN2));
    __syncthreads();  // total is written again
  }
}

// Backward of the gate activation.  dg: gradient with respect to the activated per-step gate (FP32); dx in FP32 or, for BF16
// gate inputs, rounded to BF16 once.  Per-chunk partial sums of dA_log and ddt_bias go to dA_part[(b*NT+n)*H + h] and
// dbias_part[((b*NT+n)*H + h)*128 + k] (summed over the leading index by the caller, as FLA's kda_gate_bwd does).
template <bool X_F32, bool DX_F32, bool VEC>
__global__ void __launch_bounds__(256) gate_act_bwd_kernel(const void* __restrict__ x, const float* __restrict__ A_log,
                                                            const float* __restrict__ dt_bias, const float* __restrict__ dg,
                                                            void* __restrict__ dx, float* __restrict__ dA_part,
                                                            float* __restrict__ dbias_part, int H, long long chunks_h) {
  __shared__ float2 total[SEGS][64];
  __shared__ float red[8];
  const int c = threadIdx.x & 63, seg = threadIdx.x >> 6;
  for (long long ch = blockIdx.x; ch < chunks_h; ch += gridDim.x) {
    const int h = (int)(ch % H);
    const size_t ld = (size_t)H * 128, at = ((size_t)(ch / H) * 64 + seg * SEG) * ld + h * 128 + 2 * c;
    const float a = -__expf(A_log[h]);
    float2 bias = make_float2(0.f, 0.f), sb = bias;
    if (dt_bias != nullptr) bias = make_float2(dt_bias[h * 128 + 2 * c], dt_bias[h * 128 + 2 * c + 1]);
    float sa = 0.f;
    float2 xv[SEG], d[SEG];
#pragma unroll
    for (int t = 0; t < SEG; t++) {
      xv[t] = load2<X_F32, VEC>(x, at + t * ld);
      d[t] = load2<true, VEC>(dg, at + t * ld);
    }
#pragma unroll
    for (int t = 0; t < SEG; t++) {
      xv[t].x += bias.x; xv[t].y += bias.y;
      float2 sig, sp;
      sp.x = softplus_and_sigmoid(xv[t].x, sig.x);
      sp.y = softplus_and_sigmoid(xv[t].y, sig.y);
      const float2 gx = make_float2(a * d[t].x * sig.x, a * d[t].y * sig.y);
      store2<DX_F32, VEC>(dx, at + t * ld, gx);
      sb.x += gx.x; sb.y += gx.y;
      sa += d[t].x * a * sp.x + d[t].y * a * sp.y;
    }
    total[seg][c] = sb;
    sa = warp_sum(sa);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sa;
    __syncthreads();
    if (seg == 0) {
#pragma unroll
      for (int s = 1; s < SEGS; s++) { sb.x += total[s][c].x; sb.y += total[s][c].y; }
      store2<true, VEC>(dbias_part, (size_t)ch * 128 + 2 * c, sb);
    }
    if (threadIdx.x == 128) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; w++) s += red[w];
      dA_part[ch] = s;
    }
    __syncthreads();  // total and red are written again
  }
}

int grid_for(long long work_items, int per_block) {
  long long blocks = (work_items + per_block - 1) / per_block;
  const long long cap = 148ll * 16;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

bool bad16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }
bool bad8(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) != 0; }

}  // namespace
}  // namespace rewy

using namespace rewy;

#define WRAP_REQUIRE(ptr)                                                                                \
  do {                                                                                                   \
    if ((ptr) == nullptr) return report_error(REWY_ERR_NULL, "required pointer '" #ptr "' is NULL");      \
    if (bad16(ptr)) return report_error(REWY_ERR_ALIGN, "pointer '" #ptr "' is not 16-byte aligned");      \
  } while (0)

// f(a, b, c) with the three flags as types
template <class F>
static void choose(F&& f, bool a, bool b, bool c) {
  using Y = std::true_type;
  using N = std::false_type;
  auto last = [&](auto x, auto y) { c ? f(x, y, Y()) : f(x, y, N()); };
  auto mid = [&](auto x) { b ? last(x, Y()) : last(x, N()); };
  a ? mid(Y()) : mid(N());
}

static int finish(const char* what) {
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return REWY_OK;
  char msg[160];
  snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
  return report_error(REWY_ERR_LAUNCH, msg);
}

extern "C" int rewy_l2norm_fwd(const void* x, void* y, float* rstd, int64_t rows, float eps, rewy_stream_t st) {
  WRAP_REQUIRE(x); WRAP_REQUIRE(y); WRAP_REQUIRE(rstd);
  if (rows <= 0) return report_error(REWY_ERR_SHAPE, "rows must be positive");
  l2norm_fwd_kernel<<<grid_for(rows, 8), 256, 0, (cudaStream_t)st>>>((const bf16*)x, (bf16*)y, rstd, rows, eps);
  return finish("l2norm forward");
}

extern "C" int rewy_l2norm_bwd(const void* y, const float* rstd, const void* dy, int dy_is_f32, void* dx, int64_t rows,
                               rewy_stream_t st) {
  WRAP_REQUIRE(y); WRAP_REQUIRE(rstd); WRAP_REQUIRE(dy); WRAP_REQUIRE(dx);
  if (rows <= 0) return report_error(REWY_ERR_SHAPE, "rows must be positive");
  const int grid = grid_for(rows, 8);
  if (dy_is_f32)
    l2norm_bwd_kernel<true><<<grid, 256, 0, (cudaStream_t)st>>>((const bf16*)y, rstd, dy, (bf16*)dx, rows);
  else
    l2norm_bwd_kernel<false><<<grid, 256, 0, (cudaStream_t)st>>>((const bf16*)y, rstd, dy, (bf16*)dx, rows);
  return finish("l2norm backward");
}

extern "C" int rewy_beta_sigmoid_fwd(const void* x, int x_is_f32, float* y32, void* y16, int64_t n, float scale,
                                     rewy_stream_t st) {
  if (x == nullptr || (y32 == nullptr && y16 == nullptr)) return report_error(REWY_ERR_NULL, "x or both outputs are NULL");
  if (n <= 0) return report_error(REWY_ERR_SHAPE, "n must be positive");
  const int grid = grid_for(n, 256);
  if (x_is_f32)
    beta_sigmoid_fwd_kernel<true><<<grid, 256, 0, (cudaStream_t)st>>>(x, y32, (bf16*)y16, n, scale);
  else
    beta_sigmoid_fwd_kernel<false><<<grid, 256, 0, (cudaStream_t)st>>>(x, y32, (bf16*)y16, n, scale);
  return finish("beta sigmoid forward");
}

extern "C" int rewy_beta_sigmoid_bwd(const void* x, int x_is_f32, const float* dy, float* dx, int64_t n, float scale,
                                     rewy_stream_t st) {
  if (x == nullptr || dy == nullptr || dx == nullptr) return report_error(REWY_ERR_NULL, "x, dy or dx is NULL");
  if (n <= 0) return report_error(REWY_ERR_SHAPE, "n must be positive");
  const int grid = grid_for(n, 256);
  if (x_is_f32)
    beta_sigmoid_bwd_kernel<true><<<grid, 256, 0, (cudaStream_t)st>>>(x, dy, dx, n, scale);
  else
    beta_sigmoid_bwd_kernel<false><<<grid, 256, 0, (cudaStream_t)st>>>(x, dy, dx, n, scale);
  return finish("beta sigmoid backward");
}

extern "C" int rewy_gate_cumsum_fwd(const void* x, int x_is_f32, const float* A_log, const float* dt_bias, float* g_cumsum,
                                    float* g_act, int32_t B, int32_t T, int32_t H, rewy_stream_t st) {
  if (x == nullptr || g_cumsum == nullptr) return report_error(REWY_ERR_NULL, "x or g_cumsum is NULL");
  if (B <= 0 || H <= 0 || T < C || T % C != 0) return report_error(REWY_ERR_SHAPE, "bad B/T/H");
  const long long chunks_h = (long long)B * (T / C) * H;
  const int grid = (int)(chunks_h < 148ll * 64 ? chunks_h : 148ll * 64);
  cudaStream_t s = (cudaStream_t)st;
  auto go = [&](auto act, auto f32, auto vec) {
    gate_cumsum_fwd_kernel<act.value, f32.value, vec.value><<<grid, 256, 0, s>>>(x, A_log, dt_bias, g_cumsum, g_act, T, H, chunks_h);
  };
  choose(go, A_log != nullptr, x_is_f32 != 0, !(bad8(x) || bad8(g_cumsum) || bad8(g_act)));
  return finish("gate cumulative sum");
}

static int gate_act_bwd(const void* x, int x_is_f32, const float* A_log, const float* dt_bias, const float* dg, void* dx,
                        bool dx_is_f32, float* dA_part, float* dbias_part, int32_t B, int32_t T, int32_t H, rewy_stream_t st) {
  if (x == nullptr || A_log == nullptr || dg == nullptr || dx == nullptr || dA_part == nullptr || dbias_part == nullptr)
    return report_error(REWY_ERR_NULL, "a required pointer of the gate backward is NULL");
  if (B <= 0 || H <= 0 || T < C || T % C != 0) return report_error(REWY_ERR_SHAPE, "bad B/T/H");
  const long long chunks_h = (long long)B * (T / C) * H;
  const int grid = (int)(chunks_h < 148ll * 64 ? chunks_h : 148ll * 64);
  cudaStream_t s = (cudaStream_t)st;
  auto go = [&](auto f32, auto dx_f32, auto vec) {
    gate_act_bwd_kernel<f32.value, dx_f32.value, vec.value><<<grid, 256, 0, s>>>(x, A_log, dt_bias, dg, dx, dA_part, dbias_part, H, chunks_h);
  };
  choose(go, x_is_f32 != 0, dx_is_f32, !(bad8(x) || bad8(dg) || bad8(dx) || bad8(dbias_part)));
  return finish("gate activation backward");
}

extern "C" int rewy_gate_act_bwd(const void* x, int x_is_f32, const float* A_log, const float* dt_bias, const float* dg,
                                 float* dx, float* dA_part, float* dbias_part, int32_t B, int32_t T, int32_t H,
                                 rewy_stream_t st) {
  return gate_act_bwd(x, x_is_f32, A_log, dt_bias, dg, dx, true, dA_part, dbias_part, B, T, H, st);
}

extern "C" int rewy_gate_act_bwd_bf16(const void* x, int x_is_f32, const float* A_log, const float* dt_bias, const float* dg,
                                      void* dx, float* dA_part, float* dbias_part, int32_t B, int32_t T, int32_t H,
                                      rewy_stream_t st) {
  return gate_act_bwd(x, x_is_f32, A_log, dt_bias, dg, dx, false, dA_part, dbias_part, B, T, H, st);
}
