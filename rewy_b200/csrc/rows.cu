// Row movement around the family operators: lengths that are not multiples of the 64-token chunk and grouped value heads.
//
//   rewy_rows_pad / _cut   tensors [.., tokens, ..] between the caller's token rows and the padded rows the kernels work on
//                          (every sequence extended to the next multiple of 64; the added rows hold a fill value)
//   rewy_qk_front_fwd/bwd  q and k together: optional L2 normalisation, padding and the repeat to the value heads in one
//                          pass; backward: sum over the heads of a group in FP32, normalisation backward, cut, one rounding
// FLA reaches these cases by bounds checks and head arithmetic inside its kernels; the reference's release envelope
// rejects them (src/fast_delta_rule/runtime.py:84-88).
//
// One pass over each tensor, bound by HBM: one warp per row (per row and head in the front kernels) with the widest
// accesses that the row's size and the pointers allow, up to eight tensors per launch.
// Measured against the tensor operations before (cat / index_copy / index_select / repeat / reduce and two normalisation
// kernels), DeltaNet, 12 packed sequences of 16001 tokens, 8 heads: 480 us in 24 launches -> 162 us in 6; GDN, 2 groups,
// B=2 T=4096, 32 value heads: 404 us in 8 launches -> 124 us in 2.  Half a warp per (row, head) and two items in flight
// against one warp and one item: front backward 105 -> 60 us, forward 60 -> 40 us (packed case; 16 and 64 CTAs per SM of
// grid measured for both, the better one taken). 
#include <cstdio>
#include "common.cuh"

namespace rewy {
namespace {

// caller's token row <-> padded token row; -1: no counterpart
struct RowMap {
  int B, T, Tp, nseq;
  const int *cu, *cup;  // packed: offsets of the sequences among the caller's rows and among the padded rows
};
__device__ __forceinline__ int sequence_of(const int* off, int nseq, int row) {  // the last s with off[s] <= row
  int lo = 0, hi = nseq;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= row) lo = mid; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ int caller_row(const RowMap& m, int row) {
  if (m.cu == nullptr) {
    if (m.T == m.Tp) return row;
    const int b = row / m.Tp, t = row - b * m.Tp;
    return t < m.T ? b * m.T + t : -1;
  }
  const int s = sequence_of(m.cup, m.nseq, row), at = m.cu[s] + row - m.cup[s];
  return at < m.cu[s + 1] ? at : -1;
}
__device__ __forceinline__ int padded_row(const RowMap& m, int row) {
  if (m.cu == nullptr) {
    if (m.T == m.Tp) return row;
    const int b = row / m.T;
    return b * m.Tp + row - b * m.T;
  }
  const int s = sequence_of(m.cu, m.nseq, row);
  return row < m.cu[s + 1] ? m.cup[s] + row - m.cu[s] : -1;
}

struct RowItems {
  RewyRowsItem it[REWY_MAX_ROWS_ITEMS];
  int unit[REWY_MAX_ROWS_ITEMS];  // bytes per access: 16, 8, 4, 2 or 1
};

template <class U>
__device__ __forceinline__ void move_row(const RewyRowsItem& it, long long dst, long long src, int lane) {
  const int n = (int)(it.row_bytes / sizeof(U));
  U* d = reinterpret_cast<U*>(static_cast<char*>(it.dst) + dst * it.row_bytes);
  if (src >= 0) {
    const U* s = reinterpret_cast<const U*>(static_cast<const char*>(it.src) + src * it.row_bytes);
#pragma unroll 4
    for (int i = lane; i < n; i += 32) d[i] = s[i];
  } else {
    U f;
    unsigned long long w[(sizeof(U) + 7) / 8];
    for (int i = 0; i < (int)(sizeof(w) / 8); i++) w[i] = it.fill;
    memcpy(&f, w, sizeof(U));
    for (int i = lane; i < n; i += 32) d[i] = f;
  }
}

template <bool PAD>
__global__ void __launch_bounds__(256) rows_kernel(const __grid_constant__ RowItems items, const RowMap m, int rows) {
  const RewyRowsItem& it = items.it[blockIdx.y];
  const int unit = items.unit[blockIdx.y], lane = threadIdx.x & 31;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
    const long long src = PAD ? caller_row(m, r) : padded_row(m, r);
    switch (unit) {
      case 16: move_row<uint4>(it, r, src, lane); break;
      case 8: move_row<uint2>(it, r, src, lane); break;
      case 4: move_row<uint32_t>(it, r, src, lane); break;
      case 2: move_row<uint16_t>(it, r, src, lane); break;
      default: move_row<uint8_t>(it, r, src, lane); break;
    }
  }
}

// sum_i a[i] b[i] over the 16 lanes of a half warp, in the order of the normalisation kernels in wrappers.cu (a whole warp, four
// channels per lane: lanes 2l and 2l+1 there are the two halves of lane l here, and meet last)
__device__ __forceinline__ float half_dot(const float (&a)[8], const float (&b)[8]) {
  float lo = dot4(a, b), hi = dot4(a + 4, b + 4);
#pragma unroll
  for (int m = 8; m > 0; m >>= 1) {
    lo += __shfl_xor_sync(0xffffffffu, lo, m);
    hi += __shfl_xor_sync(0xffffffffu, hi, m);
  }
  return lo + hi;
}
__device__ __forceinline__ void unpack8(const uint4& r, float (&x)[8]) {
  const uint32_t u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = unpack_bf16(u[i]);
    x[2 * i] = f.x; x[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
}

struct FrontParams {
  const bf16* x[2];  // caller's q, k [rows, H, 128]
  bf16* y[2];        // [padded rows, H * G, 128]
  float* rstd[2];    // [padded rows, H], or NULL: no normalisation
  const void* dy[2]; // gradient of y
  bf16* dx[2];       // gradient of x
  int H, G;
  float eps;
};

// Half a warp per (row, head), lane l of it owns channels 8l .. 8l+7; a warp takes ITEMS of them per half at a time, so
// that its loads are in flight together.  blockIdx.y: q or k.
constexpr int ITEMS = 2;

__global__ void __launch_bounds__(256) qk_front_fwd_kernel(const FrontParams p, const RowMap m, unsigned total) {
  const int lane = threadIdx.x & 15, z = blockIdx.y;
  const unsigned H = p.H, half = blockIdx.x * 16 + (threadIdx.x >> 4), halves = gridDim.x * 16;
  float* rstd = p.rstd[z];
  for (unsigned i0 = half & ~1u; i0 < total; i0 += halves * ITEMS) {  // both halves of a warp leave together
    uint4 u[ITEMS];
    unsigned at[ITEMS];
#pragma unroll
    for (int n = 0; n < ITEMS; n++) {
      at[n] = i0 + (half & 1u) + n * halves;
      u[n] = make_uint4(0, 0, 0, 0);
      if (at[n] < total) {
        const unsigned row = at[n] / H, h = at[n] - row * H;
        const int src = caller_row(m, (int)row);
        if (src >= 0) u[n] = *reinterpret_cast<const uint4*>(p.x[z] + ((size_t)src * H + h) * 128 + 8 * lane);
      }
    }
#pragma unroll
    for (int n = 0; n < ITEMS; n++) {
      if (rstd != nullptr) {
        float x[8];
        unpack8(u[n], x);
        const float rs = rsqrtf(half_dot(x, x) + p.eps);
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] *= rs;
        u[n] = pack8(x);
        if (lane == 0 && at[n] < total) rstd[at[n]] = rs;
      }
      if (at[n] < total) {
        bf16* y = p.y[z] + (size_t)at[n] * p.G * 128 + 8 * lane;  // heads h G .. h G + G - 1 of the row
        for (int j = 0; j < p.G; j++) *reinterpret_cast<uint4*>(y + j * 128) = u[n];
      }
    }
  }
}

template <bool DY_F32>
struct Grad8 {  // eight channels of dy as they are in memory
  uint4 a, b;
  __device__ __forceinline__ void load(const void* dy, size_t at) {
    const uint4* d = reinterpret_cast<const uint4*>(static_cast<const char*>(dy) + at * (DY_F32 ? 4 : 2));
    a = d[0];
    if (DY_F32) b = d[1];
  }
  __device__ __forceinline__ void get(float (&t)[8]) const {
    if (DY_F32) {
      t[0] = __uint_as_float(a.x); t[1] = __uint_as_float(a.y); t[2] = __uint_as_float(a.z); t[3] = __uint_as_float(a.w);
      t[4] = __uint_as_float(b.x); t[5] = __uint_as_float(b.y); t[6] = __uint_as_float(b.z); t[7] = __uint_as_float(b.w);
    } else {
      unpack8(a, t);
    }
  }
};

template <bool DY_F32>
__global__ void __launch_bounds__(256) qk_front_bwd_kernel(const FrontParams p, const RowMap m, unsigned total) {
  const int lane = threadIdx.x & 15, z = blockIdx.y;
  const unsigned H = p.H, half = blockIdx.x * 16 + (threadIdx.x >> 4), halves = gridDim.x * 16;
  const float* rstd = p.rstd[z];
  for (unsigned i0 = half & ~1u; i0 < total; i0 += halves * ITEMS) {
    Grad8<DY_F32> d[ITEMS];
    float rs[ITEMS];
    uint4 yv[ITEMS];
    size_t at[ITEMS];
    bool real[ITEMS];
#pragma unroll
    for (int n = 0; n < ITEMS; n++) {
      const unsigned item = i0 + (half & 1u) + n * halves;
      d[n].a = d[n].b = yv[n] = make_uint4(0, 0, 0, 0);
      rs[n] = 0.f;
      real[n] = false;
      if (item < total) {
        const unsigned row = item / H, h = item - row * H;
        const int src = padded_row(m, (int)row);
        if (src >= 0) {
          const size_t ph = (size_t)src * H + h;
          real[n] = true;
          at[n] = ph * p.G * 128 + 8 * lane;
          d[n].load(p.dy[z], at[n]);
          if (rstd != nullptr) {
            yv[n] = *reinterpret_cast<const uint4*>(p.y[z] + at[n]);  // the copies of a group share y
            rs[n] = rstd[ph];
          }
        }
      }
    }
#pragma unroll
    for (int n = 0; n < ITEMS; n++) {
      const unsigned item = i0 + (half & 1u) + n * halves;
      float g[8];
      d[n].get(g);
      if (real[n]) {
        for (int j = 1; j < p.G; j++) {
          Grad8<DY_F32> more;
          float t[8];
          more.load(p.dy[z], at[n] + j * 128);
          more.get(t);
#pragma unroll
          for (int e = 0; e < 8; e++) g[e] += t[e];
        }
      }
      if (rstd != nullptr) {  // dx = (dy - y <dy, y>) rstd
        float y[8];
        unpack8(yv[n], y);
        const float s = half_dot(g, y);
#pragma unroll
        for (int j = 0; j < 8; j++) g[j] = fmaf(-y[j], s, g[j]) * rs[n];
      }
      if (item < total) *reinterpret_cast<uint4*>(p.dx[z] + (size_t)item * 128 + 8 * lane) = pack8(g);
    }
  }
}

bool bad16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }
int grid_for(long long work, int per_block, int per_sm) {
  const long long blocks = (work + per_block - 1) / per_block, cap = 148ll * per_sm;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

// fills m; B = 1 and both offset arrays when packed
int make_map(const RewyRowMap* r, RowMap& m) {
  if (r == nullptr) return report_error(REWY_ERR_NULL, "row map is NULL");
  if (r->B <= 0 || r->T <= 0 || r->T_padded < r->T || (long long)r->B * r->T_padded > 0x7fffffffll)
    return report_error(REWY_ERR_SHAPE, "bad row map");
  if ((r->cu == nullptr) != (r->cu_padded == nullptr) || (r->cu != nullptr && (r->B != 1 || r->num_seqs <= 0)))
    return report_error(REWY_ERR_SHAPE, "packed rows need B = 1, num_seqs > 0 and both offset arrays");
  m.B = r->B; m.T = r->T; m.Tp = r->T_padded; m.nseq = r->num_seqs; m.cu = r->cu; m.cup = r->cu_padded;
  return REWY_OK;
}

int finish(const char* what) {
  count_launch();
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return REWY_OK;
  char msg[160];
  snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
  return report_error(REWY_ERR_LAUNCH, msg);
}

template <bool PAD>
int move_rows(const RewyRowMap* map, const RewyRowsItem* items, int n, cudaStream_t st) {
  RowMap m;
  const int rc = make_map(map, m);
  if (rc != REWY_OK) return rc;
  if (items == nullptr || n <= 0 || n > REWY_MAX_ROWS_ITEMS) return report_error(REWY_ERR_SHAPE, "1 to 8 row tensors per call");
  RowItems ri;
  for (int i = 0; i < n; i++) {
    if (items[i].src == nullptr || items[i].dst == nullptr) return report_error(REWY_ERR_NULL, "row tensor is NULL");
    if (items[i].row_bytes <= 0 || items[i].row_bytes > 0x7fffffffll) return report_error(REWY_ERR_SHAPE, "bad row size");
    ri.it[i] = items[i];
    const uintptr_t mix = reinterpret_cast<uintptr_t>(items[i].src) | reinterpret_cast<uintptr_t>(items[i].dst) |
                          (uintptr_t)items[i].row_bytes;
    ri.unit[i] = (mix & 15) == 0 ? 16 : (mix & 7) == 0 ? 8 : (mix & 3) == 0 ? 4 : (mix & 1) == 0 ? 2 : 1;
  }
  const int rows = PAD ? m.B * m.Tp : m.B * m.T;
  rows_kernel<PAD><<<dim3(grid_for(rows, 8, 16), n), 256, 0, st>>>(ri, m, rows);
  return finish(PAD ? "row padding" : "row cut");
}

}  // namespace
}  // namespace rewy

using namespace rewy;

extern "C" int rewy_rows_pad(const RewyRowMap* map, const RewyRowsItem* items, int32_t n, rewy_stream_t st) {
  return move_rows<true>(map, items, n, (cudaStream_t)st);
}
extern "C" int rewy_rows_cut(const RewyRowMap* map, const RewyRowsItem* items, int32_t n, rewy_stream_t st) {
  return move_rows<false>(map, items, n, (cudaStream_t)st);
}

static int front_common(const RewyRowMap* map, int32_t H, int32_t G, RowMap& m) {
  const int rc = make_map(map, m);
  if (rc != REWY_OK) return rc;
  if (H <= 0 || G <= 0 || (long long)m.B * m.Tp * H * G > REWY_MAX_TOKEN_HEADS)
    return report_error(REWY_ERR_SHAPE, "bad head counts, or more than 2^29 token-heads");
  return REWY_OK;
}

extern "C" int rewy_qk_front_fwd(const RewyRowMap* map, const void* q, const void* k, void* yq, void* yk, float* rq, float* rk,
                                 int32_t H, int32_t G, float eps, rewy_stream_t st) {
  RowMap m;
  const int rc = front_common(map, H, G, m);
  if (rc != REWY_OK) return rc;
  if (q == nullptr || k == nullptr || yq == nullptr || yk == nullptr || (rq == nullptr) != (rk == nullptr))
    return report_error(REWY_ERR_NULL, "a required pointer of the q/k front is NULL");
  if (bad16(q) || bad16(k) || bad16(yq) || bad16(yk)) return report_error(REWY_ERR_ALIGN, "q/k front: pointers must be 16-byte aligned");
  FrontParams p{};
  p.x[0] = (const bf16*)q; p.x[1] = (const bf16*)k; p.y[0] = (bf16*)yq; p.y[1] = (bf16*)yk; p.rstd[0] = rq; p.rstd[1] = rk;
  p.H = H; p.G = G; p.eps = eps;
  const unsigned total = (unsigned)m.B * m.Tp * H;
  qk_front_fwd_kernel<<<dim3(grid_for(total, 16 * ITEMS, 16), 2), 256, 0, (cudaStream_t)st>>>(p, m, total);
  return finish("q/k front");
}

extern "C" int rewy_qk_front_bwd(const RewyRowMap* map, const void* yq, const void* yk, const float* rq, const float* rk,
                                 const void* dyq, const void* dyk, int32_t dy_is_f32, void* dq, void* dk, int32_t H, int32_t G,
                                 rewy_stream_t st) {
  RowMap m;
  const int rc = front_common(map, H, G, m);
  if (rc != REWY_OK) return rc;
  if (dyq == nullptr || dyk == nullptr || dq == nullptr || dk == nullptr || (rq == nullptr) != (rk == nullptr) ||
      (rq != nullptr && (yq == nullptr || yk == nullptr)))
    return report_error(REWY_ERR_NULL, "a required pointer of the q/k front backward is NULL");
  if (bad16(yq) || bad16(yk) || bad16(dyq) || bad16(dyk) || bad16(dq) || bad16(dk))
    return report_error(REWY_ERR_ALIGN, "q/k front backward: pointers must be 16-byte aligned");
  FrontParams p{};
  p.y[0] = (bf16*)yq; p.y[1] = (bf16*)yk; p.rstd[0] = (float*)rq; p.rstd[1] = (float*)rk; p.dy[0] = dyq; p.dy[1] = dyk;
  p.dx[0] = (bf16*)dq; p.dx[1] = (bf16*)dk; p.H = H; p.G = G;
  const unsigned total = (unsigned)m.B * m.T * H;
  const dim3 grid(grid_for(total, 16 * ITEMS, 64), 2);
  if (dy_is_f32) qk_front_bwd_kernel<true><<<grid, 256, 0, (cudaStream_t)st>>>(p, m, total);
  else qk_front_bwd_kernel<false><<<grid, 256, 0, (cudaStream_t)st>>>(p, m, total);
  return finish("q/k front backward");
}
