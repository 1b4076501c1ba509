// Forward pass of the four families: what the autograd forward needs besides the backward's own stages.
//
//   chunk_fwd_tc_kernel      (chunk_fwd_tc.cu) per chunk: Akk = (I + tril(E Y^T, -1))^-1, Aqk = scale tril(Qg Y^T),
//                            w = Akk E, u = Akk Z, qg, kg          (E = b k gamma, Y = k / gamma, Z = w v)
//   fwd_scan_tc_kernel       (state_scan_tc.cu, state_scan_split.cu) h[n], v_new, final state
//   chunk_output_tc_kernel   (chunk_output_tc.cu, tcgen05) o = scale qg h[n] + Aqk v_new; chunk_output_kernel here is its
//                            warp-MMA cross-check (rewy_set_forward_variant(1))
// Replaces FLA's chunk_kda_fwd / chunk_gdn2_fwd / chunk_gated_delta_rule_fwd / chunk_delta_rule_fwd as the reference
// binds them (src/fast_delta_rule/_compat/kda.py:89-113, gdn2.py:94-117, gdn.py:33-125, delta.py).
#include <atomic>
#include <cstdio>
#include "warp_mma.cuh"

namespace rewy {
namespace {

constexpr int LD128 = 136;  // padded pitch of a 128-wide BF16 tile
constexpr int LD64 = 72;    // padded pitch of a 64-wide BF16 tile

// o = scale * qg h[n] + Aqk v_new for one chunk.
__global__ void __launch_bounds__(256) chunk_output_kernel(const bf16* __restrict__ qg, const bf16* __restrict__ Aqk,
                                                           const bf16* __restrict__ v_new, const bf16* __restrict__ hst,
                                                           bf16* __restrict__ o, int T, int H, float scale) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* sQ = reinterpret_cast<bf16*>(smem_raw);  // [64][136] qg, later the output tile
  bf16* sV = sQ + C * LD128;                     // [64][136] v_new
  bf16* sA = sV + C * LD128;                     // [64][72]  Aqk
  bf16* sH = sA + C * LD64;                      // [128][136] h[n]
  const int n = blockIdx.x, bh = blockIdx.y, b = bh / H, h = bh % H, NT = T / C;
  const size_t row0 = (size_t)b * T + (size_t)n * C;
  const size_t ldt = (size_t)H * 128;
  const size_t base128 = (row0 * H + h) * 128;
  const size_t base64 = (row0 * H + h) * 64;
  load_tile_bf16<C, 128>(sQ, LD128, qg + base128, ldt);
  load_tile_bf16<C, 128>(sV, LD128, v_new + base128, ldt);
  load_tile_bf16<C, 64>(sA, LD64, Aqk + base64, (size_t)H * 64);
  load_tile_bf16<128, 128>(sH, LD128, hst + (((size_t)b * NT + n) * H + h) * 128 * 128, 128);
  __syncthreads();
  Tile<64, 128, 2, 4> acc;
  acc.zero();
  acc.mma<128>(Operand<false>{sQ, LD128}, Operand<true>{sH, LD128});
  acc.for_each([&](int, int, float& x) { x *= scale; });
  acc.mma<64>(Operand<false>{sA, LD64}, Operand<true>{sV, LD128});
  __syncthreads();  // every warp has read qg
  acc.for_each_pair([&](int r, int c, float& x0, float& x1) {
    *reinterpret_cast<uint32_t*>(sQ + r * LD128 + c) = pack_bf16(x0, x1);
  });
  __syncthreads();
  store_tile_bf16<C, 128>(o + base128, ldt, sQ, LD128);
}
constexpr size_t OUTPUT_SMEM = (size_t)(2 * C * LD128 + C * LD64 + 128 * LD128) * sizeof(bf16);

// chunk-local inclusive cumulative sum of a scalar per-head gate in log2 units: one thread per (chunk, head)
__global__ void __launch_bounds__(128) scalar_gate_cumsum_kernel(const void* __restrict__ x, int x_is_f32,
                                                                  float* __restrict__ out, int H, long long chunks_h) {
  const long long ch = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= chunks_h) return;
  const int h = (int)(ch % H);
  const long long row0 = (ch / H) * 64;
  float run = 0.f;
  for (int t = 0; t < 64; t++) {
    const long long at = (row0 + t) * H + h;
    run += x_is_f32 ? static_cast<const float*>(x)[at] : bf2f(static_cast<const bf16*>(x)[at]);
    out[at] = run * 1.4426950408889634f;
  }
}

bool bad16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

std::atomic<int> g_forward_variant{0};  // output kernel: 0 = TMA + tcgen05, 1 = warp-MMA (cross-check)

}  // namespace
}  // namespace rewy

using namespace rewy;

#define FWD_REQUIRE(field)                                                                                     \
  do {                                                                                                         \
    if (a->field == nullptr) return report_error(REWY_ERR_NULL, "required pointer '" #field "' is NULL");       \
    if (bad16(a->field)) return report_error(REWY_ERR_ALIGN, "pointer '" #field "' is not 16-byte aligned");     \
  } while (0)

extern "C" int rewy_chunk_fwd(const RewyFwdArgs* a, rewy_stream_t stream) {
  if (a == nullptr) return report_error(REWY_ERR_NULL, "args is NULL");
  if (a->family < REWY_DELTA || a->family > REWY_GDN2) return report_error(REWY_ERR_UNSUPPORTED, "unknown family");
  if (a->B <= 0 || a->H <= 0 || a->T < C || a->T % C != 0) return report_error(REWY_ERR_SHAPE, "bad B/T/H");
  if ((long long)a->B * a->H > 65535) return report_error(REWY_ERR_SHAPE, "B*H exceeds the grid limit 65535");
  if ((long long)a->B * a->T * a->H > REWY_MAX_TOKEN_HEADS)
    return report_error(REWY_ERR_SHAPE, "B*T*H exceeds 2^29 token-heads (32-bit tile coordinates)");
  if (a->state_v_first != 0 && a->state_v_first != 1) return report_error(REWY_ERR_UNSUPPORTED, "state_v_first must be 0 or 1");
  if (a->cu_seqlens != nullptr && (a->B != 1 || a->num_seqs <= 0 || (long long)a->num_seqs * a->H > 65535))
    return report_error(REWY_ERR_SHAPE, "packed sequences need B = 1 and 0 < num_seqs*H <= 65535");
  FWD_REQUIRE(q); FWD_REQUIRE(k); FWD_REQUIRE(v); FWD_REQUIRE(o); FWD_REQUIRE(Aqk); FWD_REQUIRE(Akk); FWD_REQUIRE(w);
  FWD_REQUIRE(u); FWD_REQUIRE(qg); FWD_REQUIRE(kg); FWD_REQUIRE(v_new); FWD_REQUIRE(h); FWD_REQUIRE(ctrl);
  if (a->family != REWY_DELTA) FWD_REQUIRE(g);
  if (a->family == REWY_GDN2) { FWD_REQUIRE(b_gate); FWD_REQUIRE(w_gate); }
  else FWD_REQUIRE(beta);
  if (a->h0 != nullptr && bad16(a->h0)) return report_error(REWY_ERR_ALIGN, "pointer 'h0' is not 16-byte aligned");
  if (a->final_state != nullptr && bad16(a->final_state))
    return report_error(REWY_ERR_ALIGN, "pointer 'final_state' is not 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(a->ctrl, 0, sizeof(int), st);
  if (e == cudaSuccess) e = launch_chunk_fwd_tc(*a, static_cast<int*>(a->ctrl), st);
  if (e == cudaSuccess) {
    RewyBwdArgs ba{};
    ba.family = a->family; ba.B = a->B; ba.T = a->T; ba.H = a->H; ba.state_v_first = a->state_v_first; ba.scale = a->scale;
    ba.g = a->g; ba.h0 = a->h0; ba.cu_seqlens = a->cu_seqlens; ba.num_seqs = a->num_seqs;
    RewyStageBuffers sb{};
    sb.w = a->w; sb.u = a->u; sb.kg = a->kg; sb.h = a->h; sb.v_new = a->v_new;
    e = launch_fwd_scan_tc(ba, sb, static_cast<int*>(a->ctrl), st, a->final_state);
  }
  if (e == cudaSuccess && g_forward_variant.load(std::memory_order_relaxed) == 0) {
    e = launch_chunk_output_tc(*a, static_cast<int*>(a->ctrl), st);
  } else if (e == cudaSuccess) {
    e = ensure_dynamic_smem<chunk_output_kernel>(OUTPUT_SMEM);
    if (e == cudaSuccess) {
      dim3 grid(a->T / C, a->B * a->H);
      chunk_output_kernel<<<grid, 256, OUTPUT_SMEM, st>>>((const bf16*)a->qg, (const bf16*)a->Aqk, (const bf16*)a->v_new,
                                                         (const bf16*)a->h, (bf16*)a->o, a->T, a->H, a->scale);
      count_launch();
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) {
    char msg[160];
    snprintf(msg, sizeof(msg), "chunk forward: %s", cudaGetErrorString(e));
    return report_error(REWY_ERR_LAUNCH, msg);
  }
  return REWY_OK;
}

extern "C" int rewy_set_forward_variant(int variant) {
  if (variant != 0 && variant != 1) return report_error(REWY_ERR_UNSUPPORTED, "forward variant must be 0 or 1");
  g_forward_variant.store(variant, std::memory_order_relaxed);
  return REWY_OK;
}

extern "C" int rewy_scalar_gate_cumsum_fwd(const void* x, int x_is_f32, float* g_cumsum, int32_t B, int32_t T, int32_t H,
                                           rewy_stream_t stream) {
  if (x == nullptr || g_cumsum == nullptr) return report_error(REWY_ERR_NULL, "x or g_cumsum is NULL");
  if (B <= 0 || H <= 0 || T < C || T % C != 0) return report_error(REWY_ERR_SHAPE, "bad B/T/H");
  const long long chunks_h = (long long)B * (T / C) * H;
  scalar_gate_cumsum_kernel<<<(unsigned)((chunks_h + 127) / 128), 128, 0, (cudaStream_t)stream>>>(x, x_is_f32, g_cumsum, H,
                                                                                                 chunks_h);
  count_launch();
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return report_error(REWY_ERR_LAUNCH, cudaGetErrorString(e));
  return REWY_OK;
}
