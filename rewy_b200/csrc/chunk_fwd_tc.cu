// Chunk-local forward stage on the Blackwell tensor cores: Akk, Aqk, w, u, qg, kg of every chunk (definitions and the
// reference functions it replaces: chunk_fwd.cu).
//
// Persistent, two CTAs of 256 threads per SM; per chunk:
//   * TMA brings q and k (one 128-row operand [q ; k]), g, later v;
//   * vector gate: thread (row of [q ; k], 64 channels) turns its row into Qc = q alpha or Ec = b k alpha, BF16 hi and
//     lo, written straight into TENSOR MEMORY as the A operand; the q rows also write Yc = k / alpha (hi, lo) as the
//     shared-memory B operand;
//   * [Qc ; Ec] Yc^T is ONE M=128 product in three hi/lo passes (scalar gate / none: [q ; k] k^T, exact, one pass, on
//     the tiles as they landed): lanes 0..63 give Aqk, lanes 64..127 the matrix to invert.  While it runs qg and kg
//     leave in 16-byte pieces and E = b k gamma takes the place of k;
//   * (I + L)^-1 in FP32 by blocks 16 -> 32 -> 64 with all threads: X21 = -X22 (L21 X11);
//   * w = Akk E and u = Akk Z with Akk stored twice (M=128), so that lanes 0..63 finish w and lanes 64..127 u.
// A chunk outside the range of the centred factors (common.cuh) uses none: its two matrices are summed pair by pair here.
// The loops are kept rolled (two deep): a chunk's code runs once per chunk, and with everything unrolled the warps waited
// for instructions more than for anything else (1.9 of 10 cycles per issued instruction, more than for memory).
// Measured, against the warp-MMA kernel before it (three passes over the inputs, inverse by 64 threads): KDA B=1 T=8192
// H=32 336 -> 217 us (222 since the range of q and k is looked at where the gate spans 80), GDN B=2 T=4096 H=32 202 -> 148
// us, GDN2 B=2 T=2048 H=8 68 -> 41 us.  Unrolled: 251, 150, 45; with 512 threads per CTA: 237, 167, 41 (more instructions
// per result in the inverse).  Bound by instruction issue of the operand pass and by the inverse's chain (5000 of 16000
// cycles of a chunk without a vector gate).
#include "phase_log.cuh"
#include "tc05.cuh"

namespace rewy {
namespace {
using namespace tc;

constexpr int TPB = 256;
constexpr int NG = TPB / 128;  // column groups: a thread has 1/NG of its TMEM lane's columns
constexpr int LDL = 68;  // pitch of the FP32 matrix (16-byte rows, conflict-free by rows and by columns of four)
constexpr unsigned long long DRAIN_NS = 20ull * 1000 * 1000;

struct LocalParams {
  const float *g, *beta;
  const bf16 *bg, *wg;
  bf16 *Akk, *Aqk, *qg, *kg;
  int* err;
  int T, H, NT, total_chunks;
  int write_qk;  // 0: no gate and the caller's qg, kg are q and k themselves
  float scale;
};

// Shared-memory plan, byte offsets from a 1024-byte aligned base.  128-byte-swizzled BF16 panels of 64 rows are 8 KB.
struct LS {
  static constexpr uint32_t QK = 0;                // [q ; k] panel 0 (q 8 KB, k 8 KB), panel 1           32 KB
  static constexpr uint32_t KT = QK + 8192;        // k panels, 16 KB apart; become E, then w
  static constexpr uint32_t G = QK + 32768;        // vector gate: 4 panels [64 t][32 k] FP32              32 KB
  static constexpr uint32_t Y = G + 32768;         // Yc hi panels, lo panels                              32 KB
  static constexpr uint32_t L = Y;                 // over Yc: FP32 [64][68]: L, then (I + L)^-1           17 KB
  static constexpr uint32_t AK = L + 64 * LDL * 4; //          Akk twice: 128 rows K-major                 16 KB
  static constexpr uint32_t CEN = AK + 16384;      // float[128] centre of the gate
  static constexpr uint32_t GL = CEN + 512;        // float[128] last gate row
  static constexpr uint32_t MM = GL + 512;         // float[NG][2][128] min / max of the row groups
  static constexpr uint32_t BETA = MM + NG * 1024; // float[64]
  static constexpr uint32_t GS = BETA + 256;       // float[64] scalar gate rows
  static constexpr uint32_t BARS = GS + 256;
  static constexpr uint32_t TMEM = BARS + 64;
  static constexpr uint32_t TOTAL = TMEM + 64;
};
// v panels (then Z, then u): over q with a vector gate (pitch 16 KB), else where the gate tile would be (8 KB)
template <int GATE> struct VPlace {
  static constexpr uint32_t AT = GATE == GATE_VECTOR ? LS::QK : LS::G, PITCH = GATE == GATE_VECTOR ? 16384 : 8192;
};
static_assert(LS::AK % 1024 == 0 && LS::AK + 16384 >= LS::Y + 32768, "operand tiles on swizzle atoms, behind Yc");
static_assert(2 * (LS::TOTAL + 1024) <= 233472, "two forward chunk CTAs must fit one SM");
// TMEM columns: A operand hi / lo and the accumulator of the first product; then w and u
constexpr uint32_t TM_A = 0, TM_D = 128, TM_W = 0, TM_U = 128;
enum { LB_G = 0, LB_QK, LB_V, LB_D, LB_WU, LB_COUNT };

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&r)[16]) {
  uint32_t u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) r[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void split8(const float (&x)[8], uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    __nv_bfloat162 hh = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
    const float2 hf = __bfloat1622float2(hh);
    h[i] = *reinterpret_cast<uint32_t*>(&hh);
    l[i] = pack_bf16(x[2 * i] - hf.x, x[2 * i + 1] - hf.y);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  return make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
}
__device__ __forceinline__ void unpack8(const uint4& r, float (&x)[8]) {
  const uint32_t u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 f = unpack_bf16(u[i]);
    x[2 * i] = f.x; x[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load8(const unsigned char* a, const unsigned char* b, float (&x)[8]) {
  const float4 p = *reinterpret_cast<const float4*>(a), q = *reinterpret_cast<const float4*>(b);
  x[0] = p.x; x[1] = p.y; x[2] = p.z; x[3] = p.w; x[4] = q.x; x[5] = q.y; x[6] = q.z; x[7] = q.w;
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint4& v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(c0),
               "r"(c1)
               : "memory");
}

// sL holds L strictly below the diagonal of a unit lower triangular 64 x 64 matrix and zeros above; on return its lower
// triangle is the inverse (the upper right 32 x 32 block is scratch).  All 256 threads; FP32 throughout.
__device__ __forceinline__ void invert_unit_lower(float* sL, int tid) {
  if (tid < C) {  // four 16 x 16 diagonal blocks, one column per thread
    float* blk = sL + (tid >> 4) * 16 * (LDL + 1);
    const int c = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int j = 0; j < i; j += 4) {
        const float4 l4 = *reinterpret_cast<const float4*>(blk + i * LDL + j);
        s0 = fmaf(l4.x, x[j], s0);
        if (j + 1 < i) s1 = fmaf(l4.y, x[j + 1], s1);
        if (j + 2 < i) s0 = fmaf(l4.z, x[j + 2], s0);
        if (j + 3 < i) s1 = fmaf(l4.w, x[j + 3], s1);
      }
      x[i] = (i == c ? 1.f : 0.f) - (s0 + s1);
    }
    __syncwarp();  // a block's sixteen threads share a warp: all have read it
#pragma unroll
    for (int i = 0; i < 16; i++) blk[i * LDL + c] = x[i];
  }
  __syncthreads();
  {  // 16 -> 32: two pairs of blocks, two columns per thread
    const int p = tid >> 7, i = (tid >> 3) & 15, c = (tid & 7) * 2;
    float* base = sL + 32 * p * (LDL + 1);         // X11; X22 16 further along the diagonal, L21 below X11
    float* tmp = sL + (16 * p) * LDL + 32;         // scratch 16 x 16
    float a0 = 0.f, a1 = 0.f;
#pragma unroll 2
    for (int k = 0; k < 16; k += 4) {
      const float4 l4 = *reinterpret_cast<const float4*>(base + (16 + i) * LDL + k);
      const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float2 b = *reinterpret_cast<const float2*>(base + (k + e) * LDL + c);
        a0 = fmaf(l[e], b.x, a0);
        a1 = fmaf(l[e], b.y, a1);
      }
    }
    *reinterpret_cast<float2*>(tmp + i * LDL + c) = make_float2(a0, a1);
    __syncthreads();
    a0 = a1 = 0.f;
#pragma unroll 2
    for (int k = 0; k < 16; k += 4) {
      const float4 l4 = *reinterpret_cast<const float4*>(base + (16 + i) * LDL + 16 + k);
      const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float2 b = *reinterpret_cast<const float2*>(tmp + (k + e) * LDL + c);
        a0 = fmaf(l[e], b.x, a0);
        a1 = fmaf(l[e], b.y, a1);
      }
    }
    *reinterpret_cast<float2*>(base + (16 + i) * LDL + c) = make_float2(-a0, -a1);
    __syncthreads();
  }
  {  // 32 -> 64: four columns per thread
    const int i = tid >> 3, c = (tid & 7) * 4;
    float* tmp = sL + 32;  // rows 0..31, columns 32..63
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int k = 0; k < 32; k += 4) {
      const float4 l4 = *reinterpret_cast<const float4*>(sL + (32 + i) * LDL + k);
      const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float4 b = *reinterpret_cast<const float4*>(sL + (k + e) * LDL + c);
        a.x = fmaf(l[e], b.x, a.x); a.y = fmaf(l[e], b.y, a.y); a.z = fmaf(l[e], b.z, a.z); a.w = fmaf(l[e], b.w, a.w);
      }
    }
    *reinterpret_cast<float4*>(tmp + i * LDL + c) = a;
    __syncthreads();
    a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int k = 0; k < 32; k += 4) {
      const float4 l4 = *reinterpret_cast<const float4*>(sL + (32 + i) * LDL + 32 + k);
      const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float4 b = *reinterpret_cast<const float4*>(tmp + (k + e) * LDL + c);
        a.x = fmaf(l[e], b.x, a.x); a.y = fmaf(l[e], b.y, a.y); a.z = fmaf(l[e], b.z, a.z); a.w = fmaf(l[e], b.w, a.w);
      }
    }
    *reinterpret_cast<float4*>(sL + (32 + i) * LDL + c) = make_float4(-a.x, -a.y, -a.z, -a.w);
    __syncthreads();
  }
}

template <int GATE, bool VB>
__global__ void __launch_bounds__(TPB, 2)
chunk_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmG,
                    const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmU, const LocalParams p) {
  extern __shared__ __align__(1024) unsigned char sm[];
  constexpr bool VEC = GATE == GATE_VECTOR;
  constexpr uint32_t VT = VPlace<GATE>::AT, VP = VPlace<GATE>::PITCH;
  float* sL = reinterpret_cast<float*>(sm + LS::L);
  float* sCen = reinterpret_cast<float*>(sm + LS::CEN);
  float* sGl = reinterpret_cast<float*>(sm + LS::GL);
  float* sMM = reinterpret_cast<float*>(sm + LS::MM);
  float* sBeta = reinterpret_cast<float*>(sm + LS::BETA);
  float* sGs = reinterpret_cast<float*>(sm + LS::GS);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + LS::BARS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + LS::TMEM);
  const uint32_t sb = smem_u32(sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = p.T, H = p.H, NT = p.NT;
  const size_t ldt = (size_t)H * 128;
  if ((sb & 1023u) != 0) {  // the plan needs a 1024-byte aligned base
    if (tid == 0) atomicCAS(p.err, 0, 40);
    return;
  }
  // thread = (row t of q or k, half of the columns): TMEM lanes 0..63 are rows of q, 64..127 rows of k
  const int t = (warp & 1) * 32 + lane, krow = (warp >> 1) & 1, wg = warp >> 2;

  if (tid == 0) {
    for (int i = 0; i < LB_COUNT; i++) mbar_init(&bars[i], 1);
    fence_barrier_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV); prefetch_tmap(&tmW); prefetch_tmap(&tmU);
    if (VEC) prefetch_tmap(&tmG);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tb = *tmem_slot;
  const uint32_t tlane = tb + ((uint32_t)((warp & 3) * 32) << 16);
  const bool leader = warp == 0 && elect_one();
  uint32_t ph = 0;
  PhaseLog log;  // what the leader has asked for
  bool alive = true;
  auto wait = [&](int b, int code) {
    if (alive) alive = mbar_wait(&bars[b], ph, p.err, code);  // every barrier in use completes once per chunk
  };
  auto dl = [&](uint32_t off, uint32_t lbo) { return desc_lo(sb + off, lbo); };
  struct Where { int h, row0; };
  auto where = [&](int chunk) {
    const int bn = chunk / H, h = chunk - bn * H, b = bn / NT, n = bn - b * NT;  // head fastest
    return Where{h, b * T + n * C};
  };
  auto load_g = [&](int chunk) {
    const Where w = where(chunk);
    log.request(LB_G);
    mbar_expect_tx(&bars[LB_G], 32768);
    tma_load_3d(sm + LS::G, &tmG, w.h * 128, w.row0, 0, &bars[LB_G]);
  };
  auto load_qk = [&](int chunk) {
    const Where w = where(chunk);
    log.request(LB_QK);
    mbar_expect_tx(&bars[LB_QK], 32768);
    for (int pn = 0; pn < 2; pn++) {
      tma_load_2d(sm + LS::QK + pn * 16384, &tmQ, w.h * 128 + 64 * pn, w.row0, &bars[LB_QK]);
      tma_load_2d(sm + LS::KT + pn * 16384, &tmK, w.h * 128 + 64 * pn, w.row0, &bars[LB_QK]);
    }
  };
  auto load_v = [&](int chunk) {
    const Where w = where(chunk);
    log.request(LB_V);
    mbar_expect_tx(&bars[LB_V], 16384);
    for (int pn = 0; pn < 2; pn++) tma_load_2d(sm + VT + pn * VP, &tmV, w.h * 128 + 64 * pn, w.row0, &bars[LB_V]);
  };
  float next_row = 0.f;  // beta (threads 0..63) or the scalar gate (64..127) of the next chunk's rows
  auto fetch_rows = [&](int chunk) {
    if (tid < 2 * C && chunk < p.total_chunks) {
      const Where w = where(chunk);
      const size_t at = ((size_t)w.row0 + (tid & 63)) * H + w.h;
      if (!VB && tid < C) next_row = p.beta[at];
      if (GATE == GATE_SCALAR && tid >= C) next_row = p.g[at];
    }
  };
  constexpr uint32_t ID_D = instr_desc(FMT_BF16, 128, 64, false, false);   // A and B K-major
  constexpr uint32_t ID_WU = instr_desc(FMT_BF16, 128, 128, false, true);  // A K-major (Akk), B MN-major (E / Z)

  if (leader && (int)blockIdx.x < p.total_chunks) {
    load_qk(blockIdx.x);
    if (VEC) load_g(blockIdx.x);
    else load_v(blockIdx.x);
  }
  __syncwarp();
  fetch_rows(blockIdx.x);

  for (int chunk = blockIdx.x; chunk < p.total_chunks && alive; chunk += gridDim.x) {
    const Where at = where(chunk);
    const int h = at.h, row0 = at.row0, next = chunk + gridDim.x;
    const size_t base128 = ((size_t)row0 * H + h) * 128, base64 = ((size_t)row0 * H + h) * 64;
    if (!VB && tid < C) sBeta[tid] = next_row;
    if (GATE == GATE_SCALAR && tid >= C && tid < 2 * C) sGs[tid - C] = next_row;
    fetch_rows(next);
    if (leader) {  // what is requested late goes to L2 now: this chunk's v, the next one's q and k
      if (VEC)
        for (int pn = 0; pn < 2; pn++) prefetch_2d(&tmV, h * 128 + 64 * pn, row0);
      if (next < p.total_chunks) {
        const Where w = where(next);
        for (int pn = 0; pn < 2; pn++) {
          prefetch_2d(&tmQ, w.h * 128 + 64 * pn, w.row0);
          prefetch_2d(&tmK, w.h * 128 + 64 * pn, w.row0);
          if (!VEC) prefetch_2d(&tmV, w.h * 128 + 64 * pn, w.row0);
        }
      }
    }
    __syncwarp();
    bool wide = false, far = false;

    if (VEC) {
      // ---- centre of the gate per channel ---------------------------------------------------------------------
      wait(LB_G, 41);
      {
        const int ch = tid & 127, rg = tid >> 7;
        const unsigned char* gp = sm + LS::G + (ch >> 5) * 8192 + (ch & 3) * 4;
        float lo = INFINITY, hi = -INFINITY, last = 0.f;
#pragma unroll 8
        for (int r = 0; r < C / NG; r++) {
          last = *reinterpret_cast<const float*>(gp + swz(C / NG * rg + r, (ch & 31) >> 2));
          lo = fminf(lo, last);
          hi = fmaxf(hi, last);
        }
        sMM[rg * 256 + ch] = lo;
        sMM[rg * 256 + 128 + ch] = hi;
        if (rg == NG - 1) sGl[ch] = last;
      }
      __syncthreads();
      if (tid < 128) {
        float lo = sMM[tid], hi = sMM[128 + tid];
#pragma unroll
        for (int rg = 1; rg < NG; rg++) {
          lo = fminf(lo, sMM[rg * 256 + tid]);
          hi = fmaxf(hi, sMM[rg * 256 + 128 + tid]);
        }
        sCen[tid] = 0.5f * (lo + hi);
        far = !(hi - lo < VECTOR_SPAN_FREE);
        wide = !(hi - lo < VECTOR_SPAN_LIMIT);
      }
      far = __syncthreads_or(far ? 1 : 0) != 0;
      wait(LB_QK, 42);
      if (far) {  // the range of q and k counts (common.cuh): thread = half a row of one of them
        uint32_t* sMax = reinterpret_cast<uint32_t*>(sMM);
        const unsigned char* row = sm + (krow ? LS::KT : LS::QK) + wg * 16384;
        uint32_t m = 0;
#pragma unroll 2
        for (int c = 0; c < 8; c++) {
          const uint4 u = *reinterpret_cast<const uint4*>(row + swz(t, c));
          m = max_abs2(max_abs2(max_abs2(max_abs2(m, u.x), u.y), u.z), u.w);
        }
        m = __reduce_max_sync(0xffffffffu, max(m & 0xFFFFu, m >> 16));
        if (__any_sync(0xffffffffu, wide)) m = 0xFFFFu;  // out of range
        if (lane == 0) sMax[warp] = m;
        __syncthreads();
        const uint32_t mq = max(max(sMax[0], sMax[1]), max(sMax[4], sMax[5])), mk = max(max(sMax[2], sMax[3]), max(sMax[6], sMax[7]));
        wide = !centred_range(mq) || !centred_range(mk);
      }
      // ---- operands of the first product ----------------------------------------------------------------------
      if (alive) {
        const float bs = VB ? 0.f : sBeta[t];
#pragma unroll 2
        for (int c8 = 0; c8 < 16 / NG; c8++) {
          const int c = wg * (128 / NG) + c8 * 8;
          const uint32_t pn = c >> 6, off = swz(t, (c & 63) >> 3);
          const unsigned char* gp = sm + LS::G + (c >> 5) * 8192;
          float al[8], kk[8], x[8];
          uint4 hi, lo;
          load8(gp + swz(t, (c & 31) >> 2), gp + swz(t, ((c & 31) >> 2) + 1), al);
          load8(sm + LS::CEN + c * 4, sm + LS::CEN + c * 4 + 16, x);
          unpack8(*reinterpret_cast<const uint4*>(sm + LS::KT + pn * 16384 + off), kk);
#pragma unroll
          for (int j = 0; j < 8; j++) al[j] = ex2(al[j] - x[j]);  // |exponent| < 100: no flush
          if (!krow) {
            unpack8(*reinterpret_cast<const uint4*>(sm + LS::QK + pn * 16384 + off), x);
#pragma unroll
            for (int j = 0; j < 8; j++) {
              kk[j] *= rcp(al[j]);
              x[j] *= al[j];
            }
            split8(kk, hi, lo);
            *reinterpret_cast<uint4*>(sm + LS::Y + pn * 8192 + off) = hi;
            *reinterpret_cast<uint4*>(sm + LS::Y + 16384 + pn * 8192 + off) = lo;
          } else {
            if (VB) unpack8(*reinterpret_cast<const uint4*>(p.bg + base128 + (size_t)t * ldt + c), x);
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = (VB ? x[j] : bs) * kk[j] * al[j];
          }
          split8(x, hi, lo);
          tmem_st4(tlane + TM_A + c / 2, hi);
          tmem_st4(tlane + TM_A + 64 + c / 2, lo);
        }
        tmem_st_wait();
      }
      fence_async_smem();
      tc_fence_before_sync();
      __syncthreads();
      tc_fence_after_sync();
      if (wide) {
        // exact pairwise sums over the tiles, thread = (row i, every fourth column j)
        const int i = tid >> 2;
        auto bfat = [&](uint32_t tile, int r, int k) {
          return bf2f(*reinterpret_cast<const bf16*>(sm + tile + (k >> 6) * 16384 + swz(r, (k & 63) >> 3) + (k & 7) * 2));
        };
        auto gat = [&](int r, int k) {
          return *reinterpret_cast<const float*>(sm + LS::G + (k >> 5) * 8192 + swz(r, (k & 31) >> 2) + (k & 3) * 4);
        };
        const float beta_i = VB ? 0.f : sBeta[i];
        const bf16* bgi = p.bg + base128 + (size_t)i * ldt;  // key gate row of token i (vector beta)
        for (int j = tid & 3; j < C; j += 4) {
          float aq = 0.f, ak = 0.f;
          if (j <= i) {
            for (int k = 0; k < 128; k++) {
              const float f = exp2f(gat(i, k) - gat(j, k)) * bfat(LS::KT, j, k);
              aq = fmaf(bfat(LS::QK, i, k), f, aq);
              ak = fmaf((VB ? bf2f(bgi[k]) : beta_i) * bfat(LS::KT, i, k), f, ak);
            }
          }
          p.Aqk[base64 + (size_t)i * H * 64 + j] = f2bf(p.scale * aq);
          sL[i * LDL + j] = j < i ? ak : 0.f;
        }
        __syncthreads();  // the tiles are rewritten below
      } else if (warp == 0 && alive) {
        if (leader) {
#pragma unroll
          for (int pass = 0; pass < 3; pass++)  // hi hi, lo hi, hi lo
#pragma unroll
            for (int ks = 0; ks < 8; ks++)
              mma_f16_ts(tb + TM_D, tb + TM_A + (pass == 1 ? 64 : 0) + ks * 8,
                         dl(LS::Y + (pass == 2 ? 16384 : 0) + (ks >> 2) * 8192 + (ks & 3) * 32, 16), ID_D, pass > 0 || ks > 0);
        }
        __syncwarp();
      }
      if (leader) {
        log.request(LB_D);
        mma_commit(&bars[LB_D]);
      }
      __syncwarp();
    } else {
      // ---- scalar gate / none: exact products on the tiles as they landed --------------------------------------
      wait(LB_QK, 42);
      if (warp == 0 && alive) {
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < 8; ks++)
            mma_f16_lo(tb + TM_D, dl(LS::QK + (ks >> 2) * 16384 + (ks & 3) * 32, 16),
                       dl(LS::KT + (ks >> 2) * 16384 + (ks & 3) * 32, 16), ID_D, ks > 0);
          log.request(LB_D);
          mma_commit(&bars[LB_D]);
        }
        __syncwarp();
      }
      __syncthreads();  // beta and gate rows visible
      wait(LB_D, 43);   // k is rewritten in place below
    }

    // ---- qg and kg in 16-byte pieces to global memory, E in place of k -----------------------------------------------
    if (alive) {
#pragma unroll 2
      for (int i = tid; i < C * 16; i += TPB) {
        const int r = i >> 4, c = (i & 15) * 8;
        const uint32_t off = (c >> 6) * 16384 + swz(r, (c & 63) >> 3);
        const size_t go = base128 + (size_t)r * ldt + c;
        float kk[8], x[8], gam[8], kap[8];
        uint4* kat = reinterpret_cast<uint4*>(sm + LS::KT + off);
        const uint4 kraw = *kat, qraw = *reinterpret_cast<const uint4*>(sm + LS::QK + off);
        unpack8(kraw, kk);
        unpack8(qraw, x);
        if (VEC) {
          const unsigned char* gp = sm + LS::G + (c >> 5) * 8192;
          load8(gp + swz(r, (c & 31) >> 2), gp + swz(r, ((c & 31) >> 2) + 1), gam);
          load8(sm + LS::GL + c * 4, sm + LS::GL + c * 4 + 16, kap);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            kap[j] = ex2(kap[j] - gam[j]);
            gam[j] = ex2(gam[j]);
          }
        } else if (GATE == GATE_SCALAR) {
          const float g = ex2(sGs[r]), l = ex2(sGs[C - 1] - sGs[r]);
#pragma unroll
          for (int j = 0; j < 8; j++) { gam[j] = g; kap[j] = l; }
        }
        if (GATE != GATE_NONE) {
          float y[8];
#pragma unroll
          for (int j = 0; j < 8; j++) { x[j] *= gam[j]; y[j] = kk[j] * kap[j]; }
          *reinterpret_cast<uint4*>(p.qg + go) = pack8(x);
          *reinterpret_cast<uint4*>(p.kg + go) = pack8(y);
        } else if (p.write_qk) {
          *reinterpret_cast<uint4*>(p.qg + go) = qraw;
          *reinterpret_cast<uint4*>(p.kg + go) = kraw;
        }
        if (VB) unpack8(*reinterpret_cast<const uint4*>(p.bg + go), x);
        const float bs = VB ? 0.f : sBeta[r];
#pragma unroll
        for (int j = 0; j < 8; j++) kk[j] *= (VB ? x[j] : bs) * (GATE == GATE_NONE ? 1.f : gam[j]);
        *kat = pack8(kk);
      }
    }
    if (VEC) wait(LB_D, 43);
    tc_fence_after_sync();

    // ---- Aqk (rows of q) and L (rows of k, over Yc) -------------------------------------------------------------------
    if (alive && !wide) {
      const float f0 = krow ? (VEC ? 1.f : sBeta[t]) : p.scale;
#pragma unroll 1
      for (int c0 = 64 / NG * wg; c0 < 64 / NG * (wg + 1); c0 += 16) {
        float u[16];
        tmem_ld16(tlane + TM_D + c0, u);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; e++) {
          const int col = c0 + e;
          const bool keep = krow ? col < t : col <= t;
          float f = f0;
          if (GATE == GATE_SCALAR) f *= ex2(sGs[t] - sGs[keep ? col : t]);
          u[e] = keep ? u[e] * f : 0.f;
        }
        if (krow) {
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(sL + t * LDL + c0 + e) = make_float4(u[e], u[e + 1], u[e + 2], u[e + 3]);
        } else {
          uint4* dst = reinterpret_cast<uint4*>(p.Aqk + base64 + (size_t)t * H * 64 + c0);
          dst[0] = make_uint4(pack_bf16(u[0], u[1]), pack_bf16(u[2], u[3]), pack_bf16(u[4], u[5]), pack_bf16(u[6], u[7]));
          dst[1] = make_uint4(pack_bf16(u[8], u[9]), pack_bf16(u[10], u[11]), pack_bf16(u[12], u[13]), pack_bf16(u[14], u[15]));
        }
      }
    }
    fence_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (VEC) {
      if (leader && alive) {  // q and the gate tile are dead
        load_v(chunk);
        if (next < p.total_chunks) load_g(next);
      }
      __syncwarp();
    }

    invert_unit_lower(sL, tid);

    // ---- Akk: BF16, to global memory and twice into the operand tile; Z = w v in place --------------------------------
    {
#pragma unroll
      for (int e = tid; e < C * 8; e += TPB) {
        const int i = e >> 3, c0 = (e & 7) * 8;
        float x[8];
        load8(reinterpret_cast<const unsigned char*>(sL + i * LDL + c0), reinterpret_cast<const unsigned char*>(sL + i * LDL + c0 + 4), x);
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = c0 + j <= i ? x[j] : 0.f;
        const uint4 v = pack8(x);
        *reinterpret_cast<uint4*>(sm + LS::AK + swz(i, c0 / 8)) = v;
        *reinterpret_cast<uint4*>(sm + LS::AK + 8192 + swz(i, c0 / 8)) = v;
        *reinterpret_cast<uint4*>(p.Akk + base64 + (size_t)i * H * 64 + c0) = v;
      }
    }
    wait(LB_V, 44);
    if (alive) {
#pragma unroll 2
      for (int i = tid; i < C * 16; i += TPB) {
        const int r = i >> 4, c16 = i & 15;
        uint4* vat = reinterpret_cast<uint4*>(sm + VT + (c16 >> 3) * VP + swz(r, c16 & 7));
        float vv[8], ww[8];
        unpack8(*vat, vv);
        if (VB) unpack8(*reinterpret_cast<const uint4*>(p.wg + base128 + (size_t)r * ldt + c16 * 8), ww);
        const float bs = VB ? 0.f : sBeta[r];
#pragma unroll
        for (int j = 0; j < 8; j++) vv[j] *= VB ? ww[j] : bs;
        *vat = pack8(vv);
      }
    }
    fence_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0) {
      if (leader && alive) {
#pragma unroll
        for (int ks = 0; ks < 4; ks++)
          mma_f16_lo(tb + TM_W, dl(LS::AK + ks * 32, 16), dl(LS::KT + ks * 2048, 16384), ID_WU, ks > 0);
#pragma unroll
        for (int ks = 0; ks < 4; ks++)
          mma_f16_lo(tb + TM_U, dl(LS::AK + ks * 32, 16), dl(VT + ks * 2048, VP), ID_WU, ks > 0);
        log.request(LB_WU);
        mma_commit(&bars[LB_WU]);
      }
      __syncwarp();
    }
    wait(LB_WU, 45);
    tc_fence_after_sync();
    // ---- w (lanes 0..63) and u (64..127): 64 channels of row t into the dead E / Z tiles ------------------------------
    if (alive) {
      const int c0 = wg * (128 / NG);
      unsigned char* dst = sm + (krow ? VT + (c0 >> 6) * VP : LS::KT + (c0 >> 6) * 16384);
#pragma unroll 1
      for (int c = 0; c < 128 / NG; c += 16) {
        float u[16], y[8];
        tmem_ld16(tlane + (krow ? TM_U : TM_W) + c0 + c, u);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
          for (int j = 0; j < 8; j++) y[j] = u[8 * e + j];
          *reinterpret_cast<uint4*>(dst + swz(t, ((c0 & 63) + c) / 8 + e)) = pack8(y);
        }
      }
    }
    fence_async_smem();
    tc_fence_before_sync();
    alive = __syncthreads_and(alive ? 1 : 0) != 0;
    tc_fence_after_sync();
    if (leader && alive) {
      for (int pn = 0; pn < 2; pn++) {
        tma_store_2d(&tmW, sm + LS::KT + pn * 16384, h * 128 + 64 * pn, row0);
        tma_store_2d(&tmU, sm + VT + pn * VP, h * 128 + 64 * pn, row0);
      }
      tma_store_commit();
      tma_store_wait_read();
      if (next < p.total_chunks) {
        load_qk(next);
        if (!VEC) load_v(next);
      }
    }
    __syncwarp();
    ph ^= 1u;
  }
  if (leader) {
    if (!alive) {  // gave up: no copy or product may still be under way when the CTA exits
      for (int b = 0; b < LB_COUNT; b++)
        if ((log.asked >> b) & 1u) mbar_wait_limit(&bars[b], (log.odd >> b) & 1u, nullptr, 0, DRAIN_NS);
    }
    tma_store_wait_read();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tb, 256);
}

template <int GATE, bool VB>
cudaError_t run(const CUtensorMap* tm, const LocalParams& p, cudaStream_t st) {
  cudaError_t e = ensure_dynamic_smem<chunk_fwd_tc_kernel<GATE, VB>>(LS::TOTAL);
  if (e != cudaSuccess) return e;
  const int cap = 2 * 148;  // two CTAs per SM
  const int grid = p.total_chunks < cap ? p.total_chunks : cap;
  chunk_fwd_tc_kernel<GATE, VB><<<grid, TPB, LS::TOTAL, st>>>(tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], p);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_chunk_fwd_tc(const RewyFwdArgs& a, int* err, cudaStream_t st) {
  const int B = a.B, T = a.T, H = a.H, NT = T / C;
  const uint64_t rows = (uint64_t)B * T, cols = (uint64_t)H * 128, pitch = (uint64_t)H * 256;
  const bool vector = gate_mode_of(a.family) == GATE_VECTOR;
  CUtensorMap tm[6];
  bool ok = encode_tmap_2d(&tm[0], a.q, 2, cols, rows, pitch, 64, 64) && encode_tmap_2d(&tm[1], a.k, 2, cols, rows, pitch, 64, 64) &&
            encode_tmap_2d(&tm[2], a.v, 2, cols, rows, pitch, 64, 64) && encode_tmap_2d(&tm[4], a.w, 2, cols, rows, pitch, 64, 64) &&
            encode_tmap_2d(&tm[5], a.u, 2, cols, rows, pitch, 64, 64);
  tm[3] = tm[0];  // never dereferenced without a vector gate
  if (ok && vector) ok = encode_tmap_panels(&tm[3], a.g, 4, cols, rows, (uint64_t)H * 512, 64, 4);
  if (!ok) return cudaErrorInvalidValue;
  LocalParams p;
  p.g = a.g; p.beta = a.beta; p.bg = (const bf16*)a.b_gate; p.wg = (const bf16*)a.w_gate;
  p.Akk = (bf16*)a.Akk; p.Aqk = (bf16*)a.Aqk; p.qg = (bf16*)a.qg; p.kg = (bf16*)a.kg; p.err = err; p.T = T; p.H = H; p.NT = NT; p.total_chunks = B * H * NT;
  p.write_qk = a.qg != a.q || a.kg != a.k; p.scale = a.scale;
  switch (a.family) {
    case REWY_DELTA: return run<GATE_NONE, false>(tm, p, st);
    case REWY_GDN: return run<GATE_SCALAR, false>(tm, p, st);
    case REWY_KDA: return run<GATE_VECTOR, false>(tm, p, st);
    default: return run<GATE_VECTOR, true>(tm, p, st);
  }
}

}  // namespace rewy
