// Cross-chunk state scans for few (sequence, head) pairs: two CTAs per pair, each with 64 of the 128 value channels.
//
// Same recurrences, operands and roundings as the kernels of state_scan_tc.cu; a value channel's column of the state
// never meets another one, so the halves need nothing from each other.  With one CTA per pair and fewer pairs than
// SMs the time is the dependent chain of a chunk step times T / 64, whatever the rest of the chip does.  What is taken
// out of that chain here:
//   * half the state per CTA: half the TMEM reads, conversions and shared-memory writes per thread and step;
//   * every operand has its own buffer and a warp of its own refills it as soon as its last reader is complete, so no
//     tile is requested inside the chain;
//   * another warp issues the products, and those that do not depend on the state of the step run while it is waited
//     for: Aqk^T dO of the next chunk before its dh is ready, qg^T dO while the dR epilogue runs;
//   * warps hand over by mbarriers of their own instead of CTA barriers, and the global stores of dR / v_new come
//     after the hand-over.
// M = 128 products with 64 value rows: the A operand's two 64-row panels are the same tile (leading offset 0), TMEM
// lanes 64..127 repeat lanes 0..63 and their threads take the other half of the tokens.
// Measured against the whole-state kernels: reverse scan of one sequence of 8192 tokens and 16 heads (32 CTAs) 502 -> 252
// us, 3.9 -> 2.0 us per chunk step, of which the work on the state row takes 0.5 us and the wait for the dR product
// 0.7; forward scan of B=1 T=8192 H=32 494 -> 214 us; both together (side stream) at B=2 T=32768 H=32 2177 -> 1565 us,
// where HBM (7.6 GB) would allow 1160.
// Limit (SPLIT_MAX_PAIRS = 148): up to there 2 CTAs per pair all fit at two per SM.  At 96 pairs (12 sequences of 1333
// tokens on average, 8 heads) reverse 167 -> 112 us, forward 139 -> 77; above 148 pairs the whole-state kernels have two
// CTAs on every SM to hide each other's chains and run at 0.83 of the HBM peak, and this form would read kg, w, qg and
// Aqk twice for nothing.
#include "state_scan_tc.cuh"

namespace rewy {
namespace {
using namespace scan;

constexpr int WORKERS = 256;            // eight warps: thread = TMEM lane (tid & 127), column half (tid >> 7)
constexpr int TPB = WORKERS + 64;       // + one warp for TMA, one for the products
constexpr int NBARS = 12;
constexpr unsigned long long DRAIN_NS = 20ull * 1000 * 1000;  // wait for copies in flight after a give-up

__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(c0),
               "r"(c1)
               : "memory");
}

// Token range of a (sequence, head) pair; false outside the envelope of packed sequences.
struct Range {
  int bos, NT;
  bool ok;
};
__device__ __forceinline__ Range range_of(const int* cu, int b, int T, int NT) {
  Range r{b * T, NT, true};
  if (cu != nullptr) {
    r.bos = cu[b];
    const int len = cu[b + 1] - r.bos;
    r.NT = len / C;
    r.ok = len >= 0 && len % C == 0 && r.bos % C == 0;
  }
  return r;
}

// 32 columns v0 .. v0 + 31 of row k of a state tensor ([k][v], or [v][k] when value-first), times f
__device__ __forceinline__ void read_state_row(const float* st, int svf, int k, int v0, float f, float (&x)[32]) {
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    float4 v4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (st != nullptr) {
      const int v = v0 + j;
      if (svf)
        v4 = make_float4(st[(size_t)v * DK + k], st[(size_t)(v + 1) * DK + k], st[(size_t)(v + 2) * DK + k],
                         st[(size_t)(v + 3) * DK + k]);
      else
        v4 = *reinterpret_cast<const float4*>(st + (size_t)k * DV + v);
    }
    x[j] = v4.x * f; x[j + 1] = v4.y * f; x[j + 2] = v4.z * f; x[j + 3] = v4.w * f;
  }
}
__device__ __forceinline__ void write_state_row(float* st, int svf, int k, int v0, float f, const float (&x)[32]) {
  if (svf) {
#pragma unroll
    for (int j = 0; j < 32; j++) st[(size_t)(v0 + j) * DK + k] = f * x[j];
  } else {
#pragma unroll
    for (int j = 0; j < 32; j += 4)
      *reinterpret_cast<float4*>(st + (size_t)k * DV + v0 + j) = make_float4(f * x[j], f * x[j + 1], f * x[j + 2], f * x[j + 3]);
  }
}
__device__ __forceinline__ void tmem_ld32f(uint32_t taddr, float (&x)[32]) {
  uint32_t u[32];
  tmem_ld32(taddr, u);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; i++) x[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ void tmem_st32f(uint32_t taddr, const float (&x)[32]) {
  float a[16], b[16];
#pragma unroll
  for (int i = 0; i < 16; i++) { a[i] = x[i]; b[i] = x[16 + i]; }
  tmem_st16f(taddr, a);
  tmem_st16f(taddr + 16, b);
}
template <int GATE>
__device__ __forceinline__ float load_lambda(const float* g, int last_row, int H, int h, int ch) {
  if (GATE == GATE_VECTOR) return g[((size_t)last_row * H + h) * 128 + ch];
  if (GATE == GATE_SCALAR) return g[(size_t)last_row * H + h];
  return 0.f;
}

// ---- reverse scan -------------------------------------------------------------------------------------------------
struct RS {
  static constexpr uint32_t KG = 0;               // [64 i][128 k] two panels             16 KB
  static constexpr uint32_t W = KG + 16384;       // [64 i][128 k]                        16 KB
  static constexpr uint32_t QG = W + 16384;       // [64 i][128 k]                        16 KB
  static constexpr uint32_t DO0 = QG + 16384;     // [64 i][64 v]                          8 KB
  static constexpr uint32_t AQK = DO0 + 8192;     // [64 j][64 i]                          8 KB
  static constexpr uint32_t DHHI = AQK + 8192;    // [128 k][64 v]                        16 KB
  static constexpr uint32_t DHLO = DHHI + 16384;  //                                      16 KB
  static constexpr uint32_t DRHI = DHLO + 16384;  // (dR/scale)^T [64 v][64 i]             8 KB
  static constexpr uint32_t DRLO = DRHI + 8192;   //                                       8 KB
  static constexpr uint32_t BARS = DRLO + 8192;
  static constexpr uint32_t TMEM = BARS + NBARS * 8;
  static constexpr uint32_t TOTAL = TMEM + 32;
};
static_assert(2 * (RS::TOTAL + 1024) <= 233472, "two reverse-scan CTAs must fit one SM");
constexpr uint32_t TM_S = 0, TM_X = 64, TM_COLS = 128;  // state half, dR^T / (w h)^T

enum { F_KG = 0, F_AD, F_QG, F_W, B_DH, B_DR, B_Q, B_R, B_S, B_FREE, B_END };

template <int GATE>
__global__ void __launch_bounds__(TPB, 2)
bwd_scan_split_kernel(const __grid_constant__ CUtensorMap tmKg, const __grid_constant__ CUtensorMap tmW,
                      const __grid_constant__ CUtensorMap tmQg, const __grid_constant__ CUtensorMap tmDO,
                      const __grid_constant__ CUtensorMap tmAqk, const __grid_constant__ CUtensorMap tmDH, const ScanParams p) {
  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + RS::BARS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + RS::TMEM);
  const uint32_t sb = smem_u32(sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = blockIdx.x & 1, bh = blockIdx.x >> 1, b = bh / p.H, h = bh % p.H, H = p.H;
  const Range r = range_of(p.cu, b, p.T, p.NT);
  if (!r.ok || (sb & 1023u) != 0) {  // outside the envelope (or an unaligned plan): report, touch nothing
    if (tid == 0) atomicCAS(p.err, 0, 90);
    return;
  }
  const int NT = r.NT, chunk0 = r.bos / C, vb = 64 * half;  // vb: first value channel of this CTA
  const float scale = p.scale, inv_scale = 1.f / p.scale;
  if (NT == 0) {  // empty sequence: the state gradient passes through unchanged
    if (p.dh0 != nullptr)
      for (int i = tid; i < DK * DV / 2; i += TPB) {
        const size_t at = (size_t)bh * DK * DV + (size_t)half * (DK * DV / 2) + i;
        p.dh0[at] = p.dht == nullptr ? 0.f : p.dht[at];
      }
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < NBARS; i++) mbar_init(&bars[i], i == B_DH || i == B_R ? WORKERS / 32 : 1);
    fence_barrier_init();
  }
  if (warp == 8) {
    if (lane == 0) {
      prefetch_tmap(&tmKg); prefetch_tmap(&tmW); prefetch_tmap(&tmQg); prefetch_tmap(&tmDO);
      prefetch_tmap(&tmAqk); prefetch_tmap(&tmDH);
    }
    __syncwarp();
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tb = *tmem_slot;
  bool alive = true;
  // barrier phases: everything completes once per chunk step, so step `it` waits for parity it & 1
  auto wait = [&](int bar, int it, int code) {
    if (alive) alive = mbar_wait(&bars[bar], (uint32_t)it & 1u, p.err, code);
  };
  auto row_of = [&](int it) { return r.bos + (NT - 1 - it) * C; };  // step it handles chunk NT - 1 - it

  if (warp == 8) {
    // ---- copies -----------------------------------------------------------------------------------------------
    if (lane == 0) {
      auto load_kg = [&](int it) {
        mbar_expect_tx(&bars[F_KG], 16384);
        for (int pn = 0; pn < 2; pn++) tma_load_2d(sm + RS::KG + pn * 8192, &tmKg, h * 128 + 64 * pn, row_of(it), &bars[F_KG]);
      };
      auto load_ad = [&](int it) {
        mbar_expect_tx(&bars[F_AD], 16384);
        tma_load_2d(sm + RS::DO0, &tmDO, h * 128 + vb, row_of(it), &bars[F_AD]);
        tma_load_2d(sm + RS::AQK, &tmAqk, h * 64, row_of(it), &bars[F_AD]);
      };
      auto load_qg = [&](int it) {
        mbar_expect_tx(&bars[F_QG], 16384);
        for (int pn = 0; pn < 2; pn++) tma_load_2d(sm + RS::QG + pn * 8192, &tmQg, h * 128 + 64 * pn, row_of(it), &bars[F_QG]);
      };
      auto load_w = [&](int it) {
        mbar_expect_tx(&bars[F_W], 16384);
        for (int pn = 0; pn < 2; pn++) tma_load_2d(sm + RS::W + pn * 8192, &tmW, h * 128 + 64 * pn, row_of(it), &bars[F_W]);
      };
      int n_kg = 0, n_ad = 0, n_qg = 0, n_w = 0;  // last step each buffer was requested for
      load_ad(0); load_kg(0); load_qg(0); load_w(0);
      for (int it = 0; it < NT && alive; it++) {
        if (it + 2 < NT) {  // the step after next: into L2
          const int row = row_of(it + 2);
          tma_prefetch_2d(&tmDO, h * 128 + vb, row);
          if (half == 0) {
            tma_prefetch_2d(&tmKg, h * 128, row); tma_prefetch_2d(&tmKg, h * 128 + 64, row);
            tma_prefetch_2d(&tmAqk, h * 64, row);
          } else {
            tma_prefetch_2d(&tmQg, h * 128, row); tma_prefetch_2d(&tmQg, h * 128 + 64, row);
            tma_prefetch_2d(&tmW, h * 128, row); tma_prefetch_2d(&tmW, h * 128 + 64, row);
          }
        }
        wait(B_DH, it, 70);
        if (!alive) break;
        tma_store_2d(&tmDH, vb, ((chunk0 + NT - 1 - it) * H + h) * 128, sm + RS::DHHI);
        bulk_commit();
        wait(B_DR, it, 71);
        if (!alive) break;
        if (it + 1 < NT) load_kg(n_kg = it + 1);
        bulk_wait_read0();
        mbar_arrive(&bars[B_FREE]);  // the dh tile may be written again
        wait(B_Q, it, 72);
        if (!alive) break;
        if (it + 1 < NT) { load_ad(n_ad = it + 1); load_qg(n_qg = it + 1); }
        wait(B_S, it, 73);
        if (!alive) break;
        if (it + 1 < NT) load_w(n_w = it + 1);
      }
      if (!alive) {  // gave up: no copy may still be writing this CTA's shared memory when it exits
        mbar_wait_limit(&bars[F_KG], n_kg & 1, nullptr, 0, DRAIN_NS);
        mbar_wait_limit(&bars[F_AD], n_ad & 1, nullptr, 0, DRAIN_NS);
        mbar_wait_limit(&bars[F_QG], n_qg & 1, nullptr, 0, DRAIN_NS);
        mbar_wait_limit(&bars[F_W], n_w & 1, nullptr, 0, DRAIN_NS);
      }
      bulk_wait0();
    }
    __syncwarp();
  } else if (warp == 9) {
    // ---- products -----------------------------------------------------------------------------------------------
    if (elect_one()) {
      constexpr uint32_t ID_DR_A = instr_desc(FMT_BF16, 128, 64, true, false);  // A MN-major (dh^T), B K-major (kg)
      constexpr uint32_t ID_DR_B = instr_desc(FMT_BF16, 128, 64, true, true);   // A MN-major (dO^T), B MN-major (Aqk)
      constexpr uint32_t ID_S_Q = instr_desc(FMT_BF16, 128, 64, true, true);    // A MN-major (qg^T), B MN-major (dO)
      constexpr uint32_t ID_S_W = instr_desc(FMT_BF16, 128, 64, true, false, true, false);  // -(w^T) (dR/scale)^T K-major
      auto dl = [&](uint32_t off, uint32_t lbo) { return desc_lo(sb + off, lbo); };
      auto intra = [&](int it) {  // dR^T = dO^T Aqk: needs nothing of the chain
        wait(F_AD, it, 80);
        if (!alive) return;
#pragma unroll
        for (int ks = 0; ks < 4; ks++)
          mma_f16_lo(tb + TM_X, dl(RS::DO0 + ks * 2048, 0), dl(RS::AQK + ks * 2048, 8192), ID_DR_B, ks > 0);
      };
      intra(0);
      for (int it = 0; it < NT && alive; it++) {
        wait(B_DH, it, 81);
        wait(F_KG, it, 82);
        if (!alive) break;
        tc_fence_after_sync();
#pragma unroll
        for (int pass = 0; pass < 2; pass++)
#pragma unroll
          for (int ks = 0; ks < 8; ks++)
            mma_f16_lo(tb + TM_X, dl((pass == 0 ? RS::DHHI : RS::DHLO) + ks * 2048, 0),
                       dl(RS::KG + (ks >> 2) * 8192 + (ks & 3) * 32, 16), ID_DR_A, true);
        mma_commit(&bars[B_DR]);
        wait(F_QG, it, 83);
        if (!alive) break;
#pragma unroll
        for (int ks = 0; ks < 4; ks++)
          mma_f16_lo(tb + TM_S, dl(RS::QG + ks * 2048, 8192), dl(RS::DO0 + ks * 2048, 8192), ID_S_Q, true);
        mma_commit(&bars[B_Q]);
        wait(B_R, it, 84);
        wait(F_W, it, 85);
        if (!alive) break;
        tc_fence_after_sync();
#pragma unroll
        for (int pass = 0; pass < 2; pass++)
#pragma unroll
          for (int ks = 0; ks < 4; ks++)
            mma_f16_lo(tb + TM_S, dl(RS::W + ks * 2048, 8192), dl((pass == 0 ? RS::DRHI : RS::DRLO) + ks * 32, 16), ID_S_W,
                       true);
        mma_commit(&bars[B_S]);
        if (it + 1 < NT) intra(it + 1);
      }
      if (!alive) {  // gave up: the products in flight read shared memory and write TMEM
        mma_commit(&bars[B_END]);
        mbar_wait_limit(&bars[B_END], 0, nullptr, 0, DRAIN_NS);
      }
    }
    __syncwarp();
  } else {
    // ---- state, dh tiles, dR epilogue --------------------------------------------------------------------------
    const int ch = tid & 127, wg = tid >> 7;
    const uint32_t tlane = tb + ((uint32_t)((warp & 3) * 32) << 16);
    const int v = ch & 63, quarter = 2 * wg + (ch >> 6);  // dR^T: value row, 16 tokens
    const size_t ldt = (size_t)H * 128;
    float x[32];
    read_state_row(p.dht == nullptr ? nullptr : p.dht + (size_t)bh * DK * DV, p.svf, ch, vb + 32 * wg, inv_scale, x);
    float glast = load_lambda<GATE>(p.g, row_of(0) + C - 1, H, h, ch);
    for (int it = 0; it < NT; it++) {
      if (it > 0) {
        wait(B_S, it - 1, 91);
        tc_fence_after_sync();
        if (!alive) break;
        tmem_ld32f(tlane + TM_S + 32 * wg, x);
        wait(B_FREE, it - 1, 92);
        if (!alive) break;
      }
      const float lam = GATE == GATE_NONE ? 1.f : exp2f(glast);
      if (it + 1 < NT) glast = load_lambda<GATE>(p.g, row_of(it + 1) + C - 1, H, h, ch);  // needed a whole step later
      if (GATE != GATE_NONE || it == 0) {
        float y[32];
#pragma unroll
        for (int j = 0; j < 32; j++) y[j] = x[j] * lam;
        tmem_st32f(tlane + TM_S + 32 * wg, y);
      }
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float y[8];
#pragma unroll
        for (int j = 0; j < 8; j++) y[j] = scale * x[8 * c + j];
        uint4 hi, lo;
        split8s(y, hi, lo);
        *reinterpret_cast<uint4*>(sm + RS::DHHI + swz(ch, 4 * wg + c)) = hi;
        *reinterpret_cast<uint4*>(sm + RS::DHLO + swz(ch, 4 * wg + c)) = lo;
      }
      if (GATE != GATE_NONE || it == 0) tmem_st_wait();
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[B_DH]);

      wait(B_DR, it, 93);
      tc_fence_after_sync();
      if (!alive) break;
      float d[16];
      tmem_ld16f(tlane + TM_X + 16 * quarter, d);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < 2; c++) {
        float y[8];
#pragma unroll
        for (int j = 0; j < 8; j++) y[j] = d[8 * c + j] * inv_scale;
        uint4 hi, lo;
        split8s(y, hi, lo);
        *reinterpret_cast<uint4*>(sm + RS::DRHI + swz(v, 2 * quarter + c)) = hi;
        *reinterpret_cast<uint4*>(sm + RS::DRLO + swz(v, 2 * quarter + c)) = lo;
      }
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[B_R]);
      // dR as BF16 hi/lo to global memory while the state update runs
      const size_t go = ((size_t)(row_of(it) + 16 * quarter) * H + h) * 128 + vb + v;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const bf16 hi = f2bf(d[j]);
        p.dR[go + (size_t)j * ldt] = hi;
        p.dRlo[go + (size_t)j * ldt] = f2bf(d[j] - bf2f(hi));
      }
    }
    wait(B_S, NT - 1, 94);
    tc_fence_after_sync();
    if (p.dh0 != nullptr && alive) {
      tmem_ld32f(tlane + TM_S + 32 * wg, x);
      write_state_row(p.dh0 + (size_t)bh * DK * DV, p.svf, ch, vb + 32 * wg, scale, x);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tb, TM_COLS);
}

// ---- forward scan -------------------------------------------------------------------------------------------------
struct VS {
  static constexpr uint32_t STAGE = 16384 + 16384 + 8192;  // w, kg: [64 i][128 k]; u: [64 i][64 v]
  static constexpr uint32_t W = 0, KG = 16384, U = 32768;  // inside a stage; two stages
  static constexpr uint32_t HT = 2 * STAGE;                // h tile [128 k][64 v]   16 KB
  static constexpr uint32_t VNT = HT + 16384;              // v_new^T [64 v][64 i]    8 KB
  static constexpr uint32_t BARS = VNT + 8192;
  static constexpr uint32_t TMEM = BARS + NBARS * 8;
  static constexpr uint32_t TOTAL = TMEM + 32;
};
static_assert(RS::TOTAL + VS::TOTAL + 2048 <= 233472, "a forward-scan CTA fits an SM beside a reverse-scan CTA");
// full barriers of the two stages, hand-overs
enum { V_W = 0, V_KG = 2, V_U = 4, V_H = 6, V_C, V_R, V_S, V_FREE, V_END };

template <int GATE>
__global__ void __launch_bounds__(TPB, 2)
fwd_scan_split_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmKg,
                      const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmH, const FwdParams p) {
  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + VS::BARS);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + VS::TMEM);
  const uint32_t sb = smem_u32(sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = blockIdx.x & 1, bh = blockIdx.x >> 1, b = bh / p.H, h = bh % p.H, H = p.H;
  const Range r = range_of(p.cu, b, p.T, p.NT);
  if (!r.ok || (sb & 1023u) != 0) {
    if (tid == 0) atomicCAS(p.err, 0, 91);
    return;
  }
  const int NT = r.NT, chunk0 = r.bos / C, vb = 64 * half;
  if (NT == 0) {  // empty sequence: the state passes through unchanged
    if (p.final_state != nullptr)
      for (int i = tid; i < DK * DV / 2; i += TPB) {
        const size_t at = (size_t)bh * DK * DV + (size_t)half * (DK * DV / 2) + i;
        p.final_state[at] = p.h0 == nullptr ? 0.f : p.h0[at];
      }
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < NBARS; i++) mbar_init(&bars[i], i == V_H || i == V_R ? WORKERS / 32 : 1);
    fence_barrier_init();
  }
  if (warp == 8) {
    if (lane == 0) { prefetch_tmap(&tmW); prefetch_tmap(&tmKg); prefetch_tmap(&tmU); prefetch_tmap(&tmH); }
    __syncwarp();
    tmem_alloc(tmem_slot, TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tb = *tmem_slot;
  bool alive = true;
  auto wait = [&](int bar, int it, int code) {  // hand-overs: one phase per step
    if (alive) alive = mbar_wait(&bars[bar], (uint32_t)it & 1u, p.err, code);
  };
  auto wait_full = [&](int bar, int it, int code) {  // stage it & 1, its (it >> 1)th filling
    if (alive) alive = mbar_wait(&bars[bar + (it & 1)], (uint32_t)(it >> 1) & 1u, p.err, code);
  };
  auto row_of = [&](int it) { return r.bos + it * C; };

  if (warp == 8) {
    if (lane == 0) {
      auto load2 = [&](uint32_t dst, const CUtensorMap* m, int bar, int it) {
        const int s = it & 1;
        mbar_expect_tx(&bars[bar + s], 16384);
        for (int pn = 0; pn < 2; pn++)
          tma_load_2d(sm + s * VS::STAGE + dst + pn * 8192, m, h * 128 + 64 * pn, row_of(it), &bars[bar + s]);
      };
      auto load_u = [&](int it) {
        const int s = it & 1;
        mbar_expect_tx(&bars[V_U + s], 8192);
        tma_load_2d(sm + s * VS::STAGE + VS::U, &tmU, h * 128 + vb, row_of(it), &bars[V_U + s]);
      };
      int n_w = 0, n_u = 0, n_kg = 0;  // last step each tensor was requested for
      for (int it = 0; it < 2 && it < NT; it++) {
        load2(VS::W, &tmW, V_W, n_w = it);
        load_u(n_u = it);
        load2(VS::KG, &tmKg, V_KG, n_kg = it);
      }
      for (int it = 0; it < NT && alive; it++) {
        wait(V_H, it, 50);
        if (!alive) break;
        tma_store_2d(&tmH, vb, ((chunk0 + it) * H + h) * 128, sm + VS::HT);
        bulk_commit();
        wait(V_C, it, 51);
        if (!alive) break;
        if (it + 2 < NT) load2(VS::W, &tmW, V_W, n_w = it + 2);
        bulk_wait_read0();
        mbar_arrive(&bars[V_FREE]);  // the h tile may be written again
        wait(V_R, it, 52);
        if (!alive) break;
        if (it + 2 < NT) load_u(n_u = it + 2);
        wait(V_S, it, 53);
        if (!alive) break;
        if (it + 2 < NT) load2(VS::KG, &tmKg, V_KG, n_kg = it + 2);
      }
      if (!alive) {  // gave up: no copy may still be writing this CTA's shared memory when it exits
        for (int back = 0; back < 2; back++) {
          if (n_w >= back) mbar_wait_limit(&bars[V_W + ((n_w - back) & 1)], ((n_w - back) >> 1) & 1, nullptr, 0, DRAIN_NS);
          if (n_u >= back) mbar_wait_limit(&bars[V_U + ((n_u - back) & 1)], ((n_u - back) >> 1) & 1, nullptr, 0, DRAIN_NS);
          if (n_kg >= back) mbar_wait_limit(&bars[V_KG + ((n_kg - back) & 1)], ((n_kg - back) >> 1) & 1, nullptr, 0, DRAIN_NS);
        }
      }
      bulk_wait0();
    }
    __syncwarp();
  } else if (warp == 9) {
    if (elect_one()) {
      constexpr uint32_t ID_V = instr_desc(FMT_BF16, 128, 64, true, false, true, false);  // -(h^T) w^T: A MN-major negated
      constexpr uint32_t ID_S = instr_desc(FMT_BF16, 128, 64, true, false);               // kg^T (v_new^T)^T
      auto dl = [&](uint32_t off, uint32_t lbo) { return desc_lo(sb + off, lbo); };
      for (int it = 0; it < NT && alive; it++) {
        const uint32_t st = (it & 1) * VS::STAGE;
        wait_full(V_W, it, 60);
        wait(V_H, it, 61);
        if (!alive) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 8; ks++)
          mma_f16_lo(tb + TM_X, dl(VS::HT + ks * 2048, 0), dl(st + VS::W + (ks >> 2) * 8192 + (ks & 3) * 32, 16), ID_V, ks > 0);
        mma_commit(&bars[V_C]);
        wait_full(V_KG, it, 62);
        wait(V_R, it, 63);
        if (!alive) break;
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < 4; ks++)
          mma_f16_lo(tb + TM_S, dl(st + VS::KG + ks * 2048, 8192), dl(VS::VNT + ks * 32, 16), ID_S, true);
        mma_commit(&bars[V_S]);
      }
      if (!alive) {
        mma_commit(&bars[V_END]);
        mbar_wait_limit(&bars[V_END], 0, nullptr, 0, DRAIN_NS);
      }
    }
    __syncwarp();
  } else {
    const int ch = tid & 127, wg = tid >> 7;
    const uint32_t tlane = tb + ((uint32_t)((warp & 3) * 32) << 16);
    const int v = ch & 63, quarter = 2 * wg + (ch >> 6);  // v_new^T: value row, 16 tokens
    const size_t ldt = (size_t)H * 128;
    float x[32];
    read_state_row(p.h0 == nullptr ? nullptr : p.h0 + (size_t)bh * DK * DV, p.svf, ch, vb + 32 * wg, 1.f, x);
    float glast = load_lambda<GATE>(p.g, row_of(0) + C - 1, H, h, ch);
    for (int it = 0; it < NT; it++) {
      if (it > 0) {
        wait(V_S, it - 1, 64);
        tc_fence_after_sync();
        if (!alive) break;
        tmem_ld32f(tlane + TM_S + 32 * wg, x);
        wait(V_FREE, it - 1, 65);
        if (!alive) break;
      }
      const float lam = GATE == GATE_NONE ? 1.f : exp2f(glast);
      if (it + 1 < NT) glast = load_lambda<GATE>(p.g, row_of(it + 1) + C - 1, H, h, ch);
      if (GATE != GATE_NONE || it == 0) {
        float y[32];
#pragma unroll
        for (int j = 0; j < 32; j++) y[j] = x[j] * lam;
        tmem_st32f(tlane + TM_S + 32 * wg, y);
      }
#pragma unroll
      for (int c = 0; c < 4; c++) {
        uint32_t pk[4];
#pragma unroll
        for (int j = 0; j < 4; j++) pk[j] = pack_bf16(x[8 * c + 2 * j], x[8 * c + 2 * j + 1]);
        *reinterpret_cast<uint4*>(sm + VS::HT + swz(ch, 4 * wg + c)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
      if (GATE != GATE_NONE || it == 0) tmem_st_wait();
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[V_H]);

      // u while the product runs
      wait_full(V_U, it, 66);
      if (!alive) break;
      const unsigned char* su = sm + (it & 1) * VS::STAGE + VS::U;
      float d[16];
#pragma unroll
      for (int j = 0; j < 16; j++)
        d[j] = bf2f(*reinterpret_cast<const bf16*>(su + swz(16 * quarter + j, v >> 3) + (v & 7) * 2));
      wait(V_C, it, 67);
      tc_fence_after_sync();
      if (!alive) break;
      float y[16];
      tmem_ld16f(tlane + TM_X + 16 * quarter, y);
      tmem_ld_wait();
      uint32_t pk[8];
#pragma unroll
      for (int j = 0; j < 8; j++) pk[j] = pack_bf16(d[2 * j] + y[2 * j], d[2 * j + 1] + y[2 * j + 1]);
#pragma unroll
      for (int c = 0; c < 2; c++)
        *reinterpret_cast<uint4*>(sm + VS::VNT + swz(v, 2 * quarter + c)) =
            make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
      fence_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars[V_R]);
      // v_new (token-major) while the state update runs
      uint16_t* dst = reinterpret_cast<uint16_t*>(p.v_new) + ((size_t)(row_of(it) + 16 * quarter) * H + h) * 128 + vb + v;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        dst[(size_t)(2 * j) * ldt] = (uint16_t)(pk[j] & 0xFFFFu);
        dst[(size_t)(2 * j + 1) * ldt] = (uint16_t)(pk[j] >> 16);
      }
    }
    wait(V_S, NT - 1, 68);
    tc_fence_after_sync();
    if (p.final_state != nullptr && alive) {
      tmem_ld32f(tlane + TM_S + 32 * wg, x);
      write_state_row(p.final_state + (size_t)bh * DK * DV, p.svf, ch, vb + 32 * wg, 1.f, x);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tb, TM_COLS);
}

template <int GATE>
cudaError_t run_bwd(const CUtensorMap* tm, const ScanParams& p, int pairs, cudaStream_t st) {
  cudaError_t e = ensure_dynamic_smem<bwd_scan_split_kernel<GATE>>(RS::TOTAL);
  if (e != cudaSuccess) return e;
  bwd_scan_split_kernel<GATE><<<2 * pairs, TPB, RS::TOTAL, st>>>(tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], p);
  count_launch();
  return cudaGetLastError();
}
template <int GATE>
cudaError_t run_fwd(const CUtensorMap* tm, const FwdParams& p, int pairs, cudaStream_t st) {
  cudaError_t e = ensure_dynamic_smem<fwd_scan_split_kernel<GATE>>(VS::TOTAL);
  if (e != cudaSuccess) return e;
  fwd_scan_split_kernel<GATE><<<2 * pairs, TPB, VS::TOTAL, st>>>(tm[0], tm[1], tm[2], tm[3], p);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_bwd_scan_split(int gate, const CUtensorMap* tm, const scan::ScanParams& p, int pairs, cudaStream_t st) {
  switch (gate) {
    case GATE_NONE: return run_bwd<GATE_NONE>(tm, p, pairs, st);
    case GATE_SCALAR: return run_bwd<GATE_SCALAR>(tm, p, pairs, st);
    default: return run_bwd<GATE_VECTOR>(tm, p, pairs, st);
  }
}

cudaError_t launch_fwd_scan_split(int gate, const CUtensorMap* tm, const scan::FwdParams& p, int pairs, cudaStream_t st) {
  switch (gate) {
    case GATE_NONE: return run_fwd<GATE_NONE>(tm, p, pairs, st);
    case GATE_SCALAR: return run_fwd<GATE_SCALAR>(tm, p, pairs, st);
    default: return run_fwd<GATE_VECTOR>(tm, p, pairs, st);
  }
}

}  // namespace rewy
