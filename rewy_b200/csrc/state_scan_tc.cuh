// What the tcgen05 state scans share: launch parameters, 16-column TMEM accesses, bulk stores, the BF16 hi/lo split.
#pragma once
#include "tc05.cuh"

namespace rewy {
namespace scan {
using namespace tc;

struct ScanParams {
  const float *g, *dht;
  bf16 *dR, *dRlo;
  float* dh0;
  int* err;
  int T, H, NT;
  int svf;  // initial / final state tensors (dht, dh0) are stored value-first: [B,H,V,K]
  const int* cu;  // packed sequences: device int32 [sequences + 1] token offsets (multiples of 64), or nullptr
  float scale;
};

struct FwdParams {
  const float *g, *h0;
  float* final_state;  // optional: state after the last chunk, FP32 [B,H,K,V] ([B,H,V,K] when svf)
  bf16* v_new;
  int* err;
  int T, H, NT;
  int svf;  // h0 is stored value-first: [B,H,V,K]
  const int* cu;  // packed sequences: device int32 [sequences + 1] token offsets (multiples of 64), or nullptr
};
__device__ __forceinline__ void tmem_ld16f(uint32_t taddr, float (&r)[16]) {
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
__device__ __forceinline__ void tmem_st16f(uint32_t taddr, const float (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])), "r"(__float_as_uint(r[3])),
      "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])), "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7])),
      "r"(__float_as_uint(r[8])), "r"(__float_as_uint(r[9])), "r"(__float_as_uint(r[10])), "r"(__float_as_uint(r[11])),
      "r"(__float_as_uint(r[12])), "r"(__float_as_uint(r[13])), "r"(__float_as_uint(r[14])), "r"(__float_as_uint(r[15]))
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// shared -> global tile store through a tensor map (bulk async group of the issuing thread)
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, int c0, int c1, const void* src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void split8s(const float (&x)[8], uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    __nv_bfloat162 hh = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
    float2 hf = __bfloat1622float2(hh);
    h[i] = *reinterpret_cast<uint32_t*>(&hh);
    l[i] = pack_bf16(x[2 * i] - hf.x, x[2 * i + 1] - hf.y);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

constexpr int SPLIT_MAX_PAIRS = 148;  // (sequence, head) pairs up to which two CTAs share a pair: reason in state_scan_split.cu

}  // namespace scan

// state_scan_split.cu: one CTA per (sequence, head, half of the value channels); tensor maps in the order of the
// launchers of state_scan_tc.cu, `pairs` = sequences * heads.
cudaError_t launch_bwd_scan_split(int gate, const CUtensorMap* tm, const scan::ScanParams& p, int pairs, cudaStream_t st);
cudaError_t launch_fwd_scan_split(int gate, const CUtensorMap* tm, const scan::FwdParams& p, int pairs, cudaStream_t st);

}  // namespace rewy
