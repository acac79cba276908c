// Helpers shared by the reconstruction kernels (cs_recon.cu, cs_adp.cu).
#pragma once

#include <algorithm>
#include <utility>

#include "cs_solve.h"

namespace cs {

constexpr int TPB = 128;

template <typename R>
__device__ __forceinline__ R& Vat(const DStateT<R>& s, const Dims& d, int comp, int mode, int p, int i, int j, int k) {
  return s.V[d.at(mode * NVAR + comp, p, i, j, k)];
}

template <typename R>
__device__ __forceinline__ void coef10(const DGeom& g, const Dims& d, int p, int i, int j, int k, R* c) {
#pragma unroll
  for (int t = 0; t < 10; ++t) c[t] = geoR<R>(g, d, CS_G_COEF, t, p, i, j, k);
}

// ---- bulk asynchronous copies (cp.async.bulk) and mbarriers ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n selp.u32 %0, 1, 0, P;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Bounded wait on an mbarrier phase: after 2^23 polls (seconds, far beyond
// any copy) it records an error in *err and returns, so no wait can hang.
static __device__ __noinline__ void mbar_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (int it = 0; it < (1 << 23); ++it)
    if (mbar_try_wait(bar, parity)) return;
  atomicOr(err, 1);
}

// The interior zones and w layers around them.
inline Range3 around(const Dims& d, int w) { return {1 - w, d.N + w, 1 - w, d.N + w, 1 - w, d.nr + w}; }
// Layers around the interior on which STEP 8.d solves the B modes.  The stage
// reads E in one layer (the edge EMFs); P12's STEPS 9.b / 9.c run on it and
// read point values of E, made of the ADP modes, one layer further, P2's
// stencils, run on one layer more where there are four, two.  The layers beyond hold primitives and slopes for those only.
inline int adp_layers(const Solve& sv) { return (sv.p.flags & CS_FLAG_P2) ? sv.p.nghost - 1 : 2; }
inline Range3 zones_all(const Dims& d) { return {1 - d.G, d.N + d.G, 1 - d.G, d.N + d.G, 1 - d.G, d.nr + d.G}; }
inline Range3 shrink(const Dims& d, int s) {
  return {1 - d.G + s, d.N + d.G - s, 1 - d.G + s, d.N + d.G - s, 1 - d.G + s, d.nr + d.G - s};
}

}  // namespace cs
