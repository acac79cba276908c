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

// A consumer warp's release of a ring stage.  Every lane's reads are fenced
// against the async proxy first: the copy that refills the stage is not ordered
// behind loads that are still in flight, only behind this fence and the arrive.
__device__ __forceinline__ void ring_release(uint64_t* empty, int lane) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) mbar_arrive(empty);
}

// Barrier of a ring kernel's N consumer threads (the producer is not part of
// it).  It is an aligned one: lanes that skipped a masked zone's work come
// together with their warp first.
template <int N>
__device__ __forceinline__ void consumer_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory");
}

// Position in a ring of NS shared-memory stages: slot and the parity of its
// current phase.
template <int NS>
struct RingPos {
  int slot = 0;
  uint32_t par = 0;
  __device__ __forceinline__ void next() {
    if (++slot == NS) {
      slot = 0;
      par ^= 1;
    }
  }
};

// Mode mm of panel p's least-squares solution from the sums Y over panel
// 1's row weights: sign x Y at panel 1's mode (src >> 4mm) & 15, which lies
// in mm's group (the constant, x y z, xx yy zz, xy yz xz), so the choice is
// a select among three registers.  Y holds modes M0.. (M0 = 0 with the
// constant, 1 without).
template <int M0, typename R>
__device__ __forceinline__ R lsq_rotated(const R* Y, int mm, unsigned long long src, unsigned int neg) {
  const int mu = (int)((src >> (4 * mm)) & 15);
  R v;
  if (mm == 0) {
    v = Y[0 - M0];
  } else {
    const int g0 = 1 + 3 * ((mm - 1) / 3);
    v = mu == g0 ? Y[g0 - M0] : (mu == g0 + 1 ? Y[g0 + 1 - M0] : Y[g0 + 2 - M0]);
  }
  return ((neg >> mm) & 1u) ? -v : v;
}

// MRWENO weights of a quadratic least-squares solution X (modes x .. xz)
// against the linear WENO slopes lin (421:4440-4551 for the primitives,
// 421:8700-9350 for E): the quadratic polynomial's modes Phi with the linear
// part taken out, and the normalised weights of the two.
template <typename R>
__device__ __forceinline__ void mrweno_weights(const R* X, const R* lin, const R* c0, R f, R ghi, R glo, R obghi, R grat,
                                               R smallnum, R* Phi, R& Wlo, R& Whi) {
  const R ob12 = R(1.0) / R(12.0), ob180 = R(1.0) / R(180.0), ob144 = R(1.0) / R(144.0);
  const R betalo = f + (R(1.0) - f) * R(2.0);
  const R ISlo = betalo * (lin[0] * lin[0] + lin[1] * lin[1] + lin[2] * lin[2]) * ob12;
#pragma unroll
  for (int a = 0; a < 3; ++a) Phi[a] = X[a] * obghi - lin[a] * grat;
#pragma unroll
  for (int a = 3; a < 9; ++a) Phi[a] = X[a] * obghi;
  const R IShi = (Phi[0] * Phi[0] + Phi[1] * Phi[1] + Phi[2] * Phi[2]) * ob12 +
                 (Phi[3] * Phi[3]) * (sqr(c0[4] - ob12) + ob180) + (Phi[4] * Phi[4]) * (sqr(c0[5] - ob12) + ob180) +
                 (Phi[5] * Phi[5]) * (sqr(c0[6] - ob12) + ob180) + (Phi[6] * Phi[6]) * (c0[7] * c0[7] + ob144) +
                 (Phi[7] * Phi[7]) * (c0[8] * c0[8] + ob144) + (Phi[8] * Phi[8]) * (c0[9] * c0[9] + ob144);
  const R tau = fabs(IShi - ISlo);
  Wlo = glo * (R(1.0) + tau / (ISlo + smallnum));
  Whi = ghi * (R(1.0) + tau / (IShi + smallnum));
  const R aa = R(1.0) / (Wlo + Whi);
  Wlo = Wlo * aa;
  Whi = Whi * aa;
}

// The hybrid's modes x .. xz, damped by the flattener f.
template <typename R>
__device__ __forceinline__ void mrweno_hybrid(const R* X, const R* lin, const R* c0, R f, R smallnum, R* out) {
  const R ghi = f * R(0.6) + (R(1.0) - f) * R(0.95), glo = R(1.0) - ghi, obghi = R(1.0) / ghi, grat = glo / ghi;
  R Phi[9], Wlo, Whi;
  mrweno_weights(X, lin, c0, f, ghi, glo, obghi, grat, smallnum, Phi, Wlo, Whi);
  const R x = R(1.0) - f;
#pragma unroll
  for (int a = 0; a < 3; ++a) out[a] = (Whi * Phi[a] + Wlo * lin[a]) * x;
#pragma unroll
  for (int a = 3; a < 9; ++a) out[a] = (Whi * Phi[a]) * x;
}

// The central 18-zone stencil of STEPS 7.b and 9.c: (neighbour in the plane, 12
// for the zone's own column; radial offset).
struct Stencil18 {
  int v[18][2];
};
__host__ __device__ constexpr Stencil18 stencil18() {
  return {{{0, 0},  {1, 0},  {2, 0},  {3, 0},  {12, 1}, {12, -1}, {8, 0}, {9, 0},  {10, 0},
           {11, 0}, {0, 1},  {1, 1},  {0, -1}, {1, -1}, {2, 1},   {3, 1}, {2, -1}, {3, -1}}};
}

// The line of p to L2.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The resident row weights of n zones, W words a zone (STEP 7.b's 162, STEP
// 9.c's 190): blocks of 32 zones [W][32], the last one [W][what is left], so
// that a block is one contiguous run for the bulk copies.  STEP 7.b's zones
// are rounded up to 4 and STEP 9.c's copies are of whole 16 bytes.
struct WBlock {
  long long off;  // of the block's first word
  int wid;        // zones in a row
};
template <int W>
__device__ __forceinline__ WBlock w_block(long long blk, long long n) {
  return {blk * W * 32, (int)min(32LL, (W == 162 ? m9_stride(n) : n) - blk * 32)};
}
// Word e of zone t.
template <int W>
__device__ __forceinline__ long long w_at(long long t, int e, long long n) {
  const WBlock b = w_block<W>(t / 32, n);
  return b.off + (long long)e * b.wid + t % 32;
}

// The interior zones and w layers around them.
inline Range3 around(const Dims& d, int w) { return {1 - w, d.N + w, 1 - w, d.N + w, 1 - w, d.nr + w}; }
// The zones STEP 8.d solves the B modes of.
inline Range3 adp_zones(const Solve& sv) {
  const Dims& d = sv.d;
  const AdpLayers l = adp_layers(sv.p);
  return {1 - l.side, d.N + l.side, 1 - l.side, d.N + l.side, 1 - l.radial, d.nr + l.radial};
}
inline Range3 zones_all(const Dims& d) { return {1 - d.G, d.N + d.G, 1 - d.G, d.N + d.G, 1 - d.G, d.nr + d.G}; }
inline Range3 shrink(const Dims& d, int s) {
  return {1 - d.G + s, d.N + d.G - s, 1 - d.G + s, d.N + d.G - s, 1 - d.G + s, d.nr + d.G - s};
}

}  // namespace cs
