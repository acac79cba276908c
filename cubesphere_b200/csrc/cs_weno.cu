// STEPS 7.b and 9.c of LIMIT_ALL_SLOPES_P12 (400riemann_integrate/
// 421limit_all_slopes_p12.f:3869-4554, :8464-9350) from the resident
// least-squares row weights.
#include "cs_recon.cuh"

namespace cs {

namespace {

// STEP 7.b (421:3869-4551): the 18-zone quadratic least squares X = sum_r W_r
// (V_r - V_0) from the resident row weights W_r = Minv A_r^T, hybridised with
// the linear WENO slopes of STEP 7.a (MRWENO weights, flattener damping).
//
// A block takes 32 zones: four warps, two primitives each, and a producer
// warp whose bulk copies bring the weights, six rows a stage, through a ring
// that runs ahead over the tiles.  kShared: the weights are panel 1's and the
// sums are rotated to the panel; tile T is then tile T / 6 of panel T % 6, so
// that L2 serves one tile's weights to six blocks.
//
// What bounds it: HBM, 1.3 KB of weights a zone in FP64 (per panel) and 0.9 KB
// of modes.  One thread a zone for all eight primitives took 255 registers
// and waited on its loads with 8 warps an SM (2.7 TB/s); here a thread's neighbour
// values are in flight a stage ahead and the weights never wait for them, and
// the next tile's offsets and L2 lines are prepared while one is worked on.  ms
// of a 6 x 128^2 x 64 step, FP64 / FP32: 11.7 / 6.65 for the former, 9.0 / 7.2
// without and 8.3 / 6.25 with the preparation.
constexpr int W7_CONS = 4 * 32;
constexpr int W7_THREADS = W7_CONS + 32;
constexpr int W7_ROWS = 6;  // stencil rows a ring stage
constexpr int W7_NS = 3;
template <typename R>
struct W7Smem {
  R stage[W7_NS][W7_ROWS * 9 * 32];
  int nbo[2][12][32];  // in-plane neighbours of the zones as box offsets, alternating over the tiles
  uint64_t full[W7_NS];
  uint64_t empty[W7_NS];
};

template <bool kShared, typename R>
__global__ void __launch_bounds__(W7_THREADS, sizeof(R) == 4 ? 4 : 3) k_weno7b(Dims d, PhysC ph, DGeom g, DStateT<R> s,
                                                                                Range3 r) {
  extern __shared__ __align__(128) unsigned char w7_raw[];
  W7Smem<R>& S = *reinterpret_cast<W7Smem<R>*>(w7_raw);
  constexpr Stencil18 N18 = stencil18();
  const int tid = threadIdx.x;
  const long long nz = r.count(), npp = nz / 6, nw = kShared ? npp : nz;
  const unsigned ntile = (unsigned)(kShared ? 6 * ((npp + 31) / 32) : (nz + 31) / 32);
  if (tid == 0) {
    for (int q = 0; q < W7_NS; ++q) {
      mbar_init(&S.full[q], 1);
      mbar_init(&S.empty[q], W7_CONS / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  RingPos<W7_NS> ring;
  if (tid >= W7_CONS) {
    if (tid == W7_CONS) {
      bool first = true;  // the ring's first round finds every stage free
      for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x) {
        const WBlock b = w_block<162>(kShared ? T / 6 : T, nw);
        const uint32_t bytes = (uint32_t)(W7_ROWS * 9 * b.wid * sizeof(R));
        for (int c = 0; c < 3; ++c) {
          if (!first) mbar_wait(&S.empty[ring.slot], ring.par ^ 1, s.err_flag);
          mbar_expect_tx(&S.full[ring.slot], bytes);
          bulk_g2s(&S.stage[ring.slot][0], s.op_m9 + b.off + (long long)c * W7_ROWS * 9 * b.wid, bytes, &S.full[ring.slot]);
          ring.next();
          if (ring.slot == 0) first = false;
        }
      }
    }
    return;
  }
  const int lane = tid & 31, w = tid >> 5;
  const int plane = d.NI * d.NJ;
  // the tile's zone and its neighbours' offsets, prepared one tile ahead
  struct Zone {
    bool act;
    int p;
    unsigned o;
  };
  auto prepare = [&](unsigned T, int(&nbo)[12][32]) -> Zone {
    const unsigned tw = (kShared ? T / 6 : T) * 32 + lane;
    Zone z = {T < ntile && tw < (unsigned)nw, 0, 0};
    int i = r.i0, j = r.j0, k = r.k0;
    if (z.act) {
      r.decode(kShared ? (T % 6) * npp + tw : tw, z.p, i, j, k);
      z.act = mask_at(g, d, z.p, i, j) == 1;
      // of a masked zone too: its own loads must not wait for the mask
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int n = 3 * w + q;
        nbo[n][lane] = (sten(g, d, z.p, i, j, n, 1) - j) * d.NI + (sten(g, d, z.p, i, j, n, 0) - i);
      }
    }
    z.o = (unsigned)(z.p * d.S + d.idx(i, j, k));
    return z;
  };
  int buf = 0;
  Zone next = prepare(blockIdx.x, S.nbo[0]);
  for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x, buf ^= 1) {
    // opaque to the compiler, which would otherwise form the addresses of all
    // planes before the loop and spill them
    long long PS = (long long)NPANEL * d.S;
    asm volatile("" : "+l"(PS));
    const Zone zone = next;
    const bool act = zone.act;
    const int p = zone.p;
    const long long o = zone.o;
    const int wid = w_block<162>(kShared ? T / 6 : T, nw).wid;
    int(&nbo)[12][32] = S.nbo[buf];
    // the offsets are complete; the other copy is no longer read
    consumer_sync<W7_CONS>();
    const R* v = s.V + 2 * w * PS + o;  // primitives 2 w and 2 w + 1
    // differences to the neighbours of stencil rows 6 c .. 6 c + 5, loaded one
    // ring stage ahead of their use
    R D[2][W7_ROWS], v0 = R(0.0), v1 = R(0.0);
    auto load_rows = [&](int c, R (&E)[2][W7_ROWS]) {
#pragma unroll
      for (int rr = 0; rr < W7_ROWS; ++rr) {
        const int n = N18.v[c * W7_ROWS + rr][0];
        const int off = (n == 12 ? 0 : nbo[n == 12 ? 0 : n][lane]) + N18.v[c * W7_ROWS + rr][1] * plane;
        E[0][rr] = act ? v[off] : R(0.0);
        E[1][rr] = act ? v[PS + off] : R(0.0);
      }
    };
    if (act) {
      v0 = v[0];
      v1 = v[PS];
    }
    load_rows(0, D);
    next = prepare(T + gridDim.x, S.nbo[buf ^ 1]);
    // the next tile's own values and slopes, to L2 while this one is worked on
    if (T + gridDim.x < ntile) {
      const unsigned Tn = T + gridDim.x, tn = (kShared ? Tn / 6 : Tn) * 32 + lane;
      if (tn < (unsigned)nw) {
        int pn, in, jn, kn;
        r.decode(kShared ? (Tn % 6) * npp + tn : tn, pn, in, jn, kn);
        const R* z = s.V + 2 * w * PS + (long long)pn * d.S + d.idx(in, jn, kn);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          prefetch_l2(z + m * NVAR * PS);
          prefetch_l2(z + (m * NVAR + 1) * PS);
        }
      }
    }
    R Y[2][9];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int a = 0; a < 9; ++a) Y[q][a] = R(0.0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      R Dn[2][W7_ROWS];
      if (c < 2) load_rows(c + 1, Dn);
      if (!mbar_try_wait(&S.full[ring.slot], ring.par)) mbar_wait(&S.full[ring.slot], ring.par, s.err_flag);
      const R* A = &S.stage[ring.slot][lane];
#pragma unroll
      for (int rr = 0; rr < W7_ROWS; ++rr) {
        const R d0 = D[0][rr] - v0, d1 = D[1][rr] - v1;
#pragma unroll
        for (int a = 0; a < 9; ++a) {
          const R m = A[(rr * 9 + a) * wid];
          Y[0][a] = Y[0][a] + m * d0;
          Y[1][a] = Y[1][a] + m * d1;
        }
      }
      ring_release(&S.empty[ring.slot], lane);
      ring.next();
      if (c < 2)
#pragma unroll
        for (int rr = 0; rr < W7_ROWS; ++rr) {
          D[0][rr] = Dn[0][rr];
          D[1][rr] = Dn[1][rr];
        }
    }
    if (act) {
      const unsigned long long qsrc = kShared ? s.lsq_map9[p].src : LSQ_IDENTITY_SRC;
      const unsigned int qneg = kShared ? s.lsq_map9[p].neg : 0u;
      R c0[10];
#pragma unroll
      for (int m = 4; m < 10; ++m) c0[m] = (R)__ldg(g.f[CS_G_COEF] + m * PS + o);
      const R f = s.flatA[o];
      R* V = s.V + 2 * w * PS + o;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        R X[9], out[9];
#pragma unroll
        for (int a = 0; a < 9; ++a) X[a] = kShared ? lsq_rotated<1>(Y[q], a + 1, qsrc, qneg) : Y[q][a];
        const R lin[3] = {V[(NVAR + q) * PS], V[(2 * NVAR + q) * PS], V[(3 * NVAR + q) * PS]};
        mrweno_hybrid(X, lin, c0, f, R(ph.smallnum), out);
#pragma unroll
        for (int m = 1; m < 10; ++m) V[(m * NVAR + q) * PS] = out[m - 1];
      }
    }
  }
}

// STEP 9.c (421:8464-9350): the 19-point interpolation least squares (the zone
// itself first) from the resident row weights, hybridised with the slopes of
// STEP 9.b; the point value is flattened toward E_pt.  Only the point value
// (mode 1) is stored: the LLF edge solver consumes nothing else.  The weights
// are stored over the zones rs, so a block takes 32 of those, a warp one
// component; zones outside r are left out.  Ring, offsets and panel order as
// in k_weno7b.
//
// What bounds it: reads of the weights in shared memory.  One thread a zone
// for the three components, a row of weights loaded at a time, waited for L2
// nineteen times over.  ms a step, that / this: 6 x 32^2 x 1 (SSP-RK3) 0.124 /
// 0.044, 6 x 32^2 x 16 0.122 / 0.095, 6 x 128^2 x 64 4.47 / 3.74 (FP32 2.59 /
// 2.60).
constexpr int E9_CONS = 3 * 32;
constexpr int E9_THREADS = E9_CONS + 32;
constexpr int E9_ROWS = 4;  // rows a ring stage, the last one 3
constexpr int E9_NCH = 5;
constexpr int E9_NS = 3;
template <typename R>
struct E9Smem {
  R stage[E9_NS][E9_ROWS * 10 * 32 + 16 / sizeof(R)];
  int nbo[2][12][32];
  uint64_t full[E9_NS];
  uint64_t empty[E9_NS];
};

template <bool kShared, typename R>
__global__ void __launch_bounds__(E9_THREADS, sizeof(R) == 4 ? 8 : 6) k_efield_c(Dims d, PhysC ph, DGeom g, DStateT<R> s,
                                                                                 Range3 r, Range3 rs) {
  extern __shared__ __align__(128) unsigned char e9_raw[];
  E9Smem<R>& S = *reinterpret_cast<E9Smem<R>*>(e9_raw);
  constexpr Stencil18 N18 = stencil18();
  const int tid = threadIdx.x;
  const long long nz = rs.count(), npp = nz / 6, nw = kShared ? npp : nz;
  const unsigned ntile = (unsigned)(kShared ? 6 * ((npp + 31) / 32) : (nz + 31) / 32);
  // whether tile T has a layer of r (tiles of the layers around it have none)
  const unsigned layer = (unsigned)((rs.i1 - rs.i0 + 1) * (rs.j1 - rs.j0 + 1));
  auto wanted = [&](unsigned T) {
    const unsigned t0 = (kShared ? T / 6 : T) * 32;
    if (!kShared && t0 / (unsigned)npp != (t0 + 31) / (unsigned)npp) return true;
    const unsigned u0 = kShared ? t0 : t0 % (unsigned)npp;
    return (int)((u0 + 31) / layer) + rs.k0 >= r.k0 && (int)(u0 / layer) + rs.k0 <= r.k1;
  };
  if (tid == 0) {
    for (int q = 0; q < E9_NS; ++q) {
      mbar_init(&S.full[q], 1);
      mbar_init(&S.empty[q], E9_CONS / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  RingPos<E9_NS> ring;
  if (tid >= E9_CONS) {
    if (tid == E9_CONS) {
      bool first = true;  // the ring's first round finds every stage free
      for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x) {
        if (!wanted(T)) continue;
        const WBlock b = w_block<190>(kShared ? T / 6 : T, nw);
        for (int c = 0; c < E9_NCH; ++c) {
          if (!first) mbar_wait(&S.empty[ring.slot], ring.par ^ 1, s.err_flag);
          const int words = c == E9_NCH - 1 ? 190 - (E9_NCH - 1) * E9_ROWS * 10 : E9_ROWS * 10;
          const uint32_t bytes = (uint32_t)(words * b.wid * sizeof(R) + 15) / 16 * 16;
          mbar_expect_tx(&S.full[ring.slot], bytes);
          bulk_g2s(&S.stage[ring.slot][0], s.op_m10 + b.off + (long long)c * E9_ROWS * 10 * b.wid, bytes, &S.full[ring.slot]);
          ring.next();
          if (ring.slot == 0) first = false;
        }
      }
    }
    return;
  }
  const int lane = tid & 31, w = tid >> 5;
  const int plane = d.NI * d.NJ;
  const long long PS = (long long)NPANEL * d.S;
  int buf = 0;
  for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x) {
    if (!wanted(T)) continue;
    const unsigned tw = (kShared ? T / 6 : T) * 32 + lane;
    bool act = tw < (unsigned)nw;
    int p = 0, i = r.i0, j = r.j0, k = r.k0;
    int(&nbo)[12][32] = S.nbo[buf];
    if (act) {
      rs.decode(kShared ? (T % 6) * npp + tw : tw, p, i, j, k);
      act = i >= r.i0 && i <= r.i1 && j >= r.j0 && j <= r.j1 && k >= r.k0 && k <= r.k1 && mask_at(g, d, p, i, j) == 1;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int n = 4 * w + q;
        nbo[n][lane] = (sten(g, d, p, i, j, n, 1) - j) * d.NI + (sten(g, d, p, i, j, n, 0) - i);
      }
    }
    const int wid = w_block<190>(kShared ? T / 6 : T, nw).wid;
    // the offsets are complete; the other copy is no longer read
    consumer_sync<E9_CONS>();
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    const R* f = s.Esnap + w * PS + o;
    R D[19];
#pragma unroll
    for (int rr = 0; rr < 19; ++rr) {
      const int n = rr ? N18.v[rr ? rr - 1 : 0][0] : 12, dz = rr ? N18.v[rr ? rr - 1 : 0][1] : 0;
      D[rr] = act ? f[(n == 12 ? 0 : nbo[n == 12 ? 0 : n][lane]) + dz * plane] : R(0.0);
    }
    R Y[10];
#pragma unroll
    for (int a = 0; a < 10; ++a) Y[a] = R(0.0);
#pragma unroll
    for (int c = 0; c < E9_NCH; ++c) {
      if (!mbar_try_wait(&S.full[ring.slot], ring.par)) mbar_wait(&S.full[ring.slot], ring.par, s.err_flag);
      const R* A = &S.stage[ring.slot][lane];
#pragma unroll
      for (int rr = 0; rr < E9_ROWS; ++rr)
        if (c * E9_ROWS + rr < 19)
#pragma unroll
          for (int a = 0; a < 10; ++a) Y[a] = Y[a] + A[(rr * 10 + a) * wid] * D[c * E9_ROWS + rr < 19 ? c * E9_ROWS + rr : 0];
      ring_release(&S.empty[ring.slot], lane);
      ring.next();
    }
    if (act) {
      const unsigned long long qsrc = kShared ? s.lsq_map10[p].src : LSQ_IDENTITY_SRC;
      const unsigned int qneg = kShared ? s.lsq_map10[p].neg : 0u;
      R X[10], c0[10];
#pragma unroll
      for (int a = 0; a < 10; ++a) X[a] = kShared ? lsq_rotated<0>(Y, a, qsrc, qneg) : Y[a];
#pragma unroll
      for (int m = 4; m < 10; ++m) c0[m] = (R)__ldg(g.f[CS_G_COEF] + m * PS + o);
      const R* e = s.E + w * PS + o;
      const R lin[3] = {e[3 * PS], e[6 * PS], e[9 * PS]};
      const R fl = s.flatA[o];
      const R ghi = fl * R(0.6) + (R(1.0) - fl) * R(0.95), glo = R(1.0) - ghi, obghi = R(1.0) / ghi, grat = glo / ghi;
      R Wlo, Whi, Phi[9];
      mrweno_weights(X + 1, lin, c0, fl, ghi, glo, obghi, grat, R(ph.smallnum), Phi, Wlo, Whi);
      const R e0 = Whi * (X[0] * obghi - D[0] * grat) + Wlo * D[0];
      s.E[w * PS + o] = D[0] * fl + e0 * (R(1.0) - fl);
    }
    buf ^= 1;
  }
}

template <typename R>
void launch_efield_c_t(Solve& sv, const DStateT<R>& st, const Range3& r, const Range3& rs) {
  const long long n = rs.count(), nt = st.lsq_map10 ? 6 * ((n / 6 + 31) / 32) : (n + 31) / 32;
  const int nb = (int)std::min<long long>(nt, (long long)grid_sms(sv) * (sizeof(R) == 4 ? 8 : 6));
  if (st.lsq_map10)
    k_efield_c<true, R><<<nb, E9_THREADS, sizeof(E9Smem<R>), sv.stream>>>(sv.d, sv.ph, sv.g, st, r, rs);
  else
    k_efield_c<false, R><<<nb, E9_THREADS, sizeof(E9Smem<R>), sv.stream>>>(sv.d, sv.ph, sv.g, st, r, rs);
  mark(sv, "k_efield_c");
}

template <typename R>
void launch_weno7b_t(Solve& sv, const DStateT<R>& st, const Range3& r) {
  const long long n = r.count(), nt = st.lsq_map9 ? 6 * ((n / 6 + 31) / 32) : (n + 31) / 32;
  const int nb = (int)std::min<long long>(nt, (long long)grid_sms(sv) * (sizeof(R) == 4 ? 4 : 3));
  if (st.lsq_map9)
    k_weno7b<true, R><<<nb, W7_THREADS, sizeof(W7Smem<R>), sv.stream>>>(sv.d, sv.ph, sv.g, st, r);
  else
    k_weno7b<false, R><<<nb, W7_THREADS, sizeof(W7Smem<R>), sv.stream>>>(sv.d, sv.ph, sv.g, st, r);
  mark(sv, "k_weno7b");
}

}  // namespace

void launch_weno7b(Solve& sv, const Range3& r) {
  if (sv.fp32)
    launch_weno7b_t(sv, sv.stF, r);
  else
    launch_weno7b_t(sv, sv.st, r);
}

void launch_efield_c(Solve& sv, const Range3& r, const Range3& rs) {
  if (sv.fp32)
    launch_efield_c_t(sv, sv.stF, r, rs);
  else
    launch_efield_c_t(sv, sv.st, r, rs);
}

void set_weno_smem_limits() {
  cudaFuncSetAttribute(k_efield_c<false, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(E9Smem<double>));
  cudaFuncSetAttribute(k_efield_c<true, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(E9Smem<double>));
  cudaFuncSetAttribute(k_efield_c<false, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(E9Smem<float>));
  cudaFuncSetAttribute(k_efield_c<true, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(E9Smem<float>));
  cudaFuncSetAttribute(k_weno7b<false, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<double>));
  cudaFuncSetAttribute(k_weno7b<true, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<double>));
  cudaFuncSetAttribute(k_weno7b<false, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<float>));
  cudaFuncSetAttribute(k_weno7b<true, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<float>));
}

}  // namespace cs
