// STEP 7.b of LIMIT_ALL_SLOPES_P12 (400riemann_integrate/
// 421limit_all_slopes_p12.f:3869-4554) from the resident least-squares row
// weights.
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
  // central 18-zone stencil: (neighbour or 12 for the zone itself, dz)
  constexpr int N18[18][2] = {{0, 0},  {1, 0},  {2, 0},  {3, 0},  {12, 1}, {12, -1}, {8, 0}, {9, 0},  {10, 0},
                              {11, 0}, {0, 1},  {1, 1},  {0, -1}, {1, -1}, {2, 1},   {3, 1}, {2, -1}, {3, -1}};
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
        const M9Block b = m9_block(kShared ? T / 6 : T, nw);
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
    const int wid = m9_block(kShared ? T / 6 : T, nw).wid;
    int(&nbo)[12][32] = S.nbo[buf];
    // the offsets are complete; the other copy is no longer read
    asm volatile("bar.sync 1, %0;" ::"n"(W7_CONS) : "memory");
    const R* v = s.V + 2 * w * PS + o;  // primitives 2 w and 2 w + 1
    // differences to the neighbours of stencil rows 6 c .. 6 c + 5, loaded one
    // ring stage ahead of their use
    R D[2][W7_ROWS], v0 = R(0.0), v1 = R(0.0);
    auto load_rows = [&](int c, R (&E)[2][W7_ROWS]) {
#pragma unroll
      for (int rr = 0; rr < W7_ROWS; ++rr) {
        const int n = N18[c * W7_ROWS + rr][0];
        const int off = (n == 12 ? 0 : nbo[n == 12 ? 0 : n][lane]) + N18[c * W7_ROWS + rr][1] * plane;
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
      // this warp's reads are done before the copy engine may write the stage again
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.empty[ring.slot]);
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

void set_weno_smem_limits() {
  cudaFuncSetAttribute(k_weno7b<false, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<double>));
  cudaFuncSetAttribute(k_weno7b<true, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<double>));
  cudaFuncSetAttribute(k_weno7b<false, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<float>));
  cudaFuncSetAttribute(k_weno7b<true, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(W7Smem<float>));
}

}  // namespace cs
