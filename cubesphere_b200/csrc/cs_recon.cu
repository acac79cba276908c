// Reconstruction kernels of the stage: primitive variables, flattener,
// WENO-AO / MRWENO (P12) slopes, positivity limiting, face-B quadrature
// values, the ADP constrained least-squares magnetic reconstruction and the
// zone-centred electric field with its WENO limiting.
//
// Follows LIMIT_ALL_SLOPES_P12
// (pkg/inc/cubesphere/400riemann_integrate/421limit_all_slopes_p12.f) and
// ENFORCE_PRESSURE_POSITIVITY_PRIM (440enforce_pressure_positivity_prim.f);
// each kernel names the reference step it implements.  STEPS 7.b and 9.c from
// the resident row weights are in cs_weno.cu, STEP 8.d in cs_adp.cu.
#include "cs_recon.cuh"

namespace cs {

namespace {

// STEP 2 (zone part, 421:597-635) and STEP 5 (421:1497-1628) of one zone.
template <typename R>
__device__ __forceinline__ void prim_zone(const Dims& d, const PhysC& ph, const DGeom& g, const DStateT<R>& s, int p, int i,
                                          int j, int k, const AdpLayers& al) {
  const long long PS = (long long)NPANEL * d.S, o = (long long)p * d.S + d.idx(i, j, k);
  const int m = mask_at(g, d, p, i, j);
  R U[8], V[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) U[c] = s.U[c * PS + o];
  if (m == 0) {
#pragma unroll
    for (int c = 0; c < 8; ++c) U[c] = R(0.0);
    U[0] = R(ph.rhofloor);
    U[4] = R(ph.prsfloor) / (R(ph.gamma) - R(1.0));
  }
  R en = s.ent[o];
  d_cons_to_prim(ph, en, U, V);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    s.U[c * PS + o] = U[c];
    s.V[c * PS + o] = V[c];
  }
  s.ent[o] = en;
  s.ent[PS + o] = R(0.0);
  s.ent[2 * PS + o] = R(0.0);
  s.ent[3 * PS + o] = R(0.0);
  // The higher modes are zero from the start wherever no step writes them.
  // STEP 8.d writes the B modes of the active zones of its range, STEP 7.b all of
  // them on its own zones, which may be a layer less: there the B modes of the
  // last stage go.
  const int lo = 3 - d.G, hx = d.N + d.G - 2, hz = d.nr + d.G - 2;
  const bool full = i >= lo && i <= hx && j >= lo && j <= hx && k >= lo && k <= hz;
  const bool adp = m == 1 && i > -al.side && i <= d.N + al.side && j > -al.side && j <= d.N + al.side && k > -al.radial &&
                   k <= d.nr + al.radial;
  if (adp && !full)
#pragma unroll
    for (int q = 0; q < 27; ++q) s.V[((q / 3 + 1) * NVAR + 5 + q % 3) * PS + o] = R(0.0);
  const R a12 = (V[5] * V[5] + V[6] * V[6] + V[7] * V[7]) * R(ph.ob4pi);
  s.msonic[o] = sqrt((R(ph.gamma) * V[4] + a12) / V[0]);
}

// Masked-face zeroing (421:658-759; 485:383-484) of the faces at one index.
template <typename R>
__device__ __forceinline__ void mask_faces(const Dims& d, const DGeom& g, const DStateT<R>& s, int p, int i, int j, int k) {
  const int lo = 1 - d.G, hi = d.N + d.G;
  // zones are masked at the panel corners only
  const bool ci = i <= 1 || i >= d.N, cj = j <= 1 || j >= d.N;
  if (!(ci && cj)) return;
  if (k >= lo && j >= lo && mask_at(g, d, p, max(i, lo), j) == 0 && mask_at(g, d, p, min(i + 1, hi), j) == 0)
    s.Bxf[d.at(0, p, i, j, k)] = 0.0;
  if (k >= lo && i >= lo && mask_at(g, d, p, i, max(j, lo)) == 0 && mask_at(g, d, p, i, min(j + 1, hi)) == 0)
    s.Byf[d.at(0, p, i, j, k)] = 0.0;
  if (i >= lo && j >= lo && mask_at(g, d, p, i, j) == 0) s.Bzf[d.at(0, p, i, j, k)] = 0.0;
}

// The primitives of every zone and the masked faces, one thread an index
// (the box has one more face than zones along each axis).
template <typename R>
__global__ void __launch_bounds__(TPB) k_prim(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r, AdpLayers al) {
  const int lo = 1 - d.G;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    mask_faces(d, g, s, p, i, j, k);
    if (i >= lo && j >= lo && k >= lo) prim_zone(d, ph, g, s, p, i, j, k, al);
  }
}

template <typename R>
__global__ void k_zero_masked_faces(Dims d, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    mask_faces(d, g, s, p, i, j, k);
  }
}

// Tri-corner face-B synchronisation (421:779-962; 485:504-687).  One
// thread per (panel, corner, ghost column, k).
template <typename R>
__global__ void k_tricorner(Dims d, DGeom g, DStateT<R> s) {
  const long long n = 6LL * 4 * d.G * (d.NK - 1);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    long long u = t;
    const int k = (int)(u % (d.NK - 1)) + 1 - d.G;
    u /= (d.NK - 1);
    const int col = (int)(u % d.G);
    u /= d.G;
    const int corner = (int)(u % 4);
    const int p = (int)(u / 4);
    const int N = d.N;
    if (corner == 0) {  // LD
      const int i = 1 - d.G + col;
      const int xd = sten(g, d, p, i, 1, 3, 0), yd = sten(g, d, p, i, 1, 3, 1);
      double& a = s.Byf[d.at(0, p, i, 0, k)];
      double& b = s.Bxf[d.at(0, p, xd - 1, yd, k)];
      const double a11 = 0.5 * (a - b);
      a = a11;
      b = -a11;
    } else if (corner == 1) {  // RD
      const int i = N + 1 + col;
      const int xd = sten(g, d, p, i, 1, 3, 0), yd = sten(g, d, p, i, 1, 3, 1);
      double& a = s.Byf[d.at(0, p, i, 0, k)];
      double& b = s.Bxf[d.at(0, p, xd, yd, k)];
      const double a11 = 0.5 * (a + b);
      a = a11;
      b = a11;
    } else if (corner == 2) {  // RU
      const int i = N + 1 + col;
      const int xu = sten(g, d, p, i, N, 2, 0), yu = sten(g, d, p, i, N, 2, 1);
      double& a = s.Byf[d.at(0, p, i, N, k)];
      double& b = s.Bxf[d.at(0, p, xu, yu, k)];
      const double a11 = 0.5 * (a - b);
      a = a11;
      b = -a11;
    } else {  // LU
      const int i = 1 - d.G + col;
      const int xu = sten(g, d, p, i, N, 2, 0), yu = sten(g, d, p, i, N, 2, 1);
      double& a = s.Byf[d.at(0, p, i, N, k)];
      double& b = s.Bxf[d.at(0, p, xu - 1, yu, k)];
      const double a11 = 0.5 * (a + b);
      a = a11;
      b = a11;
    }
  }
}

// STEP 6.a (421:1837-2131): velocity divergence and the divergence flattener.
template <typename R>
__global__ void k_flat_a(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const int lo = 2 - d.G, hx = d.N + d.G - 1, hz = d.nr + d.G - 1;
    R fl = R(0.0);
    if (i >= lo && i <= hx && j >= lo && j <= hx && k >= lo && k <= hz) {
      const int xr = sten(g, d, p, i, j, 0, 0), yr = sten(g, d, p, i, j, 0, 1);
      const int xl = sten(g, d, p, i, j, 1, 0), yl = sten(g, d, p, i, j, 1, 1);
      const int xu = sten(g, d, p, i, j, 2, 0), yu = sten(g, d, p, i, j, 2, 1);
      const int xd = sten(g, d, p, i, j, 3, 0), yd = sten(g, d, p, i, j, 3, 1);
      const R obl0 = R(1.0) / fmax(geoR<R>(g, d, CS_G_V_SCALE, 0, p, i, j, k), R(ph.smallnum));
      const R* ms = s.msonic;
      R w = ms[d.at(0, p, i, j, k)];
      w = fmin(w, ms[d.at(0, p, xr, yr, k)]);
      w = fmin(w, ms[d.at(0, p, xl, yl, k)]);
      w = fmin(w, ms[d.at(0, p, xu, yu, k)]);
      w = fmin(w, ms[d.at(0, p, xd, yd, k)]);
      w = fmin(w, ms[d.at(0, p, i, j, k + 1)]);
      w = fmin(w, ms[d.at(0, p, i, j, k - 1)]);
      R dv = R(0.0);
      auto term = [&](int ax, int ay, int az, int bx, int by, int bz, R nx, R ny, R nz) {
        const R x = (geoR<R>(g, d, CS_G_V_CEN, 0, p, bx, by, bz) - geoR<R>(g, d, CS_G_V_CEN, 0, p, ax, ay, az)) * obl0;
        const R y = (geoR<R>(g, d, CS_G_V_CEN, 1, p, bx, by, bz) - geoR<R>(g, d, CS_G_V_CEN, 1, p, ax, ay, az)) * obl0;
        const R z = (geoR<R>(g, d, CS_G_V_CEN, 2, p, bx, by, bz) - geoR<R>(g, d, CS_G_V_CEN, 2, p, ax, ay, az)) * obl0;
        const R a11 = R(0.5) / fmax(sqrt(x * x + y * y + z * z), R(ph.smallnum));
        dv = dv + nx * a11 * (Vat(s, d, 1, 0, p, bx, by, bz) - Vat(s, d, 1, 0, p, ax, ay, az)) +
             ny * a11 * (Vat(s, d, 2, 0, p, bx, by, bz) - Vat(s, d, 2, 0, p, ax, ay, az)) +
             nz * a11 * (Vat(s, d, 3, 0, p, bx, by, bz) - Vat(s, d, 3, 0, p, ax, ay, az));
      };
      term(i, j, k, xr, yr, k, geoR<R>(g, d, CS_G_XF_N, 0, p, i, j, k), geoR<R>(g, d, CS_G_XF_N, 1, p, i, j, k),
           geoR<R>(g, d, CS_G_XF_N, 2, p, i, j, k));
      term(xl, yl, k, i, j, k, geoR<R>(g, d, CS_G_XF_N, 0, p, i - 1, j, k), geoR<R>(g, d, CS_G_XF_N, 1, p, i - 1, j, k),
           geoR<R>(g, d, CS_G_XF_N, 2, p, i - 1, j, k));
      term(i, j, k, xu, yu, k, geoR<R>(g, d, CS_G_YF_N, 0, p, i, j, k), geoR<R>(g, d, CS_G_YF_N, 1, p, i, j, k),
           geoR<R>(g, d, CS_G_YF_N, 2, p, i, j, k));
      term(xd, yd, k, i, j, k, geoR<R>(g, d, CS_G_YF_N, 0, p, i, j - 1, k), geoR<R>(g, d, CS_G_YF_N, 1, p, i, j - 1, k),
           geoR<R>(g, d, CS_G_YF_N, 2, p, i, j - 1, k));
      R nx = geoR<R>(g, d, CS_G_ZF_CEN, 0, p, i, j, k), ny = geoR<R>(g, d, CS_G_ZF_CEN, 1, p, i, j, k),
             nz = geoR<R>(g, d, CS_G_ZF_CEN, 2, p, i, j, k);
      const R a12 = R(1.0) / fmax(sqrt(nx * nx + ny * ny + nz * nz), R(ph.smallnum));
      nx = nx * a12;
      ny = ny * a12;
      nz = nz * a12;
      term(i, j, k, i, j, k + 1, nx, ny, nz);
      term(i, j, k - 1, i, j, k, nx, ny, nz);
      R a13 = fabs(dv) / (R(ph.flatten_coef) * w);
      a13 = a13 - R(1.0);
      fl = (a13 <= R(0.0)) ? R(0.0) : fmin(R(1.0), a13);
      if (mask_at(g, d, p, i, j) != 1) fl = R(0.0);
    }
    s.flatA[d.at(0, p, i, j, k)] = fl;
  }
}

// STEP 6.b (pressure-ratio raise, pass 0) and 6.c (upwinding, pass 1),
// 421:2150-2458: dst(self) = max over the six neighbours of src.
template <typename R>
__global__ void k_flat_bc(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r, const R* src, R* dst, int pass) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const int lo = 2 - d.G, hx = d.N + d.G - 1, hz = d.nr + d.G - 1;
    R fl = src[d.at(0, p, i, j, k)];
    if (i >= lo && i <= hx && j >= lo && j <= hx && k >= lo && k <= hz) {
      int xs[6], ys[6];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        xs[w] = sten(g, d, p, i, j, w, 0);
        ys[w] = sten(g, d, p, i, j, w, 1);
      }
      xs[4] = xs[5] = i;
      ys[4] = ys[5] = j;
      const int zs[6] = {k, k, k, k, k + 1, k - 1};
      const R p0 = Vat(s, d, 4, 0, p, i, j, k);
#pragma unroll
      for (int w = 0; w < 6; ++w) {
        const bool take = pass == 1 || (Vat(s, d, 4, 0, p, xs[w], ys[w], zs[w]) > R(ph.prs_flatten_coef) * p0);
        if (take) fl = fmax(fl, src[d.at(0, p, xs[w], ys[w], zs[w])]);
      }
    }
    dst[d.at(0, p, i, j, k)] = fl;
  }
}

__constant__ Stencil18 c_n18 = stencil18();  // for run-time rows

struct Nbr12 {
  int x[12], y[12];
};
__device__ __forceinline__ Nbr12 load_nbr(const DGeom& g, const Dims& d, int p, int i, int j) {
  Nbr12 n;
#pragma unroll
  for (int w = 0; w < 12; ++w) {
    n.x[w] = sten(g, d, p, i, j, w, 0);
    n.y[w] = sten(g, d, p, i, j, w, 1);
  }
  return n;
}

// STEP 7.a and STEP 9.b: the WENO-AO slopes (421:2465-3807, 421:6840-8400)
// with the work of a zone spread over three threads.  A block takes 32 zones;
// warp w first forms stencils w, w + 3, w + 6 of each zone's eight one-sided
// 3x3 stencils (two in-plane neighbours and one radial, 421:2561-3110) as
// closed-form inverses of the scaled centroid offsets into shared memory;
// then, for its variables, the eight stencil gradients and their mean and
// combines them with the WENO weights (IS + eps)^-4, central weight 100
// (421:3116-3432), so no thread keeps the 72 inverse entries in registers.
//   W7_PRIM  primitives 0-7 and (8) the entropy, variables w, w + 3, w + 6
//   W7_E     E component w
//   W7_ENT   the entropy only, by the last warp (LIMIT_ALL_SLOPES_P2's STEP
//            7.a, 420:5396-6306; k_p2_prim does its primitives)
//
// What bounds it: FP64 instructions (the weights are FP64 in every form) and
// latency at 18 (FP32: 24) warps an SM.  The neighbours are box offsets in
// shared memory (tables indexed at run time lived in local memory), a
// variable's values are loaded while the one before is worked on, and the nine
// weights take Newton reciprocals.  ms of a 6 x 128^2 x 64 step, before / now:
// STEP 7.a 7.1 / 4.6 (FP32 5.5 / 3.6), STEP 9.b 4.0 / 2.2 (3.1 / 1.8).
enum W7Kind { W7_PRIM, W7_E, W7_ENT };
constexpr int W7A_ZT = 32;
template <W7Kind kK, typename R>
__global__ void __launch_bounds__(W7A_ZT * 3, sizeof(R) == 4 ? 8 : 6) k_weno_slopes(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  __shared__ R ai[72][W7A_ZT];  // [stencil * 9 + entry][zone]
  __shared__ int nbo[4][W7A_ZT];  // box offsets of the R, L, U, D neighbours
  const int zl = threadIdx.x % W7A_ZT, w = threadIdx.x / W7A_ZT;
  const unsigned nz = (unsigned)r.count(), ntile = (nz + W7A_ZT - 1) / W7A_ZT;
  const int plane = d.NI * d.NJ;
  const long long PS = (long long)NPANEL * d.S;
  constexpr int nv = kK == W7_PRIM ? 9 : 3;
  for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x) {
    const unsigned t = T * W7A_ZT + zl;
    int p = 0, i = 0, j = 0, k = 0;
    bool act = t < nz;
    if (act) {
      r.decode(t, p, i, j, k);
      act = mask_at(g, d, p, i, j) == 1;
    }
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    if (act) {
      nbo[w][zl] = (sten(g, d, p, i, j, w, 1) - j) * d.NI + (sten(g, d, p, i, j, w, 0) - i);
      if (w == 0) nbo[3][zl] = (sten(g, d, p, i, j, 3, 1) - j) * d.NI + (sten(g, d, p, i, j, 3, 0) - i);
    }
    __syncthreads();
    // variable q's value and its differences to R, L, U, D, up, down
    auto load = [&](int q, R& f0, R (&D)[6]) {
      const R* f = (kK == W7_E ? s.Esnap + q * PS : (kK == W7_PRIM && q < 8 ? s.V + q * PS : s.ent)) + o;
      f0 = f[0];
#pragma unroll
      for (int a = 0; a < 4; ++a) D[a] = f[nbo[a][zl]];
      D[4] = f[plane];
      D[5] = f[-plane];
    };
    const bool mine = act && (kK != W7_ENT || w == 2);
    R f0 = R(0.0), D[6];
    if (mine) load(w, f0, D);
    if (act) {
      const double* cen = g.f[CS_G_V_CEN] + o;
      const R obl0 = R(1.0) / fmax((R)__ldg(g.f[CS_G_V_SCALE] + o), R(ph.smallnum));
      const R cx = (R)__ldg(cen), cy = (R)__ldg(cen + PS), cz = (R)__ldg(cen + 2 * PS);
      // stencil st: neighbour (st >> 1) & 1 (R, L), 2 + (st >> 2) (U, D), dz +1 (even) or -1
#pragma unroll 1
      for (int st = w; st < 8; st += 3) {
        const int o1 = nbo[(st >> 1) & 1][zl], o2 = nbo[2 + (st >> 2)][zl], o3 = (st & 1) ? -plane : plane;
        const R a11 = ((R)__ldg(cen + o1) - cx) * obl0, a12 = ((R)__ldg(cen + PS + o1) - cy) * obl0,
                a13 = ((R)__ldg(cen + 2 * PS + o1) - cz) * obl0;
        const R a21 = ((R)__ldg(cen + o2) - cx) * obl0, a22 = ((R)__ldg(cen + PS + o2) - cy) * obl0,
                a23 = ((R)__ldg(cen + 2 * PS + o2) - cz) * obl0;
        const R a31 = ((R)__ldg(cen + o3) - cx) * obl0, a32 = ((R)__ldg(cen + PS + o3) - cy) * obl0,
                a33 = ((R)__ldg(cen + 2 * PS + o3) - cz) * obl0;
        R ob = (-a13 * a22 * a31 + a12 * a23 * a31 + a13 * a21 * a32 - a11 * a23 * a32 - a12 * a21 * a33 + a11 * a22 * a33);
        ob = copysign(R(1.0), ob) / fmax(R(1.0e-32), fabs(ob));
        ai[st * 9 + 0][zl] = (-a23 * a32 + a22 * a33) * ob;
        ai[st * 9 + 1][zl] = (a13 * a32 - a12 * a33) * ob;
        ai[st * 9 + 2][zl] = (-a13 * a22 + a12 * a23) * ob;
        ai[st * 9 + 3][zl] = (a23 * a31 - a21 * a33) * ob;
        ai[st * 9 + 4][zl] = (-a13 * a31 + a11 * a33) * ob;
        ai[st * 9 + 5][zl] = (a13 * a21 - a11 * a23) * ob;
        ai[st * 9 + 6][zl] = (-a22 * a31 + a21 * a32) * ob;
        ai[st * 9 + 7][zl] = (a12 * a31 - a11 * a32) * ob;
        ai[st * 9 + 8][zl] = (-a12 * a21 + a11 * a22) * ob;
      }
    }
    __syncthreads();
    if (mine) {
#pragma unroll 1
      for (int q = kK == W7_ENT ? 8 : w; q < (kK == W7_ENT ? 9 : nv); q += 3) {
        R g0 = R(0.0), Dn[6];
        if (q + 3 < nv) load(q + 3, g0, Dn);
#pragma unroll
        for (int a = 0; a < 6; ++a) D[a] = D[a] - f0;
        R X[3][9];
#pragma unroll
        for (int st = 0; st < 8; ++st) {
          const R R0 = D[(st >> 1) & 1], R1 = D[2 + (st >> 2)], R2 = D[4 + (st & 1)];
#pragma unroll
          for (int rr = 0; rr < 3; ++rr)
            X[rr][st] = ai[st * 9 + rr * 3 + 0][zl] * R0 + ai[st * 9 + rr * 3 + 1][zl] * R1 + ai[st * 9 + rr * 3 + 2][zl] * R2;
        }
#pragma unroll
        for (int rr = 0; rr < 3; ++rr)
          X[rr][8] = R(0.125) * (X[rr][0] + X[rr][1] + X[rr][2] + X[rr][3] + X[rr][4] + X[rr][5] + X[rr][6] + X[rr][7]);
        // The nonlinear weights (IS + eps)^-4 span far more than the FP32
        // range, so they are formed in FP64 in every form; accumulated
        // stencil by stencil and normalised at the end.
        double sw = 0.0, t0 = 0.0, t1 = 0.0, t2 = 0.0;
#pragma unroll
        for (int st = 0; st < 9; ++st) {
          const double x0 = X[0][st], x1 = X[1][st], x2 = X[2][st];
          const double v = rcp_any(x0 * x0 + x1 * x1 + x2 * x2 + ph.smallnum), v2 = v * v;
          const double W = st < 8 ? v2 * v2 : 100.0 * (v2 * v2);
          sw = sw + W;
          t0 = t0 + W * x0;
          t1 = t1 + W * x1;
          t2 = t2 + W * x2;
        }
        const double a11 = 1.0 / sw;
        const R gr[3] = {(R)(t0 * a11), (R)(t1 * a11), (R)(t2 * a11)};
        if (kK == W7_E) {
#pragma unroll
          for (int m = 0; m < 3; ++m) s.E[(3 * (m + 1) + q) * PS + o] = gr[m];
        } else if (kK == W7_PRIM && q < 8) {
#pragma unroll
          for (int m = 0; m < 3; ++m) s.V[((m + 1) * NVAR + q) * PS + o] = gr[m];
        } else {
          const R om = R(1.0) - s.flatA[o];
#pragma unroll
          for (int m = 0; m < 3; ++m) s.ent[(m + 1) * PS + o] = gr[m] * om;
        }
        f0 = g0;
#pragma unroll
        for (int a = 0; a < 6; ++a) D[a] = Dn[a];
      }
    }
    __syncthreads();
  }
}

// Row rr of the 18 x 9 least-squares matrix of STEP 7.b (421:3869-4001)
// for zone (i,j,k): neighbour centroid offsets scaled by l0, quadratic
// modes corrected by the neighbour's own moments.
template <typename R>
__device__ __forceinline__ void w7b_row(const Dims& d, const PhysC& ph, const DGeom& g, int p, int i, int j, int k,
                                        const Nbr12& n, int rr, R cx, R cy, R cz, R l0, R obl0,
                                        const R* c0, R* A, long long& off) {
  const int w = c_n18.v[rr][0], dz = c_n18.v[rr][1];
  const int zx = w == 12 ? i : n.x[w], zy = w == 12 ? j : n.y[w], zz = k + dz;
  off = d.idx(zx, zy, zz);
  const R x = (geoR<R>(g, d, CS_G_V_CEN, 0, p, zx, zy, zz) - cx) * obl0;
  const R y = (geoR<R>(g, d, CS_G_V_CEN, 1, p, zx, zy, zz) - cy) * obl0;
  const R z = (geoR<R>(g, d, CS_G_V_CEN, 2, p, zx, zy, zz) - cz) * obl0;
  const R lj = fmax(geoR<R>(g, d, CS_G_V_SCALE, 0, p, zx, zy, zz), R(ph.smallnum));
  const R rt = lj / l0, r2 = rt * rt;
  A[0] = x;
  A[1] = y;
  A[2] = z;
  A[3] = x * x - c0[4] + geoR<R>(g, d, CS_G_COEF, 4, p, zx, zy, zz) * r2;
  A[4] = y * y - c0[5] + geoR<R>(g, d, CS_G_COEF, 5, p, zx, zy, zz) * r2;
  A[5] = z * z - c0[6] + geoR<R>(g, d, CS_G_COEF, 6, p, zx, zy, zz) * r2;
  A[6] = x * y - c0[7] + geoR<R>(g, d, CS_G_COEF, 7, p, zx, zy, zz) * r2;
  A[7] = y * z - c0[8] + geoR<R>(g, d, CS_G_COEF, 8, p, zx, zy, zz) * r2;
  A[8] = x * z - c0[9] + geoR<R>(g, d, CS_G_COEF, 9, p, zx, zy, zz) * r2;
}

// Inverse of the 9 x 9 normal matrix A^T A of STEP 7.b for one zone.
template <typename R>
__device__ __forceinline__ void w7b_minv(const Dims& d, const PhysC& ph, const DGeom& g, int p, int i, int j, int k,
                                         const Nbr12& n, R cx, R cy, R cz, R l0, R obl0,
                                         const R* c0, R* Minv) {
  R M[81];
#pragma unroll
  for (int t = 0; t < 81; ++t) M[t] = R(0.0);
  for (int rr = 0; rr < 18; ++rr) {
    R A[9];
    long long off;
    w7b_row(d, ph, g, p, i, j, k, n, rr, cx, cy, cz, l0, obl0, c0, A, off);
#pragma unroll
    for (int a = 0; a < 9; ++a)
#pragma unroll
      for (int b = a; b < 9; ++b) M[a * 9 + b] = M[a * 9 + b] + A[a] * A[b];
  }
#pragma unroll
  for (int a = 0; a < 9; ++a)
#pragma unroll
    for (int b = 0; b < a; ++b) M[a * 9 + b] = M[b * 9 + a];
  d_matinv<9>(M, Minv);
}

// STEP 7.b (421:3869-4551) without resident row weights
// (CS_FLAG_NO_OP_CACHE): 18-zone quadratic least squares hybridised with the
// linear WENO slopes (MRWENO weights, flattener damping), the rows rebuilt
// and the normal matrix inverted in every stage.  With the weights:
// k_weno7b.
template <typename R>
__global__ void __launch_bounds__(TPB) k_weno7b_rebuild(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const Nbr12 n = load_nbr(g, d, p, i, j);
    const R l0 = fmax(geoR<R>(g, d, CS_G_V_SCALE, 0, p, i, j, k), R(ph.smallnum)), obl0 = R(1.0) / l0;
    R c0[10];
    coef10(g, d, p, i, j, k, c0);
    const R cx = geoR<R>(g, d, CS_G_V_CEN, 0, p, i, j, k), cy = geoR<R>(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 cz = geoR<R>(g, d, CS_G_V_CEN, 2, p, i, j, k);
    // formed in FP64 in every form, like the resident row weights; the
    // precision form rounds the inverse once
    R Minv[81];
    {
      double c0d[10], Md[81];
      coef10(g, d, p, i, j, k, c0d);
      const double l0d = fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum);
      w7b_minv<double>(d, ph, g, p, i, j, k, n, geo(g, d, CS_G_V_CEN, 0, p, i, j, k), geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                       geo(g, d, CS_G_V_CEN, 2, p, i, j, k), l0d, 1.0 / l0d, c0d, Md);
#pragma unroll
      for (int e = 0; e < 81; ++e) Minv[e] = (R)Md[e];
    }
    const R f = s.flatA[d.at(0, p, i, j, k)];
    R v0[NVAR], Y[NVAR][9];
#pragma unroll
    for (int q = 0; q < NVAR; ++q) {
      v0[q] = s.V[((long long)q * NPANEL + p) * d.S + d.idx(i, j, k)];
#pragma unroll
      for (int a = 0; a < 9; ++a) Y[q][a] = R(0.0);
    }
#pragma unroll 1
    for (int rr = 0; rr < 18; ++rr) {
      R A[9];
      long long off;
      w7b_row(d, ph, g, p, i, j, k, n, rr, cx, cy, cz, l0, obl0, c0, A, off);
#pragma unroll
      for (int q = 0; q < NVAR; ++q) {
        const R Rv = s.V[((long long)q * NPANEL + p) * d.S + off] - v0[q];
#pragma unroll
        for (int a = 0; a < 9; ++a) Y[q][a] = Y[q][a] + A[a] * Rv;
      }
    }
#pragma unroll
    for (int q = 0; q < NVAR; ++q) {
      R X[9];
#pragma unroll
      for (int a = 0; a < 9; ++a) {
        R sacc = R(0.0);
#pragma unroll
        for (int b = 0; b < 9; ++b) sacc = sacc + Minv[a * 9 + b] * Y[q][b];
        X[a] = sacc;
      }
      const R lin[3] = {Vat(s, d, q, 1, p, i, j, k), Vat(s, d, q, 2, p, i, j, k), Vat(s, d, q, 3, p, i, j, k)};
      R out[9];
      mrweno_hybrid(X, lin, c0, f, R(ph.smallnum), out);
#pragma unroll
      for (int m = 1; m < 10; ++m) Vat(s, d, q, m, p, i, j, k) = out[m - 1];
    }
  }
}

template <typename R>
__global__ void k_ops_m9(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  // shared by the panels: panel 1's zones only (the first sixth of the range)
  const long long nr_ = s.lsq_map9 ? r.count() / 6 : r.count();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nr_; t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const Nbr12 n = load_nbr(g, d, p, i, j);
    const double l0 = fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum), obl0 = 1.0 / l0;
    double c0[10];
    coef10(g, d, p, i, j, k, c0);
    const double cx = geo(g, d, CS_G_V_CEN, 0, p, i, j, k), cy = geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 cz = geo(g, d, CS_G_V_CEN, 2, p, i, j, k);
    double Minv[81];
    w7b_minv(d, ph, g, p, i, j, k, n, cx, cy, cz, l0, obl0, c0, Minv);
    // W_rr = Minv A_rr^T for the 18 stencil rows, [rr * 9 + a][zones]
    for (int rr = 0; rr < 18; ++rr) {
      double A[9];
      long long off;
      w7b_row(d, ph, g, p, i, j, k, n, rr, cx, cy, cz, l0, obl0, c0, A, off);
      for (int a = 0; a < 9; ++a) {
        double w = 0.0;
        for (int b = 0; b < 9; ++b) w = w + Minv[a * 9 + b] * A[b];
        s.op_m9[w_at<162>(t, rr * 9 + a, nr_)] = (R)w;
      }
    }
  }
}

// Node a of the 27 positivity nodes of zone (i,j,k), as its offset from the
// centroid vc scaled by obl0: 0-7 the vertices (bit 0: +x side, bit 1: +y,
// bit 2: +z), 8-13 the face centroids (+x, -x, +y, -y, +z, -z), 14-25 the
// edge midpoints, 26 the centroid.  Read from the geometry where it is
// used, so no thread keeps the 81 coordinates.
__device__ __forceinline__ void pos_vertex(const DGeom& g, const Dims& d, int p, int i, int j, int k, int v,
                                           double* c) {
  const int vi = i - 1 + (v & 1), vj = j - 1 + ((v >> 1) & 1), vk = k - 1 + (v >> 2);
#pragma unroll
  for (int q = 0; q < 3; ++q) c[q] = geo(g, d, CS_G_VERT, q, p, vi, vj, vk);
}

__device__ __forceinline__ void pos_node(const DGeom& g, const Dims& d, int p, int i, int j, int k, int a,
                                         const double* vc, double obl0, double& x, double& y, double& z) {
  double c[3];
  if (a < 8) {
    pos_vertex(g, d, p, i, j, k, a, c);
  } else if (a < 14) {
    const int f = a - 8, dir = f >> 1, lo = f & 1;
    const int F = dir == 0 ? CS_G_XF_CEN : (dir == 1 ? CS_G_YF_CEN : CS_G_ZF_CEN);
    const int fi = i - (dir == 0 ? lo : 0), fj = j - (dir == 1 ? lo : 0), fk = k - (dir == 2 ? lo : 0);
#pragma unroll
    for (int q = 0; q < 3; ++q) c[q] = geo(g, d, F, q, p, fi, fj, fk);
  } else if (a < 26) {
    // vertex pairs along x (0-3), y (4-7), z (8-11)
    const int e = a - 14, ax = e >> 2, w = e & 3;
    int v0;
    if (ax == 0) v0 = 2 * w;
    else if (ax == 1) v0 = (w & 1) | ((w >> 1) << 2);
    else v0 = w;
    const int v1 = v0 | (1 << ax);
    double c0[3], c1[3];
    pos_vertex(g, d, p, i, j, k, v0, c0);
    pos_vertex(g, d, p, i, j, k, v1, c1);
#pragma unroll
    for (int q = 0; q < 3; ++q) c[q] = (c0[q] + c1[q]) * 0.5;
  } else {
#pragma unroll
    for (int q = 0; q < 3; ++q) c[q] = vc[q];
  }
  x = (c[0] - vc[0]) * obl0;
  y = (c[1] - vc[1]) * obl0;
  z = (c[2] - vc[2]) * obl0;
}

// Half extents of a zone over the 27 positivity nodes, max |x|, |y|, |z| of
// their scaled offsets (the edge midpoints and the centroid lie within the
// vertices'), rounded up: geometry only, once per mesh.
__global__ void k_pos_extents(Dims d, PhysC ph, DGeom g, Range3 r, float* ext) {
  const long long PS = (long long)NPANEL * d.S;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const double obl0 = 1.0 / fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum);
    const double vc[3] = {geo(g, d, CS_G_V_CEN, 0, p, i, j, k), geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                          geo(g, d, CS_G_V_CEN, 2, p, i, j, k)};
    double h[3] = {0.0, 0.0, 0.0};
    for (int a = 0; a < 14; ++a) {
      double x, y, z;
      pos_node(g, d, p, i, j, k, a, vc, obl0, x, y, z);
      h[0] = fmax(h[0], fabs(x));
      h[1] = fmax(h[1], fabs(y));
      h[2] = fmax(h[2], fabs(z));
    }
    for (int q = 0; q < 3; ++q) ext[q * PS + p * d.S + d.idx(i, j, k)] = __double2float_ru(h[q] * (1.0 + 1e-12));
  }
}

// The shrink of one zone (440:488-829): the 27 nodal values of density,
// pressure and entropy against the bounds, at most 15 passes.  Returns the
// zone's record: bit 0: gave up; bits 1-4: shrink passes applied.
template <typename R>
__device__ __noinline__ int positivity_shrink(const Dims& d, const PhysC& ph, const DGeom& g, const DStateT<R>& s, int p,
                                              int i, int j, int k, double mn0, double mx0, double mn4, double mx4,
                                              double emin, double emax) {
  const double obl0 = 1.0 / fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum);
  const double vc[3] = {geo(g, d, CS_G_V_CEN, 0, p, i, j, k), geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                        geo(g, d, CS_G_V_CEN, 2, p, i, j, k)};
  double c0[10];
  coef10(g, d, p, i, j, k, c0);
  double vr[10], vp[10], ep[4];
#pragma unroll
  for (int m = 0; m < 10; ++m) {
    vr[m] = Vat(s, d, 0, m, p, i, j, k);
    vp[m] = Vat(s, d, 4, m, p, i, j, k);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) ep[m] = s.ent[d.at(m, p, i, j, k)];
  const int niter = 15;
  const double ratio = pow(0.10, 1.0 / (double)niter);
  int gave_up = 0, nshrink = 0;
  for (int iter = 1; iter <= niter + 1; ++iter) {
    if (iter == niter + 1) {
      gave_up = 1;
      break;
    }
    bool pass = true;
    for (int a = 0; a < 27 && pass; ++a) {
      double x, y, z;
      pos_node(g, d, p, i, j, k, a, vc, obl0, x, y, z);
      const double v1 = d_poly10(vr, c0, x, y, z), v5 = d_poly10(vp, c0, x, y, z);
      const double en = ep[0] + ep[1] * x + ep[2] * y + ep[3] * z;
      if (v1 < mn0 || v1 > mx0 || v5 < mn4 || v5 > mx4 || en < emin || en > emax) pass = false;
    }
    if (pass) break;
#pragma unroll
    for (int m = 1; m < 10; ++m) {
      vr[m] = ratio * vr[m];
      vp[m] = ratio * vp[m];
    }
#pragma unroll
    for (int m = 1; m < 4; ++m) ep[m] = ratio * ep[m];
    ++nshrink;
  }
  if (gave_up || nshrink > 0) {
    for (int q = 0; q < NVAR; ++q)
      for (int m = 1; m < 10; ++m) {
        double v = Vat(s, d, q, m, p, i, j, k);
        if (gave_up) {
          v = 0.0;
        } else {
          for (int it = 0; it < nshrink; ++it) v = ratio * v;
        }
        Vat(s, d, q, m, p, i, j, k) = v;
      }
    for (int m = 1; m < 4; ++m) s.ent[d.at(m, p, i, j, k)] = gave_up ? 0.0 : ep[m];
  }
  return gave_up | (nshrink << 1);
}

// STEP 7.c (440:204-829): the 27 nodal values of density, pressure and
// entropy must lie in the expanded local range, or the zone's higher modes
// shrink.  In FP64 in every form.
//
// Almost every zone passes, so a bound decides first: no node is further
// from the mean than sum_m |mode m| max |basis m| over the zone's extents,
// and where the mean plus and minus that stays inside the range (less a
// margin for the rounding of the nodal sums) the nodes need not be formed.
// The others run the nodes (positivity_shrink), so every zone ends with the
// same record as without the bound.  A thread takes kc zones of a radial
// column and keeps the range of the last three layers: 9 neighbours' loads a
// zone instead of 27.  ms of a 6 x 128^2 x 64 step: 4.35 (FP32 form 5.0) with the
// nodes of every zone, 1.66 (1.63) so; what is left is the reads of the modes.
template <typename R>
__global__ void __launch_bounds__(TPB, 5) k_positivity(Dims d, PhysC ph, DGeom g, DStateT<R> s, const float* __restrict__ ext,
                                                       Range3 r, int kc) {
  const unsigned ni = r.i1 - r.i0 + 1, nj = r.j1 - r.j0 + 1, ncol = 6 * ni * nj;
  const unsigned nseg = (r.k1 - r.k0 + kc) / kc, nt = ncol * nseg;
  const long long PS = (long long)NPANEL * d.S;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
    const unsigned seg = t / ncol, col = t - seg * ncol, u = col / ni;
    const int i = (int)(col - u * ni) + r.i0, j = (int)(u % nj) + r.j0, p = (int)(u / nj);
    const int ka = r.k0 + (int)seg * kc, kb = min(ka + kc - 1, r.k1);
    int nbo[9];
    nbo[0] = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int w = q < 4 ? q : q + 4;
      nbo[q + 1] = (sten(g, d, p, i, j, w, 1) - j) * d.NI + (sten(g, d, p, i, j, w, 0) - i);
    }
    // range of density, pressure and entropy over the nine columns at layer k
    R lo[3][3], hi[3][3];
    auto layer = [&](int k, R (&a)[3], R (&b)[3]) {
      const long long o = (long long)p * d.S + d.idx(i, j, k);
      const R* f[3] = {s.V + o, s.V + 4 * PS + o, s.ent + o};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        a[c] = b[c] = f[c][0];
#pragma unroll
        for (int q = 1; q < 9; ++q) {
          const R v = f[c][nbo[q]];
          a[c] = fmin(a[c], v);
          b[c] = fmax(b[c], v);
        }
      }
    };
    layer(ka - 1, lo[0], hi[0]);
    layer(ka, lo[1], hi[1]);
    for (int k = ka; k <= kb; ++k) {
      layer(k + 1, lo[2], hi[2]);
      const long long o = (long long)p * d.S + d.idx(i, j, k);
      const double ef = 0.2;
      const double ff = fmax(fmin(((double)s.flatA[o] - 0.1) / 0.4, 1.0), 0.0), omff = 1.0 - ff;
      double mn[3], mx[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        mn[c] = (double)fmin(lo[0][c], fmin(lo[1][c], lo[2][c])) * (1.0 - ef * omff);
        mx[c] = (double)fmax(hi[0][c], fmax(hi[1][c], hi[2][c])) * (1.0 + ef * omff);
      }
      mn[0] = fmax(mn[0], ph.rhofloor);
      mx[0] = fmax(mx[0], ph.rhofloor);
      mn[1] = fmax(mn[1], ph.prsfloor);
      mx[1] = fmax(mx[1], ph.prsfloor);
      const double hx = ext[o], hy = ext[PS + o], hz = ext[2 * PS + o];
      const double* cf = g.f[CS_G_COEF] + o;
      const double c4 = fabs(__ldg(cf + 4 * PS)), c5 = fabs(__ldg(cf + 5 * PS)), c6 = fabs(__ldg(cf + 6 * PS));
      // |x x - c| <= max(h h, c); |x y - c| <= h h' + |c|
      const double bb[9] = {hx, hy, hz, fmax(hx * hx, c4), fmax(hy * hy, c5), fmax(hz * hz, c6),
                            hx * hy + fabs(__ldg(cf + 7 * PS)), hy * hz + fabs(__ldg(cf + 8 * PS)),
                            hx * hz + fabs(__ldg(cf + 9 * PS))};
      bool pass = true;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const R* v = c < 2 ? s.V + 4 * c * PS + o : s.ent + o;
        const long long ms = c < 2 ? NVAR * PS : PS;
        const double mean = v[0];
        double dev = 0.0;
#pragma unroll
        for (int m = 1; m < (c < 2 ? 10 : 4); ++m) dev = dev + fabs((double)v[m * ms]) * bb[m - 1];
        const double room = dev > 0.0 ? dev * (1.0 + 1e-12) + 1e-14 * (fabs(mean) + dev) : 0.0;
        pass = pass && mean - room >= mn[c] && mean + room <= mx[c];
      }
      s.giveup[o] = pass ? 0 : positivity_shrink(d, ph, g, s, p, i, j, k, mn[0], mx[0], mn[1], mx[1], mn[2], mx[2]);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        lo[0][c] = lo[1][c];
        lo[1][c] = lo[2][c];
        hi[0][c] = hi[1][c];
        hi[1][c] = hi[2][c];
      }
    }
  }
}

// STEP 8.a-c (421:4686-5567): B at the five quadrature points of each face,
// averaged from both sides and shifted to the facial mean.  One thread a
// face, the three directions in one launch (block T is tile T / 3 of
// direction T % 3, so that L2 serves a zone's modes to all three).
//
// What bounds it: the loads of 30 modes a side.  Evaluating all three
// components of both sides at once took 252 registers, 8 warps an SM.  The
// face normal is one vector on x- and y-faces, so there each side's modes are
// first contracted with it (10 values, one polynomial); on z-faces, where it
// varies over the points, the components are taken one after another.  ms of a
// 6 x 128^2 x 64 step, that / this: 7.7 / 5.6 (FP32 7.4 / 3.9); 5.8
// (4.0) since the third radial layer of ghosts is one of its zones.
template <typename R>
__global__ void __launch_bounds__(TPB, sizeof(R) == 4 ? 6 : 4) k_faceB(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r0, Range3 r1, Range3 r2) {
  const unsigned nt0 = (unsigned)((r0.count() + TPB - 1) / TPB), nt1 = (unsigned)((r1.count() + TPB - 1) / TPB),
                 nt2 = (unsigned)((r2.count() + TPB - 1) / TPB);
  for (unsigned T = blockIdx.x; T < 3 * max(nt0, max(nt1, nt2)); T += gridDim.x) {
    // opaque to the compiler, which would otherwise form the addresses of all
    // planes before the loop and spill them
    long long PS = (long long)NPANEL * d.S;
    asm volatile("" : "+l"(PS));
    const int dir = T % 3;
    const Range3 r = dir == 0 ? r0 : (dir == 1 ? r1 : r2);
    const long long t = (long long)(T / 3) * TPB + threadIdx.x;
    if (t >= r.count()) continue;
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    int lx = i, ly = j, rx = i, ry = j, rz = k;
    bool skip = false;
    if (dir == 0) {
      const int mL = mask_at(g, d, p, i, j), mR = mask_at(g, d, p, i + 1, j);
      rx = i + 1;
      if (mL == 0 && mR == 1) { lx = sten(g, d, p, rx, ry, 1, 0); ly = sten(g, d, p, rx, ry, 1, 1); }
      else if (mL == 1 && mR == 0) { rx = sten(g, d, p, lx, ly, 0, 0); ry = sten(g, d, p, lx, ly, 0, 1); }
      else if (mL == 0 && mR == 0) skip = true;
    } else if (dir == 1) {
      const int mL = mask_at(g, d, p, i, j), mR = mask_at(g, d, p, i, j + 1);
      ry = j + 1;
      if (mL == 0 && mR == 1) { lx = sten(g, d, p, rx, ry, 3, 0); ly = sten(g, d, p, rx, ry, 3, 1); }
      else if (mL == 1 && mR == 0) { rx = sten(g, d, p, lx, ly, 2, 0); ry = sten(g, d, p, lx, ly, 2, 1); }
      else if (mL == 0 && mR == 0) skip = true;
    } else {
      if (mask_at(g, d, p, i, j) == 0) skip = true;
      rz = k + 1;
    }
    const double* qp = (dir == 0 ? g.f[CS_G_XF_QP] : (dir == 1 ? g.f[CS_G_YF_QP] : g.f[CS_G_ZF_QP])) + o;
    const double* qw = (dir == 0 ? g.f[CS_G_XB_QW] : (dir == 1 ? g.f[CS_G_YB_QW] : g.f[CS_G_ZB_QW])) + o;
    const double* nf = (dir == 0 ? g.f[CS_G_XF_N] : (dir == 1 ? g.f[CS_G_YF_N] : g.f[CS_G_ZF_N])) + o;
    // the two sides' values in the state's type; the shift to the facial
    // mean in FP64, so the values average to the FP64 face B exactly
    R bq[5] = {R(0), R(0), R(0), R(0), R(0)};
    if (!skip) {
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        const long long z = (long long)p * d.S + (side ? d.idx(rx, ry, rz) : d.idx(lx, ly, k));
        const R obl = R(1.0) / fmax((R)__ldg(g.f[CS_G_V_SCALE] + z), R(ph.smallnum));
        const double* cen = g.f[CS_G_V_CEN] + z;
        const R cx = (R)__ldg(cen), cy = (R)__ldg(cen + PS), cz = (R)__ldg(cen + 2 * PS);
        R c[10];
#pragma unroll
        for (int m = 4; m < 10; ++m) c[m] = (R)__ldg(g.f[CS_G_COEF] + m * PS + z);
        R px[5], py[5], pz[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          px[q] = ((R)__ldg(qp + q * PS) - cx) * obl;
          py[q] = ((R)__ldg(qp + (5 + q) * PS) - cy) * obl;
          pz[q] = ((R)__ldg(qp + (10 + q) * PS) - cz) * obl;
        }
        const R* v = s.V + 5 * PS + z;
        if (dir < 2) {
          const R n0 = (R)__ldg(nf), n1 = (R)__ldg(nf + PS), n2 = (R)__ldg(nf + 2 * PS);
          R m[10];
#pragma unroll
          for (int a = 0; a < 10; ++a)
            m[a] = n0 * v[a * NVAR * PS] + n1 * v[(a * NVAR + 1) * PS] + n2 * v[(a * NVAR + 2) * PS];
#pragma unroll
          for (int q = 0; q < 5; ++q) bq[q] = bq[q] + d_poly10(m, c, px[q], py[q], pz[q]);
        } else {
#pragma unroll 1
          for (int b = 0; b < 3; ++b) {
            R m[10];
#pragma unroll
            for (int a = 0; a < 10; ++a) m[a] = v[(a * NVAR + b) * PS];
#pragma unroll
            for (int q = 0; q < 5; ++q)
              bq[q] = bq[q] + (R)__ldg(nf + (5 * b + q) * PS) * d_poly10(m, c, px[q], py[q], pz[q]);
          }
        }
      }
    }
    double bd = (dir == 0 ? s.Bxf : (dir == 1 ? s.Byf : s.Bzf))[o];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      bq[q] = R(0.5) * bq[q];
      bd = bd - __ldg(qw + q * PS) * (double)bq[q];
    }
    double* Bq = (dir == 0 ? s.Bq[0] : (dir == 1 ? s.Bq[1] : s.Bq[2])) + o;
#pragma unroll
    for (int q = 0; q < 5; ++q) Bq[q * PS] = (double)bq[q] + bd;
  }
}

// STEP 9.a (421:6700-6790): zone-centred E = -v x B from the point values, on
// the zones z of r.
template <typename R>
__global__ void k_efield_a(Dims d, DGeom g, DStateT<R> s, Range3 r, Range3 z) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    // a zone that exhausted STEP 7.c's shrink passes also zeroes its entropy
    // value (440:569-575), now that every zone has read its neighbours'
    if (s.giveup[d.at(0, p, i, j, k)] & 1) s.ent[d.at(0, p, i, j, k)] = 0.0;
    if (i < z.i0 || i > z.i1 || j < z.j0 || j > z.j1 || k < z.k0 || k > z.k1) continue;
    R co[10];
    coef10(g, d, p, i, j, k, co);
    R pv[8];
    for (int q = 1; q < 8; ++q) {
      if (q == 4) continue;
      R acc = Vat(s, d, q, 0, p, i, j, k);
      for (int m = 4; m < 10; ++m) acc = acc - Vat(s, d, q, m, p, i, j, k) * co[m];
      pv[q] = acc;
    }
    const R vx = pv[1], vy = pv[2], vz = pv[3], Bx = pv[5], By = pv[6], Bz = pv[7];
    const R ex = -(vy * Bz - vz * By), ey = -(vz * Bx - vx * Bz), ez = -(vx * By - vy * Bx);
    s.E[d.at(0, p, i, j, k)] = ex;
    s.E[d.at(1, p, i, j, k)] = ey;
    s.E[d.at(2, p, i, j, k)] = ez;
    s.Esnap[d.at(0, p, i, j, k)] = ex;
    s.Esnap[d.at(1, p, i, j, k)] = ey;
    s.Esnap[d.at(2, p, i, j, k)] = ez;
  }
}

// Row rr (0: the zone itself, 1..18: the STEP 7.b neighbours) of the
// 19 x 10 interpolation least-squares matrix of STEP 9.c (421:8464-8620).
template <typename R>
__device__ __forceinline__ void e9c_row(const Dims& d, const DGeom& g, int p, int i, int j, int k, const Nbr12& n,
                                        int rr, R cx, R cy, R cz, R obl0, const R* c0, R* A,
                                        long long& off) {
  if (rr == 0) {
    off = d.idx(i, j, k);
    A[0] = R(1.0);
    A[1] = R(0.0);
    A[2] = R(0.0);
    A[3] = R(0.0);
#pragma unroll
    for (int m = 4; m < 10; ++m) A[m] = R(0.0) * R(0.0) - c0[m];
    return;
  }
  const int w = c_n18.v[rr - 1][0], dz = c_n18.v[rr - 1][1];
  const int zx = w == 12 ? i : n.x[w], zy = w == 12 ? j : n.y[w], zz = k + dz;
  off = d.idx(zx, zy, zz);
  const R x = (geoR<R>(g, d, CS_G_V_CEN, 0, p, zx, zy, zz) - cx) * obl0;
  const R y = (geoR<R>(g, d, CS_G_V_CEN, 1, p, zx, zy, zz) - cy) * obl0;
  const R z = (geoR<R>(g, d, CS_G_V_CEN, 2, p, zx, zy, zz) - cz) * obl0;
  A[0] = R(1.0);
  A[1] = x;
  A[2] = y;
  A[3] = z;
  A[4] = x * x - c0[4];
  A[5] = y * y - c0[5];
  A[6] = z * z - c0[6];
  A[7] = x * y - c0[7];
  A[8] = y * z - c0[8];
  A[9] = x * z - c0[9];
}

template <typename R>
__device__ __forceinline__ void e9c_minv(const Dims& d, const DGeom& g, int p, int i, int j, int k, const Nbr12& n,
                                         R cx, R cy, R cz, R obl0, const R* c0, R* Minv) {
  R M[100];
#pragma unroll
  for (int t = 0; t < 100; ++t) M[t] = R(0.0);
  for (int rr = 0; rr < 19; ++rr) {
    R A[10];
    long long off;
    e9c_row(d, g, p, i, j, k, n, rr, cx, cy, cz, obl0, c0, A, off);
#pragma unroll
    for (int a = 0; a < 10; ++a)
#pragma unroll
      for (int b = a; b < 10; ++b) M[a * 10 + b] = M[a * 10 + b] + A[a] * A[b];
  }
#pragma unroll
  for (int a = 0; a < 10; ++a)
#pragma unroll
    for (int b = 0; b < a; ++b) M[a * 10 + b] = M[b * 10 + a];
  d_matinv<10>(M, Minv);
}

// STEP 9.c (421:8464-9350) without resident row weights
// (CS_FLAG_NO_OP_CACHE): 19-point interpolation least squares hybridised with
// the slopes, the rows rebuilt and the normal matrix inverted in every stage;
// the point value is flattened toward E_pt.  Only the point value (mode 1) is
// stored: the LLF edge solver consumes nothing else.
template <typename R>
__global__ void __launch_bounds__(TPB) k_efield_c_rebuild(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const Nbr12 n = load_nbr(g, d, p, i, j);
    const R obl0 = R(1.0) / fmax(geoR<R>(g, d, CS_G_V_SCALE, 0, p, i, j, k), R(ph.smallnum));
    R c0[10];
    coef10(g, d, p, i, j, k, c0);
    const R cx = geoR<R>(g, d, CS_G_V_CEN, 0, p, i, j, k), cy = geoR<R>(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 cz = geoR<R>(g, d, CS_G_V_CEN, 2, p, i, j, k);
    // formed in FP64 in every form, like the resident row weights
    R Minv[100];
    {
      double c0d[10], Md[100];
      coef10(g, d, p, i, j, k, c0d);
      e9c_minv<double>(d, g, p, i, j, k, n, geo(g, d, CS_G_V_CEN, 0, p, i, j, k), geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                       geo(g, d, CS_G_V_CEN, 2, p, i, j, k), 1.0 / fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum),
                       c0d, Md);
#pragma unroll
      for (int e = 0; e < 100; ++e) Minv[e] = (R)Md[e];
    }
    R Y[3][10];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int a = 0; a < 10; ++a) Y[q][a] = R(0.0);
#pragma unroll 1
    for (int rr = 0; rr < 19; ++rr) {
      R A[10];
      long long off;
      e9c_row(d, g, p, i, j, k, n, rr, cx, cy, cz, obl0, c0, A, off);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const R Rv = s.Esnap[((long long)q * NPANEL + p) * d.S + off];
#pragma unroll
        for (int a = 0; a < 10; ++a) Y[q][a] = Y[q][a] + A[a] * Rv;
      }
    }
    const R f = s.flatA[d.at(0, p, i, j, k)];
    const R ghi = f * R(0.6) + (R(1.0) - f) * R(0.95), glo = R(1.0) - ghi, obghi = R(1.0) / ghi, grat = glo / ghi;
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {
      R X[10];
#pragma unroll
      for (int a = 0; a < 10; ++a) {
        R acc = R(0.0);
#pragma unroll
        for (int b = 0; b < 10; ++b) acc = acc + Minv[a * 10 + b] * Y[q][b];
        X[a] = acc;
      }
      const R e0 = s.Esnap[((long long)q * NPANEL + p) * d.S + d.idx(i, j, k)];
      const R e[3] = {s.E[d.at(3 + q, p, i, j, k)], s.E[d.at(6 + q, p, i, j, k)], s.E[d.at(9 + q, p, i, j, k)]};
      R Wlo, Whi, Phi[9];
      mrweno_weights(X + 1, e, c0, f, ghi, glo, obghi, grat, R(ph.smallnum), Phi, Wlo, Whi);
      const R eh = Whi * (X[0] * obghi - e0 * grat) + Wlo * e0;
      s.E[d.at(q, p, i, j, k)] = e0 * f + eh * (R(1.0) - f);
    }
  }
}

template <typename R>
__global__ void k_ops_m10(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  const long long nr_ = s.lsq_map10 ? r.count() / 6 : r.count();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nr_; t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const Nbr12 n = load_nbr(g, d, p, i, j);
    const double obl0 = 1.0 / fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum);
    double c0[10];
    coef10(g, d, p, i, j, k, c0);
    const double cx = geo(g, d, CS_G_V_CEN, 0, p, i, j, k), cy = geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 cz = geo(g, d, CS_G_V_CEN, 2, p, i, j, k);
    double Minv[100];
    e9c_minv(d, g, p, i, j, k, n, cx, cy, cz, obl0, c0, Minv);
    // W_rr = Minv A_rr^T for the 19 rows (the zone and its 18 neighbours)
    for (int rr = 0; rr < 19; ++rr) {
      double A[10];
      long long off;
      e9c_row(d, g, p, i, j, k, n, rr, cx, cy, cz, obl0, c0, A, off);
      for (int a = 0; a < 10; ++a) {
        double w = 0.0;
        for (int b = 0; b < 10; ++b) w = w + Minv[a * 10 + b] * A[b];
        s.op_m10[w_at<190>(t, rr * 10 + a, nr_)] = (R)w;
      }
    }
  }
}

// ---------------------------------------------------------------------
// LIMIT_ALL_SLOPES_P2 (400riemann_integrate/420limit_all_slopes_p2.f,
// CS_FLAG_P2): STEP 7.a of the primitives (420:2459-5394) and STEP 9.b of E
// (420:8553-12285), the two steps where it differs from P12.
//
// Row rr (0..8) of one-sided stencil st around (i, j, k).  The stencils, in
// the reference's order (420:2596-4329): (R,U,+1), (L,U,+1), (L,D,+1),
// (R,D,+1), then the same with radial offset -1; with a the R / L
// neighbour, b the U / D neighbour and dz the radial direction, the rows are
// a, b, the zone at dz, aa, bb, the zone at 2 dz, the corner between a and
// b, a at dz, b at dz.  With rr a compile-time constant (unrolled loop)
// each neighbour is a select among registers, whatever st is.
__device__ __forceinline__ void p2_zone(const Nbr12& n, int st, int rr, int i, int j, int k, int& zx, int& zy,
                                        int& zz) {
  const int q = st & 3, dz = st < 4 ? 1 : -1;
  const bool R_ = q == 0 || q == 3, U_ = q < 2;
  zx = i;
  zy = j;
  zz = k;
  switch (rr) {
    case 0: case 7:  // a
      zx = R_ ? n.x[0] : n.x[1];
      zy = R_ ? n.y[0] : n.y[1];
      break;
    case 1: case 8:  // b
      zx = U_ ? n.x[2] : n.x[3];
      zy = U_ ? n.y[2] : n.y[3];
      break;
    case 3:  // aa
      zx = R_ ? n.x[4] : n.x[5];
      zy = R_ ? n.y[4] : n.y[5];
      break;
    case 4:  // bb
      zx = U_ ? n.x[6] : n.x[7];
      zy = U_ ? n.y[6] : n.y[7];
      break;
    case 6:  // corner RU, LU, LD, RD
      zx = q == 0 ? n.x[8] : (q == 1 ? n.x[9] : (q == 2 ? n.x[10] : n.x[11]));
      zy = q == 0 ? n.y[8] : (q == 1 ? n.y[9] : (q == 2 ? n.y[10] : n.y[11]));
      break;
    default: break;
  }
  if (rr == 2 || rr == 7 || rr == 8) zz = k + dz;
  if (rr == 5) zz = k + 2 * dz;
}

// The inverses of every zone's eight one-sided stencil matrices (geometry
// only), built once per mesh: STEP 7.a's 9 x 9 RECONSTRUCTION_COEFS systems
// (the modes x .. xz from the zone-average differences) into
// op_p2v (word (st * 9 + m) * 9 + rr of blocks of 32 zones,
// [block][648][32]: a stencil is one bulk copy) and STEP 9.b's 10 x 10
// INTERPOLATION_COEFS systems (the zone itself first, modes 1 .. xz from
// the point values) into op_p2e[(st * 10 + m) * 10 + rr][zone], inverted by
// MATINV's LU (121matinv.f:8).  Shared by the panels: panel 1's zones only.
template <typename R>
__global__ void k_ops_p2(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  const long long nr_ = s.p2_map ? r.count() / 6 : r.count();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nr_; t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const Nbr12 n = load_nbr(g, d, p, i, j);
    const double l0 = fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum), obl0 = 1.0 / l0;
    double c0[10];
    coef10(g, d, p, i, j, k, c0);
    const double cx = geo(g, d, CS_G_V_CEN, 0, p, i, j, k), cy = geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 cz = geo(g, d, CS_G_V_CEN, 2, p, i, j, k);
    for (int st = 0; st < 8; ++st) {
      double A[81], Ai[81], B[100], Bi[100];
      for (int m = 0; m < 10; ++m) B[m] = m == 0 ? 1.0 : (m < 4 ? 0.0 : 0.0 * 0.0 - c0[m]);
      for (int rr = 0; rr < 9; ++rr) {
        int zx, zy, zz;
        p2_zone(n, st, rr, i, j, k, zx, zy, zz);
        const double x = (geo(g, d, CS_G_V_CEN, 0, p, zx, zy, zz) - cx) * obl0;
        const double y = (geo(g, d, CS_G_V_CEN, 1, p, zx, zy, zz) - cy) * obl0;
        const double z = (geo(g, d, CS_G_V_CEN, 2, p, zx, zy, zz) - cz) * obl0;
        const double lj = fmax(geo(g, d, CS_G_V_SCALE, 0, p, zx, zy, zz), ph.smallnum);
        const double rt = lj / l0, r2 = rt * rt;
        const double sq[6] = {x * x, y * y, z * z, x * y, y * z, x * z};
        double* a = A + 9 * rr;
        a[0] = x;
        a[1] = y;
        a[2] = z;
        for (int m = 0; m < 6; ++m) a[3 + m] = sq[m] - c0[4 + m] + geo(g, d, CS_G_COEF, 4 + m, p, zx, zy, zz) * r2;
        double* e = B + 10 * (rr + 1);
        e[0] = 1.0;
        e[1] = x;
        e[2] = y;
        e[3] = z;
        for (int m = 0; m < 6; ++m) e[4 + m] = sq[m] - c0[4 + m];
      }
      d_matinv<9>(A, Ai);
      d_matinv<10>(B, Bi);
      for (int e = 0; e < 81; ++e) s.op_p2v[(t / 32 * 648 + st * 81 + e) * 32 + t % 32] = (R)Ai[e];
      for (int e = 0; e < 100; ++e) s.op_p2e[(long long)(st * 100 + e) * nr_ + t] = (R)Bi[e];
    }
  }
}

// STEP 7.a of LIMIT_ALL_SLOPES_P2.  A block takes 32 zones, a warp two of the 8
// primitives.  For each of the eight one-sided stencils a thread forms its
// primitives' modes from the resident inverse, their smoothness indicator over
// the zone's unit cube (420:5245-5257) and the WENO weight 1 / (IS +
// smallnum)^4 (in FP64 in every form), and adds the weighted modes; then the
// central stencil (STEP 7.b's resident row weights) with weight 100, and the
// sum is normalised, so that no stencil is formed twice.  Modes 2..10 are
// stored damped by the flattener.
//
// A producer warp brings the inverses, a stencil a stage, through a ring of
// bulk copies; a stencil's neighbour values are loaded while the one before is
// worked on.  With kShared the inverses are panel 1's, rotated per panel like
// the row weights, and tile T is tile T / 6 of panel T % 6, so that L2 serves
// them to six blocks.
//
// What bounds it: shared-memory reads of the inverses, one per two
// multiply-adds, at the 12 to 16 warps its registers allow.  Two warps that
// read every word from L2 themselves, twice (once for the indicators, once for
// the modes), with four primitives a thread in 255 registers, took 13.4 ms of a
// 6 x 64^2 x 32 step in FP64; this takes 7.6.
constexpr int P2_NW = 4;  // warps of a block but the producer
constexpr int P2_CONS = 32 * P2_NW;
constexpr int P2_THREADS = P2_CONS + 32;
// blocks an SM: three in FP64, with some of the sums in local memory, measured
// 7.6 ms a step, two without that 8.2
constexpr int p2_blocks(size_t word) { return word == 4 ? 4 : 3; }
template <typename R>
struct P2Smem {
  static constexpr int NS = sizeof(R) == 4 ? 3 : 2;
  R stage[NS][81][32];
  int nbo[2][13][32];  // in-plane neighbours as box offsets (12: the zone), alternating over the tiles
  uint64_t full[NS];
  uint64_t empty[NS];
};
template <bool kShared, typename R>
__global__ void __launch_bounds__(P2_THREADS, p2_blocks(sizeof(R))) k_p2_prim(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  using Smem = P2Smem<R>;
  extern __shared__ __align__(128) unsigned char p2_raw[];
  Smem& S = *reinterpret_cast<Smem*>(p2_raw);
  const int tid = threadIdx.x;
  const long long nz = r.count(), npp = nz / 6;
  const unsigned nw = (unsigned)(kShared ? npp : nz), ntile = kShared ? 6 * ((nw + 31) / 32) : (nw + 31) / 32;
  if (tid == 0) {
    for (int q = 0; q < Smem::NS; ++q) {
      mbar_init(&S.full[q], 1);
      mbar_init(&S.empty[q], P2_NW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  RingPos<Smem::NS> ring;
  if (tid >= P2_CONS) {
    if (tid == P2_CONS) {
      const R* op = s.op_p2v;
      constexpr uint32_t bytes = 81 * 32 * sizeof(R);
      bool first = true;  // the ring's first round finds every stage free
      for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x) {
        const R* src = op + (long long)(kShared ? T / 6 : T) * (8 * 81 * 32);
        for (int st = 0; st < 8; ++st) {
          if (!first) mbar_wait(&S.empty[ring.slot], ring.par ^ 1, s.err_flag);
          mbar_expect_tx(&S.full[ring.slot], bytes);
          bulk_g2s(&S.stage[ring.slot][0][0], src + st * (81 * 32), bytes, &S.full[ring.slot]);
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
  for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x, buf ^= 1) {
    const unsigned tw = (kShared ? T / 6 : T) * 32 + lane;
    bool act = tw < nw;
    const long long t = kShared ? (T % 6) * npp + tw : tw;
    int p = 0, i = r.i0, j = r.j0, k = r.k0;
    if (act) {
      r.decode(t, p, i, j, k);
      act = mask_at(g, d, p, i, j) == 1;
    }
    int(&nbo)[13][32] = S.nbo[buf];
    if (act) {
      for (int n = w; n < 12; n += P2_NW) {
        nbo[n][lane] = (sten(g, d, p, i, j, n, 1) - j) * d.NI + (sten(g, d, p, i, j, n, 0) - i);
      }
    }
    if (w == 0) nbo[12][lane] = 0;
    // the offsets are complete; the other copy is no longer read
    consumer_sync<P2_CONS>();
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    const R* f = s.V + 2 * w * PS + o;
    // smoothness weight of the modes xx .. xz over the unit cube (x y z: 1 /
    // 12).  The one-sided stencils' modes stay in panel 1's frame (with
    // kShared) and so take panel 1's moments; their sum is rotated once.
    double wis[6];
    auto cube_weights = [&](long long z) {
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        const double c = act ? __ldg(g.f[CS_G_COEF] + (4 + m) * PS + z) : 0.0;
        wis[m] = m < 3 ? sqr(c - 1.0 / 12.0) + 1.0 / 180.0 : sqr(c) + 1.0 / 144.0;
      }
    };
    cube_weights(kShared ? d.idx(i, j, k) : o);
    auto smooth = [&](const R* X) {  // X: modes x .. xz
      return ((double)X[0] * X[0] + (double)X[1] * X[1] + (double)X[2] * X[2]) * (1.0 / 12.0) +
             ((double)X[3] * X[3]) * wis[0] + ((double)X[4] * X[4]) * wis[1] + ((double)X[5] * X[5]) * wis[2] +
             ((double)X[6] * X[6]) * wis[3] + ((double)X[7] * X[7]) * wis[4] + ((double)X[8] * X[8]) * wis[5];
    };
    R f0[2];
    double sw[2], acc[2][9];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      f0[c] = act ? f[c * PS] : R(0.0);
      sw[c] = 0.0;
#pragma unroll
      for (int m = 0; m < 9; ++m) acc[c][m] = 0.0;
    }
    auto add = [&](int c, const R* X, double w0) {  // weighted modes of one stencil
      const double v = rcp_any(smooth(X) + ph.smallnum), v2 = v * v, W = w0 * (v2 * v2);
      sw[c] = sw[c] + W;
#pragma unroll
      for (int m = 0; m < 9; ++m) acc[c][m] = acc[c][m] + W * (double)X[m];
    };
    // the nine zones of stencil st (p2_zone's order)
    auto load = [&](int st, R (&D)[2][9]) {
      const int q = st & 3, dz = st < 4 ? plane : -plane, right = q == 0 || q == 3 ? 0 : 1, up = q < 2 ? 0 : 1;
      const int oa = nbo[right][lane], ob = nbo[2 + up][lane];
      const int off[9] = {oa, ob, dz, nbo[4 + right][lane], nbo[6 + up][lane], 2 * dz, nbo[8 + q][lane], oa + dz, ob + dz};
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int rr = 0; rr < 9; ++rr) D[c][rr] = act ? f[c * PS + off[rr]] : R(0.0);
    };
    R D[2][9];
    load(0, D);
#pragma unroll 1
    for (int st = 0; st < 8; ++st) {
      R Dn[2][9];
      if (st < 7) load(st + 1, Dn);
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int rr = 0; rr < 9; ++rr) D[c][rr] = D[c][rr] - f0[c];
      if (!mbar_try_wait(&S.full[ring.slot], ring.par)) mbar_wait(&S.full[ring.slot], ring.par, s.err_flag);
      const R(&A)[81][32] = S.stage[ring.slot];
      R Y[2][9];
#pragma unroll
      for (int m = 0; m < 9; ++m) {
#pragma unroll
        for (int c = 0; c < 2; ++c) Y[c][m] = R(0.0);
#pragma unroll
        for (int rr = 0; rr < 9; ++rr) {
          const R a = A[m * 9 + rr][lane];
#pragma unroll
          for (int c = 0; c < 2; ++c) Y[c][m] = Y[c][m] + a * D[c][rr];
        }
      }
      ring_release(&S.empty[ring.slot], lane);
      ring.next();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        add(c, Y[c], 1.0);
#pragma unroll
        for (int rr = 0; rr < 9; ++rr) D[c][rr] = Dn[c][rr];
      }
    }
    if (!act) continue;
    if (kShared) {
      cube_weights(o);
      const unsigned long long qsrc = s.p2_map[p].src;
      const unsigned int qneg = s.p2_map[p].neg;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        double a1[9];
#pragma unroll
        for (int m = 0; m < 9; ++m) a1[m] = acc[c][m];
#pragma unroll
        for (int m = 0; m < 9; ++m) acc[c][m] = lsq_rotated<1>(a1, m + 1, qsrc, qneg);
      }
    }
    {  // central stencil from the resident row weights
      R Y[2][9];
      const LsqPanelMap* cmap = s.lsq_map9;
      const long long tc = cmap ? t - (long long)p * npp : t, ncw = cmap ? npp : nz;
      const WBlock cb = w_block<162>(tc / 32, ncw);
      const R* wc = s.op_m9 + cb.off + tc % 32;
      const long long cstride = cb.wid;
#pragma unroll
      for (int m = 0; m < 9; ++m)
#pragma unroll
        for (int c = 0; c < 2; ++c) Y[c][m] = R(0.0);
#pragma unroll 3
      for (int rr = 0; rr < 18; ++rr) {
        const int off = nbo[c_n18.v[rr][0]][lane] + c_n18.v[rr][1] * plane;
        R v[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) v[c] = f[c * PS + off] - f0[c];
#pragma unroll
        for (int m = 0; m < 9; ++m) {
          const R a = __ldg(wc + (long long)(rr * 9 + m) * cstride);
#pragma unroll
          for (int c = 0; c < 2; ++c) Y[c][m] = Y[c][m] + a * v[c];
        }
      }
      const unsigned long long csrc = cmap ? cmap[p].src : LSQ_IDENTITY_SRC;
      const unsigned int cneg = cmap ? cmap[p].neg : 0u;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        R X[9];
#pragma unroll
        for (int m = 0; m < 9; ++m) X[m] = cmap ? lsq_rotated<1>(Y[c], m + 1, csrc, cneg) : Y[c][m];
        add(c, X, 100.0);
      }
    }
    const R fl = s.flatA[o], x = R(1.0) - fl;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double wn = 1.0 / sw[c];
#pragma unroll
      for (int m = 0; m < 9; ++m) s.V[((m + 1) * NVAR + 2 * w + c) * PS + o] = (R)(acc[c][m] * wn) * x;
    }
  }
}

// STEP 9.b of LIMIT_ALL_SLOPES_P2, a thread one zone and the three E components:
// the nine stencils' modes (eight one-sided from the resident inverses, the
// zone itself first; the central one STEP 9.c's 19-zone row weights), their
// smoothness indicators and weights as in k_p2_prim, then the weighted point
// values, summed stencil by stencil (the one-sided stencils' constants formed
// again rather than kept).  Each operator word is loaded once for the three
// components, from L2: a ring of the stencils' inverses, with a warp a
// component, measured 3.6 ms of a 6 x 64^2 x 32 step against 2.8, since its
// reads of shared memory serve one multiply-add each and its stages leave
// room for four blocks an SM.  Only the point value is stored, flattened toward
// the unlimited one (the edge solver consumes nothing else).  Panel order as
// in k_p2_prim.
template <bool kShared, typename R>
__global__ void __launch_bounds__(32) k_p2_efield(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  constexpr int NM = 10, NR = 10;
  constexpr Stencil18 N18 = stencil18();
  const int lane = threadIdx.x;
  const long long nz = r.count(), npp = nz / 6, nw = kShared ? npp : nz;
  const long long ntile = kShared ? 6 * ((npp + 31) / 32) : (nz + 31) / 32;
  const long long cstr = (long long)NPANEL * d.S;  // stride between variables
  for (long long T = blockIdx.x; T < ntile; T += gridDim.x) {
    long long t, tw;
    if (kShared) {
      tw = (T / 6) * 32 + lane;
      t = (T % 6) * npp + tw;
      if (tw >= npp) continue;
    } else {
      t = tw = T * 32 + lane;
      if (t >= nz) continue;
    }
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const Nbr12 n = load_nbr(g, d, p, i, j);
    // smoothness weight of each mode x .. xz over the unit cube
    double wis[9];
    {
      const double ob12 = 1.0 / 12.0, ob180 = 1.0 / 180.0, ob144 = 1.0 / 144.0;
      wis[0] = wis[1] = wis[2] = ob12;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const double cm = geo(g, d, CS_G_COEF, 4 + m, p, i, j, k), cc = geo(g, d, CS_G_COEF, 7 + m, p, i, j, k);
        wis[3 + m] = (cm - ob12) * (cm - ob12) + ob180;
        wis[6 + m] = cc * cc + ob144;
      }
    }
    auto smooth = [&](const R* X) {  // X: modes x .. xz
      return ((double)X[0] * X[0] + (double)X[1] * X[1] + (double)X[2] * X[2]) * wis[0] +
             ((double)X[3] * X[3]) * wis[3] + ((double)X[4] * X[4]) * wis[4] + ((double)X[5] * X[5]) * wis[5] +
             ((double)X[6] * X[6]) * wis[6] + ((double)X[7] * X[7]) * wis[7] + ((double)X[8] * X[8]) * wis[8];
    };
    const R* fb = s.Esnap + (long long)p * d.S;
    const long long o0 = d.idx(i, j, k);
    R f0[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) f0[c] = fb[c * cstr + o0];
    const unsigned long long qsrc = kShared ? s.p2_map[p].src : LSQ_IDENTITY_SRC;
    const unsigned int qneg = kShared ? s.p2_map[p].neg : 0u;
    const R* op = s.op_p2e + tw;
    // The modes of one-sided stencil st for the thread's variables, group
    // by group -- the groups the panel rotations permute within (for E the
    // constant first, then x y z, the squares, the cross terms) -- rotated
    // to this panel and handed to visit(group, X[variable][0..2]); groups
    // g0 .. g1 - 1 only.  Three modes a variable are live at a time.
    constexpr int NG = 4;
    auto stencil = [&](int st, int g0, int g1, auto&& visit) {
      R Rv[3][NR];
#pragma unroll
      for (int rr = 0; rr < NR; ++rr) {
        int zx = i, zy = j, zz = k;
        if (rr > 0) p2_zone(n, st, rr - 1, i, j, k, zx, zy, zz);
        const long long off = d.idx(zx, zy, zz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Rv[c][rr] = fb[c * cstr + off];
        }
      }
#pragma unroll
      for (int gi = 0; gi < NG; ++gi) {
        if (gi < g0 || gi >= g1) continue;
        const int mb = gi == 0 ? 0 : 3 * gi - 2;  // first mode of the group
        const int gs = gi == 0 ? 1 : 3;
        R Y[3][3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (q < gs) {
            R w[NR];
#pragma unroll
            for (int rr = 0; rr < NR; ++rr) w[rr] = __ldg(op + (long long)((st * NM + mb + q) * NR + rr) * nw);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              R acc = R(0.0);
#pragma unroll
              for (int rr = 0; rr < NR; ++rr) acc = acc + w[rr] * Rv[c][rr];
              Y[c][q] = acc;
            }
          }
        }
        R X[3][3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (q < gs) {
            const int mm = mb + q;
            const int mu = kShared ? (int)((qsrc >> (4 * mm)) & 15) - mb : q;
            const bool ng = kShared && ((qneg >> mm) & 1u);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const R v = mu == 0 ? Y[c][0] : (mu == 1 ? Y[c][1] : Y[c][2]);
              X[c][q] = ng ? -v : v;
            }
          }
        }
        visit(gi, X);
      }
    };
    double IS[3][9];
    R X8[3][NM];
    {  // central stencil from the resident row weights
      R Y[3][NM];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < NM; ++m) Y[c][m] = R(0.0);
      const LsqPanelMap* cmap = s.lsq_map10;
      const long long tc = cmap ? t - (long long)p * npp : t, ncw = cmap ? npp : nz;
      const WBlock cb = w_block<190>(tc / 32, ncw);
      const R* wc = s.op_m10 + cb.off + tc % 32;
#pragma unroll
      for (int rr = 0; rr < NR + 9; ++rr) {
        const int ro = rr - 1;  // the zone itself first
        const int w = ro < 0 ? 12 : N18.v[ro][0], dz = ro < 0 ? 0 : N18.v[ro][1];
        const long long off = d.idx(w == 12 ? i : n.x[w], w == 12 ? j : n.y[w], k + dz);
        R Rv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          Rv[c] = fb[c * cstr + off];
        }
#pragma unroll
        for (int m = 0; m < NM; ++m) {
          const R wv = __ldg(wc + (rr * NM + m) * cb.wid);
#pragma unroll
          for (int c = 0; c < 3; ++c) Y[c][m] = Y[c][m] + wv * Rv[c];
        }
      }
      const unsigned long long csrc = cmap ? cmap[p].src : LSQ_IDENTITY_SRC;
      const unsigned int cneg = cmap ? cmap[p].neg : 0u;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int m = 0; m < NM; ++m) X8[c][m] = cmap ? lsq_rotated<0>(Y[c], m, csrc, cneg) : Y[c][m];
        IS[c][8] = smooth(X8[c] + 1);
      }
    }
#pragma unroll 1
    for (int st = 0; st < 8; ++st) {
      double sm[3];
      stencil(st, 0, NG, [&](int gi, R (*X)[3]) {
        const int gg = gi - 1;  // 0: x y z, 1: the squares, 2: the cross terms
        if (gg < 0) return;     // the constant has no indicator term
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double a0 = X[c][0], a1 = X[c][1], a2 = X[c][2];
          if (gg == 0)
            sm[c] = (a0 * a0 + a1 * a1 + a2 * a2) * wis[0];
          else
            sm[c] = sm[c] + (a0 * a0) * wis[3 * gg] + (a1 * a1) * wis[3 * gg + 1] + (a2 * a2) * wis[3 * gg + 2];
        }
      });
#pragma unroll
      for (int c = 0; c < 3; ++c) IS[c][st] = sm[c];
    }
    double W[3][9];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
#pragma unroll
      for (int st = 0; st < 9; ++st) {
        const double tt = IS[c][st] + ph.smallnum, t2 = tt * tt;
        W[c][st] = (st < 8 ? 1.0 : 100.0) / (t2 * t2);
      }
      const double wn =
          1.0 / (W[c][0] + W[c][1] + W[c][2] + W[c][3] + W[c][4] + W[c][5] + W[c][6] + W[c][7] + W[c][8]);
#pragma unroll
      for (int st = 0; st < 9; ++st) W[c][st] = W[c][st] * wn;
    }
    double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int st = 0; st < 8; ++st) {
      stencil(st, 0, 1, [&](int, R (*X)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = acc[c] + W[c][st] * (double)X[c][0];
      });
    }
    const R fl = s.flatA[d.at(0, p, i, j, k)], x = R(1.0) - fl;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      acc[c] = acc[c] + W[c][8] * (double)X8[c][0];
      s.E[d.at(c, p, i, j, k)] = fl * f0[c] + x * (R)acc[c];
    }
  }
}

}  // namespace

// STEP 10 (421:9354-9976): min and max over the active interior zones of
// the 8 primitives (zone values, B from the ADP solve) and of the zone's
// net face flux of B normalised by the larger of the two sides' |B| and the
// magnetosonic scale msonic sqrt(4 3.14 rho) (the reference's constant).
// Min and max do not depend on order: each warp reduces with shuffles and
// lane 0 folds its 18 values into keys[] by atomicMin / atomicMax on
// order-preserving integer keys of the doubles.
__device__ __forceinline__ unsigned long long minmax_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}
__global__ void k_step10_reset(unsigned long long* keys) {
  if (threadIdx.x < 18) keys[threadIdx.x] = threadIdx.x < 9 ? ~0ULL : 0ULL;
}
template <typename R>
__global__ void k_step10(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r, unsigned long long* keys) {
  double mn[9], mx[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    mn[q] = 1.0e30;
    mx[q] = -1.0e30;
  }
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      v[q] = (double)Vat(s, d, q, 0, p, i, j, k);
      mn[q] = fmin(mn[q], v[q]);
      mx[q] = fmax(mx[q], v[q]);
    }
    const double bxp = s.Bxf[d.at(0, p, i, j, k)], bxm = s.Bxf[d.at(0, p, i - 1, j, k)];
    const double byp = s.Byf[d.at(0, p, i, j, k)], bym = s.Byf[d.at(0, p, i, j - 1, k)];
    const double bzp = s.Bzf[d.at(0, p, i, j, k)], bzm = s.Bzf[d.at(0, p, i, j, k - 1)];
    const double a21 = geo(g, d, CS_G_XF_AREA, 0, p, i, j, k) * bxp + geo(g, d, CS_G_YF_AREA, 0, p, i, j, k) * byp +
                       geo(g, d, CS_G_ZF_AREA, 0, p, i, j, k) * bzp - geo(g, d, CS_G_XF_AREA, 0, p, i - 1, j, k) * bxm -
                       geo(g, d, CS_G_YF_AREA, 0, p, i, j - 1, k) * bym - geo(g, d, CS_G_ZF_AREA, 0, p, i, j, k - 1) * bzm;
    const double a11 = v[5] * v[5] + v[6] * v[6] + v[7] * v[7];
    const double ms = sqrt((ph.gamma * v[4] + ph.ob4pi * a11) / v[0]);
    const double den = fmax(fmax(sqrt(bxp * bxp + byp * byp + bzp * bzp), sqrt(bxm * bxm + bym * bym + bzm * bzm)),
                            ms * sqrt(4.0 * 3.14 * v[0]));
    const double dv = a21 / den;
    mn[8] = fmin(mn[8], dv);
    mx[8] = fmax(mx[8], dv);
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn[q] = fmin(mn[q], __shfl_xor_sync(0xffffffffu, mn[q], o));
      mx[q] = fmax(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      atomicMin(keys + q, minmax_key(mn[q]));
      atomicMax(keys + 9 + q, minmax_key(mx[q]));
    }
  }
}

template <typename R>
void launch_step10_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  Range3 z = {1, d.N, 1, d.N, 1, d.nr};
  k_step10_reset<<<1, 32, 0, sv.stream>>>(sv.step10_keys);
  mark(sv, "k_step10_reset");
  k_step10<R><<<blocks_for(z.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, z, sv.step10_keys);
  mark(sv, "k_step10");
}

void launch_step10(Solve& sv) {
  if (!sv.step10_keys) return;
  if (sv.fp32)
    launch_step10_t(sv, sv.stF);
  else
    launch_step10_t(sv, sv.st);
}

inline Range3 faces_all(const Dims& d) { return {-d.G, d.N + d.G, -d.G, d.N + d.G, -d.G, d.nr + d.G}; }
template <typename R>
void launch_tricorner_t(Solve& sv, const DStateT<R>& st) {
  k_tricorner<R><<<blocks_for(6LL * 4 * sv.d.G * (sv.d.NK - 1), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.g, st);
  mark(sv, "k_tricorner");
}

template <typename R>
void launch_prim_and_masks_t(Solve& sv, DStateT<R>& st) {
  const Range3 f = faces_all(sv.d);
  k_prim<R><<<blocks_for(f.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.ph, sv.g, st, f,
                                                                                    adp_layers(sv.p));
  mark(sv, "k_prim");
  launch_tricorner_t(sv, st);
}

void launch_prim_and_masks(Solve& sv) {
  if (sv.fp32)
    launch_prim_and_masks_t(sv, sv.stF);
  else
    launch_prim_and_masks_t(sv, sv.st);
}

template <typename R>
void launch_face_masks_t(Solve& sv, DStateT<R>& st) {
  const Range3 f = faces_all(sv.d);
  k_zero_masked_faces<R><<<blocks_for(f.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.g, st, f);
  mark(sv, "k_zero_masked_faces");
  launch_tricorner_t(sv, st);
}

void launch_face_masks(Solve& sv) {
  if (sv.fp32)
    launch_face_masks_t(sv, sv.stF);
  else
    launch_face_masks_t(sv, sv.st);
}

template <typename R>
void launch_flattener_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  Range3 z = zones_all(d);
  const int nb = blocks_for(z.count(), TPB, grid_sms(sv));
  k_flat_a<R><<<nb, TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, z);
  mark(sv, "k_flat_a");
  k_flat_bc<R><<<nb, TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, z, st.flatA, st.flatB, 0);
  mark(sv, "k_flat_bc");
  k_flat_bc<R><<<nb, TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, z, st.flatB, st.flatA, 1);
  mark(sv, "k_flat_bc");
}

void launch_flattener(Solve& sv) {
  if (sv.fp32)
    launch_flattener_t(sv, sv.stF);
  else
    launch_flattener_t(sv, sv.st);
}

// 32-zone tiles of range b, panel-interleaved when the inverses are shared.
inline long long p2_tiles(const Range3& b, bool shared) {
  return shared ? 6 * ((b.count() / 6 + 31) / 32) : (b.count() + 31) / 32;
}

void set_p2_smem_limits() {
  cudaFuncSetAttribute(k_p2_prim<true, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P2Smem<double>));
  cudaFuncSetAttribute(k_p2_prim<false, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P2Smem<double>));
  cudaFuncSetAttribute(k_p2_prim<true, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P2Smem<float>));
  cudaFuncSetAttribute(k_p2_prim<false, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(P2Smem<float>));
}

template <typename R>
void launch_weno_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  Range3 a = shrink(d, 1), b = shrink(d, 2);
  if (sv.p.flags & CS_FLAG_P2) {  // LIMIT_ALL_SLOPES_P2's STEP 7.a
    const long long nt = (b.count() + W7A_ZT - 1) / W7A_ZT;
    const int nb = tile_blocks(sv, nt, 16);
    k_weno_slopes<W7_ENT, R><<<nb, W7A_ZT * 3, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
    mark(sv, "k_p2_entropy");
    const int np = (int)std::min<long long>(p2_tiles(b, st.p2_map), (long long)grid_sms(sv) * p2_blocks(sizeof(R)));
    if (st.p2_map)
      k_p2_prim<true, R><<<np, P2_THREADS, sizeof(P2Smem<R>), sv.stream>>>(d, sv.ph, sv.g, st, b);
    else
      k_p2_prim<false, R><<<np, P2_THREADS, sizeof(P2Smem<R>), sv.stream>>>(d, sv.ph, sv.g, st, b);
    mark(sv, "k_p2_prim");
    return;
  }
  {
    const long long nt = (a.count() + W7A_ZT - 1) / W7A_ZT;
    const int nb = tile_blocks(sv, nt, 16);
    k_weno_slopes<W7_PRIM, R><<<nb, W7A_ZT * 3, 0, sv.stream>>>(d, sv.ph, sv.g, st, a);
    mark(sv, "k_weno7a");
  }
  if (st.op_m9) {
    launch_weno7b(sv, b);
    return;
  }
  k_weno7b_rebuild<R><<<blocks_for(b.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
  mark(sv, "k_weno7b");
}

void launch_weno(Solve& sv) {
  if (sv.fp32)
    launch_weno_t(sv, sv.stF);
  else
    launch_weno_t(sv, sv.st);
}

template <typename R>
void launch_positivity_t(Solve& sv, DStateT<R>& st) {
  const Range3 z = shrink(sv.d, 1);
  // a thread takes 8 zones of a column where that leaves four blocks an SM
  // (fewer loads a zone), 2 otherwise (more threads)
  const long long per_k = z.count() / (z.k1 - z.k0 + 1);
  const int kc = z.count() >= (long long)grid_sms(sv) * 4 * TPB * 8 ? 8 : 2;
  const long long nt = per_k * ((z.k1 - z.k0 + kc) / kc);
  k_positivity<R><<<blocks_for(nt, TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.ph, sv.g, st, sv.mesh->pos_ext, z, kc);
  mark(sv, "k_positivity");
}

void launch_positivity(Solve& sv) {
  if (sv.fp32)
    launch_positivity_t(sv, sv.stF);
  else
    launch_positivity_t(sv, sv.st);
}

template <typename R>
void launch_faceB_adp_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  // the faces of the zones STEP 8.d solves
  Range3 fx = adp_zones(sv), fy = fx, fz = fx;
  fx.i0 -= 1;
  fy.j0 -= 1;
  fz.k0 -= 1;
  const long long nt = 3 * ((std::max(fx.count(), std::max(fy.count(), fz.count())) + TPB - 1) / TPB);
  k_faceB<R><<<tile_blocks(sv, nt, 64), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, fx, fy, fz);
  mark(sv, "k_faceB");
  launch_adp(sv);
}

void launch_faceB_adp(Solve& sv) {
  if (sv.fp32)
    launch_faceB_adp_t(sv, sv.stF);
  else
    launch_faceB_adp_t(sv, sv.st);
}

long long lsq_range_count(const Dims& d) { return shrink(d, 2).count(); }

void launch_pos_extents(Solve& sv, float* ext) {
  const Range3 z = shrink(sv.d, 1);
  k_pos_extents<<<blocks_for(z.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.ph, sv.g, z, ext);
  mark(sv, "k_pos_extents");
}

template <typename R>
void launch_ops_build_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  Range3 b = shrink(d, 2);
  if (st.op_m9) {
    k_ops_m9<R><<<blocks_for(b.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
    mark(sv, "k_ops_m9");
  }
  if (st.op_m10) {
    k_ops_m10<R><<<blocks_for(b.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
    mark(sv, "k_ops_m10");
  }
  if (st.op_p2v) {
    k_ops_p2<R><<<blocks_for(b.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
    mark(sv, "k_ops_p2");
  }
}

void launch_ops_build(Solve& sv) {
  if (sv.fp32)
    launch_ops_build_t(sv, sv.stF);
  else
    launch_ops_build_t(sv, sv.st);
}

template <typename R>
void launch_efield_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  Range3 a = around(d, 1), b = shrink(d, 2);
  // P2's stencils reach two zones beyond theirs; STEP 7.c's zones all zero
  // their entropy where they gave up
  const Range3 z = (sv.p.flags & CS_FLAG_P2) ? zones_all(d) : around(d, 2);
  const Range3 r = (sv.p.flags & CS_FLAG_P2) ? z : shrink(d, 1);
  k_efield_a<R><<<blocks_for(r.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.g, st, r, z);
  mark(sv, "k_efield_a");
  if (sv.p.flags & CS_FLAG_P2) {  // LIMIT_ALL_SLOPES_P2's STEP 9.b
    const int nb = (int)std::min<long long>(p2_tiles(b, st.p2_map), (long long)grid_sms(sv) * 16);
    if (st.p2_map)
      k_p2_efield<true, R><<<nb, 32, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
    else
      k_p2_efield<false, R><<<nb, 32, 0, sv.stream>>>(d, sv.ph, sv.g, st, b);
    mark(sv, "k_p2_efield");
    return;
  }
  {
    const long long nt = (a.count() + W7A_ZT - 1) / W7A_ZT;
    const int nb = tile_blocks(sv, nt, 16);
    k_weno_slopes<W7_E, R><<<nb, W7A_ZT * 3, 0, sv.stream>>>(d, sv.ph, sv.g, st, a);
    mark(sv, "k_efield_b");
  }
  if (st.op_m10) {
    launch_efield_c(sv, a, b);
    return;
  }
  k_efield_c_rebuild<R><<<blocks_for(a.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, a);
  mark(sv, "k_efield_c");
}

void launch_efield(Solve& sv) {
  if (sv.fp32)
    launch_efield_t(sv, sv.stF);
  else
    launch_efield_t(sv, sv.st);
}

}  // namespace cs
