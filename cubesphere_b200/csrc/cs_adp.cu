// STEP 8.d of the reconstruction: the ADP constrained least squares for the
// zones' B modes (421limit_all_slopes_p12.f:5574-6675,
// 253, 120matsolve.f), with the panel-shared inverse, the per-panel factors
// or factored in place.
#include <math_constants.h>

#include "cs_recon.cuh"

namespace cs {

namespace {

// STEP 8.d ADP (421:5617-6677): constrained least squares for the 30
// quadratic B modes matching the 6 face means exactly, solved per zone as
// the 36x36 KKT system by one warp with Gaussian elimination (scaled
// partial pivoting) in shared memory.
constexpr int ADP_WARPS = 4;
// Resident ADP factors are stored as one stream per block of ADP_ZB zones
// (zone fastest), in the order the substitution consumes them: the strict
// lower triangle row by row (630), then for rows 35..0 the entries right of
// the diagonal followed by the diagonal (666).
constexpr int ADP_ZB = 128;
__host__ __device__ constexpr int adp_stream_pos(int a, int b) {
  return b < a ? a * (a - 1) / 2 + b : 630 + (35 - a) * (36 - a) / 2 + (b == a ? 35 - a : b - a - 1);
}
// Operator of the panel-shared cache: blocks of ADP6_ZB zones with the rows
// of the inverse KKT matrix that the 30 modes need (see k_adp6), packed by
// symmetry into 645 words: with M the 30 x 30 mode block and N its 30 x 6
// columns of the face constraints, in groups a = 0..2 of 10 modes (one a
// component) and units of 15 words [5][3 groups],
//   unit f * 2 + u / 5           word u % 5:  N[10 a + u][f]
//   unit 12 + e / 5              word e % 5:  M[10 a + i][10 a + j], i <= j,
//                                             e = 10 i - i (i - 1) / 2 + j - i
//   unit 23 + (j / 5) * 10 + i   word j % 5:  M[10 a + i][10 ((a + 1) % 3) + j]
constexpr int ADP6_ZB = 32;
constexpr int ADP6_UNIT = 15;
constexpr int ADP6_WORDS = 43 * ADP6_UNIT;
__host__ __device__ constexpr int adp6_pos_n(int a, int u, int f) { return (f * 2 + u / 5) * ADP6_UNIT + (u % 5) * 3 + a; }
__host__ __device__ constexpr int adp6_tri(int i, int j) { return 10 * i - i * (i - 1) / 2 + j - i; }
__host__ __device__ constexpr int adp6_pos_d(int a, int i, int j) {
  return 12 * ADP6_UNIT + adp6_tri(i, j) / 5 * ADP6_UNIT + (adp6_tri(i, j) % 5) * 3 + a;
}
__host__ __device__ constexpr int adp6_pos_o(int a, int i, int j) {
  return (23 + (j / 5) * 10 + i) * ADP6_UNIT + (j % 5) * 3 + a;
}
static_assert(adp6_pos_n(2, 9, 5) == 12 * ADP6_UNIT - 1 && adp6_pos_d(2, 9, 9) == 23 * ADP6_UNIT - 1 &&
                  adp6_pos_o(2, 9, 9) == ADP6_WORDS - 1,
              "packed operator");
struct AdpSmem {
  double K[36][37];
  double Q[30][31];
  double bq[30], wt[30], C[6][30], D[6], rhs[36], sol[36], sc[36], vB[30];
  int piv[36];
};

// acc + err: the sum of products so far and what rounding left out of it, by
// Knuth's error-free sum and a product whose error is one fused multiply-add
// (roundings spelled out, so that none are contracted away).
__device__ __forceinline__ void add_product(double& acc, double& err, double a, double b) {
  const double p = __dmul_rn(a, b), e = __fma_rn(a, b, -p), s = __dadd_rn(acc, p), t = __dsub_rn(s, acc);
  err = __dadd_rn(err, __dadd_rn(__dadd_rn(__dsub_rn(acc, __dsub_rn(s, t)), __dsub_rn(p, t)), e));
  acc = s;
}

// kFactorOnly: assemble and factor the geometry-only KKT matrix and store
// the factors and the row permutation for k_adp_solve, or (zb == ADP6_ZB)
// the packed rows of the inverse for k_adp6 (once per mesh).
//
// The inverse's columns are refined once, with residuals carried to twice the
// precision, so that what is stored is the rounded inverse.  Without that its
// application errs up to 20 times as much as a substitution with the factors
// (thin surfaces of 12^2 x 3 zones: 7e-11 of the largest mode against 3e-12);
// with it less than half as much on every mesh, in FP32 too, where the
// substitution itself rounded at every element (12^2 x 3: 1.3e-3 for the
// factors in FP32, 8.6e-4 for the inverse).
// tmax: zones of the range handled (all of it, or panel 1's share when the
// factors are shared by the six panels); zb: zones per factor block.
template <bool kFactorOnly, typename R>
__global__ void __launch_bounds__(32 * ADP_WARPS) k_adp(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r,
                                                        long long tmax, int zb) {
  extern __shared__ unsigned char smem_raw[];
  AdpSmem& S = reinterpret_cast<AdpSmem*>(smem_raw)[threadIdx.x / 32];
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * ADP_WARPS;
  for (long long t = blockIdx.x * (long long)ADP_WARPS + threadIdx.x / 32; t < tmax; t += nw) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) == 0) continue;
    const double obl0 = 1.0 / fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum);
    const double vc0 = geo(g, d, CS_G_V_CEN, 0, p, i, j, k), vc1 = geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 vc2 = geo(g, d, CS_G_V_CEN, 2, p, i, j, k);
    double c0[10];
    coef10(g, d, p, i, j, k, c0);
    // 1. the 30 quadrature rows, one per lane
    if (lane < 30) {
      const int f = lane / 5, q = lane % 5, dir = f / 2;
      const int fx = (f == 1) ? i - 1 : i, fy = (f == 3) ? j - 1 : j, fz = (f == 5) ? k - 1 : k;
      const int QP = dir == 0 ? CS_G_XF_QP : (dir == 1 ? CS_G_YF_QP : CS_G_ZF_QP);
      const int BW = dir == 0 ? CS_G_XB_QW : (dir == 1 ? CS_G_YB_QW : CS_G_ZB_QW);
      const int NF = dir == 0 ? CS_G_XF_N : (dir == 1 ? CS_G_YF_N : CS_G_ZF_N);
      const int nq = dir == 2 ? q : 0, ns = dir == 2 ? 5 : 1;
      const double nx = geo(g, d, NF, nq, p, fx, fy, fz), ny = geo(g, d, NF, ns + nq, p, fx, fy, fz),
                   nz = geo(g, d, NF, 2 * ns + nq, p, fx, fy, fz);
      const double x = (geo(g, d, QP, q, p, fx, fy, fz) - vc0) * obl0;
      const double y = (geo(g, d, QP, 5 + q, p, fx, fy, fz) - vc1) * obl0;
      const double z = (geo(g, d, QP, 10 + q, p, fx, fy, fz) - vc2) * obl0;
      const double bfn[10] = {1.0, x, y, z, x * x - c0[4], y * y - c0[5], z * z - c0[6], x * y - c0[7], y * z - c0[8], x * z - c0[9]};
#pragma unroll
      for (int m = 0; m < 10; ++m) {
        S.Q[lane][m] = m == 0 ? nx : nx * bfn[m];
        S.Q[lane][10 + m] = m == 0 ? ny : ny * bfn[m];
        S.Q[lane][20 + m] = m == 0 ? nz : nz * bfn[m];
      }
      S.wt[lane] = geo(g, d, BW, q, p, fx, fy, fz);
      if (!kFactorOnly) {
        S.bq[lane] = s.Bq[dir][d.at(q, p, fx, fy, fz)];
        S.vB[lane] = Vat(s, d, 5 + lane / 10, lane % 10, p, i, j, k);
      } else {
        S.bq[lane] = 0.0;
        S.vB[lane] = 0.0;
      }
    }
    __syncwarp();
    // 2. constraint rows C, D and the KKT matrix
    for (int e = lane; e < 180; e += 32) {
      const int f = e / 30, m = e % 30;
      double acc = 0.0;
#pragma unroll
      for (int q = 0; q < 5; ++q) acc = acc + S.wt[f * 5 + q] * S.Q[f * 5 + q][m];
      S.C[f][m] = acc;
    }
    if (lane < 6) {
      double acc = 0.0;
#pragma unroll
      for (int q = 0; q < 5; ++q) acc = acc + S.wt[lane * 5 + q] * S.bq[lane * 5 + q];
      S.D[lane] = acc;
    }
    __syncwarp();
    // divergence-free rows (421:6586-6600) as (column, value) pairs
    const int dcol[4][3] = {{1, 12, 23}, {4, 17, 29}, {7, 15, 28}, {9, 18, 26}};
    const double dval[4][3] = {{1.0, 1.0, 1.0}, {2.0, 1.0, 1.0}, {1.0, 2.0, 1.0}, {1.0, 1.0, 2.0}};
    for (int e = lane; e < 900; e += 32) {
      const int a = e / 30, b = e % 30;
      double acc = 0.0;
      for (int q = 0; q < 30; ++q) acc = acc + S.Q[q][a] * S.Q[q][b];
      if (a == b) acc = acc + 1.0;
      for (int rr = 0; rr < 4; ++rr) {
        double va = 0.0, vb = 0.0;
        for (int c = 0; c < 3; ++c) {
          if (dcol[rr][c] == a) va = dval[rr][c];
          if (dcol[rr][c] == b) vb = dval[rr][c];
        }
        acc = acc + va * vb;
      }
      S.K[a][b] = acc;
    }
    for (int e = lane; e < 180; e += 32) {
      const int f = e / 30, m = e % 30;
      S.K[m][30 + f] = S.C[f][m];
      S.K[30 + f][m] = S.C[f][m];
    }
    if (kFactorOnly && zb == ADP6_ZB) {  // the mode block for the residuals, in place of the rows
      __syncwarp();
      for (int e = lane; e < 900; e += 32) S.Q[e / 30][e % 30] = S.K[e / 30][e % 30];
    }
    for (int e = lane; e < 36; e += 32) {
      S.K[30 + e / 6][30 + e % 6] = 0.0;
    }
    if (lane < 30) {
      double acc = 0.0;
      for (int q = 0; q < 30; ++q) acc = acc + S.Q[q][lane] * S.bq[q];
      S.rhs[lane] = acc + S.vB[lane];
    } else {
      for (int f = lane - 30; f < 6; f += 2) S.rhs[30 + f] = S.D[f];
    }
    __syncwarp();
    // 3. elimination with scaled partial pivoting
    double kmax = 0.0;  // largest entry this lane has seen
    for (int row = lane; row < 36; row += 32) {
      double m = 0.0;
      for (int c = 0; c < 36; ++c) m = fmax(m, fabs(S.K[row][c]));
      kmax = fmax(kmax, m);
      S.sc[row] = (m == 0.0) ? 0.0 : 1.0 / m;
      S.piv[row] = row;
    }
    __syncwarp();
    for (int kk = 0; kk < 36; ++kk) {
      double best = -1.0;
      int bi = kk;
      for (int row = kk + lane; row < 36; row += 32) {
        const double v = fabs(S.K[row][kk]) * S.sc[row];
        if (v > best) {
          best = v;
          bi = row;
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ob > best || (ob == best && oi < bi)) {
          best = ob;
          bi = oi;
        }
      }
      if (bi != kk) {
        for (int c = lane; c < 36; c += 32) {
          const double tmp = S.K[kk][c];
          S.K[kk][c] = S.K[bi][c];
          S.K[bi][c] = tmp;
        }
        if (lane == 0) {
          const double ts = S.sc[kk];
          S.sc[kk] = S.sc[bi];
          S.sc[bi] = ts;
          const int tp = S.piv[kk];
          S.piv[kk] = S.piv[bi];
          S.piv[bi] = tp;
        }
      }
      __syncwarp();
      if (lane == 0 && S.K[kk][kk] == 0.0) S.K[kk][kk] = 1.0e-20;
      __syncwarp();
      const double inv = 1.0 / S.K[kk][kk];
      for (int row = kk + 1 + lane; row < 36; row += 32) {
        const double l = S.K[row][kk] * inv;
        S.K[row][kk] = l;
        for (int c = kk + 1; c < 36; ++c) S.K[row][c] -= l * S.K[kk][c];
      }
      __syncwarp();
    }
    if (kFactorOnly && zb == ADP6_ZB) {
      // lane c: column c of the inverse, by symmetry row c
      double y[36];
#pragma unroll
      for (int a = 0; a < 36; ++a) {
        double acc = S.piv[a] == lane ? 1.0 : 0.0;
#pragma unroll
        for (int b = 0; b < a; ++b) acc -= S.K[a][b] * y[b];
        y[a] = acc;
      }
#pragma unroll
      for (int a = 35; a >= 0; --a) {
        double acc = y[a];
#pragma unroll
        for (int b = a + 1; b < 36; ++b) acc -= S.K[a][b] * y[b];
        y[a] = acc / S.K[a][a];
      }
      // y += K^-1 (e_c - K y); z is in local memory, so that the loops stay loops
      double z[36];
#pragma unroll 1
      for (int a = 0; a < 36; ++a) {
        const int row = S.piv[a];
        double acc = row == lane ? 1.0 : 0.0, err = 0.0;
        if (row < 30) {
          const double* k = S.Q[row];
#pragma unroll
          for (int b = 0; b < 30; ++b) add_product(acc, err, -k[b], y[b]);
#pragma unroll
          for (int f = 0; f < 6; ++f) add_product(acc, err, -S.C[f][row], y[30 + f]);
        } else {
          const double* k = S.C[row - 30];
#pragma unroll
          for (int b = 0; b < 30; ++b) add_product(acc, err, -k[b], y[b]);
        }
        acc = acc + err;
#pragma unroll 1
        for (int b = 0; b < a; ++b) acc -= S.K[a][b] * z[b];
        z[a] = acc;
      }
#pragma unroll 1
      for (int a = 35; a >= 0; --a) {
        double acc = z[a];
#pragma unroll 1
        for (int b = a + 1; b < 36; ++b) acc -= S.K[a][b] * z[b];
        z[a] = acc / S.K[a][a];
      }
#pragma unroll
      for (int a = 0; a < 36; ++a) y[a] = y[a] + z[a];
      // the size of K times that of its inverse, for the mesh build's choice
      // (infinite where an entry is not finite)
      double ymax = 0.0;
      if (lane < 30)
#pragma unroll
        for (int u = 0; u < 30; ++u) ymax = isfinite(y[u]) ? fmax(ymax, fabs(y[u])) : CUDART_INF;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        kmax = fmax(kmax, __shfl_xor_sync(0xffffffffu, kmax, off));
        ymax = fmax(ymax, __shfl_xor_sync(0xffffffffu, ymax, off));
      }
      if (lane == 0)
        atomicMax(reinterpret_cast<unsigned long long*>(s.err_flag) + 1, (unsigned long long)__double_as_longlong(kmax * ymax));
      if (lane < 30) {
        R* out = (R*)s.adp_lu + t / ADP6_ZB * (long long)(ADP6_WORDS * ADP6_ZB) + t % ADP6_ZB;
        const int g = lane / 10, j = lane % 10;
#pragma unroll
        for (int f = 0; f < 6; ++f) out[adp6_pos_n(g, j, f) * ADP6_ZB] = (R)y[30 + f];
#pragma unroll
        for (int u = 0; u < 30; ++u) {
          const int a = u / 10, i = u % 10;
          if (a == g && i <= j) out[adp6_pos_d(a, i, j) * ADP6_ZB] = (R)y[u];
          if ((a + 1) % 3 == g) out[adp6_pos_o(a, i, j) * ADP6_ZB] = (R)y[u];
        }
      }
      __syncwarp();
      continue;
    }
    if (kFactorOnly) {
      const long long blk = t / zb, z = t % zb;
      for (int e = lane; e < 36 * 36; e += 32)
        ((double*)s.adp_lu)[(blk * 1296 + adp_stream_pos(e / 36, e % 36)) * zb + z] = S.K[e / 36][e % 36];
      for (int e = lane; e < 36; e += 32) s.adp_piv[(blk * 36 + e) * zb + z] = (int8_t)S.piv[e];
      __syncwarp();
      continue;
    }
    // 4. substitution (one lane, reference order)
    if (lane == 0) {
      double y[36];
      for (int a = 0; a < 36; ++a) {
        double acc = S.rhs[S.piv[a]];
        for (int b = 0; b < a; ++b) acc -= S.K[a][b] * y[b];
        y[a] = acc;
      }
      for (int a = 35; a >= 0; --a) {
        double acc = y[a];
        for (int b = a + 1; b < 36; ++b) acc -= S.K[a][b] * S.sol[b];
        S.sol[a] = acc / S.K[a][a];
      }
    }
    __syncwarp();
    // 5. write back the modes, zone B and the energy adjustment
    if (lane < 30) Vat(s, d, 5 + lane / 10, lane % 10, p, i, j, k) = S.sol[lane];
    if (lane == 0) {
      R* U = s.U;
      const long long o5 = d.at(4, p, i, j, k);
      const double u6 = U[d.at(5, p, i, j, k)], u7 = U[d.at(6, p, i, j, k)], u8 = U[d.at(7, p, i, j, k)];
      const double aa = (u6 * u6 + u7 * u7 + u8 * u8) * ph.ob8pi;
      const double n6 = S.sol[0], n7 = S.sol[10], n8 = S.sol[20];
      U[d.at(5, p, i, j, k)] = n6;
      U[d.at(6, p, i, j, k)] = n7;
      U[d.at(7, p, i, j, k)] = n8;
      const double bb = (n6 * n6 + n7 * n7 + n8 * n8) * ph.ob8pi;
      U[o5] = U[o5] - aa + bb;
    }
    __syncwarp();
  }
}

// STEP 8.d right-hand side with the resident factors: one thread per zone
// forms the 36 entries (the same sums in the same order as k_adp) and
// stores them element-major, [36][zones of the ADP range].
constexpr int ADPR_TPB = 128;
template <typename R>
__global__ void __launch_bounds__(ADPR_TPB) k_adp_rhs(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  const long long n = r.count();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    double* out = (double*)s.adp_rhs + t;
    if (mask_at(g, d, p, i, j) != 1) {
#pragma unroll
      for (int a = 0; a < 36; ++a) out[(long long)a * n] = 0.0;
      continue;
    }
    const double obl0 = 1.0 / fmax(geo(g, d, CS_G_V_SCALE, 0, p, i, j, k), ph.smallnum);
    const double vc0 = geo(g, d, CS_G_V_CEN, 0, p, i, j, k), vc1 = geo(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 vc2 = geo(g, d, CS_G_V_CEN, 2, p, i, j, k);
    double c0[10];
    coef10(g, d, p, i, j, k, c0);
    double rhs[30];
#pragma unroll
    for (int a = 0; a < 30; ++a) rhs[a] = 0.0;
#pragma unroll 1
    for (int f = 0; f < 6; ++f) {
      const int dir = f / 2;
      const int fx = (f == 1) ? i - 1 : i, fy = (f == 3) ? j - 1 : j, fz = (f == 5) ? k - 1 : k;
      const int QP = dir == 0 ? CS_G_XF_QP : (dir == 1 ? CS_G_YF_QP : CS_G_ZF_QP);
      const int BW = dir == 0 ? CS_G_XB_QW : (dir == 1 ? CS_G_YB_QW : CS_G_ZB_QW);
      const int NF = dir == 0 ? CS_G_XF_N : (dir == 1 ? CS_G_YF_N : CS_G_ZF_N);
      const int ns = dir == 2 ? 5 : 1;
      double dacc = 0.0;
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        const int nq = dir == 2 ? q : 0;
        const double nx = geo(g, d, NF, nq, p, fx, fy, fz), ny = geo(g, d, NF, ns + nq, p, fx, fy, fz),
                     nz = geo(g, d, NF, 2 * ns + nq, p, fx, fy, fz);
        const double x = (geo(g, d, QP, q, p, fx, fy, fz) - vc0) * obl0;
        const double y = (geo(g, d, QP, 5 + q, p, fx, fy, fz) - vc1) * obl0;
        const double z = (geo(g, d, QP, 10 + q, p, fx, fy, fz) - vc2) * obl0;
        const double bfn[10] = {1.0, x, y, z, x * x - c0[4], y * y - c0[5], z * z - c0[6], x * y - c0[7],
                                y * z - c0[8], x * z - c0[9]};
        const double bq = s.Bq[dir][d.at(q, p, fx, fy, fz)];
#pragma unroll
        for (int m = 0; m < 10; ++m) {
          rhs[m] = rhs[m] + (m == 0 ? nx : nx * bfn[m]) * bq;
          rhs[10 + m] = rhs[10 + m] + (m == 0 ? ny : ny * bfn[m]) * bq;
          rhs[20 + m] = rhs[20 + m] + (m == 0 ? nz : nz * bfn[m]) * bq;
        }
        dacc = dacc + geo(g, d, BW, q, p, fx, fy, fz) * bq;
      }
      out[(long long)(30 + f) * n] = dacc;
    }
#pragma unroll
    for (int a = 0; a < 30; ++a) out[(long long)a * n] = rhs[a] + Vat(s, d, 5 + a / 10, a % 10, p, i, j, k);
  }
}

// STEP 8.d substitution with the resident factors, one thread per zone.
// The factor stream of the block's 128 zones (1296 x 1 KB, in consumption
// order) flows through a ring of ADPS_NS shared-memory stages of ADPS_CH
// elements (16 KB), filled by bulk asynchronous copies that a producer warp
// issues as soon as the four consumer warps have released a stage
// (full / empty mbarrier pairs).  The solution vector lives in shared
// memory so that the loops stay short; the arithmetic (order included) is
// that of the reference's forward and back substitution.
constexpr int ADPS_TPB = ADP_ZB;             // consumer threads (one per zone)
constexpr int ADPS_THREADS = ADPS_TPB + 32;  // + one producer warp
constexpr int ADPS_CH = 16;
constexpr int ADPS_NS = 4;
constexpr int ADPS_NCH = 1296 / ADPS_CH;
static_assert(1296 % ADPS_CH == 0, "whole chunks");
struct AdpsSmem {
  double stage[ADPS_NS][ADPS_CH][ADPS_TPB];
  double y[36][ADPS_TPB];
  uint64_t full[ADPS_NS];
  uint64_t empty[ADPS_NS];
};

template <typename R>
__global__ void __launch_bounds__(ADPS_THREADS, 2) k_adp_solve(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  extern __shared__ __align__(128) unsigned char adps_raw[];
  AdpsSmem& S = *reinterpret_cast<AdpsSmem*>(adps_raw);
  const int tid = threadIdx.x;
  const long long n = r.count();
  const long long nblk = (n + ADP_ZB - 1) / ADP_ZB;
  if ((long long)blockIdx.x >= nblk) return;
  const long long my_iters = (nblk - 1 - blockIdx.x) / gridDim.x + 1;
  const long long total_chunks = my_iters * ADPS_NCH;
  if (tid == 0) {
    for (int q = 0; q < ADPS_NS; ++q) {
      mbar_init(&S.full[q], 1);
      mbar_init(&S.empty[q], ADPS_TPB / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid >= ADPS_TPB) {
    // producer: chunk gch of this CTA is chunk gch % NCH of zone block
    // blockIdx.x + (gch / NCH) * gridDim.x
    if (tid == ADPS_TPB) {
      for (long long gch = 0; gch < total_chunks; ++gch) {
        const int slot = (int)(gch % ADPS_NS);
        if (gch >= ADPS_NS) mbar_wait(&S.empty[slot], (uint32_t)(((gch / ADPS_NS) - 1) & 1), s.err_flag);
        const long long it = gch / ADPS_NCH, c = gch % ADPS_NCH;
        const long long blk = blockIdx.x + it * gridDim.x;
        const double* src = (const double*)s.adp_lu + (blk * 1296 + c * ADPS_CH) * (long long)ADP_ZB;
        mbar_expect_tx(&S.full[slot], ADPS_CH * ADP_ZB * sizeof(double));
        bulk_g2s(&S.stage[slot][0][0], src, ADPS_CH * ADP_ZB * sizeof(double), &S.full[slot]);
      }
    }
    return;
  }
  const int lane = tid & 31;
  long long gch = 0;  // next chunk to consume
  int within = ADPS_CH;
  const double* cur = nullptr;
  // next factor element of this thread's zone
  auto next = [&]() -> double {
    if (within == ADPS_CH) {
      if (gch > 0) ring_release(&S.empty[(int)((gch - 1) % ADPS_NS)], lane);
      const int slot = (int)(gch % ADPS_NS);
      mbar_wait(&S.full[slot], (uint32_t)((gch / ADPS_NS) & 1), s.err_flag);
      cur = &S.stage[slot][0][tid];
      ++gch;
      within = 0;
    }
    return cur[(within++) * ADPS_TPB];
  };
  for (long long it = 0; it < my_iters; ++it) {
    const long long blk = blockIdx.x + it * gridDim.x;
    const long long t = blk * ADP_ZB + tid;
    const bool inr = t < n;
    const int8_t* pv = s.adp_piv + blk * 36 * ADP_ZB + tid;
    // permuted right-hand side first (36 independent loads), then the
    // substitution in place
#pragma unroll
    for (int a = 0; a < 36; ++a) S.y[a][tid] = inr ? ((const double*)s.adp_rhs)[(long long)pv[a * ADP_ZB] * n + t] : 0.0;
#pragma unroll 1
    for (int a = 1; a < 36; ++a) {
      double acc = S.y[a][tid];
#pragma unroll 4
      for (int b = 0; b < a; ++b) acc -= next() * S.y[b][tid];
      S.y[a][tid] = acc;
    }
#pragma unroll 1
    for (int a = 35; a >= 0; --a) {
      double acc = S.y[a][tid];
#pragma unroll 4
      for (int b = a + 1; b < 36; ++b) acc -= next() * S.y[b][tid];
      S.y[a][tid] = acc / next();
    }
    if (inr) {
      int p, i, j, k;
      r.decode(t, p, i, j, k);
      if (mask_at(g, d, p, i, j) == 1) {
#pragma unroll
        for (int a = 0; a < 30; ++a) Vat(s, d, 5 + a / 10, a % 10, p, i, j, k) = S.y[a][tid];
        R* U = s.U;
        const long long o5 = d.at(4, p, i, j, k);
        const double u6 = U[d.at(5, p, i, j, k)], u7 = U[d.at(6, p, i, j, k)], u8 = U[d.at(7, p, i, j, k)];
        const double aa = (u6 * u6 + u7 * u7 + u8 * u8) * ph.ob8pi;
        const double n6 = S.y[0][tid], n7 = S.y[10][tid], n8 = S.y[20][tid];
        U[d.at(5, p, i, j, k)] = n6;
        U[d.at(6, p, i, j, k)] = n7;
        U[d.at(7, p, i, j, k)] = n8;
        const double bb = (n6 * n6 + n7 * n7 + n8 * n8) * ph.ob8pi;
        U[o5] = U[o5] - aa + bb;
      }
    }
  }
}

}  // namespace

// STEP 8.d with an operator shared by the six panels.  The panels of the
// cubed sphere are rotations of panel 1 by signed permutations R_p
// (vertex(p, i,j,k) = R_p vertex(1, i,j,k), checked when the mesh is
// uploaded), so the KKT matrix of zone (i,j,k) of panel p is T_p K_1 T_p^T,
// T_p being the signed permutation of the 30 B-mode unknowns that R_p
// induces (identity on the 6 multipliers): r' = T_p^T r, y' = K_1^-1 r',
// y = T_p y', with panel 1's geometry and inverse serving all six panels.
// adp_pmap[p][0][v] is the panel-p unknown u fed by panel-1 unknown v,
// adp_pmap[p][1][v] its sign.
//
// A CTA takes ADP6_ZB zone positions and the six panels; a warp the rows of
// component w % 3 for three of them (10 modes x 3 panels of sums in
// registers).  First the 36 right-hand sides (panel 1's quadrature rows times
// the panels' face values, plus their present modes) go to shared memory;
// then the warp applies the inverse's rows to them, while a producer warp
// streams the packed inverse through a ring of bulk copies that runs ahead
// across both phases.
//
// What bounds it: the 645-word stream (5.2 KB a position in FP64) and the
// modes, about 1.8 KB a zone of HBM traffic.  Each streamed word is read from
// shared memory by six warps for 3 (6 off the diagonal) multiply-adds, where
// a triangular solve reads 1296 words for one dependent one each.  The sums (60
// registers a thread) leave two blocks an SM in FP64 and four in FP32, so what
// is left is latency.  ms of a 6 x 128^2 x 64 step: 18.6 (FP32 15.0) for right-hand
// sides in HBM and a substitution, 10.2 (8.7) for this on two layers around the
// interior, 10.6 (9.0) on all radial layers that have faces.
constexpr int ADP6_CONS = 6 * 32;
constexpr int ADP6_THREADS = ADP6_CONS + 32;
constexpr int ADP6_CH = 2 * ADP6_UNIT;  // words a ring stage
constexpr int ADP6_NS = 4;
constexpr int ADP6_FB = 4;           // faces held by the copies ahead
constexpr int ADP6_FROWS = 15 + 30;  // rows of a face
constexpr int ADP6_NCH = (ADP6_WORDS + ADP6_CH - 1) / ADP6_CH;  // the last one holds one unit
template <typename F>
struct Adp6SmemT {
  F stage[ADP6_NS][ADP6_CH][ADP6_ZB];
  F x[36][6][ADP6_ZB];  // right-hand sides in panel 1's unknowns
  F bas[2][5][9][ADP6_ZB];  // monomials of a face's points, alternating over the faces
  // the panels' new zone B [panel][component]: in the second half of bas, which
  // the next block's faces reach after a barrier
  __device__ __forceinline__ F* nb(int p, int c) { return &bas[1][0][0][0] + (p * 3 + c) * ADP6_ZB; }
  // copies ahead: a face's points (rows 0-14) and its B at them (row 15 + 5
  // panel + point), in the rows of x that hold right-hand sides later
  __device__ __forceinline__ double (*face(int f))[ADP6_ZB] {
    static_assert(sizeof(F) == 4 || ADP6_FB * ADP6_FROWS * sizeof(double) <= 30 * 6 * sizeof(F), "face rows in x");
    return reinterpret_cast<double(*)[ADP6_ZB]>(&x[0][0][0]) + f % ADP6_FB * ADP6_FROWS;
  }
  F geo[sizeof(F) == 8 ? 10 : 1][ADP6_ZB];  // copies ahead: the position's centroid, 1 / scale and moments
  uint64_t full[ADP6_NS];
  uint64_t empty[ADP6_NS];
};

// Row and column of entry e of a packed 10 x 10 triangle (adp6_tri).
struct AdpElem {
  int i, j;
};
__host__ __device__ constexpr AdpElem adp6_elem(int e) {
  int i = 0;
  while (e >= 10 - i) {
    e -= 10 - i;
    ++i;
  }
  return AdpElem{i, i + e};
}
static_assert(adp6_elem(0).j == 0 && adp6_elem(9).j == 9 && adp6_elem(10).i == 1 && adp6_elem(10).j == 1 &&
                  adp6_elem(54).i == 9 && adp6_elem(54).j == 9,
              "triangle");

// Entry E of a diagonal block, on both its sides (the indices are
// compile-time constants, so the sums stay in registers).
template <int E, typename F>
__device__ __forceinline__ void adp6_diag(F (&acc)[3][10], const F (&xr)[3][10], F m) {
  constexpr AdpElem e = adp6_elem(E);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    acc[q][e.i] += m * xr[q][e.j];
    if constexpr (e.i != e.j) acc[q][e.j] += m * xr[q][e.i];
  }
}

// One unit of the stream applied to the sums acc[panel][mode] of group a
// (w: the group's five words, wp: the group before's, x / xn / xp: the
// right-hand sides of the three panels for its own group, the next and the
// one before, [mode][panel] with stride XS).
template <int U, typename F>
__device__ __forceinline__ void adp6_unit(F (&acc)[3][10], F (&xr)[3][10], const F* w, const F* wp, const F* xm,
                                          const F* x, const F* xn, const F* xp) {
  constexpr int XM = 6 * ADP6_ZB, XP = ADP6_ZB, WS = 3 * ADP6_ZB;  // strides: mode, panel, word
  if constexpr (U < 12) {
    constexpr int f = U / 2, h = U % 2;
    F c[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) c[q] = xm[f * XM + q * XP];
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      const F m = w[t * WS];
#pragma unroll
      for (int q = 0; q < 3; ++q) acc[q][5 * h + t] += m * c[q];
    }
  } else if constexpr (U < 23) {
    if constexpr (U == 12) {
#pragma unroll
      for (int i = 0; i < 10; ++i)
#pragma unroll
        for (int q = 0; q < 3; ++q) xr[q][i] = x[i * XM + q * XP];
    }
    adp6_diag<(U - 12) * 5>(acc, xr, w[0]);
    adp6_diag<(U - 12) * 5 + 1>(acc, xr, w[WS]);
    adp6_diag<(U - 12) * 5 + 2>(acc, xr, w[2 * WS]);
    adp6_diag<(U - 12) * 5 + 3>(acc, xr, w[3 * WS]);
    adp6_diag<(U - 12) * 5 + 4>(acc, xr, w[4 * WS]);
  } else {
    constexpr int i = (U - 23) % 10, h = (U - 23) / 10;
    if constexpr (i == 0) {
#pragma unroll
      for (int t = 0; t < 5; ++t)
#pragma unroll
        for (int q = 0; q < 3; ++q) xr[q][t] = xn[(5 * h + t) * XM + q * XP];
    }
    F c[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) c[q] = xp[i * XM + q * XP];
#pragma unroll
    for (int t = 0; t < 5; ++t) {
      const F m = w[t * WS], mp = wp[t * WS];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        acc[q][i] += m * xr[q][t];
        acc[q][5 * h + t] += mp * c[q];
      }
    }
  }
}

// The whole stream of one zone block: wait for a stage, apply its two units,
// release it.
template <typename F, int... C>
__device__ __forceinline__ void adp6_apply(F (&acc)[3][10], Adp6SmemT<F>& S, RingPos<ADP6_NS>& ring, int lane, int a, int h,
                                           int* err, std::integer_sequence<int, C...>) {
  const F* xm = &S.x[30][3 * h][lane];
  const F* x = &S.x[10 * a][3 * h][lane];
  const F* xn = &S.x[10 * (a == 2 ? 0 : a + 1)][3 * h][lane];
  const F* xp = &S.x[10 * (a == 0 ? 2 : a - 1)][3 * h][lane];
  const int ap = a == 0 ? 2 : a - 1;
  F xr[3][10];
  auto chunk = [&](auto Cc) {
    constexpr int c = decltype(Cc)::value;
    if (!mbar_try_wait(&S.full[ring.slot], ring.par)) mbar_wait(&S.full[ring.slot], ring.par, err);
    const F* w = &S.stage[ring.slot][a][lane];
    const F* wp = &S.stage[ring.slot][ap][lane];
    adp6_unit<2 * c>(acc, xr, w, wp, xm, x, xn, xp);
    if constexpr (2 * c + 1 < ADP6_WORDS / ADP6_UNIT)
      adp6_unit<2 * c + 1>(acc, xr, w + ADP6_UNIT * ADP6_ZB, wp + ADP6_UNIT * ADP6_ZB, xm, x, xn, xp);
    ring_release(&S.empty[ring.slot], lane);
    ring.next();
  };
  (chunk(std::integral_constant<int, C>{}), ...);
}

__device__ __forceinline__ void adp6_sync() { consumer_sync<ADP6_CONS>(); }

// Copy of one word a lane to shared memory, in the background.
__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Box offset of face f of position zo.
__device__ __forceinline__ unsigned adp6_face(const Dims& d, int f, unsigned zo) {
  const int dir = f >> 1;
  return zo - ((f & 1) ? (dir == 0 ? 1 : (dir == 1 ? d.NI : d.NI * d.NJ)) : 0);
}

// Start the copies of face f: warp w the point w (the rows it reads itself
// before the barrier) and panel w.  A group of copies a face.
template <typename R>
__device__ __forceinline__ void adp6_fetch(Adp6SmemT<R>& S, const Dims& d, const DGeom& g, const DStateT<R>& s, int f, unsigned zo,
                                           int lane, int w) {
  const long long PS = (long long)NPANEL * d.S;
  const int dir = f >> 1;
  const unsigned fo = adp6_face(d, f, zo);
  double(*fr)[ADP6_ZB] = S.face(f);
  if (w < 5) {
    const double* qp = (dir == 0 ? g.f[CS_G_XF_QP] : (dir == 1 ? g.f[CS_G_YF_QP] : g.f[CS_G_ZF_QP])) + fo + w * PS;
#pragma unroll
    for (int c = 0; c < 3; ++c) copy8(&fr[5 * c + w][lane], qp + 5 * c * PS);
  }
  const double* Bq = (dir == 0 ? s.Bq[0] : (dir == 1 ? s.Bq[1] : s.Bq[2])) + w * d.S + fo;
#pragma unroll
  for (int c = 0; c < 5; ++c) copy8(&fr[15 + 5 * w + c][lane], Bq + c * PS);
}
template <typename R>
__device__ __forceinline__ void adp6_fetch_first(Adp6SmemT<R>& S, const Dims& d, const DGeom& g, const DStateT<R>& s, unsigned zo,
                                                 int lane, int w) {
#pragma unroll 1
  for (int f = 0; f < ADP6_FB - 1; ++f) {
    adp6_fetch(S, d, g, s, f, zo, lane, w);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
}

// The right-hand sides (see k_adp6) from copies that run three faces ahead; the
// first three are on their way.  Leaves x free.
template <typename R>
__device__ __forceinline__ void adp6_rhs_ahead(R (&acc)[3][10], Adp6SmemT<R>& S, const Dims& d, const PhysC& ph, const DGeom& g,
                                               const DStateT<R>& s, unsigned zo, int lane, int w, int a, int h) {
  const long long PS = (long long)NPANEL * d.S;
  if (w == 5) {
    const double* cen = g.f[CS_G_V_CEN] + zo;
    const double* cf = g.f[CS_G_COEF] + 4 * PS + zo;
#pragma unroll
    for (int c = 0; c < 3; ++c) S.geo[c][lane] = (R)__ldg(cen + c * PS);
    S.geo[3][lane] = R(1.0) / fmax((R)__ldg(g.f[CS_G_V_SCALE] + zo), R(ph.smallnum));
#pragma unroll
    for (int m = 0; m < 6; ++m) S.geo[4 + m][lane] = (R)__ldg(cf + m * PS);
  }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int8_t* umap = s.adp_pmap + (3 * h + q) * 72 + 10 * a;
#pragma unroll
    for (int m = 0; m < 10; ++m) {
      const int u = __ldg(umap + m);
      acc[q][m] = (R)__ldg(umap + 36 + m) * s.V[(u % 10 * NVAR + 5 + u / 10) * PS + (3 * h + q) * d.S + zo];
    }
  }
  // normals and (component 0's warps) face weights, a face ahead
  R nn[5], wt[5];
  auto scalars = [&](int f) {
    const int dir = f >> 1;
    const unsigned fo = adp6_face(d, f, zo);
    const double* nf = (dir == 0 ? g.f[CS_G_XF_N] : (dir == 1 ? g.f[CS_G_YF_N] : g.f[CS_G_ZF_N])) + fo;
    const double* bw = (dir == 0 ? g.f[CS_G_XB_QW] : (dir == 1 ? g.f[CS_G_YB_QW] : g.f[CS_G_ZB_QW])) + fo;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      nn[c] = (R)__ldg(nf + (dir == 2 ? 5 * a + c : a) * PS);
      if (a == 0) wt[c] = (R)__ldg(bw + c * PS);
    }
  };
  scalars(0);
  adp6_sync();  // geo
#pragma unroll 1
  for (int f = 0; f < 6; ++f) {
    R(&bas)[5][9][ADP6_ZB] = S.bas[f & 1];
    const double(*fr)[ADP6_ZB] = S.face(f);
    asm volatile("cp.async.wait_group %0;" ::"n"(ADP6_FB - 2) : "memory");
    if (w < 5) {
      const R ob = S.geo[3][lane], x = ((R)fr[w][lane] - S.geo[0][lane]) * ob, y = ((R)fr[5 + w][lane] - S.geo[1][lane]) * ob,
              z = ((R)fr[10 + w][lane] - S.geo[2][lane]) * ob;
      bas[w][0][lane] = x;
      bas[w][1][lane] = y;
      bas[w][2][lane] = z;
      bas[w][3][lane] = x * x - S.geo[4][lane];
      bas[w][4][lane] = y * y - S.geo[5][lane];
      bas[w][5][lane] = z * z - S.geo[6][lane];
      bas[w][6][lane] = x * y - S.geo[7][lane];
      bas[w][7][lane] = y * z - S.geo[8][lane];
      bas[w][8][lane] = x * z - S.geo[9][lane];
    }
    // this face's rows and monomials are complete, the face before's no longer
    // read
    adp6_sync();
    if (a == 0) {
      R dacc[3] = {R(0.0), R(0.0), R(0.0)};
#pragma unroll
      for (int c = 0; c < 5; ++c)
#pragma unroll
        for (int q = 0; q < 3; ++q) dacc[q] = dacc[q] + wt[c] * (R)fr[15 + 5 * (3 * h + q) + c][lane];
#pragma unroll
      for (int q = 0; q < 3; ++q) S.x[30 + f][3 * h + q][lane] = dacc[q];
    }
    R n5[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) n5[c] = nn[c];
    if (f + ADP6_FB - 1 < 6) adp6_fetch(S, d, g, s, f + ADP6_FB - 1, zo, lane, w);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (f < 5) scalars(f + 1);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      R bq[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) bq[q] = (R)fr[15 + 5 * (3 * h + q) + c][lane];
#pragma unroll
      for (int q = 0; q < 3; ++q) acc[q][0] = acc[q][0] + n5[c] * bq[q];
#pragma unroll
      for (int m = 0; m < 9; ++m) {
        const R e = n5[c] * bas[c][m][lane];
#pragma unroll
        for (int q = 0; q < 3; ++q) acc[q][1 + m] = acc[q][1 + m] + e * bq[q];
      }
    }
  }
  adp6_sync();  // the last face's rows have been read
}

// The stream, the right-hand sides and the sums are in the state's type R
// (FP32 in the precision form: half the stream's bytes).
//
// In FP64 a face's points and values come through copies that run three faces
// ahead, into the next block's too: 13.1 -> 10.2 ms of a 6 x 128^2 x 64 step,
// 0.300 -> 0.279 of a 6 x 32^2 x 16 one, the same on the smallest.  The FP32
// form's right-hand sides leave room for two faces only, with which it was
// slower (8.7 -> 9.0 ms, 0.57 -> 0.66 ms on 6 x 50^2 x 13): its threads load
// their own.
template <typename R>
__global__ void __launch_bounds__(ADP6_THREADS, sizeof(R) == 4 ? 4 : 2) k_adp6(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  extern __shared__ __align__(128) unsigned char adp6_raw[];
  Adp6SmemT<R>& S = *reinterpret_cast<Adp6SmemT<R>*>(adp6_raw);
  const int tid = threadIdx.x;
  const long long n1 = r.count() / 6;
  const long long nblk = (n1 + ADP6_ZB - 1) / ADP6_ZB;
  if ((long long)blockIdx.x >= nblk) return;
  if (tid == 0) {
    for (int q = 0; q < ADP6_NS; ++q) {
      mbar_init(&S.full[q], 1);
      mbar_init(&S.empty[q], ADP6_CONS / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (tid >= ADP6_CONS) {
    if (tid == ADP6_CONS) {
      RingPos<ADP6_NS> ring;
      bool first = true;  // the ring's first round finds every stage free
      for (long long blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
        const R* src = (const R*)s.adp_lu + blk * (long long)(ADP6_WORDS * ADP6_ZB);
        for (int c = 0; c < ADP6_NCH; ++c) {
          if (!first) mbar_wait(&S.empty[ring.slot], ring.par ^ 1, s.err_flag);
          const int words = min(ADP6_CH, ADP6_WORDS - c * ADP6_CH);
          const uint32_t bytes = (uint32_t)(words * ADP6_ZB * sizeof(R));
          mbar_expect_tx(&S.full[ring.slot], bytes);
          bulk_g2s(&S.stage[ring.slot][0][0], src + c * ADP6_CH * ADP6_ZB, bytes, &S.full[ring.slot]);
          ring.next();
          if (ring.slot == 0) first = false;
        }
      }
    }
    return;
  }
  const int lane = tid & 31, w = tid >> 5;
  const long long PS = (long long)NPANEL * d.S;
  constexpr bool kAhead = sizeof(R) == 8;
  RingPos<ADP6_NS> ring;
  auto fetch_first = [&](long long blk) {  // of a block's position
    const long long t1 = blk * ADP6_ZB + lane;
    int p0 = 0, i = r.i0, j = r.j0, k = r.k0;
    if (t1 < n1) r.decode(t1, p0, i, j, k);
    adp6_fetch_first(S, d, g, s, (unsigned)d.idx(i, j, k), lane, w);
  };
  if constexpr (kAhead) fetch_first(blockIdx.x);
  for (long long blk = blockIdx.x; blk < nblk; blk += gridDim.x) {
    const long long t1 = blk * ADP6_ZB + lane;
    const bool inr = t1 < n1;
    // lanes past the range work on its first position and store nothing
    int p0 = 0, i = r.i0, j = r.j0, k = r.k0;
    if (inr) r.decode(t1, p0, i, j, k);
    // right-hand sides r1 = sum_q row_1(q) bq_p(q) + T_p^T vB_p, rows of
    // component a for panels 3 h .. 3 h + 2: panel 1's quadrature points one
    // face at a time, their monomials formed once by a warp a point
    const int a = w % 3, h = w / 3;
    R acc[3][10];
    {
      const unsigned zo = (unsigned)d.idx(i, j, k);  // box offset of the position
      if constexpr (kAhead) {
        adp6_rhs_ahead(acc, S, d, ph, g, s, zo, lane, w, a, h);
      } else {
        const double* cen = g.f[CS_G_V_CEN] + zo;
        const double* cf = g.f[CS_G_COEF] + zo;
        const R obl0 = R(1.0) / fmax((R)__ldg(g.f[CS_G_V_SCALE] + zo), R(ph.smallnum));
        const R vc0 = (R)__ldg(cen), vc1 = (R)__ldg(cen + PS), vc2 = (R)__ldg(cen + 2 * PS);
        R c0[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) c0[m] = (R)__ldg(cf + (4 + m) * PS);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int8_t* umap = s.adp_pmap + (3 * h + q) * 72 + 10 * a;
#pragma unroll
          for (int m = 0; m < 10; ++m) {
            const int u = __ldg(umap + m);
            acc[q][m] = (R)__ldg(umap + 36 + m) * s.V[(u % 10 * NVAR + 5 + u / 10) * PS + (3 * h + q) * d.S + zo];
          }
        }
#pragma unroll 1
        for (int f = 0; f < 6; ++f) {
          const int dir = f >> 1;
          const unsigned fo = zo - ((f & 1) ? (dir == 0 ? 1 : (dir == 1 ? d.NI : d.NI * d.NJ)) : 0);
          R(&bas)[5][9][ADP6_ZB] = S.bas[f & 1];
          if (w < 5) {
            const double* qp = (dir == 0 ? g.f[CS_G_XF_QP] : (dir == 1 ? g.f[CS_G_YF_QP] : g.f[CS_G_ZF_QP])) + fo;
            const R x = ((R)__ldg(qp + w * PS) - vc0) * obl0, y = ((R)__ldg(qp + (5 + w) * PS) - vc1) * obl0,
                    z = ((R)__ldg(qp + (10 + w) * PS) - vc2) * obl0;
            bas[w][0][lane] = x;
            bas[w][1][lane] = y;
            bas[w][2][lane] = z;
            bas[w][3][lane] = x * x - c0[0];
            bas[w][4][lane] = y * y - c0[1];
            bas[w][5][lane] = z * z - c0[2];
            bas[w][6][lane] = x * y - c0[3];
            bas[w][7][lane] = y * z - c0[4];
            bas[w][8][lane] = x * z - c0[5];
          }
          const double* Bq = (dir == 0 ? s.Bq[0] : (dir == 1 ? s.Bq[1] : s.Bq[2])) + 3 * h * d.S + fo;
          const double* nf = (dir == 0 ? g.f[CS_G_XF_N] : (dir == 1 ? g.f[CS_G_YF_N] : g.f[CS_G_ZF_N])) + fo;
          R bq[3][5], nn[5];
#pragma unroll
          for (int c = 0; c < 5; ++c) {
            nn[c] = (R)__ldg(nf + (dir == 2 ? 5 * a + c : a) * PS);
#pragma unroll
            for (int q = 0; q < 3; ++q) bq[q][c] = (R)Bq[c * PS + q * d.S];
          }
          if (a == 0) {
            const double* bw = (dir == 0 ? g.f[CS_G_XB_QW] : (dir == 1 ? g.f[CS_G_YB_QW] : g.f[CS_G_ZB_QW])) + fo;
            R dacc[3] = {R(0.0), R(0.0), R(0.0)};
#pragma unroll
            for (int c = 0; c < 5; ++c) {
              const R wt = (R)__ldg(bw + c * PS);
#pragma unroll
              for (int q = 0; q < 3; ++q) dacc[q] = dacc[q] + wt * bq[q][c];
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) S.x[30 + f][3 * h + q][lane] = dacc[q];
          }
          adp6_sync();
#pragma unroll
          for (int c = 0; c < 5; ++c) {
#pragma unroll
            for (int q = 0; q < 3; ++q) acc[q][0] = acc[q][0] + nn[c] * bq[q][c];
#pragma unroll
            for (int m = 0; m < 9; ++m) {
              const R e = nn[c] * bas[c][m][lane];
#pragma unroll
              for (int q = 0; q < 3; ++q) acc[q][1 + m] = acc[q][1 + m] + e * bq[q][c];
            }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int m = 0; m < 10; ++m) S.x[10 * a + m][3 * h + q][lane] = acc[q][m];
    }
    adp6_sync();
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int m = 0; m < 10; ++m) acc[q][m] = R(0.0);
    adp6_apply(acc, S, ring, lane, a, h, s.err_flag, std::make_integer_sequence<int, ADP6_NCH>{});
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int p = 3 * h + q;
      if (inr && mask_at(g, d, p, i, j) == 1) {
        const int8_t* umap = s.adp_pmap + p * 72 + 10 * a;
#pragma unroll
        for (int m = 0; m < 10; ++m) {
          const int u = __ldg(umap + m);
          const R val = (R)__ldg(umap + 36 + m) * acc[q][m];
          Vat(s, d, 5 + u / 10, u % 10, p, i, j, k) = val;
          if (m == 0) S.nb(p, u / 10)[lane] = val;
        }
      }
    }
    adp6_sync();
    if constexpr (kAhead) {  // x has been read
      if (blk + gridDim.x < nblk) fetch_first(blk + gridDim.x);
    }
    if (inr && mask_at(g, d, w, i, j) == 1) {
      R* U = s.U;
      const long long o5 = d.at(4, w, i, j, k);
      const double nb0 = S.nb(w, 0)[lane], nb1 = S.nb(w, 1)[lane], nb2 = S.nb(w, 2)[lane];
      const double u6 = U[d.at(5, w, i, j, k)], u7 = U[d.at(6, w, i, j, k)], u8 = U[d.at(7, w, i, j, k)];
      const double aa = (u6 * u6 + u7 * u7 + u8 * u8) * ph.ob8pi;
      U[d.at(5, w, i, j, k)] = nb0;
      U[d.at(6, w, i, j, k)] = nb1;
      U[d.at(7, w, i, j, k)] = nb2;
      const double bb = (nb0 * nb0 + nb1 * nb1 + nb2 * nb2) * ph.ob8pi;
      U[o5] = U[o5] - aa + bb;
    }
  }
}

template <typename R>
void launch_adp_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  const Range3 a = adp_zones(sv);
  if (st.adp_lu && st.adp_pmap) {
    const long long nblk = (a.count() / 6 + ADP6_ZB - 1) / ADP6_ZB;
    const int grid = (int)std::min<long long>(nblk, (long long)grid_sms(sv) * (sizeof(R) == 4 ? 4 : 2));
    k_adp6<R><<<grid, ADP6_THREADS, sizeof(Adp6SmemT<R>), sv.stream>>>(d, sv.ph, sv.g, st, a);
    mark(sv, "k_adp6");
    return;
  }
  if (st.adp_lu) {
    k_adp_rhs<R><<<blocks_for(a.count(), ADPR_TPB, grid_sms(sv)), ADPR_TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, a);
    mark(sv, "k_adp_rhs");
    const long long nblk = (a.count() + ADP_ZB - 1) / ADP_ZB;
    const int grid = (int)std::min<long long>(nblk, (long long)grid_sms(sv) * 2);
    k_adp_solve<R><<<grid, ADPS_THREADS, sizeof(AdpsSmem), sv.stream>>>(d, sv.ph, sv.g, st, a);
    mark(sv, "k_adp_solve");
    return;
  }
  const size_t smem = sizeof(AdpSmem) * ADP_WARPS;
  long long nwarps = a.count();
  long long nblk = (nwarps + ADP_WARPS - 1) / ADP_WARPS;
  long long cap = (long long)grid_sms(sv) * 16;
  if (nblk > cap) nblk = cap;
  k_adp<false, R><<<(int)nblk, 32 * ADP_WARPS, smem, sv.stream>>>(d, sv.ph, sv.g, st, a, a.count(), ADP_ZB);
  mark(sv, "k_adp");
}

void launch_adp(Solve& sv) {
  if (sv.fp32)
    launch_adp_t(sv, sv.stF);
  else
    launch_adp_t(sv, sv.st);
}

long long adp_range_count(const Solve& sv) { return adp_zones(sv).count(); }
long long adp_factor_doubles(const Solve& sv, bool shared) {
  const long long n = adp_range_count(sv);
  if (shared) return (n / 6 + ADP6_ZB - 1) / ADP6_ZB * (long long)ADP6_ZB * ADP6_WORDS;
  return (n + ADP_ZB - 1) / ADP_ZB * (long long)ADP_ZB * 1296;
}

void set_adp_smem_limits() {
  const int smem = (int)(sizeof(AdpSmem) * ADP_WARPS);
  cudaFuncSetAttribute(k_adp_solve<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AdpsSmem));
  cudaFuncSetAttribute(k_adp_solve<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AdpsSmem));
  cudaFuncSetAttribute(k_adp6<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Adp6SmemT<double>));
  cudaFuncSetAttribute(k_adp6<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Adp6SmemT<float>));
  cudaFuncSetAttribute(k_adp<false, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaFuncSetAttribute(k_adp<true, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaFuncSetAttribute(k_adp<false, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaFuncSetAttribute(k_adp<true, float>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

template <typename R>
void launch_adp_factor_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  const Range3 a = adp_zones(sv);
  const size_t smem = sizeof(AdpSmem) * ADP_WARPS;
  // shared factors: panel 1's zones only, in blocks of ADP6_ZB
  const long long tmax = st.adp_pmap ? a.count() / 6 : a.count();
  long long nblk = (tmax + ADP_WARPS - 1) / ADP_WARPS;
  long long cap = (long long)grid_sms(sv) * 16;
  if (nblk > cap) nblk = cap;
  k_adp<true, R><<<(int)nblk, 32 * ADP_WARPS, smem, sv.stream>>>(d, sv.ph, sv.g, st, a, tmax,
                                                                 st.adp_pmap ? ADP6_ZB : ADP_ZB);
  mark(sv, "k_adp_factor");
}

void launch_adp_factor(Solve& sv) {
  if (sv.fp32)
    launch_adp_factor_t(sv, sv.stF);
  else
    launch_adp_factor_t(sv, sv.st);
}

}  // namespace cs
