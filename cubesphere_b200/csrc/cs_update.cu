// Ghost exchange across the panel edges, radial padding, the RK stage
// combine, the conservative update with the constrained-transport face-B
// update, the post-update clean-up and the CFL reduction.
//
// Follows FETCH_BUFFERS_FILL_IN_UX / _UY (300riemann_module/330-332),
// PAD_BOUNDARY_R (800applications_cs/826pad_boundary_r.f:190-420),
// UPDATE_IMEX_RK_STEP_P1 (400riemann_integrate/484update_imex_rk_step_p1.f:212-906),
// CLEANUP_AFTER_UPDATE (485cleanup_after_update.f:383-1273),
// EVALUATE_TIMESTEP (490evaluate_timestep.f:121-286) and the RK combine of
// the driver (_I/_1000riemann_geomesh_cs_mhd/1000riemann_geomesh_cs_mhd.f:2661-2773).
#include <algorithm>

#include "cs_solve.h"

namespace cs {

namespace {

constexpr int TPB = 128;

// Fields the ghost exchange moves: 0 U, 1 entropy (the state's type R),
// 2..4 face B (always FP64).  Values travel as doubles.
template <typename R>
__device__ __forceinline__ double fill_load(const DStateT<R>& s, int f, int32_t at) {
  switch (f) {
    case 0: return (double)s.U[at];
    case 1: return (double)s.ent[at];
    case 2: return s.Bxf[at];
    case 3: return s.Byf[at];
    default: return s.Bzf[at];
  }
}
template <typename R>
__device__ __forceinline__ void fill_store(const DStateT<R>& s, int f, int32_t at, double v) {
  switch (f) {
    case 0: s.U[at] = (R)v; break;
    case 1: s.ent[at] = (R)v; break;
    case 2: s.Bxf[at] = v; break;
    case 3: s.Byf[at] = v; break;
    default: s.Bzf[at] = v;
  }
}

// Phase 1 of the exchange: every destination value is computed from the
// pre-exchange arrays (the reference reads all sources from buffers packed
// before any ghost is written).
template <typename R>
__global__ void k_fill_gather(DStateT<R> s, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                              const uint8_t* __restrict__ meta, double* __restrict__ tmp, long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int m = meta[t];
    double v = fill_load(s, (m >> 5) & 7, src[t]);
    if (m & 8) v = -v;
    if (m & 16) v = (fill_load(s, m & 7, dst[t]) + v) * 0.5;
    tmp[t] = v;
  }
}

template <typename R>
__global__ void k_fill_scatter(DStateT<R> s, const int32_t* __restrict__ dst, const uint8_t* __restrict__ meta,
                               const double* __restrict__ tmp, long long n) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    fill_store(s, meta[t] & 7, dst[t], tmp[t]);
}

// Radial outflow padding below k = 1 and above k = nr (826:190-420), one
// thread a column and ghost layer.  Two columns that share an x- or y-face
// copy the same value into it.
template <typename R>
__global__ void k_pad_radial(Dims d, DGeom g, DStateT<R> s, int bc_lower, int bc_upper) {
  const unsigned n1 = d.N + 2 * d.G, ncol = 6 * n1 * n1;
  const long long PS = (long long)NPANEL * d.S;
  const int dj = d.NI;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < 2 * d.G * ncol; t += gridDim.x * blockDim.x) {
    const unsigned layer = t / ncol, col = t - layer * ncol, u = col / n1;
    const int i = (int)(col - u * n1) + 1 - d.G, j = (int)(u % n1) + 1 - d.G, p = (int)(u / n1);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const bool upper = (int)layer >= d.G;
    const int kk = (int)layer - (upper ? d.G : 0) + 1;
    const long long b = (long long)p * d.S;
    if (!upper) {
      if (bc_lower != 2) continue;
      const long long l = b + d.idx(i, j, 1 - kk), r = b + d.idx(i, j, 1), dk = (long long)d.NI * d.NJ;
#pragma unroll
      for (int q = 0; q < NVAR; ++q) s.U[q * PS + l] = s.U[q * PS + r];
      s.Bxf[l] = s.Bxf[r];
      s.Bxf[l - 1] = s.Bxf[r - 1];
      s.Byf[l] = s.Byf[r];
      s.Byf[l - dj] = s.Byf[r - dj];
      s.Bzf[l - dk] = s.Bzf[r - dk];
    } else {
      if (bc_upper != 2) continue;
      const long long l = b + d.idx(i, j, d.nr + kk), r = b + d.idx(i, j, d.nr);
      const double *vol = g.f[CS_G_V_VOL], *xa = g.f[CS_G_XF_AREA], *ya = g.f[CS_G_YF_AREA], *za = g.f[CS_G_ZF_AREA];
      const double vr = __ldg(vol + r), vl = __ldg(vol + l);
#pragma unroll
      for (int q = 0; q < NVAR; ++q) s.U[q * PS + l] = s.U[q * PS + r] * vr / vl;
      s.Bzf[l] = s.Bzf[r] * __ldg(za + r) / __ldg(za + l);
      s.Bxf[l] = s.Bxf[r] * __ldg(xa + r) / __ldg(xa + l);
      s.Byf[l] = s.Byf[r] * __ldg(ya + r) / __ldg(ya + l);
      s.Bxf[l - 1] = s.Bxf[r - 1] * __ldg(xa + r - 1) / __ldg(xa + l - 1);
      s.Byf[l - dj] = s.Byf[r - dj] * __ldg(ya + r - dj) / __ldg(ya + l - dj);
    }
  }
}

// What one pass of the update does besides U += scale dt dU/dt.  A stage's save,
// combine and restore need no passes of their own: with them, the copies and the
// gravity a 6 x 32^2 x 1 step was 111 launches, now 73.  Both updates are bound by
// HBM on large meshes (1.3 and 1.0 ms of a 6 x 128^2 x 64 step):
//   UP_PLAIN  nothing (the routine by itself)
//   UP_SAVE   first stage: also saves the state
//   UP_MEAN   (x + x0) / 2 first (RK2's second stage)
//   UP_MIX    a0 x0 + (1 - a0) x first (SSP-RK3)
//   UP_IMEX1  UP_SAVE with the first stage's rates, then the implicit gravity
//   UP_IMEX2  from the saved state: scale0 dt of the first stage's rates, then
//             scale dt of the current ones with cg S(U) of the current state
//             added, then the implicit gravity
enum UpMode { UP_PLAIN, UP_SAVE, UP_MEAN, UP_MIX, UP_IMEX1, UP_IMEX2 };
struct UpArgs {
  double scale;   // of the time step, for the current rates
  double scale0;  // for the first stage's
  double a0;      // UP_MIX
  double cg;      // UP_IMEX2
  double gam;     // implicit gravity
  bool gravity;
};

// RK combine of a value with the saved one, in FP64.
template <int M>
__device__ __forceinline__ double up_combine(double x, double x0, double a0) {
  return M == UP_MIX ? a0 * x0 + (1.0 - a0) * x : (x + x0) * 0.5;
}

// The entropy update (484:330-372) of interior zone (i,j,k) and the
// conserved->primitive repair.
template <typename R>
__device__ __forceinline__ void up_entropy(const Dims& d, const PhysC& ph, const DGeom& g, R* const* EF, long long o,
                                           long long dk, R dt, R& en, R* U) {
  const double *xa = g.f[CS_G_XF_AREA] + o, *ya = g.f[CS_G_YF_AREA] + o, *za = g.f[CS_G_ZF_AREA] + o;
  const R div = (R)__ldg(xa) * EF[0][o] - (R)__ldg(xa - 1) * EF[0][o - 1] + (R)__ldg(ya) * EF[1][o] -
                (R)__ldg(ya - d.NI) * EF[1][o - d.NI] + (R)__ldg(za) * EF[2][o] - (R)__ldg(za - dk) * EF[2][o - dk];
  R V[8];
  en = en - dt * div / (R)__ldg(g.f[CS_G_V_VOL] + o);
  d_cons_to_prim(ph, en, U, V);
}

// Zone update (484:212-372): U += dt dU/dt on the zones r, then on the
// interior the entropy update and the conserved->primitive repair, with the
// stage's combine and the IMEX gravity in the same pass.  The time step is
// scale times the device-resident step of the solve.
//
// Gravity S(U) = (0, -rho g, -m . g), g = GM x / r^3, on the active zones
// 0..N+1 (the zones of BUILD_NON_STIFF_SOURCES).  rho is unchanged by it, so
// the implicit stage U = U* + a S(U) has the closed form m = m* - a rho g,
// E = E* - a m . g.
template <int M, typename R>
__global__ void __launch_bounds__(TPB) k_update_zones(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r, UpArgs a) {
  const long long PS = (long long)NPANEL * d.S, dk = (long long)d.NI * d.NJ;
  const R dt = (R)(a.scale * *s.dt), dt0 = (R)(a.scale0 * *s.dt), ag = (R)(a.gam * *s.dt);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    const bool inside = i >= 1 && i <= d.N && j >= 1 && j <= d.N && k >= 1 && k <= d.nr;
    const bool heavy = (M == UP_IMEX1 || M == UP_IMEX2) && a.gravity && i >= 0 && i <= d.N + 1 && j >= 0 && j <= d.N + 1 &&
                       k >= 0 && k <= d.nr + 1 && mask_at(g, d, p, i, j) == 1;
    R gx = R(0.0), gy = R(0.0), gz = R(0.0);
    if (heavy) {
      const double* cen = g.f[CS_G_V_CEN] + o;
      const R x = (R)__ldg(cen), y = (R)__ldg(cen + PS), z = (R)__ldg(cen + 2 * PS);
      const R rad = sqrt(x * x + y * y + z * z);
      const R gmb = R(ph.gm) * (R(1.0) / (rad * rad * rad));
      gx = gmb * x;
      gy = gmb * y;
      gz = gmb * z;
    }
    const R* K = (M == UP_IMEX1 ? s.K1 : s.dUdt) + o;
    R* const* EF = M == UP_IMEX1 ? s.EF1 : s.EF;
    R U[8], en = R(0.0);
    if (M == UP_IMEX2) {
      R dU[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) dU[q] = K[q * PS];
      if (heavy) {
        const R c = (R)a.cg, rho = s.U[o], m1 = s.U[PS + o], m2 = s.U[2 * PS + o], m3 = s.U[3 * PS + o];
        dU[1] += c * (-(gx * rho));
        dU[2] += c * (-(gy * rho));
        dU[3] += c * (-(gz * rho));
        dU[4] += c * (-(gx * m1 + gy * m2 + gz * m3));
#pragma unroll
        for (int q = 1; q < 5; ++q) s.dUdt[q * PS + o] = dU[q];  // part of the rates from here on
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) U[q] = s.U0[q * PS + o] + dt0 * s.K1[q * PS + o];
      if (inside) {
        en = s.ent0[o];
        up_entropy(d, ph, g, s.EF1, o, dk, dt0, en, U);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) U[q] = U[q] + dt * dU[q];
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        U[q] = s.U[q * PS + o];
        if (M == UP_SAVE || M == UP_IMEX1) s.U0[q * PS + o] = U[q];
        if (M == UP_MEAN || M == UP_MIX) U[q] = (R)up_combine<M>((double)U[q], (double)s.U0[q * PS + o], a.a0);
        U[q] = U[q] + dt * K[q * PS];
      }
      en = s.ent[o];
      if (M == UP_SAVE || M == UP_IMEX1) s.ent0[o] = en;
      if (M == UP_MEAN || M == UP_MIX) en = (R)up_combine<M>((double)en, (double)s.ent0[o], a.a0);
    }
    if (inside) up_entropy(d, ph, g, EF, o, dk, dt, en, U);
    else if (M == UP_IMEX2) en = s.ent0[o];
    if (M != UP_PLAIN || inside) s.ent[o] = en;
    if (heavy) {
      U[1] = U[1] - ag * (gx * U[0]);
      U[2] = U[2] - ag * (gy * U[0]);
      U[3] = U[3] - ag * (gz * U[0]);
      U[4] = U[4] - ag * (gx * U[1] + gy * U[2] + gz * U[3]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) s.U[q * PS + o] = U[q];
  }
}

__device__ __forceinline__ double vrad(const DGeom& g, const Dims& d, int p, int i, int j, int k) {
  const double x = geo(g, d, CS_G_VERT, 0, p, i, j, k), y = geo(g, d, CS_G_VERT, 1, p, i, j, k),
               z = geo(g, d, CS_G_VERT, 2, p, i, j, k);
  return sqrt(x * x + y * y + z * z);
}
// Angle between the vertices a and b on the sphere of radius 1/inv.
__device__ __forceinline__ double vang(const DGeom& g, const Dims& d, int p, int ax, int ay, int bx, int by, int k,
                                       double inv) {
  const double c = (geo(g, d, CS_G_VERT, 0, p, ax, ay, k) * inv) * (geo(g, d, CS_G_VERT, 0, p, bx, by, k) * inv) +
                   (geo(g, d, CS_G_VERT, 1, p, ax, ay, k) * inv) * (geo(g, d, CS_G_VERT, 1, p, bx, by, k) * inv) +
                   (geo(g, d, CS_G_VERT, 2, p, ax, ay, k) * inv) * (geo(g, d, CS_G_VERT, 2, p, bx, by, k) * inv);
  return acos(c);
}

// Constrained-transport face update (484:376-906): Stokes circulation of
// the edge EMFs with spherical arc lengths for the angular edges, with the
// stage's save, combine or restore of face B in the same pass.  One launch
// for the three face directions over the faces r; only the interior zones'
// faces have a circulation.
template <int M, typename R>
__global__ void __launch_bounds__(TPB) k_ct(Dims d, DGeom g, DStateT<R> s, Range3 r, UpArgs a) {
  const double dt = a.scale * *s.dt, dt0 = a.scale0 * *s.dt;
  const long long dk = (long long)d.NI * d.NJ;
  const unsigned nb = (unsigned)((r.count() + TPB - 1) / TPB);
  for (unsigned T = blockIdx.x; T < 3 * nb; T += gridDim.x) {
    const int dir = T % 3;
    const long long t = (long long)(T / 3) * TPB + threadIdx.x;
    if (t >= r.count()) continue;
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    double* B = dir == 0 ? s.Bxf : (dir == 1 ? s.Byf : s.Bzf);
    double* B0 = dir == 0 ? s.B0[0] : (dir == 1 ? s.B0[1] : s.B0[2]);
    const bool inside = i >= (dir != 0) && i <= d.N && j >= (dir != 1) && j <= d.N && k >= (dir != 2) && k <= d.nr;
    if (M == UP_PLAIN && !inside) continue;
    double b;
    if (M == UP_IMEX2) {
      b = B0[o];
    } else {
      b = B[o];
      if (M == UP_SAVE || M == UP_IMEX1) B0[o] = b;
      if (M == UP_MEAN || M == UP_MIX) b = up_combine<M>(b, B0[o], a.a0);
    }
    if (inside) {
      // circulation: the lengths of the four edges once, then the EMFs of the
      // current rates (and of the first stage's)
      double w[4];
      long long e[4];
      const double area = __ldg((dir == 0 ? g.f[CS_G_XF_AREA] : (dir == 1 ? g.f[CS_G_YF_AREA] : g.f[CS_G_ZF_AREA])) + o);
      const double rout = vrad(g, d, p, i, j, k);
      int c0, c2;  // EMF components of edges 0, 1 and 2, 3
      if (dir == 2) {
        const double inv = 1.0 / rout;
        w[0] = rout * vang(g, d, p, i, j, i, j - 1, k, inv);
        w[1] = -rout * vang(g, d, p, i - 1, j, i - 1, j - 1, k, inv);
        w[2] = -rout * vang(g, d, p, i, j, i - 1, j, k, inv);
        w[3] = rout * vang(g, d, p, i, j - 1, i - 1, j - 1, k, inv);
        c0 = 1;
        c2 = 0;
        e[0] = o;
        e[1] = o - 1;
        e[2] = o;
        e[3] = o - d.NI;
      } else {
        const double rin = vrad(g, d, p, i, j, k - 1), dr = rout - rin;
        const double th = dir == 0 ? vang(g, d, p, i, j, i, j - 1, k, 1.0 / rout) : vang(g, d, p, i, j, i - 1, j, k, 1.0 / rout);
        const double sg = dir == 0 ? 1.0 : -1.0;
        w[0] = sg * dr;
        w[1] = -sg * dr;
        w[2] = -sg * (rout * th);
        w[3] = sg * (rin * th);
        c0 = 2;
        c2 = dir == 0 ? 1 : 0;
        e[0] = o;
        e[1] = o - (dir == 0 ? d.NI : 1);
        e[2] = o;
        e[3] = o - dk;
      }
      if (M == UP_IMEX2) {
        const double* Ea = c0 == 2 ? s.Ef1[2] : s.Ef1[1];
        const double* Eb = c2 == 1 ? s.Ef1[1] : s.Ef1[0];
        b = b - dt0 * (w[0] * Ea[e[0]] + w[1] * Ea[e[1]] + w[2] * Eb[e[2]] + w[3] * Eb[e[3]]) / area;
      }
      double* const* Ef = M == UP_IMEX1 ? s.Ef1 : s.Ef;
      const double* Ea = c0 == 2 ? Ef[2] : Ef[1];
      const double* Eb = c2 == 1 ? Ef[1] : Ef[0];
      b = b - dt * (w[0] * Ea[e[0]] + w[1] * Ea[e[1]] + w[2] * Eb[e[2]] + w[3] * Eb[e[3]]) / area;
    }
    B[o] = b;
  }
}

// Clean-up zone pass (485:688-1273): least-squares zone-centred B from the
// six face values on active zones with the matching total-energy fix, then
// the conserved->primitive repair on every zone.
template <typename R>
__global__ void k_cleanup_zones(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    double U[8], V[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) U[q] = s.U[d.at(q, p, i, j, k)];
    if (mask_at(g, d, p, i, j) == 1) {
      double nv[3] = {geo(g, d, CS_G_ZF_CEN, 0, p, i, j, k), geo(g, d, CS_G_ZF_CEN, 1, p, i, j, k),
                      geo(g, d, CS_G_ZF_CEN, 2, p, i, j, k)};
      const double a = 1.0 / fmax(ph.smallnum, sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]));
      nv[0] = nv[0] * a;
      nv[1] = nv[1] * a;
      nv[2] = nv[2] * a;
      double Am[6][3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        Am[0][q] = geo(g, d, CS_G_XF_N, q, p, i, j, k);
        Am[1][q] = geo(g, d, CS_G_XF_N, q, p, i - 1, j, k);
        Am[2][q] = geo(g, d, CS_G_YF_N, q, p, i, j, k);
        Am[3][q] = geo(g, d, CS_G_YF_N, q, p, i, j - 1, k);
        Am[4][q] = nv[q];
        Am[5][q] = nv[q];
      }
      const double Rm[6] = {s.Bxf[d.at(0, p, i, j, k)], s.Bxf[d.at(0, p, i - 1, j, k)], s.Byf[d.at(0, p, i, j, k)],
                            s.Byf[d.at(0, p, i, j - 1, k)], s.Bzf[d.at(0, p, i, j, k)], s.Bzf[d.at(0, p, i, j, k - 1)]};
      double M[3][3], rhs[3];
#pragma unroll
      for (int a1 = 0; a1 < 3; ++a1) {
#pragma unroll
        for (int a2 = 0; a2 < 3; ++a2) {
          double sm = 0.0;
#pragma unroll
          for (int q = 0; q < 6; ++q) sm = sm + Am[q][a1] * Am[q][a2];
          M[a1][a2] = sm;
        }
        double sm = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) sm = sm + Am[q][a1] * Rm[q];
        rhs[a1] = sm;
      }
      const double a11 = M[0][0], a12 = M[0][1], a13 = M[0][2], a21 = M[1][0], a22 = M[1][1], a23 = M[1][2],
                   a31 = M[2][0], a32 = M[2][1], a33 = M[2][2];
      const double det = a11 * (a22 * a33 - a32 * a23) - a12 * (a21 * a33 - a31 * a23) + a13 * (a21 * a32 - a31 * a22);
      const double ob = copysign(1.0, det) / fmax(1.0e-32, fabs(det));
      const double b11 = (a22 * a33 - a23 * a32) * ob, b12 = (a13 * a32 - a12 * a33) * ob, b13 = (a12 * a23 - a22 * a13) * ob;
      const double b21 = (a23 * a31 - a21 * a33) * ob, b22 = (a11 * a33 - a13 * a31) * ob, b23 = (a13 * a21 - a11 * a23) * ob;
      const double b31 = (a21 * a32 - a22 * a31) * ob, b32 = (a12 * a31 - a11 * a32) * ob, b33 = (a11 * a22 - a12 * a21) * ob;
      const double nb0 = b11 * rhs[0] + b12 * rhs[1] + b13 * rhs[2];
      const double nb1 = b21 * rhs[0] + b22 * rhs[1] + b23 * rhs[2];
      const double nb2 = b31 * rhs[0] + b32 * rhs[1] + b33 * rhs[2];
      const double Bx = U[5], By = U[6], Bz = U[7];
      U[5] = nb0;
      U[6] = nb1;
      U[7] = nb2;
      U[4] = U[4] - (Bx * Bx + By * By + Bz * Bz) * ph.ob8pi + (nb0 * nb0 + nb1 * nb1 + nb2 * nb2) * ph.ob8pi;
    }
    double en = s.ent[d.at(0, p, i, j, k)];
    d_cons_to_prim(ph, en, U, V);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      s.U[d.at(q, p, i, j, k)] = U[q];
      s.V[d.at(q, p, i, j, k)] = V[q];
    }
    s.ent[d.at(0, p, i, j, k)] = en;
  }
}

// The solve's time step, and the start of the next CFL reduction: 1.1 times
// it (490:121-286).
__global__ void k_set_dt(double* dt, unsigned long long* dtmin, double v) {
  *dt = v;
  *dtmin = (unsigned long long)__double_as_longlong(1.1 * v);
}

// CFL limit over the active interior zones; the minimum positive double is
// found with an integer atomicMin on its bit pattern (positive IEEE doubles
// order like their bit patterns).  The last block to finish makes the result
// the solve's next step and starts the reduction after it.
template <typename R>
__global__ void k_timestep(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  double dtl = 1.0e300;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) == 0) continue;
    double U[8], V[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) U[q] = s.U[d.at(q, p, i, j, k)];
    double en = s.ent[d.at(0, p, i, j, k)];
    d_cons_to_prim(ph, en, U, V);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      s.U[d.at(q, p, i, j, k)] = U[q];
      s.V[d.at(q, p, i, j, k)] = V[q];
    }
    s.ent[d.at(0, p, i, j, k)] = en;
    const double b2 = V[5] * V[5] + V[6] * V[6] + V[7] * V[7];
    const double ms = sqrt((ph.gamma * V[4] + ph.ob4pi * b2) / V[0]);
    s.msonic[d.at(0, p, i, j, k)] = ms;
    const double a21 = sqrt(V[1] * V[1] + V[2] * V[2] + V[3] * V[3]) + ms;
    dtl = fmin(dtl, ph.cfl * geo(g, d, CS_G_V_SCALE, 0, p, i, j, k) / a21);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dtl = fmin(dtl, __shfl_down_sync(0xffffffffu, dtl, o));
  if ((threadIdx.x & 31) == 0 && dtl < 1.0e300 && dtl > 0.0)
    atomicMin(s.dtmin, (unsigned long long)__double_as_longlong(dtl));
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned* done = reinterpret_cast<unsigned*>(s.dtmin + 1);
    __threadfence();
    if (atomicAdd(done, 1u) == gridDim.x - 1) {
      *done = 0;
      const double dt = __longlong_as_double((long long)atomicAdd(s.dtmin, 0ULL));
      *s.dt = dt;
      *s.dtmin = (unsigned long long)__double_as_longlong(1.1 * dt);
    }
  }
}

inline Range3 zones_all(const Dims& d) { return {1 - d.G, d.N + d.G, 1 - d.G, d.N + d.G, 1 - d.G, d.nr + d.G}; }

}  // namespace

template <typename R>
void launch_fill_ghosts_t(Solve& sv, const DStateT<R>& st) {
  const FillMap& f = sv.fill;
  if (f.n > 0) {
    const int nb = blocks_for(f.n, 256, grid_sms(sv));
    k_fill_gather<R><<<nb, 256, 0, sv.stream>>>(st, f.d_src, f.d_dst, f.d_meta, f.d_tmp, f.n);
    mark(sv, "k_fill_gather");
    k_fill_scatter<R><<<nb, 256, 0, sv.stream>>>(st, f.d_dst, f.d_meta, f.d_tmp, f.n);
    mark(sv, "k_fill_scatter");
  }
  const int n1 = sv.d.N + 2 * sv.d.G;
  k_pad_radial<R><<<blocks_for(12LL * sv.d.G * n1 * n1, TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.g, st, sv.p.bc_lower,
                                                                                      sv.p.bc_upper);
  mark(sv, "k_pad_radial");
}
void launch_fill_ghosts(Solve& sv) {
  if (sv.fp32)
    launch_fill_ghosts_t(sv, sv.stF);
  else
    launch_fill_ghosts_t(sv, sv.st);
}

template <int M, typename R>
void launch_update_mode(Solve& sv, const DStateT<R>& st, const UpArgs& a) {
  const Dims& d = sv.d;
  const Range3 z = own_columns(d, d.G);
  k_update_zones<M, R><<<blocks_for(z.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, z, a);
  mark(sv, "k_update_zones");
  // UP_PLAIN touches the interior zones' faces only
  const Range3 f = M == UP_PLAIN ? Range3{0, d.N, 0, d.N, 0, d.nr} : Range3{0, d.N, 0, d.N, z.k0 - 1, z.k1};
  const long long nb = 3 * ((f.count() + TPB - 1) / TPB);
  k_ct<M, R><<<(int)std::min<long long>(nb, (long long)grid_sms(sv) * 64), TPB, 0, sv.stream>>>(d, sv.g, st, f, a);
  mark(sv, "k_ct");
}
template <typename R>
void launch_update_t(Solve& sv, const DStateT<R>& st, int mode, const UpArgs& a) {
  switch (mode) {
    case UP_PLAIN: launch_update_mode<UP_PLAIN>(sv, st, a); break;
    case UP_SAVE: launch_update_mode<UP_SAVE>(sv, st, a); break;
    case UP_MEAN: launch_update_mode<UP_MEAN>(sv, st, a); break;
    case UP_MIX: launch_update_mode<UP_MIX>(sv, st, a); break;
    case UP_IMEX1: launch_update_mode<UP_IMEX1>(sv, st, a); break;
    default: launch_update_mode<UP_IMEX2>(sv, st, a);
  }
}
static void launch_update_args(Solve& sv, int mode, UpArgs a) {
  a.gravity = sv.ph.gm > sv.p.smallnum;
  if (sv.fp32)
    launch_update_t(sv, sv.stF, mode, a);
  else
    launch_update_t(sv, sv.st, mode, a);
}
void launch_update(Solve& sv, double scale) { launch_update_args(sv, UP_PLAIN, {scale, 0.0, 0.0, 0.0, 0.0, false}); }
void launch_update_rk(Solve& sv, int irk, double a0, double scale) {
  launch_update_args(sv, irk == 1 ? UP_SAVE : (a0 > 0.0 ? UP_MIX : UP_MEAN), {scale, 0.0, a0, 0.0, 0.0, false});
}
void launch_update_imex(Solve& sv, int irk, double gam, double del) {
  if (irk == 1)
    launch_update_args(sv, UP_IMEX1, {gam, 0.0, 0.0, 0.0, gam, false});
  else
    launch_update_args(sv, UP_IMEX2, {1.0 - del, del, 0.0, (1.0 - gam) / (1.0 - del), gam, false});
}

template <typename R>
void launch_cleanup_t(Solve& sv, const DStateT<R>& st, const Range3& z) {
  k_cleanup_zones<R><<<blocks_for(z.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(sv.d, sv.ph, sv.g, st, z);
  mark(sv, "k_cleanup_zones");
}
void launch_cleanup(Solve& sv, bool masks) {
  if (masks) launch_face_masks(sv);
  const Range3 z = masks ? zones_all(sv.d) : own_columns(sv.d, sv.d.G);
  if (sv.fp32)
    launch_cleanup_t(sv, sv.stF, z);
  else
    launch_cleanup_t(sv, sv.st, z);
}

template <typename R>
void launch_timestep_t(Solve& sv, const DStateT<R>& st) {
  Range3 r = {1, sv.d.N, 1, sv.d.N, 1, sv.d.nr};
  k_timestep<R><<<blocks_for(r.count(), 256, grid_sms(sv)), 256, 0, sv.stream>>>(sv.d, sv.ph, sv.g, st, r);
  mark(sv, "k_timestep");
}
void launch_timestep(Solve& sv) {
  if (sv.fp32)
    launch_timestep_t(sv, sv.stF);
  else
    launch_timestep_t(sv, sv.st);
}

// Conservation diagnostics over the interior zones (FP64): volume-weighted
// sums of rho and of the total energy, and the largest |div B| (face-area
// weighted circulation of the face B over the zone volume).  A fixed grid
// of DIAG_BLOCKS blocks writes partial sums that one block then adds in a
// fixed order, so the result does not depend on launch shapes or timing.
constexpr int DIAG_BLOCKS = 512, DIAG_TPB = 256;
template <typename R>
__global__ void __launch_bounds__(DIAG_TPB) k_diag_partial(Dims d, DGeom g, DStateT<R> s, Range3 r, double* part) {
  double m = 0.0, e = 0.0, dv = 0.0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    const double vol = geo(g, d, CS_G_V_VOL, 0, p, i, j, k);
    m += (double)s.U[d.at(0, p, i, j, k)] * vol;
    e += (double)s.U[d.at(4, p, i, j, k)] * vol;
    const double flux = geo(g, d, CS_G_XF_AREA, 0, p, i, j, k) * s.Bxf[d.at(0, p, i, j, k)] -
                        geo(g, d, CS_G_XF_AREA, 0, p, i - 1, j, k) * s.Bxf[d.at(0, p, i - 1, j, k)] +
                        geo(g, d, CS_G_YF_AREA, 0, p, i, j, k) * s.Byf[d.at(0, p, i, j, k)] -
                        geo(g, d, CS_G_YF_AREA, 0, p, i, j - 1, k) * s.Byf[d.at(0, p, i, j - 1, k)] +
                        geo(g, d, CS_G_ZF_AREA, 0, p, i, j, k) * s.Bzf[d.at(0, p, i, j, k)] -
                        geo(g, d, CS_G_ZF_AREA, 0, p, i, j, k - 1) * s.Bzf[d.at(0, p, i, j, k - 1)];
    dv = fmax(dv, fabs(flux) / vol);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m += __shfl_down_sync(0xffffffffu, m, o);
    e += __shfl_down_sync(0xffffffffu, e, o);
    dv = fmax(dv, __shfl_down_sync(0xffffffffu, dv, o));
  }
  __shared__ double red[3][DIAG_TPB / 32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    red[0][w] = m;
    red[1][w] = e;
    red[2][w] = dv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int q = 0; q < DIAG_TPB / 32; ++q) {
      a += red[0][q];
      b += red[1][q];
      c = fmax(c, red[2][q]);
    }
    part[3 * blockIdx.x] = a;
    part[3 * blockIdx.x + 1] = b;
    part[3 * blockIdx.x + 2] = c;
  }
}
__global__ void k_diag_final(const double* part, int n, double* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int q = 0; q < n; ++q) {
      a += part[3 * q];
      b += part[3 * q + 1];
      c = fmax(c, part[3 * q + 2]);
    }
    out[0] = a;
    out[1] = b;
    out[2] = c;
  }
}

template <typename R>
void launch_diag_t(Solve& sv, const DStateT<R>& st, double* part, double* out) {
  const Range3 r = {1, sv.d.N, 1, sv.d.N, 1, sv.d.nr};
  k_diag_partial<R><<<DIAG_BLOCKS, DIAG_TPB, 0, sv.stream>>>(sv.d, sv.g, st, r, part);
  mark(sv, "k_diag_partial");
  k_diag_final<<<1, 32, 0, sv.stream>>>(part, DIAG_BLOCKS, out);
  mark(sv, "k_diag_final");
}
void launch_diag(Solve& sv, double* part, double* out) {
  if (sv.fp32)
    launch_diag_t(sv, sv.stF, part, out);
  else
    launch_diag_t(sv, sv.st, part, out);
}
size_t diag_scratch_doubles() { return 3 * DIAG_BLOCKS + 4; }

void launch_set_dt(Solve& sv, double dt) {
  k_set_dt<<<1, 1, 0, sv.stream>>>(sv.fp32 ? sv.stF.dt : sv.st.dt, sv.fp32 ? sv.stF.dtmin : sv.st.dtmin, dt);
  mark(sv, "k_set_dt");
}

}  // namespace cs
