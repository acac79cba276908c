// Edge electric fields for the constrained-transport update: three-point
// Simpson rule along every edge, four-state multidimensional HLL solver
// with the symmetrised (LLF) speeds, and the three-state solver on the
// radial edges at the four cube corners of each panel.
//
// Follows MAKE_EDGE_EFIELDS_P1 with USE_2D_LLF_RS_FOR_EZ = 1
// (pkg/inc/cubesphere/400riemann_integrate/460make_edge_fields_p1.f:335-7037),
// Two_D_RS_Ez_4State_HLL (620riemann_2d/630...:10-372) and
// Two_D_RS_Ez_3State_HLL (620riemann_2d/631...:9-338).  One thread per edge.
#include <algorithm>

#include "cs_solve.h"

namespace cs {

namespace {

constexpr int TPB = 128;

template <typename R>
__device__ __forceinline__ double E1(const DStateT<R>& s, const Dims& d, int q, int p, int i, int j, int k) {
  return s.E[d.at(q, p, i, j, k)];
}
template <typename T>
__device__ __forceinline__ double Sg(const T* a, const Dims& d, int p, int i, int j, int k) {
  return a[d.at(0, p, i, j, k)];
}
template <typename R>
__device__ __forceinline__ double Bqa(const DStateT<R>& s, const Dims& d, int dir, int q, int p, int i, int j, int k) {
  return s.Bq[dir][d.at(q, p, i, j, k)];
}

// E along the tangent of the edge between the vertices va and vb (one sphere)
// by Simpson's rule: at each point P (the two ends and the middle) the tangent
// t = va - vb is made orthogonal to the radial direction and normalised,
//   E . n = (t.E - (t.P)(P.E) / P.P) / sqrt(t.t - (t.P)^2 / P.P).
__device__ __forceinline__ double along_edge(const double* va, const double* vb, const double* E) {
  double t[3], m[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    t[q] = va[q] - vb[q];
    m[q] = va[q] + vb[q];
  }
  const double tt = t[0] * t[0] + t[1] * t[1] + t[2] * t[2], tE = t[0] * E[0] + t[1] * E[1] + t[2] * E[2];
  auto at = [&](const double* P) {
    const double tP = t[0] * P[0] + t[1] * P[1] + t[2] * P[2];
    const double f = tP / (P[0] * P[0] + P[1] * P[1] + P[2] * P[2]);
    return (tE - f * (P[0] * E[0] + P[1] * E[1] + P[2] * E[2])) / sqrt(tt - f * tP);
  };
  return (4.0 / 6.0) * at(m) + (1.0 / 6.0) * (at(va) + at(vb));
}
__device__ __forceinline__ double llf_speed(double a, double b, double c, double e) {
  return fmax(fmax(fabs(a), fabs(b)), fmax(fabs(c), fabs(e)));
}

// The symmetrised (LLF) speeds and one E for the four states, USE_2D_LLF_RS_FOR_EZ:
// with S_R = S_U = -S_L = -S_D = s the four-state solver (d_rs4, 630:10-372)
// has its interaction region's centroid at the origin, and its two averages
// agree and reduce to
//   E + s / (2 sin) ((B_y,R - B_y,L) - (B_n,U - B_n,D)).
__device__ __forceinline__ double llf_emf(double s, double sin_t, double E, double BnU, double BnD, double ByR, double ByL) {
  return E + 0.5 * s * ((ByR - ByL) - (BnU - BnD)) / sin_t;
}

// x-edges (460:393-1493): i in 1..N, j in 0..N, k in 0..nr.
template <typename R>
__device__ __forceinline__ void edge_x(const Dims& d, const DGeom& g, const DStateT<R>& s, int p, int i, int j, int k) {
  const long long PS = (long long)NPANEL * d.S, o = (long long)p * d.S + d.idx(i, j, k);
  const int dj = d.NI, dk = d.NI * d.NJ;
  double E[3], va[3], vb[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const R* e = s.E + q * PS + o;
    E[q] = ((double)e[0] + (double)e[dj] + (double)e[dj + dk] + (double)e[dk]) * 0.25;
    va[q] = __ldg(g.f[CS_G_VERT] + q * PS + o);
    vb[q] = __ldg(g.f[CS_G_VERT] + q * PS + o - 1);
  }
  const double sp = fmax(llf_speed(s.S[3][o + dk], s.S[3][o], s.S[2][o + dk], s.S[2][o]),
                         llf_speed(s.S[5][o + dj], s.S[5][o], s.S[4][o + dj], s.S[4][o]));
  s.Ef[0][o] = llf_emf(sp, 1.0, along_edge(va, vb, E), s.Bq[1][2 * PS + o + dk], s.Bq[1][PS + o], s.Bq[2][4 * PS + o + dj],
                       s.Bq[2][3 * PS + o]);
}

// y-edges (460:1497-2587): i in 0..N, j in 1..N, k in 0..nr.
template <typename R>
__device__ __forceinline__ void edge_y(const Dims& d, const DGeom& g, const DStateT<R>& s, int p, int i, int j, int k) {
  const long long PS = (long long)NPANEL * d.S, o = (long long)p * d.S + d.idx(i, j, k);
  const int dk = d.NI * d.NJ;
  double E[3], va[3], vb[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const R* e = s.E + q * PS + o;
    E[q] = ((double)e[0] + (double)e[dk] + (double)e[dk + 1] + (double)e[1]) * 0.25;
    va[q] = __ldg(g.f[CS_G_VERT] + q * PS + o);
    vb[q] = __ldg(g.f[CS_G_VERT] + q * PS + o - d.NI);
  }
  const double sp = fmax(llf_speed(s.S[5][o + 1], s.S[5][o], s.S[4][o + 1], s.S[4][o]),
                         llf_speed(s.S[1][o + dk], s.S[1][o], s.S[0][o + dk], s.S[0][o]));
  s.Ef[1][o] = llf_emf(sp, 1.0, along_edge(va, vb, E), s.Bq[2][2 * PS + o + 1], s.Bq[2][PS + o], s.Bq[0][4 * PS + o + dk],
                       s.Bq[0][3 * PS + o]);
}

// z-edges (460:2591-3721): i, j in 0..N, k in 1..nr, zero where a neighbour
// is masked; the four cube corners (460:3725-7037) use the three-state
// solver.  The vertices of a radial edge are radii times one unit vector, so
// the three points of the rule share one frame.
template <typename R>
__device__ __forceinline__ void edge_z(const Dims& d, const DGeom& g, const DStateT<R>& s, int p, int i, int j, int k) {
  const int N = d.N, dj = d.NI;
  const long long PS = (long long)NPANEL * d.S, o = (long long)p * d.S + d.idx(i, j, k);
  double e[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) e[q] = __ldg(g.f[CS_G_VERT] + q * PS + o);
  const double en = 1.0 / sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
#pragma unroll
  for (int q = 0; q < 3; ++q) e[q] = e[q] * en;
  const bool corner = (i == 0 || i == N) && (j == 0 || j == N);
  if (!corner) {
    if (mask_at(g, d, p, i, j) == 0 || mask_at(g, d, p, i + 1, j) == 0 || mask_at(g, d, p, i + 1, j + 1) == 0 ||
        mask_at(g, d, p, i, j + 1) == 0) {
      s.Ef[2][o] = 0.0;
      return;
    }
    double E = 0.0, n1[3], ta[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const R* z = s.E + q * PS + o;
      E = E + ((double)z[0] + (double)z[1] + (double)z[1 + dj] + (double)z[dj]) * 0.25 * e[q];
      const double* v = g.f[CS_G_VERT] + q * PS + o;
      n1[q] = __ldg(v + 1) - __ldg(v - 1);
      ta[q] = __ldg(v + dj) - __ldg(v - dj);
    }
    // cosine of the angle between the two families' normals, made orthogonal
    // to the edge
    const double ne = n1[0] * e[0] + n1[1] * e[1] + n1[2] * e[2], te = ta[0] * e[0] + ta[1] * e[1] + ta[2] * e[2];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      n1[q] = n1[q] - ne * e[q];
      ta[q] = ta[q] - te * e[q];
    }
    const double nn = n1[0] * n1[0] + n1[1] * n1[1] + n1[2] * n1[2], tt = ta[0] * ta[0] + ta[1] * ta[1] + ta[2] * ta[2];
    const double cos_t = (ta[0] * n1[0] + ta[1] * n1[1] + ta[2] * n1[2]) / sqrt(nn * tt);
    const double sp = fmax(llf_speed(s.S[1][o + dj], s.S[1][o], s.S[0][o + dj], s.S[0][o]),
                           llf_speed(s.S[3][o + 1], s.S[3][o], s.S[2][o + 1], s.S[2][o]));
    s.Ef[2][o] = llf_emf(sp, sqrt(1.0 - cos_t * cos_t), E, s.Bq[0][2 * PS + o + dj], s.Bq[0][PS + o], s.Bq[1][4 * PS + o + 1],
                         s.Bq[1][3 * PS + o]);
  } else {
    const int c = (i == 0 && j == 0) ? 0 : (i == N && j == 0) ? 1 : (i == N && j == N) ? 2 : 3;
    int z1x, z1y, z2x, z2y, z3x, z3y;
    if (c == 0) { z1x = i + 1; z1y = j + 1; z2x = i; z2y = j + 1; z3x = i + 1; z3y = j; }
    else if (c == 1) { z1x = i + 1; z1y = j + 1; z2x = i; z2y = j + 1; z3x = i; z3y = j; }
    else if (c == 2) { z1x = i; z1y = j + 1; z2x = i; z2y = j; z3x = i + 1; z3y = j; }
    else { z1x = i + 1; z1y = j + 1; z2x = i; z2y = j; z3x = i + 1; z3y = j; }
    const double ob3 = 1.0 / 3.0;
    const double Ex = (E1(s, d, 0, p, z1x, z1y, k) + E1(s, d, 0, p, z2x, z2y, k) + E1(s, d, 0, p, z3x, z3y, k)) * ob3;
    const double Ey = (E1(s, d, 1, p, z1x, z1y, k) + E1(s, d, 1, p, z2x, z2y, k) + E1(s, d, 1, p, z3x, z3y, k)) * ob3;
    const double Ez = (E1(s, d, 2, p, z1x, z1y, k) + E1(s, d, 2, p, z2x, z2y, k) + E1(s, d, 2, p, z3x, z3y, k)) * ob3;
    double Bn1, Bn2, Bn3, SR1, SL1, SR2, SL2, SR3, SL3;
    if (c == 0) {
      Bn1 = -Bqa(s, d, 1, 4, p, z3x, z3y, k); Bn2 = Bqa(s, d, 0, 2, p, z2x, z2y, k); Bn3 = Bqa(s, d, 1, 3, p, z2x, z2y - 1, k);
      SR1 = -Sg(s.S[2], d, p, z3x, z3y, k); SL1 = -Sg(s.S[3], d, p, z3x, z3y, k);
      SR2 = Sg(s.S[1], d, p, z2x, z2y, k); SL2 = Sg(s.S[0], d, p, z2x, z2y, k);
      SR3 = Sg(s.S[3], d, p, z2x, z2y - 1, k); SL3 = Sg(s.S[2], d, p, z2x, z2y - 1, k);
    } else if (c == 1) {
      Bn1 = -Bqa(s, d, 1, 4, p, z1x, z1y - 1, k); Bn2 = Bqa(s, d, 0, 2, p, z2x, z2y, k); Bn3 = Bqa(s, d, 1, 3, p, z3x, z3y, k);
      SR1 = -Sg(s.S[0], d, p, z3x, z3y, k); SL1 = -Sg(s.S[1], d, p, z3x, z3y, k);
      SR2 = Sg(s.S[1], d, p, z2x, z2y, k); SL2 = Sg(s.S[0], d, p, z2x, z2y, k);
      SR3 = Sg(s.S[3], d, p, z3x, z3y, k); SL3 = Sg(s.S[2], d, p, z3x, z3y, k);
    } else if (c == 2) {
      Bn1 = Bqa(s, d, 0, 2, p, z1x, z1y, k); Bn2 = Bqa(s, d, 1, 3, p, z2x, z2y, k); Bn3 = -Bqa(s, d, 0, 1, p, z2x, z2y, k);
      SR1 = Sg(s.S[1], d, p, z1x, z1y, k); SL1 = Sg(s.S[0], d, p, z1x, z1y, k);
      SR2 = Sg(s.S[3], d, p, z2x, z2y, k); SL2 = Sg(s.S[2], d, p, z2x, z2y, k);
      SR3 = -Sg(s.S[0], d, p, z2x, z2y, k); SL3 = -Sg(s.S[1], d, p, z2x, z2y, k);
    } else {
      Bn1 = -Bqa(s, d, 1, 4, p, z3x, z3y, k); Bn2 = Bqa(s, d, 1, 3, p, z2x, z2y, k); Bn3 = -Bqa(s, d, 0, 1, p, z2x, z2y, k);
      SR1 = -Sg(s.S[2], d, p, z3x, z3y, k); SL1 = -Sg(s.S[3], d, p, z3x, z3y, k);
      SR2 = Sg(s.S[3], d, p, z2x, z2y, k); SL2 = Sg(s.S[2], d, p, z2x, z2y, k);
      SR3 = -Sg(s.S[0], d, p, z2x, z2y, k); SL3 = -Sg(s.S[1], d, p, z2x, z2y, k);
    }
    const double tm = fmax(fmax(fmax(fabs(SR1), fabs(SL1)), fmax(fabs(SR2), fabs(SL2))), fmax(fabs(SR3), fabs(SL3)));
    // one direction along the edge, so the rule's three points agree
    s.Ef[2][o] = d_rs3(tm, -tm, tm, -tm, tm, -tm, Ex * e[0] + Ey * e[1] + Ez * e[2], Bn1, Bn2, Bn3);
  }
}

// The three edge directions in one launch: block T is tile T / 3 of
// direction T % 3.
//
// What bounds it: latency of about 30 loads an edge.  Solving the four-state
// problem in its general form at each of the rule's three points took 136
// registers and most of the time in FP64 divisions: 2.9 ms of a 6 x 128^2 x 64
// step against 1.2.
template <typename R>
__global__ void __launch_bounds__(TPB, 6) k_edges(Dims d, DGeom g, DStateT<R> s, Range3 r0, Range3 r1, Range3 r2) {
  const unsigned nb = (unsigned)((max(r0.count(), max(r1.count(), r2.count())) + TPB - 1) / TPB);
  for (unsigned T = blockIdx.x; T < 3 * nb; T += gridDim.x) {
    const int dir = T % 3;
    const Range3 r = dir == 0 ? r0 : (dir == 1 ? r1 : r2);
    const long long t = (long long)(T / 3) * TPB + threadIdx.x;
    if (t >= r.count()) continue;
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (dir == 0)
      edge_x(d, g, s, p, i, j, k);
    else if (dir == 1)
      edge_y(d, g, s, p, i, j, k);
    else
      edge_z(d, g, s, p, i, j, k);
  }
}

// Panel-edge ownership for the EMFs: a non-owner copy of a shared edge
// takes the owner's value, negated where the two panels run the edge in
// opposite directions.
template <typename R>
__global__ void k_sync_emf(DStateT<R> s, PanelSync ps) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < ps.ne; t += (long long)gridDim.x * blockDim.x)
    s.Ef[ps.e_df[t]][ps.e_dst[t]] = (double)ps.e_sign[t] * s.Ef[ps.e_sf[t]][ps.e_src[t]];
}

// The reference's rule for a shared edge (CS_FLAG_PANEL_AVERAGE): all
// copies take the average of the panels' EMFs, signed where a panel runs the
// edge the other way; two copies (own + other) * 0.5, the three of a
// cube-corner radial edge their sum / 3 (334fetch_buffers_fill_in_flux_x.f:
// 341-395, 335fetch_buffers_fill_in_flux_y.f:761-795).  One thread an edge:
// its owner's copy, then the one or two entries from e_cls[q].
template <typename R>
__global__ void k_avg_emf(DStateT<R> s, PanelSync ps) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < ps.ncls; q += (long long)gridDim.x * blockDim.x) {
    const int h = ps.e_cls[q], n = ps.e_cls[q + 1] - h;
    double* own = s.Ef[ps.e_sf[h]] + ps.e_src[h];
    double sum = *own;
    for (int m = h; m < h + n; ++m) sum += (double)ps.e_sign[m] * s.Ef[ps.e_df[m]][ps.e_dst[m]];
    const double avg = n == 1 ? sum * 0.5 : sum / 3.0;
    *own = avg;
    for (int m = h; m < h + n; ++m) s.Ef[ps.e_df[m]][ps.e_dst[m]] = (double)ps.e_sign[m] * avg;
  }
}

}  // namespace

template <typename R>
void launch_edges_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  const int N = d.N, nr = d.nr;
  Range3 ex = {1, N, 0, N, 0, nr};
  Range3 ey = {0, N, 1, N, 0, nr};
  Range3 ez = {0, N, 0, N, 1, nr};
  const long long nb = 3 * ((std::max(ex.count(), std::max(ey.count(), ez.count())) + TPB - 1) / TPB);
  k_edges<R><<<(int)std::min<long long>(nb, (long long)grid_sms(sv) * 64), TPB, 0, sv.stream>>>(d, sv.g, st, ex, ey, ez);
  mark(sv, "k_edges");
  if (sv.psync.ncls > 0 && (sv.p.flags & CS_FLAG_PANEL_AVERAGE)) {
    k_avg_emf<R><<<blocks_for(sv.psync.ncls, 128, grid_sms(sv)), 128, 0, sv.stream>>>(st, sv.psync);
    mark(sv, "k_avg_emf");
  } else if (sv.psync.ne > 0) {
    k_sync_emf<R><<<blocks_for(sv.psync.ne, 128, grid_sms(sv)), 128, 0, sv.stream>>>(st, sv.psync);
    mark(sv, "k_sync_emf");
  }
}

void launch_edges(Solve& sv) {
  if (sv.fp32)
    launch_edges_t(sv, sv.stF);
  else
    launch_edges_t(sv, sv.st);
}

}  // namespace cs

// Known-answer access to the multidimensional Riemann solvers, one thread a
// case: the three-state solver and the four-state one's closed form, which
// k_edges calls, and the four-state solver in general, which it does not.
namespace {
__global__ void k_twod_rs_ez(int n, int kind, const double* in, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  if (kind == 4) {
    const double* a = in + (long long)t * 11;
    out[t] = cs::d_rs4(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10]);
  } else if (kind == 5) {
    const double* a = in + (long long)t * 7;
    out[t] = cs::llf_emf(a[0], a[1], a[2], a[3], a[4], a[5], a[6]);
  } else {
    const double* a = in + (long long)t * 10;
    out[t] = cs::d_rs3(a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9]);
  }
}
}  // namespace

extern "C" int cs_twod_rs_ez(int32_t kind, int32_t n, const double* in, double* out) {
  if (kind < 3 || kind > 5 || n < 0 || (n > 0 && (!in || !out))) return CS_ERR_ARG;
  if (n == 0) return CS_OK;
  const size_t nin = (size_t)n * (kind == 4 ? 11 : (kind == 5 ? 7 : 10));
  double *din = nullptr, *dout = nullptr;
  if (cudaMalloc(&din, nin * sizeof(double)) != cudaSuccess) return CS_ERR_CUDA;
  if (cudaMalloc(&dout, (size_t)n * sizeof(double)) != cudaSuccess) {
    cudaFree(din);
    return CS_ERR_CUDA;
  }
  cudaError_t e = cudaMemcpy(din, in, nin * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_twod_rs_ez<<<(n + 127) / 128, 128>>>(n, kind, din, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(din);
  cudaFree(dout);
  return e == cudaSuccess ? CS_OK : CS_ERR_CUDA;
}
