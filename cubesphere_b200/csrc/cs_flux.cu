// Face fluxes of the stage: five-point quadrature per face, rotation to
// the face frame, HLL solve, rotation back, and the race-free gather of
// the per-face contributions into the zone time derivative; plus the
// explicit point-mass gravity source.
//
// Follows MAKE_FACIAL_FLUXES (pkg/inc/cubesphere/400riemann_integrate/
// 450make_facial_fluxes.f:405-2933), OneD_RS_MHD_Ptwise
// (600riemann_1d/610_1d_rs_oned_rs_mhd_ptwise.f) and
// BUILD_NON_STIFF_SOURCES (470build_non_stiff_sources.f:147-244).
// The reference scatters each face into both neighbours inside one
// parallel loop; here each face writes its two one-sided contributions and
// each zone sums its own six faces in a fixed order.
#include <algorithm>

#include "cs_solve.h"

namespace cs {

namespace {

constexpr int TPB = 128;

// A block takes 32 faces with five warps, in three phases.  Basis: warp q
// forms, for both sides, the nine centred monomials of quadrature point q in
// the side zone's scaled coordinates.  Face states (450:545-2931): the 18
// (side, primitive or entropy) polynomials of each face at the five points,
// four primitives of a side a warp, so that a mode is read once and a basis
// value once for four primitives; the fifth warp takes the entropies, the frame
// of the x- and y-faces and the two area / volume ratios, once
// a face.  Fluxes: one quadrature point per thread (warp = point) rotates the
// two states to the face frame, solves the HLL problem and rotates the
// contributions back; they meet in shared memory and are summed in point
// order (the order of the reference's quadrature loop).  No face state goes
// through HBM.  One launch covers the three face directions: tile T is tile
// T / 3 of direction T % 3, so the x, y and z faces of about the same zone
// rows run side by side and L2 serves a zone's modes to all three.
//
// What bounds it: L1 (73 % busy, mostly shared-memory words) and FP64 latency
// at the 20 warps its registers and shared memory allow.  ms of a 6 x 128^2 x
// 64 step, FP64 / FP32: 29.5 / 19.8 with every thread forming its point's basis
// per variable, 22.3 / 14.6 with the basis kept and two primitives a warp at a
// time, 21.3 / 14.1 with four, 20.7 / 13.1 with the tiles in order (tile_blocks),
// 21.7 / 13.3 since it forms the second radial faces beyond the ends too.
constexpr int FLUX_FACES = 32;
// Registers / occupancy: 4 blocks per SM suit the FP64 instantiation, 7 the
// FP32 one (measured on the 6 x 128^2 x 64 shell).
template <typename R>
__global__ void __launch_bounds__(FLUX_FACES * 5, sizeof(R) == 4 ? 7 : 4) k_flux(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r0, Range3 r1, Range3 r2) {
  // the basis is dead once the face states are formed, so it shares its space
  // with the flux contributions
  union Scratch {
    R red[5][16][FLUX_FACES];
    R bs[2][5][9][FLUX_FACES];  // [side][point][x y z xx yy zz xy yz xz][face]
  };
  __shared__ Scratch sc;
  __shared__ R fs[2][9][5][FLUX_FACES];  // [side][primitive 0-7, entropy][point][face]
  __shared__ R fr[9][FLUX_FACES];        // frame of an x- or y-face: A, B, C
  __shared__ R av[2][FLUX_FACES];        // area / volume of each side
  const int lane = threadIdx.x % FLUX_FACES, jq = threadIdx.x / FLUX_FACES;
  const long long PS = (long long)NPANEL * d.S;
  const unsigned nt0 = (unsigned)((r0.count() + FLUX_FACES - 1) / FLUX_FACES),
                 nt1 = (unsigned)((r1.count() + FLUX_FACES - 1) / FLUX_FACES),
                 nt2 = (unsigned)((r2.count() + FLUX_FACES - 1) / FLUX_FACES);
  const unsigned ntile = 3 * max(nt0, max(nt1, nt2));
  for (unsigned T = blockIdx.x; T < ntile; T += gridDim.x) {
    const int dir = T % 3;
    const unsigned tile = T / 3;
    const Range3 r = dir == 0 ? r0 : (dir == 1 ? r1 : r2);
    if (tile >= (dir == 0 ? nt0 : (dir == 1 ? nt1 : nt2))) continue;  // uniform over the block
    const double* qp = dir == 0 ? g.f[CS_G_XF_QP] : (dir == 1 ? g.f[CS_G_YF_QP] : g.f[CS_G_ZF_QP]);
    const double* qw = dir == 0 ? g.f[CS_G_XF_QW] : (dir == 1 ? g.f[CS_G_YF_QW] : g.f[CS_G_ZF_QW]);
    const double* ar = dir == 0 ? g.f[CS_G_XF_AREA] : (dir == 1 ? g.f[CS_G_YF_AREA] : g.f[CS_G_ZF_AREA]);
    R* F = dir == 0 ? s.fcon[0] : (dir == 1 ? s.fcon[1] : s.fcon[2]);
    const unsigned t = tile * FLUX_FACES + lane;
    const bool valid = t < (unsigned)r.count();
    int p = 0, i = 0, j = 0, k = 0;
    if (valid) r.decode(t, p, i, j, k);
    const long long o = (long long)p * d.S + d.idx(i, j, k);
    // the two side zones; one remapped through istencil at a panel corner
    long long zo0 = o, zo1 = o;
    bool skip = !valid;
    if (valid) {
      int lx = i, ly = j, rx = i, ry = j, rz = k;
      if (dir == 2) {
        if (mask_at(g, d, p, i, j) == 0) skip = true;
        rz = k + 1;
      } else {
        const int w = 2 * dir;  // istencil entry of the upper neighbour, w + 1 of the lower
        rx += dir == 0;
        ry += dir == 1;
        const int mL = mask_at(g, d, p, i, j), mR = mask_at(g, d, p, rx, ry);
        if (mL == 0 && mR == 1) {
          lx = sten(g, d, p, rx, ry, w + 1, 0);
          ly = sten(g, d, p, rx, ry, w + 1, 1);
        } else if (mL == 1 && mR == 0) {
          rx = sten(g, d, p, lx, ly, w, 0);
          ry = sten(g, d, p, lx, ly, w, 1);
        } else if (mL == 0 && mR == 0) {
          skip = true;
        }
      }
      zo0 = (long long)p * d.S + d.idx(lx, ly, k);
      zo1 = (long long)p * d.S + d.idx(rx, ry, rz);
    }
    if (!skip) {
      const R qx = (R)__ldg(qp + jq * PS + o), qy = (R)__ldg(qp + (5 + jq) * PS + o), qz = (R)__ldg(qp + (10 + jq) * PS + o);
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const long long z = side ? zo1 : zo0;
        const double* cen = g.f[CS_G_V_CEN] + z;
        const double* cf = g.f[CS_G_COEF] + z;
        const R obl = rcp_newton(fmax((R)__ldg(g.f[CS_G_V_SCALE] + z), R(ph.smallnum)));
        const R x = (qx - (R)__ldg(cen)) * obl, y = (qy - (R)__ldg(cen + PS)) * obl, zz = (qz - (R)__ldg(cen + 2 * PS)) * obl;
        R(&b)[9][FLUX_FACES] = sc.bs[side][jq];
        b[0][lane] = x;
        b[1][lane] = y;
        b[2][lane] = zz;
        b[3][lane] = x * x - (R)__ldg(cf + 4 * PS);
        b[4][lane] = y * y - (R)__ldg(cf + 5 * PS);
        b[5][lane] = zz * zz - (R)__ldg(cf + 6 * PS);
        b[6][lane] = x * y - (R)__ldg(cf + 7 * PS);
        b[7][lane] = y * zz - (R)__ldg(cf + 8 * PS);
        b[8][lane] = x * zz - (R)__ldg(cf + 9 * PS);
      }
    }
    __syncthreads();
    if (!skip) {
      if (jq < 4) {  // primitives 4 (jq & 1) .. + 3 of side jq >> 1
        const int side = jq >> 1, c = 4 * (jq & 1);
        const R* v = s.V + c * PS + (side ? zo1 : zo0);
        R u[5][4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const R m = v[n * PS];
#pragma unroll
          for (int q = 0; q < 5; ++q) u[q][n] = m;
        }
#pragma unroll
        for (int a = 1; a < 10; ++a) {
          R m[4];
#pragma unroll
          for (int n = 0; n < 4; ++n) m[n] = v[(a * NVAR + n) * PS];
#pragma unroll
          for (int q = 0; q < 5; ++q) {
            const R bv = sc.bs[side][q][a - 1][lane];
#pragma unroll
            for (int n = 0; n < 4; ++n) u[q][n] = u[q][n] + m[n] * bv;
          }
        }
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
          for (int n = 0; n < 4; ++n) fs[side][c + n][q][lane] = u[q][n];
      } else {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const R* e = s.ent + (side ? zo1 : zo0);
          const R e0 = e[0], e1 = e[PS], e2 = e[2 * PS], e3 = e[3 * PS];
#pragma unroll
          for (int q = 0; q < 5; ++q) {
            const R(&b)[9][FLUX_FACES] = sc.bs[side][q];
            fs[side][8][q][lane] = e0 + e1 * b[0][lane] + e2 * b[1][lane] + e3 * b[2][lane];
          }
        }
        const R area = (R)__ldg(ar + o);
        av[0][lane] = area * rcp_newton((R)__ldg(g.f[CS_G_V_VOL] + zo0));
        av[1][lane] = area * rcp_newton((R)__ldg(g.f[CS_G_V_VOL] + zo1));
        if (dir < 2) {
          const double* nv = (dir == 0 ? g.f[CS_G_XF_N] : g.f[CS_G_YF_N]) + o;
          const double* fc = (dir == 0 ? g.f[CS_G_XF_CEN] : g.f[CS_G_YF_CEN]) + o;
          const R Ax = (R)__ldg(nv), Ay = (R)__ldg(nv + PS), Az = (R)__ldg(nv + 2 * PS);
          R ex = (R)__ldg(fc), ey = (R)__ldg(fc + PS), ez = (R)__ldg(fc + 2 * PS);
          const R tt = rcp_newton(fmax(sqrt(ex * ex + ey * ey + ez * ez), R(ph.smallnum)));
          ex = ex * tt;
          ey = ey * tt;
          ez = ez * tt;
          // the radial direction and its product with the normal: C and
          // B = C x A on x-faces; B and C = A x B on y-faces
          const R sx = ey * Az - ez * Ay, sy = ez * Ax - ex * Az, sz = ex * Ay - ey * Ax;
          const bool xf = dir == 0;
          fr[0][lane] = Ax;
          fr[1][lane] = Ay;
          fr[2][lane] = Az;
          fr[3][lane] = xf ? sx : ex;
          fr[4][lane] = xf ? sy : ey;
          fr[5][lane] = xf ? sz : ez;
          fr[6][lane] = xf ? ex : -sx;
          fr[7][lane] = xf ? ey : -sy;
          fr[8][lane] = xf ? ez : -sz;
        }
      }
    }
    __syncthreads();
    // the flux at point jq of face lane
    if (skip) {
#pragma unroll
      for (int c = 0; c < 16; ++c) sc.red[jq][c][lane] = R(0.0);
    } else {
      R Ax, Ay, Az, Bx, By, Bz, Cx, Cy, Cz;
      if (dir < 2) {
        Ax = fr[0][lane];
        Ay = fr[1][lane];
        Az = fr[2][lane];
        Bx = fr[3][lane];
        By = fr[4][lane];
        Bz = fr[5][lane];
        Cx = fr[6][lane];
        Cy = fr[7][lane];
        Cz = fr[8][lane];
      } else {
        const double* nv = g.f[CS_G_ZF_N] + o;
        const double* vt = g.f[CS_G_VERT] + o;
        const int dj = d.NI;
        Ax = (R)__ldg(nv + jq * PS);
        Ay = (R)__ldg(nv + (5 + jq) * PS);
        Az = (R)__ldg(nv + (10 + jq) * PS);
        R tt = rcp_newton(fmax(sqrt(Ax * Ax + Ay * Ay + Az * Az), R(ph.smallnum)));
        Ax = Ax * tt;
        Ay = Ay * tt;
        Az = Az * tt;
        auto across = [&](const double* v) {
          return (R)__ldg(v) + (R)__ldg(v - dj) - (R)__ldg(v - 1) - (R)__ldg(v - 1 - dj);
        };
        Bx = across(vt);
        By = across(vt + PS);
        Bz = across(vt + 2 * PS);
        tt = Bx * Ax + By * Ay + Bz * Az;
        Bx = Bx - tt * Ax;
        By = By - tt * Ay;
        Bz = Bz - tt * Az;
        tt = rcp_newton(fmax(sqrt(Bx * Bx + By * By + Bz * Bz), R(ph.smallnum)));
        Bx = Bx * tt;
        By = By * tt;
        Bz = Bz * tt;
        Cx = Ay * Bz - Az * By;
        Cy = Az * Bx - Ax * Bz;
        Cz = Ax * By - Ay * Bx;
        tt = rcp_newton(fmax(sqrt(Cx * Cx + Cy * Cy + Cz * Cz), R(ph.smallnum)));
        Cx = Cx * tt;
        Cy = Cy * tt;
        Cz = Cz * tt;
      }
      R V[2][8];
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        V[side][0] = fs[side][0][jq][lane];
        V[side][4] = fs[side][4][jq][lane];
#pragma unroll
        for (int u = 1; u <= 5; u += 4) {
          const R w0 = fs[side][u][jq][lane], w1 = fs[side][u + 1][jq][lane], w2 = fs[side][u + 2][jq][lane];
          V[side][u] = Ax * w0 + Ay * w1 + Az * w2;
          V[side][u + 1] = Bx * w0 + By * w1 + Bz * w2;
          V[side][u + 2] = Cx * w0 + Cy * w1 + Cz * w2;
        }
      }
      R FlL[8], FlR[8], FL[8], FR[8], SL, SR, entF;
      d_hll(ph, V[0], V[1], fs[0][8][jq][lane], fs[1][8][jq][lane], FlL, FlR, FL, FR, SL, SR, entF);
      if (jq == 0) {
        (dir == 0 ? s.S[0] : (dir == 1 ? s.S[2] : s.S[4]))[o] = SL;
        (dir == 0 ? s.S[1] : (dir == 1 ? s.S[3] : s.S[5]))[o] = SR;
        (dir == 0 ? s.EF[0] : (dir == 1 ? s.EF[1] : s.EF[2]))[o] = entF;
      }
      const R wt = (R)__ldg(qw + jq * PS + o);
      // the two sides' net contributions (fluctuation + flux) summed in the
      // face frame and rotated back once, and area / volume once per side
      // (the reference rotates each term and divides every term; the
      // results differ from it in the last bits only)
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        FlL[c] = FlL[c] + FL[c];
        FlR[c] = FlR[c] - FR[c];
      }
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const R* G = side ? FlR : FlL;
        const R a = av[side][lane];
        R(*out)[FLUX_FACES] = sc.red[jq] + 8 * side;
        out[0][lane] = wt * G[0] * a;
        out[4][lane] = wt * G[4] * a;
#pragma unroll
        for (int u = 1; u <= 5; u += 4) {
          out[u][lane] = wt * (Ax * G[u] + Bx * G[u + 1] + Cx * G[u + 2]) * a;
          out[u + 1][lane] = wt * (Ay * G[u] + By * G[u + 1] + Cy * G[u + 2]) * a;
          out[u + 2][lane] = wt * (Az * G[u] + Bz * G[u + 1] + Cz * G[u + 2]) * a;
        }
      }
    }
    __syncthreads();
    if (valid) {
      for (int c = jq; c < 16; c += 5) {
        R acc = R(0.0);
#pragma unroll
        for (int q = 0; q < 5; ++q) acc = acc + sc.red[q][c][lane];
        F[c * PS + o] = acc;
      }
    }
    __syncthreads();
  }
}

// Panel-edge ownership for the face fluxes: a non-owner copy of a shared
// face takes the owner's two one-sided contributions with the sides
// exchanged (their normals are opposite) and the negated entropy flux.
template <typename R>
__global__ void k_sync_flux(Dims d, DStateT<R> s, PanelSync ps) {
  const unsigned n = (unsigned)ps.nf;
  const long long PS = (long long)NPANEL * d.S;
  // one thread an entry and value: 16 contributions, then the entropy flux
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < 17 * n; t += gridDim.x * blockDim.x) {
    const unsigned c = t / n, e = t - c * n;
    const unsigned dst = ps.f_dst[e], src = ps.f_src[e];
    const int dd = ps.f_ddir[e], sd = ps.f_sdir[e];
    R* Fd = dd == 0 ? s.fcon[0] : s.fcon[1];  // panel edges have x- and y-faces only
    const R* Fs = sd == 0 ? s.fcon[0] : s.fcon[1];
    if (c < 16)
      Fd[c * PS + dst] = Fs[(c ^ 8) * PS + src];
    else
      (dd == 0 ? s.EF[0] : s.EF[1])[dst] = -(sd == 0 ? s.EF[0] : s.EF[1])[src];
  }
}

// The reference's rule for a shared face (CS_FLAG_PANEL_AVERAGE): both
// copies take the average of the two panels' one-sided contributions (the
// sides exchanged between them) and of their entropy fluxes (negated), as
// its defect correction does (FETCH_BUFFERS_FILL_IN_FLUX_X / _Y,
// 334fetch_buffers_fill_in_flux_x.f:295-309).  Each face is in one entry.
template <typename R>
__global__ void k_avg_flux(Dims d, DStateT<R> s, PanelSync ps) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < ps.nf; t += (long long)gridDim.x * blockDim.x) {
    const long long dst = ps.f_dst[t], src = ps.f_src[t];
    const int dd = ps.f_ddir[t], sd = ps.f_sdir[t];
    const int dp = (int)(dst / d.S), sp = (int)(src / d.S);
    const long long dof = dst % d.S, sof = src % d.S;
    R* Fd = s.fcon[dd];
    R* Fs = s.fcon[sd];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      R& dl = Fd[((long long)c * NPANEL + dp) * d.S + dof];
      R& dr = Fd[((long long)(8 + c) * NPANEL + dp) * d.S + dof];
      R& sl = Fs[((long long)c * NPANEL + sp) * d.S + sof];
      R& sr = Fs[((long long)(8 + c) * NPANEL + sp) * d.S + sof];
      const R a = (dl + sr) * R(0.5), b = (dr + sl) * R(0.5);
      dl = a;
      sr = a;
      dr = b;
      sl = b;
    }
    const R e = (s.EF[dd][dst] - s.EF[sd][src]) * R(0.5);
    s.EF[dd][dst] = e;
    s.EF[sd][src] = -e;
  }
}

// dU/dt of each zone from its six faces (x, then y, then z; lower face,
// upper face).  The fluxes end with the radial face at the far side of the
// first ghost (face -1 and face nr + 1), so the second ghost has that one face
// only, as in the reference, which adds each face to both its zones.
template <typename R>
__global__ void k_gather(Dims d, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    R acc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = R(0.0);
    if (mask_at(g, d, p, i, j) == 1) {
      const long long PS = (long long)NPANEL * d.S, o = (long long)p * d.S + d.idx(i, j, k);
      const int dk = d.NI * d.NJ;
      if (k >= 0 && k <= d.nr + 1) {
#pragma unroll
        for (int dir = 0; dir < 3; ++dir) {
          const R *Fl = s.fcon[dir] + o, *Fr = Fl + 8 * PS - (dir == 0 ? 1 : (dir == 1 ? d.NI : dk));
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            acc[c] = acc[c] - Fr[c * PS];
            acc[c] = acc[c] - Fl[c * PS];
          }
        }
      } else {  // a second ghost: its face toward the interior
        const R* F = s.fcon[2] + o + (k < 0 ? 0 : 8 * PS - dk);
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = acc[c] - F[c * PS];
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) s.dUdt[d.at(c, p, i, j, k)] = acc[c];
  }
}

// Point-mass gravity (470:147-244).
template <typename R>
__global__ void k_sources(Dims d, PhysC ph, DGeom g, DStateT<R> s, Range3 r) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < r.count(); t += (long long)gridDim.x * blockDim.x) {
    int p, i, j, k;
    r.decode(t, p, i, j, k);
    if (mask_at(g, d, p, i, j) != 1) continue;
    const R x = geoR<R>(g, d, CS_G_V_CEN, 0, p, i, j, k), y = geoR<R>(g, d, CS_G_V_CEN, 1, p, i, j, k),
                 z = geoR<R>(g, d, CS_G_V_CEN, 2, p, i, j, k);
    const R rho = s.V[d.at(0, p, i, j, k)], vx = s.V[d.at(1, p, i, j, k)], vy = s.V[d.at(2, p, i, j, k)],
                 vz = s.V[d.at(3, p, i, j, k)];
    const R rad = sqrt(x * x + y * y + z * z);
    const R gmb = R(ph.gm) * (R(1.0) / (rad * rad * rad));
    const R S2 = -(gmb * x * rho), S3 = -(gmb * y * rho), S4 = -(gmb * z * rho);
    const R S5 = vx * S2 + vy * S3 + vz * S4;
    s.dUdt[d.at(1, p, i, j, k)] += S2;
    s.dUdt[d.at(2, p, i, j, k)] += S3;
    s.dUdt[d.at(3, p, i, j, k)] += S4;
    s.dUdt[d.at(4, p, i, j, k)] += S5;
  }
}

}  // namespace

template <typename R>
void launch_fluxes_t(Solve& sv, DStateT<R>& st) {
  const Dims& d = sv.d;
  const int N = d.N, nr = d.nr;
  // the faces of the zones to gather, and the layer across the interior's whose
  // speeds and fluxes its edges read
  const Range3 z = own_columns(d, 2);
  Range3 fx = {0, N, 0, N + 1, 0, nr + 1};
  Range3 fy = {0, N + 1, 0, N, 0, nr + 1};
  Range3 fz = {0, N + 1, 0, N + 1, -1, nr + 1};
  {
    const long long nt = 3 * ((std::max(fx.count(), std::max(fy.count(), fz.count())) + FLUX_FACES - 1) / FLUX_FACES);
    k_flux<R><<<tile_blocks(sv, nt, 32), FLUX_FACES * 5, 0, sv.stream>>>(d, sv.ph, sv.g, st, fx, fy, fz);
    mark(sv, "k_flux");
  }
  if (sv.psync.nf > 0 && (sv.p.flags & CS_FLAG_PANEL_AVERAGE)) {
    k_avg_flux<R><<<blocks_for(sv.psync.nf, 128, grid_sms(sv)), 128, 0, sv.stream>>>(d, st, sv.psync);
    mark(sv, "k_avg_flux");
  } else if (sv.psync.nf > 0) {
    k_sync_flux<R><<<blocks_for(17 * sv.psync.nf, 128, grid_sms(sv)), 128, 0, sv.stream>>>(d, st, sv.psync);
    mark(sv, "k_sync_flux");
  }
  k_gather<R><<<blocks_for(z.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.g, st, z);
  mark(sv, "k_gather");
}

void launch_fluxes(Solve& sv) {
  if (sv.fp32)
    launch_fluxes_t(sv, sv.stF);
  else
    launch_fluxes_t(sv, sv.st);
}

template <typename R>
void launch_sources_t(Solve& sv, DStateT<R>& st) {
  if (!(sv.ph.gm > sv.p.smallnum)) return;
  const Dims& d = sv.d;
  const Range3 z = own_columns(d, 1);
  k_sources<R><<<blocks_for(z.count(), TPB, grid_sms(sv)), TPB, 0, sv.stream>>>(d, sv.ph, sv.g, st, z);
  mark(sv, "k_sources");
}

void launch_sources(Solve& sv) {
  if (sv.fp32)
    launch_sources_t(sv, sv.stF);
  else
    launch_sources_t(sv, sv.st);
}

}  // namespace cs
