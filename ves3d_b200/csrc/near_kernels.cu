// Near-singular correction of the velocity at off-surface targets (FP64): the
// interpolation scheme of NearSingular<Real_t>::operator() (src/NearSingular.cc:1356-1555)
// as StokesVelocity<Real>::operator() composes it for SetTrgCoord targets
// (src/StokesVelocity.cc:475-500).
//
//   every target: the smooth quadrature of every vesicle at the far upsampling order
//   p_up (the reference's far field over its upsampled sources, :476-489);
//   a target closer than r_near = r_ves 2 / sqrt(p_up) to a vesicle (r_ves the largest
//   distance of a surface point from its vesicle's centroid, src/NearSingular.cc:119-160):
//   that vesicle's smooth contribution (SubtractDirect, :1144-1212) is replaced by the
//   Lagrange interpolation (InterPoints / InterPoly, :1356-1374) of 8 values along the line
//   from the target's projection P on the surface through the target: at x = 0 the
//   vesicle's own singular-quadrature velocity at P (plus, with a double layer, g(P)/2
//   outside and -g(P)/2 inside: the jump, :1474-1481), at x_l = 1 + (l - 1)/6, l = 1..7,
//   the smooth quadrature at P + r_near x_l d; evaluated at x = |T - P| / r_near.
//
// The reference finds near pairs with a pvfmm octree and projects on quadratic patches of
// 3 x 3 grid points; here a target's near vesicles come from a bounding-sphere test and
// its distance to the vesicle's upsampled points (up to kNearMax per target, ascending
// vesicle order), and the projection is Gauss-Newton on the spherical-harmonic surface
// itself from the nearest upsampled point: a warp or half a warp per (target, vesicle) pair, lane
// m carrying the order-m Legendre recurrence. The on-surface velocity and density at P come
// from their coefficients the same way. Each pair's correction is written to its own slot
// and the slots are added in order (deterministic).
#include <cmath>
#include <vector>

#include "common.cuh"
#include "kernels.h"

namespace ves3d {

namespace {

constexpr int kInterpDeg = 8;
constexpr double kSqrt2Pi = 2.5066282746310002;
constexpr double kStepDone = 1e-15;  // a Gauss-Newton step (radians) below the rounding of the angles

__device__ __forceinline__ double inter_point(int i) { return i ? 1.0 + (i - 1.0) / (kInterpDeg - 2) : 0.0; }

__device__ double inter_poly(double x, int j) {
  double y = 1.0;
  const double x0 = inter_point(j);
  for (int k = 0; k < kInterpDeg; k++)
    if (k != j) y *= (x - inter_point(k)) / (x0 - inter_point(k));
  return y;
}

// Per vesicle: centroid of its order-p points, the largest distance of a point from it
// (cen_r[v] = (cx, cy, cz, R)), and the global maximum R as an ordered integer.
__global__ void k_centroid_radius(const double* __restrict__ X, int ng, double* __restrict__ cen_r,
                                  unsigned long long* __restrict__ rmax_bits) {
  __shared__ double red[3][256];
  const long v = blockIdx.x;
  const double* x = X + v * 3 * ng;
  double s[3] = {0, 0, 0};
  for (int i = threadIdx.x; i < ng; i += blockDim.x)
    for (int d = 0; d < 3; d++) s[d] += x[d * ng + i];
  for (int d = 0; d < 3; d++) red[d][threadIdx.x] = s[d];
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h)
      for (int d = 0; d < 3; d++) red[d][threadIdx.x] += red[d][threadIdx.x + h];
    __syncthreads();
  }
  const double c0 = red[0][0] / ng, c1 = red[1][0] / ng, c2 = red[2][0] / ng;
  __syncthreads();
  double m = 0.0;
  for (int i = threadIdx.x; i < ng; i += blockDim.x) {
    const double dx = x[i] - c0, dy = x[ng + i] - c1, dz = x[2 * ng + i] - c2;
    m = fmax(m, dx * dx + dy * dy + dz * dz);
  }
  red[0][threadIdx.x] = m;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) red[0][threadIdx.x] = fmax(red[0][threadIdx.x], red[0][threadIdx.x + h]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double R = sqrt(red[0][0]);
    cen_r[4 * v] = c0;
    cen_r[4 * v + 1] = c1;
    cen_r[4 * v + 2] = c2;
    cen_r[4 * v + 3] = R;
    atomicMax(rmax_bits, (unsigned long long)__double_as_longlong(R));  // R >= 0: bits order as values
  }
}

// r_near = r_ves 2 / sqrt(p_up), r_ves from the bits of the largest vesicle radius
__device__ __forceinline__ double near_radius(const unsigned long long* rmax_bits, int p_up) {
  return __longlong_as_double((long long)rmax_bits[0]) * 2.0 / sqrt((double)p_up);
}

// Near vesicles of each target: up to kNearMax in ascending vesicle order, with the index
// of the nearest upsampled point; count[t] = their number, or kNearMax + 1 when more (the first
// such target goes to *over). One warp per target: its lanes test 32 vesicles' spheres at a time
// and share the points of those in reach (a thread per target left 27 vesicles' tests and 1,200
// points per near vesicle to one lane: 1.34 ms for 20,000 targets, now 44 us).
__global__ void __launch_bounds__(128) k_near_find(const double* __restrict__ trg, long M,
                                                   const double* __restrict__ cen_r, long nv,
                                                   const double* __restrict__ pos_up, int p_up,
                                                   const unsigned long long* __restrict__ rmax_bits,
                                                   unsigned long long* __restrict__ over, int* __restrict__ count,
                                                   int* __restrict__ near_v, int* __restrict__ near_k) {
  const int lane = threadIdx.x & 31;
  const long t = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= M) return;
  const int ng1 = 2 * p_up * (p_up + 1);
  const double r_near = near_radius(rmax_bits, p_up);
  const double tx = trg[3 * t], ty = trg[3 * t + 1], tz = trg[3 * t + 2];
  int cnt = 0;
  for (long v0 = 0; v0 < nv; v0 += 32) {
    bool reach = false;
    if (v0 + lane < nv) {
      const double* c = cen_r + 4 * (v0 + lane);
      const double dx = tx - c[0], dy = ty - c[1], dz = tz - c[2];
      // upsampled points lie within about R of the centroid; a generous bound
      const double r = 1.25 * c[3] + r_near;
      reach = !(dx * dx + dy * dy + dz * dz > r * r);
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, reach); todo; todo &= todo - 1) {
      const long v = v0 + __ffs(todo) - 1;
      const double* P = pos_up + 3 * v * (long)ng1;
      double best = r_near * r_near;
      int kb = ng1;
      for (int k = lane; k < ng1; k += 32) {
        const double ex = P[3 * k] - tx, ey = P[3 * k + 1] - ty, ez = P[3 * k + 2] - tz;
        const double d2 = ex * ex + ey * ey + ez * ez;
        if (d2 < best) {
          best = d2;
          kb = k;
        }
      }
      // the nearest point, the first of equally near ones
      for (int o = 16; o > 0; o >>= 1) {
        const double d2 = __shfl_xor_sync(0xffffffffu, best, o);
        const int k = __shfl_xor_sync(0xffffffffu, kb, o);
        if (k < ng1 && (kb == ng1 || d2 < best || (d2 == best && k < kb))) {
          best = d2;
          kb = k;
        }
      }
      if (kb == ng1) continue;
      if (lane == 0 && cnt < kNearMax) {
        near_v[t * kNearMax + cnt] = (int)v;
        near_k[t * kNearMax + cnt] = kb;
      }
      cnt++;
    }
  }
  if (lane) return;
  count[t] = cnt <= kNearMax ? cnt : kNearMax + 1;
  if (cnt > kNearMax) atomicMin(over, (unsigned long long)t);
}

// Recurrence tables of the normalised associated Legendre functions (near_tables): rows n = 0..p
// of [3][32] (order m): a and b of P(m, n) = x a P(m, n - 1) - b P(m, n - 2), and c of the
// derivative's P(m + 1, n) term; then [32] factors of P(m, m) = -P(m - 1, m - 1) s diag.
__host__ __device__ constexpr int near_table_doubles(int p) { return 96 * (p + 1) + 32; }

// Value, d/dtheta and d/dphi of the 3 functions S[3][nc] at (x = cos theta, phi), summed over the
// G lanes of a group (all its lanes get them): lane m < p + 1 runs the recurrence of order m and
// the order-m blocks (the reference's LegPoly / LegPolyDeriv, src/SphericalHarmonics.cc:889-950;
// P(m + 1, n) for the derivative comes from lane m + 1).
// Where a target lies near the surface's centres of curvature the Gauss-Newton steps do not
// settle, and forty of them amplify a rounding to 1e-6 of the velocity and more: the order of the
// operations here is part of the result. (Sums of each block before its cosine, and a multiplication
// by 1 / s alone, took 0.23 ms less for 15,000 pairs at p = 12, and moved such targets.)
template <int G>
__device__ __forceinline__ void sh_point(const double* __restrict__ S, const double* __restrict__ tab, int p,
                                         const int* __restrict__ blk_off, double x, double phi, bool grads,
                                         double* val) {
  const int m = threadIdx.x & (G - 1);
  const int nc = p * (p + 2);
  const double s = sqrt(fmax(1.0 - x * x, 0.0)), si = s > 0.0 ? 1.0 / s : 0.0;
  const bool act = m <= p;
  double pmm = 0.28209479177387814;  // 1/sqrt(4 pi)
  for (int i = 1; i <= p; i++) {
    const double rt = tab[96 * (p + 1) + i];
    if (i <= m) pmm = -pmm * s * rt;
  }
  double cm = 1.0, sm = 0.0, dcm = 0.0, dsm = 0.0;
  if (act) {
    sincos(m * phi, &sm, &cm);
    dcm = -m * sm;
    dsm = m * cm;
  }
  const int jc = m == 0 ? 0 : (m == p ? 2 * p - 1 : 2 * m - 1);  // cos block of order m
  const bool sine = m >= 1 && m < p;                              // it has a sin block
  const double* Sc = S + (act ? blk_off[jc] : 0) - m;
  const double* Ss = S + (sine ? blk_off[2 * m] : 0) - m;
  double acc[9];
#pragma unroll
  for (int i = 0; i < 9; i++) acc[i] = 0.0;
  double pm2 = 0.0, pm1 = pmm;
  for (int n = 0; n <= p; n++) {
    const double* row = tab + 96 * n + m;
    double pn = 0.0;
    if (act && n >= m) {
      if (n == m) {
        pn = pmm;
      } else {
        const double a = row[0], b = row[32];
        pn = x * a * pm1 - b * pm2;
        pm2 = pm1;
        pm1 = pn;
      }
    }
    // P(m + 1, n) from the next lane (0 beyond the diagonal) for the theta derivative
    const double pnext = __shfl_down_sync(0xffffffffu, pn, 1, G);
    if (act && n >= m) {
      const double c2 = row[64];
      // -(legpoly_deriv) = d/dtheta of P(m, n)(cos theta)
      const double num = m * x * pn + c2 * s * (m + 1 <= n ? pnext : 0.0);
      const double dpn = s > 0.0 ? quotient_by(num, s, si) : 0.0;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const double a = Sc[d * nc + n];
        acc[d] += a * pn * cm;
        if (grads) {
          acc[3 + d] += a * dpn * cm;
          acc[6 + d] += a * pn * dcm;
        }
      }
      if (sine) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const double a = Ss[d * nc + n];
          acc[d] += a * pn * sm;
          if (grads) {
            acc[3 + d] += a * dpn * sm;
            acc[6 + d] += a * pn * dsm;
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 9; i++) {
    if (i >= 3 && !grads) break;
    double v = acc[i];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
    val[i] = kSqrt2Pi * v;
  }
}

struct NearArgs {
  const double* trg;
  long M;
  const int* count;
  const int* near_v;
  const int* near_k;
  const unsigned long long* rmax_bits;
  const double* Sx;      // [nv][3][nc] position coefficients
  const double* Vc;      // [nv][3][nc] self-velocity coefficients (single + double layer)
  const double* Gc;      // [nv][3][nc] double-layer density coefficients, or null
  const double* pos_up;  // [nv ng1][3]
  const double* den_up;
  const double* nrm_up;  // null without a double layer
  const double* dden_up;
  const double* theta_up;  // [p_up + 1] latitudes of the upsampled grid
  const double* tab;       // near_tables
  const int* blk_off;
  int p, p_up;
  double* proj;  // [kNearMax M][10]: projection, unit direction, value there, |T - P| / r_near
  double* corr;  // [M][kNearMax][3]
};

constexpr int kProjWarps = 4;

// Projection of each near target on its vesicle and the on-surface values there: one group of G
// lanes per (slot, target) pair, slot-major (most targets have one near vesicle, so the groups in
// use are neighbours). The vesicle's coefficients and the recurrence tables are staged in shared
// memory. What bounds it is the serial chain of up to 40 Gauss-Newton steps of p + 1 recurrence
// steps each: with the square roots and divisions of the recurrence in tables, 16 lanes per pair
// at p <= 15 and every warp at it, 15,000 pairs at p = 12 take 0.98 ms (one warp of a 128-thread CTA
// per pair, three waiting, and the coefficients recomputed took 14.5 ms with the sums of
// k_near_correct).
template <int G>
__global__ void __launch_bounds__(32 * kProjWarps) k_near_project(NearArgs A) {
  extern __shared__ double smn[];
  const int p = A.p, nc = p * (p + 2);
  double* tab = smn;
  int* bo = reinterpret_cast<int*>(tab + near_table_doubles(p));
  double* Sall = tab + near_table_doubles(p) + p + 1;
  const int grp = threadIdx.x / G, gl = threadIdx.x & (G - 1);
  const long i = (long)blockIdx.x * (32 * kProjWarps / G) + grp;
  const int slot = (int)(i / A.M);
  const long t = i - (long)slot * A.M;
  const int cnt = slot < kNearMax ? A.count[t] : 0;
  const bool on = slot < cnt && cnt <= kNearMax;
  if (__syncthreads_or(on) == 0) return;
  for (int k = threadIdx.x; k < near_table_doubles(p); k += 32 * kProjWarps) tab[k] = A.tab[k];
  for (int k = threadIdx.x; k <= 2 * p; k += 32 * kProjWarps) bo[k] = A.blk_off[k];
  double* S = Sall + grp * 3 * nc;
  const int v = on ? A.near_v[t * kNearMax + slot] : 0, k0 = on ? A.near_k[t * kNearMax + slot] : 0;
  if (on)
    for (int k = gl; k < 3 * nc; k += G) S[k] = A.Sx[(long)v * 3 * nc + k];
  __syncthreads();
  // the groups of a warp run their steps together (one finished early repeats nothing: its
  // angles stay); an idle group follows on its staged (unused) values
  const double tx = on ? A.trg[3 * t] : 0.0, ty = on ? A.trg[3 * t + 1] : 0.0, tz = on ? A.trg[3 * t + 2] : 0.0;
  double th = A.theta_up[k0 / (2 * A.p_up)], ph = M_PI * (k0 % (2 * A.p_up)) / A.p_up;
  double val[9];
  const double* Sg = on ? S : A.Sx;
  bool done = !on;
  for (int itn = 0; itn < 40; itn++) {  // Gauss-Newton on |X(theta, phi) - T|^2
    if (__all_sync(0xffffffffu, done)) break;
    sh_point<G>(Sg, tab, p, bo, cos(th), ph, true, val);
    const double rx = val[0] - tx, ry = val[1] - ty, rz = val[2] - tz;
    const double a11 = val[3] * val[3] + val[4] * val[4] + val[5] * val[5];
    const double a12 = val[3] * val[6] + val[4] * val[7] + val[5] * val[8];
    const double a22 = val[6] * val[6] + val[7] * val[7] + val[8] * val[8];
    const double g1 = val[3] * rx + val[4] * ry + val[5] * rz, g2 = val[6] * rx + val[7] * ry + val[8] * rz;
    const double reg = 1e-14 * (a11 + a22);
    const double b11 = a11 + reg, b22 = a22 + reg, det = b11 * b22 - a12 * a12;
    const double d1 = -(b22 * g1 - a12 * g2) / det, d2 = -(b11 * g2 - a12 * g1) / det;
    if (!done) {
      th += d1;
      ph += d2;
    }
    // at this length the steps are the rounding of the angles
    done = done || fmax(fabs(d1), fabs(d2)) < kStepDone;
  }
  sh_point<G>(Sg, tab, p, bo, cos(th), ph, true, val);
  const double px = val[0], py = val[1], pz = val[2];
  // outward normal X_theta x X_phi (the orientation of the library's unit normals)
  double nx = val[4] * val[8] - val[5] * val[7], ny = val[5] * val[6] - val[3] * val[8],
         nz = val[3] * val[7] - val[4] * val[6];
  const double nn = sqrt(nx * nx + ny * ny + nz * nz);
  nx /= nn;
  ny /= nn;
  nz /= nn;
  const double dx = tx - px, dy = ty - py, dz = tz - pz;
  const double dist = sqrt(dx * dx + dy * dy + dz * dz);
  const bool exterior = dx * nx + dy * ny + dz * nz >= 0.0;
  double ux = nx, uy = ny, uz = nz;
  if (dist > 0.0) {
    ux = dx / dist;
    uy = dy / dist;
    uz = dz / dist;
  }
  double y0[9];
  sh_point<G>(A.Vc + (long)v * 3 * nc, tab, p, bo, cos(th), ph, false, y0);
  if (A.Gc) {
    double gs[9];
    sh_point<G>(A.Gc + (long)v * 3 * nc, tab, p, bo, cos(th), ph, false, gs);
    const double jump = exterior ? 0.5 : -0.5;
    for (int d = 0; d < 3; d++) y0[d] += jump * gs[d];
  }
  if (on && gl == 0) {
    double* o = A.proj + 10 * i;
    o[0] = px;
    o[1] = py;
    o[2] = pz;
    o[3] = ux;
    o[4] = uy;
    o[5] = uz;
    o[6] = y0[0];
    o[7] = y0[1];
    o[8] = y0[2];
    o[9] = dist / near_radius(A.rmax_bits, A.p_up);
  }
}

// The correction of each pair: one CTA of 128 threads sums the smooth upsampled quadrature of the
// vesicle at the 7 line points and at the target; threads 0..2 interpolate. Bound by the FP64 pipe
// (8 targets x 1,200 sources per pair; 0.54 ms for 15,000 pairs at p = 12).
template <bool DL>
__global__ void __launch_bounds__(128) k_near_correct(NearArgs A) {
  const long i = blockIdx.x;
  const int slot = (int)(i / A.M);
  const long t = i - (long)slot * A.M;
  const int cnt = A.count[t];
  if (slot >= cnt || cnt > kNearMax) return;
  __shared__ double red[4][8 * 3];
  const int v = A.near_v[t * kNearMax + slot];
  const int ng1 = 2 * A.p_up * (A.p_up + 1);
  const double* o = A.proj + 10 * i;
  const double r_near = near_radius(A.rmax_bits, A.p_up);
  double pt[8][3];  // line points (7) and the target
#pragma unroll
  for (int q = 0; q < 8; q++)
#pragma unroll
    for (int d = 0; d < 3; d++) pt[q][d] = q < 7 ? o[d] + r_near * inter_point(q + 1) * o[3 + d] : A.trg[3 * t + d];
  double acc[24];
#pragma unroll
  for (int k = 0; k < 24; k++) acc[k] = 0.0;
  const double* P = A.pos_up + 3 * (long)v * ng1;
  const double* D = A.den_up + 3 * (long)v * ng1;
  const double* Nn = DL ? A.nrm_up + 3 * (long)v * ng1 : nullptr;
  const double* Gd = DL ? A.dden_up + 3 * (long)v * ng1 : nullptr;
  for (int s = threadIdx.x; s < ng1; s += blockDim.x) {
    const double sx = P[3 * s], sy = P[3 * s + 1], sz = P[3 * s + 2];
    const double fx = D[3 * s], fy = D[3 * s + 1], fz = D[3 * s + 2];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      // single layer: r = source - point (src/CPUKernels.cc:1011-1057)
      const double rx = sx - pt[q][0], ry = sy - pt[q][1], rz = sz - pt[q][2];
      const double r2 = rx * rx + ry * ry + rz * rz;
      double ri = rsqrt_f64_int_seed(r2);
      ri = r2_in_range(r2) ? ri : 0.0;
      const double ri2 = ri * ri;
      double c = (rx * fx + ry * fy + rz * fz) * ri2 * ri;
      if (DL) {  // double layer, r = point - source: 3/(4 pi) (r.n)(r.g) r / |r|^5, 6 times 1/(8 pi)
        const double rn = rx * Nn[3 * s] + ry * Nn[3 * s + 1] + rz * Nn[3 * s + 2];
        const double rg = rx * Gd[3 * s] + ry * Gd[3 * s + 1] + rz * Gd[3 * s + 2];
        c -= 6.0 * rn * rg * (ri2 * ri2 * ri);
      }
      acc[3 * q] = fma(c, rx, fma(fx, ri, acc[3 * q]));
      acc[3 * q + 1] = fma(c, ry, fma(fy, ri, acc[3 * q + 1]));
      acc[3 * q + 2] = fma(c, rz, fma(fz, ri, acc[3 * q + 2]));
    }
  }
  // fixed-order reduction: warp shuffles, then the 4 warps in order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 24; k++) {
    double a = acc[k];
    for (int of = 16; of > 0; of >>= 1) a += __shfl_xor_sync(0xffffffffu, a, of);
    if (lane == 0) red[warp][k] = a * kInv8Pi;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    const int d = threadIdx.x;
    double y[kInterpDeg];
    y[0] = o[6 + d];
    for (int l = 1; l < kInterpDeg; l++)
      y[l] = ((red[0][3 * (l - 1) + d] + red[1][3 * (l - 1) + d]) + (red[2][3 * (l - 1) + d] + red[3][3 * (l - 1) + d]));
    const double direct = (red[0][21 + d] + red[1][21 + d]) + (red[2][21 + d] + red[3][21 + d]);
    double interp = 0.0;
    for (int l = 0; l < kInterpDeg; l++) interp += y[l] * inter_poly(o[9], l);
    A.corr[(t * kNearMax + slot) * 3 + d] = interp - direct;
  }
}

// vel[t] += the corrections of its near vesicles, in slot order
__global__ void k_near_add(const int* __restrict__ count, const double* __restrict__ corr, long M,
                           double* __restrict__ vel) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= M) return;
  const int cnt = count[t];
  for (int s = 0; s < cnt && s < kNearMax; s++)
    for (int d = 0; d < 3; d++) vel[3 * t + d] += corr[(t * kNearMax + s) * 3 + d];
}

}  // namespace

int launch_centroid_radius(const double* X, long nv, int p, double* cen_r, unsigned long long* rmax_bits,
                           cudaStream_t st) {
  if (nv <= 0) return VES3D_OK;
  VES3D_CK(cudaMemsetAsync(rmax_bits, 0, sizeof(unsigned long long), st));
  k_centroid_radius<<<(unsigned)nv, 256, 0, st>>>(X, ngrid_(p), cen_r, rmax_bits);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// Recurrence tables of k_near_project (see near_table_doubles).
std::vector<double> near_tables(int p) {
  std::vector<double> t(near_table_doubles(p), 0.0);
  for (int m = 0; m <= p; m++) {
    t[96 * (p + 1) + m] = m > 0 ? std::sqrt((2.0 * m + 1.0) / (2.0 * m)) : 0.0;
    for (int n = m + 1; n <= p; n++) {
      t[96 * n + m] = std::sqrt(((2.0 * n - 1) * (2.0 * n + 1)) / ((double)(n - m) * (n + m)));
      if (n > m + 1)
        t[96 * n + 32 + m] =
            std::sqrt(((2.0 * n + 1) * (n + m - 1) * (n - m - 1)) / ((double)(n - m) * (n + m) * (2 * n - 3)));
      t[96 * n + 64 + m] = std::sqrt(n + m + 1.0) * std::sqrt((double)(n - m));
    }
  }
  return t;
}

int launch_near_find(const double* trg, long M, const double* cen_r, long nv, const double* pos_up, int p_up,
                     unsigned long long* rmax_over, int* count, int* near_v, int* near_k, cudaStream_t st) {
  if (M <= 0) return VES3D_OK;
  VES3D_CK(cudaMemsetAsync(rmax_over + 1, 0xff, sizeof(unsigned long long), st));
  k_near_find<<<(unsigned)((M + 3) / 4), 128, 0, st>>>(trg, M, cen_r, nv, pos_up, p_up, rmax_over, rmax_over + 1, count,
                                                       near_v, near_k);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

template <int G>
static int launch_project(const NearArgs& a, cudaStream_t st) {
  const int per = 32 * kProjWarps / G, p = a.p;
  const size_t smem = ((size_t)near_table_doubles(p) + p + 1 + (size_t)per * 3 * p * (p + 2)) * sizeof(double);
  if (const int s = allow_smem(k_near_project<G>, smem)) return s;
  k_near_project<G><<<(unsigned)((a.M * kNearMax + per - 1) / per), 32 * kProjWarps, smem, st>>>(a);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

int launch_near_correct(const double* trg, long M, const int* count, const int* near_v, const int* near_k,
                        const unsigned long long* rmax_over, const double* Sx, const double* Vc, const double* Gc,
                        const double* pos_up, const double* den_up, const double* nrm_up, const double* dden_up,
                        const double* theta_up, const double* tab, const int* blk_off, int p, int p_up, double* proj,
                        double* corr, double* vel, cudaStream_t st) {
  if (M <= 0) return VES3D_OK;
  if (p + 1 > 32) {
    set_error("near-singular correction: orders up to 31");
    return VES3D_ERR_ARG;
  }
  const NearArgs a{trg, M, count, near_v, near_k, rmax_over, Sx, Vc, Gc, pos_up, den_up, nrm_up, dden_up, theta_up,
                   tab, blk_off, p, p_up, proj, corr};
  const int s = p + 1 <= 16 ? launch_project<16>(a, st) : launch_project<32>(a, st);
  if (s) return s;
  if (nrm_up)
    k_near_correct<true><<<(unsigned)(M * kNearMax), 128, 0, st>>>(a);
  else
    k_near_correct<false><<<(unsigned)(M * kNearMax), 128, 0, st>>>(a);
  VES3D_LAUNCHED();
  k_near_add<<<(unsigned)((M + 127) / 128), 128, 0, st>>>(count, corr, M, vel);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

}  // namespace ves3d
