// Fused singular-quadrature kernel of the self-matrix build (FP64), for the single and the
// double layer:
//
//   R (rotated coefficients, 3 x Nc)
//     -> Legendre synthesis at the order-q nodes, values and theta-derivatives
//     -> DFT synthesis: X, X_theta, X_phi on the upsampled grid
//     -> the singular kernel to the two pole targets, 2 poles x 6 components
//     -> transposed DFT -> transposed Legendre sums
//     -> C (2 x 6 x Nc): the kernel contracted back to order-p coefficients
//
// i.e. SHC2Grid(p -> q, grads) + the kernel loop + SHC2GridTranspose(q -> p) of
// SphericalHarmonics<Real>::StokesSingularInteg_ (src/SphericalHarmonics.cc:963-1082), every
// intermediate in shared memory.
//
// The work is FP64 multiply-adds on operands in shared memory, so the grid's symmetries come first:
// latitudes l and q - l share the Legendre sums of the even and of the odd degrees, and longitudes j
// and -j the cosine and sine sums. That halves the dense transforms' multiply-adds, which a matrix
// instruction has no use for (FP64 DMMA runs at the vector units' rate); one thread then holds a row's
// coefficients in registers and meets compile-time cosines as constant operands. A CTA takes one
// rotation, LPG latitude pairs through all phases at a time.
// Bound by the FP64 pipe (39% busy at p = 16) and, where it is not, by the barriers between the
// phases and instruction fetch of the unrolled transforms. Self matrices of
//   512 / 64 vesicles, p = 16:  32.8 -> 18.3 ms / 4.12 -> 2.28 ms  (before: dense, DMMA from shared memory)
//   64 vesicles, p = 24:        32.4 -> 16.3 ms
//   64 vesicles, p = 12:        1.29 -> 0.66 ms
//   double layer, 48 at p = 16: 20 -> 1.72 ms  (before: a kernel per stage, intermediates in HBM)
// Thread groups that take a pair each through all phases with their own barriers were slower
// (2.91 ms for 64 vesicles), as were three or five parts per row (the code outgrows the cache).
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "cos_table.cuh"
#include "kernels.h"

namespace ves3d {

namespace {

struct RingArgs {
  const double* R;        // [nrot][3][nc]
  double* C;              // [nrot][12][nc]
  const double* leg;      // [q + 1][ring_leg_offsets(p, ..)], times sqrt(2 pi)
  const double* dleg;
  const double* sing_w;   // [q + 1]
  const double* qp;       // [2][p + 1]
  const double* twiddle;  // GEN: [J][PM + 1][2] cos / sin of m phi_j
  const int* blk_off;     // [2 p + 1]
  const int* leg_off;     // [4 p]: starts of the blocks' even and odd parts in a row of leg
  long nrot;
  int p, q, lpg, ldl;     // lpg: latitude pairs at a time; ldl: row stride of leg
};

// Items of the transposed Legendre sums: (block, parity, up to qc coefficients), times two
// halves of the 12 kernel components.
__host__ __device__ constexpr int legt_items(int p, int qc) {
  int t = 0;
  for (int k = 0; k < 2 * p; k++) {
    const int len = p + 1 - (k + 1) / 2;
    t += ((len + 1) / 2 + qc - 1) / qc + (len / 2 + qc - 1) / qc;
  }
  return 2 * t;
}

// Least n' >= n with n' = r (mod 16): row strides in doubles that keep the lanes of a half warp on
// distinct banks.
__host__ __device__ constexpr int round16(int n, int r) { return n + ((r - n % 16) + 16) % 16; }

// Shape of the instance for (at most) order P: threads, CTAs per SM, and the pairs of latitudes that
// a CTA takes through the phases at a time (fewer where a large p_up leaves no room for them).
// Threads are the items of the transposed Legendre sums; CTAs per SM what registers and shared memory
// allow, several so that one CTA's barriers are another's work.
// p = 12 in two CTAs of 192 threads and five pairs against three of 128 and three pairs (13 pairs in three
// rounds for five): 64 vesicles 746 -> 660 us, 8 vesicles 111 -> 96 us, p_up = 40 2.72 -> 2.19 ms; p = 10
// so was slower (310 -> 360 us).
template <int P>
struct RingShape {
  static constexpr int NT = P <= 10 ? 128 : P <= 16 ? 192 : 384;
  static constexpr int MINB = P <= 8 ? 4 : P <= 10 ? 3 : P <= 16 ? 2 : 1;
  static constexpr int LPG = P <= 10 || P == 16 ? 4 : 5;
  static constexpr int QC = 4;  // coefficients of one transposed-Legendre item
  static constexpr int NP = 2;  // parts of a row in the DFT synthesis
  static_assert(legt_items(P, QC) <= NT, "one item per thread");
};

struct RingLayout {
  int ldj, ldx, ldc, off_leg, off_dleg, off_a, off_x, off_tw, off_sw, off_qp, off_trg, off_bo, off_lo, off_it, total;
};

__host__ __device__ inline RingLayout ring_layout(int p, int q, int lpg, int qc, int ldl, int tw_doubles) {
  RingLayout L;
  const int nc = p * (p + 2);
  L.ldj = (2 * q) | 1;
  L.ldx = round16(12 * L.ldj, 2);  // slots of X / K and of C: eight of them times two rows fill 16 banks
  L.ldc = round16(2 * p * 12, 2);
  int o = (3 * nc + 1) & ~1;
  L.off_leg = o;
  o += lpg * ldl;
  L.off_dleg = o;
  o += lpg * ldl;
  L.off_a = o;  // A, dA [2 lpg][6][2 p + 1], then C [2 lpg][2 p][12]
  const int sz_a = 2 * lpg * 6 * (2 * p + 1), sz_c = 2 * lpg * L.ldc;
  o += (sz_a > sz_c ? sz_a : sz_c) + 1 & ~1;
  L.off_x = o;  // X, X_theta, X_phi [2 lpg][9 of 12][ldj], then K [2 lpg][12][ldj]
  o += 2 * lpg * L.ldx;
  L.off_tw = o;
  o += tw_doubles;
  L.off_sw = o;
  o += q + 1;
  L.off_qp = o;
  o += 2 * (p + 1);
  L.off_trg = o;
  o += 6;
  L.off_bo = o;
  o += (2 * p + 2) / 2 + 1;
  L.off_lo = o;
  o += 2 * p;
  L.off_it = o;  // items of the transposed Legendre sums (int)
  o += legt_items(p, qc) / 2;
  L.total = o;
  return L;
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// The kernel values of one source point at the two pole targets: v[t * 6 + component].
template <bool DL>
__device__ __forceinline__ void pole_kernel(const double* x, int ldj, const double* trg, double w0, double w1,
                                            double* v) {
  const double px = x[0], py = x[ldj], pz = x[2 * ldj];
  const double ax = x[3 * ldj], ay = x[4 * ldj], az = x[5 * ldj];
  const double bx = x[6 * ldj], by = x[7 * ldj], bz = x[8 * ldj];
  const double nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
  double area = 0.0;
  if (!DL) {
    const double n2 = nx * nx + ny * ny + nz * nz;
    area = n2 * rsqrt_f64_int_seed(n2);  // |X_theta x X_phi| > 0 on the upsampled grid
  }
#pragma unroll
  for (int t = 0; t < 2; t++) {
    const double dx = trg[t] - px, dy = trg[2 + t] - py, dz = trg[4 + t] - pz;
    const double r2 = dx * dx + dy * dy + dz * dz;
    double rinv = rsqrt_f64_int_seed(r2);  // (r2 below 2^-126 is cut off here too)
    if (r2 <= 2.220446049250313e-16) rinv = 0.0;
    const double rinv2 = rinv * rinv;
    double* k = v + 6 * t;
    if (DL) {
      const double a2 = kDl * (t ? w1 : w0) * (nx * dx + ny * dy + nz * dz) * (rinv2 * rinv2 * rinv);
      const double bx2 = dx * a2, by2 = dy * a2;
      k[0] = dx * bx2;
      k[1] = dy * bx2;
      k[2] = dz * bx2;
      k[3] = dy * by2;
      k[4] = dz * by2;
      k[5] = dz * dz * a2;
    } else {
      const double a1 = kInv8Pi * (t ? w1 : w0) * area * rinv;
      const double a2 = a1 * rinv2;
      const double bx2 = dx * a2, by2 = dy * a2;
      k[0] = fma(dx, bx2, a1);
      k[1] = dy * bx2;
      k[2] = dz * bx2;
      k[3] = fma(dy, by2, a1);
      k[4] = dz * by2;
      k[5] = fma(dz * dz, a2, a1);
    }
  }
}

// Transposed DFT of one row at the frequencies of parity PAR: the row's values at the four
// images j, -j, q - j, q + j of a longitude are folded first.
template <int P, bool GEN, int PAR>
__device__ __forceinline__ void dft_transpose_row(const double* __restrict__ x, int p, int q, const double* tw,
                                                  double* __restrict__ out) {
  constexpr int NM = (P - PAR) / 2 + 1;  // m = PAR, PAR + 2, .. <= P
  double c[NM], s[NM];
#pragma unroll
  for (int i = 0; i < NM; i++) c[i] = s[i] = 0.0;
  const int N = 2 * q, J = q / 2;
  auto fold = [&](int j, double& fc, double& fs) {
    const double v1 = x[j];
    const double v2 = j == 0 ? 0.0 : x[N - j];
    const bool own = 2 * j == q;  // its image q - j is itself
    const double v3 = own ? 0.0 : x[q - j];
    const double v4 = j == 0 || own ? 0.0 : x[q + j];
    if (PAR == 0) {
      fc = (v1 + v2) + (v3 + v4);
      fs = (v1 - v2) - (v3 - v4);
    } else {
      fc = (v1 + v2) - (v3 + v4);
      fs = (v1 - v2) + (v3 - v4);
    }
  };
  if constexpr (!GEN) {
    constexpr int N1 = 4 * P;
#pragma unroll
    for (int j = 0; j <= P; j++) {
      double fc, fs;
      fold(j, fc, fs);
#pragma unroll
      for (int i = 0; i < NM; i++) {
        const int m = PAR + 2 * i;
        c[i] = fma(fc, c_cos<N1>.v[(m * j) % N1], c[i]);
        if (m > 0 && m < P) s[i] = fma(fs, c_cos<N1>.v[(m * j + 3 * P) % N1], s[i]);
      }
    }
  } else {
#pragma unroll 1
    for (int j = 0; j <= J; j++) {
      double fc, fs;
      fold(j, fc, fs);
      const double2* t = reinterpret_cast<const double2*>(tw) + j * (P + 1) + PAR;
#pragma unroll
      for (int i = 0; i < NM; i++) {
        const double2 w = t[2 * i];
        c[i] = fma(fc, w.x, c[i]);
        s[i] = fma(fs, w.y, s[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NM; i++) {
    const int m = PAR + 2 * i;
    if (m == 0) {
      out[0] = c[i];
    } else if (m <= p) {
      out[(2 * m - 1) * 12] = c[i];
      if (m < p) out[2 * m * 12] = s[i];
    }
  }
}

// DFT synthesis of one row at the longitudes of part PT of NP: j = PT, PT + NP, .. <= q / 2 and
// their images, from the row's cosine and sine coefficients.
template <int P, bool GEN, int NP, int PT>
__device__ __forceinline__ void dft_row_part(const double (&c)[P + 1], const double (&s)[P + 1], int part, int q,
                                             const double* tw, double* __restrict__ x) {
  const int N = 2 * q;
  auto put = [&](int j, double ce, double co, double se, double so) {
    const double a = ce + co, b = se + so, d = ce - co, e = so - se;
    x[j] = a + b;
    if (j > 0) x[N - j] = a - b;
    if (2 * j != q) {
      x[q - j] = d + e;
      if (j > 0) x[q + j] = d - e;
    }
  };
  if constexpr (!GEN) {
    constexpr int N1 = 4 * P;
#pragma unroll
    for (int j = PT; j <= P; j += NP) {
      double ce = c[0], co = 0.0, se = 0.0, so = 0.0;
#pragma unroll
      for (int m = 1; m <= P; m++) {
        const double w = c_cos<N1>.v[(m * j) % N1], z = c_cos<N1>.v[(m * j + 3 * P) % N1];
        if (m & 1) {
          co = fma(c[m], w, co);
          so = fma(s[m], z, so);
        } else {
          ce = fma(c[m], w, ce);
          se = fma(s[m], z, se);
        }
      }
      put(j, ce, co, se, so);
    }
  } else {
    const int J = q / 2;
#pragma unroll 1
    for (int j = part; j <= J; j += NP) {
      const double2* t = reinterpret_cast<const double2*>(tw) + j * (P + 1);
      double ce = c[0], co = 0.0, se = 0.0, so = 0.0;
#pragma unroll
      for (int m = 1; m <= P; m++) {
        const double2 w = t[m];
        if (m & 1) {
          co = fma(c[m], w.x, co);
          so = fma(s[m], w.y, so);
        } else {
          ce = fma(c[m], w.x, ce);
          se = fma(s[m], w.y, se);
        }
      }
      put(j, ce, co, se, so);
    }
  }
}

template <int P, bool GEN, bool DL>
__global__ void __launch_bounds__(RingShape<P>::NT, RingShape<P>::MINB) k_ring(const RingArgs A) {
  using Sh = RingShape<P>;
  constexpr int NT = Sh::NT, QC = Sh::QC, NP = Sh::NP;
  const int p = GEN ? A.p : P, q = GEN ? A.q : 2 * P;
  const int nc = p * (p + 2), ldl = A.ldl, F = 2 * p, lda = F + 1;
  const int npair = q / 2 + 1;
  extern __shared__ __align__(16) double sm[];
  const RingLayout L = ring_layout(p, q, A.lpg, QC, ldl, GEN ? 2 * (q / 2 + 1) * (P + 1) : 0);
  double *sR = sm, *sLeg = sm + L.off_leg, *sdLeg = sm + L.off_dleg, *sA = sm + L.off_a, *sC = sA, *sX = sm + L.off_x;
  double *sTw = sm + L.off_tw, *sSw = sm + L.off_sw, *sQp = sm + L.off_qp, *trg = sm + L.off_trg;
  int* sBo = reinterpret_cast<int*>(sm + L.off_bo);
  int* sLo = reinterpret_cast<int*>(sm + L.off_lo);
  int2* sIt = reinterpret_cast<int2*>(sm + L.off_it);
  const int ldj = L.ldj, ldx = L.ldx, ldc = L.ldc;
  const int tid = threadIdx.x;
  const int nit = legt_items(p, QC);
  for (int i = tid; i <= F; i += NT) sBo[i] = __ldg(A.blk_off + i);
  for (int i = tid; i < 2 * F; i += NT) sLo[i] = __ldg(A.leg_off + i);
  for (int i = tid; i <= q; i += NT) sSw[i] = __ldg(A.sing_w + i);
  for (int i = tid; i < 2 * (p + 1); i += NT) sQp[i] = __ldg(A.qp + i);
  if (GEN)
    for (int i = tid; i < 2 * (q / 2 + 1) * (P + 1); i += NT) sTw[i] = __ldg(A.twiddle + i);
  if (tid == 0) {
    // items: the coefficients t, t + T, .. of one parity of a block, so that neighbouring items
    // read neighbouring values: x: block | parity << 8 | count << 9 | T << 13, y: place in a row of
    // leg | first coefficient << 16
    int n = 0;
    for (int k = 0; k < F; k++) {
      const int b0 = __ldg(A.blk_off + k), len = __ldg(A.blk_off + k + 1) - b0;
      for (int par = 0; par < 2; par++) {
        const int cnt = (len + 1 - par) / 2, T = (cnt + QC - 1) / QC;
        for (int t = 0; t < T; t++)
          sIt[n++] = make_int2(k | par << 8 | (cnt - t + T - 1) / T << 9 | T << 13,
                               (__ldg(A.leg_off + 2 * k + par) + t) | (b0 + par + 2 * t) << 16);
      }
    }
  }
  const long first = blockIdx.x;
  if (first < A.nrot)
    for (int i = tid; i < 3 * nc; i += NT) cp_async8(sR + i, A.R + first * 3 * nc + i);
  for (long rot = first; rot < A.nrot; rot += gridDim.x) {
    double acc[QC][6];
#pragma unroll
    for (int i = 0; i < QC; i++)
#pragma unroll
      for (int h = 0; h < 6; h++) acc[i][h] = 0.0;
    // pairs per round: lpg, or one fewer where they do not divide evenly
    const int nround = (npair + A.lpg - 1) / A.lpg;
    for (int g = 0; g < nround; g++) {
      const int l0 = g * npair / nround, np = (g + 1) * npair / nround - l0;
      // the round's pairs: latitudes l0 + l (slot 2 l) and their mirror images q - l0 - l (slot
      // 2 l + 1), which the middle latitude of an even q has not
      for (int i = tid; i < np * ldl; i += NT) {
        cp_async8(sLeg + i, A.leg + (long)l0 * ldl + i);
        cp_async8(sdLeg + i, A.dleg + (long)l0 * ldl + i);
      }
      cp_async_wait();
      __syncthreads();
      if (g == 0 && tid < 32) {  // pole targets
#pragma unroll
        for (int i = 0; i < 6; i++) {
          const int c = i >> 1, t = i & 1;
          double s = tid <= p ? sR[c * nc + tid] * sQp[t * (p + 1) + tid] : 0.0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
          if (tid == 0) trg[i] = s;
        }
      }
      // ---- Legendre synthesis: even and odd parts of a block serve both latitudes of a pair ----------
      for (int i = tid; i < np * F; i += NT) {
        const int k = i / np, l = i - k * np;
        const int c0 = sBo[k], len = sBo[k + 1] - c0, ne = (len + 1) / 2, no = len / 2;
        const double *Le = sLeg + l * ldl + sLo[2 * k], *Lo = sLeg + l * ldl + sLo[2 * k + 1], *r = sR + c0;
        const double *De = sdLeg + l * ldl + sLo[2 * k], *Do = sdLeg + l * ldl + sLo[2 * k + 1];
        double e[6], o[6];
#pragma unroll
        for (int d = 0; d < 6; d++) e[d] = o[d] = 0.0;
#pragma unroll 2
        for (int n = 0; n < no; n++) {
          const double a = Le[n], b = Lo[n], da = De[n], db = Do[n];
#pragma unroll
          for (int d = 0; d < 3; d++) {
            const double r0 = r[d * nc + 2 * n], r1 = r[d * nc + 2 * n + 1];
            e[d] = fma(a, r0, e[d]);
            o[d] = fma(b, r1, o[d]);
            e[3 + d] = fma(da, r0, e[3 + d]);
            o[3 + d] = fma(db, r1, o[3 + d]);
          }
        }
        if (ne > no) {
          const double a = Le[no], da = De[no];
#pragma unroll
          for (int d = 0; d < 3; d++) {
            const double r0 = r[d * nc + 2 * no];
            e[d] = fma(a, r0, e[d]);
            e[3 + d] = fma(da, r0, e[3 + d]);
          }
        }
        double* a0 = sA + (2 * l) * 6 * lda + k;
        double* a1 = a0 + 6 * lda;
#pragma unroll
        for (int d = 0; d < 3; d++) {
          a0[d * lda] = e[d] + o[d];
          a1[d * lda] = e[d] - o[d];
          a0[(3 + d) * lda] = e[3 + d] + o[3 + d];
          a1[(3 + d) * lda] = o[3 + d] - e[3 + d];
        }
      }
      __syncthreads();
      // ---- DFT synthesis: rows (X | X_theta | X_phi, component, slot) -----------------------------
      {
        const int nrow = 18 * np;
        for (int i = tid; i < NP * nrow; i += NT) {
          const int part = i / nrow, r = i - part * nrow;
          const int f = r / (2 * np), slot = r - f * 2 * np, kind = f / 3, d = f - kind * 3;
          const double* a = sA + (slot * 6 + (kind == 2 ? 3 : 0) + d) * lda;
          double c[P + 1], s[P + 1];
          c[0] = kind == 1 ? 0.0 : a[0];
          s[0] = 0.0;
#pragma unroll
          for (int m = 1; m <= P; m++) {
            const bool in = !GEN || m <= p;
            const double ac = in ? a[2 * m - 1] : 0.0;
            const double as = (GEN ? m < p : m < P) ? a[2 * m] : 0.0;
            c[m] = kind == 1 ? m * as : ac;
            s[m] = kind == 1 ? -m * ac : as;
          }
          double* x = sX + slot * ldx + f * ldj;
          if (GEN || part == 0)
            dft_row_part<P, GEN, NP, 0>(c, s, part, q, sTw, x);
          else
            dft_row_part<P, GEN, NP, 1>(c, s, part, q, sTw, x);
        }
      }
      __syncthreads();
      // ---- the kernel at a pair's points (la, j) and (lb, j): their sum and difference, in place of
      // the surface values of that column ---------------------------------------------------------
      for (int i = tid; i < np * 2 * q; i += NT) {
        const int l = i / (2 * q), j = i - l * 2 * q;
        const int la = l0 + l, lb = q - la;
        double* xa = sX + 2 * l * ldx + j;
        double* xb = xa + ldx;
        double va[12], vb[12];
        pole_kernel<DL>(xa, ldj, trg, sSw[lb], sSw[la], va);  // pole 0 is weighted from the other end
        if (la != lb) {
          pole_kernel<DL>(xb, ldj, trg, sSw[la], sSw[lb], vb);
        } else {
#pragma unroll
          for (int h = 0; h < 12; h++) vb[h] = 0.0;
        }
#pragma unroll
        for (int h = 0; h < 12; h++) {
          xa[h * ldj] = va[h] + vb[h];
          xb[h * ldj] = la != lb ? va[h] - vb[h] : 0.0;
        }
      }
      __syncthreads();
      // ---- transposed DFT: rows (component, slot), one item per parity of the frequency -----------
      {
        const int nrow = 24 * np;
        for (int i = tid; i < 2 * nrow; i += NT) {
          const int par = i >= nrow, r = i - (par ? nrow : 0), h = r / (2 * np), slot = r - h * 2 * np;
          if (par == 0)
            dft_transpose_row<P, GEN, 0>(sX + slot * ldx + h * ldj, p, q, sTw, sC + slot * ldc + h);
          else
            dft_transpose_row<P, GEN, 1>(sX + slot * ldx + h * ldj, p, q, sTw, sC + slot * ldc + h);
        }
      }
      __syncthreads();
      if (g + 1 == nround && rot + gridDim.x < A.nrot)  // sR is free: the next rotation's
        for (int i = tid; i < 3 * nc; i += NT) cp_async8(sR + i, A.R + (rot + gridDim.x) * 3 * nc + i);
      // ---- transposed Legendre sums: even degrees meet the sum of the pair, odd ones the difference
      if (tid < nit) {
        const int half = tid >= nit / 2;
        const int2 it = sIt[half ? tid - nit / 2 : tid];
        const int k = it.x & 0xff, par = (it.x >> 8) & 1, cnt = (it.x >> 9) & 0xf, T = it.x >> 13;
        const double* cc = sC + par * ldc + k * 12 + half * 6;
        for (int l = 0; l < np; l++) {
          const double2* c2 = reinterpret_cast<const double2*>(cc + 2 * l * ldc);
          const double2 x0 = c2[0], x1 = c2[1], x2 = c2[2];
          const double* lg = sLeg + l * ldl + (it.y & 0xffff);
#pragma unroll
          for (int n = 0; n < QC; n++) {
            const double w = n < cnt ? lg[n * T] : 0.0;
            acc[n][0] = fma(w, x0.x, acc[n][0]);
            acc[n][1] = fma(w, x0.y, acc[n][1]);
            acc[n][2] = fma(w, x1.x, acc[n][2]);
            acc[n][3] = fma(w, x1.y, acc[n][3]);
            acc[n][4] = fma(w, x2.x, acc[n][4]);
            acc[n][5] = fma(w, x2.y, acc[n][5]);
          }
        }
      }
      __syncthreads();
    }
    if (tid < nit) {
      const int half = tid >= nit / 2;
      const int2 it = sIt[half ? tid - nit / 2 : tid];
      const int cnt = (it.x >> 9) & 0xf, T = it.x >> 13;
      double* out = A.C + rot * 12 * nc + half * 6 * nc + (it.y >> 16);
#pragma unroll
      for (int n = 0; n < QC; n++)
        if (n < cnt)
#pragma unroll
          for (int h = 0; h < 6; h++) out[h * nc + 2 * n * T] = acc[n][h];
    }
  }
}

constexpr size_t kSmemPerSm = 227 * 1024;

// Persistent CTAs per SM: what fits, or with VES3D_RING_CTAS=1 one, which leaves room beside it
// for far-field CTAs when the far field runs concurrently (VES3D_FAR_OVERLAP=1).
int ring_ctas_cap() {
  static const int n = [] {
    const char* e = getenv("VES3D_RING_CTAS");
    return e && e[0] == '1' && !e[1] ? 1 : 32;
  }();
  return n;
}

template <int P, bool GEN, bool DL>
int launch_ring(const double* R, long nrot, const DevTables& T, double* C, cudaStream_t st) {
  using Sh = RingShape<P>;
  RingArgs a;
  a.R = R;
  a.C = C;
  a.leg = T.ring_leg;
  a.dleg = T.ring_dleg;
  a.sing_w = T.sing_w;
  a.qp = T.qp;
  a.twiddle = T.ring_twiddle;
  a.blk_off = T.blk_off;
  a.leg_off = T.ring_off;
  a.ldl = T.ring_ldl;
  a.nrot = nrot;
  a.p = T.p0;
  a.q = T.p1;
  const int tw = GEN ? 2 * (T.p1 / 2 + 1) * (P + 1) : 0;
  auto bytes = [&](int lpg) {
    return (size_t)ring_layout(T.p0, T.p1, lpg, Sh::QC, T.ring_ldl, tw).total * sizeof(double);
  };
  int lpg = Sh::LPG;
  while (lpg > 1 && bytes(lpg) > kSmemPerSm / Sh::MINB - 1024) lpg--;
  a.lpg = lpg;
  const size_t smem = bytes(lpg);
  if (smem > kSmemPerSm) {
    set_error("internal: fused self-matrix build at p = %d, p_up = %d needs %zu bytes of shared memory", T.p0, T.p1, smem);
    return VES3D_ERR_ARG;
  }
  if (const int s = allow_smem(k_ring<P, GEN, DL>, smem)) return s;
  int dev = 0, nsm = 148, per = 1;
  VES3D_CK(cudaGetDevice(&dev));
  VES3D_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  VES3D_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_ring<P, GEN, DL>, Sh::NT, smem));
  const long grid = std::min(nrot, (long)nsm * std::max(1, std::min(per, ring_ctas_cap())));
  k_ring<P, GEN, DL><<<(unsigned)grid, Sh::NT, smem, st>>>(a);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

}  // namespace

// orders with a compile-time transform at q = 2 p
#define VES3D_RING_ORDERS(X) X(4) X(6) X(8) X(10) X(12) X(16) X(20) X(24)

// Orders and upsampled orders whose padded tables fit shared memory; the others take the stage by
// stage pipeline. Within the range the fused kernel is the faster at every order, the run-time
// instances included (they pad p to the next instance and read their cosines from shared memory).
// Builds of 8 vesicles, fused and stage by stage, at (p, p_up): (4, 8) 31 and 42 us, (7, 14) 96 and
// 122 us, (8, 56) 0.38 and 0.95 ms, (12, 18) 0.21 and 0.48 ms, (16, 32) 0.55 and 2.7 ms, (22, 44) 7.7 and
// 15.5 ms, (24, 56) 9.7 and 30.2 ms.
bool ring_supported(int p0, int p1) { return p0 >= 2 && p0 <= 24 && p1 >= p0 && p1 <= 56; }

// Starts of the blocks' even-degree and odd-degree parts in a row of the fused build's Legendre
// tables, then the row length. The i-th part starts at i (mod 4) and rows are 4 (mod 16) long, so
// that the four latitudes times four parts that a half warp reads are on distinct banks.
std::vector<int> ring_leg_offsets(int p0) {
  std::vector<int> off;
  int o = 0;
  for (int i = 0; i < 4 * p0; i++) {
    const int len = p0 + 1 - (i / 2 + 1) / 2;
    o += (i % 4 - o % 4 + 4) % 4;
    off.push_back(o);
    o += (len + 1 - i % 2) / 2;
  }
  off.push_back(round16(o, 4));
  return off;
}

// The padded order of the run-time instance that takes order p0 (its twiddle rows).
int ring_padded_order(int p0, int p1) {
  if (p1 == 2 * p0) {
#define VES3D_RING_HAS(P) \
  if (p0 == P) return 0;
    VES3D_RING_ORDERS(VES3D_RING_HAS)
#undef VES3D_RING_HAS
  }
  for (int P : {8, 12, 16, 20, 24})
    if (p0 <= P) return P;
  return 0;
}

int launch_ring_build(bool dl, const double* R, long nrot, const DevTables& T, double* C, cudaStream_t st) {
  if (nrot <= 0) return VES3D_OK;
  const int pad = ring_padded_order(T.p0, T.p1);
  if (pad == 0) {
    switch (T.p0) {
#define VES3D_RING_CASE(P) \
  case P: return dl ? launch_ring<P, false, true>(R, nrot, T, C, st) : launch_ring<P, false, false>(R, nrot, T, C, st);
      VES3D_RING_ORDERS(VES3D_RING_CASE)
#undef VES3D_RING_CASE
      default: break;
    }
  }
  switch (pad) {
#define VES3D_RING_CASE(P) \
  case P: return dl ? launch_ring<P, true, true>(R, nrot, T, C, st) : launch_ring<P, true, false>(R, nrot, T, C, st);
    VES3D_RING_CASE(8) VES3D_RING_CASE(12) VES3D_RING_CASE(16) VES3D_RING_CASE(20) VES3D_RING_CASE(24)
#undef VES3D_RING_CASE
    default: break;
  }
  set_error("internal: fused self-matrix build at p = %d, p_up = %d", T.p0, T.p1);
  return VES3D_ERR_ARG;
}

}  // namespace ves3d
