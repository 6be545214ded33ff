// FP64 kernels of the singular self-interaction build (plain form): coefficient
// rotation to every target, the pole-singular Stokes kernel, and the adjoint rotation
// that scatters the result into the per-vesicle self-matrix layout.
// Math: SphericalHarmonics<Real>::RotateAll / StokesSingularInteg_ / RotateTranspose
// (src/SphericalHarmonics.cc:363-541, 954-1180).
#include <cstdlib>

#include "common.cuh"
#include "kernels.h"

namespace ves3d {

// Most threads (coefficients) a CTA takes: the rotation blocks of larger orders outgrow shared memory.
constexpr int kRotAllMax = 768;

// CTAs (vesicle v, latitude rotation t, part of the p0 longitude phases j), JB phases at a time (4,
// or fewer where the staging would not fit: p = 24).
// out[c'] = sum_b (P_j s)[perm_n[b]] * Mr[t][n][b][pos(c')],   n = degree(c').
// A thread per coefficient: it keeps the coefficient and its partner in registers, writes their JB
// phases to shared memory in degree-major order, and forms one degree-major output of the three
// components and JB phases (a warp's lanes share a degree: one loop length, broadcast inputs in
// 16-byte loads, consecutive block columns), so a block element is loaded once per 3 JB
// multiply-adds. The outputs return to their order in shared memory and leave as one contiguous run.
// The data (R written once) would take a third of its time; bound by the shared-memory loads and the
// barriers around them. With four multiply-adds per block element, one component a pass, and outputs
// stored in degree-major order (8 bytes per line) it took
//   p = 16, 512 / 64 vesicles  1.71 ms / 240 us, now 1.10 ms / 154 us
//   p = 24, 64 vesicles        2.59 ms, now 0.86 ms
template <int JB>
__global__ void __launch_bounds__(kRotAllMax) k_rotate_all(const double* __restrict__ S, int p0, int mr_per_t,
                                                           DevTables T, double* __restrict__ R) {
  constexpr int ND = 3 * JB, LDB = JB == 4 ? 14 : ND + (JB & 1);  // (row stride: even, off the multiples of 16)
  extern __shared__ __align__(16) double sm[];
  const int nc = p0 * (p0 + 2);
  double* sB = sm;                                  // phases [nc][LDB], then outputs [JB][3][nc]
  double* sM = sB + (size_t)LDB * nc;               // blocks of t, rows b
  double* sCs = sM + mr_per_t;                      // cos_tab [2 p0]
  double* sSn = sCs + 2 * p0;                       // sin_tab [2 p0]
  const int t = blockIdx.x;
  const long v = blockIdx.y;
  const int tid = threadIdx.x;
  const int mbase = __ldg(T.mr_off + t * (p0 + 1));
  for (int i = tid; i < mr_per_t; i += blockDim.x) sM[i] = __ldg(T.mr + mbase + i);
  for (int i = tid; i < 2 * p0; i += blockDim.x) {
    sCs[i] = __ldg(T.cos_tab + i);
    sSn[i] = __ldg(T.sin_tab + i);
  }
  // thread tid holds coefficient c = tid for the phases and degree-major position e = tid for the sums
  const bool active = tid < nc;
  const int c = active ? tid : 0;
  const int pc = __ldg(T.partner + c), m = __ldg(T.m_of_coef + c), n = __ldg(T.n_of_coef + c);
  const bool sine = __ldg(T.is_sin + c);
  const int dm = __ldg(T.perm_off + n) + __ldg(T.pos_in_block + c);
  double own[3], other[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    own[d] = S[(v * 3 + d) * nc + c];
    other[d] = pc >= 0 ? S[(v * 3 + d) * nc + pc] : 0.0;
  }
  const int ce = __ldg(T.perm + c), ne = __ldg(T.n_of_coef + ce);  // the output's coefficient and degree
  const int po = __ldg(T.perm_off + ne), bn = __ldg(T.perm_off + ne + 1) - po;
  const double* M = sM + __ldg(T.mr_off + t * (p0 + 1) + ne) - mbase + (c - po);
  const int rounds = (p0 + JB - 1) / JB;
  for (int r = blockIdx.z; r < rounds; r += gridDim.z) {
    const int j0 = r * JB, nj = min(JB, p0 - j0);
    __syncthreads();
    if (active) {
      int q = (m * j0) % (2 * p0);
#pragma unroll
      for (int jj = 0; jj < JB; jj++) {
        const double cs = sCs[q], sn = sSn[q];
#pragma unroll
        for (int d = 0; d < 3; d++) {
          double val = own[d];
          if (pc >= 0) val = sine ? -other[d] * sn + own[d] * cs : own[d] * cs + other[d] * sn;
          sB[dm * LDB + jj * 3 + d] = val;
        }
        q += m;
        if (q >= 2 * p0) q -= 2 * p0;
      }
    }
    __syncthreads();
    double acc[ND];
#pragma unroll
    for (int u = 0; u < ND; u++) acc[u] = 0.0;
    if (active) {
      const double* b = sB + po * LDB;
      for (int k = 0; k < bn; k++) {
        const double w = M[k * bn];
        double x[ND + (ND & 1)];
#pragma unroll
        for (int u = 0; u < (ND + 1) / 2; u++) {
          const double2 y = reinterpret_cast<const double2*>(b + k * LDB)[u];
          x[2 * u] = y.x;
          x[2 * u + 1] = y.y;
        }
#pragma unroll
        for (int u = 0; u < ND; u++) acc[u] = fma(x[u], w, acc[u]);
      }
    }
    __syncthreads();
    if (active)
#pragma unroll
      for (int u = 0; u < ND; u++) sB[u * nc + ce] = acc[u];
    __syncthreads();
    double* out = R + ((v * (p0 + 1) + t) * p0 + j0) * 3 * (long)nc;
    for (int i = tid; i < nj * 3 * nc; i += blockDim.x) out[i] = sB[i];
  }
}

static int mr_per_t(const DevTables& T) { return T.mr_total / (T.p0 + 1); }

// One rotation of n_fun coefficient vectors: the grid point (latitude t, longitude j) of
// order p0 moved to the x = -1 pole, j in [0, 2 p0) (the step of RotateAll for one (t, j),
// src/SphericalHarmonics.cc:363-449: longitude phase P_j, then the per-degree blocks of
// MatRotate for latitude t). One CTA per function.
__global__ void __launch_bounds__(256) k_rotate_one(const double* __restrict__ S, int p0, int t, int j, DevTables T,
                                                    double* __restrict__ R) {
  extern __shared__ double sB[];  // phase-shifted coefficients [nc]
  const int nc = p0 * (p0 + 2);
  const long f = blockIdx.x;
  const double* s = S + f * nc;
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    const int pc = __ldg(T.partner + c);
    if (pc < 0) {
      sB[c] = s[c];
    } else {
      const int q = (__ldg(T.m_of_coef + c) * j) % (2 * p0);
      const double cs = __ldg(T.cos_tab + q), sn = __ldg(T.sin_tab + q);
      sB[c] = __ldg(T.is_sin + c) ? -s[pc] * sn + s[c] * cs : s[c] * cs + s[pc] * sn;
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    const int n = __ldg(T.n_of_coef + c), bp = __ldg(T.pos_in_block + c);
    const int po = __ldg(T.perm_off + n), bn = __ldg(T.perm_off + n + 1) - po;
    const double* M = T.mr + __ldg(T.mr_off + t * (p0 + 1) + n);
    double acc = 0.0;
    for (int k = 0; k < bn; k++) acc = fma(sB[__ldg(T.perm + po + k)], __ldg(M + k * bn + bp), acc);
    R[f * nc + c] = acc;
  }
}

int launch_rotate_one(const double* S, long n_fun, int t, int j, const DevTables& T, double* R, cudaStream_t st) {
  if (n_fun <= 0) return VES3D_OK;
  const int nc = ncoef_(T.p0);
  k_rotate_one<<<(unsigned)n_fun, 256, nc * sizeof(double), st>>>(S, T.p0, t, j, T, R);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

int launch_rotate_all(const double* S, long nv, const DevTables& T, double* R, cudaStream_t st) {
  if (nv <= 0) return VES3D_OK;
  const int p0 = T.p0;
  const int mpt = mr_per_t(T);
  const size_t nc = ncoef_(p0);
  if (p0 > 127) {  // the on-chip tables hold orders and block positions in one byte
    set_error("rotation kernels support SH orders up to 127");
    return VES3D_ERR_ARG;
  }
  const size_t cap = 227 * 1024;
  int jb = 0;
  size_t smem = 0;
  for (int k : {4, 2, 1}) {
    smem = ((size_t)(k == 4 ? 14 : 3 * k + (k & 1)) * nc + mpt + 4 * p0) * sizeof(double);
    if (smem <= cap) {
      jb = k;
      break;
    }
  }
  if (jb == 0 || nc > kRotAllMax) {
    set_error("RotateAll: the rotation blocks of p = %d do not fit in shared memory", p0);
    return VES3D_ERR_ARG;
  }
  // few vesicles: the phases of a (vesicle, rotation) over several CTAs, up to two per SM
  const int rounds = (p0 + jb - 1) / jb;
  int parts = 1;
  while (parts < rounds && (p0 + 1) * nv * parts < 2 * 148) parts++;
  const dim3 grid(p0 + 1, (unsigned)nv, (unsigned)parts);
  const int nt = ((int)nc + 31) / 32 * 32;
  auto launch = [&](auto kernel) {
    if (const int s = allow_smem(kernel, smem)) return s;
    kernel<<<grid, nt, smem, st>>>(S, p0, mpt, T, R);
    return (int)VES3D_OK;
  };
  const int s = jb == 4 ? launch(k_rotate_all<4>) : jb == 2 ? launch(k_rotate_all<2>) : launch(k_rotate_all<1>);
  if (s) return s;
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// One CTA per rotated surface. Pole targets from the m = 0 block (SHC2Pole, :325-360),
// then for every upsampled source point s (latitude j0) and pole t, with r = target - source,
// n = X_theta x X_phi (area-weighted outward normal), qs = SingularWeights(p1)[t ? j0 : p1 - j0]
// and |r|^-1 := 0 when |r|^2 <= 2^-52 (src/SphericalHarmonics.cc:989-1068):
//   single layer  a1 + r_a r_b a2 with a1 = qs |n| / (8 pi |r|), a2 = a1 / |r|^2
//   double layer  r_a r_b q      with q  = 3 qs (n . r) / (4 pi |r|^5)
template <bool DL>
__global__ void __launch_bounds__(256) k_singular(const double* __restrict__ X, const double* __restrict__ Xt,
                                                  const double* __restrict__ Xp, const double* __restrict__ R,
                                                  int p0, int p1, const double* __restrict__ qp,
                                                  const double* __restrict__ sw, double* __restrict__ K) {
  __shared__ double trg[6];
  const long rot = blockIdx.x;
  const int nc = p0 * (p0 + 2), M1 = 2 * p1 * (p1 + 1);
  if (threadIdx.x < 6) {
    const int c = threadIdx.x >> 1, t = threadIdx.x & 1;
    const double* r = R + (rot * 3 + c) * nc;
    double s = 0.0;
    for (int n = 0; n <= p0; n++) s += r[n] * __ldg(qp + t * (p0 + 1) + n);
    trg[c * 2 + t] = s;
  }
  __syncthreads();
  const double eps = 2.220446049250313e-16;
  const double* x = X + rot * 3 * M1;
  const double* xt = Xt + rot * 3 * M1;
  const double* xp = Xp + rot * 3 * M1;
  double* k = K + rot * 12 * (long)M1;
  for (int s = threadIdx.x; s < M1; s += blockDim.x) {
    const int j0 = s / (2 * p1);
    const double px = x[s], py = x[M1 + s], pz = x[2 * M1 + s];
    const double ax = xt[s], ay = xt[M1 + s], az = xt[2 * M1 + s];
    const double bx = xp[s], by = xp[M1 + s], bz = xp[2 * M1 + s];
    const double nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
    const double area = DL ? 0.0 : sqrt(nx * nx + ny * ny + nz * nz);
#pragma unroll
    for (int t = 0; t < 2; t++) {
      const double dx = trg[t] - px, dy = trg[2 + t] - py, dz = trg[4 + t] - pz;
      const double r2 = dx * dx + dy * dy + dz * dz;
      double rinv = 1.0 / sqrt(r2);
      if (r2 <= eps) rinv = 0.0;
      const double rinv2 = rinv * rinv;
      double* kt = k + (long)t * 6 * M1;
      if (DL) {
        const double q = kDl * __ldg(sw + (t ? j0 : p1 - j0)) * (nx * dx + ny * dy + nz * dz) * (rinv2 * rinv2 * rinv);
        kt[s] = dx * dx * q;
        kt[M1 + s] = dx * dy * q;
        kt[2 * M1 + s] = dx * dz * q;
        kt[3 * M1 + s] = dy * dy * q;
        kt[4 * M1 + s] = dy * dz * q;
        kt[5 * M1 + s] = dz * dz * q;
      } else {
        const double a1 = kInv8Pi * __ldg(sw + (t ? j0 : p1 - j0)) * area * rinv;
        const double a2 = a1 * rinv2;
        kt[s] = a1 + dx * dx * a2;
        kt[M1 + s] = dx * dy * a2;
        kt[2 * M1 + s] = dx * dz * a2;
        kt[3 * M1 + s] = a1 + dy * dy * a2;
        kt[4 * M1 + s] = dy * dz * a2;
        kt[5 * M1 + s] = a1 + dz * dz * a2;
      }
    }
  }
}

int launch_singular_sl(const double* X, const double* Xt, const double* Xp, const double* R, long nrot,
                       const DevTables& T, double* K, cudaStream_t st) {
  if (nrot <= 0) return VES3D_OK;
  k_singular<false><<<(unsigned)nrot, 256, 0, st>>>(X, Xt, Xp, R, T.p0, T.p1, T.qp, T.sing_w, K);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

int launch_singular_dl(const double* X, const double* Xt, const double* Xp, const double* R, long nrot,
                       const DevTables& T, double* K, cudaStream_t st) {
  if (nrot <= 0) return VES3D_OK;
  k_singular<true><<<(unsigned)nrot, 256, 0, st>>>(X, Xt, Xp, R, T.p0, T.p1, T.qp, T.sing_w, K);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// One CTA per (vesicle, latitude rotation t), looping over (pole, component) and over
// chunks of jb longitude rotations. For each input vector a (coefficients of one
// (t, j, pole, comp) function): b = Mr_t^T a per degree block, then the inverse phase
// P_j^T, then scatter into SL3[v][c_in][k][c_out][grid] at grid (t, j) for pole 0 and
// (p0 - t, p0 + j) for pole 1, for both (c_in, c_out) orders of the symmetric component.
// The blocks Mr[t][.] are staged in shared memory; each input vector is stored in
// degree-major order (coefficients of one degree contiguous) so the block products read
// contiguous data, and every thread forms one coefficient for 4 rotations at a time.
constexpr int kRtJ = 4;

__global__ void __launch_bounds__(256) k_rotate_transpose_scatter(const double* __restrict__ C, int p0, int jb,
                                                                  int mr_per_t, DevTables T,
                                                                  double* __restrict__ SL3) {
  extern __shared__ double sm[];
  const int nc = p0 * (p0 + 2), ng = 2 * p0 * (p0 + 1);
  const int lda = nc + 2;      // row padding against bank conflicts between rotations
  double* sA = sm;             // jb * lda, degree-major
  double* sB = sm + jb * lda;  // jb * lda, coefficient order
  double* sM = sm + 2 * jb * lda;
  const int t = blockIdx.x;
  const long v = blockIdx.y;
  const int mbase = __ldg(T.mr_off + t * (p0 + 1));
  for (int i = threadIdx.x; i < mr_per_t; i += blockDim.x) sM[i] = __ldg(T.mr + mbase + i);
  for (int pole = 0; pole < 2; pole++) {
    for (int comp = 0; comp < 6; comp++) {
      for (int j0 = 0; j0 < p0; j0 += jb) {
        const int nj = min(jb, p0 - j0);
        __syncthreads();
        for (int i = threadIdx.x; i < nj * nc; i += blockDim.x) {
          const int jj = i / nc, c = i % nc;
          const int n = __ldg(T.n_of_coef + c);
          const int dm = __ldg(T.perm_off + n) + __ldg(T.pos_in_block + c);
          sA[jj * lda + dm] = C[((((v * (p0 + 1) + t) * p0 + j0 + jj) * 2 + pole) * 6 + comp) * (long)nc + c];
        }
        __syncthreads();
        const int njq = (nj + kRtJ - 1) / kRtJ;
        for (int i = threadIdx.x; i < njq * nc; i += blockDim.x) {
          const int c = i % nc, jq = i / nc;
          const int n = __ldg(T.n_of_coef + c), b = __ldg(T.pos_in_block + c);
          const int po = __ldg(T.perm_off + n), bn = __ldg(T.perm_off + n + 1) - po;
          const double* M = sM + (__ldg(T.mr_off + t * (p0 + 1) + n) - mbase) + b * bn;
          const double* a = sA + jq * kRtJ * lda + po;
          double acc[kRtJ];
#pragma unroll
          for (int q = 0; q < kRtJ; q++) acc[q] = 0.0;
          for (int k = 0; k < bn; k++) {
            const double m = M[k];
#pragma unroll
            for (int q = 0; q < kRtJ; q++) acc[q] = fma(a[q * lda + k], m, acc[q]);
          }
#pragma unroll
          for (int q = 0; q < kRtJ; q++)
            if (jq * kRtJ + q < nj) sB[(jq * kRtJ + q) * lda + c] = acc[q];
        }
        __syncthreads();
        // inverse phase and scatter; consecutive threads take consecutive j for coalescing
        for (int i = threadIdx.x; i < nj * nc; i += blockDim.x) {
          const int jj = i % nj, c = i / nj;
          const int j = j0 + jj;
          const int pc = __ldg(T.partner + c);
          double val;
          if (pc < 0) {
            val = sB[jj * lda + c];
          } else {
            const int q = (__ldg(T.m_of_coef + c) * j) % (2 * p0);
            const double cs = __ldg(T.cos_tab + q), sn = __ldg(T.sin_tab + q);
            if (!__ldg(T.is_sin + c)) {
              val = sB[jj * lda + c] * cs - sB[jj * lda + pc] * sn;
            } else {
              val = sB[jj * lda + pc] * sn + sB[jj * lda + c] * cs;
            }
          }
          const int grid = pole == 0 ? t * 2 * p0 + j : (p0 - t) * 2 * p0 + p0 + j;
          const int cin = comp < 3 ? 0 : (comp < 5 ? 1 : 2), cout = comp < 3 ? comp : (comp < 5 ? comp - 2 : 2);  // (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)
          SL3[(((v * 3 + cin) * nc + c) * 3 + cout) * (long)ng + grid] = val;
          if (cin != cout) SL3[(((v * 3 + cout) * nc + c) * 3 + cin) * (long)ng + grid] = val;
        }
      }
    }
  }
}

// The rotate-transpose per (degree, order) item, in the arithmetic type TV: one CTA per
// (latitude rotation t, vesicle v); for each pole and symmetric component the P longitude
// rows of C are staged in degree-major order, then each thread takes one item (degree n,
// order m) -- the coefficient of cos(m phi) and its sin(m phi) partner (one coefficient for
// m = 0 and m = P) -- and JH of the P rows, and forms the rotation back
//     B[row][po + b] = sum_k A[row][po + k] Mr_{t,n}[b][k]
// at its two positions b, then the inverse longitude phase of the pair in registers. The
// values pass through shared memory (in place of the rows) to the self-matrix grid SL3, laid
// out as the other forms', as whole rows of P consecutive grid values. A thread's rows share
// the staged inputs (broadcast to the lanes of its degree) and its two rotation rows.
// TV = float in the mixed form (C is FP32 after the tensor-core build, FP64 after the FP64 ring
// and rounded when staged; the FP32 grid goes to the FP32 Grid2SHC); TV = double in the FP64
// form (the DMMA kernel below keeps the odd orders).
// Its data (C read and SL3 written once) would take a fifth of its time: what bounds it is
// latency, with few warps per SM beside the tables in shared memory. So the rows of an item are
// split over H threads, the next plane's inputs are sent for while this one is formed (to L2: in
// registers they spill), and the output leaves in 16-byte stores of neighbouring lanes. A thread per
// item that stored its own rows (32 lines per instruction) and now:
//   FP64, p = 16, 512 / 64 vesicles  5.80 -> 3.86 ms / 775 -> 533 us
//   FP32 of FP64, p = 24, 64         5.09 -> 2.30 ms
//   FP32, p = 16, 512                2.84 -> 2.50 ms
// The 16-byte vector of 16 / sizeof(T) values starting at o[i] (destinations 16-byte aligned).
__device__ __forceinline__ float4 vec16(const float* o, int i) { return make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]); }
__device__ __forceinline__ double2 vec16(const double* o, int i) { return make_double2(o[i], o[i + 1]); }

template <int P, typename TV>
struct RtItemCfg {
  static constexpr int NI = (P + 1) * (P + 2) / 2;  // items (n, m <= n), degree-major: n (n + 1) / 2 + m
  static constexpr int NTI = (NI + 31) / 32 * 32;
  static constexpr int W = 16 / sizeof(TV);  // values per 16-byte vector
  // threads per item: whole vectors of rows each
  static constexpr int H = P % (2 * W) == 0 ? 2 : P % (3 * W) == 0 ? 3 : 1;
  static constexpr int JH = P / H, NT = H * NTI;
  // CTAs per SM the registers are sized for (shared memory allows 4 in FP32, 2 in FP64 at p = 16)
  static constexpr int MINB = P <= 8 || (P <= 16 && sizeof(TV) == 4) ? 4 : P <= 12 ? 3 : P <= 16 ? 2 : 1;
  // output row stride: 16-byte stores of eight neighbouring items fall on distinct banks
  static constexpr int LDO = P + (sizeof(TV) == 4 ? (P % 8 == 4 ? 0 : 4) : (P % 4 == 2 ? 0 : 2));
  // values of the rows [P][nc + 1], or of the outputs [2 NI][LDO] that take their place
  static constexpr int SZA = (P * (P * (P + 2) + 1) > 2 * NI * LDO ? P * (P * (P + 2) + 1) : 2 * NI * LDO) + W - 1 & ~(W - 1);
  static_assert(P % W == 0 && JH % W == 0, "rows of whole vectors");
};

template <int P, typename TC, typename TV>
__global__ void __launch_bounds__(RtItemCfg<P, TV>::NT, RtItemCfg<P, TV>::MINB)
    k_rotate_transpose_item(const TC* __restrict__ C, int mr_per_t, DevTables T, TV* __restrict__ SL3) {
  using Cf = RtItemCfg<P, TV>;
  constexpr int nc = P * (P + 2), ng = 2 * P * (P + 1), lda = nc + 1;
  constexpr int NI = Cf::NI, NT = Cf::NT, JH = Cf::JH, W = Cf::W, LDO = Cf::LDO;
  constexpr int LINE = 128 / sizeof(TC);
  using V = decltype(vec16((const TV*)nullptr, 0));
  extern __shared__ __align__(16) unsigned char smraw[];
  TV* sA = reinterpret_cast<TV*>(smraw);  // [P rows][lda], degree-major, then the outputs [2][NI][LDO]
  TV* sM = sA + Cf::SZA;                  // blocks of degree n at sMo[n], rows of bn | 1
  const int msz = mr_per_t + (P + 1) * 2 * P;  // (upper bound of the padded size)
  TV* sCs = sM + msz;                     // cos_tab [2P]
  TV* sSn = sCs + 2 * P;                  // sin_tab [2P]
  int* sMo = reinterpret_cast<int*>(sSn + 2 * P);                        // [P + 2] padded block offsets
  unsigned short* sDm = reinterpret_cast<unsigned short*>(sMo + P + 2);  // degree-major position [nc]
  unsigned short* sOr = sDm + nc;                                        // output row of a coefficient [nc]
  short* sI0 = reinterpret_cast<short*>(sOr + nc);                       // cos (or single) coefficient [NI]
  short* sI1 = sI0 + NI;                                                 // its sin partner or -1 [NI]
  const int t = blockIdx.x;
  const long v = blockIdx.y;
  const int tid = threadIdx.x;
  const TC* Cv = C + (v * (P + 1) + t) * P * 12 * (long)nc;  // [j][pole][comp][c]
  if (tid == 0) {
    int o = 0;
    for (int n = 0; n <= P; n++) {
      sMo[n] = o;
      const int bn = __ldg(T.perm_off + n + 1) - __ldg(T.perm_off + n);
      o += bn * (bn | 1);
    }
    sMo[P + 1] = o;
  }
  for (int i = tid; i < NI; i += NT) sI0[i] = sI1[i] = -1;
  for (int i = tid; i < 2 * P; i += NT) {
    sCs[i] = (TV)__ldg(T.cos_tab + i);
    sSn[i] = (TV)__ldg(T.sin_tab + i);
  }
  __syncthreads();
  for (int c = tid; c < nc; c += NT) {
    const int n = __ldg(T.n_of_coef + c), item = n * (n + 1) / 2 + __ldg(T.m_of_coef + c);
    const bool sine = __ldg(T.is_sin + c);
    sDm[c] = (unsigned short)(__ldg(T.perm_off + n) + __ldg(T.pos_in_block + c));
    sOr[c] = (unsigned short)(item + (sine ? NI : 0));
    (sine ? sI1 : sI0)[item] = (short)c;
  }
  // the rotation blocks of this t, rows padded to bn | 1
  for (int n = 0; n <= P; n++) {
    const int bn = __ldg(T.perm_off + n + 1) - __ldg(T.perm_off + n);
    const double* M = T.mr + __ldg(T.mr_off + t * (P + 1) + n);
    for (int i = tid; i < bn * bn; i += NT) {
      const int b = i / bn, k = i - b * bn;
      sM[sMo[n] + b * (bn | 1) + k] = (TV)__ldg(M + i);
    }
  }
  __syncthreads();
  // this thread's item and first row
  const int item = tid % Cf::NTI, j0 = tid / Cf::NTI * JH;
  int n = 0;
  while ((n + 1) * (n + 2) / 2 <= item && n < P) n++;
  const bool active = item < NI && sI0[item] >= 0;  // (every (n, m <= n) has its cos coefficient)
  const int m = active ? item - n * (n + 1) / 2 : 0;
  const int c0 = active ? sI0[item] : 0, c1 = active ? sI1[item] : -1;
  const int po = __ldg(T.perm_off + n), bn = __ldg(T.perm_off + n + 1) - po;
  const TV* M0 = active ? sM + sMo[n] + (sDm[c0] - po) * (bn | 1) : sM;
  const TV* M1 = c1 >= 0 ? sM + sMo[n] + (sDm[c1] - po) * (bn | 1) : M0;
  for (int pc = blockIdx.z; pc < 12; pc += gridDim.z) {
    const int pole = pc / 6, comp = pc - 6 * pole;
    const int grid0 = pole == 0 ? t * 2 * P : (P - t) * 2 * P + P;
    // stage A[j][dm(c)], eight loads in flight per thread
#pragma unroll 1
    for (int i0 = tid; i0 < P * nc; i0 += NT * 8) {
      TC val[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = i0 + u * NT, j = i / nc;
        if (i < P * nc) val[u] = Cv[((long)j * 12 + pc) * nc + (i - j * nc)];
      }
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = i0 + u * NT, j = i / nc;
        if (i < P * nc) sA[j * lda + sDm[i - j * nc]] = (TV)val[u];
      }
    }
    __syncthreads();
    // the next plane on its way to L2
    if (pc + gridDim.z < 12)
      for (int i = tid; i < P * ((nc + LINE - 1) / LINE); i += NT) {
        const int j = i % P, l = i / P;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(Cv + ((long)j * 12 + pc + gridDim.z) * nc + min(l * LINE, nc - 1)));
      }
    TV acc0[JH], acc1[JH];
#pragma unroll
    for (int j = 0; j < JH; j++) acc0[j] = acc1[j] = TV(0);
    if (active) {
      const TV* a = sA + j0 * lda + po;
      for (int k = 0; k < bn; k++) {
        const TV m0 = M0[k], m1 = M1[k];
#pragma unroll
        for (int j = 0; j < JH; j++) {
          const TV x = a[j * lda + k];
          acc0[j] = fma(x, m0, acc0[j]);
          acc1[j] = fma(x, m1, acc1[j]);
        }
      }
      // inverse longitude phase of the pair: cos row c0, sin row c1
      if (c1 >= 0) {
#pragma unroll
        for (int j = 0; j < JH; j++) {
          const int q = (m * (j0 + j)) % (2 * P);
          const TV cs = sCs[q], sn = sSn[q];
          const TV x0 = acc0[j], x1 = acc1[j];
          acc0[j] = fma(-x1, sn, x0 * cs);
          acc1[j] = fma(x0, sn, x1 * cs);
        }
      }
    }
    __syncthreads();
    if (active) {
      V* o = reinterpret_cast<V*>(sA + item * LDO + j0);
#pragma unroll
      for (int q = 0; q < JH / W; q++) {
        o[q] = vec16(acc0, W * q);
        if (c1 >= 0) o[q + NI * LDO / W] = vec16(acc1, W * q);
      }
    }
    __syncthreads();
    // symmetric component -> (c_in, c_out): (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)
    const int cin = comp < 3 ? 0 : (comp < 5 ? 1 : 2), cout = comp < 3 ? comp : (comp < 5 ? comp - 2 : 2);
    TV* d0 = SL3 + ((v * 3 + cin) * nc * 3 + cout) * (long)ng + grid0;
    TV* d1 = SL3 + ((v * 3 + cout) * nc * 3 + cin) * (long)ng + grid0;
#pragma unroll 4
    for (int i = tid; i < nc * (P / W); i += NT) {
      const int c = i / (P / W), q = i - c * (P / W);
      const V w = reinterpret_cast<const V*>(sA + sOr[c] * LDO)[q];
      reinterpret_cast<V*>(d0 + (long)c * 3 * ng)[q] = w;
      if (cin != cout) reinterpret_cast<V*>(d1 + (long)c * 3 * ng)[q] = w;
    }
    __syncthreads();
  }
}

template <int P, typename TV>
static size_t rt_item_smem(int mpt) {
  const size_t fl = (size_t)RtItemCfg<P, TV>::SZA + mpt + (size_t)(P + 1) * 2 * P + 4 * P;
  return fl * sizeof(TV) + (size_t)(P + 2) * sizeof(int) + (size_t)P * (P + 2) * 4 + (size_t)RtItemCfg<P, TV>::NI * 4 + 16;
}

template <int P, typename TC, typename TV = float>
static int launch_rt_item(const TC* C, long nv, const DevTables& T, TV* SL3, cudaStream_t st) {
  const int mpt = mr_per_t(T);
  // few vesicles: the 12 (pole, component) planes of a (vesicle, rotation) over several CTAs, up to
  // four per SM (each plane's arithmetic stays as it is)
  int planes = 1;
  while (planes < 12 && (P + 1) * nv * planes < 4 * 148) planes = planes < 4 ? planes + 1 : planes == 4 ? 6 : 12;
  dim3 grid(P + 1, (unsigned)nv, (unsigned)planes);
  const size_t smem = rt_item_smem<P, TV>(mpt);  // FP32: 53 KB at p = 16 (four CTAs per SM), 163 KB at p = 24
  VES3D_CK(cudaFuncSetAttribute(k_rotate_transpose_item<P, TC, TV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem));
  k_rotate_transpose_item<P, TC, TV><<<grid, RtItemCfg<P, TV>::NT, smem, st>>>(C, mpt, T, SL3);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

int launch_rotate_transpose_f32(const float* C, long nv, const DevTables& T, float* SL3, cudaStream_t st) {
  if (nv <= 0) return VES3D_OK;
  // the FP32 results come from the tensor-core build, which is laid out for p = 16 only
  if (T.p0 != 16) {
    set_error("internal: FP32 rotate-transpose at p = %d (built for p = 16)", T.p0);
    return VES3D_ERR_ARG;
  }
  return launch_rt_item<16>(C, nv, T, SL3, st);
}

bool rotate_transpose_f32_from_f64_supported(int p0) { return p0 == 12 || p0 == 24; }

int launch_rotate_transpose_f32(const double* C, long nv, const DevTables& T, float* SL3, cudaStream_t st) {
  if (nv <= 0) return VES3D_OK;
  switch (T.p0) {
    case 12: return launch_rt_item<12>(C, nv, T, SL3, st);
    case 24: return launch_rt_item<24>(C, nv, T, SL3, st);
    default: break;
  }
  set_error("internal: FP32 rotate-transpose of FP64 results at p = %d (built for p in {12, 24})", T.p0);
  return VES3D_ERR_ARG;
}

// VES3D_TC_ROTATE=0 selects the CUDA-core form of the rotate-transpose (for comparison).
static bool tc_rotate_disabled() {
  static const bool off = [] {
    const char* e = getenv("VES3D_TC_ROTATE");
    return e && e[0] == '0';
  }();
  return off;
}

constexpr int kRtMaxK = 8;  // K steps of 4: rotation blocks up to 32 wide (p0 <= 16)

__device__ __forceinline__ void dmma_rt(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Row stride >= n with stride = 4 (mod 16) doubles: conflict-free m8n8k4 A fragments.
__host__ __device__ constexpr int pad4_16(int n) { return ((n + 11) / 16) * 16 + 4; }

// RotateTranspose + inverse phase + Rearrange on the FP64 tensor cores. One CTA per
// (latitude rotation t, vesicle v); rows are (pole, component, longitude j), processed in
// blocks of cb components x p0 longitudes. A block's coefficients are staged degree-major
// in shared memory; for every degree n the rotation back is one GEMM
//     Out[row][b] = sum_k In[row][po(n) + k] * M_{t,n}[b][k]       (b, k < bn)
// on mma.sync m8n8k4 (A = In from shared memory, B = M from the L1/L2-resident table,
// masked to the block), written back in place after a barrier; reads of the K padding
// land in the next degree's (finite) columns and meet zeros in B. Then the longitude
// phase is undone and the values are scattered into the self-matrix grid layout, as in
// k_rotate_transpose_scatter.
__global__ void __launch_bounds__(256, 2) k_rotate_transpose_tc(const double* __restrict__ C, int p0, int cb, int ldi,
                                                                DevTables T, double* __restrict__ SL3) {
  extern __shared__ __align__(16) double sm[];
  const int nc = p0 * (p0 + 2), ng = 2 * p0 * (p0 + 1);
  const int rows = cb * p0, rows8 = (rows + 7) & ~7;
  double* sIn = sm;                                                        // rows8 x ldi
  double* sCs = sm + (size_t)rows8 * ldi;                                  // cos_tab [2 p0]
  double* sSn = sCs + 2 * p0;                                              // sin_tab [2 p0]
  unsigned short* sDm = reinterpret_cast<unsigned short*>(sSn + 2 * p0);   // degree-major position [nc]
  short* sPc = reinterpret_cast<short*>(sDm + nc);                        // partner (or -1) [nc]
  unsigned char* sMs = reinterpret_cast<unsigned char*>(sPc + nc);        // m | (is_sin << 7) [nc]
  const int t = blockIdx.x;
  const long v = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int grow = lane >> 2, gcol = lane & 3;
  // per-coefficient tables of the phase / scatter step, on chip (the L1 left beside the
  // staging buffer is small, and every element needs them)
  for (int c = tid; c < nc; c += 256) {
    sDm[c] = (unsigned short)(__ldg(T.perm_off + __ldg(T.n_of_coef + c)) + __ldg(T.pos_in_block + c));
    sPc[c] = (short)__ldg(T.partner + c);
    sMs[c] = (unsigned char)(__ldg(T.m_of_coef + c) | (__ldg(T.is_sin + c) ? 0x80 : 0));
  }
  for (int i = tid; i < 2 * p0; i += 256) {
    sCs[i] = __ldg(T.cos_tab + i);
    sSn[i] = __ldg(T.sin_tab + i);
  }
  // zero the K padding of every row and the padding rows once (never overwritten)
  for (int i = tid; i < rows8 * ldi; i += 256) {
    const int r = i / ldi, col = i - r * ldi;
    if (r >= rows || col >= nc) sIn[i] = 0.0;
  }
  const int mtiles = rows8 / 8;
  for (int pole = 0; pole < 2; pole++) {
    for (int comp0 = 0; comp0 < 6; comp0 += cb) {
      __syncthreads();
      // stage: In[(cc, j)][dm(c)] = C[v][t][j][pole][comp0 + cc][c], eight loads in flight
      // per thread before the shared-memory stores
      for (int i0 = tid; i0 < rows * nc; i0 += 256 * 8) {
        double val[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int i = i0 + u * 256;
          if (i < rows * nc) {
            const int r = i / nc, c = i - r * nc;
            const int cc = r / p0, j = r - cc * p0;
            val[u] = C[((((v * (p0 + 1) + t) * p0 + j) * 2 + pole) * 6 + comp0 + cc) * (long)nc + c];
          }
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int i = i0 + u * 256;
          if (i < rows * nc) {
            const int r = i / nc, c = i - r * nc;
            sIn[r * ldi + sDm[c]] = val[u];
          }
        }
      }
      __syncthreads();
      for (int n = 0; n <= p0; n++) {
        const int po = __ldg(T.perm_off + n), bn = __ldg(T.perm_off + n + 1) - po;
        const double* M = T.mr + __ldg(T.mr_off + t * (p0 + 1) + n);
        const int ntiles = (bn + 7) / 8, ksteps = (bn + 3) / 4;
        const int nitems = mtiles * ntiles;
        // at most 3 items per warp held in registers across the barrier (nitems <= 24
        // for rows8 <= 48 and bn <= 32; larger problems loop in rounds)
        for (int base = 0; base < nitems; base += 24) {
          double acc[3][2];
          int item[3];
#pragma unroll
          for (int q = 0; q < 3; q++) {
            item[q] = base + warp + 8 * q;
            acc[q][0] = acc[q][1] = 0.0;
            if (item[q] < nitems) {
              const int mt = item[q] / ntiles, nt = item[q] - mt * ntiles;
              const double* a = sIn + (mt * 8 + grow) * ldi + po + gcol;
              const int nn = nt * 8 + grow;
              // B fragments first (independent loads in flight together), then the MMAs
              double bv[kRtMaxK];
#pragma unroll
              for (int ks = 0; ks < kRtMaxK; ks++) {
                const int kk = ks * 4 + gcol;
                bv[ks] = (ks < ksteps && nn < bn && kk < bn) ? __ldg(M + nn * bn + kk) : 0.0;
              }
#pragma unroll
              for (int ks = 0; ks < kRtMaxK; ks++)
                if (ks < ksteps) dmma_rt(acc[q][0], acc[q][1], a[ks * 4], bv[ks]);
            }
          }
          __syncthreads();
#pragma unroll
          for (int q = 0; q < 3; q++) {
            if (item[q] < nitems) {
              const int mt = item[q] / ntiles, nt = item[q] - mt * ntiles;
              const int row = mt * 8 + grow, col = nt * 8 + 2 * gcol;
              if (row < rows) {
                if (col < bn) sIn[row * ldi + po + col] = acc[q][0];
                if (col + 1 < bn) sIn[row * ldi + po + col + 1] = acc[q][1];
              }
            }
          }
          __syncthreads();
        }
      }
      // inverse phase and scatter; consecutive threads take consecutive j
      for (int i = tid; i < rows * nc; i += 256) {
        const int j = i % p0, rest = i / p0;
        const int c = rest % nc, cc = rest / nc;
        const double* in = sIn + (cc * p0 + j) * ldi;
        const int pc = sPc[c];
        double val;
        if (pc < 0) {
          val = in[sDm[c]];
        } else {
          const int ms = sMs[c];
          const int q = ((ms & 0x7f) * j) % (2 * p0);
          const double cs = sCs[q], sn = sSn[q];
          if (!(ms & 0x80))
            val = in[sDm[c]] * cs - in[sDm[pc]] * sn;
          else
            val = in[sDm[pc]] * sn + in[sDm[c]] * cs;
        }
        const int grid = pole == 0 ? t * 2 * p0 + j : (p0 - t) * 2 * p0 + p0 + j;
        const int comp = comp0 + cc;
        const int cin = comp < 3 ? 0 : (comp < 5 ? 1 : 2), cout = comp < 3 ? comp : (comp < 5 ? comp - 2 : 2);  // (0,0) (0,1) (0,2) (1,1) (1,2) (2,2)
        SL3[(((v * 3 + cin) * nc + c) * 3 + cout) * (long)ng + grid] = val;
        if (cin != cout) SL3[(((v * 3 + cout) * nc + c) * 3 + cin) * (long)ng + grid] = val;
      }
    }
  }
}

int launch_rotate_transpose_scatter(const double* C, long nv, const DevTables& T, double* SL3, cudaStream_t st) {
  if (nv <= 0) return VES3D_OK;
  const int p0 = T.p0, nc = ncoef_(p0);
  // the per-item kernel in FP64 at its even orders (p = 16: 3.9 ms per 512-vesicle build against
  // 9.5 ms for the DMMA form below, which keeps the odd orders; p = 12, 8 vesicles: 51 against 128 us;
  // whole builds of 27 vesicles at p = 4 38 against 54 us, p = 20 4.9 against 7.6 ms)
  if (!tc_rotate_disabled()) switch (p0) {
      case 4: return launch_rt_item<4, double, double>(C, nv, T, SL3, st);
      case 6: return launch_rt_item<6, double, double>(C, nv, T, SL3, st);
      case 8: return launch_rt_item<8, double, double>(C, nv, T, SL3, st);
      case 10: return launch_rt_item<10, double, double>(C, nv, T, SL3, st);
      case 12: return launch_rt_item<12, double, double>(C, nv, T, SL3, st);
      case 14: return launch_rt_item<14, double, double>(C, nv, T, SL3, st);
      case 16: return launch_rt_item<16, double, double>(C, nv, T, SL3, st);
      case 18: return launch_rt_item<18, double, double>(C, nv, T, SL3, st);
      case 20: return launch_rt_item<20, double, double>(C, nv, T, SL3, st);
      default: break;
    }
  {
    // tensor-core form: the largest component block (3, 2 or 1 components x p0 rows)
    // whose staging fits two CTAs per SM; 6 must be a multiple of the block
    const int ldi = pad4_16(nc + 3);
    for (int cb : {3, 2, 1}) {
      const int rows8 = ((cb * p0) + 7) & ~7;
      const size_t smem = ((size_t)rows8 * ldi + 4 * p0) * sizeof(double) + ((size_t)nc * 5 + 15) / 16 * 16;
      if (p0 <= 16 && smem <= 113 * 1024 && !tc_rotate_disabled()) {
        if (const int s = allow_smem(k_rotate_transpose_tc, smem)) return s;
        dim3 grid(p0 + 1, (unsigned)nv);
        k_rotate_transpose_tc<<<grid, 256, smem, st>>>(C, p0, cb, ldi, T, SL3);
        VES3D_LAUNCHED();
        return VES3D_OK;
      }
    }
  }
  const int mpt = mr_per_t(T);
  // two CTAs per SM: keep shared memory under ~110 KB; whole groups of kRtJ rotations
  long budget = (110 * 1024) / (long)sizeof(double) - mpt;
  int jb = (int)(budget / (2 * (long)(nc + 2)));
  jb = (jb / kRtJ) * kRtJ;
  if (jb > p0) jb = ((p0 + kRtJ - 1) / kRtJ) * kRtJ;
  if (jb < kRtJ) jb = kRtJ;
  size_t smem = ((size_t)2 * jb * (nc + 2) + mpt) * sizeof(double);
  if (smem > 48 * 1024)
    if (const int s = allow_smem(k_rotate_transpose_scatter, smem)) return s;
  dim3 grid(p0 + 1, (unsigned)nv);
  k_rotate_transpose_scatter<<<grid, 256, smem, st>>>(C, p0, jb, mpt, T, SL3);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// V[v][col] = sum_row F[v][row] * SL[v][row][col]. A CTA takes 32 VEC columns; its warps share the
// rows, eight row loads of VEC consecutive columns in flight per lane, and their sums are added in
// warp order. Bound by the one read of SL: a thread per column with four loads in flight ran
// 32 vesicles of p = 16 (191 MB) in 229 us, latency-bound on 224 CTAs; now 43 us (4.4 TB/s). 64
// vesicles 234 -> 68 us, 512 vesicles (3.06 GB) 555 -> 442 us (6.9 TB/s).
constexpr int kGemvWarps = 8;

template <bool ACC, int VEC>
__global__ void __launch_bounds__(32 * kGemvWarps) k_self_gemv(const double* __restrict__ F,
                                                               const double* __restrict__ SL, int n,
                                                               double* __restrict__ V) {
  __shared__ double red[kGemvWarps][32 * VEC];
  const long v = blockIdx.y;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = (blockIdx.x * 32 + lane) * VEC;
  const double* f = F + v * n;
  double s[VEC];
#pragma unroll
  for (int k = 0; k < VEC; k++) s[k] = 0.0;
  if (col < n) {
    const double* M = SL + v * (long)n * n + col;
    constexpr int U = 8;
    int r = w;
    for (; r + (U - 1) * kGemvWarps < n; r += U * kGemvWarps) {
      double m[U][VEC], x[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const double* row = M + (long)(r + u * kGemvWarps) * n;
        if (VEC == 2) {
          const double2 a = __ldg(reinterpret_cast<const double2*>(row));
          m[u][0] = a.x;
          m[u][VEC - 1] = a.y;
        } else {
          m[u][0] = __ldg(row);
        }
        x[u] = __ldg(f + r + u * kGemvWarps);
      }
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int k = 0; k < VEC; k++) s[k] = fma(x[u], m[u][k], s[k]);
    }
    for (; r < n; r += kGemvWarps)
#pragma unroll
      for (int k = 0; k < VEC; k++) s[k] = fma(__ldg(f + r), __ldg(M + (long)r * n + k), s[k]);
  }
#pragma unroll
  for (int k = 0; k < VEC; k++) red[w][lane * VEC + k] = s[k];
  __syncthreads();
  const int c = blockIdx.x * 32 * VEC + threadIdx.x;
  if (threadIdx.x < 32 * VEC && c < n) {
    double sum = 0.0;
#pragma unroll
    for (int q = 0; q < kGemvWarps; q++) sum += red[q][threadIdx.x];
    V[v * n + c] = ACC ? V[v * n + c] + sum : sum;
  }
}

// Several density vectors per vesicle at once (batched operator applications):
// V[q nv + v][col] = sum_row F[q nv + v][row] SL[v][row][col], q < nvec; every SL column is
// read once for all nvec vectors (the single-vector form reads it per vector).
constexpr int kGemvMaxVec = 8;
template <bool ACC>
__global__ void __launch_bounds__(128) k_self_gemv_multi(const double* __restrict__ F, const double* __restrict__ SL,
                                                         long nv, int nvec, int n, double* __restrict__ V) {
  extern __shared__ double sF[];  // [nvec][n]
  const long v = blockIdx.y;
  for (int i = threadIdx.x; i < nvec * n; i += blockDim.x) {
    const int q = i / n, r = i - q * n;
    sF[i] = F[((long)q * nv + v) * n + r];
  }
  __syncthreads();
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= n) return;
  const double* M = SL + v * (long)n * n + col;
  double acc[kGemvMaxVec];
#pragma unroll
  for (int q = 0; q < kGemvMaxVec; q++) acc[q] = 0.0;
  for (int r = 0; r < n; r++) {
    const double m = __ldg(M + (long)r * n);
#pragma unroll
    for (int q = 0; q < kGemvMaxVec; q++)
      if (q < nvec) acc[q] = fma(sF[q * n + r], m, acc[q]);
  }
#pragma unroll
  for (int q = 0; q < kGemvMaxVec; q++)
    if (q < nvec) {
      double* o = V + ((long)q * nv + v) * n + col;
      *o = ACC ? *o + acc[q] : acc[q];
    }
}

int launch_self_gemv_multi(const double* F, const double* SL, long nv, int nvec, int n, double* V, cudaStream_t st,
                           bool accumulate) {
  if (nv <= 0 || nvec <= 0) return VES3D_OK;
  if (nvec > kGemvMaxVec) {
    set_error("launch_self_gemv_multi: at most %d vectors", kGemvMaxVec);
    return VES3D_ERR_ARG;
  }
  dim3 grid((n + 127) / 128, (unsigned)nv);
  const size_t smem = (size_t)nvec * n * sizeof(double);
  if (accumulate) {
    if (smem > 48 * 1024)
      if (const int s = allow_smem(k_self_gemv_multi<true>, smem)) return s;
    k_self_gemv_multi<true><<<grid, 128, smem, st>>>(F, SL, nv, nvec, n, V);
  } else {
    if (smem > 48 * 1024)
      if (const int s = allow_smem(k_self_gemv_multi<false>, smem)) return s;
    k_self_gemv_multi<false><<<grid, 128, smem, st>>>(F, SL, nv, nvec, n, V);
  }
  VES3D_LAUNCHED();
  return VES3D_OK;
}

int launch_self_gemv(const double* F, const double* SL, long nv, int n, double* V, cudaStream_t st, bool accumulate) {
  if (nv <= 0) return VES3D_OK;
  // 16-byte loads need even rows (n = 3 p (p + 2) is odd for odd p)
  const int vec = n % 2 == 0 ? 2 : 1;
  const dim3 grid((n + 32 * vec - 1) / (32 * vec), (unsigned)nv);
  auto kernel = vec == 2 ? (accumulate ? k_self_gemv<true, 2> : k_self_gemv<false, 2>)
                         : (accumulate ? k_self_gemv<true, 1> : k_self_gemv<false, 1>);
  kernel<<<grid, 32 * kGemvWarps, 0, st>>>(F, SL, n, V);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

}  // namespace ves3d
