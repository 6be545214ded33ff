// Grid2SHC(p, p) of FP64 grid functions (src/SphericalHarmonics.cc:152-235) at the usual orders, by
// the grid's symmetries: latitudes l and p - l meet the even and the odd degrees of a block as their
// sum and difference, and the longitudes j, -j, p - j, p + j the cosines and sines of even and odd
// m, which leaves 10 of the dense transform's 22 thousand multiply-adds per function at p = 16.
//
// Persistent CTAs of one thread per coefficient, which keeps its Legendre row in registers, walk
// rounds of FB functions: the next round's grid values arrive by cp.async while this one's rows go
// through the folded DFT (a thread per row and parity of m, its factors constant operands) and the
// Legendre sums (shared-memory reads that a block's coefficients share). Bound by the FP64 pipe and
// the shared-memory reads together; the dense form on FP64 tensor cores took 5.37 ms for the build of
// 512 vesicles at p = 16 (1.3 million functions), this 3.63 (64 vesicles 709 -> 476 us).
#include <algorithm>

#include "common.cuh"
#include "cos_table.cuh"
#include "kernels.h"

namespace ves3d {

namespace {

template <int P>
struct G2sCfg {
  static constexpr int NLON = 2 * P, NC = P * (P + 2), NG = NLON * (P + 1), H = P / 2 + 1;
  static constexpr int NT = (NC + 31) / 32 * 32;
  static constexpr int FB = P <= 8 ? 4 : P <= 16 ? 8 : 6;          // functions per round
  static constexpr int MINB = P <= 8 ? 4 : P <= 16 ? 2 : 1;
  static constexpr int LD = NLON + 1;                              // row strides (odd)
  static constexpr int SZ_X = FB * (P + 1) * LD, SZ_G = FB * 2 * H * LD;
  static constexpr size_t SMEM = (size_t)(2 * SZ_X + SZ_G) * sizeof(double);
};

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The DFT sums of parity PAR of the row a + sign b (b null: a alone), unscaled.
template <int P, int PAR>
__device__ __forceinline__ void fold_row(const double* __restrict__ a, const double* __restrict__ b, double sign,
                                         double* __restrict__ out) {
  constexpr int N = 2 * P, NM = (P - PAR) / 2 + 1;
  double c[NM], s[NM];
#pragma unroll
  for (int i = 0; i < NM; i++) c[i] = s[i] = 0.0;
#pragma unroll
  for (int j = 0; j <= P / 2; j++) {
    auto at = [&](int k) { return fma(sign, b[k], a[k]); };
    const double v1 = at(j), v2 = j ? at(N - j) : 0.0, v3 = 2 * j == P ? 0.0 : at(P - j),
                 v4 = j == 0 || 2 * j == P ? 0.0 : at(P + j);
    const double fc = PAR ? (v1 + v2) - (v3 + v4) : (v1 + v2) + (v3 + v4);
    const double fs = PAR ? (v1 - v2) + (v3 - v4) : (v1 - v2) - (v3 - v4);
#pragma unroll
    for (int i = 0; i < NM; i++) {
      const int m = PAR + 2 * i;
      c[i] = fma(fc, c_cos<N>.v[(m * j) % N], c[i]);
      if (m > 0 && m < P) s[i] = fma(fs, c_cos<N>.v[(m * j + 3 * N / 4) % N], s[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < NM; i++) {
    const int m = PAR + 2 * i;
    out[m ? 2 * m - 1 : 0] = c[i];
    if (m > 0 && m < P) out[2 * m] = s[i];
  }
}

template <int P>
__global__ void __launch_bounds__(G2sCfg<P>::NT, G2sCfg<P>::MINB)
    k_grid2shc(const double* __restrict__ in, long nfun, const double* __restrict__ leg, const int* __restrict__ jf,
               double* __restrict__ out) {
  using C = G2sCfg<P>;
  extern __shared__ __align__(16) double sm[];
  double* sG = sm + 2 * C::SZ_X;
  const int tid = threadIdx.x;
  const bool has_c = tid < C::NC;
  const int k = has_c ? __ldg(jf + tid) : 0, m = (k + 1) >> 1;
  int par = 0;  // parity of the degree within its block
  double lr[C::H];
  {
    // first coefficient of block k: its place in the block gives the degree
    int c0 = 0;
    if (k > 0) {
      const int full = P + 1 + 2 * ((m - 1) * (P + 1) - (m - 1) * m / 2);
      c0 = (k & 1) ? full : full + P + 1 - m;
    }
    par = has_c ? (tid - c0) & 1 : 0;
    // weights and the DFT's factor 1 / (sqrt(2 pi) p), half at m = 0 and p
    const double e = (m == 0 || m == P ? 0.5 : 1.0) * 0.3989422804014327 / P;
#pragma unroll
    for (int l = 0; l < C::H; l++) lr[l] = has_c ? __ldg(leg + tid * (P + 1) + l) * e : 0.0;
  }
  const long nround = (nfun + C::FB - 1) / C::FB;
  auto load = [&](long r, double* dst) {
    const long f0 = r * C::FB;
    const int n = (int)min((long)C::FB, nfun - f0) * C::NG;
    const double* src = in + f0 * C::NG;
    for (int i = tid; i < n; i += C::NT) {
      const int row = i / C::NLON, j = i - row * C::NLON;
      cp_async8(dst + row * C::LD + j, src + i);
    }
  };
  if ((long)blockIdx.x < nround) load(blockIdx.x, sm);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int buf = 0;
  for (long r = blockIdx.x; r < nround; r += gridDim.x, buf ^= 1) {
    const double* sX = sm + buf * C::SZ_X;
    if (r + gridDim.x < nround) load(r + gridDim.x, sm + (buf ^ 1) * C::SZ_X);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // this round's rows are in; the last round's Legendre sums are done
    const long f0 = r * C::FB;
    const int nf = (int)min((long)C::FB, nfun - f0), rows = nf * 2 * C::H;
    for (int i = tid; i < 2 * rows; i += C::NT) {
      const int odd_m = i >= rows, q = i - (odd_m ? rows : 0), f = q / (2 * C::H), l = (q - f * 2 * C::H) >> 1;
      const double* a = sX + (f * (P + 1) + l) * C::LD;
      const double* b = sX + (f * (P + 1) + P - l) * C::LD;
      const double sign = 2 * l == P ? 0.0 : (q & 1) ? -1.0 : 1.0;  // the middle latitude has no partner
      if (odd_m)
        fold_row<P, 1>(a, b, sign, sG + q * C::LD);
      else
        fold_row<P, 0>(a, b, sign, sG + q * C::LD);
    }
    __syncthreads();
    if (has_c) {
      const double* g = sG + par * C::LD + k;
      for (int f = 0; f < nf; f++, g += 2 * C::H * C::LD) {
        double s = 0.0, t = 0.0;
#pragma unroll
        for (int l = 0; l < C::H; l += 2) {
          s = fma(g[2 * l * C::LD], lr[l], s);
          if (l + 1 < C::H) t = fma(g[(2 * l + 2) * C::LD], lr[l + 1], t);
        }
        out[(f0 + f) * C::NC + tid] = s + t;
      }
    }
  }
}

template <int P>
int launch_g2s(const double* in, long nfun, const double* leg, const int* jf, double* out, cudaStream_t st) {
  using C = G2sCfg<P>;
  VES3D_CK(cudaFuncSetAttribute(k_grid2shc<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
  int dev = 0, nsm = 148, per = 1;
  VES3D_CK(cudaGetDevice(&dev));
  VES3D_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  VES3D_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_grid2shc<P>, C::NT, C::SMEM));
  const long grid = std::min((nfun + C::FB - 1) / C::FB, (long)nsm * std::max(per, 1));
  k_grid2shc<P><<<(unsigned)grid, C::NT, C::SMEM, st>>>(in, nfun, leg, jf, out);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

}  // namespace

// Even orders from 6 to 20, and 24. 27 vesicles' builds with it against the dense forms: p = 6 65 and
// 73 us, p = 12 563 and 606, p = 20 4.9 and 8.6 ms, p = 24 19.1 and 27.9 ms; at p = 4 the dense form on
// tensor cores is the faster (two vesicles 30 against 32 us).
bool grid2shc_folded(int p) { return p >= 6 && p <= 24 && p % 2 == 0 && p != 22; }

int launch_grid2shc_folded(const double* in, long nfun, int p, const double* leg, const int* jf, double* out,
                           cudaStream_t st) {
  switch (p) {
    case 6: return launch_g2s<6>(in, nfun, leg, jf, out, st);
    case 8: return launch_g2s<8>(in, nfun, leg, jf, out, st);
    case 10: return launch_g2s<10>(in, nfun, leg, jf, out, st);
    case 12: return launch_g2s<12>(in, nfun, leg, jf, out, st);
    case 14: return launch_g2s<14>(in, nfun, leg, jf, out, st);
    case 16: return launch_g2s<16>(in, nfun, leg, jf, out, st);
    case 18: return launch_g2s<18>(in, nfun, leg, jf, out, st);
    case 20: return launch_g2s<20>(in, nfun, leg, jf, out, st);
    case 24: return launch_g2s<24>(in, nfun, leg, jf, out, st);
    default: break;
  }
  set_error("internal: folded Grid2SHC at p = %d", p);
  return VES3D_ERR_ARG;
}

}  // namespace ves3d
