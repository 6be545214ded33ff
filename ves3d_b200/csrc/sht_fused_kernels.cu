// The SHTrans entry points' transforms at one order, in one launch each: analysis, synthesis, and
// analysis - scaling - synthesis (the frequency filters). Math as in sht_kernels.cu.
//
// The tables (Gauss-Legendre nodes and weights, normalised Legendre functions of half the
// latitudes, cosines and sines) are formed by every CTA in shared memory, a few microseconds of
// latency, instead of on the host: building, allocating, uploading and freeing them took 360 us of
// each call against 50 us of kernels. Rows are folded by the grid's symmetries first -- latitudes l
// and p - l, longitudes j, -j, p - j and p + j -- which leaves 7.8 thousand multiply-adds per
// function at p = 16 of the dense transform's 22. 768 functions of p = 16: 17.8 us analysis, 18.8 us
// synthesis, 26.8 us filter, bound by the latency of forming the tables and one wave of CTAs; the three
// calls with their set-up took 1,097 us, now 99.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace ves3d {

namespace {

constexpr int kShtMaxP = 32;
constexpr int kShtThreads = 256;
enum { kShtForward, kShtBackward, kShtFilter };

struct ShtArgs {
  const double* in;
  double* out;
  long nfun;
  int p, fb;                    // functions per CTA and round
  double scale[kShtMaxP + 1];   // the filter's factor of each degree
};

struct ShtLayout {
  int J, H, ldq, x, s, w, ab, ca, cb, dg, q, tw, deg, koc, fold, g, coef, total;
};

__host__ __device__ inline ShtLayout sht_layout(int p, int fb, int mode) {
  ShtLayout L;
  const int nc = p * (p + 2);
  L.J = (p / 2 + 1) | 1;  // folded longitudes, padded to an odd stride
  L.H = p / 2 + 1;        // latitude pairs
  L.ldq = nc | 1;
  int o = 0;
  auto take = [&](int n) {
    const int at = o;
    o += n;
    return at;
  };
  L.x = take(L.H);
  L.s = take(L.H);
  L.w = take(L.H);
  L.ab = take(2 * (p + 2));
  L.ca = take((p + 1) * (p + 1));
  L.cb = take((p + 1) * (p + 1));
  L.dg = take(p + 1);
  L.q = take(L.H * L.ldq);
  L.tw = take(2 * p * L.J);
  L.deg = take((nc + 7) / 8 + 1);       // degree of each coefficient (unsigned char)
  L.koc = take((nc + 7) / 8 + 1);       // its Fourier block (unsigned char)
  L.fold = take(mode == kShtBackward ? 0 : fb * 2 * L.H * 4 * L.J);
  L.g = take(fb * 2 * L.H * 2 * p);
  L.coef = take(mode == kShtForward ? 0 : fb * nc);
  L.total = o;
  return L;
}

// First coefficient of Fourier block k.
__device__ __forceinline__ int sht_block(int p, int k) {
  const int m = (k + 1) >> 1;  // blocks before it: m = 0 once, each 0 < m' < m twice, and m's cosines
  if (k == 0) return 0;
  const int full = p + 1 + 2 * ((m - 1) * (p + 1) - (m - 1) * m / 2);
  return (k & 1) ? full : full + p + 1 - m;
}

template <int MODE>
__global__ void __launch_bounds__(kShtThreads) k_sht(const ShtArgs A) {
  extern __shared__ double sm[];
  const int p = A.p, nc = p * (p + 2), F = 2 * p, nlon = 2 * p, ng = nlon * (p + 1);
  const ShtLayout L = sht_layout(p, A.fb, MODE);
  const int J = L.J, H = L.H, ldq = L.ldq, nj = p / 2 + 1, tid = threadIdx.x;
  double *sx = sm + L.x, *ss = sm + L.s, *sw = sm + L.w, *ab = sm + L.ab, *ca = sm + L.ca, *cb = sm + L.cb;
  double *dg = sm + L.dg, *Q = sm + L.q, *tw = sm + L.tw, *fold = sm + L.fold, *G = sm + L.g, *coef = sm + L.coef;
  unsigned char* sdeg = reinterpret_cast<unsigned char*>(sm + L.deg);
  unsigned char* skoc = reinterpret_cast<unsigned char*>(sm + L.koc);

  // ---- tables ---------------------------------------------------------------------------------
  for (int k = tid; k <= p + 1; k += kShtThreads) {  // P_k = a x P_{k-1} - b P_{k-2}
    ab[2 * k] = k ? (2.0 * k - 1.0) / k : 0.0;
    ab[2 * k + 1] = k ? (k - 1.0) / k : 0.0;
  }
  for (int i = tid; i < (p + 1) * (p + 1); i += kShtThreads) {
    const int m = i / (p + 1), n = i - m * (p + 1);
    double a = 0.0, b = 0.0;
    if (n > m) {
      a = sqrt(((2.0 * n - 1) * (2.0 * n + 1)) / ((double)(n - m) * (n + m)));
      if (n > m + 1) b = sqrt(((2.0 * n + 1) * (n + m - 1) * (n - m - 1)) / ((double)(n - m) * (n + m) * (2 * n - 3)));
    }
    ca[i] = a;
    cb[i] = b;
  }
  for (int i = tid; i <= p; i += kShtThreads) dg[i] = i ? sqrt((2.0 * i + 1.0) / (2.0 * i)) : 0.70710678118654752;
  for (int i = tid; i < F * J; i += kShtThreads) {
    const int k = i / J, j = i - k * J, m = (k + 1) >> 1, a = m * j % nlon;
    tw[i] = (k & 1) || k == 0 ? cospi((double)a / p) : sinpi((double)a / p);
  }
  for (int k = tid; k < F; k += kShtThreads) {
    const int c0 = sht_block(p, k), m = (k + 1) >> 1;
    for (int n = m; n <= p; n++) {
      sdeg[c0 + n - m] = (unsigned char)n;
      skoc[c0 + n - m] = (unsigned char)k;
    }
  }
  __syncthreads();
  if (tid < H) {  // node and weight of latitude tid (cos theta ascending: the negative half and 0)
    const int n = p + 1;
    double z = -cospi((tid + 0.75) / (n + 0.5)), pp = 1.0;
    for (int it = 0; it < 6; it++) {
      double p0 = 1.0, p1 = z;
      for (int k = 2; k <= n; k++) {
        const double p2 = ab[2 * k] * z * p1 - ab[2 * k + 1] * p0;
        p0 = p1;
        p1 = p2;
      }
      pp = n * (z * p1 - p0) / (z * z - 1.0);
      if (it < 5) z = 2 * tid == p ? 0.0 : z - p1 / pp;
    }
    sx[tid] = z;
    ss[tid] = sqrt(1.0 - z * z);
    sw[tid] = 2.0 / ((1.0 - z * z) * pp * pp);
  }
  __syncthreads();
  // sqrt(2 pi) times the normalised Legendre functions at the latitudes l <= p / 2
  for (int i = tid; i < H * (p + 1); i += kShtThreads) {
    const int m = i / H, l = i - m * H;
    const double x = sx[l], s = ss[l];
    double pm2 = 0.0, pm1 = dg[0];
    for (int q = 1; q <= m; q++) pm1 *= -s * dg[q];
    double *qc = Q + l * ldq + (m ? sht_block(p, 2 * m - 1) : 0),
           *qs = m > 0 && m < p ? Q + l * ldq + sht_block(p, 2 * m) : nullptr;
    for (int n = m; n <= p; n++) {
      if (n > m) {
        const double pn = ca[m * (p + 1) + n] * x * pm1 - cb[m * (p + 1) + n] * pm2;
        pm2 = pm1;
        pm1 = pn;
      }
      qc[n - m] = pm1;
      if (qs) qs[n - m] = pm1;
    }
  }
  __syncthreads();

  const long ngroups = (A.nfun + A.fb - 1) / A.fb;
  for (long grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    const long f0 = grp * A.fb;
    const int nf = (int)min((long)A.fb, A.nfun - f0);
    if (MODE != kShtBackward) {
      // ---- analysis: fold, DFT, Legendre sums -----------------------------------------------------
      const double* X = A.in + f0 * ng;
      for (int i = tid; i < nf * H * nj; i += kShtThreads) {
        const int j = i % nj, r = i / nj, l = r % H, f = r / H;
        const double* a = X + (long)f * ng + l * nlon;
        const double* b = X + (long)f * ng + (p - l) * nlon;
        const bool mid = 2 * l == p, own = 2 * j == p;
        double v[4], u[4];
        v[0] = a[j];
        u[0] = mid ? 0.0 : b[j];
        v[1] = j ? a[nlon - j] : 0.0;
        u[1] = j && !mid ? b[nlon - j] : 0.0;
        v[2] = own ? 0.0 : a[p - j];
        u[2] = own || mid ? 0.0 : b[p - j];
        v[3] = j == 0 || own ? 0.0 : a[p + j];
        u[3] = j == 0 || own || mid ? 0.0 : b[p + j];
        double* o = fold + (size_t)(f * H + l) * 8 * J + j;
#pragma unroll
        for (int h = 0; h < 2; h++) {  // the pair's sum, its difference
          double t[4];
#pragma unroll
          for (int q = 0; q < 4; q++) t[q] = h ? v[q] - u[q] : v[q] + u[q];
          if (h && mid) t[0] = t[1] = t[2] = t[3] = 0.0;
          o[(4 * h + 0) * J] = (t[0] + t[1]) + (t[2] + t[3]);  // cosines of even m
          o[(4 * h + 1) * J] = (t[0] + t[1]) - (t[2] + t[3]);  // of odd m
          o[(4 * h + 2) * J] = (t[0] - t[1]) - (t[2] - t[3]);  // sines of even m
          o[(4 * h + 3) * J] = (t[0] - t[1]) + (t[2] - t[3]);  // of odd m
        }
      }
      __syncthreads();
      const int rows = nf * 2 * H;
      for (int i = tid; i < F * ((rows + 3) / 4); i += kShtThreads) {
        const int k = i % F, r0 = 4 * (i / F), m = (k + 1) >> 1;
        const int cls = ((k & 1) || k == 0 ? 0 : 2) + (m & 1);
        const double* t = tw + k * J;
        const double* d[4];
        double s[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; q++) d[q] = fold + (size_t)min(r0 + q, rows - 1) * 4 * J + cls * J;
        for (int j = 0; j < nj; j++) {
          const double c = t[j];
#pragma unroll
          for (int q = 0; q < 4; q++) s[q] = fma(d[q][j], c, s[q]);
        }
        const double e = (m == 0 || m == p ? 0.5 : 1.0) / p;
#pragma unroll
        for (int q = 0; q < 4; q++)
          if (r0 + q < rows) G[(r0 + q) * F + k] = s[q] * (e * sw[(r0 + q) / 2 % H]);
      }
      __syncthreads();
      double* S = MODE == kShtFilter ? coef : A.out + f0 * nc;
      for (int i = tid; i < nc * ((nf + 1) / 2); i += kShtThreads) {
        const int c = i % nc, f = 2 * (i / nc), k = skoc[c], n = sdeg[c];
        const bool two = f + 1 < nf;
        const double* g0 = G + (size_t)f * 2 * H * F + ((n - ((k + 1) >> 1)) & 1) * F + k;
        const double* g1 = two ? g0 + 2 * H * F : g0;
        double s0 = 0.0, s1 = 0.0;
        for (int l = 0; l < H; l++) {
          const double q = Q[l * ldq + c];
          s0 = fma(q, g0[2 * l * F], s0);
          s1 = fma(q, g1[2 * l * F], s1);
        }
        const double sc = MODE == kShtFilter ? A.scale[n] : 1.0;
        S[(long)f * nc + c] = s0 * sc;
        if (two) S[(long)(f + 1) * nc + c] = s1 * sc;
      }
    } else {
      for (int i = tid; i < nf * nc; i += kShtThreads) coef[i] = A.in[f0 * nc + i];
    }
    __syncthreads();
    if (MODE == kShtForward) continue;
    // ---- synthesis: Legendre sums (even and odd degrees of a block serve a pair), DFT ----------------
    for (int i = tid; i < nf * F * H; i += kShtThreads) {
      const int l = i % H, r = i / H, k = r % F, f = r / F;
      const int c0 = sht_block(p, k), len = p + 1 - ((k + 1) >> 1);
      const double *q = Q + l * ldq + c0, *s = coef + f * nc + c0;
      double e = 0.0, o = 0.0;
      int n = 0;
      for (; n + 1 < len; n += 2) {
        e = fma(q[n], s[n], e);
        o = fma(q[n + 1], s[n + 1], o);
      }
      if (n < len) e = fma(q[n], s[n], e);
      double* g = G + (size_t)(f * H + l) * 2 * F + k;
      g[0] = e + o;
      g[F] = e - o;
    }
    __syncthreads();
    double* X = A.out + f0 * ng;
    for (int i = tid; i < nf * 2 * H * nj; i += kShtThreads) {
      const int j = i % nj, r = i / nj, slot = r & 1, l = (r >> 1) % H, f = (r >> 1) / H;
      if (slot && 2 * l == p) continue;
      const double *g = G + (size_t)r * F, *t = tw + j;
      double ce = g[0], co = 0.0, se = 0.0, so = 0.0;
      for (int m = 1; m < p; m++) {
        const double wc = t[(2 * m - 1) * J], ws = t[2 * m * J], gc = g[2 * m - 1], gs = g[2 * m];
        if (m & 1) {
          co = fma(gc, wc, co);
          so = fma(gs, ws, so);
        } else {
          ce = fma(gc, wc, ce);
          se = fma(gs, ws, se);
        }
      }
      if (p & 1)
        co = fma(g[F - 1], t[(F - 1) * J], co);
      else
        ce = fma(g[F - 1], t[(F - 1) * J], ce);
      double* x = X + (long)f * ng + (slot ? p - l : l) * nlon;
      x[j] = (ce + co) + (se + so);
      if (j) x[nlon - j] = (ce + co) - (se + so);
      if (2 * j != p) {
        x[p - j] = (ce - co) + (so - se);
        if (j) x[p + j] = (ce - co) - (so - se);
      }
    }
    __syncthreads();
  }
}

template <int MODE>
int launch_sht_mode(ShtArgs a, cudaStream_t st) {
  int dev = 0, nsm = 148;
  VES3D_CK(cudaGetDevice(&dev));
  VES3D_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  // functions per round: the whole batch over one CTA per SM, within 200 KB of shared memory
  auto bytes = [&](int fb) { return (size_t)sht_layout(a.p, fb, MODE).total * sizeof(double); };
  int fb = (int)std::min(16L, (a.nfun + nsm - 1) / nsm);
  while (fb > 1 && bytes(fb) > 200 * 1024) fb--;
  a.fb = fb;
  const size_t smem = bytes(fb);
  if (const int s = allow_smem(k_sht<MODE>, smem)) return s;
  int per = 1;
  VES3D_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sht<MODE>, kShtThreads, smem));
  const long grid = std::min((a.nfun + fb - 1) / fb, (long)nsm * std::max(per, 1));
  k_sht<MODE><<<(unsigned)grid, kShtThreads, smem, st>>>(a);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

}  // namespace

bool sht_fused_supported(int p) { return p >= 2 && p <= kShtMaxP; }

int launch_sht_fused(int mode, const double* in, long nfun, int p, const double* scale, double* out, cudaStream_t st) {
  if (nfun <= 0) return VES3D_OK;
  ShtArgs a{};
  a.in = in;
  a.out = out;
  a.nfun = nfun;
  a.p = p;
  for (int n = 0; scale && n <= p; n++) a.scale[n] = scale[n];
  return mode == kShtForward    ? launch_sht_mode<kShtForward>(a, st)
         : mode == kShtBackward ? launch_sht_mode<kShtBackward>(a, st)
                                : launch_sht_mode<kShtFilter>(a, st);
}

}  // namespace ves3d
