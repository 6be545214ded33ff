// FP64 direct Stokes single-layer sums (plain form) and the far-field source packing.
//
// Pair kernel (StokesAlltoAll, src/CPUKernels.cc:1011-1057; DirectStokesKernel, :123-178):
//   r = x_s - x_t,  u_t += [ d_s / |r| + (r . d_s) r / |r|^3 ] / (8 pi),
// and a coincident pair (|r| = 0) contributes nothing.
//
// (The far field with same-vesicle exclusion is in far_kernels.cu.)
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace ves3d {

constexpr int kFarBS = 128;

struct PairAcc {
  double x = 0.0, y = 0.0, z = 0.0;
};

__device__ __forceinline__ void pair_f64(double tx, double ty, double tz, double sx, double sy, double sz, double dx_,
                                         double dy_, double dz_, bool skip, PairAcc& a) {
  const double dx = sx - tx, dy = sy - ty, dz = sz - tz;
  const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  double rinv = rsqrt_f64(r2);
  rinv = (skip || r2 == 0.0) ? 0.0 : rinv;
  const double cc = fma(dz, dz_, fma(dy, dy_, dx * dx_)) * rinv * rinv;
  a.x = fma(fma(cc, dx, dx_), rinv, a.x);
  a.y = fma(fma(cc, dy, dy_), rinv, a.y);
  a.z = fma(fma(cc, dz, dz_), rinv, a.z);
}

// Sums over N sources at M targets, both point-major: the single layer of den and, with DL, the
// double layer of unit normals nrm and densities dden. A CTA of kSumWarps warps takes 64 targets,
// two per lane, each warp its 32 of the sources of every staged tile (so that a few thousand
// targets fill the chip without partial sums in memory), and adds the warps' sums in order.
// grid (chunks of targets, source segments); out gets the sums, or out[segment] those of its
// sources for k_sum_segments. Bound by the FP64 pipe: 22 operations a pair, 47 with the double
// layer. 20,000 targets of 32,400 sources, single layer: 3.57 -> 1.10 ms (one target per thread
// before, a barrier per 128 sources, 157 CTAs).
constexpr int kSumWarps = 8, kSumTrg = 64, kSumTile = 32 * kSumWarps;

template <bool DL>
__global__ void __launch_bounds__(32 * kSumWarps, DL ? 2 : 4)
    k_sum_f64(const double* __restrict__ pos, const double* __restrict__ den, const double* __restrict__ nrm,
              const double* __restrict__ dden, long N, long seg_len, const double* __restrict__ trg, long M,
              double* __restrict__ out) {
  constexpr int WS = DL ? 12 : 6, WO = DL ? 6 : 3;
  __shared__ __align__(16) double sm[kSumTile * WS];
  static_assert(kSumTile * WS >= kSumWarps * kSumTrg * WO, "the warps' sums reuse the tile");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long m0 = (long)blockIdx.x * kSumTrg;
  double t[2][3];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const long m = min(m0 + lane + 32 * j, M - 1);  // idle lanes repeat the last target
#pragma unroll
    for (int d = 0; d < 3; d++) t[j][d] = trg[3 * m + d];
  }
  PairAcc a[2], b[2];
  const long b0 = (long)blockIdx.y * seg_len, b1 = min(N, b0 + seg_len);
  for (long s0 = b0; s0 < b1; s0 += kSumTile) {
    const int ns = (int)min((long)kSumTile, b1 - s0);
    __syncthreads();
    if (threadIdx.x < ns) {
      const long s = 3 * (s0 + threadIdx.x);
      double* q = sm + WS * threadIdx.x;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        q[d] = pos[s + d];
        q[3 + d] = den[s + d];
        if (DL) {
          q[6 + d] = nrm[s + d];
          q[9 + d] = dden[s + d];
        }
      }
    }
    __syncthreads();
    const int k1 = min(32 * (w + 1), ns);
#pragma unroll 2
    for (int k = 32 * w; k < k1; k++) {
      const double* q = sm + WS * k;
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const double dx = q[0] - t[j][0], dy = q[1] - t[j][1], dz = q[2] - t[j][2];
        const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
        double rinv = rsqrt_f64_int_seed(r2);
        rinv = r2_in_range(r2) ? rinv : 0.0;  // a coincident pair contributes nothing
        const double rinv2 = rinv * rinv;
        const double c = fma(dz, q[5], fma(dy, q[4], dx * q[3])) * rinv2;
        a[j].x = fma(fma(c, dx, q[3]), rinv, a[j].x);
        a[j].y = fma(fma(c, dy, q[4]), rinv, a[j].y);
        a[j].z = fma(fma(c, dz, q[5]), rinv, a[j].z);
        if (DL) {  // r = target - source = -(dx, dy, dz)
          const double e = fma(dz, q[8], fma(dy, q[7], dx * q[6])) * fma(dz, q[11], fma(dy, q[10], dx * q[9])) *
                           -(rinv2 * rinv2 * rinv);
          b[j].x = fma(e, dx, b[j].x);
          b[j].y = fma(e, dy, b[j].y);
          b[j].z = fma(e, dz, b[j].z);
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 2; j++) {
    double* o = sm + (w * kSumTrg + lane + 32 * j) * WO;
    o[0] = a[j].x;
    o[1] = a[j].y;
    o[2] = a[j].z;
    if (DL) {
      o[3] = b[j].x;
      o[4] = b[j].y;
      o[5] = b[j].z;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * kSumTrg; i += 32 * kSumWarps) {
    const int m = i / 3, d = i - 3 * m;
    if (m0 + m >= M) continue;
    double s = 0.0, g = 0.0;
#pragma unroll
    for (int q = 0; q < kSumWarps; q++) {
      s += sm[(q * kSumTrg + m) * WO + d];
      if (DL) g += sm[(q * kSumTrg + m) * WO + 3 + d];
    }
    out[(long)blockIdx.y * 3 * M + 3 * (m0 + m) + d] = DL ? s * kInv8Pi + g * kDl : s * kInv8Pi;
  }
}

// out[i] = scale sum over the sets of partial sums, in order
__global__ void k_sum_segments(const double* __restrict__ part, int nseg, long n, double scale,
                               double* __restrict__ out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
#pragma unroll 8
  for (int q = 0; q < nseg; q++) s += part[(long)q * n + i];
  out[i] = s * scale;
}

// Source segments of a sum at M targets: about sixteen CTAs per SM in all, four at a time, so that
// the last wave is a small part (20,000 targets at one segment: three CTAs on some SMs, two on others).
static long sum_segments(long M) {
  const long chunks = (M + kSumTrg - 1) / kSumTrg;
  return std::max(1L, std::min(32L, 16L * 148 / chunks));
}

// (not monotonic in M: more targets take fewer segments)
size_t targets_part_doubles(long M) { return sum_segments(M) > 1 ? 3 * (size_t)M * sum_segments(M) : 0; }

// Segments of N sources at M targets with room for part_doubles partial sums.
long targets_segments(long N, long M, size_t part_doubles, long* tiles_each) {
  const long room = std::max(1L, (long)(part_doubles / (3 * (size_t)M)));
  const long tiles = (N + kSumTile - 1) / kSumTile, nseg = std::min(sum_segments(M), room);
  const long per = std::max(1L, (tiles + nseg - 1) / nseg);
  if (tiles_each) *tiles_each = per;
  return std::max(1L, (tiles + per - 1) / per);
}

int launch_alltoall_f64(const double* pos, const double* den, long np, double* pot, double* part, long slots,
                        cudaStream_t st) {
  if (np <= 0) return VES3D_OK;
  if (part) {
    int G = 0;
    const int s = launch_far_sym(pos, den, nullptr, nullptr, 0, np, part, slots, st, &G);
    if (s) return s;
    k_sum_segments<<<(unsigned)((3 * np + 255) / 256), 256, 0, st>>>(part, G, 3 * np, kInv8Pi, pot);
  } else {
    k_sum_f64<false><<<(unsigned)((np + kSumTrg - 1) / kSumTrg), 32 * kSumWarps, 0, st>>>(pos, den, nullptr, nullptr,
                                                                                          np, np, pos, np, pot);
  }
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// Device<GPU>::DirectStokes / cuda_stokes (src/CudaKernels.cu:1840-1916, 1996-2006):
// per surface v, targets t in [t_head, t_tail) of T[v] (stride trg_m), sources all
// src_m points of S[v] with density D * Q. grid = (target chunks, n surfaces).
__global__ void __launch_bounds__(kFarBS) k_direct_stokes_f64(int src_m, int trg_m, int t_head, int t_tail,
                                                              const double* __restrict__ T,
                                                              const double* __restrict__ S,
                                                              const double* __restrict__ D, double* __restrict__ U,
                                                              const double* __restrict__ Q) {
  __shared__ double sp[kFarBS * 3];
  __shared__ double sd[kFarBS * 3];
  const long v = blockIdx.y;
  const int t = t_head + blockIdx.x * kFarBS + threadIdx.x;
  const bool active = t < t_tail;
  const double* Tv = T + v * 3 * (long)trg_m;
  const double* Sv = S + v * 3 * (long)src_m;
  const double* Dv = D + v * 3 * (long)src_m;
  double tx = 0, ty = 0, tz = 0;
  if (active) {
    tx = Tv[t];
    ty = Tv[trg_m + t];
    tz = Tv[2 * trg_m + t];
  }
  PairAcc acc;
  for (int s0 = 0; s0 < src_m; s0 += kFarBS) {
    const int ns = min(kFarBS, src_m - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < ns; i += kFarBS) {
      const int s = s0 + i;
      const double q = Q ? Q[s] : 1.0;
      sp[3 * i] = Sv[s];
      sp[3 * i + 1] = Sv[src_m + s];
      sp[3 * i + 2] = Sv[2 * src_m + s];
      sd[3 * i] = Dv[s] * q;
      sd[3 * i + 1] = Dv[src_m + s] * q;
      sd[3 * i + 2] = Dv[2 * src_m + s] * q;
    }
    __syncthreads();
    if (!active) continue;
    for (int k = 0; k < ns; k++)
      pair_f64(tx, ty, tz, sp[3 * k], sp[3 * k + 1], sp[3 * k + 2], sd[3 * k], sd[3 * k + 1], sd[3 * k + 2], false,
               acc);
  }
  if (!active) return;
  double* Uv = U + v * 3 * (long)trg_m;
  Uv[t] = acc.x * kInv8Pi;
  Uv[trg_m + t] = acc.y * kInv8Pi;
  Uv[2 * trg_m + t] = acc.z * kInv8Pi;
}

int launch_direct_stokes_f64(int src_m, int trg_m, int n, int t_head, int t_tail, const double* T,
                             const double* S, const double* D, double* U, const double* Q, cudaStream_t st) {
  if (n <= 0 || t_tail <= t_head) return VES3D_OK;
  dim3 grid((t_tail - t_head + kFarBS - 1) / kFarBS, n);
  k_direct_stokes_f64<<<grid, kFarBS, 0, st>>>(src_m, trg_m, t_head, t_tail, T, S, D, U, Q);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// The single-precision overload of cuda_stokes (src/CudaKernels.cu:594-761, the kernel
// `stokes` on float arrays, used by SINGLE_PREC builds of the reference): FP32 inputs and
// outputs and FP32 pair arithmetic (hardware reciprocal square root, a coincident pair
// contributes nothing), each thread's FP32 sum over a tile of 128 sources added into an
// FP64 accumulator. Q may be NULL (unit weights), as in the reference's second kernel.
__global__ void __launch_bounds__(kFarBS) k_direct_stokes_f32(int src_m, int trg_m, int t_head, int t_tail,
                                                              const float* __restrict__ T,
                                                              const float* __restrict__ S,
                                                              const float* __restrict__ D, float* __restrict__ U,
                                                              const float* __restrict__ Q) {
  __shared__ float sp[kFarBS * 3];
  __shared__ float sd[kFarBS * 3];
  const long v = blockIdx.y;
  const int t = t_head + blockIdx.x * kFarBS + threadIdx.x;
  const bool active = t < t_tail;
  const float* Tv = T + v * 3 * (long)trg_m;
  const float* Sv = S + v * 3 * (long)src_m;
  const float* Dv = D + v * 3 * (long)src_m;
  float tx = 0.f, ty = 0.f, tz = 0.f;
  if (active) {
    tx = Tv[t];
    ty = Tv[trg_m + t];
    tz = Tv[2 * trg_m + t];
  }
  double ax = 0.0, ay = 0.0, az = 0.0;
  for (int s0 = 0; s0 < src_m; s0 += kFarBS) {
    const int ns = min(kFarBS, src_m - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < ns; i += kFarBS) {
      const int s = s0 + i;
      const float q = Q ? Q[s] : 1.f;
      sp[3 * i] = Sv[s];
      sp[3 * i + 1] = Sv[src_m + s];
      sp[3 * i + 2] = Sv[2 * src_m + s];
      sd[3 * i] = Dv[s] * q;
      sd[3 * i + 1] = Dv[src_m + s] * q;
      sd[3 * i + 2] = Dv[2 * src_m + s] * q;
    }
    __syncthreads();
    if (!active) continue;
    float ux = 0.f, uy = 0.f, uz = 0.f;
    for (int k = 0; k < ns; k++) {
      const float dx = sp[3 * k] - tx, dy = sp[3 * k + 1] - ty, dz = sp[3 * k + 2] - tz;
      const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      const float rinv = r2 > 0.f ? rsqrtf(r2) : 0.f;
      const float cc = fmaf(dz, sd[3 * k + 2], fmaf(dy, sd[3 * k + 1], dx * sd[3 * k])) * rinv * rinv;
      ux = fmaf(fmaf(cc, dx, sd[3 * k]), rinv, ux);
      uy = fmaf(fmaf(cc, dy, sd[3 * k + 1]), rinv, uy);
      uz = fmaf(fmaf(cc, dz, sd[3 * k + 2]), rinv, uz);
    }
    ax += ux;
    ay += uy;
    az += uz;
  }
  if (!active) return;
  float* Uv = U + v * 3 * (long)trg_m;
  Uv[t] = (float)(ax * kInv8Pi);
  Uv[trg_m + t] = (float)(ay * kInv8Pi);
  Uv[2 * trg_m + t] = (float)(az * kInv8Pi);
}

int launch_direct_stokes_f32(int src_m, int trg_m, int n, int t_head, int t_tail, const float* T, const float* S,
                             const float* D, float* U, const float* Q, cudaStream_t st) {
  if (n <= 0 || t_tail <= t_head) return VES3D_OK;
  dim3 grid((t_tail - t_head + kFarBS - 1) / kFarBS, n);
  k_direct_stokes_f32<<<grid, kFarBS, 0, st>>>(src_m, trg_m, t_head, t_tail, T, S, D, U, Q);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// Double-layer pair (DirectStokesDoubleLayerKernel, src/CPUKernels.cc:1060-1120;
// stokes_double_layer, src/CudaKernels.cu:783-868): r = x_t - x_s,
// u_t += (r . n_s)(r . d_s) r / |r|^5, scaled by 3/(4 pi) after the sum; a coincident pair
// contributes nothing.
__device__ __forceinline__ void pair_dl_f64(double tx, double ty, double tz, const double* sp, const double* sn,
                                            const double* sd, PairAcc& a) {
  const double dx = tx - sp[0], dy = ty - sp[1], dz = tz - sp[2];
  const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
  double rinv = rsqrt_f64(r2);
  rinv = r2 > 0.0 ? rinv : 0.0;
  const double rinv2 = rinv * rinv;
  const double q = fma(dz, sn[2], fma(dy, sn[1], dx * sn[0])) * fma(dz, sd[2], fma(dy, sd[1], dx * sd[0])) *
                   (rinv2 * rinv2 * rinv);
  a.x = fma(dx, q, a.x);
  a.y = fma(dy, q, a.y);
  a.z = fma(dz, q, a.z);
}

// Device<GPU>::DirectStokesDoubleLayer / cuda_stokes_double_layer (src/CudaKernels.cu:895-918,
// src/DeviceGPU.cc:263-271): per surface v, targets t in [t_head, t_tail) of T[v] (stride
// trg_m), sources all src_m points of S[v] with normals N and densities D (times Q when
// given). grid = (target chunks, n surfaces).
__global__ void __launch_bounds__(kFarBS) k_direct_stokes_dl_f64(int src_m, int trg_m, int t_head, int t_tail,
                                                                 const double* __restrict__ T,
                                                                 const double* __restrict__ S,
                                                                 const double* __restrict__ N,
                                                                 const double* __restrict__ D, double* __restrict__ U,
                                                                 const double* __restrict__ Q) {
  __shared__ double sp[kFarBS * 3];
  __shared__ double sn[kFarBS * 3];
  __shared__ double sd[kFarBS * 3];
  const long v = blockIdx.y;
  const int t = t_head + blockIdx.x * kFarBS + threadIdx.x;
  const bool active = t < t_tail;
  const double* Tv = T + v * 3 * (long)trg_m;
  const double* Sv = S + v * 3 * (long)src_m;
  const double* Nv = N + v * 3 * (long)src_m;
  const double* Dv = D + v * 3 * (long)src_m;
  double tx = 0, ty = 0, tz = 0;
  if (active) {
    tx = Tv[t];
    ty = Tv[trg_m + t];
    tz = Tv[2 * trg_m + t];
  }
  PairAcc acc;
  for (int s0 = 0; s0 < src_m; s0 += kFarBS) {
    const int ns = min(kFarBS, src_m - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < ns; i += kFarBS) {
      const int s = s0 + i;
      const double q = Q ? Q[s] : 1.0;
      sp[3 * i] = Sv[s];
      sp[3 * i + 1] = Sv[src_m + s];
      sp[3 * i + 2] = Sv[2 * src_m + s];
      sn[3 * i] = Nv[s];
      sn[3 * i + 1] = Nv[src_m + s];
      sn[3 * i + 2] = Nv[2 * src_m + s];
      sd[3 * i] = Dv[s] * q;
      sd[3 * i + 1] = Dv[src_m + s] * q;
      sd[3 * i + 2] = Dv[2 * src_m + s] * q;
    }
    __syncthreads();
    if (!active) continue;
    for (int k = 0; k < ns; k++) pair_dl_f64(tx, ty, tz, sp + 3 * k, sn + 3 * k, sd + 3 * k, acc);
  }
  if (!active) return;
  double* Uv = U + v * 3 * (long)trg_m;
  Uv[t] = acc.x * kDl;
  Uv[trg_m + t] = acc.y * kDl;
  Uv[2 * trg_m + t] = acc.z * kDl;
}

int launch_direct_stokes_dl_f64(int src_m, int trg_m, int n, int t_head, int t_tail, const double* T,
                                const double* S, const double* N, const double* D, double* U, const double* Q,
                                cudaStream_t st) {
  if (n <= 0 || t_tail <= t_head) return VES3D_OK;
  dim3 grid((t_tail - t_head + kFarBS - 1) / kFarBS, n);
  k_direct_stokes_dl_f64<<<grid, kFarBS, 0, st>>>(src_m, trg_m, t_head, t_tail, T, S, N, D, U, Q);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// Velocity at M off-surface targets (point-major) from all N surface points (point-major):
// the single layer of den and, with nrm, the double layer of unit normals nrm and densities
// dden (both densities times area and weights). Few targets split the sources over segments.
int launch_targets_f64(const double* pos, const double* den, const double* nrm, const double* dden, long N,
                       const double* trg, long M, double* out, double* part, size_t part_doubles, cudaStream_t st) {
  if (M <= 0) return VES3D_OK;
  long per = 1;
  const long nseg = targets_segments(N, M, part_doubles, &per);
  const dim3 grid((unsigned)((M + kSumTrg - 1) / kSumTrg), (unsigned)nseg);
  double* dst = nseg > 1 ? part : out;
  if (nrm)
    k_sum_f64<true><<<grid, 32 * kSumWarps, 0, st>>>(pos, den, nrm, dden, N, per * kSumTile, trg, M, dst);
  else
    k_sum_f64<false><<<grid, 32 * kSumWarps, 0, st>>>(pos, den, nullptr, nullptr, N, per * kSumTile, trg, M, dst);
  VES3D_LAUNCHED();
  if (nseg == 1) return VES3D_OK;
  k_sum_segments<<<(unsigned)((3 * M + 255) / 256), 256, 0, st>>>(part, (int)nseg, 3 * M, 1.0, out);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// Unit outward normals, point-major (src/StokesVelocity.cc:245-275).
__global__ void k_unit_normals(const double* __restrict__ Xt, const double* __restrict__ Xp, long nv, int p0,
                               double* __restrict__ nrm) {
  const int ng = 2 * p0 * (p0 + 1);
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nv * ng) return;
  const long v = g / ng;
  const int k = (int)(g - v * ng);
  const long b = v * 3 * ng + k;
  const double ax = Xt[b], ay = Xt[b + ng], az = Xt[b + 2 * ng];
  const double bx = Xp[b], by = Xp[b + ng], bz = Xp[b + 2 * ng];
  const double nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
  const double inv = 1.0 / sqrt(nx * nx + ny * ny + nz * nz);
  nrm[3 * g] = nx * inv;
  nrm[3 * g + 1] = ny * inv;
  nrm[3 * g + 2] = nz * inv;
}

int launch_unit_normals(const double* Xt, const double* Xp, long nv, int p0, double* nrm, cudaStream_t st) {
  const long N = nv * ngrid_(p0);
  if (N <= 0) return VES3D_OK;
  k_unit_normals<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(Xt, Xp, nv, p0, nrm);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

// area = |X_theta x X_phi|; pos point-major; den = f * area * w[lat].
__global__ void k_far_sources(const double* __restrict__ X, const double* __restrict__ f,
                              const double* __restrict__ Xt, const double* __restrict__ Xp, long nv, int p0,
                              const double* __restrict__ w, double* __restrict__ area, double* __restrict__ pos,
                              double* __restrict__ den) {
  const int ng = 2 * p0 * (p0 + 1);
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nv * ng) return;
  const long v = g / ng;
  const int k = (int)(g - v * ng);
  const long b = v * 3 * ng + k;
  const double ax = Xt[b], ay = Xt[b + ng], az = Xt[b + 2 * ng];
  const double bx = Xp[b], by = Xp[b + ng], bz = Xp[b + 2 * ng];
  const double nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
  const double a = sqrt(nx * nx + ny * ny + nz * nz);
  area[g] = a;
  const double q = a * w[k / (2 * p0)];
  pos[3 * g] = X[b];
  pos[3 * g + 1] = X[b + ng];
  pos[3 * g + 2] = X[b + 2 * ng];
  if (f) {
    den[3 * g] = f[b] * q;
    den[3 * g + 1] = f[b + ng] * q;
    den[3 * g + 2] = f[b + 2 * ng] * q;
  }
}

int launch_far_sources(const double* X, const double* f, const double* Xt, const double* Xp, long nv, int p0,
                       const double* smooth_w, double* area, double* pos, double* den, cudaStream_t st) {
  const long N = nv * ngrid_(p0);
  if (N <= 0) return VES3D_OK;
  k_far_sources<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(X, f, Xt, Xp, nv, p0, smooth_w, area, pos, den);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

__global__ void k_far_density(const double* __restrict__ f, const double* __restrict__ area, long nv, int p0,
                              const double* __restrict__ w, double* __restrict__ den) {
  const int ng = 2 * p0 * (p0 + 1);
  const long g = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nv * ng) return;
  const long v = g / ng;
  const int k = (int)(g - v * ng);
  const long b = v * 3 * ng + k;
  const double q = area[g] * w[k / (2 * p0)];
  den[3 * g] = f[b] * q;
  den[3 * g + 1] = f[b + ng] * q;
  den[3 * g + 2] = f[b + 2 * ng] * q;
}

int launch_far_density(const double* f, const double* area, long nv, int p0, const double* smooth_w, double* den,
                       cudaStream_t st) {
  const long N = nv * ngrid_(p0);
  if (N <= 0) return VES3D_OK;
  k_far_density<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(f, area, nv, p0, smooth_w, den);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

__global__ void k_scale_vesicles(const double* __restrict__ x, long n, long per, const double* __restrict__ c, long nc,
                                 const double* __restrict__ z, double beta, double* __restrict__ out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = c[(i / per) % nc] * x[i];
  out[i] = z ? fma(beta, z[i], v) : v;
}

int launch_scale_vesicles(const double* x, long n, long per, const double* c, long nc, const double* z, double beta,
                          double* out, cudaStream_t st) {
  if (n <= 0) return VES3D_OK;
  k_scale_vesicles<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, n, per, c, nc, z, beta, out);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

__global__ void k_add(const double* __restrict__ a, const double* __restrict__ b, long n, double* __restrict__ out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = a[i] + b[i];
}

int launch_add(const double* a, const double* b, long n, double* out, cudaStream_t st) {
  if (n <= 0) return VES3D_OK;
  k_add<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a, b, n, out);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

}  // namespace ves3d
