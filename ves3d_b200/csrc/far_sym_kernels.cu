// FP64 all-pairs sums that evaluate each unordered pair of points once. The distance, its
// reciprocal and the tensor's structure are the same seen from either point (the Stokeslet is
// even in r, the double layer's kernel odd), so the two directions of a pair share the FP64
// operations up to 1/|r|: 32 per unordered pair of the single layer against 2 x 22 one-sided (36
// against 2 x 25 of the double layer).
//
// Bound by the FP64 pipe (68.7% busy; 88% of the slots of the last wave filled at 34,816 points). A
// lane keeps T targets and their sums in registers, the staged sources' sums stay in shared memory,
// and lane l meets source (l + k) mod 32 in step k, so no sum is ever shared between two lanes and
// the order of every sum is fixed. Before (one-sided) and now:
//   single layer, 278,528 points 123.2 -> 98.9 ms, 34,816 points 2.20 -> 1.59 ms
//   double layer, 26,112 points  1.36 -> 1.17 ms
//   all pairs of 19,000 points   2.14 -> 0.53 ms (one target per thread before)
// The partial sums are the price: G sets of 24 bytes a point (up to 80, within a GiB; 78 sets, 521 MB, at
// 278,528 points), where a group of several target blocks reads and adds to what it has written: 734 MB
// of DRAM traffic a launch against 105 one-sided, of the 640 GB that the launch's time would move.
// Other shapes (2 to 6 targets, 2 to 16 warps, 80 to 255 registers) ran 97 to 139 ms at 278,528
// points; two sources a step with sums in shuffles 106 ms.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace ves3d {

namespace {

constexpr long kMaxSlots = 80;  // sets of partial sums
// All pairs of points: from this many on the paired sums are the faster (one call of the interaction
// handle with 4,000 points 97 us against 149, 10,000 points 234 against 427).
constexpr long kPairsMin = 4000;

// Warps per CTA, targets per lane, 32-source rounds per warp between two barriers. SMALL: two targets
// per lane, for groups of half the points and four times the items.
template <bool DL, bool SMALL>
struct SymCfg {
  static constexpr int W = 4, T = SMALL ? 2 : DL ? 3 : 4, SUB = 2, MINB = 3;
  static constexpr int NT = 32 * W, TB = NT * T;  // targets per block
  static constexpr int ST = 32 * W * SUB;         // sources per staged tile
  static constexpr int WS = DL ? 9 : 6;           // doubles per staged source
  static constexpr size_t SMEM = (size_t)ST * (WS + 3) * sizeof(double);
};

template <bool DL>
struct SymTarget {
  double p[3], d[3], n[DL ? 3 : 1], a[3];
};

// One round: the lane's T targets against 32 staged sources.
// e0, e1: the staged indices (relative to base) of the target's own vesicle, skipped when MASK.
template <bool DL, bool SMALL, bool SYM, bool MASK>
__device__ __forceinline__ void sym_round(const double2* __restrict__ src, const double* __restrict__ nz,
                                          double2* __restrict__ axy, double* __restrict__ az,
                                          SymTarget<DL> (&t)[SymCfg<DL, SMALL>::T],
                                          const int (&e0)[SymCfg<DL, SMALL>::T],
                                          const int (&e1)[SymCfg<DL, SMALL>::T], int base) {
  constexpr int ST = SymCfg<DL, SMALL>::ST, T = SymCfg<DL, SMALL>::T;
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int k = 0; k < 32; k++) {
    const int i = (lane + k) & 31;
    const double2 q0 = src[i], q1 = src[ST + i], q2 = src[2 * ST + i];  // (x, y) (z, d_x) (d_y, d_z)
    double2 q3;
    double snz = 0.0;
    if (DL) {  // (n_x, n_y), n_z
      q3 = src[3 * ST + i];
      snz = nz[i];
    }
    double ux = 0.0, uy = 0.0, uz = 0.0;
    if (SYM) {
      const double2 u = axy[i];
      ux = u.x;
      uy = u.y;
      uz = az[i];
    }
#pragma unroll
    for (int j = 0; j < T; j++) {
      const double dx = q0.x - t[j].p[0], dy = q0.y - t[j].p[1], dz = q1.x - t[j].p[2];
      const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
      double rinv = rsqrt_f64_int_seed(r2);
      bool ok = r2_in_range(r2);  // a coincident pair contributes nothing
      if (MASK) ok = ok && !(base + i >= e0[j] && base + i < e1[j]);
      rinv = ok ? rinv : 0.0;
      const double rinv2 = rinv * rinv;
      if (!DL) {
        const double c = fma(dz, q2.y, fma(dy, q2.x, dx * q1.y)) * rinv2;
        t[j].a[0] = fma(fma(c, dx, q1.y), rinv, t[j].a[0]);
        t[j].a[1] = fma(fma(c, dy, q2.x), rinv, t[j].a[1]);
        t[j].a[2] = fma(fma(c, dz, q2.y), rinv, t[j].a[2]);
        if (SYM) {
          const double e = fma(dz, t[j].d[2], fma(dy, t[j].d[1], dx * t[j].d[0])) * rinv2;
          ux = fma(fma(e, dx, t[j].d[0]), rinv, ux);
          uy = fma(fma(e, dy, t[j].d[1]), rinv, uy);
          uz = fma(fma(e, dz, t[j].d[2]), rinv, uz);
        }
      } else {
        // seen from the target r = -(dx, dy, dz): the odd kernel changes sign
        const double rinv5 = rinv2 * rinv2 * rinv;
        const double c = fma(dz, snz, fma(dy, q3.y, dx * q3.x)) * fma(dz, q2.y, fma(dy, q2.x, dx * q1.y)) * -rinv5;
        t[j].a[0] = fma(c, dx, t[j].a[0]);
        t[j].a[1] = fma(c, dy, t[j].a[1]);
        t[j].a[2] = fma(c, dz, t[j].a[2]);
        if (SYM) {
          const double e = fma(dz, t[j].n[2], fma(dy, t[j].n[1], dx * t[j].n[0])) *
                           fma(dz, t[j].d[2], fma(dy, t[j].d[1], dx * t[j].d[0])) * rinv5;
          ux = fma(e, dx, ux);
          uy = fma(e, dy, uy);
          uz = fma(e, dz, uz);
        }
      }
    }
    if (SYM) {
      axy[i] = make_double2(ux, uy);
      az[i] = uz;
      __syncwarp();  // the neighbouring lane meets this source next
    }
  }
}

__device__ __forceinline__ long vesicle_at(const long* __restrict__ off, long nves, long g) {
  long lo = 0, hi = nves;
  while (hi - lo > 1) {
    const long mid = (lo + hi) >> 1;
    if (off[mid] <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

// The points are cut into G groups of GS; CTA (I, J), I <= J, takes the pairs between two groups.
// It writes the sums of group I's points over group J to slot J of those points and those of
// group J's points over group I to slot I, so every (point, slot) is written once: part
// [G][N][3]. A group with itself is summed one-sided (as many operations as two groups with
// each other). off null: every pair counts but coincident ones.
template <bool DL, bool SMALL>
__global__ void __launch_bounds__(SymCfg<DL, SMALL>::NT, SymCfg<DL, SMALL>::MINB)
    k_far_sym_f64(const double* __restrict__ pos, const double* __restrict__ den, const double* __restrict__ nrm,
                  const long* __restrict__ off, long nves, long N, int G, long GS, double* __restrict__ part) {
  using Cf = SymCfg<DL, SMALL>;
  constexpr int NT = Cf::NT, T = Cf::T, ST = Cf::ST, W = Cf::W, SUB = Cf::SUB;
  extern __shared__ __align__(16) double2 sm2[];
  double2* src = sm2;
  double2* axy = src + (DL ? 4 * ST + ST / 2 : 3 * ST);
  double* az = reinterpret_cast<double*>(axy + ST);
  double* nz = reinterpret_cast<double*>(src + 4 * ST);  // (DL only)
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nsym = G * (G - 1) / 2;
  int I, J;
  if ((int)blockIdx.x < nsym) {  // pairs of distinct groups first: they are the longer items
    const int b = blockIdx.x;
    J = (int)((1.0f + sqrtf(1.0f + 8.0f * b)) * 0.5f);
    while (J * (J - 1) / 2 > b) J--;
    while ((J + 1) * J / 2 <= b) J++;
    I = b - J * (J - 1) / 2;
  } else {
    I = J = blockIdx.x - nsym;
  }
  const long i0 = I * GS, i1 = min(N, i0 + GS), j0 = J * GS, j1 = min(N, j0 + GS);
  const bool sym = I != J;
  // a vesicle in both groups (the last of I reaches into J): its points skip one another
  const bool mask = !sym || (off && off[vesicle_at(off, nves, i1 - 1) + 1] > j0);
  for (long t0 = i0; t0 < i1; t0 += Cf::TB) {
    SymTarget<DL> t[T];
    int e0[T], e1[T];
#pragma unroll
    for (int j = 0; j < T; j++) {
      const long g = t0 + (w * T + j) * 32 + lane;
      const bool v = g < i1;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        t[j].p[d] = v ? pos[3 * g + d] : 0.0;
        t[j].d[d] = v ? den[3 * g + d] : 0.0;
        if (DL) t[j].n[d] = v ? nrm[3 * g + d] : 0.0;
        t[j].a[d] = 0.0;
      }
      e0[j] = e1[j] = 0;
      if (mask && off && v) {
        const long ves = vesicle_at(off, nves, g);
        e0[j] = (int)max(0L, off[ves] - j0);
        e1[j] = (int)max(0L, off[ves + 1] - j0);
      }
    }
    for (long s0 = j0; s0 < j1; s0 += ST) {
      const int ns = (int)min((long)ST, j1 - s0);
      __syncthreads();  // the previous tile is written out
      for (int i = threadIdx.x; i < ST; i += NT) {
        const bool v = i < ns;  // padding sources carry no density
        const long s = 3 * (s0 + i);
        src[i] = v ? make_double2(pos[s], pos[s + 1]) : make_double2(0.0, 0.0);
        src[ST + i] = v ? make_double2(pos[s + 2], den[s]) : make_double2(0.0, 0.0);
        src[2 * ST + i] = v ? make_double2(den[s + 1], den[s + 2]) : make_double2(0.0, 0.0);
        if (DL) {
          src[3 * ST + i] = v ? make_double2(nrm[s], nrm[s + 1]) : make_double2(0.0, 0.0);
          nz[i] = v ? nrm[s + 2] : 0.0;
        }
        axy[i] = make_double2(0.0, 0.0);
        az[i] = 0.0;
      }
      __syncthreads();
      // warp w starts at the w-th part of the tile: the warps hold distinct sources at any time
#pragma unroll 1
      for (int sp = 0; sp < W; sp++) {
        const int part0 = ((w + sp) % W) * SUB * 32;
#pragma unroll 1
        for (int o = part0; o < min(part0 + SUB * 32, ns); o += 32) {
          const int base = (int)(s0 - j0) + o;
          if (!sym)
            sym_round<DL, SMALL, false, true>(src + o, DL ? nz + o : nullptr, axy + o, az + o, t, e0, e1, base);
          else if (mask)
            sym_round<DL, SMALL, true, true>(src + o, DL ? nz + o : nullptr, axy + o, az + o, t, e0, e1, base);
          else
            sym_round<DL, SMALL, true, false>(src + o, DL ? nz + o : nullptr, axy + o, az + o, t, e0, e1, base);
        }
        if (sym) __syncthreads();
      }
      if (sym) {  // this CTA alone writes group J's slot I: the first block of targets sets it
        double* P = part + (long)I * 3 * N;
        for (int i = threadIdx.x; i < ns; i += NT) {
          const long s = 3 * (s0 + i);
          const double2 u = axy[i];
          const double z = az[i];
          if (t0 == i0) {
            P[s] = u.x;
            P[s + 1] = u.y;
            P[s + 2] = z;
          } else {
            P[s] += u.x;
            P[s + 1] += u.y;
            P[s + 2] += z;
          }
        }
      }
    }
    double* P = part + (long)J * 3 * N;
#pragma unroll
    for (int j = 0; j < T; j++) {
      const long g = t0 + (w * T + j) * 32 + lane;
      if (g < i1)
#pragma unroll
        for (int d = 0; d < 3; d++) P[3 * g + d] = t[j].a[d];
    }
  }
}

// Group size: whole target blocks, at most max_slots groups, so that the G (G + 1) / 2 equal
// items fill their last wave of CTAs; the fewest groups (partial sums) within 2% of the best.
template <class Cf>
void sym_groups(long N, long max_slots, int nsm, int* G, long* GS) {
  const long tb = Cf::TB;
  auto eff = [&](long g, long gs) {
    const double items = 0.5 * g * (g + 1), slots = (double)nsm * Cf::MINB;
    return (double)N * N / (std::ceil(items / slots) * slots * gs * gs);
  };
  *GS = tb * ((N + tb - 1) / tb);  // one group
  *G = 1;
  double best = 0.0;
  for (int pass = 0; pass < 2; pass++)
    for (long g = 2; g <= max_slots; g++) {
      const long gs = ((N + g - 1) / g + tb - 1) / tb * tb;
      if ((N + gs - 1) / gs != g) continue;
      const double e = eff(g, gs);
      if (pass == 0) {
        best = std::max(best, e);
      } else if (e >= 0.98 * best) {
        *G = (int)g;
        *GS = gs;
        return;
      }
    }
}

struct SymPlan {
  bool small = false;
  int G = 1;
  long GS = 0;
};

// SMALL while its groups can be single blocks of targets: N <= kMaxSlots blocks (20,480 points). One
// block of the larger form against another is 233 us on an SM by itself and 99 us beside two more, so
// few items take it long. us at 8,704 / 13,056 / 17,408 / 21,760 points, SMALL and not: single layer 134 and
// 262, 253 and 318, 426 and 519, 846 and 738; double layer 149 and 194, 276 and 348, 465 and 571, 897 and 830.
template <bool DL>
SymPlan sym_plan(long N, long max_slots, int nsm) {
  SymPlan p;
  p.small = N <= kMaxSlots * SymCfg<DL, true>::TB;
  max_slots = std::min(max_slots, kMaxSlots);
  if (p.small)
    sym_groups<SymCfg<DL, true>>(N, max_slots, nsm, &p.G, &p.GS);
  else
    sym_groups<SymCfg<DL, false>>(N, max_slots, nsm, &p.G, &p.GS);
  return p;
}

int sm_count() {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

template <bool DL, bool SMALL>
int launch_sym(const SymPlan& pl, const double* pos, const double* den, const double* nrm, const long* off, long nves,
               long N, double* part, cudaStream_t st) {
  using Cf = SymCfg<DL, SMALL>;
  VES3D_CK(cudaFuncSetAttribute(k_far_sym_f64<DL, SMALL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cf::SMEM));
  k_far_sym_f64<DL, SMALL><<<(unsigned)(pl.G * (pl.G + 1) / 2), Cf::NT, Cf::SMEM, st>>>(pos, den, nrm, off, nves, N,
                                                                                      pl.G, pl.GS, part);
  VES3D_LAUNCHED();
  return VES3D_OK;
}

template <bool DL>
int launch_plan(const double* pos, const double* den, const double* nrm, const long* off, long nves, long N,
                double* part, long max_slots, cudaStream_t st, int* nslots) {
  const SymPlan pl = sym_plan<DL>(N, max_slots, sm_count());
  *nslots = pl.G;
  return pl.small ? launch_sym<DL, true>(pl, pos, den, nrm, off, nves, N, part, st)
                  : launch_sym<DL, false>(pl, pos, den, nrm, off, nves, N, part, st);
}

}  // namespace

// Groups (sets of partial sums) that the sums over N points are cut into, given room for max_slots.
static long groups_of(long N, long max_slots) {
  const int nsm = sm_count();
  return std::max(sym_plan<false>(N, max_slots, nsm).G, sym_plan<true>(N, max_slots, nsm).G);
}

// Partial sums within a GiB, or kFarMaxSegments sets.
static long slot_limit(long N) {
  return std::max(kFarMaxSegments, std::min(kMaxSlots, (long)((size_t)1 << 30) / (24 * std::max(N, 1L))));
}

long far_slots(long N) {
  return N < kFarSymMin ? kMaxSlots : std::max(kFarMaxSegments, groups_of(N, slot_limit(N)));
}

long alltoall_slots(long np) {
  if (np < kPairsMin || slot_limit(np) <= kFarMaxSegments) return 0;
  return groups_of(np, slot_limit(np));
}

int launch_far_sym(const double* pos, const double* den, const double* nrm, const long* off, long nves, long N,
                   double* part, long max_slots, cudaStream_t st, int* nslots) {
  return nrm ? launch_plan<true>(pos, den, nrm, off, nves, N, part, max_slots, st, nslots)
             : launch_plan<false>(pos, den, nrm, off, nves, N, part, max_slots, st, nslots);
}

}  // namespace ves3d
