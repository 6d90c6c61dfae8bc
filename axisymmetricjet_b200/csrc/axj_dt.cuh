// axj_dt.cuh -- the point scan of ComputeTimeStep (ModInputOutput.f90:389-438), shared by the
// handle-based and the allocation-free time-step kernels.
//
// dt is the minimum of CFL / x over the points, x the point's inviscid plus viscous rate. In
// FP64 x costs about fifty instructions per point (two square roots, T**0.666 with its table
// loads), which bound the kernels at 35-48 us for 2.8 M points when the 24 B/point they read
// take 10 us; but only the points near the largest x need it. A block therefore first forms an
// FP32 estimate of x for its points with the approximate square root, log2 and exp2 units
// (relative error of the parts well below 1e-5), takes the largest estimate, and evaluates
// x in FP64 only where the estimate lies within DT_SCREEN of the parts' magnitudes of that.
// The margin is an order of magnitude wider than the estimate's error, so the point of the
// largest x is always among them and the result is the full FP64 scan's, bit for bit.
// Estimates that are not finite (NaN or infinite inputs, FP32 overflow) and points where FP32
// underflows (below) are always evaluated in FP64. The largest lower bound seen so far is handed
// from block to block through a word in global memory (a hint: any value it holds is a valid
// bound), so that most blocks evaluate no point in FP64 at all.
// Measured at 4400 x 640 on a B200: a call of the allocation-free entry point 55.4 -> 22.7 us, the
// handle's kernel 27.0 -> 20.1 us (within a step, with the state out of the caches, 35.4 -> 21.2).
#pragma once

#include <cuda_runtime.h>

#include "axj_common.cuh"

namespace axj {

// Screened, a warp takes strips of 32 columns by DT_K rows: the z metric is loaded and converted
// once per strip, the row's by one lane. Otherwise one point per thread, in row order.
constexpr int DT_K = 4;
constexpr int DT_WARPS = DT_THREADS / 32;
// A scan in FP64 throughout takes 8.5 us + 19 ps a point (a call of the allocation-free entry
// point on a B200), a screened one 9.6 us + 4.6 ps for each of its strips' 32-column slots, used
// or not: the screened one wins above DT_FULL points in full strips, above ever more
// points the more slots are idle, and in no grid of 10 columns or fewer. Measured (FP64 / screened):
// 256 x 384 10.1 / 10.3 us, 787 x 203 10.8 / 10.3, 1801 x 333 18.5 / 12.4, 4400 x 640 55 / 22; 33 x 10000
// 14.0 / 13.1, 12 x 20000 12.5 / 12.8, 12 x 200000 47 / 37, 8 x 500000 78 / 81, 1 x 2097152 42 / 287.
constexpr long long DT_FULL = 98304;
__host__ __device__ inline bool dt_screened(int Nz, int Nr) {
  const long long n = (long long)Nz * Nr, slots = (long long)((Nz + 31) / 32 * 32) * Nr;
  return 3 * n > slots + 2 * DT_FULL;
}
// Strips of a screened grid, and a scan's blocks: a strip per warp up to one resident wave, or a
// point per thread.
__host__ __device__ inline long long dt_strips(int Nz, int Nr) {
  return (long long)((Nz + 31) / 32) * ((Nr + DT_K - 1) / DT_K);
}
constexpr long long DT_WAVE = 148 * 4;  // (a launch shape only: the blocks loop, on any number of SMs)
__host__ __device__ inline long long dt_blocks(int Nz, int Nr, bool screen) {
  if (!screen) return ((long long)Nz * Nr + DT_THREADS - 1) / DT_THREADS;
  const long long b = (dt_strips(Nz, Nr) + DT_WARPS - 1) / DT_WARPS;
  return b < DT_WAVE ? b : DT_WAVE;
}
constexpr float DT_SCREEN = 1.220703125e-4f;   // 2**-13
constexpr float DT_TINY = 1.0e-30f;            // absolute margin (subnormal products)
// Underflow: the approximate units flush subnormals, so a T, or a sum of squared metrics, below FP32's
// normal range loses its part of the estimate, and a T that is negative but small is no NaN. The
// points of a lane whose z metric's square or least T is below that range are therefore evaluated
// in FP64 whatever their estimates (which, being too small, are still valid lower bounds).
// Otherwise what underflows is below the margin, for velocities up to 1e15 or metrics that are
// zero or normal in FP32; the stale T and the viscous factors are tested once per launch
// (dt_factors). Overflow needs no test: an infinite estimate is evaluated too.
constexpr float DT_NORMAL = 1.17549435e-38f;

__device__ __forceinline__ float f_sqrt(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float f_lg2(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float f_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct DtScan {
  const double* U;       // 5 planes of Nr rows, pitch P
  long long P, plane;    // row pitch, plane size
  int Nz, Nr;
  const double* dxidz;
  const double* detadr;
  bool phys;     // sound speed from the point's T (else sqrt_stale)
  float sqrt_stale, inv_Re, inv_RePr;
  bool factors_ok;  // these are in the estimate's range (dt_factors)
};
__device__ __forceinline__ void dt_factors(DtScan& s, double staleT, double inv_Re, double inv_RePr) {
  s.sqrt_stale = f_sqrt((float)staleT);
  s.inv_Re = (float)inv_Re;
  s.inv_RePr = (float)inv_RePr;
  const float inv = fminf(fabsf(s.inv_Re), fabsf(s.inv_RePr));
  // (a stale T of zero, as before the first step, leaves no sound term to cover a lost viscous one)
  s.factors_ok = s.phys || (staleT >= DT_NORMAL ? inv >= DT_NORMAL : staleT == 0.0 && inv >= 1.0e-12f);
}

// One strip of 32 columns x DT_K rows of a screened scan, by one warp. blanked(o): whether the
// point at offset o is blanked (counted in nblank); exact(i, j, o): the FP64 evaluation. sL: the
// largest lower bound the block knows (float bits in shared memory, zeroed by the caller before
// a barrier; it only grows, any value it holds is a valid bound, and no warp waits for
// another's); hint: the launch's.
template <class Blanked, class Exact>
__device__ __forceinline__ void dt_scan_strip(const DtScan& s, unsigned strip, unsigned* sL, unsigned* hint,
                                              int& nblank, Blanked blanked, Exact exact) {
  constexpr int K = DT_K;
  // (a grid that fits the device has far fewer than 2**31 strips)
  const unsigned ncs = (unsigned)(s.Nz + 31) / 32u, lane = threadIdx.x & 31u;
  const unsigned rg = strip / ncs;
  const int j0 = (int)(rg * K), nrow = min(K, s.Nr - j0);
  const int iu = (int)((strip - rg * ncs) * 32u + lane), i = min(iu, s.Nz - 1);
  const long long o0 = (long long)j0 * s.P + i;
  unsigned cand = 0;  // rows to evaluate in FP64
  // every load of the strip first (none depends on another), then the estimates
  double vr[K], vz[K], tt[K];
  bool bl[K];
  const double* u = s.U + o0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const long long o = min(k, nrow - 1) * s.P;  // rows past the grid repeat the last one
    bl[k] = blanked(o0 + o);
    vr[k] = __ldg(u + s.plane + o);
    vz[k] = __ldg(u + 3 * s.plane + o);
    tt[k] = __ldg(u + 4 * s.plane + o);
  }
  const float x = (float)__ldg(s.dxidz + i);
  const float yl = (float)__ldg(s.detadr + j0 + min((int)lane, nrow - 1));
  float up[K];      // upper bound of x
  float lo = 0.0f;  // largest lower bound
  float tl = DT_NORMAL;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float y = __shfl_sync(0xffffffffu, yl, k);
    const float Vr = (float)vr[k], Vz = (float)vz[k], T = (float)tt[k];
    const float a = Vz * x, b = Vr * y;
    const float g2 = x * x + y * y;
    const float gs = f_sqrt(g2);
    const float snd = (s.phys ? f_sqrt(T) : s.sqrt_stale) * gs;
    const float mu = f_ex2(0.666f * f_lg2(T));
    tl = fminf(tl, T);  // (a NaN makes its own estimate one)
    const float lam = (0.6f - 2.0f / 3.0f) * mu;
    const float mx = fmaxf(fmaxf(mu, lam) * s.inv_Re, mu * s.inv_RePr);
    const float d = fabsf(x) + fabsf(y);
    const float visc = 2.0f * mx * (d * d);
    const float est = fabsf(a + b) + snd + visc;
    const float mar = DT_SCREEN * (fabsf(a) + fabsf(b) + snd + fabsf(visc)) + DT_TINY;
    up[k] = est + mar;
    // (a repeated row or column counts once more: the same bound, no point of its own)
    if (bl[k]) {
      nblank = 1;
    } else {
      lo = fmaxf(lo, est - mar);  // (fmaxf drops a NaN)
      if (k < nrow && iu < s.Nz) cand |= 1u << k;
    }
  }
  // a lower bound that overflowed says nothing
  const unsigned lob = lo <= 3.0e38f ? __float_as_uint(lo) : 0u;
  const unsigned w = __reduce_max_sync(0xffffffffu, lob);
  const unsigned b = max(*reinterpret_cast<volatile unsigned*>(sL), w);
  if (lane == 0 && b == w) atomicMax(sL, w);
  if (threadIdx.x == 0) {
    const unsigned h = *reinterpret_cast<volatile unsigned*>(hint);
    if (h > b) atomicMax(sL, h);  // for the strips to come
    else if (h < b) atomicMax(hint, b);
  }
  const bool ok = s.factors_ok && x * x >= DT_NORMAL && tl >= DT_NORMAL;
  const float thr = ok ? __uint_as_float(b) : -1.0f / 0.0f;
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (up[k] < thr) cand &= ~(1u << k);
#pragma unroll 1
  for (int k = 0; k < K; ++k)
    if ((cand >> k) & 1u) exact(i, j0 + k, o0 + k * s.P);
}

// The points of block blk of nblk.
template <bool SCREEN, class Blanked, class Exact>
__device__ __forceinline__ void dt_scan(const DtScan& s, unsigned blk, unsigned nblk, unsigned* sL, unsigned* hint,
                                        int& nblank, Blanked blanked, Exact exact) {
  if constexpr (SCREEN) {
    const unsigned n = (unsigned)dt_strips(s.Nz, s.Nr);
    for (unsigned st = blk * DT_WARPS + (threadIdx.x >> 5); st < n; st += nblk * DT_WARPS)
      dt_scan_strip(s, st, sL, hint, nblank, blanked, exact);
  } else {
    // (a grid that fits the device has fewer than 2**32 points)
    const unsigned n = (unsigned)s.Nz * (unsigned)s.Nr, step = nblk * DT_THREADS;
    for (unsigned p = blk * DT_THREADS + threadIdx.x; p < n; p += step) {
      const int j = (int)(p / (unsigned)s.Nz), i = (int)(p - (unsigned)j * (unsigned)s.Nz);
      const long long o = (long long)j * s.P + i;
      if (blanked(o)) nblank = 1;
      else exact(i, j, o);
      if (p + step < p) break;
    }
  }
}

}  // namespace axj
