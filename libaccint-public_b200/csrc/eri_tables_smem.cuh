// Lookup tables staged in shared memory by the persistent ERI kernels: the Boys
// grid (one-root classes) or the class's Rys root table, with row strides padded
// so that lanes reading different rows fall into different banks (a warp's
// per-lane gathers from global memory would touch up to 32 cache lines per load
// instruction).  Same arithmetic as rys_eval.h.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "eri_device.cuh"
#include "rys_eval.h"

namespace lai {

// Shared-memory table layouts, in elements of the compute type R (the FP32 kernels
// stage FP32 copies: half the shared memory, and single-width loads).
//
// (A layout with the Taylor coefficients pre-divided by j!, which saves the x/j
// products, was measured slower: its 18-double rows take more shared memory, and
// the carve-out shrinks L1, which these kernels lean on.)
// FP64 rows: F_0..F_9 at T0 = k / 10 (five 16-byte units, odd, so lanes on
// different rows spread over the banks).
constexpr int kBoysRowsS = kBoysNGrid;
constexpr double kBoysTmaxS = kBoysTmax;
constexpr int kBoysRowS = 10;
constexpr int kBoysRowF = 12;     // FP32: F_0..F_11, three 16-byte units (odd)
template <typename R>
__host__ __device__ constexpr int boys_row() { return sizeof(R) == 8 ? kBoysRowS : kBoysRowF; }
template <typename R>
__host__ __device__ constexpr int boys_rows() { return sizeof(R) == 8 ? kBoysRowsS : kBoysNGrid; }
template <int NR>
__host__ __device__ constexpr int rys_row() { return 24 * NR + 2; }  // 12 degrees x NR x (u,w) + pad
template <int NR, typename R>
__host__ __device__ constexpr int table_elems() {
  return NR == 1 ? boys_rows<R>() * boys_row<R>() : rys_tmax_c(NR) * rys_row<NR>();
}
// 1.5 * 2^52: adding it to a double y with 0 <= |y| < 2^31 leaves rint(y) in the
// low word of the sum (round to nearest even), with no conversion instruction.
constexpr double kRoundMagicD = 6755399441055744.0;
template <int NR, typename R>
__host__ __device__ constexpr size_t table_bytes() {
  return (sizeof(R) * table_elems<NR, R>() + 15) & ~size_t(15);  // what follows stays 16-byte aligned
}

template <int NR, typename R>
__device__ __forceinline__ void stage_table(R* __restrict__ st, const RysTablesView& tab) {
  if constexpr (NR == 1 && sizeof(R) == 8) {
    constexpr int NV = kBoysRowS;
    for (int i = threadIdx.x; i < kBoysRowsS * NV; i += blockDim.x) {
      const int k = i / NV, j = i - k * NV;
      st[k * NV + j] = __ldg(tab.boys + k * kBoysNM + j);
    }
  } else if constexpr (NR == 1) {
    constexpr int NV = boys_row<R>();  // values per row (the row holds no padding)
    for (int i = threadIdx.x; i < kBoysNGrid * NV; i += blockDim.x) {
      const int k = i / NV, j = i - k * NV;
      st[k * NV + j] = R(__ldg(tab.boys + k * kBoysNM + j));
    }
  } else {
    constexpr int W = 24 * NR;
    const double* src = tab.coef + rys_off(NR);
    for (int i = threadIdx.x; i < rys_tmax_c(NR) * W; i += blockDim.x) {
      const int k = i / W, j = i - k * W;
      st[k * rys_row<NR>() + j] = R(__ldg(src + i));
    }
  }
}

// F_0(T) and F_1(T) from the staged Boys grid (the Taylor series of boys01 in
// rys_eval.h; FP64 from the pre-divided rows).
template <typename R>
__device__ __forceinline__ void boys01_smem(R T, const R* __restrict__ st, R& F0, R& F1) {
  constexpr bool F64 = sizeof(R) == 8;
  if constexpr (F64) {
    // FP64: nearest grid point by the rounding constant (no conversion
    // instructions), 8-term Taylor series (first omitted term below 6e-17 relative)
    if (T < kBoysTmaxS) {
      const double km = fma(double(T), 10.0, kRoundMagicD);
      const int k = min(__double2loint(km), kBoysRowsS - 1);
      const double x = fma(km - kRoundMagicD, 0.1, -double(T));
      const double2* f = reinterpret_cast<const double2*>(st + k * kBoysRowS);
      double g[10];
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const double2 v = f[j];
        g[2 * j] = v.x;
        g[2 * j + 1] = v.y;
      }
      double a, b;
      boys_taylor<double>(x, g, a, b);
      F0 = R(a);
      F1 = R(b);
    } else {
      const R rt = fast_rsqrt(T);
      F0 = R(0.88622692545275801365) * rt;  // sqrt(pi)/2
      F1 = R(0.5) * F0 * rt * rt;
    }
  } else {
    // FP32: nearest grid point; T just below kBoysTmax can round up to the row past
    // the end, hence the clamp
    if (T < R(kBoysTmax)) {
      const int k = min(__float2int_rn(float(T) * 10.0f), kBoysNGrid - 1);
      const R x = R(k) * R(0.1) - T;
      constexpr int NG = boys_terms<R>() + 1;  // grid values used: F_0..F_N
      R g[12];
      const float4* f = reinterpret_cast<const float4*>(st + k * kBoysRowF);
#pragma unroll
      for (int j = 0; j < (NG + 3) / 4; ++j) {
        const float4 v = f[j];
        g[4 * j] = v.x;
        g[4 * j + 1] = v.y;
        g[4 * j + 2] = v.z;
        g[4 * j + 3] = v.w;
      }
      boys_taylor<R>(x, g, F0, F1);
    } else {
      const R rt = fast_rsqrt(T);
      F0 = R(0.88622692545275801365) * rt;  // sqrt(pi)/2
      F1 = R(0.5) * F0 * rt * rt;
    }
  }
}

// Boys rows for F_0 .. F_L, L <= 3 (the thread-per-quartet kernels of the low classes).
// Row k, of 10 doubles (five 16-byte units, odd, so lanes on different rows spread over
// the banks), holds Taylor coefficients about T0 = k / 10, divided by j!:
//   L = 0: F_j / j!, j < 8;  L = 1: F_j / j!, j < 9 (F_1 is the derivative of the same
//   polynomial);  L >= 2: F_{L+j} / j!, j < 8, and exp(-T0), for the downward recursion
//   F_{m-1} = (2 T F_m + exp(-T)) / (2m - 1).
// The first omitted term is below 0.05^8/8!/17 = 6e-17.  Above the grid the asymptotic
// forms hold to 1e-16 of F_L: from 39.95 (L <= 1), 45.95 (L = 2, 3; the rows past the
// stored grid come from F_0 = sqrt(pi/T)/2 and the upward recursion).
constexpr int kBoysRowLen = 10;
template <int L>
__host__ __device__ constexpr int boys_rows_n() { return L <= 1 ? kBoysNGrid : 461; }
template <int L>
__host__ __device__ constexpr double boys_rows_tmax() { return L <= 1 ? kBoysTmax : 45.95; }
template <int L>
__host__ __device__ constexpr size_t boys_rows_bytes() { return sizeof(double) * kBoysRowLen * boys_rows_n<L>(); }

template <int L>
__device__ __forceinline__ void stage_boys_rows(double* __restrict__ st, const RysTablesView& tab) {
  constexpr int NV = L == 1 ? 9 : 8;
  for (int k = threadIdx.x; k < boys_rows_n<L>(); k += blockDim.x) {
    double* row = st + k * kBoysRowLen;
    double F[L + 9];
    const double T = k * 0.1, e = L >= 2 ? exp(-T) : 0.0;
    if (k < kBoysNGrid) {
#pragma unroll
      for (int j = 0; j < L + 9; ++j) F[j] = __ldg(tab.boys + k * kBoysNM + j);
    } else {
      F[0] = 0.88622692545275801365 * rsqrt(T);
#pragma unroll
      for (int j = 0; j < L + 8; ++j) F[j + 1] = ((2 * j + 1) * F[j] - e) / (2.0 * T);
    }
    constexpr int m0 = L >= 2 ? L : 0;
    double f = 1.0;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      row[j] = F[m0 + j] * f;
      f /= j + 1;
    }
    if (L >= 2) row[8] = e;
  }
}

template <int L>
__device__ __forceinline__ void boys_rows(double T, const double* __restrict__ st, double (&F)[L + 1]) {
  static_assert(L >= 0 && L <= 3, "F_0 .. F_3");
  if (T < boys_rows_tmax<L>()) {
    const double km = fma(T, 10.0, kRoundMagicD);  // nearest row (no conversion instructions)
    const int k = min(__double2loint(km), boys_rows_n<L>() - 1);
    const double x = fma(km - kRoundMagicD, 0.1, -T);
    const double2* r = reinterpret_cast<const double2*>(st + k * kBoysRowLen);
    double g[10];
#pragma unroll
    for (int j = 0; j < (L == 0 ? 4 : 5); ++j) {
      const double2 v = r[j];
      g[2 * j] = v.x;
      g[2 * j + 1] = v.y;
    }
    if constexpr (L == 1) {
      double a = fma(g[8], x, g[7]), d = g[8];  // polynomial and its derivative
#pragma unroll
      for (int j = 6; j >= 0; --j) {
        d = fma(d, x, a);
        a = fma(a, x, g[j]);
      }
      F[0] = a;
      F[1] = d;
    } else {
      double a = g[7];
#pragma unroll
      for (int j = 6; j >= 0; --j) a = fma(a, x, g[j]);
      F[L] = a;
      if constexpr (L >= 2) {
        // exp(-T) = exp(-T0) exp(x), |x| <= 0.05: degree 8 leaves 0.05^9/9! = 5e-18
        constexpr double c[9] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320};
        double ex = c[8];
#pragma unroll
        for (int j = 7; j >= 0; --j) ex = fma(ex, x, c[j]);
        ex *= g[8];
        const double t2 = T + T;
#pragma unroll
        for (int m = L; m >= 1; --m) F[m - 1] = fma(t2, F[m], ex) * (1.0 / (2 * m - 1));
      }
    }
  } else {
    const double rt = fast_rsqrt(T);
    F[0] = 0.88622692545275801365 * rt;  // sqrt(pi)/2
    const double h = 0.5 * rt * rt;
#pragma unroll
    for (int m = 1; m <= L; ++m) F[m] = (2 * m - 1) * h * F[m - 1];
  }
}

// Roots/weights of the NR-point Rys rule from the staged table (same arithmetic
// as rys_roots_table in rys_eval.h).
template <int NR, typename R>
__device__ __forceinline__ void rys_smem(R T, const R* __restrict__ st, const RysTablesView& tab,
                                         R* __restrict__ u, R* __restrict__ w) {
  constexpr bool F64 = sizeof(R) == 8;
  if constexpr (NR == 1) {
    if (T < R(kBoysTmax)) {
      R F0, F1;
      boys01_smem<R>(T, st, F0, F1);
      u[0] = fast_div(F1, F0);
      w[0] = F0;
    } else {
      rys1_asymptotic<R>(T, u[0], w[0]);
    }
  } else {
    if (T < R(rys_tmax_c(NR))) {
      int k;
      R x;
      if constexpr (F64) {
        // unit interval by the rounding constant: rint(T - 1/2) (an integer T may
        // land on the interval below, at its end x = 1)
        const double km = (double(T) - 0.5) + kRoundMagicD;
        k = __double2loint(km);
        x = fma(2.0, double(T) - (km - kRoundMagicD), -1.0);
      } else {
        k = (int)T;
        x = R(2) * (T - R(k)) - R(1);
      }
      using V2 = typename std::conditional<F64, double2, float2>::type;
      const V2* c = reinterpret_cast<const V2*>(st + k * rys_row<NR>());
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const V2 v = c[kRysDeg * NR + r];
        u[r] = v.x;
        w[r] = v.y;
      }
#pragma unroll
      for (int j = kRysDeg - 1; j >= 0; --j)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const V2 v = c[j * NR + r];
          u[r] = u[r] * x + v.x;
          w[r] = w[r] * x + v.y;
        }
    } else {
      const R rt = fast_rsqrt(T);
      const R it = rt * rt;
      const int h = rys_hoff(NR);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        u[r] = R(__ldg(tab.herm_x2 + h + r)) * it;
        w[r] = R(__ldg(tab.herm_w + h + r)) * rt;
      }
    }
  }
}

}  // namespace lai
