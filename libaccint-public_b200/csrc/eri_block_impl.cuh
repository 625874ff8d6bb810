// Block-per-quartet Rys ERI kernel for the classes with too many integrals for one
// thread: compile-time specialised on the ket (lc, ld), any bra (la, lb).  J/K digestion
// only (the raw-integral and Schwarz modes stay on the tiled kernel).
//
// One block of 32-192 threads per quartet; thread e owns row e of the contracted
// (e0|f0) block, e over the Cartesian components of shells la..la+lb, and holds
// G[f] for every component f of the ket shells F0..F1 in registers:
//   1. table phase: for up to `batch` primitive quartets at once, one thread per
//      (primitive quartet, root, direction) builds I(e, f) by the vertical recurrence
//      of eri_device.cuh, columns in registers, and stores it to shared memory;
//   2. accumulation: per root every thread reads its rows Ix(ex, .), Iy(ey, .),
//      Iz(ez, .), 3 (lc+ld+1) values, and updates all its G[f] from them, so a shared
//      load feeds NF / (3 (lc+ld+1)) products (74/21 for an (ff| ket) where a kernel
//      that owns scattered integrals needs three loads for each;
//   3. once per contracted quartet, for a chunk of ket components c at a time: the ket
//      transfer (e0|f0) -> (e0|c d) from registers, the bra transfer -> (ab|c d) per
//      thread (a, b), and the six Fock blocks from it.  Everything after G is linear in
//      G, and the chunks are independent, which gives three freedoms: with few quartets
//      in a launch, a quartet's primitive quartets and then its chunks are split over
//      several blocks, and the two largest kets, whose G does not fit a thread's
//      registers ((gf| 100 and (gg| 145 values), run as two launches over the shells
//      F0..F1 of f.
// The density blocks arrive by cp.async behind the table phase.
//
// Expansion centre.  The transfer writes (x-A)^a (x-B)^b in powers of x-A, and where A lies
// far from the charge the terms are large and cancel: on one side by up to some ten times, on
// both sides by the product.  Applied per root to the 2-D tables, as the tiled kernel does,
// it costs the sum over directions; applied to the contracted block the product over
// directions and sides: K' of (ff|ff) in H2O/cc-pVQZ was off by 4.8e-14 of its norm where the
// tiled kernel is off by 2.1e-15.  So a ket with ld >= 2, and a bra with la >= 3 and lb >= 2
// against a ket with ld >= 1 (from lb = 3 also (ds|, (fs| and (gs| kets; template parameter
// BM), are expanded about M, the centre P of the pair's first primitive: powers 0..la+lb of
// x-M, (x-A)^a = (x-M + M-A)^a and the same for B, whose terms are as large as the charge
// makes them.  K' of (ff|ff): 1.5e-15; J and K of H2O/cc-pVQZ, in three geometries, 7e-15 to
// 1e-14 before and 4e-15 now.  The other classes are as exact as the tiled kernel without it.
// It costs rows ((fd| 56 for 46) and longer bra sums (prod (a_x + b_x + 1) terms for
// prod (b_x + 1)): (fd|dp) of C6H14/cc-pVTZ 2.37 -> 2.72 ms, the build 84.2 -> 86.1 ms.
//
// R = double, or float for the FP32 part of a mixed-precision build (roots, tables and the
// primitive sums in G in FP32; the primitive-pair quantities up to T and the prefactor,
// and everything after G, in FP64).
// The row strides in shared memory are odd multiples of 16 bytes, so that the 16-byte
// loads of threads on different rows fall into different banks.
//
// Bound: latency (tables, block syncs) for small blocks, FP64 issue for the f and g
// kets.  Against the tiled kernel, which repeated its table and digestion sweeps for
// every 512 integrals: see the dispatch rule in eri_block.cu.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "eri_device.cuh"
#include "eri_kernels.h"

namespace lai {
namespace block_detail {

template <int B, int E, typename F>
__device__ __forceinline__ void bfor(F&& f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    bfor<B + 1, E>(f);
  }
}

// smallest odd number of 16-byte units that holds n values of type R, in values
template <typename R = double>
__host__ __device__ constexpr int odd_stride(int n) {
  constexpr int u = 16 / sizeof(R);
  return u * (((n + u - 1) / u) | 1);
}

constexpr int kMaxThreads = 160;     // components of (gg| about A: 145
constexpr int kMaxThreadsMid = 192;  // and about M: 165
constexpr int kMaxTerms = 12;     // transfer terms of a g component: (2,1,1) -> 3 * 2 * 2
constexpr int kMaxLab = 2 * kMaxL;
constexpr int kMaxSmem = 226 * 1024;  // of 227 KB, less the static part

// Registers: left alone, ptxas takes 255 for any ket and a block of 32 threads ends up with
// 8 warps per SM, each waiting on its own arithmetic and shared-memory latency (ncu, (dd|dp):
// issue active 30 %, stalls `wait` and `short_scoreboard`).  Caps of 96 and 128 registers
// (65536 / (160 * blocks)) pay for the kets of few components, C6H14/cc-pVTZ without and
// with them: (fd|ps) 4.9 -> 3.5 ms, (ff|ps) 1.6 -> 0.9, (fs|dp) 4.8 -> 4.0, but (dd|pp) 2.5
// -> 2.8; with the bra about M (fd|pp) 3.07 -> 2.79, (ff|pp) 1.26 -> 0.73; from 25 components on the spills cost more ((dd|fp) 1.2 ->
// 1.6 with 128).
template <int F0, int F1, bool BM>
__host__ __device__ constexpr int min_blocks() {  // (BM: blocks of 192 threads, nearly the same caps)
  constexpr int nf = ncart_range(F0, F1);
  return nf <= 10 ? 4 - BM : nf <= 16 ? 3 - BM : 1;
}

__host__ __device__ constexpr int block_binom(int n, int k) {
  int r = 1;
  for (int i = 0; i < k; ++i) r = r * (n - i) / (i + 1);
  return r;
}
__device__ __forceinline__ double block_pow(double x, int m) {
  double r = 1.0;
  for (int i = 0; i < m; ++i) r *= x;
  return r;
}

// Expansion about M instead of the first shell's centre (see above).
template <int LD, typename R>
__host__ __device__ constexpr bool mid_ket() { return sizeof(R) == 8 && LD >= 2; }
template <int LC, int LD, typename R>
__host__ __device__ constexpr bool mid_bra_possible() { return sizeof(R) == 8 && (LD >= 1 || LC >= 2); }
__host__ __device__ constexpr bool mid_bra(int la, int lb, int ld) { return la >= 3 && lb >= (ld > 0 ? 2 : 3); }

// out[k] = coefficient of x^k in (x + p)^i (x + q)^j, k <= i + j < N.
template <int N>
__device__ __forceinline__ void mid_coefs(double p, double q, int i, int j, double* out) {
  double c[N];
  c[0] = 1.0;
#pragma unroll
  for (int k = 1; k < N; ++k) c[k] = 0.0;
  for (int m = 0; m < i + j; ++m) {
    const double r = m < i ? p : q;
#pragma unroll
    for (int k = N - 1; k > 0; --k) c[k] = c[k - 1] + r * c[k];
    c[0] *= r;
  }
#pragma unroll
  for (int k = 0; k < N; ++k)
    if (k <= i + j) out[k] = c[k];
}

// Ket components c per digestion chunk (a divisor of the shell's count): enough values
// per thread (a, b) to keep a chunk's phases busy, few enough to stay in registers
// beside G.
__host__ __device__ constexpr int chunk_components(int lc, int ld) {
  return lc == 0 ? 1 : lc == 1 ? 3 : lc == 2 ? (ld == 2 ? 3 : 6)
         : lc == 3 ? (ld == 0 ? 10 : ld == 1 ? 5 : ld == 2 ? 2 : 1)
                   : (ld == 0 ? 15 : ld == 1 ? 5 : ld == 2 ? 3 : 1);
}

// Runtime geometry of a launch and its shared-memory layout (in doubles).
struct BlockGeom {
  int la, lb, nroots, ne, nab, na, nb;
  int batch;     // primitive quartets per table phase
  int chunk;     // consecutive work items a block takes at a time
  int ts;        // one direction's table: (la + lb + 1) * row stride, in values
  int nacc;      // density elements of a quartet: D_ab, D_cd, D_ac, D_ad, D_bc, D_bd
  int o_tab, o_h, o_v, o_r1, o_r2, o_jp, o_d, o_jab, o_kad, o_kbd, o_cob, o_cod, o_nab, o_ncd, o_int;
  int doubles;   // total, including the integer tables at o_int
};

template <int LC, int LD, typename R, bool BM>
__host__ BlockGeom make_geom(int la, int lb, int threads, int batch) {
  constexpr int W = LC + LD + 1, WS = odd_stride<R>(W), ND = ncart(LD), NC = ncart(LC);
  constexpr int CB = chunk_components(LC, LD), NV = CB * ND, NVP = odd_stride(NV);
  static_assert(NC % CB == 0, "chunks of equal size");
  BlockGeom g{};
  g.la = la; g.lb = lb;
  g.nroots = (la + lb + LC + LD) / 2 + 1;
  g.ne = ncart_range(BM ? 0 : la, la + lb);
  g.na = ncart(la); g.nb = ncart(lb); g.nab = g.na * g.nb;
  g.nacc = g.nab + NC * ND + g.na * NC + g.na * ND + g.nb * NC + g.nb * ND;
  g.batch = batch;
  g.ts = (la + lb + 1) * WS;
  int o = 0;
  auto take = [&](int n) { const int at = o; o += (n + 1) & ~1; return at; };
  g.o_tab = take((int)(batch * g.nroots * 3 * g.ts * sizeof(R) / 8));
  g.o_h = take(g.ne * NVP);
  g.o_v = take(g.nab * NVP);
  g.o_r1 = take(g.nab * CB);
  g.o_r2 = take(g.nab * CB);
  g.o_jp = take(g.na * NV);
  g.o_d = take(g.nacc);
  g.o_jab = take(g.nab);
  g.o_kad = take(g.na * ND + g.nb * ND);
  g.o_kbd = g.o_kad + g.na * ND;
  g.o_cob = take(BM ? 3 * (la + 1) * (lb + 1) * (la + lb + 1) : g.nb * kMaxTerms);
  g.o_cod = take(mid_ket<LD, R>() ? 3 * (LC + 1) * (LD + 1) * W : ND * kMaxTerms);
  g.o_nab = take(g.nab);
  g.o_ncd = take(NC * ND);
  g.o_int = o;
  // integers: list of primitive quartets (64-bit), (e0| index of every bra term (BM: of every
  // power of x, y and z), per-b term count, coefficient and powers, the same coefficients
  // and powers for the ket, row and column of every density element
  const int terms = BM ? (la + lb + 1) * (la + lb + 1) * (la + lb + 1) : g.nab * kMaxTerms;
  const int ints = 2 * threads + terms + g.nb * (1 + 2 * kMaxTerms) + ND * 2 * kMaxTerms + g.nacc + 8;
  o += (ints + 1) / 2;
  g.doubles = (o + 1) & ~1;
  return g;
}

// 8-byte asynchronous copy to shared memory, and the wait for this thread's copies
__device__ __forceinline__ void copy_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// largest p with offsets[p] <= t, by a 32-way search of the whole warp
__device__ __forceinline__ int find_bra_warp(const int64_t* __restrict__ offsets, int npairs, int64_t t) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = npairs;  // offsets[lo] <= t < offsets[hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32;
    const int at = lo + lane * step;
    const bool le = at < hi && __ldg(offsets + at) <= t;
    const unsigned m = __ballot_sync(0xffffffffu, le);  // lane 0 always holds
    const int k = 31 - __clz(m);
    lo += k * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

template <int LC, int LD, int F0, int F1, typename R, bool BM>
__global__ void __launch_bounds__((BM ? kMaxThreadsMid : kMaxThreads), (min_blocks<F0, F1, BM>()))
    eri_block_kernel(QuartetBlock one, JKArgs args, RysTablesView tab, BlockGeom g, int nsplit1, int csplit1,
                     const MultiEntry* list_of_blocks, int nblocks, int64_t nwork) {
  constexpr int LCD = LC + LD, W = LCD + 1, WS = odd_stride<R>(W);
  constexpr int NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
  constexpr int CB = chunk_components(LC, LD), NV = CB * ND, NVP = odd_stride(NV);
  constexpr int NF = ncart_range(F0, F1);
  constexpr bool KM = mid_ket<LD, R>();
  extern __shared__ __align__(16) double smem_b[];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  const int la = g.la, lb = g.lb, LAB = la + lb, NR = g.nroots;
  const int NE = g.ne, NA = g.na, NB = g.nb, NAB = g.nab;
  R* const Tb = reinterpret_cast<R*>(smem_b + g.o_tab);
  double* const Hs = smem_b + g.o_h;      // (e0|c d) of the current chunk: [e][NVP]
  double* const Vs = smem_b + g.o_v;      // (ab|c d) of the current chunk: [ab][NVP]
  double* const R1 = smem_b + g.o_r1;     // sum_d V D_bd per (a, b, c)
  double* const R2 = smem_b + g.o_r2;     // sum_d V D_ad per (a, b, c)
  double* const JP = smem_b + g.o_jp;     // sum_b V D_ab per (a, c, d)
  double* const Dab = smem_b + g.o_d;
  double* const Dcd = Dab + NAB;
  double* const Dac = Dcd + NCD;
  double* const Dad = Dac + NA * NC;
  double* const Dbc = Dad + NA * ND;
  double* const Dbd = Dbc + NB * NC;
  double* const Jab = smem_b + g.o_jab;
  double* const Kxd = smem_b + g.o_kad;   // K'_ad, then K'_bd
  double* const CoB = smem_b + g.o_cob;   // per quartet: coefficient of bra term (b, t), or (BM) of
                                          // x^k in (x+M-A)^i (x+M-B)^j by direction, i, j and k
  double* const CoD = smem_b + g.o_cod;   // the same for the ket: term (d, t), or (KM) direction, i, j, k
  double* const Nab = smem_b + g.o_nab;   // normalization of (a, b)
  double* const Ncd = smem_b + g.o_ncd;
  int64_t* const list = reinterpret_cast<int64_t*>(smem_b + g.o_int);
  int* const be = reinterpret_cast<int*>(list + nt);  // [ab][term] index of a + k
  int* const bn = be + (BM ? (LAB + 1) * (LAB + 1) * (LAB + 1) : NAB * kMaxTerms);
  int* const bc = bn + NB;
  int* const bp = bc + NB * kMaxTerms;
  int* const dc = bp + NB * kMaxTerms;
  int* const dp = dc + ND * kMaxTerms;
  int* const dpos = dp + ND * kMaxTerms;  // row shell | column shell << 2 | row << 4 | column << 12
  int* const nlist = dpos + g.nacc;

  // ---- tables of the class, once per block ----
  if constexpr (BM)
    for (int i = tid; i < (LAB + 1) * (LAB + 1) * (LAB + 1); i += nt) {
      const int x = i / ((LAB + 1) * (LAB + 1)), yz = i - x * (LAB + 1) * (LAB + 1);
      const int y = yz / (LAB + 1), z = yz - y * (LAB + 1);
      be[i] = x + y + z <= LAB ? ncart_before(0, x + y + z) + cart_index(x, y, z) : 0;
    }
  for (int i = tid; i < NAB; i += nt) {
    const int a = i / NB, b = i - a * NB;
    Nab[i] = norm_factor(la, a) * norm_factor(lb, b);
    if constexpr (BM) continue;
    const int ca = cart_comp(la, a), cb = cart_comp(lb, b);
    const int bx = comp_x(cb), by = comp_y(cb), bz = comp_z(cb);
    int t = 0;
    for (int kx = 0; kx <= bx; ++kx)
      for (int ky = 0; ky <= by; ++ky)
        for (int kz = 0; kz <= bz; ++kz, ++t) {
          be[i * kMaxTerms + t] = ncart_before(la, la + kx + ky + kz) +
                                  cart_index(comp_x(ca) + kx, comp_y(ca) + ky, comp_z(ca) + kz);
          if (a == 0) {
            bc[b * kMaxTerms + t] = block_binom(bx, kx) * block_binom(by, ky) * block_binom(bz, kz);
            bp[b * kMaxTerms + t] = (bx - kx) | ((by - ky) << 4) | ((bz - kz) << 8);
          }
        }
    if (a == 0) bn[b] = t;
  }
  for (int i = tid; i < NCD; i += nt) {
    Ncd[i] = norm_factor(LC, i / ND) * norm_factor(LD, i % ND);
    if (!KM && i < ND) {
      const int cd = cart_comp(LD, i);
      const int dx = comp_x(cd), dy = comp_y(cd), dz = comp_z(cd);
      int t = 0;
      for (int kx = 0; kx <= dx; ++kx)
        for (int ky = 0; ky <= dy; ++ky)
          for (int kz = 0; kz <= dz; ++kz, ++t) {
            dc[i * kMaxTerms + t] = block_binom(dx, kx) * block_binom(dy, ky) * block_binom(dz, kz);
            dp[i * kMaxTerms + t] = (dx - kx) | ((dy - ky) << 4) | ((dz - kz) << 8);
          }
      for (; t < kMaxTerms; ++t) dc[i * kMaxTerms + t] = dp[i * kMaxTerms + t] = 0;
    }
  }
  for (int i = tid; i < g.nacc; i += nt) {
    int k = i, rs = 0, cs = 1, nc = NB;  // shells 0..3 = a, b, c, d
    auto next = [&](int n, int r, int c, int w) {
      if (k < n) return false;
      k -= n; rs = r; cs = c; nc = w;
      return true;
    };
    if (next(NAB, 2, 3, ND) && next(NCD, 0, 2, NC) && next(NA * NC, 0, 3, ND) && next(NA * ND, 1, 2, NC))
      next(NB * NC, 1, 3, ND);
    dpos[i] = rs | (cs << 2) | ((k / nc) << 4) | ((k % nc) << 12);
  }
  // this thread's rows of the tables
  int ox = 0, oy = g.ts, oz = 2 * g.ts;
  if (tid < NE) {
    int l = BM ? 0 : la, r = tid;
    while (r >= ncart(l)) r -= ncart(l++);
    const int ce = cart_comp(l, r);
    ox += comp_x(ce) * WS;
    oy += comp_y(ce) * WS;
    oz += comp_z(ce) * WS;
  }
  __syncthreads();

  // the quartets' block: `one`, or the entry of the list that holds the work item
  __shared__ MultiEntry entry;
  if (!list_of_blocks && tid == 0) {
    entry.blk = one;
    entry.work0 = 0;
    entry.nsplit = nsplit1;
    entry.csplit = csplit1;
  }
  __syncthreads();
  const QuartetBlock& blk = entry.blk;
  int cur = list_of_blocks ? -1 : 0;
  const int64_t nchunk = (nwork + g.chunk - 1) / g.chunk;
  unsigned int nprim_done = 0;

  for (int64_t ch = blockIdx.x; ch < nchunk; ch += gridDim.x) {
    const int64_t w0 = ch * g.chunk, w1 = min(nwork, w0 + g.chunk);
    int p = -1;
    for (int64_t wi = w0; wi < w1; ++wi) {
      if (list_of_blocks) {
        int e = cur < 0 ? 0 : cur;  // work items only move forward
        while (e + 1 < nblocks && __ldg(&list_of_blocks[e + 1].work0) <= wi) ++e;
        if (e != cur) {  // (all are past the last quartet: it ended with a sync)
          const int* src = reinterpret_cast<const int*>(list_of_blocks + e);
          for (int i = tid; i < (int)(sizeof(MultiEntry) / sizeof(int)); i += nt)
            reinterpret_cast<int*>(&entry)[i] = __ldg(src + i);
          cur = e;
          p = -1;
          __syncthreads();
        }
      }
      const int nbra = blk.bra.npairs, nket = blk.ket.npairs;
      const int Kcd = blk.ket.Ka * blk.ket.Kb;
      const int Kab = blk.bra.Ka * blk.bra.Kb;
      const int64_t P = (int64_t)Kab * Kcd;
      const int nsplit = entry.nsplit, csplit = entry.csplit, parts = nsplit * csplit;
      const int64_t wl = wi - entry.work0, tq = parts == 1 ? wl : wl / parts;
      const int part = (int)(wl - tq * parts), cpart = part / nsplit, split = part - cpart * nsplit;
      // this part's ket components [c_begin, c_end), whole chunks
      const int c_begin = cpart * (NC / CB) / csplit * CB, c_end = (cpart + 1) * (NC / CB) / csplit * CB;
      const int64_t t = blk.t_begin + tq;
      if (p < 0) p = find_bra_warp(blk.offsets, nbra, t);
      else while (t >= __ldg(blk.offsets + p + 1)) ++p;
      const int q = (blk.qbegin ? __ldg(blk.qbegin + p) : 0) + (int)(t - __ldg(blk.offsets + p));
      const int fa = __ldg(blk.bra.func_a + p), fb = __ldg(blk.bra.func_b + p);
      const int fc = __ldg(blk.ket.func_a + q), fd = __ldg(blk.ket.func_b + q);
      const double sym = quartet_weight(blk, p, q);
      const SysMats mats = sys_mats(args, blk, p);
      const size_t n = (size_t)mats.nbf;
      const double* __restrict__ pbra = blk.bra.primb + (size_t)p * Kab * kBraRec;
      const double* __restrict__ pket = blk.ket.primb + (size_t)q * Kcd * kBraRec;
      const bool one_centre = BM && __ldg(blk.bra.AB + p) == 0.0 && __ldg(blk.bra.AB + nbra + p) == 0.0 &&
                              __ldg(blk.bra.AB + 2 * nbra + p) == 0.0;
      {  // density blocks, transfer coefficients, zeroed sums
        const double* __restrict__ D = mats.D;
        auto first = [&](int sh) { return sh == 0 ? fa : sh == 1 ? fb : sh == 2 ? fc : fd; };
        for (int i = tid; i < g.nacc; i += nt) {
          const int k = dpos[i];
          copy_async8(Dab + i, D + (size_t)(first(k & 3) + ((k >> 4) & 255)) * n + first((k >> 2) & 3) + (k >> 12));
        }
        for (int i = tid; i < NAB; i += nt) Jab[i] = 0.0;
        for (int i = tid; i < (NA + NB) * ND; i += nt) Kxd[i] = 0.0;
        const double ABx = __ldg(blk.bra.AB + p), ABy = __ldg(blk.bra.AB + nbra + p),
                     ABz = __ldg(blk.bra.AB + 2 * nbra + p);
        if constexpr (BM) {
          const int per = (la + 1) * (lb + 1);
          for (int i = tid; i < 3 * per; i += nt) {
            const int x = i / per, ij = i - x * per, ia = ij / (lb + 1);
            const double pa = __ldg(pbra + BR_PAX + x);
            mid_coefs<kMaxLab + 1>(pa, pa + (x == 0 ? ABx : x == 1 ? ABy : ABz), ia, ij - ia * (lb + 1),
                                   CoB + i * (LAB + 1));
          }
        } else {
          for (int i = tid; i < NB * kMaxTerms; i += nt) {
            if (i % kMaxTerms >= bn[i / kMaxTerms]) continue;
            const int k = bp[i];
            CoB[i] = (double)bc[i] * block_pow(ABx, k & 15) * block_pow(ABy, (k >> 4) & 15) * block_pow(ABz, k >> 8);
          }
        }
        const double CDx = __ldg(blk.ket.AB + q), CDy = __ldg(blk.ket.AB + nket + q),
                     CDz = __ldg(blk.ket.AB + 2 * nket + q);
        if constexpr (KM) {
          constexpr int per = (LC + 1) * (LD + 1);
          for (int i = nt - 1 - tid; i < 3 * per; i += nt) {
            const int x = i / per, ij = i - x * per, ic = ij / (LD + 1);
            const double qc = __ldg(pket + BR_PAX + x);
            mid_coefs<W>(qc, qc + (x == 0 ? CDx : x == 1 ? CDy : CDz), ic, ij - ic * (LD + 1), CoD + i * W);
          }
        } else
        for (int i = tid; i < ND * kMaxTerms; i += nt) {
          const int k = dp[i];
          CoD[i] = (double)dc[i] * block_pow(CDx, k & 15) * block_pow(CDy, (k >> 4) & 15) * block_pow(CDz, k >> 8);
        }
      }
      R G[NF];
#pragma unroll
      for (int i = 0; i < NF; ++i) G[i] = R(0);

      // ---- primitive quartets: this block's candidates split + k * nsplit, those above
      // the cut collected in a list, the list processed `batch` at a time ----
      for (int64_t c0 = split; c0 < P; c0 += (int64_t)nt * nsplit) {
        int cnt;
        if (P == 1) {  // (the usual case of the d, f and g shells): no list
          cnt = __ldg(pbra + BR_Q) * __ldg(pket + BR_Q) < args.prim_eps ? 0 : 1;
        } else {
          if (tid == 0) *nlist = 0;
          __syncthreads();
          const int64_t ci = c0 + (int64_t)tid * nsplit;
          bool pass = false;
          if (ci < P) {
            const int64_t ib = ci / Kcd, ik = ci - ib * Kcd;
            pass = !(__ldg(pbra + ib * kBraRec + BR_Q) * __ldg(pket + ik * kBraRec + BR_Q) < args.prim_eps);
          }
          const unsigned m = __ballot_sync(0xffffffffu, pass);
          int at = 0;
          if (lane == 0 && m) at = atomicAdd(nlist, __popc(m));
          at = __shfl_sync(0xffffffffu, at, 0);
          if (pass) list[at + __popc(m & ((1u << lane) - 1))] = ci;
          __syncthreads();
          cnt = *nlist;
          if (cnt == 0) __syncthreads();  // all have read it before it is reset
        }
        if (cpart == 0) nprim_done += cnt;
        for (int base = 0; base < cnt; base += g.batch) {
          const int nb_ = min(g.batch, cnt - base);
          if (tid < nb_ * 3 * NR) {
            const int s = tid / (3 * NR), rx = tid - s * 3 * NR, r = rx / 3, x = rx - 3 * r;
            const int64_t ci = P == 1 ? 0 : list[base + s], ib = ci / Kcd;
            const double* pb = pbra + ib * kBraRec;
            const double* pk = pket + (ci - ib * Kcd) * kBraRec;
            const double zeta = __ldg(pb + BR_ZETA), eta = __ldg(pk + BR_ZETA);
            const double hz = __ldg(pb + BR_HZ), he = __ldg(pk + BR_HZ);
            const double PQx = __ldg(pb + BR_PX) - __ldg(pk + BR_PX), PQy = __ldg(pb + BR_PY) - __ldg(pk + BR_PY),
                         PQz = __ldg(pb + BR_PZ) - __ldg(pk + BR_PZ);
            const double rs = rsqrt(zeta + eta);
            const double inv = rs * rs, rz = eta * inv, re = zeta * inv;
            const double T = zeta * rz * (PQx * PQx + PQy * PQy + PQz * PQz);
            const double pref = __ldg(pb + BR_C) * __ldg(pk + BR_C) * rs;
            R u, w;
            rys_root_one<R>(NR, r, R(T), tab, u, w);
            const R pqx = R(x == 0 ? PQx : x == 1 ? PQy : PQz), rzr = R(rz), rer = R(re);
            // P - A and Q - C, or P - M and Q - M (0 in the first primitive)
            const double pc = BM ? __ldg(pb + BR_PX + x) - __ldg(pbra + BR_PX + x) : __ldg(pb + BR_PAX + x);
            const double qd = KM ? __ldg(pk + BR_PX + x) - __ldg(pket + BR_PX + x) : __ldg(pk + BR_PAX + x);
            const R pa = R(pc) - rzr * u * pqx, qc = R(qd) + rer * u * pqx;
            const R b00 = R(0.5) * R(inv) * u, b10 = R(hz) - R(hz) * rzr * u, b01 = R(he) - R(he) * rer * u;
            R* dst = Tb + (size_t)(s * NR * 3 + rx) * g.ts;
            R cur[kMaxLab + 1], prev[kMaxLab + 1];
            cur[0] = x == 2 ? w * R(pref) : R(1);
            dst[0] = cur[0];
#pragma unroll
            for (int e = 0; e < kMaxLab; ++e) {
              prev[e] = R(0);
              if (e < LAB) {
                cur[e + 1] = pa * cur[e] + (e ? R(e) * b10 * cur[e > 0 ? e - 1 : 0] : R(0));
                dst[(e + 1) * WS] = cur[e + 1];
              }
            }
            prev[kMaxLab] = R(0);
#pragma unroll
            for (int f = 0; f < LCD; ++f) {
              const R fb01 = R(f) * b01;
#pragma unroll
              for (int e = kMaxLab; e >= 0; --e)
                if (e <= LAB) {
                  R v = qc * cur[e];
                  if (f) v += fb01 * prev[e];
                  if (e) v += R(e) * b00 * cur[e > 0 ? e - 1 : 0];
                  prev[e] = v;
                  dst[e * WS + f + 1] = v;
                }
#pragma unroll
              for (int e = 0; e <= kMaxLab; ++e) {
                const R v = prev[e];
                prev[e] = cur[e];
                cur[e] = v;
              }
            }
          }
          __syncthreads();
          if (tid < NE) {
            const R* row = Tb;
            using V = typename std::conditional<sizeof(R) == 8, double2, float4>::type;
            constexpr int U = 16 / sizeof(R), NU = (F1 + U) / U;  // 16-byte loads that cover columns 0..F1
            for (int k = 0; k < nb_ * NR; ++k, row += 3 * g.ts) {
              R X[NU * U], Y[NU * U], Z[NU * U];
#pragma unroll
              for (int j = 0; j < NU; ++j) {
                reinterpret_cast<V*>(X)[j] = *reinterpret_cast<const V*>(row + ox + U * j);
                reinterpret_cast<V*>(Y)[j] = *reinterpret_cast<const V*>(row + oy + U * j);
                reinterpret_cast<V*>(Z)[j] = *reinterpret_cast<const V*>(row + oz + U * j);
              }
              bfor<0, F1 + 1>([&](auto FX) {
                constexpr int fx = decltype(FX)::value;
                bfor<0, F1 - fx + 1>([&](auto FY) {
                  constexpr int fy = decltype(FY)::value;
                  const R xy = X[fx] * Y[fy];
                  constexpr int z0 = F0 - fx - fy > 0 ? F0 - fx - fy : 0;
                  bfor<z0, F1 - fx - fy + 1>([&](auto FZ) {
                    constexpr int fz = decltype(FZ)::value;
                    constexpr int i = ncart_before(F0, fx + fy + fz) + cart_index(fx, fy, fz);
                    G[i] += xy * Z[fz];
                  });
                });
              });
            }
          }
          __syncthreads();
        }
      }

      // ---- transfer and digestion, a chunk of ket components at a time ----
      copy_async_wait();
      __syncthreads();
      const double s2 = 2.0 * sym;
      // J'_cd of the chunk at c0, from its (a, c, d) sums (by the block's last threads)
      auto flush_jcd = [&](int c0) {
        for (int i = nt - 1 - tid; i < NV; i += nt) {
          double s = 0.0;
          for (int a = 0; a < NA; ++a) s += JP[a * NV + i];
          atomicAdd(mats.J + (size_t)(fc + c0 + i / ND) * n + fd + i % ND, s2 * s);
        }
      };
      for (int c0 = c_begin; c0 < c_end; c0 += CB) {
        if (tid < NE) {
          bfor<0, NC / CB>([&](auto CH) {
            constexpr int c0_ = decltype(CH)::value * CB;
            if (c0 == c0_) {
              bfor<0, NV>([&](auto II) {
                constexpr int i = decltype(II)::value;
                constexpr int cc = cart_comp(LC, c0_ + i / ND), d = i % ND, cd = cart_comp(LD, d);
                double h = 0.0;
                if constexpr (KM) {
                  constexpr int per = (LC + 1) * (LD + 1) * W;
                  const double* cx = CoD + (comp_x(cc) * (LD + 1) + comp_x(cd)) * W;
                  const double* cy = CoD + per + (comp_y(cc) * (LD + 1) + comp_y(cd)) * W;
                  const double* cz = CoD + 2 * per + (comp_z(cc) * (LD + 1) + comp_z(cd)) * W;
                  bfor<0, comp_x(cc) + comp_x(cd) + 1>([&](auto KX) {
                    bfor<0, comp_y(cc) + comp_y(cd) + 1>([&](auto KY) {
                      constexpr int kx = decltype(KX)::value, ky = decltype(KY)::value;
                      constexpr int z0 = F0 - kx - ky > 0 ? F0 - kx - ky : 0;
                      constexpr int z1 = comp_z(cc) + comp_z(cd) < F1 - kx - ky ? comp_z(cc) + comp_z(cd) : F1 - kx - ky;
                      if constexpr (z0 <= z1) {
                        double hz = 0.0;
                        bfor<z0, z1 + 1>([&](auto KZ) {
                          constexpr int kz = decltype(KZ)::value;
                          hz += cz[kz] * G[ncart_before(F0, kx + ky + kz) + cart_index(kx, ky, kz)];
                        });
                        h += cx[kx] * cy[ky] * hz;
                      }
                    });
                  });
                } else
                bfor<0, comp_x(cd) + 1>([&](auto KX) {
                  bfor<0, comp_y(cd) + 1>([&](auto KY) {
                    bfor<0, comp_z(cd) + 1>([&](auto KZ) {
                      constexpr int kx = decltype(KX)::value, ky = decltype(KY)::value, kz = decltype(KZ)::value;
                      constexpr int lf = LC + kx + ky + kz;
                      if constexpr (lf >= F0 && lf <= F1) {
                        constexpr int f = ncart_before(F0, lf) +
                                          cart_index(comp_x(cc) + kx, comp_y(cc) + ky, comp_z(cc) + kz);
                        constexpr int t = (kx * (comp_y(cd) + 1) + ky) * (comp_z(cd) + 1) + kz;
                        h += CoD[d * kMaxTerms + t] * double(G[f]);
                      }
                    });
                  });
                });
                Hs[tid * NVP + i] = h;
              });
            }
          });
        }
        __syncthreads();
        if (c0 > c_begin) flush_jcd(c0 - CB);
        for (int i = tid; i < NAB; i += nt) {
          const int a = i / NB, b = i - a * NB;
          double v[NVP];
#pragma unroll
          for (int j = 0; j < NV; ++j) v[j] = 0.0;
          auto add = [&](double co, int e) {
            const double* h = Hs + e * NVP;
#pragma unroll
            for (int j = 0; j < (NV + 1) / 2; ++j) {
              const double2 hv = *reinterpret_cast<const double2*>(h + 2 * j);
              v[2 * j] += co * hv.x;
              if (2 * j + 1 < NV) v[2 * j + 1] += co * hv.y;
            }
          };
          if constexpr (BM) {
            const int ca = cart_comp(la, a), cb = cart_comp(lb, b), per = (la + 1) * (lb + 1) * (LAB + 1);
            const int ax = comp_x(ca), ay = comp_y(ca), az = comp_z(ca);
            const int bx = comp_x(cb), by = comp_y(cb), bz = comp_z(cb);
            const double* cx = CoB + (ax * (lb + 1) + bx) * (LAB + 1);
            const double* cy = CoB + per + (ay * (lb + 1) + by) * (LAB + 1);
            const double* cz = CoB + 2 * per + (az * (lb + 1) + bz) * (LAB + 1);
            // one loop over all powers, whose length is all that differs between the lanes (a
            // pair on one centre has the highest powers only)
            const int nx = ax + bx, ny = ay + by, nz = az + bz;
            int kx = one_centre ? nx : 0, ky = one_centre ? ny : 0, kz = one_centre ? nz : 0;
            const int terms = one_centre ? 1 : (nx + 1) * (ny + 1) * (nz + 1);
            for (int k = 0; k < terms; ++k) {
              add(cx[kx] * cy[ky] * cz[kz], be[(kx * (LAB + 1) + ky) * (LAB + 1) + kz]);
              if (++kz > nz) {
                kz = 0;
                if (++ky > ny) {
                  ky = 0;
                  ++kx;
                }
              }
            }
          } else {
            const int terms = bn[b];
            for (int k = 0; k < terms; ++k) add(CoB[b * kMaxTerms + k], be[i * kMaxTerms + k]);
          }
          double sj = 0.0;
          const double nab = Nab[i];
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            double s1 = 0.0, s3 = 0.0;
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const double x = v[c * ND + d] * (nab * Ncd[c0 * ND + c * ND + d]);
              Vs[i * NVP + c * ND + d] = x;
              sj += x * Dcd[c0 * ND + c * ND + d];
              s1 += x * Dbd[b * ND + d];
              s3 += x * Dad[a * ND + d];
            }
            R1[i * CB + c] = s1;
            R2[i * CB + c] = s3;
          }
          Jab[i] += sj;
        }
        __syncthreads();
        // K'_ad = sum_bc V D_bc and K'_bd = sum_ac V D_ac, one loop with the strides of
        // either, so that both share the warps' instructions
        for (int i = tid; i < (NA + NB) * ND; i += nt) {
          const bool ad = i < NA * ND;
          const int j = ad ? i : i - NA * ND;
          const int ab = j / ND, d = j - ab * ND;
          const double* v = Vs + (ad ? ab * NB * NVP : ab * NVP) + d;
          const double* dm = (ad ? Dbc : Dac) + c0;
          const int sv = ad ? NVP : NB * NVP, len = ad ? NB : NA;
          double k = 0.0;
          for (int m = 0; m < len; ++m, v += sv, dm += NC) {
#pragma unroll
            for (int c = 0; c < CB; ++c) k += v[c * ND] * dm[c];
          }
          Kxd[i] += k;
        }
        for (int i = tid; i < NA * NV; i += nt) {  // the J'_cd sums
          const int a = i / NV, cd = i - a * NV;
          const double* v = Vs + a * NB * NVP + cd;
          double j = 0.0;
          for (int b = 0; b < NB; ++b) j += v[b * NVP] * Dab[a * NB + b];
          JP[i] = j;
        }
        for (int i = nt - 1 - tid; i < (NA + NB) * CB; i += nt) {  // K'_ac, K'_bc
          const bool ac = i < NA * CB;
          const int j = ac ? i : i - NA * CB;
          const int ab = j / CB, c = j - ab * CB;
          const double* r = (ac ? R1 + ab * NB * CB : R2 + ab * CB) + c;
          const int sr = ac ? CB : NB * CB, len = ac ? NB : NA;
          double k = 0.0;
          for (int m = 0; m < len; ++m) k += r[m * sr];
          atomicAdd(mats.K + (size_t)((ac ? fa : fb) + ab) * n + fc + c0 + c, sym * k);
        }
        // (the next chunk's H overwrites Hs only; its V waits for the sync after that)
      }
      __syncthreads();
      flush_jcd(c_end - CB);
      for (int i = tid; i < NAB; i += nt) {
        const int k = dpos[i];
        atomicAdd(mats.J + (size_t)(fa + ((k >> 4) & 255)) * n + fb + (k >> 12), s2 * Jab[i]);
      }
      for (int i = tid; i < (NA + NB) * ND; i += nt) {
        const bool ad = i < NA * ND;
        const int j = ad ? i : i - NA * ND;
        atomicAdd(mats.K + (size_t)((ad ? fa : fb) + j / ND) * n + fd + j % ND, sym * Kxd[i]);
      }
      __syncthreads();  // before the next quartet's blocks overwrite these
    }
  }
  if (F0 == (KM ? 0 : LC)) count_prims(args.prim_count, tid == 0 ? nprim_done : 0u);
}

// Geometry of a bra and its resident blocks per SM; -3 on a CUDA error.
template <int LC, int LD, int F0, int F1, typename R, bool BM>
int block_geometry(int la, int lb, int64_t P, BlockGeom* g, int* threads, size_t* smem) {
  *threads = (ncart_range(BM ? 0 : la, la + lb) + 31) / 32 * 32;
  const int nroots = (la + lb + LC + LD) / 2 + 1;
  // table batch: one thread per (primitive quartet, root, direction); a block of 32 has
  // room for at least one primitive quartet of its class (27 >= 3 nroots)
  int batch = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(P, 8), *threads / (3 * nroots)));
  *g = make_geom<LC, LD, R, BM>(la, lb, *threads, batch);
  while (g->doubles * 8 > kMaxSmem && batch > 1) *g = make_geom<LC, LD, R, BM>(la, lb, *threads, --batch);
  *smem = sizeof(double) * (size_t)g->doubles;
  auto kern = eri_block_kernel<LC, LD, F0, F1, R, BM>;
  // resident blocks per SM, per bra and batch (0: not asked yet)
  static std::atomic<int> occ[kMaxL + 1][kMaxL + 1][9];
  int per_sm = occ[la][lb][batch].load(std::memory_order_relaxed);
  if (per_sm == 0) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, *threads, *smem) != cudaSuccess || per_sm < 1)
      return -3;
    occ[la][lb][batch].store(per_sm, std::memory_order_relaxed);
  }
  return per_sm;
}

// Blocks that share a quartet, where a launch has too few quartets (nq) for the `slots`
// blocks the device holds: first by primitive quartets (at least two table batches each),
// then by chunks of ket components.
inline void block_split(int64_t nq, int64_t P, int batch, int nchunks, int64_t slots, int* nsplit, int* csplit) {
  *nsplit = (int)std::max<int64_t>(1, std::min<int64_t>(P / (2 * batch), slots / nq));
  *csplit = (int)std::max<int64_t>(1, std::min<int64_t>(nchunks, slots / (nq * *nsplit)));
}

template <int LC, int LD, int F0, int F1, typename R, bool BM>
int launch_range_at(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab, cudaStream_t stream,
                    int num_sms) {
  const int64_t P = (int64_t)blk.bra.Ka * blk.bra.Kb * blk.ket.Ka * blk.ket.Kb;
  BlockGeom g;
  int threads;
  size_t smem;
  const int per_sm = block_geometry<LC, LD, F0, F1, R, BM>(blk.bra.la, blk.bra.lb, P, &g, &threads, &smem);
  if (per_sm < 0) return per_sm;
  const int64_t nq = blk.total - blk.t_begin, slots = (int64_t)num_sms * per_sm;
  int nsplit, csplit;
  block_split(nq, P, g.batch, ncart(LC) / chunk_components(LC, LD), slots, &nsplit, &csplit);
  const int64_t nwork = nq * nsplit * csplit;
  // consecutive quartets per block (one search for the bra pair, its data cached), at
  // least eight turns per block for balance
  g.chunk = (int)std::max<int64_t>(1, std::min<int64_t>(16, nwork / (slots * 8)));
  const int64_t want = (nwork + g.chunk - 1) / g.chunk;
  eri_block_kernel<LC, LD, F0, F1, R, BM><<<(unsigned)std::min<int64_t>(want, slots), threads, smem, stream>>>(
      blk, args, tab, g, nsplit, csplit, nullptr, 0, nwork);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

template <int LC, int LD, int F0, int F1, bool BM>
int launch_range_list_at(int la, int lb, int64_t Pmax, const MultiEntry* list, int n, int64_t nwork,
                         const JKArgs& args, const RysTablesView& tab, cudaStream_t stream, int num_sms) {
  BlockGeom g;
  int threads;
  size_t smem;
  const int per_sm = block_geometry<LC, LD, F0, F1, double, BM>(la, lb, Pmax, &g, &threads, &smem);
  if (per_sm < 0) return per_sm;
  const int64_t slots = (int64_t)num_sms * per_sm;
  g.chunk = (int)std::max<int64_t>(1, std::min<int64_t>(16, nwork / (slots * 8)));
  const int64_t want = (nwork + g.chunk - 1) / g.chunk;
  eri_block_kernel<LC, LD, F0, F1, double, BM><<<(unsigned)std::min<int64_t>(want, slots), threads, smem, stream>>>(
      QuartetBlock{}, args, tab, g, 1, 1, list, n, nwork);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// 0 when launched, -3 on a CUDA error.
template <int LC, int LD, int F0, int F1, typename R>
int launch_range(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab, cudaStream_t stream,
                 int num_sms) {
  if constexpr (mid_bra_possible<LC, LD, R>())
    if (mid_bra(blk.bra.la, blk.bra.lb, LD))
      return launch_range_at<LC, LD, F0, F1, R, true>(blk, args, tab, stream, num_sms);
  return launch_range_at<LC, LD, F0, F1, R, false>(blk, args, tab, stream, num_sms);
}

// The n blocks of a list (device memory; one bra (la, lb), Pmax the most primitive quartets
// of an entry) as one launch of nwork work items.
template <int LC, int LD, int F0, int F1>
int launch_range_list(int la, int lb, int64_t Pmax, const MultiEntry* list, int n, int64_t nwork, const JKArgs& args,
                      const RysTablesView& tab, cudaStream_t stream, int num_sms) {
  if constexpr (mid_bra_possible<LC, LD, double>())
    if (mid_bra(la, lb, LD))
      return launch_range_list_at<LC, LD, F0, F1, true>(la, lb, Pmax, list, n, nwork, args, tab, stream, num_sms);
  return launch_range_list_at<LC, LD, F0, F1, false>(la, lb, Pmax, list, n, nwork, args, tab, stream, num_sms);
}

}  // namespace block_detail
}  // namespace lai
