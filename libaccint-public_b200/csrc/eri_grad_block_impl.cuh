// Block-per-quartet nuclear gradient of E = 1/2 tr(D J[D]) - 1/4 tr(D K[D]) for the classes
// outside the thread-per-quartet set: compile-time specialised on the ket (lc, ld), any
// bra, the layout of the J/K kernel in eri_block_impl.cuh.
//
// The energy of a quartet is linear in its contracted integrals G[e][f] = (e0|f0), so the
// transfer is applied to the density instead of to derivative integrals: with
// Gamma_abcd = 4 D_ab D_cd - D_ac D_bd - D_ad D_bc,
//   E = sum_ef W[e][f] G[e][f],
//   W[e][f] = sum_{a+k=e, c+l=f} C(b,k) AB^(b-k) C(d,l) CD^(d-l) Gamma_abcd,
// formed once per quartet.  Then per primitive quartet and root the derivatives of the
// uncontracted (e0|f0) contract with W directly,
//   d/dA_x: 2 alpha (e+1x 0|f0) - e_x (e-1x 0|f0),   d/dC_x: the same on f with gamma,
//   d/dD_x: 2 delta ((e0|f+1x 0) + CD_x (e0|f0)),     d/dB = -(d/dA + d/dC + d/dD),
// and what is left is the dependence of W on AB and CD, which moves weight between A and B
// (C and D) only:  T_x = sum (dW[e][f]/dAB_x) G[e][f], once per quartet from G.
// One thread per row e holds W[e][.] and G[e][.] in registers; for one direction the sums
// over f collapse to P_x[f_x] = sum W Iy Iz first, so the three centres cost one pass.
// Against transferring the 2-D tables of the raised and lowered functions per primitive
// quartet and root, and combining nine products per integral, this leaves about three times
// the work of the J/K kernel.
//
// Where A (or C) lies far from the charge the terms of the transfer are large and cancel, and
// with both sides transferred once per quartet the factors multiply (eri_block_impl.cuh).
// So the bras that are there, (dd| against (dd| and larger kets (template parameter BM), and
// the kets (dd|, (fd|, (ff| and (gd| are expanded about M, the centre P of the pair's first
// primitive.  With u = x - M + (M-A),
//   d/dA_x: 2 alpha ((e+1x 0|f0) + (M-A)_x (e0|f0)) contracted with W, less the contraction
// of dW/d(M-A)_x with G; the same for C and D with their own exponents.  Error of the
// gradient of H2O/cc-pVQZ's f shells alone, four geometries: 3e-14 to 1e-13 of its norm about
// A and C, 1.4e-15 to 3.1e-15 about M (the kernel that transferred per primitive quartet:
// 2.6e-15 to 6.7e-15); d shells 5e-15 to 1e-14, 9e-16 to 2.2e-15 (1.4e-15 to 5.8e-15).
// (H2O)6/cc-pVDZ gradient 11.46 -> 11.45 ms.  The kets (gf| and (gg| stay about C: their
// unrolled derivatives would be 25000 and 50000 products, and with the bra about M the error
// with g shells is 1e-15 to 4.5e-15.
//
// A ket's f shells are split over launches (F0..F1) where W and G do not fit the
// registers; every term is linear in W.
#pragma once

#include "eri_block_impl.cuh"

namespace lai {
namespace grad_block {

using namespace block_detail;

template <int LC, int LD>
__host__ __device__ constexpr bool grad_mid_ket() { return LD >= 2 && LC + LD <= 6; }

struct GradBlockArgs {
  const double* D;
  int nbf;
  const int* shell_atom;
  double* grad;        // kGradCopies accumulators of grad_stride doubles each
  int grad_stride;
  double prim_eps;
};

struct GradBlockGeom {
  int la, lb, nroots, ne, nab, na, nb;
  int batch, nsplit, chunk;
  int ts;        // one direction's table: (la + lb + 2) * row stride
  int nacc, nentry;
  int o_tab, o_v, o_d, o_cob, o_cod, o_nab, o_ncd, o_exp, o_int;
  int doubles;
};

constexpr int transfer_terms(int l) {  // sum over the components of shell l of prod (b_x + 1)
  int n = 0;
  for (int x = 0; x <= l; ++x)
    for (int y = 0; x + y <= l; ++y) n += (x + 1) * (y + 1) * (l - x - y + 1);
  return n;
}

// the same about M: sum over a and b of prod (a_x + b_x + 1)
inline int mid_transfer_terms(int la, int lb) {
  int n = 0;
  for (int a = 0; a < ncart(la); ++a)
    for (int b = 0; b < ncart(lb); ++b) {
      const int ca = cart_comp(la, a), cb = cart_comp(lb, b);
      n += (comp_x(ca) + comp_x(cb) + 1) * (comp_y(ca) + comp_y(cb) + 1) * (comp_z(ca) + comp_z(cb) + 1);
    }
  return n;
}

template <int LC, int LD, bool BM>
__host__ GradBlockGeom make_grad_block_geom(int la, int lb, int threads, int batch) {
  constexpr int WS = odd_stride(LC + LD + 2), ND = ncart(LD), NC = ncart(LC);
  constexpr int NVP = odd_stride(chunk_components(LC, LD) * ND);
  GradBlockGeom g{};
  g.la = la; g.lb = lb;
  g.nroots = (la + lb + LC + LD + 1) / 2 + 1;
  g.ne = ncart_range(BM ? 0 : la, la + lb);
  g.na = ncart(la); g.nb = ncart(lb); g.nab = g.na * g.nb;
  g.nacc = g.nab + NC * ND + g.na * NC + g.na * ND + g.nb * NC + g.nb * ND;
  g.nentry = BM ? mid_transfer_terms(la, lb) : g.na * transfer_terms(lb);
  g.batch = batch;
  g.ts = (la + lb + 2) * WS;
  int o = 0;
  auto take = [&](int n) { const int at = o; o += (n + 1) & ~1; return at; };
  g.o_tab = take(batch * g.nroots * 3 * g.ts);
  g.o_v = take(g.nab * NVP);
  g.o_d = take(g.nacc);
  // coefficients, then their derivatives by AB_x (BM: by M-A in the same direction)
  g.o_cob = take(BM ? 6 * (la + 1) * (lb + 1) * (la + lb + 1) : 4 * g.nb * kMaxTerms);
  g.o_cod = take(grad_mid_ket<LC, LD>() ? 3 * (LC + 1) * (LD + 1) * (LC + LD + 1) : 4 * ND * kMaxTerms);
  g.o_nab = take(g.nab);
  g.o_ncd = take(NC * ND);
  g.o_exp = take(3 * batch);             // alpha, gamma, delta of every batched primitive quartet
  g.o_int = o;
  const int ints = 2 * threads + g.nentry + 2 * (g.ne + 1) + g.nb * 2 * kMaxTerms + ND * 2 * kMaxTerms + g.nacc + 8;
  o += (ints + 1) / 2;
  g.doubles = (o + 1) & ~1;
  return g;
}

template <int LC, int LD, int F0, int F1, bool BM>
__global__ void __launch_bounds__((BM ? kMaxThreadsMid : kMaxThreads))
    grad_block_kernel(QuartetBlock blk, GradBlockArgs ga, RysTablesView tab, GradBlockGeom g) {
  constexpr bool KM = grad_mid_ket<LC, LD>();
  constexpr int LCD = LC + LD, WS = odd_stride(LCD + 2);
  constexpr int NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
  constexpr int CB = chunk_components(LC, LD), NV = CB * ND, NVP = odd_stride(NV);
  constexpr int NF = ncart_range(F0, F1);
  extern __shared__ __align__(16) double smem_g[];
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
  const int la = g.la, lb = g.lb, LABp = la + lb + 1, NR = g.nroots;
  const int NE = g.ne, NA = g.na, NB = g.nb, NAB = g.nab;
  double* const Tb = smem_g + g.o_tab;
  double* const Vs = smem_g + g.o_v;   // Gamma of the current chunk: [ab][NVP]
  double* const Dab = smem_g + g.o_d;
  double* const Dcd = Dab + NAB;
  double* const Dac = Dcd + NCD;
  double* const Dad = Dac + NA * NC;
  double* const Dbc = Dad + NA * ND;
  double* const Dbd = Dbc + NB * NC;
  double* const CoB = smem_g + g.o_cob;
  double* const CoD = smem_g + g.o_cod;
  double* const Nab = smem_g + g.o_nab;
  double* const Ncd = smem_g + g.o_ncd;
  double* const Ex = smem_g + g.o_exp;
  int64_t* const list = reinterpret_cast<int64_t*>(smem_g + g.o_int);
  // by row e: ab | (b kMaxTerms + term) << 16, or (BM) ab | (a_x, b_x) << 8 | (a_y, b_y) << 13 | (a_z, b_z) << 18
  int* const entry = reinterpret_cast<int*>(list + nt);
  int* const first = entry + g.nentry;                   // [NE + 1] first entry of each row
  int* const fill = first + NE + 1;
  int* const bc = fill + NE + 1;
  int* const bp = bc + NB * kMaxTerms;
  int* const dc = bp + NB * kMaxTerms;
  int* const dp = dc + ND * kMaxTerms;
  int* const dpos = dp + ND * kMaxTerms;
  int* const nlist = dpos + g.nacc;
  const int sB = NB * kMaxTerms, sD = ND * kMaxTerms;

  // ---- tables of the class, once per block ----
  for (int i = tid; i < NE + 1; i += nt) first[i] = fill[i] = 0;
  for (int i = tid; i < NB * kMaxTerms; i += nt) bc[i] = bp[i] = 0;
  __syncthreads();
  auto each_term = [&](int i, auto&& f) {  // f(term, row e, coefficient, powers) of bra pair i
    const int a = i / NB, b = i - a * NB;
    const int ca = cart_comp(la, a), cb = cart_comp(lb, b);
    const int bx = comp_x(cb), by = comp_y(cb), bz = comp_z(cb);
    int t = 0;
    if constexpr (BM) {
      const int ax = comp_x(ca), ay = comp_y(ca), az = comp_z(ca);
      const int pairs = (ax * (lb + 1) + bx) | ((ay * (lb + 1) + by) << 5) | ((az * (lb + 1) + bz) << 10);
      for (int kx = 0; kx <= ax + bx; ++kx)
        for (int ky = 0; ky <= ay + by; ++ky)
          for (int kz = 0; kz <= az + bz; ++kz)
            f(0, ncart_before(0, kx + ky + kz) + cart_index(kx, ky, kz), 0, pairs);
      return;
    }
    for (int kx = 0; kx <= bx; ++kx)
      for (int ky = 0; ky <= by; ++ky)
        for (int kz = 0; kz <= bz; ++kz, ++t)
          f(t, ncart_before(la, la + kx + ky + kz) + cart_index(comp_x(ca) + kx, comp_y(ca) + ky, comp_z(ca) + kz),
            block_binom(bx, kx) * block_binom(by, ky) * block_binom(bz, kz),
            (bx - kx) | ((by - ky) << 4) | ((bz - kz) << 8));
  };
  for (int i = tid; i < NAB; i += nt) {
    each_term(i, [&](int t, int e, int c, int pw) {
      atomicAdd(first + e + 1, 1);
      if (!BM && i < NB) {
        bc[i * kMaxTerms + t] = c;
        bp[i * kMaxTerms + t] = pw;
      }
    });
    Nab[i] = norm_factor(la, i / NB) * norm_factor(lb, i % NB);
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
  __syncthreads();
  if (tid == 0)
    for (int e = 0; e < NE; ++e) first[e + 1] += first[e];
  __syncthreads();
  for (int i = tid; i < NAB; i += nt)
    each_term(i, [&](int t, int e, int, int pw) {
      entry[first[e] + atomicAdd(fill + e, 1)] = BM ? i | (pw << 8) : i | (((i % NB) * kMaxTerms + t) << 16);
    });
  // this thread's rows of the tables, and its component
  int ox = 0, oy = g.ts, oz = 2 * g.ts, ex = 0, ey = 0, ez = 0;
  if (tid < NE) {
    int l = BM ? 0 : la, r = tid;
    while (r >= ncart(l)) r -= ncart(l++);
    const int ce = cart_comp(l, r);
    ex = comp_x(ce); ey = comp_y(ce); ez = comp_z(ce);
    ox += ex * WS;
    oy += ey * WS;
    oz += ez * WS;
  }
  __syncthreads();
  const int e_first = tid < NE ? first[tid] : 0, e_last = tid < NE ? first[tid + 1] : 0;

  const int nbra = blk.bra.npairs, nket = blk.ket.npairs;
  const int Kab = blk.bra.Ka * blk.bra.Kb, Kcd = blk.ket.Ka * blk.ket.Kb;
  const int64_t P = (int64_t)Kab * Kcd;
  const int64_t nwork = (blk.total - blk.t_begin) * g.nsplit;
  const int64_t nchunk = (nwork + g.chunk - 1) / g.chunk;
  double* const grad = ga.grad + (size_t)(blockIdx.x % kGradCopies) * ga.grad_stride;
  const size_t n = (size_t)ga.nbf;

  for (int64_t ch = blockIdx.x; ch < nchunk; ch += gridDim.x) {
    const int64_t w0 = ch * g.chunk, w1 = min(nwork, w0 + g.chunk);
    int p = -1;
    for (int64_t wi = w0; wi < w1; ++wi) {
      const int64_t tq = g.nsplit == 1 ? wi : wi / g.nsplit;
      const int split = (int)(wi - tq * g.nsplit);
      const int64_t t = blk.t_begin + tq;
      if (p < 0) p = find_bra_warp(blk.offsets, nbra, t);
      else while (t >= __ldg(blk.offsets + p + 1)) ++p;
      const int q = (blk.qbegin ? __ldg(blk.qbegin + p) : 0) + (int)(t - __ldg(blk.offsets + p));
      const int fa = __ldg(blk.bra.func_a + p), fb = __ldg(blk.bra.func_b + p);
      const int fc = __ldg(blk.ket.func_a + q), fd = __ldg(blk.ket.func_b + q);
      const double sym = quartet_weight(blk, p, q);
      const double CD[3] = {__ldg(blk.ket.AB + q), __ldg(blk.ket.AB + nket + q), __ldg(blk.ket.AB + 2 * nket + q)};
      const double* __restrict__ pbra = blk.bra.primb + (size_t)p * Kab * kBraRec;
      const double* __restrict__ pket = blk.ket.primb + (size_t)q * Kcd * kBraRec;
      {  // density blocks; transfer coefficients C(b,k) AB^(b-k) and their derivatives
        const double* __restrict__ D = ga.D;
        auto func = [&](int sh) { return sh == 0 ? fa : sh == 1 ? fb : sh == 2 ? fc : fd; };
        for (int i = tid; i < g.nacc; i += nt) {
          const int k = dpos[i];
          copy_async8(Dab + i, D + (size_t)(func(k & 3) + ((k >> 4) & 255)) * n + func((k >> 2) & 3) + (k >> 12));
        }
        const double AB[3] = {__ldg(blk.bra.AB + p), __ldg(blk.bra.AB + nbra + p), __ldg(blk.bra.AB + 2 * nbra + p)};
        if constexpr (BM) {
          const int per = (la + 1) * (lb + 1), S = la + lb + 1;
          for (int i = tid; i < 3 * per; i += nt) {
            const int x = i / per, ij = i - x * per, ia = ij / (lb + 1), jb = ij - ia * (lb + 1);
            const double ma = __ldg(pbra + BR_PAX + x), mb = ma + (x == 0 ? AB[0] : x == 1 ? AB[1] : AB[2]);
            mid_coefs<kMaxLab + 1>(ma, mb, ia, jb, CoB + i * S);
            double* d = CoB + (3 * per + i) * S;  // ia times the coefficients of one power less
            if (ia) mid_coefs<kMaxLab + 1>(ma, mb, ia - 1, jb, d);
            for (int k = 0; k < ia + jb; ++k) d[k] = ia ? ia * d[k] : 0.0;
            d[ia + jb] = 0.0;
          }
        }
        if constexpr (KM) {
          constexpr int per = (LC + 1) * (LD + 1), S = LCD + 1;
          for (int i = nt - 1 - tid; i < 3 * per; i += nt) {
            const int x = i / per, ij = i - x * per, ic = ij / (LD + 1);
            const double mc = __ldg(pket + BR_PAX + x), md = mc + (x == 0 ? CD[0] : x == 1 ? CD[1] : CD[2]);
            mid_coefs<S>(mc, md, ic, ij - ic * (LD + 1), CoD + i * S);
          }
        }
        for (int i = tid + (BM ? sB : 0); i < (KM ? sB : sB + sD); i += nt) {
          const bool bra = i < sB;
          const int j = bra ? i : i - sB;
          const int k = bra ? bp[j] : dp[j], m[3] = {k & 15, (k >> 4) & 15, k >> 8};
          const double c = (double)(bra ? bc[j] : dc[j]);
          double v[3], dv[3];
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            const double r = bra ? AB[x] : CD[x];
            v[x] = block_pow(r, m[x]);
            dv[x] = m[x] ? m[x] * block_pow(r, m[x] - 1) : 0.0;
          }
          double* o = (bra ? CoB : CoD) + j;
          const int s = bra ? sB : sD;
          o[0] = c * v[0] * v[1] * v[2];
          o[s] = c * dv[0] * v[1] * v[2];
          o[2 * s] = c * v[0] * dv[1] * v[2];
          o[3 * s] = c * v[0] * v[1] * dv[2];
        }
      }
      copy_async_wait();
      __syncthreads();

      // Gamma of a chunk of ket components, normalized and weighted: Vs[ab][c d]
      auto gamma_chunk = [&](int c0) {
        for (int i = tid; i < NAB; i += nt) {
          const int a = i / NB, b = i - a * NB;
          const double w = sym * Nab[i], dab4 = 4.0 * Dab[i];
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            const double dac = Dac[a * NC + c0 + c], dbc = Dbc[b * NC + c0 + c];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              const int cd = (c0 + c) * ND + d;
              Vs[i * NVP + c * ND + d] =
                  w * Ncd[cd] * (dab4 * Dcd[cd] - dac * Dbd[b * ND + d] - Dad[a * ND + d] * dbc);
            }
          }
        }
      };
      // row e of the bra-transposed chunk: out[cd] = sum over the row's terms of
      // coefficient * Gamma[ab][cd]; dir = 0, 1, 2: the coefficients' derivative by AB_x
      // (BM: by (M-A)_x), 3: the coefficients
      auto gather_row = [&](int dir, double (&out)[NVP]) {
        const int S = la + lb + 1, per = (la + 1) * (lb + 1) * S;
        const double* cx = CoB + (dir == 0 ? 3 * per : 0) + ex;
        const double* cy = CoB + (dir == 1 ? 4 * per : per) + ey;
        const double* cz = CoB + (dir == 2 ? 5 * per : 2 * per) + ez;
        const double* co = CoB + (dir == 3 ? 0 : (dir + 1) * sB);
#pragma unroll
        for (int j = 0; j < NV; ++j) out[j] = 0.0;
        for (int k = e_first; k < e_last; ++k) {
          const int en = entry[k];
          double c;
          if constexpr (BM) c = cx[((en >> 8) & 31) * S] * cy[((en >> 13) & 31) * S] * cz[((en >> 18) & 31) * S];
          else c = co[en >> 16];
          const double* v = Vs + (en & (BM ? 0xff : 0xffff)) * NVP;
#pragma unroll
          for (int j = 0; j < (NV + 1) / 2; ++j) {
            const double2 x = *reinterpret_cast<const double2*>(v + 2 * j);
            out[2 * j] += c * x.x;
            if (2 * j + 1 < NV) out[2 * j + 1] += c * x.y;
          }
        }
      };

      // coefficients of (x-M + M-C)^i (x-M + M-D)^j in one direction (KM)
      auto ket_co = [&](int x, int i, int j) {
        return CoD + ((x * (LC + 1) + i) * (LD + 1) + j) * (LCD + 1);
      };

      // ---- W[e][f] ----
      double Wt[NF], G[NF];
#pragma unroll
      for (int i = 0; i < NF; ++i) Wt[i] = G[i] = 0.0;
      for (int c0 = 0; c0 < NC; c0 += CB) {
        gamma_chunk(c0);
        __syncthreads();
        if (tid < NE) {
          double row[NVP];
          gather_row(3, row);
          bfor<0, NC / CB>([&](auto CH) {
            constexpr int c0_ = decltype(CH)::value * CB;
            if (c0 == c0_) {
              bfor<0, NV>([&](auto II) {
                constexpr int i = decltype(II)::value;
                constexpr int cc = cart_comp(LC, c0_ + i / ND), d = i % ND, cd = cart_comp(LD, d);
                if constexpr (KM) {
                  bfor<0, comp_x(cc) + comp_x(cd) + 1>([&](auto KX) {
                    bfor<0, comp_y(cc) + comp_y(cd) + 1>([&](auto KY) {
                      constexpr int kx = decltype(KX)::value, ky = decltype(KY)::value;
                      constexpr int z0 = F0 - kx - ky > 0 ? F0 - kx - ky : 0;
                      constexpr int mz = comp_z(cc) + comp_z(cd), z1 = mz < F1 - kx - ky ? mz : F1 - kx - ky;
                      if constexpr (z0 <= z1) {
                        const double w = row[i] * (ket_co(0, comp_x(cc), comp_x(cd))[kx] *
                                                   ket_co(1, comp_y(cc), comp_y(cd))[ky]);
                        bfor<z0, z1 + 1>([&](auto KZ) {
                          constexpr int kz = decltype(KZ)::value;
                          Wt[ncart_before(F0, kx + ky + kz) + cart_index(kx, ky, kz)] +=
                              w * ket_co(2, comp_z(cc), comp_z(cd))[kz];
                        });
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
                        constexpr int tt = (kx * (comp_y(cd) + 1) + ky) * (comp_z(cd) + 1) + kz;
                        Wt[f] += CoD[d * kMaxTerms + tt] * row[i];
                      }
                    });
                  });
                });
              });
            }
          });
        }
        __syncthreads();
      }

      // ---- primitive quartets ----
      double gA[3] = {0.0, 0.0, 0.0}, gC[3] = {0.0, 0.0, 0.0}, gD[3] = {0.0, 0.0, 0.0};
      for (int64_t c0 = split; c0 < P; c0 += (int64_t)nt * g.nsplit) {
        int cnt;
        if (P == 1) {
          cnt = __ldg(pbra + BR_Q) * __ldg(pket + BR_Q) < ga.prim_eps ? 0 : 1;
        } else {
          if (tid == 0) *nlist = 0;
          __syncthreads();
          const int64_t ci = c0 + (int64_t)tid * g.nsplit;
          bool pass = false;
          if (ci < P) {
            const int64_t ib = ci / Kcd, ik = ci - ib * Kcd;
            pass = !(__ldg(pbra + ib * kBraRec + BR_Q) * __ldg(pket + ik * kBraRec + BR_Q) < ga.prim_eps);
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
            if (rx == 0) {
              const double gamma = __ldg(pk + BR_ALPHA);
              Ex[3 * s] = __ldg(pb + BR_ALPHA);
              Ex[3 * s + 1] = gamma;
              Ex[3 * s + 2] = eta - gamma;
            }
            double u, w;
            rys_root_one<double>(NR, r, T, tab, u, w);
            const double pqx = x == 0 ? PQx : x == 1 ? PQy : PQz;
            // P - A and Q - C, or P - M and Q - M (0 in the first primitive)
            const double pc = BM ? __ldg(pb + BR_PX + x) - __ldg(pbra + BR_PX + x) : __ldg(pb + BR_PAX + x);
            const double qd = KM ? __ldg(pk + BR_PX + x) - __ldg(pket + BR_PX + x) : __ldg(pk + BR_PAX + x);
            const double pa = pc - rz * u * pqx, qc = qd + re * u * pqx;
            const double b00 = 0.5 * inv * u, b10 = hz - hz * rz * u, b01 = he - he * re * u;
            double* dst = Tb + (size_t)(s * NR * 3 + rx) * g.ts;
            constexpr int E = kMaxLab + 1;
            double cur[E + 1], prev[E + 1];
            cur[0] = x == 2 ? w * pref : 1.0;
            dst[0] = cur[0];
#pragma unroll
            for (int e = 0; e < E; ++e) {
              prev[e] = 0.0;
              if (e < LABp) {
                cur[e + 1] = pa * cur[e] + (e ? e * b10 * cur[e > 0 ? e - 1 : 0] : 0.0);
                dst[(e + 1) * WS] = cur[e + 1];
              }
            }
            prev[E] = 0.0;
#pragma unroll
            for (int f = 0; f < F1 + 1; ++f) {
              const double fb01 = f * b01;
#pragma unroll
              for (int e = E; e >= 0; --e)
                if (e <= LABp) {
                  double v = qc * cur[e];
                  if (f) v += fb01 * prev[e];
                  if (e) v += e * b00 * cur[e > 0 ? e - 1 : 0];
                  prev[e] = v;
                  dst[e * WS + f + 1] = v;
                }
#pragma unroll
              for (int e = 0; e <= E; ++e) {
                const double v = prev[e];
                prev[e] = cur[e];
                cur[e] = v;
              }
            }
          }
          __syncthreads();
          if (tid < NE) {
            const double* row = Tb;
            for (int s = 0; s < nb_; ++s) {
              double up[3] = {0.0, 0.0, 0.0}, lo[3] = {0.0, 0.0, 0.0}, uc[3] = {0.0, 0.0, 0.0},
                     lc[3] = {0.0, 0.0, 0.0}, S = 0.0;
              for (int r = 0; r < NR; ++r, row += 3 * g.ts) {
                constexpr int NU = (F1 + 3) / 2;  // 16-byte loads that cover columns 0..F1+1
                double X[2 * NU], Y[2 * NU], Z[2 * NU];
#pragma unroll
                for (int j = 0; j < NU; ++j) {
                  reinterpret_cast<double2*>(X)[j] = *reinterpret_cast<const double2*>(row + ox + 2 * j);
                  reinterpret_cast<double2*>(Y)[j] = *reinterpret_cast<const double2*>(row + oy + 2 * j);
                  reinterpret_cast<double2*>(Z)[j] = *reinterpret_cast<const double2*>(row + oz + 2 * j);
                }
                double Px[F1 + 1], Py[F1 + 1], Pz[F1 + 1];
#pragma unroll
                for (int j = 0; j <= F1; ++j) Px[j] = Py[j] = Pz[j] = 0.0;
                bfor<0, F1 + 1>([&](auto FX) {
                  constexpr int fx = decltype(FX)::value;
                  bfor<0, F1 - fx + 1>([&](auto FY) {
                    constexpr int fy = decltype(FY)::value;
                    const double xy = X[fx] * Y[fy];
                    constexpr int z0 = F0 - fx - fy > 0 ? F0 - fx - fy : 0;
                    double wz = 0.0;  // sum over fz of W Iz
                    bfor<z0, F1 - fx - fy + 1>([&](auto FZ) {
                      constexpr int fz = decltype(FZ)::value;
                      constexpr int i = ncart_before(F0, fx + fy + fz) + cart_index(fx, fy, fz);
                      G[i] += xy * Z[fz];
                      Pz[fz] += Wt[i] * xy;
                      wz += Wt[i] * Z[fz];
                    });
                    Px[fx] += wz * Y[fy];
                    Py[fy] += wz * X[fx];
                  });
                });
                auto dir = [&](const double (&Pf)[F1 + 1], const double (&I)[2 * NU], int at, int e, double& u_,
                               double& l_, double& uc_, double& lc_) {
                  const double* hi = row + at + WS;
                  const double* lw = row + (e ? at - WS : at);
                  double a = 0.0, b = 0.0;
#pragma unroll
                  for (int j = 0; j <= F1; ++j) {
                    a += Pf[j] * hi[j];
                    if (!BM) b += Pf[j] * lw[j];
                    uc_ += Pf[j] * I[j + 1];
                    if (!KM && j) lc_ += Pf[j] * (j * I[j > 0 ? j - 1 : 0]);
                  }
                  u_ += a;
                  if (!BM) l_ += e * b;
                };
                dir(Px, X, ox, ex, up[0], lo[0], uc[0], lc[0]);
                dir(Py, Y, oy, ey, up[1], lo[1], uc[1], lc[1]);
                dir(Pz, Z, oz, ez, up[2], lo[2], uc[2], lc[2]);
#pragma unroll
                for (int j = 0; j <= F1; ++j) S += Px[j] * X[j];
              }
              const double al2 = 2.0 * Ex[3 * s], ga2 = 2.0 * Ex[3 * s + 1], de2 = 2.0 * Ex[3 * s + 2];
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                if constexpr (BM) gA[x] += al2 * (up[x] + __ldg(pbra + BR_PAX + x) * S);
                else gA[x] += al2 * up[x] - lo[x];
                if constexpr (KM) {
                  const double mc = __ldg(pket + BR_PAX + x);
                  gC[x] += ga2 * (uc[x] + mc * S);
                  gD[x] += de2 * (uc[x] + (mc + CD[x]) * S);
                } else {
                  gC[x] += ga2 * uc[x] - lc[x];
                  gD[x] += de2 * (uc[x] + CD[x] * S);
                }
              }
            }
          }
          __syncthreads();
        }
      }

      // ---- the dependence of W on AB and CD (about M: on M-A, M-C and M-D), from the
      // contracted G ----
      double tAB[3] = {0.0, 0.0, 0.0}, tCD[3] = {0.0, 0.0, 0.0}, tD[3] = {0.0, 0.0, 0.0};
      if (LD > 0 || lb > 0)
        for (int c0 = 0; c0 < NC; c0 += CB) {
          gamma_chunk(c0);
          __syncthreads();
          if (tid < NE) {
            double H[NV], row[NVP];
            gather_row(3, row);
            bfor<0, NC / CB>([&](auto CH) {
              constexpr int c0_ = decltype(CH)::value * CB;
              if (c0 == c0_) {
                bfor<0, NV>([&](auto II) {
                  constexpr int i = decltype(II)::value;
                  constexpr int cc = cart_comp(LC, c0_ + i / ND), d = i % ND, cd = cart_comp(LD, d);
                  double h = 0.0;
                  if constexpr (KM) {
                    constexpr int c_x = comp_x(cc), c_y = comp_y(cc), c_z = comp_z(cc);
                    constexpr int d_x = comp_x(cd), d_y = comp_y(cd), d_z = comp_z(cd);
                    double hc[3] = {0.0, 0.0, 0.0}, hd[3] = {0.0, 0.0, 0.0};
                    bfor<0, c_x + d_x + 1>([&](auto KX) {
                      bfor<0, c_y + d_y + 1>([&](auto KY) {
                        constexpr int kx = decltype(KX)::value, ky = decltype(KY)::value;
                        constexpr int z0 = F0 - kx - ky > 0 ? F0 - kx - ky : 0;
                        constexpr int mz = c_z + d_z, z1 = mz < F1 - kx - ky ? mz : F1 - kx - ky;
                        if constexpr (z0 <= z1) {
                          double sz = 0.0, sc = 0.0, sd = 0.0;  // over z: coefficients, derivatives by M-C and M-D
                          bfor<z0, z1 + 1>([&](auto KZ) {
                            constexpr int kz = decltype(KZ)::value;
                            const double gf = G[ncart_before(F0, kx + ky + kz) + cart_index(kx, ky, kz)];
                            sz += ket_co(2, c_z, d_z)[kz] * gf;
                            if constexpr (c_z > 0 && kz < mz) sc += ket_co(2, c_z - 1, d_z)[kz] * gf;
                            if constexpr (d_z > 0 && kz < mz) sd += ket_co(2, c_z, d_z - 1)[kz] * gf;
                          });
                          const double cx = ket_co(0, c_x, d_x)[kx], cy = ket_co(1, c_y, d_y)[ky];
                          h += cx * cy * sz;
                          hc[2] += cx * cy * sc;
                          hd[2] += cx * cy * sd;
                          if constexpr (c_x > 0 && kx < c_x + d_x) hc[0] += ket_co(0, c_x - 1, d_x)[kx] * (cy * sz);
                          if constexpr (d_x > 0 && kx < c_x + d_x) hd[0] += ket_co(0, c_x, d_x - 1)[kx] * (cy * sz);
                          if constexpr (c_y > 0 && ky < c_y + d_y) hc[1] += ket_co(1, c_y - 1, d_y)[ky] * (cx * sz);
                          if constexpr (d_y > 0 && ky < c_y + d_y) hd[1] += ket_co(1, c_y, d_y - 1)[ky] * (cx * sz);
                        }
                      });
                    });
                    if constexpr (c_x > 0) tCD[0] += row[i] * (c_x * hc[0]);
                    if constexpr (c_y > 0) tCD[1] += row[i] * (c_y * hc[1]);
                    if constexpr (c_z > 0) tCD[2] += row[i] * (c_z * hc[2]);
                    if constexpr (d_x > 0) tD[0] += row[i] * (d_x * hd[0]);
                    if constexpr (d_y > 0) tD[1] += row[i] * (d_y * hd[1]);
                    if constexpr (d_z > 0) tD[2] += row[i] * (d_z * hd[2]);
                  } else
                  bfor<0, comp_x(cd) + 1>([&](auto KX) {
                    bfor<0, comp_y(cd) + 1>([&](auto KY) {
                      bfor<0, comp_z(cd) + 1>([&](auto KZ) {
                        constexpr int kx = decltype(KX)::value, ky = decltype(KY)::value, kz = decltype(KZ)::value;
                        constexpr int lf = LC + kx + ky + kz;
                        if constexpr (lf >= F0 && lf <= F1) {
                          constexpr int f = ncart_before(F0, lf) +
                                            cart_index(comp_x(cc) + kx, comp_y(cc) + ky, comp_z(cc) + kz);
                          constexpr int tt = (kx * (comp_y(cd) + 1) + ky) * (comp_z(cd) + 1) + kz;
                          const double* co = CoD + d * kMaxTerms + tt;
                          h += co[0] * G[f];
                          const double rg = row[i] * G[f];
                          if constexpr (kx < comp_x(cd)) tCD[0] += co[sD] * rg;
                          if constexpr (ky < comp_y(cd)) tCD[1] += co[2 * sD] * rg;
                          if constexpr (kz < comp_z(cd)) tCD[2] += co[3 * sD] * rg;
                        }
                      });
                    });
                  });
                  H[i] = h;
                });
              }
            });
            if (lb > 0) {
#pragma unroll
              for (int x = 0; x < 3; ++x) {
                gather_row(x, row);
#pragma unroll
                for (int j = 0; j < NV; ++j) tAB[x] += row[j] * H[j];
              }
            }
          }
          __syncthreads();
        }

      // ---- sums over the block's rows (each warp adds its own) ----
      double v[9];
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        v[x] = BM ? gA[x] - tAB[x] : gA[x] + tAB[x];
        v[3 + x] = KM ? gC[x] - tCD[x] : gC[x] + tCD[x];
        v[6 + x] = KM ? gD[x] - tD[x] : gD[x] - tCD[x];
      }
#pragma unroll
      for (int i = 0; i < 9; ++i)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
      if (lane == 0) {
        const int atA = __ldg(ga.shell_atom + __ldg(blk.bra.shell_a + p));
        const int atB = __ldg(ga.shell_atom + __ldg(blk.bra.shell_b + p));
        const int atC = __ldg(ga.shell_atom + __ldg(blk.ket.shell_a + q));
        const int atD = __ldg(ga.shell_atom + __ldg(blk.ket.shell_b + q));
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          atomicAdd(grad + 3 * atA + x, v[x]);
          atomicAdd(grad + 3 * atB + x, -(v[x] + v[3 + x] + v[6 + x]));
          atomicAdd(grad + 3 * atC + x, v[3 + x]);
          atomicAdd(grad + 3 * atD + x, v[6 + x]);
        }
      }
      __syncthreads();  // before the next quartet's blocks overwrite these
    }
  }
}

template <int LC, int LD, int F0, int F1, bool BM>
int launch_grad_range_at(const QuartetBlock& blk, const GradBlockArgs& ga, const RysTablesView& tab, cudaStream_t stream,
                      int num_sms) {
  const int la = blk.bra.la, lb = blk.bra.lb;
  const int threads = (ncart_range(BM ? 0 : la, la + lb) + 31) / 32 * 32;
  const int nroots = (la + lb + LC + LD + 1) / 2 + 1;
  const int64_t P = (int64_t)blk.bra.Ka * blk.bra.Kb * blk.ket.Ka * blk.ket.Kb;
  int batch = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(P, 8), threads / (3 * nroots)));
  GradBlockGeom g = make_grad_block_geom<LC, LD, BM>(la, lb, threads, batch);
  while (g.doubles * 8 > kMaxSmem && batch > 1) g = make_grad_block_geom<LC, LD, BM>(la, lb, threads, --batch);
  const size_t smem = sizeof(double) * (size_t)g.doubles;
  auto kern = grad_block_kernel<LC, LD, F0, F1, BM>;
  static std::atomic<int> occ[kMaxL + 1][kMaxL + 1][9];
  int per_sm = occ[la][lb][batch].load(std::memory_order_relaxed);
  if (per_sm == 0) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess || per_sm < 1)
      return -3;
    occ[la][lb][batch].store(per_sm, std::memory_order_relaxed);
  }
  // the split of few quartets and the turns per block of the J/K kernel (launch_range)
  const int64_t nq = blk.total - blk.t_begin, slots = (int64_t)num_sms * per_sm;
  g.nsplit = (int)std::max<int64_t>(1, std::min<int64_t>(P / (2 * batch), slots / nq));
  const int64_t nwork = nq * g.nsplit;
  g.chunk = (int)std::max<int64_t>(1, std::min<int64_t>(16, nwork / (slots * 8)));
  const int64_t want = (nwork + g.chunk - 1) / g.chunk;
  kern<<<(unsigned)std::min<int64_t>(want, slots), threads, smem, stream>>>(blk, ga, tab, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// 0 when launched, -3 on a CUDA error.
template <int LC, int LD, int F0, int F1>
int launch_grad_range(const QuartetBlock& blk, const GradBlockArgs& ga, const RysTablesView& tab, cudaStream_t stream,
                      int num_sms) {
  if constexpr (mid_bra_possible<LC, LD, double>())
    if (mid_bra(blk.bra.la, blk.bra.lb, LD) || (LD == 2 && blk.bra.lb == 2))
      return launch_grad_range_at<LC, LD, F0, F1, true>(blk, ga, tab, stream, num_sms);
  return launch_grad_range_at<LC, LD, F0, F1, false>(blk, ga, tab, stream, num_sms);
}

}  // namespace grad_block
}  // namespace lai
