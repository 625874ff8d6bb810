// Device side of an engine's set-up: the pair tables of every class are formed by one
// kernel from the shells, the Schwarz bounds of the shell pairs and of their primitive
// pairs come from the diagonal launches, and the sorted tables are written by the same
// kernel again.  The host orders and screens the pairs (it needs their bounds anyway for
// the quartet ranges) and copies a few packed arrays.
//
// Forming the tables on the host took most of a small engine's set-up, through one
// allocation and one synchronous copy for each of the twelve arrays of each class, in
// three rounds: (H2O)6/cc-pVDZ needed 1100 allocations, copies and frees.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <numeric>
#include <utility>

#include "engine_internal.h"
#include "fp32_tables.h"
#include "rys_tables.inc"

static_assert(RYS_DEG == lai::kRysDeg, "table degree mismatch");
static_assert(BOYS_NM == lai::kBoysNM, "Boys table width mismatch");
static_assert(BOYS_NGRID == lai::kBoysNGrid, "Boys grid mismatch");

namespace lai {
namespace host {

namespace {

struct DevShell {
  double x[3];
  int K, prim0, func, pad;
};

// One class of a build_tables launch.  Elements (primitive t of pair p) are numbered
// t * npairs + p within the class, so that consecutive threads write consecutive
// addresses of the SoA tables.
struct ClassTables {
  int Kb, Kab, npairs;
  int parentK;              // > 0: every pair is one primitive pair of a parent class
  int64_t elem0;            // first element of the class in the launch
  int64_t pair0;            // its pairs in the launch's pair list (the parent's, if any)
  int64_t src0;             // first primitive bound of the class in qprim (order != nullptr)
  int64_t ord0;             // first entry of the class in order
  PairClassDev out;         // tables to write (FP32 copies only where not null)
  unsigned long long* qmax; // largest primitive bound of the class, as its bit pattern
};

// Pairs [pair0, pair0 + n) of the pair list, of one class, in the bounds of one stage: shell
// pairs (0) or their primitive pairs, prim0 the first (1).
struct Piece {
  int stage, n;
  int64_t pair0, prim0;
  ClassTables tab;
};
constexpr size_t kBoundBytes = size_t(256) << 20;

__device__ __forceinline__ int find_class(const ClassTables* __restrict__ cls, int ncls, int64_t e) {
  int lo = 0, hi = ncls;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (cls[mid].elem0 <= e) lo = mid; else hi = mid;
  }
  return lo;
}

__global__ void build_tables_kernel(const ClassTables* __restrict__ cls, int ncls, int64_t total,
                                    const int2* __restrict__ pairs, const int* __restrict__ src,
                                    const int* __restrict__ order, const double* __restrict__ qprim,
                                    const DevShell* __restrict__ shells, const double* __restrict__ exps,
                                    const double* __restrict__ coefs) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  const ClassTables& c = cls[find_class(cls, ncls, e)];
  const int64_t l = e - c.elem0;
  const int n = c.npairs, t = (int)(l / n), p = (int)(l - (int64_t)t * n);
  int pp = p, ti = t;  // pair in the pair list, primitive pair of the two shells
  if (c.parentK > 0) {
    pp = p / c.parentK;
    ti = p - pp * c.parentK;
  } else if (order) {
    ti = order[c.ord0 + (int64_t)p * c.Kab + t];
  }
  const int2 ab = pairs[c.pair0 + pp];
  const DevShell A = shells[ab.x], B = shells[ab.y];
  const int Kb = c.parentK > 0 ? B.K : c.Kb;
  const int ia = ti / Kb, ib = ti - ia * Kb;
  const double al = exps[A.prim0 + ia], be = exps[B.prim0 + ib], z = al + be;
  double f[PF_COUNT], ab2 = 0.0, d[3];
  for (int x = 0; x < 3; ++x) {
    d[x] = A.x[x] - B.x[x];
    ab2 += d[x] * d[x];
    f[PF_PX + x] = (al * A.x[x] + be * B.x[x]) / z;
    f[PF_PAX + x] = f[PF_PX + x] - A.x[x];
  }
  f[PF_ZETA] = z;
  f[PF_HZ] = 0.5 / z;
  f[PF_ALPHA] = al;
  const double pi54s2 = 5.9149671727956128778;  // sqrt(2) pi^(5/4)
  f[PF_C] = pi54s2 * coefs[A.prim0 + ia] * coefs[B.prim0 + ib] * exp(-al * be / z * ab2) / z;
  f[PF_Q] = order ? qprim[c.src0 + (int64_t)src[c.pair0 + p] * c.Kab + ti] : 0.0;
  const PairClassDev& o = c.out;
  const size_t sf = (size_t)c.Kab * n, at = (size_t)t * n + p;
  double* prim = const_cast<double*>(o.prim);
  for (int k = 0; k < PF_COUNT; ++k) prim[k * sf + at] = f[k];
  double* rb = const_cast<double*>(o.primb) + ((size_t)p * c.Kab + t) * kBraRec;
  const double rec[kBraRec] = {f[PF_Q],  f[PF_ZETA], f[PF_HZ], f[PF_C], f[PF_PX], f[PF_PY],
                               f[PF_PZ], f[PF_ALPHA], f[PF_PAX], f[PF_PAY], f[PF_PAZ], 0.0};
  for (int k = 0; k < kBraRec; ++k) rb[k] = rec[k];
  const double ket[kKetRec] = {f[PF_Q],   f[PF_ZETA], f[PF_HZ],  f[PF_PX], f[PF_PY], f[PF_PZ],
                               f[PF_PAX], f[PF_PAY],  f[PF_PAZ], f[PF_C],  f[PF_ALPHA]};
  const size_t kt = ((size_t)(p / kKetTile) * c.Kab + t) * kKetRec * kKetTile + p % kKetTile;
  for (int k = 0; k < kKetRec; ++k) const_cast<double*>(o.primk)[kt + k * kKetTile] = ket[k];
  if (o.primf) {
    for (int k = 0; k < PF_COUNT; ++k) const_cast<float*>(o.primf)[k * sf + at] = (float)f[k];
    float* rbf = const_cast<float*>(o.primbf) + ((size_t)p * c.Kab + t) * kBraRec;
    for (int k = 0; k < kBraRec; ++k) rbf[k] = (float)rec[k];
    for (int k = 0; k < kKetRec; ++k) const_cast<float*>(o.primkf)[kt + k * kKetTile] = (float)ket[k];
  }
  if (t == 0) {
    for (int x = 0; x < 3; ++x) {
      const_cast<double*>(o.AB)[(size_t)x * n + p] = d[x];
      const_cast<double*>(o.Acen)[(size_t)x * n + p] = A.x[x];
    }
    const_cast<int*>(o.shell_a)[p] = ab.x;
    const_cast<int*>(o.shell_b)[p] = ab.y;
    const_cast<int*>(o.func_a)[p] = A.func;
    const_cast<int*>(o.func_b)[p] = B.func;
    // non-negative doubles order like their bit patterns
    if (order) atomicMax(c.qmax, (unsigned long long)__double_as_longlong(f[PF_Q]));
  }
}

// order[ord0 + p Kab + r] = the primitive pair of rank r (descending bound; equal bounds
// in their original order) of pair p.
__global__ void rank_kernel(const ClassTables* __restrict__ cls, int ncls, int64_t total,
                            const int* __restrict__ src, const double* __restrict__ qprim, int* __restrict__ order) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  const ClassTables& c = cls[find_class(cls, ncls, e)];
  const int64_t l = e - c.elem0;
  const int p = (int)(l / c.Kab), t = (int)(l - (int64_t)p * c.Kab);
  const double* q = qprim + c.src0 + (int64_t)src[c.pair0 + p] * c.Kab;
  const double mine = q[t];
  int r = 0;
  for (int k = 0; k < c.Kab; ++k) r += q[k] > mine || (q[k] == mine && k < t);
  order[c.ord0 + (int64_t)p * c.Kab + r] = t;
}

__global__ void iota_kernel(int64_t* __restrict__ a, int* __restrict__ b, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (int)i;
  if (i <= n) a[i] = i;
}

unsigned blocks_for(int64_t n) { return (unsigned)((n + 255) / 256); }

// Room for a class's tables in an arena layout (two passes: sizes, then pointers).
struct Layout {
  char* base = nullptr;
  size_t at = 0;
  template <typename T>
  T* take(size_t n) {
    T* p = base ? reinterpret_cast<T*>(base + at) : nullptr;
    at += (n * sizeof(T) + 255) & ~size_t(255);
    return p;
  }
};

void lay_out_class(Layout& L, PairClassDev& v, bool fp32) {
  const size_t n = v.npairs, K = (size_t)v.Ka * v.Kb;
  const size_t ket = (n + kKetTile - 1) / kKetTile * K * kKetRec * kKetTile;
  v.shell_a = L.take<int>(n);
  v.shell_b = L.take<int>(n);
  v.func_a = L.take<int>(n);
  v.func_b = L.take<int>(n);
  v.AB = L.take<double>(3 * n);
  v.Acen = L.take<double>(3 * n);
  v.prim = L.take<double>(PF_COUNT * K * n);
  v.primb = L.take<double>(K * n * kBraRec);
  v.primk = L.take<double>(ket);
  v.primf = fp32 ? L.take<float>(PF_COUNT * K * n) : nullptr;
  v.primbf = fp32 ? L.take<float>(K * n * kBraRec) : nullptr;
  v.primkf = fp32 ? L.take<float>(ket) : nullptr;
}

// Pads of the last ket tile of a class are read (never used): keep them defined.
int clear_ket_pads(const PairClassDev& v, cudaStream_t s) {
  const size_t n = v.npairs, K = (size_t)v.Ka * v.Kb;
  if (n == 0 || n % kKetTile == 0) return LAI_OK;
  const size_t tile = K * kKetRec * kKetTile, first = n / kKetTile * tile;
  LAI_CUDA_TRY(cudaMemsetAsync(const_cast<double*>(v.primk) + first, 0, tile * sizeof(double), s));
  if (v.primkf) LAI_CUDA_TRY(cudaMemsetAsync(const_cast<float*>(v.primkf) + first, 0, tile * sizeof(float), s));
  return LAI_OK;
}

// The lookup tables (Rys fits, Hermite limits, Boys grids) are the same for every engine:
// one copy in device memory (0.8 MB) for the life of the process, like module constants.
int shared_tables(lai::RysTablesView* out) {
  static std::mutex m;
  static bool ready = false;
  static lai::RysTablesView view;
  std::lock_guard<std::mutex> lock(m);
  if (!ready) {
    std::vector<float> bf((size_t)lai::kBoysF32Rows * lai::kBoysF32Stride), rf(2 * (size_t)lai::kRysF32Len);
    lai::build_boys_f32(BOYS_GRID_H, bf.data());
    lai::build_rys_f32(RYS_COEF_H, rf.data());
    Layout L;
    for (int pass = 0; pass < 2; ++pass) {
      L.at = 0;
      view.coef = L.take<double>(RYS_COEF_LEN);
      view.herm_x2 = L.take<double>(RYS_HERM_LEN);
      view.herm_w = L.take<double>(RYS_HERM_LEN);
      view.boys = L.take<double>(BOYS_NGRID * BOYS_NM);
      view.boys_f32 = L.take<float>(bf.size());
      view.rys_f32 = L.take<float>(rf.size());
      if (pass == 0) {
        void* p = nullptr;
        LAI_CUDA_TRY(cudaMalloc(&p, L.at));
        L.base = static_cast<char*>(p);
      }
    }
    auto put = [](const void* dst, const void* s, size_t n) {
      return cudaMemcpy(const_cast<void*>(dst), s, n, cudaMemcpyHostToDevice);
    };
    cudaError_t e = put(view.coef, RYS_COEF_H, sizeof(double) * RYS_COEF_LEN);
    if (e == cudaSuccess) e = put(view.herm_x2, RYS_HERM_X2_H, sizeof(double) * RYS_HERM_LEN);
    if (e == cudaSuccess) e = put(view.herm_w, RYS_HERM_W_H, sizeof(double) * RYS_HERM_LEN);
    if (e == cudaSuccess) e = put(view.boys, BOYS_GRID_H, sizeof(double) * BOYS_NGRID * BOYS_NM);
    if (e == cudaSuccess) e = put(view.boys_f32, bf.data(), sizeof(float) * bf.size());
    if (e == cudaSuccess) e = put(view.rys_f32, rf.data(), sizeof(float) * rf.size());
    if (e != cudaSuccess) {
      cudaFree(L.base);
      return fail(LAI_ECUDA, std::string("lookup tables: ") + cudaGetErrorString(e));
    }
    ready = true;
  }
  *out = view;
  return LAI_OK;
}

}  // namespace

int setup_tables(lai_engine* E) { return shared_tables(&E->tab); }

int setup_pairs(lai_engine* E) {
  const auto& sh = E->basis->shells;
  const int ns = (int)sh.size();
  const int nc = (int)E->classes.size();
  const bool batched = E->nsys > 1;
  cudaStream_t s = E->stream;
  if (!batched) E->Q_all.assign((size_t)ns * ns, 0.0);  // (a full matrix only for one system)
  if (nc == 0) return LAI_OK;

  // ---- shells and pair lists ----
  std::vector<DevShell> hs(ns);
  std::vector<double> hexp, hcoef;
  for (int i = 0; i < ns; ++i) {
    hs[i] = DevShell{{sh[i].center[0], sh[i].center[1], sh[i].center[2]},
                     (int)sh[i].exps.size(), (int)hexp.size(), (int)sh[i].func, 0};
    hexp.insert(hexp.end(), sh[i].exps.begin(), sh[i].exps.end());
    hcoef.insert(hcoef.end(), sh[i].coefs.begin(), sh[i].coefs.end());
  }
  int64_t npairs = 0, nelem = 0;
  std::vector<int2> hp;
  std::vector<ClassTables> raw(nc);
  for (int c = 0; c < nc; ++c) {
    const auto& cl = *E->classes[c];
    const int Kab = cl.Ka * cl.Kb, n = cl.n();
    for (int p = 0; p < n; ++p) hp.push_back(int2{cl.sa[p], cl.sb[p]});
    ClassTables a{};
    a.Kb = cl.Kb; a.Kab = Kab; a.npairs = n;
    a.elem0 = nelem; a.pair0 = npairs; a.src0 = nelem;
    a.out.la = cl.la; a.out.lb = cl.lb; a.out.Ka = cl.Ka; a.out.Kb = cl.Kb; a.out.npairs = n;
    raw[c] = a;
    npairs += n;
    nelem += (int64_t)n * Kab;
  }
  // temporary buffers of the set-up
  DevBuf d_in, d_tmp, d_bounds, d_meta;
  DevShell* ds; double *de, *dcf; int2* dp; int64_t* iota64; int* iota32;
  {
    Layout L;
    for (int pass = 0; pass < 2; ++pass) {
      L.at = 0;
      ds = L.take<DevShell>(ns);
      de = L.take<double>(hexp.size());
      dcf = L.take<double>(hcoef.size());
      dp = L.take<int2>(npairs);
      if (pass == 0) {
        LAI_CUDA_TRY(d_in.alloc(L.at));
        L.base = d_in.as<char>();
      }
    }
    // one packed copy
    std::vector<char> pack(L.at);
    auto put = [&](const void* dst, const void* from, size_t n) {
      std::memcpy(pack.data() + (static_cast<const char*>(dst) - d_in.as<char>()), from, n);
    };
    put(ds, hs.data(), hs.size() * sizeof(DevShell));
    put(de, hexp.data(), hexp.size() * sizeof(double));
    put(dcf, hcoef.data(), hcoef.size() * sizeof(double));
    put(dp, hp.data(), hp.size() * sizeof(int2));
    LAI_CUDA_TRY(cudaMemcpyAsync(d_in.p, pack.data(), pack.size(), cudaMemcpyHostToDevice, s));
    LAI_CUDA_TRY(cudaStreamSynchronize(s));
  }
  // ---- bounds: of the shell pairs (ab|ab), and of every primitive pair run as a
  // one-primitive pair (by the Schwarz inequality a primitive quartet contributes at most
  // q_ab q_cd to any integral of its quartet).  Their unsorted tables, 340 bytes for each
  // primitive pair of the basis, most of them far below the cut in a large one, are formed
  // in pieces: ranges of a class's pairs, as many at a time as fit kBoundBytes. ----
  std::vector<Piece> pieces;
  for (int stage = 0; stage < 2; ++stage)
    for (int c = nc - 1; c >= 0; --c) {
      ClassTables a = raw[c];
      if (stage == 1) {
        a.parentK = a.Kab;
        a.Kb = a.Kab = 1;
        a.out.Ka = a.out.Kb = 1;
      }
      const int n = raw[c].npairs, per = stage == 0 ? 1 : raw[c].Kab;
      const size_t pair = (size_t)raw[c].Kab * (PF_COUNT + kBraRec + kKetRec) * sizeof(double) +
                          per * (6 * sizeof(double) + 4 * sizeof(int));
      const int most = (int)std::max<size_t>(kKetTile, std::min<size_t>(INT_MAX / per, kBoundBytes / 2 / pair));
      for (int p = 0; p < n; p += most) {
        const int np = std::min(most, n - p);
        Piece pc{stage, np, raw[c].pair0 + p, raw[c].elem0 + (int64_t)p * raw[c].Kab, a};
        pc.tab.pair0 = pc.pair0;
        pc.tab.npairs = pc.tab.out.npairs = np * per;
        pieces.push_back(pc);
      }
    }
  // batches [first, last) of pieces of one stage
  std::vector<std::pair<size_t, size_t>> batches;
  size_t need = 0, batch_pieces = 0;
  int64_t maxn = 0;
  for (size_t i = 0; i < pieces.size();) {
    Layout L;
    size_t j = i;
    while (j < pieces.size() && pieces[j].stage == pieces[i].stage) {
      Layout next = L;
      PairClassDev v = pieces[j].tab.out;
      lay_out_class(next, v, false);
      if (j > i && next.at > kBoundBytes) break;
      L = next;
      maxn = std::max<int64_t>(maxn, pieces[j].tab.npairs);
      ++j;
    }
    need = std::max(need, L.at);
    batch_pieces = std::max(batch_pieces, j - i);
    batches.emplace_back(i, j);
    i = j;
  }
  double *d_q, *d_qprim;
  {
    Layout L;
    for (int pass = 0; pass < 2; ++pass) {
      L.at = 0;
      d_q = L.take<double>(npairs);
      d_qprim = L.take<double>(nelem);
      iota64 = L.take<int64_t>(maxn + 1);
      iota32 = L.take<int>(maxn);
      if (pass == 0) {
        LAI_CUDA_TRY(d_bounds.alloc(L.at));
        L.base = d_bounds.as<char>();
      }
    }
  }
  iota_kernel<<<blocks_for(maxn + 1), 256, 0, s>>>(iota64, iota32, maxn);
  LAI_CUDA_TRY(d_tmp.alloc(need));
  LAI_CUDA_TRY(d_meta.alloc(sizeof(ClassTables) * batch_pieces));
  for (const auto& [first, last] : batches) {
    Layout L;
    L.base = d_tmp.as<char>();
    std::vector<ClassTables> meta;
    int64_t elems = 0;
    for (size_t i = first; i < last; ++i) {
      ClassTables& t = pieces[i].tab;
      lay_out_class(L, t.out, false);
      if (int rc = clear_ket_pads(t.out, s)) return rc;
      t.elem0 = elems;
      elems += (int64_t)t.Kab * t.npairs;
      meta.push_back(t);
    }
    LAI_CUDA_TRY(cudaMemcpyAsync(d_meta.p, meta.data(), sizeof(ClassTables) * meta.size(), cudaMemcpyHostToDevice, s));
    build_tables_kernel<<<blocks_for(elems), 256, 0, s>>>(d_meta.as<ClassTables>(), (int)meta.size(), elems, dp,
                                                          nullptr, nullptr, nullptr, ds, de, dcf);
    LAI_CUDA_TRY(cudaGetLastError());
    LaunchLanes lanes(E, s, kLanes);
    for (size_t i = first; i < last; ++i) {
      const Piece& pc = pieces[i];
      const auto& o = pc.tab.out;
      lai::QuartetBlock blk{};
      blk.bra = blk.ket = o;
      blk.offsets = iota64;
      blk.qbegin = iota32;
      blk.total = o.npairs;
      blk.same_class = 1;
      lai::JKArgs args{};
      args.mode = lai::MODE_SCHWARZ;
      args.schwarz_out = pc.stage == 0 ? d_q + pc.pair0 : d_qprim + pc.prim0;
      cudaError_t ce = lanes.pick(alg_work(o.la, o.lb, o.la, o.lb, o.Ka, o.Kb, o.Ka, o.Kb) * o.npairs, &E->stream);
      const int rc = ce == cudaSuccess ? launch_block(E, blk, args) : fail(LAI_ECUDA, cudaGetErrorString(ce));
      E->stream = s;
      if (rc) return rc;
    }
    LAI_CUDA_TRY(lanes.join());
  }
  std::vector<double> Q(npairs);
  LAI_CUDA_TRY(cudaMemcpyAsync(Q.data(), d_q, sizeof(double) * npairs, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaStreamSynchronize(s));
  LAI_CUDA_TRY(d_tmp.alloc(0));  // given back before the engine's own tables are taken

  // ---- screening and order (host) ----
  double qmax = 0.0;
  for (int c = 0; c < nc; ++c) {
    const auto& cl = *E->classes[c];
    for (int p = 0; p < cl.n(); ++p) {
      const double q = Q[raw[c].pair0 + p];
      qmax = std::max(qmax, q);
      if (!batched) E->Q_all[(size_t)cl.sa[p] * ns + cl.sb[p]] = E->Q_all[(size_t)cl.sb[p] * ns + cl.sa[p]] = q;
    }
  }
  std::vector<int2> kp;
  std::vector<int> ksrc, ksys;
  std::vector<double> kq;
  std::vector<ClassTables> fin(nc);
  int64_t kelem = 0;
  for (int c = 0; c < nc; ++c) {
    auto& cl = *E->classes[c];
    const int n = cl.n();
    const double* q = Q.data() + raw[c].pair0;
    // pairs ordered by system, then by Schwarz bound (descending); pairs that pass
    // with no partner dropped -- each system's kept pairs are a prefix of its segment
    std::vector<int> idx;
    idx.reserve(n);
    for (int i = 0; i < n; ++i)
      if (q[i] * qmax >= E->thr) idx.push_back(i);
    std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) {
      return cl.sys[x] != cl.sys[y] ? cl.sys[x] < cl.sys[y] : q[x] > q[y];
    });
    const int keep = (int)idx.size();
    ClassTables a = raw[c];
    a.npairs = a.out.npairs = keep;
    a.pair0 = (int64_t)kp.size();
    a.elem0 = a.ord0 = kelem;
    kelem += (int64_t)keep * a.Kab;
    auto perm = [&](std::vector<int>& v) {
      std::vector<int> o(keep);
      for (int i = 0; i < keep; ++i) o[i] = v[idx[i]];
      v = std::move(o);
    };
    perm(cl.sa); perm(cl.sb); perm(cl.fa); perm(cl.fb); perm(cl.sys);
    cl.Q.resize(keep);
    for (int i = 0; i < keep; ++i) {
      cl.Q[i] = q[idx[i]];
      kp.push_back(int2{cl.sa[i], cl.sb[i]});
      ksrc.push_back(idx[i]);
      ksys.push_back(cl.sys[i]);
      kq.push_back(cl.Q[i]);
    }
    cl.seg.assign(E->nsys + 1, 0);
    for (int i = 0, t = 0; t <= E->nsys; ++t) {
      while (i < keep && cl.sys[i] < t) ++i;
      cl.seg[t] = i;
    }
    cl.batched = batched;
    fin[c] = a;
  }

  // ---- quartet ranges of every class pair: the kets of a bra pair that pass are a prefix
  // of its system's segment, which shrinks along the segment's bra pairs ----
  int64_t noff = 0, nqb = 0;
  for (int A = 0; A < nc; ++A)
    for (int B = 0; B <= A; ++B) {
      const auto& ca = *E->classes[A];
      const auto& cb = *E->classes[B];
      if (ca.n() == 0 || cb.n() == 0) continue;
      auto blk = std::make_unique<ClassPairBlock>();
      blk->bra = A;
      blk->ket = B;
      blk->offsets.resize(ca.n() + 1);
      blk->offsets[0] = 0;
      if (batched) blk->qbegin.resize(ca.n());
      int last = -1, hi = 0;
      for (int p = 0; p < ca.n(); ++p) {
        const int s0 = cb.seg[ca.sys[p]];
        if (ca.sys[p] != last) {
          last = ca.sys[p];
          hi = cb.seg[last + 1];
        }
        while (hi > s0 && !(ca.Q[p] * cb.Q[hi - 1] >= E->thr)) --hi;
        int cnt = hi - s0;
        if (A == B) cnt = std::min(cnt, p - s0 + 1);  // canonical q <= p (same segment)
        blk->offsets[p + 1] = blk->offsets[p] + cnt;
        if (batched) blk->qbegin[p] = s0;
      }
      blk->total = blk->offsets[ca.n()];
      if (blk->total == 0) continue;
      blk->alg_flops = alg_work(ca.la, ca.lb, cb.la, cb.lb, ca.Ka, ca.Kb, cb.Ka, cb.Kb);
      blk->flops_per_prim = alg_per_prim(ca.la, ca.lb, cb.la, cb.lb);
      blk->flops_per_quartet = alg_per_quartet(ca.la, ca.lb, cb.la, cb.lb);
      noff += (int64_t)blk->offsets.size();
      nqb += (int64_t)blk->qbegin.size();
      E->blocks.push_back(std::move(blk));
    }

  // ---- final tables: one allocation for what the host copies, one for what the device
  // forms ----
  int2* kpd; int *ksd, *kyd, *qbd; double* kqd; int64_t* offd; ClassTables* fmeta; unsigned long long* qm;
  size_t packed = 0;
  {
    Layout L;
    for (int pass = 0; pass < 2; ++pass) {
      L.at = 0;
      kqd = L.take<double>(kq.size());
      offd = L.take<int64_t>(noff);
      qbd = L.take<int>(nqb);
      kyd = L.take<int>(batched ? ksys.size() : 0);
      kpd = L.take<int2>(kp.size());
      ksd = L.take<int>(ksrc.size());
      fmeta = L.take<ClassTables>(nc);
      qm = L.take<unsigned long long>(nc);
      packed = L.at;
      for (auto& c : fin) lay_out_class(L, c.out, true);
      if (pass == 0) {
        LAI_CUDA_TRY(E->d_pairs.alloc(L.at));
        L.base = E->d_pairs.as<char>();
      }
    }
  }
  std::vector<char> pack(packed, 0);
  auto put = [&](const void* dst, const void* from, size_t n) {
    if (n) std::memcpy(pack.data() + (static_cast<const char*>(dst) - E->d_pairs.as<char>()), from, n);
  };
  put(kqd, kq.data(), kq.size() * sizeof(double));
  put(kpd, kp.data(), kp.size() * sizeof(int2));
  put(ksd, ksrc.data(), ksrc.size() * sizeof(int));
  if (batched) put(kyd, ksys.data(), ksys.size() * sizeof(int));
  int64_t o1 = 0, o2 = 0;
  for (auto& b : E->blocks) {
    put(offd + o1, b->offsets.data(), b->offsets.size() * sizeof(int64_t));
    put(qbd + o2, b->qbegin.data(), b->qbegin.size() * sizeof(int));
    b->dev_offsets = offd + o1;
    b->dev_qbegin = b->qbegin.empty() ? nullptr : qbd + o2;
    o1 += (int64_t)b->offsets.size();
    o2 += (int64_t)b->qbegin.size();
  }
  for (int c = 0; c < nc; ++c) {
    fin[c].qmax = qm + c;
    fin[c].out.Q = kqd + fin[c].pair0;
    fin[c].out.sys = batched ? kyd + fin[c].pair0 : nullptr;
    if (int rc = clear_ket_pads(fin[c].out, s)) return rc;
  }
  put(fmeta, fin.data(), sizeof(ClassTables) * nc);
  LAI_CUDA_TRY(cudaMemcpyAsync(E->d_pairs.p, pack.data(), packed, cudaMemcpyHostToDevice, s));
  DevBuf d_order;
  LAI_CUDA_TRY(d_order.alloc(sizeof(int) * std::max<int64_t>(kelem, 1)));
  if (kelem > 0) {
    rank_kernel<<<blocks_for(kelem), 256, 0, s>>>(fmeta, nc, kelem, ksd, d_qprim, d_order.as<int>());
    build_tables_kernel<<<blocks_for(kelem), 256, 0, s>>>(fmeta, nc, kelem, kpd, ksd, d_order.as<int>(), d_qprim, ds,
                                                          de, dcf);
    LAI_CUDA_TRY(cudaGetLastError());
  }
  std::vector<unsigned long long> bits(nc);
  LAI_CUDA_TRY(cudaMemcpyAsync(bits.data(), qm, sizeof(unsigned long long) * nc, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaStreamSynchronize(s));
  for (int c = 0; c < nc; ++c) {
    auto& cl = *E->classes[c];
    std::memcpy(&cl.qprim_max, &bits[c], sizeof(double));
    cl.dev = fin[c].out;
    cl.dev.qprim_max = cl.qprim_max;
    cl.on_device = true;
  }
  return LAI_OK;
}

}  // namespace host
}  // namespace lai
