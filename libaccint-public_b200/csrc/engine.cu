// Host orchestration of the J/K engine and the C ABI (include/libaccint_b200.h).
//
// Pipeline of one engine (built once per basis, reused for every density):
//   1. lai_basis_create: normalize contraction coefficients like the reference
//      Shell constructor (src/shared/basis/shell.cpp:32-113); drop primitives whose
//      normalized coefficient is exactly zero (general-contraction padding kept by
//      the reference's BSE reader, src/shared/data/bse_json_parser.cpp:43-57 --
//      their contribution is exactly zero).
//   2. Shell pairs (i >= j) oriented so la >= lb, grouped into pair classes
//      (la, lb, Ka, Kb); primitive-pair data (zeta, P, P-A, prefactor) in SoA.
//   3. Schwarz bounds from the diagonal quartets (ab|ab) on the device
//      (src/shared/screening/schwarz_bounds.cpp:20-59 computes the same on the host).
//   4. Pairs sorted by Q (descending) within their class; pairs with
//      Q * Q_max < threshold dropped; for every ordered class pair (bra >= ket) the
//      number of passing kets of each bra pair is a prefix length (binary search),
//      prefix-summed into the launch's flat quartet range.
//   5. lai_jk_build: one launch per class pair (thread-per-quartet kernels for the
//      small classes, block-per-quartet otherwise), then J = J' + J'^T, K = K' + K'^T.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/libaccint_b200.h"
#include "engine_internal.h"
#include "eri_kernels.h"

namespace lai {
void spherical_forget_basis(const lai_basis* basis);  // spherical.cu
}  // namespace lai

using namespace lai::host;

namespace lai {
namespace host {

thread_local std::string g_last_error;

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

double dfact_odd(int l) {
  double r = 1;
  for (int k = 2 * l - 1; k > 1; k -= 2) r *= k;
  return r;
}

}  // namespace host
}  // namespace lai

// ---------------------------------------------------------------------------
// Basis
// ---------------------------------------------------------------------------

extern "C" {

const char* lai_last_error(void) { return g_last_error.c_str(); }
int lai_abi_version(void) { return LAI_ABI_VERSION; }

int lai_basis_create(int nshell, const int* l, const int* nprim, const double* centers,
                     const double* exps, const double* coefs, const int* atom_index, int flags,
                     lai_basis** out) {
  if (!out) return fail(LAI_EINVAL, "lai_basis_create: out is NULL");
  *out = nullptr;
  if (nshell < 0 || (nshell > 0 && (!l || !nprim || !centers || !exps || !coefs)))
    return fail(LAI_EINVAL, "lai_basis_create: null array");
  auto b = std::make_unique<lai_basis>();
  long off = 0;
  for (int s = 0; s < nshell; ++s) {
    if (l[s] < 0 || l[s] > lai::kMaxL)
      return fail(LAI_EINVAL, "lai_basis_create: shell " + std::to_string(s) +
                                  " angular momentum outside [0, 4]");
    if (nprim[s] < 1) return fail(LAI_EINVAL, "lai_basis_create: shell with no primitive");
    HostShell sh;
    sh.l = l[s];
    for (int x = 0; x < 3; ++x) sh.center[x] = centers[3 * s + x];
    sh.atom = atom_index ? atom_index[s] : -1;
    sh.exps_all.assign(exps + off, exps + off + nprim[s]);
    sh.coefs_all.assign(coefs + off, coefs + off + nprim[s]);
    off += nprim[s];
    for (double e : sh.exps_all)
      if (!(e > 0.0)) return fail(LAI_EINVAL, "lai_basis_create: non-positive exponent");
    if (!(flags & LAI_BASIS_PRENORMALIZED)) {
      // Reference Shell normalization (shell.cpp:32-113): primitive factor
      // (2a/pi)^{3/4} (4a)^{l/2} / sqrt((2l-1)!!), then unit (l,0,0) self-overlap.
      const int L = sh.l;
      const int n = (int)sh.exps_all.size();
      for (int p = 0; p < n; ++p) {
        const double a = sh.exps_all[p];
        sh.coefs_all[p] *= std::pow(2.0 * a / M_PI, 0.75) * std::pow(4.0 * a, 0.5 * L) /
                           std::sqrt(dfact_odd(L));
      }
      double ov = 0.0;
      for (int p = 0; p < n; ++p)
        for (int q = 0; q < n; ++q) {
          const double z = sh.exps_all[p] + sh.exps_all[q];
          double o = std::pow(M_PI / z, 1.5);
          for (int k = 0; k < L; ++k) o *= 0.5 / z;
          ov += sh.coefs_all[p] * sh.coefs_all[q] * o;
        }
      if (!(ov > 0.0)) return fail(LAI_EINVAL, "lai_basis_create: zero contraction");
      const double sc = 1.0 / std::sqrt(ov);
      for (auto& c : sh.coefs_all) c *= sc;
    }
    for (size_t p = 0; p < sh.exps_all.size(); ++p)
      if (sh.coefs_all[p] != 0.0) {
        sh.exps.push_back(sh.exps_all[p]);
        sh.coefs.push_back(sh.coefs_all[p]);
      }
    if (sh.exps.empty()) return fail(LAI_EINVAL, "lai_basis_create: all coefficients zero");
    sh.func = b->nbf;
    b->nbf += lai::ncart(sh.l);
    b->shells.push_back(std::move(sh));
  }
  *out = b.release();
  return LAI_OK;
}

void lai_basis_destroy(lai_basis* basis) {
  if (!basis) return;
  lai::spherical_forget_basis(basis);
  delete basis;
}
long lai_basis_nbf(const lai_basis* basis) { return basis ? basis->nbf : 0; }
int lai_basis_nshell(const lai_basis* basis) { return basis ? (int)basis->shells.size() : 0; }

int lai_basis_shell(const lai_basis* basis, int s, int* l, int* nprim, double* center,
                    double* exps, double* coefs, long* func_index) {
  if (!basis || s < 0 || s >= (int)basis->shells.size())
    return fail(LAI_EINVAL, "lai_basis_shell: bad shell index");
  const HostShell& sh = basis->shells[s];
  if (l) *l = sh.l;
  if (nprim) *nprim = (int)sh.exps_all.size();
  if (center) for (int x = 0; x < 3; ++x) center[x] = sh.center[x];
  if (exps) std::copy(sh.exps_all.begin(), sh.exps_all.end(), exps);
  if (coefs) std::copy(sh.coefs_all.begin(), sh.coefs_all.end(), coefs);
  if (func_index) *func_index = sh.func;
  return LAI_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Engine
// ---------------------------------------------------------------------------
namespace lai {
namespace host {


// Algorithmic FP work of one canonical quartet (one unit), the single accounting
// used for roofline fractions:  P (40 + 64 n + n (20 + T2D + 4 Ncart)) + 25 Ncart
// with P the product of nonzero primitive counts, n the root count and
// T2D = 3 [5 (La+Lb+1)(Lc+Ld+1) + 2 Lb (La+Lb+1)(Lc+Ld+1)(Ld+1) + 2 Ld (La+1)(Lb+1)(Lc+Ld+1)].
double alg_per_prim(int la, int lb, int lc, int ld) {
  const int n = (la + lb + lc + ld) / 2 + 1;
  const double nc = (double)lai::ncart(la) * lai::ncart(lb) * lai::ncart(lc) * lai::ncart(ld);
  const double t2d = 3.0 * (5.0 * (la + lb + 1) * (lc + ld + 1) +
                            2.0 * lb * (la + lb + 1) * (lc + ld + 1) * (ld + 1) +
                            2.0 * ld * (la + 1) * (lb + 1) * (lc + ld + 1));
  return 40.0 + 64.0 * n + n * (20.0 + t2d + 4.0 * nc);
}
double alg_per_quartet(int la, int lb, int lc, int ld) {
  return 25.0 * lai::ncart(la) * lai::ncart(lb) * lai::ncart(lc) * lai::ncart(ld);
}
double alg_work(int la, int lb, int lc, int ld, int Ka, int Kb, int Kc, int Kd) {
  const double P = (double)Ka * Kb * Kc * Kd;
  return P * alg_per_prim(la, lb, lc, ld) + alg_per_quartet(la, lb, lc, ld);
}

// J = J' + J'^T, K = K' + K'^T, J' and K' the sums of `copies` accumulators of n^2 elements.
__global__ void symmetrize_kernel(const double* __restrict__ Jp, const double* __restrict__ Kp,
                                  double* __restrict__ J, double* __restrict__ K, int n, int copies) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nn = (int64_t)n * n;
  if (idx >= nn) return;
  const int i = (int)(idx / n), j = (int)(idx - (int64_t)i * n);
  const int64_t tr = (int64_t)j * n + i;
  double sj = 0.0, sk = 0.0;
#pragma unroll 4
  for (int c = 0; c < copies; ++c, Jp += nn, Kp += nn) {
    sj += Jp[idx] + Jp[tr];
    sk += Kp[idx] + Kp[tr];
  }
  J[idx] = sj;
  K[idx] = sk;
}

}  // namespace host
}  // namespace lai


namespace lai {
namespace host {

int build_classes(lai_engine* E) {
  const auto& sh = E->basis->shells;
  const int ns = (int)sh.size();
  // class key -> index
  std::vector<std::array<int, 4>> keys;
  std::map<std::array<int, 4>, int> index;
  auto class_of = [&](int la, int lb, int Ka, int Kb) {
    std::array<int, 4> k{la, lb, Ka, Kb};
    const auto it = index.emplace(k, (int)keys.size());
    if (!it.second) return it.first->second;
    keys.push_back(k);
    E->classes.push_back(std::make_unique<PairClassHost>());
    auto& c = *E->classes.back();
    c.la = la; c.lb = lb; c.Ka = Ka; c.Kb = Kb;
    return (int)keys.size() - 1;
  };
  // pairs within one system only (shells of a system are contiguous)
  int sys_first = 0;
  for (int i = 0; i < ns; ++i) {
    if (i > 0 && sh[i].sys != sh[i - 1].sys) sys_first = i;
    for (int j = sys_first; j <= i; ++j) {
      int a = i, b = j;
      const int Ki = (int)sh[i].exps.size(), Kj = (int)sh[j].exps.size();
      // orient: higher l first, then more primitives first
      if (sh[j].l > sh[i].l || (sh[j].l == sh[i].l && Kj > Ki)) std::swap(a, b);
      const HostShell& A = sh[a];
      const HostShell& B = sh[b];
      const int ci = class_of(A.l, B.l, (int)A.exps.size(), (int)B.exps.size());
      auto& c = *E->classes[ci];
      c.sa.push_back(a); c.sb.push_back(b);
      c.fa.push_back((int)A.func); c.fb.push_back((int)B.func);
      c.sys.push_back(A.sys);
    }
  }
  // sort classes by key so that bra >= ket implies (la,lb) >= (lc,ld)
  std::vector<int> order(keys.size());
  std::iota(order.begin(), order.end(), 0);
  std::sort(order.begin(), order.end(), [&](int x, int y) { return keys[x] < keys[y]; });
  std::vector<std::unique_ptr<PairClassHost>> sorted;
  for (int o : order) sorted.push_back(std::move(E->classes[o]));
  E->classes = std::move(sorted);
  return LAI_OK;
}

void fill_pair_data(const lai_basis* basis, PairClassHost& c) {
  const auto& sh = basis->shells;
  const int n = c.n();
  const int Kab = c.Ka * c.Kb;
  c.AB.assign(3 * (size_t)n, 0.0);
  c.Acen.assign(3 * (size_t)n, 0.0);
  c.prim.assign((size_t)lai::PF_COUNT * Kab * n, 0.0);
  const double pi54s2 = std::sqrt(2.0) * std::pow(M_PI, 1.25);
  for (int p = 0; p < n; ++p) {
    const HostShell& A = sh[c.sa[p]];
    const HostShell& B = sh[c.sb[p]];
    double AB[3], ab2 = 0;
    for (int x = 0; x < 3; ++x) {
      AB[x] = A.center[x] - B.center[x];
      ab2 += AB[x] * AB[x];
      c.AB[(size_t)x * n + p] = AB[x];
      c.Acen[(size_t)x * n + p] = A.center[x];
    }
    for (int ia = 0; ia < c.Ka; ++ia)
      for (int ib = 0; ib < c.Kb; ++ib) {
        const int t = ia * c.Kb + ib;
        const double al = A.exps[ia], be = B.exps[ib];
        const double z = al + be;
        auto at = [&](int f) -> double& { return c.prim[((size_t)f * Kab + t) * n + p]; };
        at(lai::PF_ZETA) = z;
        at(lai::PF_ALPHA) = al;
        at(lai::PF_HZ) = 0.5 / z;
        for (int x = 0; x < 3; ++x) {
          const double P = (al * A.center[x] + be * B.center[x]) / z;
          at(lai::PF_PX + x) = P;
          at(lai::PF_PAX + x) = P - A.center[x];
        }
        at(lai::PF_C) = pi54s2 * A.coefs[ia] * B.coefs[ib] * std::exp(-al * be / z * ab2) / z;
      }
  }
}

int upload_class(PairClassHost& c) {
  LAI_CUDA_TRY(upload(c.d_sa, c.sa));
  LAI_CUDA_TRY(upload(c.d_sb, c.sb));
  LAI_CUDA_TRY(upload(c.d_fa, c.fa));
  LAI_CUDA_TRY(upload(c.d_fb, c.fb));
  LAI_CUDA_TRY(upload(c.d_AB, c.AB));
  LAI_CUDA_TRY(upload(c.d_Acen, c.Acen));
  LAI_CUDA_TRY(upload(c.d_prim, c.prim));
  if (c.Q.empty()) c.Q.assign(c.n(), 0.0);
  LAI_CUDA_TRY(upload(c.d_Q, c.Q));
  {  // per-pair primitive records (lai::BraRecField), FP64 and FP32
    const int n = c.n(), Kab = c.Ka * c.Kb;
    std::vector<double> rb((size_t)n * Kab * lai::kBraRec, 0.0);
    static const int from[lai::kBraRec] = {lai::PF_Q,  lai::PF_ZETA, lai::PF_HZ,  lai::PF_C,
                                           lai::PF_PX, lai::PF_PY,   lai::PF_PZ,  lai::PF_ALPHA,
                                           lai::PF_PAX, lai::PF_PAY, lai::PF_PAZ, -1};
    for (int p = 0; p < n; ++p)
      for (int t = 0; t < Kab; ++t)
        for (int f = 0; f < lai::kBraRec; ++f)
          if (from[f] >= 0)
            rb[((size_t)p * Kab + t) * lai::kBraRec + f] = c.prim[((size_t)from[f] * Kab + t) * n + p];
    std::vector<float> rbf(rb.size());
    for (size_t i = 0; i < rb.size(); ++i) rbf[i] = (float)rb[i];
    LAI_CUDA_TRY(upload(c.d_primb, rb));
    LAI_CUDA_TRY(upload(c.d_primbf, rbf));
  }
  {  // ket tiles of 32 pairs (lai::KetRecField), FP64 and FP32; pad lanes stay 0
    const int n = c.n(), Kab = c.Ka * c.Kb;
    const size_t ntile = ((size_t)n + lai::kKetTile - 1) / lai::kKetTile;
    std::vector<double> rk(ntile * Kab * lai::kKetRec * lai::kKetTile, 0.0);
    static const int from[lai::kKetRec] = {lai::PF_Q,   lai::PF_ZETA, lai::PF_HZ,  lai::PF_PX,
                                           lai::PF_PY,  lai::PF_PZ,   lai::PF_PAX, lai::PF_PAY,
                                           lai::PF_PAZ, lai::PF_C,    lai::PF_ALPHA};
    for (int p = 0; p < n; ++p)
      for (int t = 0; t < Kab; ++t)
        for (int f = 0; f < lai::kKetRec; ++f)
          rk[(((size_t)(p / lai::kKetTile) * Kab + t) * lai::kKetRec + f) * lai::kKetTile + p % lai::kKetTile] =
              c.prim[((size_t)from[f] * Kab + t) * n + p];
    std::vector<float> rkf(rk.size());
    for (size_t i = 0; i < rk.size(); ++i) rkf[i] = (float)rk[i];
    LAI_CUDA_TRY(upload(c.d_primk, rk));
    LAI_CUDA_TRY(upload(c.d_primkf, rkf));
  }
  return LAI_OK;
}

int ensure_scratch(lai_engine* E, size_t doubles) {
  if (E->d_scratch.bytes >= doubles * sizeof(double)) return LAI_OK;
  E->release_graph();
  LAI_CUDA_TRY(E->d_scratch.alloc(doubles * sizeof(double)));
  return LAI_OK;
}

cudaError_t scratch_pool(cudaMemPool_t* out) {
  static std::mutex m;
  static cudaMemPool_t pool = nullptr;  // engines of one process use one device
  std::lock_guard<std::mutex> lock(m);
  if (!pool) {
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t made = nullptr;
    if (cudaError_t e = cudaMemPoolCreate(&made, &props)) return e;
    uint64_t keep = 32 << 20;
    if (cudaError_t e = cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep)) {
      cudaMemPoolDestroy(made);
      return e;
    }
    pool = made;
  }
  *out = pool;
  return cudaSuccess;
}

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  cudaMemPool_t pool = nullptr;
  if (cudaError_t e = scratch_pool(&pool)) return e;
  return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

namespace {
std::mutex g_lane_mutex;
std::vector<LaneSet>& lane_pool() {  // never destroyed: the streams go with the CUDA context
  static auto* pool = new std::vector<LaneSet>;
  return *pool;
}
void destroy_lanes(LaneSet& set) {
  for (auto e : set.ev)
    if (e) cudaEventDestroy(e);
  for (auto s : set.side)
    if (s) cudaStreamDestroy(s);
  for (auto e : {set.t0, set.t1})
    if (e) cudaEventDestroy(e);
  if (set.main) cudaStreamDestroy(set.main);
  set = LaneSet{};
}
}  // namespace

int acquire_lanes(LaneSet& out) {
  {
    std::lock_guard<std::mutex> lock(g_lane_mutex);
    if (!lane_pool().empty()) {
      out = std::move(lane_pool().back());
      lane_pool().pop_back();
      return LAI_OK;
    }
  }
  while (out.ev.size() < (size_t)kLanes) {
    cudaEvent_t e = nullptr;
    LAI_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    out.ev.push_back(e);
  }
  while (out.side.size() + 1 < (size_t)kLanes) {
    cudaStream_t s = nullptr;
    LAI_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    out.side.push_back(s);
  }
  LAI_CUDA_TRY(cudaStreamCreateWithFlags(&out.main, cudaStreamNonBlocking));
  LAI_CUDA_TRY(cudaEventCreate(&out.t0));
  LAI_CUDA_TRY(cudaEventCreate(&out.t1));
  return LAI_OK;
}

// Work still queued on the set's streams was joined to the caller's stream, and the next
// engine's work on them simply follows it.
void release_lanes(LaneSet& set) {
  if (set.side.size() + 1 < (size_t)kLanes || !set.t1)
    return destroy_lanes(set);
  std::lock_guard<std::mutex> lock(g_lane_mutex);
  if (lane_pool().size() >= kPooledLaneSets) return destroy_lanes(set);
  lane_pool().push_back(std::move(set));
  set = LaneSet{};
}

// Id of the capture that the stream is part of, 0 if none.
static unsigned long long capture_of(cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(stream, &status, &id) != cudaSuccess) return 0;
  return status == cudaStreamCaptureStatusNone ? 0 : id;
}

LaunchLanes::LaunchLanes(lai_engine* E, cudaStream_t stream, size_t lanes) : E_(E), main_(stream), load_(1, 0.0), lock_(E->lanes_mutex) {
  E->fork_stream = stream;
  lanes = std::min(lanes, E->lanes.side.size() + 1);
  if (lanes < 2) return;
  // A side stream of an earlier call inside a capture belongs to that capture until it
  // ends, and another stream's work may not be queued on it.
  const unsigned long long own = capture_of(stream);
  load_.resize(lanes, -1.0);
  bool any = false;
  for (size_t i = 1; i < lanes; ++i) {
    const unsigned long long c = capture_of(E->lanes.side[i - 1]);
    if (c && c != own) load_[i] = kClosed;
    else any = true;
  }
  if (!any || cudaEventRecord(E->lanes.ev[0], stream) != cudaSuccess) load_.resize(1);  // one lane: the caller's stream
}

cudaError_t LaunchLanes::pick(double work, cudaStream_t* s) {
  size_t best = 0;
  for (size_t i = 1; i < load_.size(); ++i)
    if (std::max(load_[i], 0.0) < load_[best]) best = i;
  *s = best ? E_->lanes.side[best - 1] : main_;
  if (load_[best] < 0.0) {
    load_[best] = 0.0;
    if (cudaError_t e = cudaStreamWaitEvent(*s, E_->lanes.ev[0], 0)) return e;
  }
  load_[best] += work;
  return cudaSuccess;
}

cudaError_t LaunchLanes::join() {
  cudaError_t rc = cudaSuccess;
  for (size_t i = 1; i < load_.size(); ++i) {
    if (load_[i] < 0.0 || load_[i] == kClosed) continue;
    cudaError_t e = cudaEventRecord(E_->lanes.ev[i], E_->lanes.side[i - 1]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, E_->lanes.ev[i], 0);
    if (e != cudaSuccess) rc = e;
  }
  load_.assign(1, 0.0);
  if (lock_.owns_lock()) {
    E_->fork_stream = nullptr;
    lock_.unlock();
  }
  return rc;
}

// Launches the kernel of the block's class.  fp32 asks for the FP32 variant; the
// classes without one (generic kernel) run in FP64, and *ran_fp32 says which ran.
int launch_block(lai_engine* E, const lai::QuartetBlock& blk, const lai::JKArgs& args,
                 bool fp32, bool* ran_fp32, lai::LaunchTune tune) {
  const int la = blk.bra.la, lb = blk.bra.lb, lc = blk.ket.la, ld = blk.ket.lb;
  if (ran_fp32) *ran_fp32 = false;
  const bool untuned = tune.ps == 0 && tune.ksuper == 0 && tune.kernel == lai::KERNEL_DEFAULT;
  if (untuned && !fp32 && args.mode == lai::MODE_JK && lai::block_for_few(blk, E->num_sms)) tune.kernel = lai::KERNEL_BLOCK;
  if (lai::small_class_supported(la, lb, lc, ld) && tune.kernel != lai::KERNEL_BLOCK) {
    fp32 = fp32 && lai::small_fp32_class(la, lb, lc, ld);
    const int rc = lai::launch_small(blk, args, E->tab, E->stream, fp32, E->num_sms, tune);
    if (ran_fp32) *ran_fp32 = fp32;
    if (rc < 0) return fail(LAI_ECUDA, std::string("small-class launch failed: ") +
                                           cudaGetErrorString(cudaGetLastError()));
    return LAI_OK;
  }
  // the other classes: block-per-quartet, bra-sliced or tiled kernel, as tuned for this
  // block (lai_engine_autotune) or by default_kernel; FP32 requests go to the sliced
  // kernel where it exists, else to the block-per-quartet kernel's FP32 variant (the
  // tiled and generic kernels are FP64 only).  The raw-integral and Schwarz modes run on
  // the sliced and tiled kernels.
  int kern = tune.kernel != lai::KERNEL_DEFAULT ? tune.kernel
             : lai::default_kernel(la, lb, lc, ld, blk.total - blk.t_begin, E->num_sms);
  if (fp32) kern = lai::sliced_class_supported(la, lb, lc, ld) ? lai::KERNEL_SLICED : lai::KERNEL_BLOCK;
  if (kern == lai::KERNEL_BLOCK) {
    const bool f32 = fp32 && lai::block_fp32_class(la, lb, lc, ld);
    const int rc = lai::launch_blockq(blk, args, E->tab, E->stream, E->num_sms, f32);
    if (rc == 0) {
      if (ran_fp32) *ran_fp32 = f32;
      return LAI_OK;
    }
    if (rc < -1) return fail(LAI_ECUDA, std::string("block-per-quartet launch failed: ") +
                                            cudaGetErrorString(cudaGetLastError()));
  }
  if (kern != lai::KERNEL_TILED && lai::sliced_class_supported(la, lb, lc, ld)) {
    const int rc = lai::launch_sliced(blk, args, E->tab, E->stream, fp32, E->num_sms);
    if (ran_fp32) *ran_fp32 = fp32;
    if (rc < 0) return fail(LAI_ECUDA, std::string("sliced launch failed: ") +
                                           cudaGetErrorString(cudaGetLastError()));
    return LAI_OK;
  }
  {
    const int rc = lai::launch_tiled(blk, args, E->tab, E->stream, E->num_sms);
    if (rc == 0) return LAI_OK;
    if (rc < -1) return fail(LAI_ECUDA, std::string("tiled launch failed: ") +
                                            cudaGetErrorString(cudaGetLastError()));
  }
  const size_t need = lai::generic_global_scratch_doubles(la, lb, lc, ld, E->num_sms);
  if (int rc = ensure_scratch(E, need)) return rc;
  // one scratch buffer: launches that use it follow one another on the caller's stream
  const int rc = lai::launch_generic(blk, args, E->tab, E->fork_stream ? E->fork_stream : E->stream,
                                     E->d_scratch.as<double>(), E->d_scratch.bytes / sizeof(double), E->num_sms);
  if (rc < 0) return fail(LAI_ECUDA, std::string("generic launch failed: ") +
                                         cudaGetErrorString(cudaGetLastError()));
  return LAI_OK;
}

lai::QuartetBlock make_block(const lai_engine* E, const ClassPairBlock& b) {
  lai::QuartetBlock q{};
  q.bra = E->classes[b.bra]->view();
  q.ket = E->classes[b.ket]->view();
  q.offsets = b.dev_offsets;
  q.qbegin = b.dev_qbegin;
  q.total = b.total;
  q.same_class = (b.bra == b.ket);
  return q;
}

__global__ void absmax_kernel(const double* __restrict__ x, size_t n, unsigned long long* out) {
  double m = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    m = fmax(m, fabs(x[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  // non-negative doubles order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// max |x_i| of a device array (one stream synchronisation).
int device_absmax(lai_engine* E, const double* x, size_t n, cudaStream_t stream, double* out) {
  LAI_CUDA_TRY(E->d_absmax.ensure(sizeof(unsigned long long)));
  LAI_CUDA_TRY(cudaMemsetAsync(E->d_absmax.p, 0, sizeof(unsigned long long), stream));
  if (n > 0) {
    const size_t want = (n + 255) / 256;
    const unsigned grid = (unsigned)std::min<size_t>(want, (size_t)E->num_sms * 8);
    absmax_kernel<<<grid, 256, 0, stream>>>(x, n, E->d_absmax.as<unsigned long long>());
    LAI_CUDA_TRY(cudaGetLastError());
  }
  unsigned long long bits = 0;
  LAI_CUDA_TRY(cudaMemcpyAsync(&bits, E->d_absmax.p, sizeof(bits), cudaMemcpyDeviceToHost, stream));
  LAI_CUDA_TRY(cudaStreamSynchronize(stream));
  std::memcpy(out, &bits, sizeof(double));
  return LAI_OK;
}

// Elements of the engine's D/J/K arrays: nbf^2, or the packed blocks of a batched engine.
size_t engine_mat_elems(const lai_engine* E) {
  if (E->nsys > 1) return (size_t)E->sys_off[E->nsys];
  return (size_t)E->basis->nbf * (size_t)E->basis->nbf;
}

// Builds (once per cut value) the FP64/FP32 split of every block.
int build_split(lai_engine* E, double cut) {
  if (E->split_cut == cut) return LAI_OK;
  E->release_graph();  // a captured graph points into the buffers rebuilt here
  E->split_cut = -1.0;
  for (auto& bp : E->blocks) {
    auto& b = *bp;
    const auto& ca = *E->classes[b.bra];
    const auto& cb = *E->classes[b.ket];
    const int n = ca.n();
    std::vector<int64_t> o64(n + 1), o32(n + 1);
    std::vector<int> qb32(n);
    o64[0] = o32[0] = 0;
    for (int p = 0; p < n; ++p) {
      const int64_t cnt = b.offsets[p + 1] - b.offsets[p];
      const int base = b.qbegin.empty() ? 0 : b.qbegin[p];  // first ket of the bra's range
      int lo = 0, hi = (int)cnt;  // first ket with Q_p Q_q < cut
      while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (ca.Q[p] * cb.Q[base + mid] >= cut) lo = mid + 1; else hi = mid;
      }
      o64[p + 1] = o64[p] + lo;
      o32[p + 1] = o32[p] + (cnt - lo);
      qb32[p] = base + lo;
    }
    b.total64 = o64[n];
    b.total32 = o32[n];
    LAI_CUDA_TRY(upload(b.d_off64, o64));
    LAI_CUDA_TRY(upload(b.d_off32, o32));
    LAI_CUDA_TRY(upload(b.d_qb32, qb32));
  }
  E->split_cut = cut;
  return LAI_OK;
}

// Accumulators of J' (and of K') in a build: an element collects thousands of additions, in
// an order that the concurrent launches change, and four short sums carry a third of the
// rounding of one long one.  Norm of K against the sum of 24 shards, one -> four: 1.9e-15 ->
// 6.5e-16 at 175 functions, 4.5e-15 -> 1.5e-15 at 725, 5.8e-15 -> 1.9e-15 at 1600 (12
// shards); the time is the same at every size ((H2O)4/cc-pVDZ 1.17 ms, (H2O)64 1.32 s).  Above
// 2^24 elements, where they would take more than a gigabyte, one.
int accumulator_copies(size_t elems) { return elems <= (size_t(1) << 24) ? 4 : 1; }

// J' and K' of a build, elems each, one buffer (J' first).
int ensure_accumulators(lai_engine* E, size_t elems) {
  const size_t bytes = 2 * sizeof(double) * elems;
  if (E->d_JKp.bytes >= bytes) return LAI_OK;
  E->release_graph();
  LAI_CUDA_TRY(E->d_JKp.alloc(bytes));
  return LAI_OK;
}

// J = J' + J'^T, K = K' + K'^T on every system block of a batched engine's packed
// matrices (block s = nbf_s x nbf_s at element offset off[s]).
__global__ void symmetrize_batched_kernel(const double* __restrict__ Jp, const double* __restrict__ Kp,
                                          double* __restrict__ J, double* __restrict__ K,
                                          const int64_t* __restrict__ off, const int* __restrict__ nbfs,
                                          int nsys, int copies) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= off[nsys]) return;
  int lo = 0, hi = nsys;  // off[lo] <= idx < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= idx) lo = mid; else hi = mid;
  }
  const int n = nbfs[lo];
  const int64_t l = idx - off[lo];
  const int i = (int)(l / n), j = (int)(l - (int64_t)i * n);
  const int64_t tr = off[lo] + (int64_t)j * n + i, all = off[nsys];
  double sj = 0.0, sk = 0.0;
#pragma unroll 4
  for (int c = 0; c < copies; ++c, Jp += all, Kp += all) {
    sj += Jp[idx] + Jp[tr];
    sk += Kp[idx] + Kp[tr];
  }
  J[idx] = sj;
  K[idx] = sk;
}

// The launches of a plain build.  An engine has a block per pair of classes (la, lb, Ka, Kb),
// H2O/cc-pVQZ 666 of them for 120 angular classes; a launch each leaves the device to
// their set-up (lookup tables, class tables, 15 - 25 us of latency whatever the work).
// The blocks of one angular class that do not fill the device alone go out as one launch,
// each with its own split of a quartet, the heaviest items first.  Larger ones keep a launch
// of their own: a list has one geometry for all its entries, the table batch of the longest
// contraction, and holds its items together in time.
int build_launches(lai_engine* E) {
  const int nb = (int)E->blocks.size();
  std::map<std::array<int, 5>, std::vector<int>> groups;  // kernel and class -> blocks
  std::vector<int> single;
  for (int b = 0; b < nb; ++b) {
    const lai::QuartetBlock q = make_block(E, *E->blocks[b]);
    const int la = q.bra.la, lb = q.bra.lb, lc = q.ket.la, ld = q.ket.lb;
    int kind = 0;  // 1: thread-per-quartet, split; 2: block-per-quartet
    if (lai::small_class_supported(la, lb, lc, ld))
      kind = lai::block_for_few(q, E->num_sms) ? 2 : q.total < (int64_t)E->num_sms * lai::kSplitQuartetsPerSm ? 1 : 0;
    else if (lai::default_kernel(la, lb, lc, ld, q.total, E->num_sms) == lai::KERNEL_BLOCK &&
             q.total < (int64_t)E->num_sms * lai::kListBlocksPerSm)
      kind = 2;
    if (kind) groups[{kind, la, lb, lc, ld}].push_back(b);
    else single.push_back(b);
  }
  std::vector<lai::MultiEntry> entries;
  auto work_of = [&](int b) { return E->blocks[b]->alg_flops * (double)E->blocks[b]->total; };
  auto add_single = [&](int b) {
    lai_engine::LaunchItem it;
    it.block = b;
    it.work = work_of(b);
    E->launches.push_back(it);
  };
  for (int b : single) add_single(b);
  for (auto& [key, blocks] : groups) {
    if (blocks.size() == 1) {
      add_single(blocks[0]);
      continue;
    }
    lai_engine::LaunchItem it;
    it.block_kernel = key[0] == 2;
    it.la = key[1]; it.lb = key[2]; it.lc = key[3]; it.ld = key[4];
    it.first = (int)entries.size();
    it.n = (int)blocks.size();
    double prims = 0.0;
    std::vector<lai::MultiEntry> es;
    std::vector<int64_t> P;
    for (int b : blocks) {
      lai::MultiEntry e{};
      e.blk = make_block(E, *E->blocks[b]);
      P.push_back((int64_t)e.blk.bra.Ka * e.blk.bra.Kb * e.blk.ket.Ka * e.blk.ket.Kb);
      prims += (double)P.back() * (double)e.blk.total;
      it.Pmax = std::max(it.Pmax, P.back());
      it.work += work_of(b);
      e.ps = e.nsplit = e.csplit = 1;
      es.push_back(e);
    }
    if (!it.block_kernel) {
      // lanes per quartet: no lane with more than a quarter of its share of the launch in
      // one quartet (or 24 primitive quartets), and enough lanes to fill the device
      const double lanes = 512.0 * E->num_sms, most = std::max(24.0, 0.25 * prims / lanes);
      double used = 0.0;
      for (size_t i = 0; i < es.size(); ++i) {
        const int Kab = es[i].blk.bra.Ka * es[i].blk.bra.Kb;
        while (es[i].ps < 32 && es[i].ps < Kab && (double)P[i] / es[i].ps > most) es[i].ps <<= 1;
        es[i].nsplit = (int)std::max(1.0, std::min((double)(P[i] / Kab), (double)P[i] / es[i].ps / most));
        used += (double)es[i].blk.total * es[i].ps;
      }
      for (bool grew = true; grew && used < lanes;) {
        grew = false;
        for (auto& e : es)
          if (e.ps < 32 && e.ps < e.blk.bra.Ka * e.blk.bra.Kb) {
            used += (double)e.blk.total * e.ps;
            e.ps <<= 1;
            grew = true;
          }
      }
    } else {
      // the same over blocks: four per SM, a quartet's primitive quartets first
      const double slots = 4.0 * E->num_sms;
      const int nroots = (it.la + it.lb + it.lc + it.ld) / 2 + 1;
      const int rows = lai::ncart_range(it.la, it.la + it.lb);
      const double least = 2.0 * std::max(1, (rows + 31) / 32 * 32 / (3 * nroots));
      const double most = std::max(least, prims / (2.0 * slots));
      double used = 0.0;
      for (size_t i = 0; i < es.size(); ++i) {
        es[i].nsplit = (int)std::max(1.0, std::min((double)P[i] / most, 1024.0));
        used += (double)es[i].blk.total * es[i].nsplit;
      }
      const int nchunks = lai::block_ket_chunks(it.lc, it.ld);
      const int cs = (int)std::max(1.0, std::min((double)nchunks, slots / used));
      for (auto& e : es) e.csplit = cs;
    }
    // heaviest work items first
    std::vector<int> order(es.size());
    std::iota(order.begin(), order.end(), 0);
    auto cost = [&](int i) { return (double)P[i] / es[i].nsplit / (it.block_kernel ? 1 : es[i].ps); };
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost(x) > cost(y); });
    for (int i : order) {
      lai::MultiEntry e = es[i];
      e.work0 = it.nwork;
      const int per = 32 / e.ps;
      it.nwork += it.block_kernel ? e.blk.total * e.nsplit * e.csplit : (e.blk.total + per - 1) / per * e.nsplit;
      entries.push_back(e);
    }
    E->launches.push_back(it);
  }
  std::stable_sort(E->launches.begin(), E->launches.end(),
                   [](const auto& x, const auto& y) { return x.work > y.work; });
  return upload(E->d_multi, entries) == cudaSuccess ? LAI_OK : fail(LAI_ECUDA, "launch list upload failed");
}

// J' = K' = 0 and every class-pair launch of a build of the density dD, on `stream`
// (spread over the lanes).  Part 1 of a mixed build's blocks runs in FP32.
int enqueue_jk(lai_engine* E, const double* dD, cudaStream_t stream, const lai_jk_opts& o, double cut, bool timed,
               lai_jk_report& rep) {
  const int nbf = (int)E->basis->nbf;
  const bool batched = E->nsys > 1;
  const size_t elems = engine_mat_elems(E);
  struct Restore {
    lai_engine* E;
    cudaStream_t saved;
    ~Restore() { E->stream = saved; }
  } restore{E, E->stream};
  E->stream = stream;
  const int copies = accumulator_copies(elems);
  LAI_CUDA_TRY(cudaMemsetAsync(E->d_JKp.p, 0, 2 * sizeof(double) * copies * elems, stream));
  if (timed) LAI_CUDA_TRY(cudaEventRecord(E->ev0, stream));
  lai::JKArgs args{};
  args.D = dD;
  args.J = E->jp();
  args.K = E->kp(copies * elems);
  args.copy_mask = copies - 1;
  args.copy_stride = (int64_t)elems;
  args.nbf = nbf;
  args.mode = lai::MODE_JK;
  args.prim_eps = E->prim_eps;
  args.prim_rel32 = o.fp32_prim_rel;
  if (batched) {
    args.sys_off = E->d_sys_off.as<int64_t>();
    args.sys_nbf = E->d_sys_nbf.as<int>();
  }
  int launches = 0;
  int64_t nq = 0, nq32 = 0;
  double flops = 0;
  const bool mixed = cut > 0.0;
  const int nparts = mixed ? 2 : 1;
  if (o.profile) {
    const size_t need = 2 * nparts * E->blocks.size();
    while (E->prof_ev.size() < need) {
      cudaEvent_t ev;
      LAI_CUDA_TRY(cudaEventCreate(&ev));
      E->prof_ev.push_back(ev);
    }
    E->prof_block.clear();
    E->prof_quartets.clear();
    LAI_CUDA_TRY(E->d_prof_prims.ensure(sizeof(unsigned long long) * std::max<size_t>(1, nparts * E->blocks.size())));
    LAI_CUDA_TRY(cudaMemsetAsync(E->d_prof_prims.p, 0, E->d_prof_prims.bytes, stream));
  }
  E->prof_n = 0;
  // profiled builds time every launch by itself, in block order on one stream
  LaunchLanes lanes(E, stream, o.profile ? 1 : kLanes);
  if (!o.profile && !mixed && o.shard_count == 1 && !E->tuned) {
    for (const auto& it : E->launches) {
      LAI_CUDA_TRY(lanes.pick(it.work, &E->stream));
      if (it.block >= 0) {
        if (int rc = launch_block(E, make_block(E, *E->blocks[it.block]), args)) return rc;
      } else {
        const lai::MultiEntry* list = E->d_multi.as<lai::MultiEntry>() + it.first;
        const int rc = it.block_kernel
                           ? lai::launch_blockq_list(it.la, it.lb, it.lc, it.ld, it.Pmax, list, it.n, it.nwork, args,
                                                     E->tab, E->stream, E->num_sms)
                           : lai::launch_small_list(it.la, it.lb, it.lc, it.ld, list, it.n, it.nwork, args, E->tab,
                                                    E->stream, E->num_sms);
        if (rc < 0) return fail(LAI_ECUDA, std::string("launch failed: ") + cudaGetErrorString(cudaGetLastError()));
      }
      ++launches;
    }
    for (const auto& b : E->blocks) {
      nq += b->total;
      flops += b->alg_flops * (double)b->total;
    }
  } else
  for (size_t i = 0; i < E->blocks.size(); ++i) {
    const size_t b = o.profile ? i : (size_t)E->launch_order[i];
    const auto& bp = *E->blocks[b];
    for (int part = 0; part < nparts; ++part) {
      // part 0: the whole block (FP64), or its FP64 prefix when mixed; part 1: the
      // FP32 suffix
      lai::QuartetBlock q = make_block(E, bp);
      int64_t total = bp.total;
      if (mixed) {
        total = part == 0 ? bp.total64 : bp.total32;
        q.offsets = (part == 0 ? bp.d_off64 : bp.d_off32).as<int64_t>();
        if (part == 1) q.qbegin = bp.d_qb32.as<int>();  // the FP64 part keeps the block's ket starts
      }
      // this shard's contiguous slice of the part
      int64_t lo = 0, hi = 0;
      lai_shard_range(total, o.shard_index, o.shard_count, &lo, &hi);
      if (hi <= lo) continue;
      q.t_begin = lo;
      q.total = hi;
      args.prim_count = o.profile ? E->d_prof_prims.as<unsigned long long>() + E->prof_n : nullptr;
      if (o.profile) LAI_CUDA_TRY(cudaEventRecord(E->prof_ev[2 * E->prof_n], stream));
      bool ran32 = false;
      LAI_CUDA_TRY(lanes.pick(bp.alg_flops * (double)(hi - lo), &E->stream));
      if (int rc = launch_block(E, q, args, part == 1, &ran32, bp.tune)) return rc;
      if (o.profile) {
        LAI_CUDA_TRY(cudaEventRecord(E->prof_ev[2 * E->prof_n + 1], stream));
        E->prof_block.push_back((int)b);
        E->prof_quartets.push_back(hi - lo);
        ++E->prof_n;
      }
      ++launches;
      nq += hi - lo;
      if (ran32) nq32 += hi - lo;
      flops += bp.alg_flops * (double)(hi - lo);
    }
  }
  LAI_CUDA_TRY(lanes.join());
  rep.quartets_fp64 = nq - nq32;
  rep.quartets_fp32 = nq32;
  rep.fp32_schwarz_cut = cut;
  rep.alg_flops = flops;
  rep.kernel_launches = launches;
  rep.seconds_device = 0;
  return LAI_OK;
}

// forced_cut >= 0: use this Schwarz cut for the FP32 split instead of deriving it
// from max|D| (which synchronizes the stream; not allowed while capturing a graph).
int run_jk(lai_engine* E, const double* dD, double* dJ, double* dK, cudaStream_t stream,
           const lai_jk_opts& o, lai_jk_report* rep, bool timed, double forced_cut = -1.0) {
  const int nbf = (int)E->basis->nbf;
  const bool batched = E->nsys > 1;
  const size_t elems = engine_mat_elems(E);
  if (o.shard_count < 1 || o.shard_index < 0 || o.shard_index >= o.shard_count)
    return fail(LAI_EINVAL, "lai_jk: bad shard_index/shard_count");
  const int copies = accumulator_copies(elems);
  if (int rc = ensure_accumulators(E, copies * elems)) return rc;
  // Mixed precision: a quartet runs in FP32 when Q_ij Q_kl max|D| < fp32_cut.  The
  // Schwarz cut fp32_cut / max|D| is rounded down to a power of two (conservative:
  // fewer FP32 quartets), so that the split, built on the host, is rebuilt only
  // when max|D| moves past a power of two.
  double cut = forced_cut >= 0.0 ? forced_cut : 0.0;
  if (o.fp32_cut > 0.0 && forced_cut < 0.0) {
    double maxd = 0.0;
    if (int rc = device_absmax(E, dD, elems, stream, &maxd)) return rc;
    if (maxd > 0.0 && std::isfinite(maxd)) cut = std::exp2(std::floor(std::log2(o.fp32_cut / maxd)));
  }
  if (cut > 0.0)
    if (int rc = build_split(E, cut)) return rc;
  lai_jk_report r{};
  if (int rc = enqueue_jk(E, dD, stream, o, cut, timed, r)) return rc;
  const int64_t nn = (int64_t)elems;
  if (nn > 0) {
    if (batched)
      symmetrize_batched_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, stream>>>(
          E->jp(), E->kp(copies * elems), dJ, dK, E->d_sys_off.as<int64_t>(), E->d_sys_nbf.as<int>(), E->nsys, copies);
    else
      symmetrize_kernel<<<(unsigned)((nn + 255) / 256), 256, 0, stream>>>(E->jp(), E->kp(copies * elems), dJ, dK, nbf,
                                                                          copies);
    ++r.kernel_launches;
  }
  LAI_CUDA_TRY(cudaGetLastError());
  if (timed) LAI_CUDA_TRY(cudaEventRecord(E->ev1, stream));
  if (rep) {
    const double total = rep->seconds_total;
    *rep = r;
    rep->seconds_total = total;
  }
  return LAI_OK;
}

// Launch choices of every block, timed one launch at a time, and whether builds use them.
int tune_blocks(lai_engine* engine, const double* d_D, cudaStream_t s, double* ms_before, double* ms_after) {
  const size_t elems = engine_mat_elems(engine);
  const int copies = accumulator_copies(elems);
  lai::JKArgs args{};
  args.D = d_D;
  args.J = engine->jp();
  args.K = engine->kp(copies * elems);
  args.copy_mask = copies - 1;
  args.copy_stride = (int64_t)elems;
  args.nbf = (int)engine->basis->nbf;
  args.mode = lai::MODE_JK;
  args.prim_eps = engine->prim_eps;
  if (engine->nsys > 1) {
    args.sys_off = engine->d_sys_off.as<int64_t>();
    args.sys_nbf = engine->d_sys_nbf.as<int>();
  }
  struct Events {
    cudaEvent_t e[2] = {nullptr, nullptr};
    ~Events() { for (auto x : e) if (x) cudaEventDestroy(x); }
  } ev;
  for (auto& x : ev.e)
    if (cudaEventCreate(&x) != cudaSuccess) return LAI_ECUDA;
  const cudaEvent_t e0 = ev.e[0], e1 = ev.e[1];
  struct Restore {
    lai_engine* E;
    cudaStream_t saved;
    ~Restore() { E->stream = saved; }
  } restore{engine, engine->stream};
  engine->stream = s;
  double before = 0.0, after = 0.0;
  auto time_launch = [&](const lai::QuartetBlock& q, lai::LaunchTune t, float* ms) -> int {
    float best = 1e30f;
    for (int rep = 0; rep < 2; ++rep) {  // the first run warms caches, the minimum counts
      if (cudaEventRecord(e0, s) != cudaSuccess) return LAI_ECUDA;
      if (int r = launch_block(engine, q, args, false, nullptr, t)) return r;
      if (cudaEventRecord(e1, s) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) return LAI_ECUDA;
      float m = 0;
      cudaEventElapsedTime(&m, e0, e1);
      best = std::min(best, m);
    }
    *ms = best;
    return LAI_OK;
  };
  for (auto& bp : engine->blocks) {
    const lai::QuartetBlock q = make_block(engine, *bp);
    float base = 0;
    if (const int rc = time_launch(q, bp->tune, &base)) return rc;
    before += base;
    if (!lai::small_class_supported(q.bra.la, q.bra.lb, q.ket.la, q.ket.lb)) {
      // kernel family: block-per-quartet, bra-sliced, tiled
      lai::LaunchTune best = bp->tune;
      float best_ms = base;
      for (int k : {lai::KERNEL_BLOCK, lai::KERNEL_SLICED, lai::KERNEL_TILED}) {
        if (k == lai::KERNEL_SLICED && !lai::sliced_class_supported(q.bra.la, q.bra.lb, q.ket.la, q.ket.lb))
          continue;
        lai::LaunchTune t;
        t.kernel = k;
        float m = 0;
        if (const int rc = time_launch(q, t, &m)) return rc;
        if (m < 0.98f * best_ms) { best_ms = m; best = t; }
      }
      bp->tune = best;
      after += best_ms;
      continue;
    }
    const int Kab = q.bra.Ka * q.bra.Kb;
    lai::LaunchTune best = bp->tune;
    float best_ms = base;
    for (int ps = 1; ps <= 8 && ps < 2 * Kab; ps <<= 1)
      for (int ks : {1, 4, 16}) {
        float m = 0;
        if (const int rc = time_launch(q, lai::LaunchTune{ps, ks}, &m)) return rc;
        if (m < 0.98f * best_ms) { best_ms = m; best = lai::LaunchTune{ps, ks}; }
      }
    if (q.total - q.t_begin < (int64_t)engine->num_sms * 64) {
      float m = 0;
      lai::LaunchTune t;
      t.kernel = lai::KERNEL_BLOCK;
      if (const int rc = time_launch(q, t, &m)) return rc;
      if (m < 0.98f * best_ms) { best_ms = m; best = t; }
    }
    bp->tune = best;
    after += best_ms;
  }
  // The launches were timed one at a time, a build runs them side by side: the choices stay
  // only if a whole build is faster with them than with the built-in schedule.
  float build[2] = {1e30f, 1e30f};
  lai_jk_opts o;
  lai_jk_opts_default(&o);
  for (int rep = 0; rep < 3; ++rep)  // the first of each warms up
    for (int k = 0; k < 2; ++k) {
      engine->tuned = k == 1;
      lai_jk_report r{};
      if (cudaEventRecord(e0, s) != cudaSuccess) return LAI_ECUDA;
      const int rc = enqueue_jk(engine, d_D, s, o, 0.0, false, r);
      engine->tuned = false;
      if (rc) return rc;
      float m = 0;
      if (cudaEventRecord(e1, s) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
          cudaEventElapsedTime(&m, e0, e1) != cudaSuccess)
        return LAI_ECUDA;
      if (rep > 0) build[k] = std::min(build[k], m);
    }
  engine->tuned = build[1] < 0.99f * build[0];
  if (!engine->tuned)
    for (auto& bp : engine->blocks) bp->tune = lai::LaunchTune{};
  if (ms_before) *ms_before = before;
  if (ms_after) *ms_after = engine->tuned ? after : before;
  return LAI_OK;
}

// splitmix64
inline uint64_t mix64(uint64_t& x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void fp64_fma_probe(double* out, int iters) {
  double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-10, a2 = a0 + 2e-10, a3 = a0 + 3e-10;
  double a4 = a0 + 4e-10, a5 = a0 + 5e-10, a6 = a0 + 6e-10, a7 = a0 + 7e-10;
  const double m = 0.999999, c = 1e-7;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
      a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
    }
  }
  const double r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (r == 12345.678) out[0] = r;  // keep the chain alive
}

}  // namespace host
}  // namespace lai

extern "C" {

int lai_shard_range(int64_t total, int index, int count, int64_t* lo, int64_t* hi) {
  if (count < 1 || index < 0 || index >= count || total < 0 || !lo || !hi)
    return fail(LAI_EINVAL, "lai_shard_range: bad arguments");
  // 128-bit products: total * count may exceed 63 bits for huge blocks
  *lo = (int64_t)((__int128)total * index / count);
  *hi = (int64_t)((__int128)total * (index + 1) / count);
  return LAI_OK;
}

void lai_engine_opts_default(lai_engine_opts* opts) {
  if (!opts) return;
  opts->schwarz_threshold = 1e-12;
  opts->device = 0;
  opts->prim_threshold = -1.0;
}

void lai_jk_opts_default(lai_jk_opts* opts) {
  if (!opts) return;
  opts->fp32_cut = 0.0;
  opts->check_symmetric = 0;
  opts->shard_index = 0;
  opts->shard_count = 1;
  opts->profile = 0;
  opts->graph = 0;
  opts->fp32_prim_rel = 0.0;
}

}  // extern "C"

namespace lai {
namespace host {

// Engine over `basis`; for a batched engine, `merged` is the concatenation of the
// systems' shells (each tagged with its system) and sys_nbf their function counts.
int create_engine(const lai_basis* basis, std::unique_ptr<lai_basis> merged, const std::vector<int>& sys_nbf,
                  const lai_engine_opts* opts, lai_engine** out) {
  lai_engine_opts o;
  lai_engine_opts_default(&o);
  if (opts) o = *opts;
  if (!(o.schwarz_threshold >= 0.0)) return fail(LAI_EINVAL, "negative Schwarz threshold");
  int ndev = 0;
  LAI_CUDA_TRY(cudaGetDeviceCount(&ndev));
  if (o.device < 0 || o.device >= ndev) return fail(LAI_EINVAL, "lai_engine_create: bad device");
  // The kernel launchers set their launch attributes (dynamic shared-memory
  // limits) and cache occupancies once per process, and CUDA keeps those per
  // device: every engine of a process therefore uses the first engine's device.
  static std::atomic<int> process_device{-1};
  int first = -1;
  if (!process_device.compare_exchange_strong(first, o.device) && first != o.device)
    return fail(LAI_ENOTSUP, "lai_engine_create: this process already runs engines on another CUDA device "
                             "(one device per process: run one process per GPU)");
  LAI_CUDA_TRY(cudaSetDevice(o.device));
  auto E = std::make_unique<lai_engine>();
  if (merged) {
    E->merged = std::move(merged);
    E->basis = E->merged.get();
    E->nsys = (int)sys_nbf.size();
    E->sys_nbf = sys_nbf;
    E->sys_off.assign(E->nsys + 1, 0);
    for (int i = 0; i < E->nsys; ++i) E->sys_off[i + 1] = E->sys_off[i] + (int64_t)sys_nbf[i] * sys_nbf[i];
    LAI_CUDA_TRY(upload(E->d_sys_nbf, E->sys_nbf));
    LAI_CUDA_TRY(upload(E->d_sys_off, E->sys_off));
  } else {
    E->basis = basis;
  }
  basis = E->basis;
  E->device = o.device;
  E->thr = o.schwarz_threshold;
  E->prim_eps = o.prim_threshold < 0.0 ? 1e-3 * o.schwarz_threshold : o.prim_threshold;
  LAI_CUDA_TRY(cudaDeviceGetAttribute(&E->num_sms, cudaDevAttrMultiProcessorCount, o.device));
  cudaMemPool_t pool = nullptr;
  LAI_CUDA_TRY(scratch_pool(&pool));
  if (int rc = acquire_lanes(E->lanes)) return rc;
  E->stream = E->lanes.main;
  E->ev0 = E->lanes.t0;
  E->ev1 = E->lanes.t1;
  if (int rc = setup_tables(E.get())) return rc;
  if (int rc = build_classes(E.get())) return rc;
  if (int rc = setup_pairs(E.get())) return rc;
  E->launch_order.resize(E->blocks.size());
  std::iota(E->launch_order.begin(), E->launch_order.end(), 0);
  std::stable_sort(E->launch_order.begin(), E->launch_order.end(), [&](int x, int y) {
    return E->blocks[x]->alg_flops * (double)E->blocks[x]->total >
           E->blocks[y]->alg_flops * (double)E->blocks[y]->total;
  });
  if (int rc = build_launches(E.get())) return rc;
  *out = E.release();
  return LAI_OK;
}

}  // namespace host
}  // namespace lai

extern "C" {

int lai_engine_create(const lai_basis* basis, const lai_engine_opts* opts, lai_engine** out) {
  if (!out || !basis) return fail(LAI_EINVAL, "lai_engine_create: null argument");
  *out = nullptr;
  return create_engine(basis, nullptr, {}, opts, out);
}

int lai_engine_create_batched(int nsys, const lai_basis* const* bases, const lai_engine_opts* opts,
                              lai_engine** out) {
  if (!out || nsys < 1 || !bases) return fail(LAI_EINVAL, "lai_engine_create_batched: null argument");
  *out = nullptr;
  auto merged = std::make_unique<lai_basis>();
  std::vector<int> nbf(nsys);
  for (int s = 0; s < nsys; ++s) {
    if (!bases[s]) return fail(LAI_EINVAL, "lai_engine_create_batched: null basis");
    for (const HostShell& sh : bases[s]->shells) {
      merged->shells.push_back(sh);
      merged->shells.back().sys = s;  // func stays local to the system
    }
    nbf[s] = (int)bases[s]->nbf;
  }
  merged->nbf = 0;  // no single matrix size: D/J/K are packed per system
  return create_engine(nullptr, std::move(merged), nbf, opts, out);
}

int lai_engine_batch_layout(lai_engine* engine, int* nsys, int64_t* offsets, int* nbf) {
  if (!engine) return fail(LAI_EINVAL, "lai_engine_batch_layout: null engine");
  if (nsys) *nsys = engine->nsys;
  if (engine->nsys == 1) {
    if (offsets) { offsets[0] = 0; offsets[1] = (int64_t)engine->basis->nbf * engine->basis->nbf; }
    if (nbf) nbf[0] = (int)engine->basis->nbf;
    return LAI_OK;
  }
  if (offsets) std::copy(engine->sys_off.begin(), engine->sys_off.end(), offsets);
  if (nbf) std::copy(engine->sys_nbf.begin(), engine->sys_nbf.end(), nbf);
  return LAI_OK;
}

void lai_engine_destroy(lai_engine* engine) {
  if (engine) {
    cudaSetDevice(engine->device);
    delete engine;
  }
}

int lai_engine_schwarz(lai_engine* engine, double* Q) {
  if (engine && engine->nsys > 1) return fail(LAI_ENOTSUP, "lai_engine_schwarz: not available for a batched engine");
  if (!engine || !Q) return fail(LAI_EINVAL, "lai_engine_schwarz: null argument");
  std::copy(engine->Q_all.begin(), engine->Q_all.end(), Q);
  return LAI_OK;
}

int lai_jk_build_device(lai_engine* engine, const double* d_D, double* d_J, double* d_K,
                        void* stream, const lai_jk_opts* opts, lai_jk_report* report) {
  if (!engine || !d_D || !d_J || !d_K) return fail(LAI_EINVAL, "lai_jk_build_device: null argument");
  lai_jk_opts o;
  lai_jk_opts_default(&o);
  if (opts) o = *opts;
  if (!(o.fp32_cut >= 0.0)) return fail(LAI_EINVAL, "lai_jk_build_device: fp32_cut must be >= 0");
  if (!(o.fp32_prim_rel >= 0.0 && o.fp32_prim_rel < 1.0))
    return fail(LAI_EINVAL, "lai_jk_build_device: fp32_prim_rel must be in [0, 1)");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!o.graph) return run_jk(engine, d_D, d_J, d_K, s, o, report, false);
  if (!s || o.profile) return fail(LAI_EINVAL, "lai_jk_build_device: graph mode needs a stream and profile = 0");
  lai_engine::GraphKey key{d_D, d_J, d_K, s, o.fp32_cut, o.shard_index, o.shard_count, o.fp32_prim_rel};
  if (engine->graph_exec && engine->graph_key == key) {
    LAI_CUDA_TRY(cudaGraphLaunch(engine->graph_exec, s));
    if (report) *report = engine->graph_report;
    return LAI_OK;
  }
  // First call: an ordinary build (allocations, the FP32 split and its cut), whose
  // result is this call's; then the same launch sequence captured for the replays.
  lai_jk_report rep{};
  if (int rc = run_jk(engine, d_D, d_J, d_K, s, o, &rep, false)) return rc;
  engine->release_graph();
  cudaGraph_t graph = nullptr;
  LAI_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  lai_jk_report rep2{};
  const int rc = run_jk(engine, d_D, d_J, d_K, s, o, &rep2, false, rep.fp32_schwarz_cut);
  const cudaError_t ce = cudaStreamEndCapture(s, &graph);
  if (rc) {
    if (graph) cudaGraphDestroy(graph);
    return rc;
  }
  LAI_CUDA_TRY(ce);
  const cudaError_t ie = cudaGraphInstantiate(&engine->graph_exec, graph, 0);
  cudaGraphDestroy(graph);
  LAI_CUDA_TRY(ie);
  engine->graph_key = key;
  engine->graph_report = rep;
  if (report) *report = rep;
  return LAI_OK;
}

int lai_jk_build(lai_engine* engine, const double* D, size_t nbf, double* J, double* K,
                 const lai_jk_opts* opts, lai_jk_report* report) {
  auto t0 = std::chrono::steady_clock::now();
  if (!engine || !D || !J || !K) return fail(LAI_EINVAL, "lai_jk_build: null argument");
  if (engine->nsys > 1) return fail(LAI_EINVAL, "lai_jk_build: batched engine (use lai_jk_build_batched)");
  if ((long)nbf != engine->basis->nbf)
    return fail(LAI_EINVAL, "lai_jk_build: nbf mismatch (expected " +
                                std::to_string(engine->basis->nbf) + ", got " +
                                std::to_string(nbf) + ")");
  lai_jk_opts o;
  lai_jk_opts_default(&o);
  if (opts) o = *opts;
  if (!(o.fp32_cut >= 0.0)) return fail(LAI_EINVAL, "lai_jk_build: fp32_cut must be >= 0");
  if (!(o.fp32_prim_rel >= 0.0 && o.fp32_prim_rel < 1.0))
    return fail(LAI_EINVAL, "lai_jk_build: fp32_prim_rel must be in [0, 1)");
  if (o.check_symmetric) {
    for (size_t i = 0; i < nbf; ++i)
      for (size_t j = 0; j < i; ++j)
        if (std::fabs(D[i * nbf + j] - D[j * nbf + i]) > 1e-12 * (1.0 + std::fabs(D[i * nbf + j])))
          return fail(LAI_EINVAL, "lai_jk_build: density matrix is not symmetric");
  }
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  const size_t bytes = sizeof(double) * nbf * nbf;
  for (DevBuf* b : {&engine->d_D, &engine->d_J, &engine->d_K}) LAI_CUDA_TRY(b->ensure(bytes));
  cudaStream_t s = engine->stream;
  LAI_CUDA_TRY(cudaMemcpyAsync(engine->d_D.p, D, bytes, cudaMemcpyHostToDevice, s));
  if (int rc = run_jk(engine, engine->d_D.as<double>(), engine->d_J.as<double>(),
                      engine->d_K.as<double>(), s, o, report, true))
    return rc;
  LAI_CUDA_TRY(cudaMemcpyAsync(J, engine->d_J.p, bytes, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaMemcpyAsync(K, engine->d_K.p, bytes, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaStreamSynchronize(s));
  if (report) {
    float ms = 0;
    cudaEventElapsedTime(&ms, engine->ev0, engine->ev1);
    report->seconds_device = ms * 1e-3;
    report->seconds_total =
        std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  }
  return LAI_OK;
}

int lai_jk_build_batched(lai_engine* engine, const double* D, double* J, double* K, const lai_jk_opts* opts,
                         lai_jk_report* report) {
  auto t0 = std::chrono::steady_clock::now();
  if (!engine || !D || !J || !K) return fail(LAI_EINVAL, "lai_jk_build_batched: null argument");
  lai_jk_opts o;
  lai_jk_opts_default(&o);
  if (opts) o = *opts;
  if (!(o.fp32_cut >= 0.0)) return fail(LAI_EINVAL, "lai_jk_build_batched: fp32_cut must be >= 0");
  if (!(o.fp32_prim_rel >= 0.0 && o.fp32_prim_rel < 1.0))
    return fail(LAI_EINVAL, "lai_jk_build_batched: fp32_prim_rel must be in [0, 1)");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  const size_t bytes = sizeof(double) * engine_mat_elems(engine);
  for (DevBuf* b : {&engine->d_D, &engine->d_J, &engine->d_K}) LAI_CUDA_TRY(b->ensure(bytes));
  cudaStream_t s = engine->stream;
  LAI_CUDA_TRY(cudaMemcpyAsync(engine->d_D.p, D, bytes, cudaMemcpyHostToDevice, s));
  if (int rc = run_jk(engine, engine->d_D.as<double>(), engine->d_J.as<double>(), engine->d_K.as<double>(), s, o,
                      report, true))
    return rc;
  LAI_CUDA_TRY(cudaMemcpyAsync(J, engine->d_J.p, bytes, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaMemcpyAsync(K, engine->d_K.p, bytes, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaStreamSynchronize(s));
  if (report) {
    float ms = 0;
    cudaEventElapsedTime(&ms, engine->ev0, engine->ev1);
    report->seconds_device = ms * 1e-3;
    report->seconds_total = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  }
  return LAI_OK;
}

int lai_eri_batch_screened(lai_engine* engine, double* out, size_t out_capacity,
                           lai_quartet_meta* meta, size_t meta_capacity, int64_t* n_quartets,
                           int64_t* n_values) {
  if (engine && engine->nsys > 1) return fail(LAI_ENOTSUP, "lai_eri_batch_screened: not available for a batched engine");
  if (!engine) return fail(LAI_EINVAL, "lai_eri_batch_screened: null engine");
  int64_t nq = 0, nv = 0;
  std::vector<int64_t> vals_per(engine->blocks.size());
  for (size_t b = 0; b < engine->blocks.size(); ++b) {
    const auto& bp = *engine->blocks[b];
    const auto& ca = *engine->classes[bp.bra];
    const auto& cb = *engine->classes[bp.ket];
    vals_per[b] = (int64_t)lai::ncart(ca.la) * lai::ncart(ca.lb) * lai::ncart(cb.la) * lai::ncart(cb.lb);
    nq += bp.total;
    nv += bp.total * vals_per[b];
  }
  if (n_quartets) *n_quartets = nq;
  if (n_values) *n_values = nv;
  if (!out || !meta) return LAI_OK;
  if ((int64_t)out_capacity < nv || (int64_t)meta_capacity < nq)
    return fail(LAI_EINVAL, "lai_eri_batch_screened: output capacity too small");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  DevBuf d_out, d_meta;
  LAI_CUDA_TRY(d_out.alloc(sizeof(double) * (size_t)std::max<int64_t>(nv, 1)));
  LAI_CUDA_TRY(d_meta.alloc(sizeof(int) * 4 * (size_t)std::max<int64_t>(nq, 1)));
  int64_t qo = 0, vo = 0;
  for (size_t b = 0; b < engine->blocks.size(); ++b) {
    const auto& bp = *engine->blocks[b];
    lai::JKArgs args{};
    args.mode = lai::MODE_RAW;
    args.raw_out = d_out.as<double>() + vo;
    args.raw_meta = d_meta.as<int>() + 4 * qo;
    if (int rc = launch_block(engine, make_block(engine, bp), args)) return rc;
    qo += bp.total;
    vo += bp.total * vals_per[b];
  }
  std::vector<int> hmeta(4 * (size_t)nq);
  LAI_CUDA_TRY(cudaMemcpyAsync(out, d_out.p, sizeof(double) * nv, cudaMemcpyDeviceToHost, engine->stream));
  LAI_CUDA_TRY(cudaMemcpyAsync(hmeta.data(), d_meta.p, sizeof(int) * 4 * nq, cudaMemcpyDeviceToHost,
                               engine->stream));
  LAI_CUDA_TRY(cudaStreamSynchronize(engine->stream));
  qo = 0;
  vo = 0;
  for (size_t b = 0; b < engine->blocks.size(); ++b) {
    const auto& bp = *engine->blocks[b];
    const auto& ca = *engine->classes[bp.bra];
    const auto& cb = *engine->classes[bp.ket];
    for (int64_t t = 0; t < bp.total; ++t) {
      lai_quartet_meta& m = meta[qo + t];
      m.offset = vo + t * vals_per[b];
      m.fa = hmeta[4 * (qo + t)]; m.fb = hmeta[4 * (qo + t) + 1];
      m.fc = hmeta[4 * (qo + t) + 2]; m.fd = hmeta[4 * (qo + t) + 3];
      m.na = lai::ncart(ca.la); m.nb = lai::ncart(ca.lb);
      m.nc = lai::ncart(cb.la); m.nd = lai::ncart(cb.lb);
    }
    qo += bp.total;
    vo += bp.total * vals_per[b];
  }
  return LAI_OK;
}

int lai_jk_last_profile(lai_engine* engine, int capacity, double* ms, double* alg_flops,
                        double* alg_flops_executed, int64_t* quartets, int64_t* prim_quartets,
                        int* lclass) {
  if (!engine) return fail(LAI_EINVAL, "lai_jk_last_profile: null engine");
  const int n = engine->prof_n;
  if (capacity < n || !ms) return n;
  std::vector<unsigned long long> prims(n, 0);
  if (n > 0) {
    LAI_CUDA_TRY(cudaEventSynchronize(engine->prof_ev[2 * n - 1]));
    LAI_CUDA_TRY(cudaMemcpy(prims.data(), engine->d_prof_prims.p, sizeof(unsigned long long) * n,
                            cudaMemcpyDeviceToHost));
  }
  for (int i = 0; i < n; ++i) {
    float t = 0;
    LAI_CUDA_TRY(cudaEventElapsedTime(&t, engine->prof_ev[2 * i], engine->prof_ev[2 * i + 1]));
    ms[i] = t;
    const auto& b = *engine->blocks[engine->prof_block[i]];
    const auto& ca = *engine->classes[b.bra];
    const auto& cb = *engine->classes[b.ket];
    const double nq = (double)engine->prof_quartets[i];
    if (alg_flops) alg_flops[i] = b.alg_flops * nq;
    if (alg_flops_executed)
      alg_flops_executed[i] = b.flops_per_prim * (double)prims[i] + b.flops_per_quartet * nq;
    if (quartets) quartets[i] = engine->prof_quartets[i];
    if (prim_quartets) prim_quartets[i] = (int64_t)prims[i];
    if (lclass) {
      lclass[4 * i] = ca.la; lclass[4 * i + 1] = ca.lb;
      lclass[4 * i + 2] = cb.la; lclass[4 * i + 3] = cb.lb;
    }
  }
  return n;
}

int64_t lai_engine_quartet_count(lai_engine* engine) {
  if (!engine) return -1;
  int64_t n = 0;
  for (auto& b : engine->blocks) n += b->total;
  return n;
}

int lai_engine_sample_quartets(lai_engine* engine, int64_t n, uint64_t seed, int32_t* quartets) {
  if (engine && engine->nsys > 1) return fail(LAI_ENOTSUP, "lai_engine_sample_quartets: not available for a batched engine");
  if (!engine || n < 0 || (n > 0 && !quartets)) return fail(LAI_EINVAL, "lai_engine_sample_quartets");
  std::vector<int64_t> pref(engine->blocks.size() + 1, 0);
  for (size_t b = 0; b < engine->blocks.size(); ++b) pref[b + 1] = pref[b] + engine->blocks[b]->total;
  const int64_t total = pref.back();
  if (total == 0) return n == 0 ? LAI_OK : fail(LAI_ESTATE, "engine has no quartets");
  uint64_t st = seed;
  for (int64_t i = 0; i < n; ++i) {
    const int64_t t = (int64_t)(mix64(st) % (uint64_t)total);
    const size_t b = std::upper_bound(pref.begin(), pref.end(), t) - pref.begin() - 1;
    const auto& bp = *engine->blocks[b];
    const int64_t tl = t - pref[b];
    const int p = (int)(std::upper_bound(bp.offsets.begin(), bp.offsets.end(), tl) - bp.offsets.begin() - 1);
    const int q = (int)(tl - bp.offsets[p]);
    const auto& ca = *engine->classes[bp.bra];
    const auto& cb = *engine->classes[bp.ket];
    quartets[4 * i] = ca.sa[p];
    quartets[4 * i + 1] = ca.sb[p];
    quartets[4 * i + 2] = cb.sa[q];
    quartets[4 * i + 3] = cb.sb[q];
  }
  return LAI_OK;
}

int lai_engine_autotune(lai_engine* engine, const double* d_D, void* stream, double* ms_before,
                        double* ms_after) {
  if (!engine || !d_D) return fail(LAI_EINVAL, "lai_engine_autotune: null argument");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // one ordinary build first: allocations and accumulators
  lai_jk_opts o;
  lai_jk_opts_default(&o);
  const size_t elems = engine_mat_elems(engine);
  DevBuf dJ, dK;
  LAI_CUDA_TRY(dJ.alloc(sizeof(double) * elems));
  LAI_CUDA_TRY(dK.alloc(sizeof(double) * elems));
  if (int rc = run_jk(engine, d_D, dJ.as<double>(), dK.as<double>(), s, o, nullptr, false)) return rc;
  engine->release_graph();
  engine->tuned = false;
  for (auto& bp : engine->blocks) bp->tune = lai::LaunchTune{};
  const int rc = tune_blocks(engine, d_D, s, ms_before, ms_after);
  if (rc) {
    for (auto& bp : engine->blocks) bp->tune = lai::LaunchTune{};
    return fail(rc, "lai_engine_autotune: a timing launch failed");
  }
  return LAI_OK;
}

int lai_engine_tune_table(lai_engine* engine, int capacity, int* rows) {
  if (!engine) return fail(LAI_EINVAL, "lai_engine_tune_table: null engine");
  const int n = (int)engine->blocks.size();
  if (!rows || capacity < n) return n;
  for (int b = 0; b < n; ++b) {
    const auto& bp = *engine->blocks[b];
    const auto& ca = *engine->classes[bp.bra];
    const auto& cb = *engine->classes[bp.ket];
    int* r = rows + 10 * b;
    r[0] = ca.la; r[1] = ca.lb; r[2] = cb.la; r[3] = cb.lb;
    r[4] = ca.Ka * ca.Kb; r[5] = cb.Ka * cb.Kb;
    r[6] = (int)std::min<int64_t>(bp.total, INT32_MAX);
    r[7] = bp.tune.kernel ? -bp.tune.kernel : bp.tune.ps; r[8] = bp.tune.ksuper;
    r[9] = (int)std::min<int64_t>(bp.total / 1000, INT32_MAX);
  }
  return n;
}

int lai_probe_fp64_peak(int device, double* tflops) {
  if (!tflops) return fail(LAI_EINVAL, "lai_probe_fp64_peak: null output");
  LAI_CUDA_TRY(cudaSetDevice(device));
  int sms = 0;
  LAI_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  DevBuf out;
  LAI_CUDA_TRY(out.alloc(8));
  cudaEvent_t a, b;
  LAI_CUDA_TRY(cudaEventCreate(&a));
  LAI_CUDA_TRY(cudaEventCreate(&b));
  const int threads = 256, blocks = sms * 8, iters = 4096;
  fp64_fma_probe<<<blocks, threads>>>(out.as<double>(), 64);  // warm-up
  double best = 0;
  for (int rep = 0; rep < 3; ++rep) {
    LAI_CUDA_TRY(cudaEventRecord(a));
    fp64_fma_probe<<<blocks, threads>>>(out.as<double>(), iters);
    LAI_CUDA_TRY(cudaEventRecord(b));
    LAI_CUDA_TRY(cudaEventSynchronize(b));
    float ms = 0;
    LAI_CUDA_TRY(cudaEventElapsedTime(&ms, a, b));
    const double fl = 2.0 * 8 * 16 * (double)iters * threads * blocks;
    best = std::max(best, fl / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  *tflops = best;
  return LAI_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Read-only accessors for other translation units of the library (not C ABI).
// ---------------------------------------------------------------------------
namespace lai {

int engine_device(const lai_engine* E) { return E->device; }
int engine_num_sms(const lai_engine* E) { return E->num_sms; }
int engine_nbf(const lai_engine* E) { return (int)E->basis->nbf; }
double engine_prim_eps(const lai_engine* E) { return E->prim_eps; }
RysTablesView engine_tables(const lai_engine* E) { return E->tab; }
const lai_basis* engine_basis(const lai_engine* E) { return E->basis; }
int engine_nsys(const lai_engine* E) { return E->nsys; }
int engine_block_count(const lai_engine* E) { return (int)E->blocks.size(); }
QuartetBlock engine_block(const lai_engine* E, int i) { return make_block(E, *E->blocks[i]); }
void engine_set_error(const char* msg) { g_last_error = msg; }

}  // namespace lai
