// Host-side types shared by the translation units of the engine: device buffers,
// shells and bases, pair classes, quartet blocks and the engine object behind the
// opaque C handles of include/libaccint_b200.h.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/libaccint_b200.h"
#include "dev_buf.h"
#include "eri_device.cuh"
#include "eri_kernels.h"

namespace lai {
namespace host {

// Records msg as the thread's last error (lai_last_error) and returns code.
int fail(int code, const std::string& msg);

#define LAI_CUDA_TRY(expr)                                                              \
  do {                                                                                  \
    cudaError_t e_ = (expr);                                                            \
    if (e_ != cudaSuccess)                                                              \
      return fail(e_ == cudaErrorMemoryAllocation ? LAI_ENOMEM : LAI_ECUDA,             \
                  std::string(#expr) + ": " + cudaGetErrorString(e_));                  \
  } while (0)

// Stream-ordered scratch of one call (cudaFreeAsync gives it back), from a memory pool of
// this library that keeps up to 32 MB: the default pool returns its memory at every
// synchronization, and an allocation after one takes 0.3 - 2 ms.  lai_engine_create makes
// the pool, so that no call under stream capture does.
cudaError_t scratch_pool(cudaMemPool_t* out);
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);

template <typename T>
cudaError_t upload(DevBuf& b, const std::vector<T>& v) {
  cudaError_t e = b.alloc(v.size() * sizeof(T));
  if (e != cudaSuccess || v.empty()) return e;
  return cudaMemcpy(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
}

}  // namespace host
}  // namespace lai

// ---------------------------------------------------------------------------
// Basis
// ---------------------------------------------------------------------------
struct HostShell {
  int l;
  double center[3];
  std::vector<double> exps_all, coefs_all;  // normalized, all primitives as given
  std::vector<double> exps, coefs;          // nonzero-coefficient primitives only
  int atom;
  long func;     // first function of the shell within its system
  int sys = 0;   // system index (batched engines merge independent systems)
};

struct lai_basis {
  std::vector<HostShell> shells;
  long nbf = 0;
};

namespace lai {
namespace host {

// An engine's streams and events.  Builds (LaunchLanes) run on the caller's stream, lane 0,
// and side[i - 1], lane i.  Creating them takes about 0.4 ms, which would be a sixth of a
// small engine's set-up, so a destroyed engine's set goes back to a process-wide pool
// (at most kPooledLaneSets kept; mutex) and the next engine takes it.
struct LaneSet {
  cudaStream_t main = nullptr;        // the engine's own stream
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> ev;        // [0] fork, [i] end of side[i - 1]
  cudaEvent_t t0 = nullptr, t1 = nullptr;  // timed builds
};
constexpr int kLanes = 8;
constexpr size_t kPooledLaneSets = 4;
int acquire_lanes(LaneSet& out);
void release_lanes(LaneSet& set);

struct PairClassHost {
  int la, lb, Ka, Kb;
  double qprim_max = 0.0;
  std::vector<int> sa, sb, fa, fb;  // shell and function indices (oriented)
  std::vector<int> sys;             // system of each pair (batched engines)
  std::vector<int> seg;             // [nsys + 1] first pair of each system (pairs sorted by system)
  std::vector<double> Q;
  std::vector<double> AB;          // SoA [3][n]
  std::vector<double> Acen;        // SoA [3][n] centre of the first shell (a)
  std::vector<double> prim;        // SoA [PF_COUNT][Kab][n]
  int n() const { return (int)sa.size(); }
  // device copies
  DevBuf d_sa, d_sb, d_fa, d_fb, d_Q, d_AB, d_Acen, d_prim, d_primb, d_primbf, d_primk, d_primkf;
  bool batched = false;             // more than one system
  bool on_device = false;           // an engine's class: its tables are in the engine's d_pairs
  lai::PairClassDev dev{};
  lai::PairClassDev view() const {
    if (on_device) return dev;
    lai::PairClassDev v;
    v.la = la; v.lb = lb; v.Ka = Ka; v.Kb = Kb; v.npairs = n();
    v.shell_a = d_sa.as<int>(); v.shell_b = d_sb.as<int>();
    v.func_a = d_fa.as<int>(); v.func_b = d_fb.as<int>();
    v.Q = d_Q.as<double>(); v.AB = d_AB.as<double>(); v.Acen = d_Acen.as<double>();
    v.prim = d_prim.as<double>();
    v.qprim_max = qprim_max;
    v.sys = nullptr;
    v.primf = nullptr;
    v.primb = d_primb.as<double>();
    v.primbf = d_primbf.as<float>();
    v.primk = d_primk.as<double>();
    v.primkf = d_primkf.as<float>();
    return v;
  }
};

struct ClassPairBlock {
  int bra, ket;                 // class indices, bra >= ket
  std::vector<int64_t> offsets; // host copy
  const int64_t* dev_offsets = nullptr;
  std::vector<int> qbegin;      // first ket of each bra pair (batched engines: its system's segment)
  const int* dev_qbegin = nullptr;  // null for a single system (every ket range starts at 0)
  int64_t total = 0;
  double alg_flops = 0;         // per quartet of this block (all nonzero primitives)
  double flops_per_prim = 0;    // per primitive quartet
  double flops_per_quartet = 0; // per contracted quartet (normalization + digestion)
  // Mixed-precision split of this block for one FP32 cut: the kets of bra pair p
  // are sorted by Schwarz bound, so those with Q_p Q_q >= cut form a prefix (the
  // FP64 part, offsets64) and the rest a suffix (the FP32 part: offsets32, with
  // qbegin32[p] its first ket).
  int64_t total64 = 0, total32 = 0;
  DevBuf d_off64, d_off32, d_qb32;

  lai::LaunchTune tune;         // launch parameters chosen by lai_engine_autotune (0 = heuristic)
};

}  // namespace host
}  // namespace lai

struct lai_engine {
  ~lai_engine();
  const lai_basis* basis = nullptr;
  // batched engines: the merged basis (owned) and the per-system layout of the
  // packed D/J/K arrays (block s = nbf_s x nbf_s at element offset sys_off[s])
  std::unique_ptr<lai_basis> merged;
  int nsys = 1;
  std::vector<int> sys_nbf;
  std::vector<int64_t> sys_off;   // [nsys + 1]
  lai::host::DevBuf d_sys_nbf, d_sys_off;
  int device = 0;
  int num_sms = 148;
  double thr = 1e-12;
  double prim_eps = 1e-15;
  cudaStream_t stream = nullptr;
  lai::RysTablesView tab{};
  lai::host::DevBuf d_pairs;     // pair tables of every class and quartet ranges of every block
  std::vector<std::unique_ptr<lai::host::PairClassHost>> classes;
  std::vector<std::unique_ptr<lai::host::ClassPairBlock>> blocks;
  std::vector<double> Q_all;     // nshell x nshell Schwarz matrix
  lai::host::DevBuf d_JKp, d_D, d_J, d_K;
  double* jp() const { return d_JKp.as<double>(); }
  double* kp(size_t elems) const { return d_JKp.as<double>() + elems; }  // elems: all of J' (every accumulator)
  lai::host::DevBuf d_scratch;    // of the generic kernel
  lai::host::DevBuf d_status;
  double split_cut = -1.0;       // FP32 cut the blocks' mixed-precision split was built for
  lai::host::DevBuf d_absmax;
  lai::host::DevBuf d_shell_atom;  // [nshell] atom of each shell (gradients)
  int natom = -1;
  lai::host::DevBuf d_grad_acc;    // accumulators of a gradient, after grad_done
  cudaEvent_t grad_done = nullptr;
  std::mutex grad_mutex;
  // one-electron integrals: shell table, primitives and shell pairs grouped by
  // (la, lb) class (built on first use; one_electron.cu)
  lai::host::DevBuf d_1e_shell, d_1e_exp, d_1e_coef, d_1e_pairs, d_1e_charges;
  std::vector<int> one_e_class;    // per class: la, lb, first pair, pair count
  // CUDA graph of one device build (lai_jk_opts.graph) and what it was captured for
  struct GraphKey {
    const double* D;
    double* J;
    double* K;
    cudaStream_t stream;
    double fp32_cut;
    int shard_index, shard_count;
    double fp32_prim_rel;
    bool operator==(const GraphKey& o) const {
      return D == o.D && J == o.J && K == o.K && stream == o.stream && fp32_cut == o.fp32_cut &&
             shard_index == o.shard_index && shard_count == o.shard_count && fp32_prim_rel == o.fp32_prim_rel;
    }
  };
  cudaGraphExec_t graph_exec = nullptr;
  GraphKey graph_key{};
  lai_jk_report graph_report{};
  void release_graph() {
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    graph_exec = nullptr;
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // per-launch profile of the last build with opts.profile
  std::vector<cudaEvent_t> prof_ev;
  std::vector<int> prof_block;
  std::vector<int64_t> prof_quartets;
  lai::host::DevBuf d_prof_prims;
  int prof_n = 0;
  // streams the independent class-pair launches of one build are spread over
  lai::host::LaneSet lanes;
  std::mutex lanes_mutex;             // held while launches are queued on the lanes
  cudaStream_t fork_stream = nullptr; // caller's stream while a build is spread over lanes
  std::vector<int> launch_order;      // blocks by descending estimated work
  // The launches of a plain build (FP64, one shard, untuned), by descending estimated
  // work: single blocks, and groups of a class's smaller blocks that share a launch
  // (build_launches).
  struct LaunchItem {
    int block = -1;                   // a single block, or
    bool block_kernel = false;        // a group for the block-per-quartet kernel, or for the split thread-per-quartet one
    int la = 0, lb = 0, lc = 0, ld = 0;
    int first = 0, n = 0;             // its entries in d_multi
    int64_t nwork = 0, Pmax = 0;
    double work = 0.0;
  };
  std::vector<LaunchItem> launches;
  lai::host::DevBuf d_multi;          // MultiEntry of every group
  bool tuned = false;                 // lai_engine_autotune has chosen per-block launches
};

inline lai_engine::~lai_engine() {
  release_graph();
  for (auto e : prof_ev) cudaEventDestroy(e);
  if (grad_done) cudaEventDestroy(grad_done);
  classes.clear();
  blocks.clear();
  lai::host::release_lanes(lanes);
}

namespace lai {
namespace host {

// Implemented in engine.cu.
void fill_pair_data(const lai_basis* basis, PairClassHost& c);
int upload_class(PairClassHost& c);
int launch_block(lai_engine* E, const lai::QuartetBlock& blk, const lai::JKArgs& args,
                 bool fp32 = false, bool* ran_fp32 = nullptr, lai::LaunchTune tune = lai::LaunchTune{});
lai::QuartetBlock make_block(const lai_engine* E, const ClassPairBlock& b);
int ensure_scratch(lai_engine* E, size_t doubles);
int ensure_accumulators(lai_engine* E, size_t elems);

// Spreads independent launches over the engine's lanes: pick(w) returns the stream of
// the lane with the least estimated work so far; join() makes the caller's stream wait
// for all of them.  The class-pair launches of one build only add to J'/K' (or the
// gradient) with atomics, so their order does not matter, and most of them do not fill
// the device alone: H2O / cc-pVQZ has 666 class pairs, most with work for a few warps.  The blocks
// go out by descending estimated work, so that the small launches fill the large ones'
// last waves.  kLanes is the number of hardware queues a process gets by default; more
// streams would share them.  One stream -> eight, with the kernels of the time (device time
// of a build): H2O/STO-3G 106 -> 49 us, (H2O)16/cc-pVDZ 53.2 -> 39.3 ms, (H2O)64/cc-pVDZ
// 1505 -> 1390 ms; (H2O)6/cc-pVDZ gradient 82.5 -> 30.5 ms.  Now, every launch by itself on
// one stream against a build: H2O/cc-pVQZ 19.6 -> 3.3 ms (small launches shared as well),
// C6H14/cc-pVTZ 90.6 -> 86.1 ms.
class LaunchLanes {
 public:
  LaunchLanes(lai_engine* E, cudaStream_t stream, size_t lanes);
  ~LaunchLanes() { join(); }
  LaunchLanes(const LaunchLanes&) = delete;
  cudaError_t pick(double work, cudaStream_t* s);
  cudaError_t join();

 private:
  lai_engine* E_;
  cudaStream_t main_;
  static constexpr double kClosed = 1e300;
  std::vector<double> load_;   // estimated work per lane; < 0: not forked yet
  // Gradients and density-fitting integrals of several threads on one engine queue their
  // launches one after another: they share the lanes' events.  (J/K builds share the
  // accumulators as well, and are the caller's to serialize.)
  std::unique_lock<std::mutex> lock_;
};
double alg_work(int la, int lb, int lc, int ld, int Ka, int Kb, int Kc, int Kd);
double alg_per_prim(int la, int lb, int lc, int ld);
double alg_per_quartet(int la, int lb, int lc, int ld);

// Implemented in setup.cu: the lookup tables, and the pair tables, bounds and quartet
// ranges of the engine's classes (build_classes has listed their pairs).
int setup_tables(lai_engine* E);
int setup_pairs(lai_engine* E);

}  // namespace host
}  // namespace lai
