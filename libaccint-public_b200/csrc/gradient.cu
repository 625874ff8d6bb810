// Nuclear gradient of the two-electron energy E = 1/2 tr(D J) - 1/4 tr(D K) at
// fixed density over the engine's screened canonical quartets (the quartets the
// J/K build computes), and the C ABI around it.  dE/dD = J - K/2 comes from the
// J/K build itself.  No counterpart in the reference (MAX_DERIVATIVE_ORDER = 0,
// config.hpp.in:49).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "engine_internal.h"
#include "eri_kernels.h"

using namespace lai::host;

namespace {

int ensure_atoms(lai_engine* E) {
  if (E->natom >= 0) return LAI_OK;
  const auto& sh = E->basis->shells;
  std::vector<int> at(sh.size());
  int natom = 0;
  for (size_t s = 0; s < sh.size(); ++s) {
    if (sh[s].atom < 0) return fail(LAI_EINVAL, "gradient: the basis was created without atom indices");
    at[s] = sh[s].atom;
    natom = std::max(natom, sh[s].atom + 1);
  }
  LAI_CUDA_TRY(upload(E->d_shell_atom, at));
  E->natom = natom;
  return LAI_OK;
}

// grad[i] = sum over the kGradCopies accumulators, stride doubles apart
__global__ void sum_copies_kernel(const double* __restrict__ copies, int stride, int n, double* __restrict__ grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int c = 0; c < lai::kGradCopies; ++c) s += copies[(size_t)c * stride + i];
  grad[i] = s;
}

// The accumulators of one call.  A call outside a capture uses the engine's, after the work
// of the call before it, whatever stream that went to: an allocation per call, also from a
// pool, is refused in a thread that is capturing, and breaks a global capture of another
// thread.  Inside a capture they are the graph's own.
struct Accumulators {
  lai_engine* E;
  cudaStream_t s;
  std::unique_lock<std::mutex> lock;  // until the call's work is queued
  void* p = nullptr;
  bool owned = false;
  Accumulators(lai_engine* engine, cudaStream_t stream) : E(engine), s(stream), lock(engine->grad_mutex) {}
  int take(size_t bytes) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    LAI_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) {
      LAI_CUDA_TRY(scratch_alloc(&p, bytes, s));
      owned = true;
      return LAI_OK;
    }
    if (!E->grad_done) LAI_CUDA_TRY(cudaEventCreateWithFlags(&E->grad_done, cudaEventDisableTiming));
    LAI_CUDA_TRY(E->d_grad_acc.ensure(bytes));
    LAI_CUDA_TRY(cudaStreamWaitEvent(s, E->grad_done, 0));
    p = E->d_grad_acc.p;
    return LAI_OK;
  }
  ~Accumulators() {
    if (owned) cudaFreeAsync(p, s);
    else if (p) cudaEventRecord(E->grad_done, s);
  }
};

}  // namespace

extern "C" {

int lai_engine_natom(lai_engine* engine) {
  if (!engine) return fail(LAI_EINVAL, "lai_engine_natom: null engine");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  if (int rc = ensure_atoms(engine)) return rc;
  return engine->natom;
}

int lai_jk_gradient_device(lai_engine* engine, const double* d_D, double* d_grad, void* stream) {
  if (engine && engine->nsys > 1) return fail(LAI_ENOTSUP, "lai_jk_gradient: not available for a batched engine");
  if (!engine || !d_D || !d_grad) return fail(LAI_EINVAL, "lai_jk_gradient_device: null argument");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  if (int rc = ensure_atoms(engine)) return rc;
  cudaStream_t stream_of_call = static_cast<cudaStream_t>(stream);
  const int n3 = 3 * engine->natom, stride = (n3 + 15) / 16 * 16;
  const size_t bytes = sizeof(double) * stride * lai::kGradCopies;
  Accumulators copies(engine, stream_of_call);
  if (int rc = copies.take(bytes)) return rc;
  double* const acc = static_cast<double*>(copies.p);
  LAI_CUDA_TRY(cudaMemsetAsync(acc, 0, bytes, stream_of_call));
  const int nbf = (int)engine->basis->nbf;
  LaunchLanes lanes(engine, stream_of_call, kLanes);
  for (const int b : engine->launch_order) {
    const auto& bp = engine->blocks[b];
    const lai::QuartetBlock q = make_block(engine, *bp);
    cudaStream_t s = stream_of_call;
    LAI_CUDA_TRY(lanes.pick(bp->alg_flops * (double)bp->total, &s));
    const int rs = lai::launch_grad_small(q, d_D, nbf, engine->d_shell_atom.as<int>(), acc, stride, engine->prim_eps,
                                          engine->tab, s, engine->num_sms);
    if (rs == 0) continue;
    if (rs != -1)
      return fail(LAI_ECUDA, std::string("gradient launch failed: ") + cudaGetErrorString(cudaGetLastError()));
    const int rc = lai::launch_grad_block(q, d_D, nbf, engine->d_shell_atom.as<int>(), acc, stride, engine->prim_eps,
                                          engine->tab, s, engine->num_sms);
    if (rc < 0)
      return fail(LAI_ECUDA, std::string("gradient launch failed: ") + cudaGetErrorString(cudaGetLastError()));
  }
  LAI_CUDA_TRY(lanes.join());
  if (n3 > 0) sum_copies_kernel<<<(n3 + 127) / 128, 128, 0, stream_of_call>>>(acc, stride, n3, d_grad);
  LAI_CUDA_TRY(cudaGetLastError());
  return LAI_OK;
}

int lai_jk_gradient(lai_engine* engine, const double* D, size_t nbf, double* grad) {
  if (!engine || !D || !grad) return fail(LAI_EINVAL, "lai_jk_gradient: null argument");
  if ((long)nbf != engine->basis->nbf) return fail(LAI_EINVAL, "lai_jk_gradient: nbf mismatch");
  LAI_CUDA_TRY(cudaSetDevice(engine->device));
  if (int rc = ensure_atoms(engine)) return rc;
  const size_t bytes = sizeof(double) * nbf * nbf;
  DevBuf dD, dG;
  LAI_CUDA_TRY(dD.alloc(bytes));
  LAI_CUDA_TRY(dG.alloc(sizeof(double) * 3 * engine->natom));
  cudaStream_t s = engine->stream;
  LAI_CUDA_TRY(cudaMemcpyAsync(dD.p, D, bytes, cudaMemcpyHostToDevice, s));
  if (int rc = lai_jk_gradient_device(engine, dD.as<double>(), dG.as<double>(), s)) return rc;
  LAI_CUDA_TRY(cudaMemcpyAsync(grad, dG.p, sizeof(double) * 3 * engine->natom, cudaMemcpyDeviceToHost, s));
  LAI_CUDA_TRY(cudaStreamSynchronize(s));
  return LAI_OK;
}

}  // extern "C"
