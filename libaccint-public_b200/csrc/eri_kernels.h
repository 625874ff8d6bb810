// Launch entry points of the ERI/J-K kernels (host side).
#pragma once

#include <cuda_runtime.h>

#include "eri_device.cuh"

namespace lai {

// Thread-per-quartet kernels for the small classes (eri_small.cu).  Returns 1 if
// the class (la,lb|lc,ld) has a specialised kernel and it was launched, 0 if the
// class is not covered (use the generic kernel), <0 on a launch error.
// Launch parameters of the thread-per-quartet kernels chosen by the autotuner
// (lai_engine_autotune); 0 = the built-in heuristic.  ps = lanes per quartet
// (primitive split, power of two), ksuper = chunks per super-chunk.
struct LaunchTune {
  int ps = 0;
  int ksuper = 0;
  int kernel = 0;  // classes outside the thread-per-quartet set: 0 = default choice,
                   // KERNEL_TILED, KERNEL_SLICED or KERNEL_BLOCK
};
enum { KERNEL_DEFAULT = 0, KERNEL_TILED = 2, KERNEL_SLICED = 3, KERNEL_BLOCK = 4 };
// One of several blocks of a class that share a launch: work items [work0, next entry's
// work0) are its chunks of 32 / ps quartets, nsplit parts by ket primitive each
// (thread-per-quartet kernels), or its quartets times nsplit * csplit parts
// (block-per-quartet kernel).
struct MultiEntry {
  QuartetBlock blk;
  int64_t work0;
  int ps;
  int nsplit, csplit;
  int pad;
};
// A launch with fewer quartets per SM than this splits them over lanes.
constexpr int kSplitQuartetsPerSm = 1024;
// A block-kernel launch with fewer quartets per SM than this shares a launch.  Without a
// limit -> 1024 -> 256 -> 64 -> 16: C6H14/cc-pVTZ 84.4, 83.3, 81.7, 79.7, 79.5 ms, (H2O)2/cc-pVQZ
// 27.3, 27.4, 27.4, 27.1, 26.5, (H2O)23/cc-pVDZ 91.5, 91.5, 89.8, 89.8, 89.8, (H2O)64/cc-pVDZ
// 1318, 1306, 1307, 1307, 1308; below 16 the small ones wait for launches again
// ((H2O)4/cc-pVTZ 13.6, 13.5, 13.6, 13.5, 13.7, (H2O)8/cc-pVDZ 5.13, 5.14, 5.14, 5.14, 5.17).
constexpr int kListBlocksPerSm = 64;
int launch_small_list(int la, int lb, int lc, int ld, const MultiEntry* list, int n, int64_t nwork,
                      const JKArgs& args, const RysTablesView& tab, cudaStream_t stream, int num_sms);
int launch_small(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab,
                 cudaStream_t stream, bool fp32, int num_sms, LaunchTune tune = LaunchTune{});
bool small_class_supported(int la, int lb, int lc, int ld);
// Whether the class has an FP32 variant.  Of the g classes only (gs|ss) has: the FP32
// primitive sums are compensated up to 18 (e0|f0) integrals, and (gs|ps) has 45.
constexpr bool small_fp32_class(int la, int lb, int lc, int ld) { return la <= 3 || lb + lc + ld == 0; }

// Bra-sliced kernels for the medium classes (eri_sliced.cu); same return codes.
int launch_sliced(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab,
                  cudaStream_t stream, bool fp32, int num_sms);
bool sliced_class_supported(int la, int lb, int lc, int ld);

// Kernel family of a J/K launch of nq quartets of a class outside the thread-per-quartet
// set when no tuned choice exists (measured per class on B200: eri_block.cu).
int default_kernel(int la, int lb, int lc, int ld, int64_t nq, int num_sms);
// Warp-per-quartet kernel with lanes over the output integrals (eri_tiled.cu),
// any class with l <= 4, all modes; 0 on success, -1 if the class does not fit shared
// memory.
int launch_tiled(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab, cudaStream_t stream,
                 int num_sms);

// Block-per-quartet kernel (eri_block.cu), any class with l <= 4, J/K mode only: 0 on
// success, -1 for another mode, -3 on a CUDA error.
// fp32 asks for the FP32 variant (block_fp32_class).
int launch_blockq(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab, cudaStream_t stream,
                  int num_sms, bool fp32);
int launch_blockq_list(int la, int lb, int lc, int ld, int64_t Pmax, const MultiEntry* list, int n, int64_t nwork,
                       const JKArgs& args, const RysTablesView& tab, cudaStream_t stream, int num_sms);
int block_ket_chunks(int lc, int ld);  // digestion chunks of a ket, the most parts of csplit
bool block_fp32_class(int la, int lb, int lc, int ld);
// whether a J/K launch of a thread-per-quartet class goes to the block-per-quartet kernel
bool block_for_few(const QuartetBlock& blk, int num_sms);

// Warp-per-quartet generic kernel (eri_generic.cu), any class with l <= 4.
int launch_generic(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab,
                   cudaStream_t stream, double* gscratch, size_t gscratch_doubles, int num_sms);
// Global scratch (doubles) the generic kernel needs for class (la,lb|lc,ld) when
// its (e0|f0) block does not fit in shared memory; 0 if it fits.
size_t generic_global_scratch_doubles(int la, int lb, int lc, int ld, int num_sms);

// Block-per-quartet gradient kernel (eri_grad_block.cu), any class: adds dE/dR of the block's quartets
// (E = 1/2 tr DJ - 1/4 tr DK at fixed D) to grad.  0 on success.  grad holds kGradCopies
// accumulators [natom][3], grad_stride doubles apart, that the caller sums: a gradient has
// so few elements that the atomics of a whole launch would queue up on them.
constexpr int kGradCopies = 64;
int launch_grad_block(const QuartetBlock& blk, const double* D, int nbf, const int* shell_atom, double* grad,
                      int grad_stride, double prim_eps, const RysTablesView& tab, cudaStream_t stream, int num_sms);
// Thread-per-quartet gradient kernels for the low classes (eri_grad_small.cu): 0 when
// launched, -1 when the class is not covered (use launch_grad_block), -3 on a CUDA error.
int launch_grad_small(const QuartetBlock& blk, const double* D, int nbf, const int* shell_atom, double* grad,
                      int grad_stride, double prim_eps, const RysTablesView& tab, cudaStream_t stream, int num_sms);
bool grad_small_supported(int la, int lb, int lc, int ld);

}  // namespace lai
