// Dispatch of the block-per-quartet kernel (eri_block_impl.cuh) over its kets, which are
// instantiated in eri_block_k*.cu, and the choice of kernel family for the classes
// outside the thread-per-quartet set.
#include <cuda_runtime.h>

#include "eri_block_impl.cuh"

namespace lai {

// FP64: from ld = 2 on the f shells start at 0 (expansion about M, eri_block_impl.cuh)
#define LAI_BLOCK_KETS(K)                                                                              \
  K(0, 0, 0, 0) K(1, 0, 1, 1) K(1, 1, 1, 2) K(2, 0, 2, 2) K(2, 1, 2, 3) K(2, 2, 0, 4) K(3, 0, 3, 3)     \
  K(3, 1, 3, 4) K(3, 2, 0, 5) K(3, 3, 0, 6) K(4, 0, 4, 4) K(4, 1, 4, 5) K(4, 2, 0, 6)                  \
  /* more components than a thread's registers hold: two launches, each digests its part */           \
  K(4, 3, 0, 5) K(4, 3, 6, 7) K(4, 4, 0, 6) K(4, 4, 7, 8)
#define LAI_BLOCK_KETS_F32(K)                                                                          \
  K(0, 0, 0, 0) K(1, 0, 1, 1) K(1, 1, 1, 2) K(2, 0, 2, 2) K(2, 1, 2, 3) K(2, 2, 2, 4) K(3, 0, 3, 3)     \
  K(3, 1, 3, 4) K(3, 2, 3, 5) K(3, 3, 3, 6)

namespace block_detail {
#define K(c, d, f0, f1)                                                                                       \
  extern template int launch_range<c, d, f0, f1, double>(const QuartetBlock&, const JKArgs&,                  \
                                                         const RysTablesView&, cudaStream_t, int);            \
  extern template int launch_range_list<c, d, f0, f1>(int, int, int64_t, const MultiEntry*, int, int64_t,     \
                                                      const JKArgs&, const RysTablesView&, cudaStream_t, int);
LAI_BLOCK_KETS(K)
#undef K
#define K(c, d, f0, f1) \
  extern template int launch_range<c, d, f0, f1, float>(const QuartetBlock&, const JKArgs&, const RysTablesView&, \
                                                        cudaStream_t, int);
LAI_BLOCK_KETS_F32(K)
#undef K
}  // namespace block_detail

int launch_blockq_list(int la, int lb, int lc, int ld, int64_t Pmax, const MultiEntry* list, int n, int64_t nwork,
                       const JKArgs& args, const RysTablesView& tab, cudaStream_t stream, int num_sms) {
#define K(c, d, f0, f1)                                                                                        \
  if (lc == c && ld == d)                                                                                      \
    if (const int rc = block_detail::launch_range_list<c, d, f0, f1>(la, lb, Pmax, list, n, nwork, args, tab,   \
                                                                     stream, num_sms)) return rc;
  LAI_BLOCK_KETS(K)
#undef K
  return 0;
}

int launch_blockq(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab, cudaStream_t stream,
                  int num_sms, bool fp32) {
  if (args.mode != MODE_JK) return -1;
  if (blk.total - blk.t_begin <= 0) return 0;
  const int lc = blk.ket.la, ld = blk.ket.lb;
  if (fp32) {
#define K(c, d, f0, f1) \
  if (lc == c && ld == d) return block_detail::launch_range<c, d, f0, f1, float>(blk, args, tab, stream, num_sms);
    LAI_BLOCK_KETS_F32(K)
#undef K
  }
#define K(c, d, f0, f1)                                                                               \
  if (lc == c && ld == d)                                                                             \
    if (const int rc = block_detail::launch_range<c, d, f0, f1, double>(blk, args, tab, stream, num_sms)) return rc;
  LAI_BLOCK_KETS(K)
#undef K
  return 0;
}

int block_ket_chunks(int lc, int ld) { return ncart(lc) / block_detail::chunk_components(lc, ld); }

// FP32 covers the d and f classes with at most 1024 contracted (e0|f0) integrals: up to
// (dd|dd), 961.  The larger ones, from (fd|fp) with 1150 on, and the g classes run in FP64
// in a mixed-precision build.
bool block_fp32_class(int la, int lb, int lc, int ld) {
  return la <= 3 && ncart_range(la, la + lb) * ncart_range(lc, lc + ld) <= 1024;
}

// Launches of the thread-per-quartet classes with three roots or more and few quartets:
// the block kernel splits a quartet over threads and blocks, where a thread holds all its
// roots, blocks and outputs (one (pp|pp) quartet of H2O/STO-3G, 81 primitive quartets: 41 us
// by threads, 23 us by a block).  The classes below stay with the threads, which split the
// primitive quartets over lanes and warps: a block has one row there, three or six.
bool block_for_few(const QuartetBlock& blk, int num_sms) {
  return blk.bra.la + blk.bra.lb + blk.ket.la + blk.ket.lb >= 4 &&
         blk.total - blk.t_begin <= 8 * (int64_t)num_sms;
}

// The block-per-quartet kernel, except large launches of the bra-sliced classes.  Those,
// (dp|pp), (dp|dp) and (dd|ds), leave half of a block's threads without a row (16 of 32; 31
// for (dd|) and their digestion is short: one launch of (dp|pp), C2H6/cc-pVQZ, 1.3e5
// quartets of one primitive quartet, takes 0.248 ms on either kernel.  With fewer
// quartets than the device holds blocks the block kernel, which splits a quartet, takes
// them too: the same class in H2O/cc-pVQZ with 25 - 36 primitive quartets.
//
// What the block kernel replaced in the other classes was the tiled kernel (one warp per
// quartet, its table and digestion sweeps repeated for every 512 integrals) and a
// warp-per-quartet kernel with scattered (e0|f0) ownership.  Device time per class,
// C6H14/cc-pVTZ, before -> now: (fd|dp) 21.6 -> 2.7 ms, (fp|dp) 23.1 -> 3.2, (fd|dd) 10.3
// -> 1.4, (ff|fd) 8.1 -> 0.4, (dd|dp) 6.2 -> 3.8; one (gg|gg) quartet 74 ms -> 0.07 ms.
// Whole builds when it came: C6H14/cc-pVTZ 199 -> 90 ms, H2O/cc-pVQZ 120 -> 5.1 ms.
int default_kernel(int la, int lb, int lc, int ld, int64_t nq, int num_sms) {
  if (nq >= (int64_t)32 * num_sms && sliced_class_supported(la, lb, lc, ld)) return KERNEL_SLICED;
  return KERNEL_BLOCK;
}

}  // namespace lai
