// Dispatch of the block-per-quartet gradient kernel (eri_grad_block_impl.cuh) over its
// kets, which are instantiated in eri_grad_block_k*.cu; the larger kets take several
// launches, each with a range of f shells.
#include "eri_grad_block_impl.cuh"

namespace lai {
namespace grad_block {
#define LAI_GRAD_KETS(K) \
  K(0, 0, 0, 0) K(1, 0, 1, 1) K(1, 1, 1, 2) K(2, 0, 2, 2) K(2, 1, 2, 3) K(2, 2, 0, 4) K(3, 0, 3, 3) \
  K(3, 1, 3, 4) K(3, 2, 0, 4) K(3, 2, 5, 5) K(3, 3, 0, 4) K(3, 3, 5, 5) K(3, 3, 6, 6) K(4, 0, 4, 4) \
  K(4, 1, 4, 5) K(4, 2, 0, 4) K(4, 2, 5, 5) K(4, 2, 6, 6) K(4, 3, 4, 5) K(4, 3, 6, 6) K(4, 3, 7, 7) \
  K(4, 4, 4, 5) K(4, 4, 6, 6) K(4, 4, 7, 7) K(4, 4, 8, 8)
#define K(c, d, f0, f1)                                                                                    \
  extern template int launch_grad_range<c, d, f0, f1>(const QuartetBlock&, const GradBlockArgs&,          \
                                                      const RysTablesView&, cudaStream_t, int);
LAI_GRAD_KETS(K)
#undef K
}  // namespace grad_block

int launch_grad_block(const QuartetBlock& blk, const double* D, int nbf, const int* shell_atom, double* grad,
                      int grad_stride, double prim_eps, const RysTablesView& tab, cudaStream_t stream, int num_sms) {
  if (blk.total - blk.t_begin <= 0) return 0;
  const int lc = blk.ket.la, ld = blk.ket.lb;
  const grad_block::GradBlockArgs ga{D, nbf, shell_atom, grad, grad_stride, prim_eps};
#define K(c, d, f0, f1)    \
  if (lc == c && ld == d)  \
    if (const int rc = grad_block::launch_grad_range<c, d, f0, f1>(blk, ga, tab, stream, num_sms)) return rc;
  LAI_GRAD_KETS(K)
#undef K
  return 0;
}

}  // namespace lai
