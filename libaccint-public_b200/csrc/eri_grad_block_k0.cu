// Kets of the block-per-quartet gradient kernel (eri_grad_block_impl.cuh), part 1 of 9
// (compiled in parallel).
#include "eri_grad_block_impl.cuh"

namespace lai {
namespace grad_block {

template int launch_grad_range<0, 0, 0, 0>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<1, 0, 1, 1>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<2, 0, 2, 2>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<1, 1, 1, 2>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);

}  // namespace grad_block
}  // namespace lai
