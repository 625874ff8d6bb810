// Kets of the block-per-quartet gradient kernel (eri_grad_block_impl.cuh), part 7 of 9
// (compiled in parallel).
#include "eri_grad_block_impl.cuh"

namespace lai {
namespace grad_block {

template int launch_grad_range<4, 2, 0, 4>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<4, 2, 5, 5>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<4, 2, 6, 6>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);

}  // namespace grad_block
}  // namespace lai
