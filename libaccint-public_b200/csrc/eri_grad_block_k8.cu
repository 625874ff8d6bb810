// Kets of the block-per-quartet gradient kernel (eri_grad_block_impl.cuh), part 9 of 9
// (compiled in parallel).
#include "eri_grad_block_impl.cuh"

namespace lai {
namespace grad_block {

template int launch_grad_range<4, 4, 4, 5>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<4, 4, 6, 6>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<4, 4, 7, 7>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);
template int launch_grad_range<4, 4, 8, 8>(const QuartetBlock&, const GradBlockArgs&,
                                           const RysTablesView&, cudaStream_t, int);

}  // namespace grad_block
}  // namespace lai
