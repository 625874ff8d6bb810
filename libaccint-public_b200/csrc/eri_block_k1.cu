// Kets of the block-per-quartet kernel (eri_block_impl.cuh), part 2 of 8 (compiled in
// parallel).
#include "eri_block_impl.cuh"

namespace lai {
namespace block_detail {

template int launch_range<2, 1, 2, 3, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<2, 1, 2, 3, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<3, 1, 3, 4, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<3, 1, 3, 4, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);

}  // namespace block_detail
}  // namespace lai
