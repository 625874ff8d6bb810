// Kets of the block-per-quartet kernel (eri_block_impl.cuh), part 4 of 8 (compiled in
// parallel).
#include "eri_block_impl.cuh"

namespace lai {
namespace block_detail {

template int launch_range<3, 2, 0, 5, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<3, 2, 0, 5>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<3, 2, 3, 5, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);

}  // namespace block_detail
}  // namespace lai
