// Kets of the block-per-quartet kernel (eri_block_impl.cuh), part 3 of 8 (compiled in
// parallel).
#include "eri_block_impl.cuh"

namespace lai {
namespace block_detail {

template int launch_range<2, 2, 0, 4, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<2, 2, 0, 4>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<2, 2, 2, 4, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<4, 1, 4, 5, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<4, 1, 4, 5>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);

}  // namespace block_detail
}  // namespace lai
