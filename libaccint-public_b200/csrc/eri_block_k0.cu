// Kets of the block-per-quartet kernel (eri_block_impl.cuh), part 1 of 8 (compiled in
// parallel).
#include "eri_block_impl.cuh"

namespace lai {
namespace block_detail {

template int launch_range<0, 0, 0, 0, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<0, 0, 0, 0>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<0, 0, 0, 0, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<1, 0, 1, 1, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<1, 0, 1, 1>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<1, 0, 1, 1, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<2, 0, 2, 2, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<2, 0, 2, 2>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<2, 0, 2, 2, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<3, 0, 3, 3, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<3, 0, 3, 3>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<3, 0, 3, 3, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range<4, 0, 4, 4, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<4, 0, 4, 4>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<1, 1, 1, 2, double>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);
template int launch_range_list<1, 1, 1, 2>(int, int, int64_t, const MultiEntry*, int, int64_t,
                                          const JKArgs&, const RysTablesView&, cudaStream_t, int);
template int launch_range<1, 1, 1, 2, float>(const QuartetBlock&, const JKArgs&,
                                             const RysTablesView&, cudaStream_t, int);

}  // namespace block_detail
}  // namespace lai
