// Dispatch of the thread-per-quartet small-class kernels (eri_small_impl.cuh);
// the kernels themselves are instantiated in eri_small_i*.cu.
#include <cuda_runtime.h>

#include "eri_kernels.h"

namespace lai {
namespace small_detail {
template <int LA, int LB, int LC, int LD>
int launch_one(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab,
               cudaStream_t stream, bool fp32, int num_sms, LaunchTune tune);
template <int LA, int LB, int LC, int LD>
int launch_list(const MultiEntry* list, int n, int64_t nwork, const JKArgs& args, const RysTablesView& tab,
                cudaStream_t stream, int num_sms);
}  // namespace small_detail

// Up to some 90 contracted (e0|f0) integrals a thread per quartet is faster than a block,
// even where ptxas spills a part of them (C6H14/cc-pVTZ, block -> thread: (fp|ps) 5.1 -> 1.7
// ms with 1.3 KB of spills, (fs|ds) 5.6 -> 1.6, (fs|pp) 3.6 -> 1.7, (fd|ss) 2.2 -> 0.5); from
// 138 on ((fd|ps), (dp|pp), (fp|ds), (fs|dp)) it is 3 to 7 times slower.
#define LAI_SMALL_CLASSES(X) \
  X(0, 0, 0, 0) X(1, 0, 0, 0) X(1, 0, 1, 0) X(1, 1, 0, 0) X(1, 1, 1, 0) X(2, 0, 0, 0) \
  X(2, 0, 1, 0) X(2, 0, 2, 0) X(2, 1, 0, 0) X(2, 2, 0, 0) X(3, 0, 0, 0) X(3, 0, 1, 0)   \
  X(3, 1, 0, 0) X(4, 0, 0, 0) X(1, 1, 1, 1) X(2, 0, 1, 1) X(2, 1, 1, 0) X(2, 1, 2, 0) X(2, 2, 1, 0) \
  X(3, 0, 1, 1) X(3, 0, 2, 0) X(3, 1, 1, 0) X(3, 2, 0, 0) X(4, 0, 1, 0) X(4, 1, 0, 0)

bool small_class_supported(int la, int lb, int lc, int ld) {
#define X(a, b, c, d) if (la == a && lb == b && lc == c && ld == d) return true;
  LAI_SMALL_CLASSES(X)
#undef X
  return false;
}

int launch_small(const QuartetBlock& blk, const JKArgs& args, const RysTablesView& tab,
                 cudaStream_t stream, bool fp32, int num_sms, LaunchTune tune) {
  const int la = blk.bra.la, lb = blk.bra.lb, lc = blk.ket.la, ld = blk.ket.lb;
#define X(a, b, c, d) \
  if (la == a && lb == b && lc == c && ld == d) return small_detail::launch_one<a, b, c, d>(blk, args, tab, stream, fp32, num_sms, tune);
  LAI_SMALL_CLASSES(X)
#undef X
  return 0;
}

int launch_small_list(int la, int lb, int lc, int ld, const MultiEntry* list, int n, int64_t nwork,
                      const JKArgs& args, const RysTablesView& tab, cudaStream_t stream, int num_sms) {
#define X(a, b, c, d) \
  if (la == a && lb == b && lc == c && ld == d) return small_detail::launch_list<a, b, c, d>(list, n, nwork, args, tab, stream, num_sms);
  LAI_SMALL_CLASSES(X)
#undef X
  return 0;
}

}  // namespace lai
