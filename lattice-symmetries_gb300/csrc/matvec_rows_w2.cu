// matvec_rows_w2.cu -- row-group matvec kernels on bit planes of 2 words (groups of at most 64 elements).
#include "rowkernel.cuh"

namespace lsg {
template int launch_rows_mode<2>(const MatvecProblem&, const RowsLaunch&, int, int*, const uint64_t*, cudaStream_t);
}
