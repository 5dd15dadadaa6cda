// matvec_rows_w5.cu -- row-group matvec kernels on bit planes of 5 words (groups of at most 160 elements).
#include "rowkernel.cuh"

namespace lsg {
template int launch_rows_mode<5>(const MatvecProblem&, const RowsLaunch&, int, int*, const uint64_t*, cudaStream_t);
}
