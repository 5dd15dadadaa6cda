// matvec_rows_w16.cu -- row-group matvec kernels on bit planes of 16 words (groups of at most 512 elements).
#include "rowkernel.cuh"

namespace lsg {
template int launch_rows_mode<16>(const MatvecProblem&, const RowsLaunch&, int, int*, const uint64_t*, cudaStream_t);
}
