// matvec_rows_w9.cu -- row-group matvec kernels on bit planes of 9 words (groups of at most 288 elements).
#include "rowkernel.cuh"

namespace lsg {
template int launch_rows_mode<9>(const MatvecProblem&, const RowsLaunch&, int, int*, const uint64_t*, cudaStream_t);
}
