// rowkernel.cuh -- the row-group matvec kernel and its launcher for one scan mode (instantiated by
// matvec_rows.cu and matvec_rows_w*.cu, so that the modes compile in parallel).
#pragma once

#include "matvec_launch.cuh"
#include "rowsums.cuh"

namespace lsg {

template <int MODE, bool INV, bool FERMI, int COL, bool KEEP>
__global__ void __launch_bounds__(kRowsThreads<KEEP>, 1)
    k_matvec_rows(const MatvecProblem p, const RowsLayout L, const RowsSums s, int* __restrict__ err,
                  const uint64_t* __restrict__ binom) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Group = RowGroup<MODE, INV, FERMI, KEEP>;
  Group::stage(L, p, smem);
  auto* coef = reinterpret_cast<typename Column<COL>::C*>(smem + L.off_coef);
  stage_coefficients<COL>(L, p.off.rows, p.group.chars, coef);
  __syncthreads();
  Group g(L, p, smem);
  // blocks of rows are dealt across the CTAs first: a last round that does not fill the grid
  // leaves a few warps on every SM instead of whole SMs without work (28-site chain, 16 columns:
  // the busiest SM had 17 % more FP64 work than the mean)
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t b = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; b < s.n_blocks; b += n_warps) {
    const int64_t begin = b * s.rows_per_block, end = min(begin + s.rows_per_block, p.n_rows);
    g.restart();
    for (int64_t row = begin; row < end; row += L.R) {
      g.load_rows(p.index, row, (int)min((int64_t)L.R, end - row));
      if constexpr (KEEP) {
        g.resolve(p.index, err, binom);
        sum_rows<COL>(g, s, coef, row);
      } else {
        resolve_and_sum<COL>(g, s, p.index, coef, row, err, binom);
      }
    }
  }
}

template <int MODE>
int launch_rows_mode(const MatvecProblem& p, const RowsLaunch& q, int col, int* d_err, const uint64_t* binom,
                     cudaStream_t st) {
  auto go = [&](auto kern) -> int {
    if (!ensure_smem_limit((const void*)kern, q.L.total)) return LS_GPU_ERR_CUDA;
    kern<<<(unsigned)q.blocks, q.L.threads, q.L.total, st>>>(p, q.L, q.s, d_err, binom);
    return cuda_ok(cudaGetLastError(), "k_matvec_rows") ? 0 : LS_GPU_ERR_CUDA;
  };
  const bool keep = q.s.cols > 1;
  auto with_col = [&](auto itag, auto ftag) -> int {
    constexpr bool I = decltype(itag)::value, F = decltype(ftag)::value;
    if (col == kColReal) return go(k_matvec_rows<MODE, I, F, kColReal, false>);
    if (col == kColPair)
      return keep ? go(k_matvec_rows<MODE, I, F, kColPair, true>) : go(k_matvec_rows<MODE, I, F, kColPair, false>);
    return keep ? go(k_matvec_rows<MODE, I, F, kColComplex, true>) : go(k_matvec_rows<MODE, I, F, kColComplex, false>);
  };
  const bool inv = p.group.spin_inversion != 0;
  if (p.group.fermionic) {
    if (inv) return fail(LS_GPU_ERR_INVALID, "fermionic groups have no spin inversion");
    if constexpr (MODE <= 5) return with_col(std::false_type{}, std::true_type{});
    return fail(LS_GPU_ERR_INVALID, "fermionic lattice symmetries: at most 128 group elements");
  }
  return inv ? with_col(std::true_type{}, std::false_type{}) : with_col(std::false_type{}, std::false_type{});
}

}  // namespace lsg
