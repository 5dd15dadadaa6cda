// matvec_rows_sectors.cu -- y_s = H_s x_s for many symmetry sectors in one launch of the row-group kernels
// (rowgroup.cuh, rowsums.cuh): complex128, up to 16 columns.
//
// The sectors share the group's images, the terms and the constraint; each has its own states,
// index, characters (a coefficient table per sector in shared memory) and vectors.  Work is dealt
// in blocks of consecutive rows of one sector.  Sectors with real matrix elements take the real
// sums (2 FMAs per element instead of 4).
//
// Bound by the FP64 pipe at 16 columns.  48 sectors of the 24-site XXZ chain (2.7e6 rows), 16
// columns: 11.55 ms with the warp-per-row kernel, 4.88 ms here; ~4.0 ms is the time of the
// products alone at the FP64 rate.
#include <algorithm>

#include "matvec_launch.cuh"
#include "rowsums.cuh"

namespace lsg {

template <int MODE, bool INV, bool KEEP>
__global__ void __launch_bounds__(kRowsThreads<false>, 1)
    k_matvec_rows_sectors(const MatvecProblem p, const RowsLayout L, const RowsSums sums,
                          const SectorDesc* __restrict__ sectors, int n_sectors, int64_t total_rows,
                          const double* __restrict__ xs_all, int col, int* __restrict__ err,
                          const uint64_t* __restrict__ binom) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Group = RowGroup<MODE, INV, false, KEEP>;
  SectorDesc* sd = (SectorDesc*)(smem + L.off_sectors);
  const uint64_t* src = reinterpret_cast<const uint64_t*>(sectors);
  for (int i = threadIdx.x; i < n_sectors * (int)(sizeof(SectorDesc) / 8); i += blockDim.x)
    reinterpret_cast<uint64_t*>(sd)[i] = __ldg(src + i);
  Group::stage(L, p, smem);  // synchronises the block after the copies above
  double2* coef = (double2*)(smem + L.off_coef);
  const int table = p.off.rows.n_cls * L.G;
  for (int i = threadIdx.x; i < n_sectors * table; i += blockDim.x) {
    const int s = i / table, e = i - s * table;
    const double2 v = __ldg(p.off.rows.cval + e / L.G), chi = __ldg(sd[s].chars + e % L.G);
    const C2 f = cmul_conj_b(C2{v.x, v.y}, C2{chi.x, chi.y});
    // real sectors: the first half of their table as plain doubles
    if (sd[s].real_elements) reinterpret_cast<double*>(coef + s * table)[e] = f.re;
    else coef[i] = make_double2(f.re, f.im);
  }
  int64_t* first = (int64_t*)(smem + L.off_first);  // first block of every sector
  if (threadIdx.x == 0) {
    int64_t b = 0;
    for (int s = 0; s < n_sectors; ++s) {
      first[s] = b;
      const int64_t rows = (s + 1 < n_sectors ? sd[s + 1].row_begin : total_rows) - sd[s].row_begin;
      b += (rows + sums.rows_per_block - 1) / sums.rows_per_block;
    }
    first[n_sectors] = b;
  }
  __syncthreads();
  Group g(L, p, smem);
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5, n_blocks = first[n_sectors];
  int cur = 0;
  for (int64_t b = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; b < n_blocks; b += n_warps) {
    while (b >= first[cur + 1]) ++cur;  // blocks of a warp ascend; empty sectors have none
    const SectorDesc& S = sd[cur];
    const int64_t rows = (cur + 1 < n_sectors ? sd[cur + 1].row_begin : total_rows) - S.row_begin;
    const int64_t begin = (b - first[cur]) * sums.rows_per_block, end = min(begin + sums.rows_per_block, rows);
    RowsSums s = sums;
    s.x = S.x;
    s.y = S.y;
    s.xs = xs_all + ((size_t)S.row_begin * s.ldxs + col) * 2;
    const bool real = S.real_elements != 0;
    const DeviceIndex ix = S.index;
    const double2* cz = coef + cur * table;
    g.minus = S.spin_inversion == -1;
    g.restart();
    for (int64_t row = begin; row < end; row += L.R) {
      g.load_rows(ix, row, (int)min((int64_t)L.R, end - row));
      if constexpr (KEEP) {
        g.resolve(ix, err, binom);
        if (real) sum_rows<kColPair>(g, s, reinterpret_cast<const double*>(cz), row);
        else sum_rows<kColComplex>(g, s, cz, row);
      } else {
        if (real) resolve_and_sum<kColPair>(g, s, ix, reinterpret_cast<const double*>(cz), row, err, binom);
        else resolve_and_sum<kColComplex>(g, s, ix, cz, row, err, binom);
      }
    }
  }
}

int launch_rows_sectors(const MatvecProblem& p, int k, int col, const SectorDesc* d_desc, int n_sectors,
                        int64_t total_rows, int64_t ldx, int64_t ldy, const double* xs_all, int64_t ldxs, int* d_err,
                        const uint64_t* binom, cudaStream_t st) {
  RowsLaunch q{};
  if (!rows_plan(p, kColComplex, k, total_rows, n_sectors, &q))
    return fail(LS_GPU_ERR_INVALID, "row-group tables do not fit in shared memory");
  q.s.ldx = ldx;
  q.s.ldy = ldy;
  q.s.ldxs = ldxs;
  auto go = [&](auto kern) -> int {
    if (!ensure_smem_limit((const void*)kern, q.L.total)) return LS_GPU_ERR_CUDA;
    kern<<<(unsigned)q.blocks, q.L.threads, q.L.total, st>>>(p, q.L, q.s, d_desc, n_sectors, total_rows, xs_all, col,
                                                             d_err, binom);
    return cuda_ok(cudaGetLastError(), "k_matvec_rows_sectors") ? 0 : LS_GPU_ERR_CUDA;
  };
  const bool inv = p.group.spin_inversion != 0, keep = q.s.cols > 1;
  auto with_keep = [&](auto mtag, auto itag) -> int {
    constexpr int M = decltype(mtag)::value;
    constexpr bool I = decltype(itag)::value;
    return keep ? go(k_matvec_rows_sectors<M, I, true>) : go(k_matvec_rows_sectors<M, I, false>);
  };
  auto with_inv = [&](auto mtag) -> int {
    return inv ? with_keep(mtag, std::true_type{}) : with_keep(mtag, std::false_type{});
  };
  switch (q.mode) {  // groups of at most 128 elements
    case kModeN32: return with_inv(std::integral_constant<int, kModeN32>{});
    case 2: return with_inv(std::integral_constant<int, 2>{});
    case 5: return with_inv(std::integral_constant<int, 5>{});
    default: return fail(LS_GPU_ERR_INVALID, "sector batches: at most 128 group elements");
  }
}

}  // namespace lsg
