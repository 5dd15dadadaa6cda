// matvec_rows.cu -- y = H x from the row-group orbit scan (rowgroup.cuh, rowsums.cuh): projected bases, real
// or complex vectors, up to 16 complex or 32 real columns per launch.
#include <algorithm>

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

// Dynamic shared memory of a row-group kernel (the coupling products keep 2.2 KB more, statically).
constexpr size_t kRowsSmem = kMaxDynamicSmem - 4096;

// Layout for `warps` warps of R rows (keep: the resolved elements are kept in shared memory); false when it exceeds the shared memory of a CTA.
static bool rows_layout(const MatvecProblem& p, int mode, bool complex_elements, bool keep, int n_sectors,
                        int warps, int R, RowsLayout* out) {
  RowsLayout L{};
  uint32_t o = 0;
  auto take = [&](size_t bytes) {
    const uint32_t at = o;
    o += (uint32_t)((bytes + 15) & ~(size_t)15);
    return at;
  };
  const DeviceRowTerms& t = p.off.rows;
  const DeviceRowTerms& d = p.diag.rows;
  const size_t state = mode == kModeN32 ? 4 : 8;  // bytes of a state word
  L.threads = 32 * warps;
  L.R = R;
  L.lanes_per_row = 32 / R;
  L.lane_shift = 31 - __builtin_clz((unsigned)L.lanes_per_row);
  L.cap = std::max(t.n_slots, 1);
  L.T = p.off.n;
  L.n_slots = t.n_slots;
  L.slot_blocks = t.slot_blocks;
  L.n_pat = t.n_pat;
  L.n_diag_blocks = d.slot_blocks;
  L.G = p.group.n_elems;
  L.words = mode == kModeN32 ? (L.G + 7) / 8 * 8 : (L.G + 15) / 16 * 8;
  L.stride = L.words + 1;  // odd: patterns (and rows) next to each other fall into different banks
  L.site_words = (L.words + 31) / 32 * 32;
  L.nlow = mode == kModeP16 ? p.group.n_bits - 16 : 0;
  const int pw = (L.nlow + 3) / 4;
  L.nlow_pad = 4 * pw;
  L.perm_stride = 4 * (pw % 2 ? pw : pw + 1);
  // a table beyond the shared memory of a CTA cannot fit (and would overflow the 32-bit offsets)
  const size_t big = (size_t)L.n_pat * L.stride * 4 + (size_t)t.n_cls * L.G * 16 * std::max(n_sectors, 1) +
                     (size_t)R * L.cap * 10;
  if (big > kMaxDynamicSmem || (size_t)p.off.n * 64 > 4 * kMaxDynamicSmem || (size_t)R * L.cap > 65535) {
    *out = L;  // warp_bytes 0
    return false;
  }
  L.off_coef = take((size_t)t.n_cls * L.G * (complex_elements ? 16 : 8) * std::max(n_sectors, 1));
  L.off_site = take((size_t)p.group.n_bits * L.site_words * 4);
  L.off_img = take((size_t)L.n_pat * L.stride * 4);
  L.off_perm = take(mode == kModeP16 ? (size_t)L.G * L.perm_stride : 0);
  L.off_sm = take((size_t)32 * L.slot_blocks * state);
  L.off_sl1 = take((size_t)32 * L.slot_blocks * state);
  L.off_sl2 = take((size_t)32 * L.slot_blocks * state);
  L.off_st = take((size_t)32 * L.slot_blocks * 4);
  L.off_ti = take((size_t)L.T * 4);
  L.off_ts = take((size_t)L.T * state);
  L.off_xm = take((size_t)L.n_pat * state);
  L.off_dm = take((size_t)32 * L.n_diag_blocks * state);
  L.off_dr = take((size_t)32 * L.n_diag_blocks * state);
  L.off_ds = take((size_t)32 * L.n_diag_blocks * state);
  L.off_db = take((size_t)L.n_diag_blocks * 8);
  L.off_dv = take((size_t)d.n_cls * 16);
  L.off_fs = take(p.group.fermionic ? (size_t)p.group.n_bits * 32 * p.group.gpl * state : 0);
  L.off_sectors = take((size_t)n_sectors * sizeof(SectorDesc));
  L.off_first = take(n_sectors > 0 ? (size_t)(n_sectors + 1) * 8 : 0);
  L.off_warp = o;
  o = 0;
  take((size_t)R * L.stride * 4);
  L.w_list = take((size_t)R * L.cap * 2);
  L.w_ent = take(keep ? (size_t)R * L.cap * 8 : 0);
  L.w_a = take((size_t)R * state);
  L.warp_bytes = o;
  L.total = L.off_warp + (uint32_t)warps * L.warp_bytes;
  *out = L;
  return L.total <= kRowsSmem;
}

// Modes that `p` can run in order of preference: N32 where the state fits 32 bits (whole states, no
// second comparison), else, or when its pattern images do not fit, P16 (half the table, two
// elements per word; at most 32 chunks of 16 elements in the scan's mask).
static bool rows_mode_allowed(const MatvecProblem& p, int mode) {
  const int n = p.group.n_bits;
  if (p.group.n_elems < 1 || !p.off.rows.ok || !p.diag.rows.ok) return false;
  if (p.group.fermionic && (p.group.gpl < 1 || p.group.gpl > 4)) return false;  // as the packed kernels
  return mode == kModeN32 ? n <= 32 : n >= 17 && n <= 63 && p.group.n_elems <= 512;
}

constexpr int kLeastWarps = 4;

bool rows_fit(const MatvecProblem& p, int n_sectors) {
  RowsLayout L;
  if (p.projection != 2) return false;
  for (const int m : {kModeN32, kModeP16})
    if (rows_mode_allowed(p, m) && rows_layout(p, m, n_sectors > 0 || p.real_elements == 0, true, n_sectors, kLeastWarps, 1, &L)) return true;
  return false;
}

// Shape for p (rows_fit): the cheapest number of rows per warp among those that leave enough warps
// their area.
static bool rows_shape(const MatvecProblem& p, bool complex_elements, bool keep, int64_t n_rows, int n_sectors,
                       int max_warps, int sms, int* mode, RowsLayout* L) {
  for (const int m : {kModeN32, kModeP16}) {
    if (!rows_mode_allowed(p, m)) continue;
    RowsLayout t[4];
    int warps[4];
    for (int i = 0; i < 4; ++i) {
      rows_layout(p, m, complex_elements, keep, n_sectors, 1, 8 >> i, &t[i]);
      const int64_t room = (int64_t)kRowsSmem - t[i].off_warp;
      warps[i] = t[i].warp_bytes == 0 || room < 0 ? 0 : (int)std::min<int64_t>(max_warps, room / t[i].warp_bytes);
    }
    for (const int enough : {24, 16, 8, kLeastWarps}) {
      int pick = -1;
      double least = 0.0;
      for (int i = 0; i < 4; ++i) {
        if (warps[i] < std::min(enough, max_warps) || warps[i] < 1) continue;
        // rounds of row groups over all warps x steps of a group: images and lists row by row, the
        // scan of 64 elements (about half the slots match) over all words
        const int64_t R = 8 >> i, all = (int64_t)sms * warps[i], groups = (n_rows + R - 1) / R;
        const double scans = (double)((t[i].n_slots * R / 2 + 63) / 64) * (2.0 + t[i].words / 16.0);
        const double cost = (double)((groups + all - 1) / all) * (4.0 + (double)R + scans);
        if (pick < 0 || cost < least) {
          pick = i;
          least = cost;
        }
      }
      if (pick < 0) continue;
      *mode = m;
      return rows_layout(p, m, complex_elements, keep, n_sectors, warps[pick], 8 >> pick, L);
    }
  }
  return false;
}

void rows_launch_config(int* max_threads, int* waves);

bool rows_plan(const MatvecProblem& p, int col, int k, int64_t n_rows, int n_sectors, RowsLaunch* out,
               int most_threads) {
  const int units = col == kColPair && out->s.real_cols ? (k + 1) / 2 : k;  // columns of the lanes
  const bool keep = units > 1, complex_elements = n_sectors > 0 || col == kColComplex;
  // (the batched kernel holds the sector's description in registers, too)
  int max_threads = keep && n_sectors == 0 ? kRowsThreads<true> : kRowsThreads<false>, waves = 1;
  if (most_threads > 0) max_threads = most_threads;
  else rows_launch_config(&max_threads, &waves);
  const int sms = num_sms();
  RowsLayout& L = out->L;
  if (!rows_shape(p, complex_elements, keep, n_rows, n_sectors, max_threads / 32, sms, &out->mode, &L)) return false;
  int warps = L.threads / 32;
  // few rows: one group of rows per warp, the warps spread over the SMs
  const int64_t groups = (n_rows + L.R - 1) / L.R;
  const int64_t per_sm = std::max<int64_t>(kLeastWarps, (groups + sms - 1) / sms);
  if (per_sm < warps) {
    warps = (int)per_sm;
    if (!rows_layout(p, out->mode, complex_elements, keep, n_sectors, warps, L.R, &L)) return false;
  }
  RowsSums& s = out->s;
  s.cols = units;
  s.rp = std::max(1, std::min(L.R, 32 / s.cols));
  s.q = 1;
  while (2 * s.q * s.rp * s.cols <= 32) s.q *= 2;
  // rows of one warp: consecutive (the images follow from row to row), enough blocks to balance
  const int64_t total_warps = (int64_t)sms * warps * waves;
  s.rows_per_block = std::max<int64_t>(L.R, std::min<int64_t>(64, n_rows / (16 * total_warps) / L.R * L.R));
  s.n_blocks = (n_rows + s.rows_per_block - 1) / s.rows_per_block;
  out->blocks = std::max<int64_t>(1, std::min<int64_t>((s.n_blocks + warps - 1) / warps, (int64_t)sms * waves));
  return true;
}

int launch_rows(const MatvecProblem& p, Scalar sc, int k, const double* d_x, int64_t ldx, double* d_y, int64_t ldy,
                int* d_err, const uint64_t* binom, cudaStream_t st) {
  const bool cplx = sc == Scalar::Complex;
  const int col = cplx ? (p.real_elements ? kColPair : kColComplex) : (k == 1 ? kColReal : kColPair);
  RowsLaunch q{};
  RowsSums& s = q.s;
  s.real_cols = (!cplx && col == kColPair) ? k : 0;
  if (!rows_plan(p, col, k, p.n_rows, 0, &q))
    return fail(LS_GPU_ERR_INVALID, "row-group tables do not fit in shared memory");
  s.x = d_x;
  s.xs = p.xs != nullptr ? p.xs : d_x;
  s.norms = p.xs != nullptr ? nullptr : p.index.norms;
  s.y = d_y;
  s.ldx = ldx;
  s.ldxs = p.xs != nullptr ? p.ldxs : ldx;
  s.ldy = ldy;
  const RowsLayout& L = q.L;
  const bool keep = s.cols > 1;
  auto go = [&](auto kern) -> int {
    if (!ensure_smem_limit((const void*)kern, L.total)) return LS_GPU_ERR_CUDA;
    kern<<<(unsigned)q.blocks, L.threads, L.total, st>>>(p, L, s, d_err, binom);
    return cuda_ok(cudaGetLastError(), "k_matvec_rows") ? 0 : LS_GPU_ERR_CUDA;
  };
  const bool inv = p.group.spin_inversion != 0;
  auto with_col = [&](auto mtag, auto itag, auto ftag) -> int {
    constexpr int M = decltype(mtag)::value;
    constexpr bool I = decltype(itag)::value, F = decltype(ftag)::value;
    if (col == kColReal) return go(k_matvec_rows<M, I, F, kColReal, false>);
    if (col == kColPair)
      return keep ? go(k_matvec_rows<M, I, F, kColPair, true>) : go(k_matvec_rows<M, I, F, kColPair, false>);
    return keep ? go(k_matvec_rows<M, I, F, kColComplex, true>) : go(k_matvec_rows<M, I, F, kColComplex, false>);
  };
  auto with_mode = [&](auto mtag) -> int {
    if (p.group.fermionic) {
      if (inv) return fail(LS_GPU_ERR_INVALID, "fermionic groups have no spin inversion");
      return with_col(mtag, std::false_type{}, std::true_type{});
    }
    return inv ? with_col(mtag, std::true_type{}, std::false_type{})
               : with_col(mtag, std::false_type{}, std::false_type{});
  };
  return q.mode == kModeN32 ? with_mode(std::integral_constant<int, kModeN32>{})
                          : with_mode(std::integral_constant<int, kModeP16>{});
}

}  // namespace lsg
