// matvec_rows.cu -- y = H x from the row-group orbit scan (rowgroup.cuh): projected bases, real or
// complex vectors, up to 16 complex or 32 real columns per launch, FP64 multiply-adds.
//
// Sums.  A row's resolved elements are {column index j, coefficient word}; the coefficient
// v conj(chi_g) comes from a shared-memory table over (class of v, group element) and its sign from
// the word's top bit, so that forming it costs no FP64 instruction.  The lanes of a warp are split
// into `rp` rows x `q` elements x `cols` columns; q = 1 (no cross-lane sum) from 4 columns on.
// The norms are folded in through the gather source x_j n_j and one multiplication by 1 / n_i
// per output, the diagonal element is a class count times the class value: per row and column the
// FP64 pipe sees little more than the products themselves (2 FMAs per element for real
// elements, 4 for complex ones).  GB300's FP64 pipe (2 lanes per clock and SM) bounds blocks of 16
// columns on small groups; the scan bounds single vectors.
#include <algorithm>

#include "matvec_launch.cuh"
#include "rowgroup.cuh"

namespace lsg {

// Columns of a launch: real scalars, real elements times complex columns (or pairs of real
// columns), complex elements times complex columns.
constexpr int kColReal = 0, kColPair = 1, kColComplex = 2;

struct RowsSums {
  const double* x;   // the caller's vectors (diagonal), leading dimension ldx in scalars
  const double* xs;  // x_j n_j, leading dimension ldxs in scalars
  double* y;
  int64_t ldx, ldxs, ldy;
  int64_t rows_per_block, n_blocks;  // consecutive rows of one warp
  int cols, q, rp;                   // lanes: column + cols * (element + q * row)
  int real_cols;                     // real vectors: number of real columns (pairs), else 0
};

template <int COL>
struct Column;
template <>
struct Column<kColReal> {
  using V = double;
  using C = double;
  __device__ __forceinline__ static void mac(double& a, double c, double x) { a += c * x; }
  __device__ __forceinline__ static double zero() { return 0.0; }
};
template <>
struct Column<kColPair> {
  using V = double2;
  using C = double;
  __device__ __forceinline__ static void mac(double2& a, double c, double2 x) {
    a.x += c * x.x;
    a.y += c * x.y;
  }
  __device__ __forceinline__ static double2 zero() { return make_double2(0.0, 0.0); }
};
template <>
struct Column<kColComplex> {
  using V = double2;
  using C = double2;
  __device__ __forceinline__ static void mac(double2& a, double2 c, double2 x) {
    a.x += c.x * x.x;
    a.y += c.x * x.y;
    a.x -= c.y * x.y;
    a.y += c.y * x.x;
  }
  __device__ __forceinline__ static double2 zero() { return make_double2(0.0, 0.0); }
};

__device__ __forceinline__ double flip_sign(double v, uint32_t sign) {
  return __hiloint2double(__double2hiint(v) ^ (int)sign, __double2loint(v));
}
__device__ __forceinline__ double2 flip_sign(double2 v, uint32_t sign) {
  return make_double2(flip_sign(v.x, sign), flip_sign(v.y, sign));
}
__device__ __forceinline__ double shfl_down_v(double v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }
__device__ __forceinline__ double2 shfl_down_v(double2 v, int d) {
  return make_double2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double add_v(double a, double b) { return a + b; }
__device__ __forceinline__ double2 add_v(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// Step 4: sums of the group's resolved rows.
template <int COL, typename Group>
__device__ __forceinline__ void sum_rows(const Group& g, const RowsSums& s, int64_t row0) {
  using Col = Column<COL>;
  using V = typename Col::V;
  using C = typename Col::C;
  constexpr unsigned FULL = 0xffffffffu;
  const RowsLayout& L = g.L;
  const int lane = g.lane;
  const int c = lane % s.cols, rest = lane / s.cols;
  const int q = rest & (s.q - 1), rl = rest / s.q;
  const bool active = rl < s.rp;
  const C* coef = g.template tab<C>(L.off_coef);
  const V* __restrict__ xs = reinterpret_cast<const V*>(s.xs) + c;
  const int64_t ldv = COL == kColReal ? s.ldxs : (s.real_cols ? s.ldxs / 2 : s.ldxs);
  const double2 diag = g.diagonal();
  for (int r0 = 0; r0 < g.nr; r0 += s.rp) {
    const int r = r0 + rl;
    const bool act = active && r < g.nr;
    const int rr = act ? r : 0;
    const int cnt = __shfl_sync(FULL, g.cnt_l, rr);
    const int n = act ? cnt : 0;
    const int steps = (int)__reduce_max_sync(FULL, (unsigned)(n + s.q - 1)) / s.q;
    const uint2* e = g.entries + rr * L.cap + q;
    V acc = Col::zero();
    for (int i = 0; i < steps; i += 4) {
      uint2 w[4];
      V xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int at = (i + u) * s.q;
        w[u] = at + q < n ? e[at] : make_uint2(Group::kAbsent, 0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = w[u].x != Group::kAbsent ? __ldg(xs + (int64_t)w[u].x * ldv) : Col::zero();
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (w[u].x != Group::kAbsent) Col::mac(acc, flip_sign(coef[w[u].y & 0x7fffffffu], w[u].y & 0x80000000u), xv[u]);
    }
    for (int d = s.q / 2; d > 0; d >>= 1) acc = add_v(acc, shfl_down_v(acc, d * s.cols));
    const double inv = __shfl_sync(FULL, g.inv_l, rr);
    const double dre = __shfl_sync(FULL, diag.x, rr);
    const double dim = COL == kColReal ? 0.0 : __shfl_sync(FULL, diag.y, rr);
    if (act && q == 0) {
      const int64_t row = row0 + r;
      if constexpr (COL == kColReal) {
        s.y[row * s.ldy] = inv == 0.0 ? 0.0 : acc * inv + dre * __ldg(s.x + row * s.ldx);
      } else {
        if (s.real_cols) {
          const int c0 = 2 * c;
          s.y[row * s.ldy + c0] = inv == 0.0 ? 0.0 : acc.x * inv + dre * __ldg(s.x + row * s.ldx + c0);
          if (c0 + 1 < s.real_cols)
            s.y[row * s.ldy + c0 + 1] = inv == 0.0 ? 0.0 : acc.y * inv + dre * __ldg(s.x + row * s.ldx + c0 + 1);
        } else {
          const double2 xi = __ldg(reinterpret_cast<const double2*>(s.x) + row * s.ldx + c);
          double2 out = make_double2(0.0, 0.0);
          if (inv != 0.0) {
            out.x = acc.x * inv + dre * xi.x;
            out.y = acc.y * inv + dre * xi.y;
            if (dim != 0.0) {
              out.x -= dim * xi.y;
              out.y += dim * xi.x;
            }
          }
          reinterpret_cast<double2*>(s.y)[row * s.ldy + c] = out;
        }
      }
    }
  }
}

// Coefficient table v conj(chi) over (class, element); chars in element order.
template <int COL>
__device__ __forceinline__ void stage_coefficients(const RowsLayout& L, const DeviceRowTerms& t, const double2* chars,
                                                   unsigned char* smem) {
  for (int i = threadIdx.x; i < t.n_cls * L.G; i += blockDim.x) {
    const double2 v = __ldg(t.cval + i / L.G), chi = __ldg(chars + i % L.G);
    const C2 f = cmul_conj_b(C2{v.x, v.y}, C2{chi.x, chi.y});
    if constexpr (COL == kColComplex) reinterpret_cast<double2*>(smem + L.off_coef)[i] = make_double2(f.re, f.im);
    else reinterpret_cast<double*>(smem + L.off_coef)[i] = f.re;
  }
}

template <int MODE, bool INV, bool FERMI, int COL>
__global__ void __launch_bounds__(1024, 1)
    k_matvec_rows(const MatvecProblem p, const RowsLayout L, const RowsSums s, int* __restrict__ err,
                  const uint64_t* __restrict__ binom) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Group = RowGroup<MODE, INV, FERMI>;
  Group::stage(L, p, smem);
  stage_coefficients<COL>(L, p.off.rows, p.group.chars, smem);
  __syncthreads();
  Group g(L, p, smem);
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < s.n_blocks; b += n_warps) {
    const int64_t begin = b * s.rows_per_block, end = min(begin + s.rows_per_block, p.n_rows);
    g.restart();
    for (int64_t row = begin; row < end; row += L.R) {
      const int total = g.load_rows(p.index, row, (int)min((int64_t)L.R, end - row));
      g.resolve(p.index, total, err, binom);
      sum_rows<COL>(g, s, row);
    }
  }
}

// Layout for `warps` warps of R rows; false when it exceeds the shared memory of a CTA.
static bool rows_layout(const MatvecProblem& p, int mode, bool complex_elements, int warps, int R, RowsLayout* out) {
  RowsLayout L{};
  uint32_t o = 0;
  auto take = [&](size_t bytes) {
    const uint32_t at = o;
    o += (uint32_t)((bytes + 15) & ~(size_t)15);
    return at;
  };
  const DeviceRowTerms& t = p.off.rows;
  const DeviceRowTerms& d = p.diag.rows;
  L.threads = 32 * warps;
  L.R = R;
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
  L.perm_stride = 4 * (pw % 2 ? pw : pw + 1);
  // a table beyond the shared memory of a CTA cannot fit (and would overflow the 32-bit offsets)
  const size_t big = (size_t)L.n_pat * L.stride * 4 + (size_t)t.n_cls * L.G * 16 + (size_t)R * L.cap * 10;
  if (big > kMaxDynamicSmem || (size_t)p.off.n * 64 > 4 * kMaxDynamicSmem || (size_t)R * L.cap > 65535) return false;
  L.off_coef = take((size_t)t.n_cls * L.G * (complex_elements ? 16 : 8));
  L.off_site = take((size_t)p.group.n_bits * L.site_words * 4);
  L.off_img = take((size_t)L.n_pat * L.stride * 4);
  L.off_perm = take(mode == kModeP16 ? (size_t)L.G * L.perm_stride : 0);
  L.off_sm = take((size_t)32 * L.slot_blocks * 8);
  L.off_sl1 = take((size_t)32 * L.slot_blocks * 8);
  L.off_sl2 = take((size_t)32 * L.slot_blocks * 8);
  L.off_st = take((size_t)32 * L.slot_blocks * 4);
  L.off_ti = take((size_t)L.T * 4);
  L.off_ts = take((size_t)L.T * 8);
  L.off_xm = take((size_t)L.n_pat * 8);
  L.off_dm = take((size_t)32 * L.n_diag_blocks * 8);
  L.off_dr = take((size_t)32 * L.n_diag_blocks * 8);
  L.off_ds = take((size_t)32 * L.n_diag_blocks * 8);
  L.off_db = take((size_t)L.n_diag_blocks * 8);
  L.off_dv = take((size_t)d.n_cls * 16);
  L.off_fs = take(p.group.fermionic ? (size_t)p.group.n_bits * 32 * p.group.gpl * 8 : 0);
  L.off_warp = o;
  o = 0;
  take((size_t)R * L.stride * 4);
  L.w_ent = take((size_t)R * L.cap * 8);
  L.w_ord = take((size_t)R * L.cap * 2);
  L.w_a = take((size_t)R * 8);
  L.warp_bytes = o;
  L.total = L.off_warp + (uint32_t)warps * L.warp_bytes;
  *out = L;
  return L.total <= kMaxDynamicSmem;
}

// Mode and shape: N32 where the state fits and the group is small, P16 otherwise (half the loads
// and minima per element, a second look at the winners); then as many warps as fit, with as many
// rows each as leave all of them room.
static bool rows_shape(const MatvecProblem& p, bool complex_elements, int max_warps, int64_t warps_wanted, int* mode,
                       RowsLayout* L) {
  const int n = p.group.n_bits;
  if (n > 63 || p.group.n_elems < 1 || !p.off.rows.ok || !p.diag.rows.ok) return false;
  if (p.group.fermionic && (p.group.gpl < 1 || p.group.gpl > 4)) return false;  // as the packed kernels
  for (const int m : {kModeN32, kModeP16}) {
    if (m == kModeN32 && n > 32) continue;
    if (m == kModeP16 && n < 17) continue;
    if (m == kModeP16 && p.group.n_elems > 512) continue;  // 32 chunks of 16 elements in the scan's mask
    for (const int least : {24, 16, 8, 4}) {
      if (least > max_warps && least != 4) continue;
      for (const int R : {8, 4, 2, 1}) {
        int warps = max_warps;
        while (warps > 1 && !rows_layout(p, m, complex_elements, warps, R, L)) --warps;
        if (!rows_layout(p, m, complex_elements, warps, R, L)) continue;
        if (warps < std::min(least, max_warps)) continue;
        // few rows: fewer per warp, so that all SMs have some
        int rows = R;
        while (rows > 1 && (p.n_rows + rows - 1) / rows < warps_wanted) rows /= 2;
        if (rows != R && !rows_layout(p, m, complex_elements, warps, rows, L)) continue;
        *mode = m;
        return true;
      }
    }
  }
  return false;
}

bool rows_fit(const MatvecProblem& p) {
  RowsLayout L{};
  int mode = 0;
  return p.projection == 2 && rows_shape(p, p.real_elements == 0, 32, 1, &mode, &L);
}

void rows_launch_config(int* max_threads, int* waves);

int launch_rows(const MatvecProblem& p, Scalar sc, int k, const double* d_x, int64_t ldx, double* d_y, int64_t ldy,
                int* d_err, const uint64_t* binom, cudaStream_t st) {
  const bool cplx = sc == Scalar::Complex;
  const int col = cplx ? (p.real_elements ? kColPair : kColComplex) : (k == 1 ? kColReal : kColPair);
  int max_threads = 1024, waves = 1;
  rows_launch_config(&max_threads, &waves);
  const int sms = num_sms();
  RowsLayout L{};
  int mode = 0;
  if (!rows_shape(p, col == kColComplex, max_threads / 32, (int64_t)sms * 16, &mode, &L))
    return fail(LS_GPU_ERR_INVALID, "row-group tables do not fit in shared memory");
  int warps = L.threads / 32;
  // few rows: one group of rows per warp, the warps spread over the SMs
  const int64_t groups = (p.n_rows + L.R - 1) / L.R;
  const int64_t per_sm = std::max<int64_t>(4, (groups + sms - 1) / sms);
  if (per_sm < warps) {
    warps = (int)per_sm;
    if (!rows_layout(p, mode, col == kColComplex, warps, L.R, &L)) return LS_GPU_ERR_INVALID;
  }
  RowsSums s{};
  s.x = d_x;
  s.xs = p.xs;
  s.y = d_y;
  s.ldx = ldx;
  s.ldxs = p.ldxs;
  s.ldy = ldy;
  s.real_cols = (!cplx && col == kColPair) ? k : 0;
  s.cols = s.real_cols ? (k + 1) / 2 : k;
  s.rp = std::max(1, std::min(L.R, 32 / s.cols));
  s.q = 1;
  while (2 * s.q * s.rp * s.cols <= 32) s.q *= 2;
  // rows of one warp: consecutive (the images follow from row to row), enough blocks to balance
  const int64_t total_warps = (int64_t)sms * warps * waves;
  s.rows_per_block = std::max<int64_t>(L.R, std::min<int64_t>(64, p.n_rows / (8 * total_warps) / L.R * L.R));
  s.n_blocks = (p.n_rows + s.rows_per_block - 1) / s.rows_per_block;
  const int64_t ctas = (s.n_blocks + warps - 1) / warps;
  auto go = [&](auto kern) -> int {
    if (!ensure_smem_limit((const void*)kern, L.total)) return LS_GPU_ERR_CUDA;
    int resident = 0;
    if (!cuda_ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kern, L.threads, L.total), "occupancy"))
      return LS_GPU_ERR_CUDA;
    const int64_t blocks = std::min<int64_t>(ctas, (int64_t)sms * std::max(1, resident) * waves);
    kern<<<(unsigned)std::max<int64_t>(1, blocks), L.threads, L.total, st>>>(p, L, s, d_err, binom);
    return cuda_ok(cudaGetLastError(), "k_matvec_rows") ? 0 : LS_GPU_ERR_CUDA;
  };
  const bool inv = p.group.spin_inversion != 0;
  auto with_col = [&](auto mtag, auto itag, auto ftag) -> int {
    constexpr int M = decltype(mtag)::value;
    constexpr bool I = decltype(itag)::value, F = decltype(ftag)::value;
    switch (col) {
      case kColReal: return go(k_matvec_rows<M, I, F, kColReal>);
      case kColPair: return go(k_matvec_rows<M, I, F, kColPair>);
      default: return go(k_matvec_rows<M, I, F, kColComplex>);
    }
  };
  auto with_mode = [&](auto mtag) -> int {
    if (p.group.fermionic) {
      if (inv) return fail(LS_GPU_ERR_INVALID, "fermionic groups have no spin inversion");
      return with_col(mtag, std::false_type{}, std::true_type{});
    }
    return inv ? with_col(mtag, std::true_type{}, std::false_type{})
               : with_col(mtag, std::false_type{}, std::false_type{});
  };
  return mode == kModeN32 ? with_mode(std::integral_constant<int, kModeN32>{})
                          : with_mode(std::integral_constant<int, kModeP16>{});
}

}  // namespace lsg
