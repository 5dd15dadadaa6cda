// rowsums.cuh -- sums over the elements that the row-group orbit scan (rowgroup.cuh) resolves: y = H x for one or
// several real or complex columns, FP64 multiply-adds.
//
// Sums.  A row's resolved elements are {column index j, coefficient word}; the coefficient
// v conj(chi_g) comes from a shared-memory table over (class of v, group element) and its sign from
// the word's top bit, so that forming it costs no FP64 instruction.  For several columns the lanes
// of a warp are split into `rp` rows x `q` elements x `cols` columns; q = 1 (no cross-lane sum)
// from 4 columns on.  The norms are folded in through the gather source x_j n_j and one
// multiplication by 1 / n_i per output, the diagonal element is a class count times the class
// value: per row and column the FP64 pipe sees little more than the products themselves (2 FMAs
// per element for real elements, 4 for complex ones).  GB300's FP64 pipe (2 lanes per clock and SM)
// bounds blocks of 16 columns on small groups (28-site chain, complex sector: 90 % of it busy); the
// scan bounds single vectors.
#pragma once

#include "rowgroup.cuh"

namespace lsg {

// Threads per CTA (one CTA per SM: 64 or 80 registers per thread).
template <bool KEEP>
constexpr int kRowsThreads = KEEP ? 1024 : 768;
constexpr int kColReal = 0, kColPair = 1, kColComplex = 2;

struct RowsSums {
  const double* x;   // the caller's vectors (diagonal), leading dimension ldx in scalars
  const double* xs;  // x_j n_j, leading dimension ldxs in scalars; x itself where norms != null
  const double* norms;  // the orbit norms n_j where xs is not scaled (small problems), else null
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
__device__ __forceinline__ double scaled(double v, double n) { return v * n; }
__device__ __forceinline__ double2 scaled(double2 v, double n) { return make_double2(v.x * n, v.y * n); }
__device__ __forceinline__ double shfl_down_v(double v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }
__device__ __forceinline__ double2 shfl_down_v(double2 v, int d) {
  return make_double2(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double add_v(double a, double b) { return a + b; }
__device__ __forceinline__ double2 add_v(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// x_j (n_j) of column unit c: a vector load from a scaled copy or of complex columns; pairs of the
// caller's real columns are only 8-byte aligned and may lack the second.
template <int COL>
__device__ __forceinline__ typename Column<COL>::V load_x(const RowsSums& s, uint32_t j, int c) {
  using V = typename Column<COL>::V;
  if constexpr (COL == kColPair) {
    if (s.norms != nullptr && s.real_cols) {
      const double* q = s.xs + (int64_t)j * s.ldxs + 2 * c;
      return make_double2(__ldg(q), 2 * c + 1 < s.real_cols ? __ldg(q + 1) : 0.0);
    }
  }
  const int64_t ldv = COL == kColPair && s.real_cols ? s.ldxs / 2 : s.ldxs;
  return __ldg(reinterpret_cast<const V*>(s.xs) + (int64_t)j * ldv + c);
}

// y of one row and column: the sum over n_i plus the diagonal (zero for a zero-norm row).
template <int COL>
__device__ __forceinline__ void write_output(const RowsSums& s, int64_t row, int c, typename Column<COL>::V acc,
                                             double inv, double dre, double dim) {
  if constexpr (COL == kColReal) {
    s.y[row * s.ldy + c] = inv == 0.0 ? 0.0 : acc * inv + dre * __ldg(s.x + row * s.ldx + c);
  } else if (s.real_cols) {
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

// One column: every lane sums its own elements as they are resolved, then the lanes of a row add up.
template <int COL, typename Group>
__device__ __forceinline__ void resolve_and_sum(Group& g, const RowsSums& s, const DeviceIndex& ix,
                                                const typename Column<COL>::C* coef, int64_t row0,
                                                int* __restrict__ err, const uint64_t* __restrict__ binom) {
  using Col = Column<COL>;
  using V = typename Col::V;
  constexpr unsigned FULL = 0xffffffffu;
  const RowsLayout& L = g.L;
  V acc = Col::zero();
  g.resolve(ix, err, binom, [&](const auto& j, const auto& w, const auto&) {
    constexpr int E = sizeof(j) / sizeof(j[0]);
    V xv[E];
#pragma unroll
    for (int e = 0; e < E; ++e) xv[e] = j[e] != Group::kAbsent ? load_x<COL>(s, j[e], 0) : Col::zero();
    if (s.norms != nullptr) {
#pragma unroll
      for (int e = 0; e < E; ++e) xv[e] = scaled(xv[e], j[e] != Group::kAbsent ? __ldg(s.norms + j[e]) : 0.0);
    }
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (j[e] != Group::kAbsent) Col::mac(acc, flip_sign(coef[w[e] & 0x7fffffffu], w[e] & 0x80000000u), xv[e]);
  });
  const double2 diag = g.diagonal();
  for (int d = L.lanes_per_row / 2; d > 0; d >>= 1) acc = add_v(acc, shfl_down_v(acc, d));
  const int r = g.lane >> L.lane_shift;
  const double inv = __shfl_sync(FULL, g.inv_l, r);
  const double dre = __shfl_sync(FULL, diag.x, r);
  const double dim = COL == kColReal ? 0.0 : __shfl_sync(FULL, diag.y, r);
  if ((g.lane & (L.lanes_per_row - 1)) == 0 && r < g.nr) write_output<COL>(s, row0 + r, 0, acc, inv, dre, dim);
}

// Several columns: the resolved elements go to shared memory, then the warp sums them with lanes
// split into rows, elements and columns.
template <int COL, typename Group>
__device__ __forceinline__ void sum_rows(const Group& g, const RowsSums& s, const typename Column<COL>::C* coef,
                                         int64_t row0) {
  using Col = Column<COL>;
  using V = typename Col::V;
  constexpr unsigned FULL = 0xffffffffu;
  const RowsLayout& L = g.L;
  const int lane = g.lane;
  const int c = lane % s.cols, rest = lane / s.cols;
  const int q = rest & (s.q - 1), rl = rest / s.q;
  const bool active = rl < s.rp;
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
      for (int u = 0; u < 4; ++u) xv[u] = w[u].x != Group::kAbsent ? load_x<COL>(s, w[u].x, c) : Col::zero();
      if (s.norms != nullptr) {
#pragma unroll
        for (int u = 0; u < 4; ++u) xv[u] = scaled(xv[u], w[u].x != Group::kAbsent ? __ldg(s.norms + w[u].x) : 0.0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (w[u].x != Group::kAbsent) Col::mac(acc, flip_sign(coef[w[u].y & 0x7fffffffu], w[u].y & 0x80000000u), xv[u]);
    }
    for (int d = s.q / 2; d > 0; d >>= 1) acc = add_v(acc, shfl_down_v(acc, d * s.cols));
    const double inv = __shfl_sync(FULL, g.inv_l, rr);
    const double dre = __shfl_sync(FULL, diag.x, rr);
    const double dim = COL == kColReal ? 0.0 : __shfl_sync(FULL, diag.y, rr);
    if (act && q == 0) write_output<COL>(s, row0 + r, c, acc, inv, dre, dim);
  }
}

// Coefficient table v conj(chi) over (class, element); chars in element order.
template <int COL>
__device__ __forceinline__ void stage_coefficients(const RowsLayout& L, const DeviceRowTerms& t, const double2* chars,
                                                   typename Column<COL>::C* coef) {
  for (int i = threadIdx.x; i < t.n_cls * L.G; i += blockDim.x) {
    const double2 v = __ldg(t.cval + i / L.G), chi = __ldg(chars + i % L.G);
    const C2 f = cmul_conj_b(C2{v.x, v.y}, C2{chi.x, chi.y});
    if constexpr (COL == kColComplex) coef[i] = make_double2(f.re, f.im);
    else coef[i] = f.re;
  }
}


// Host side (matvec_rows.cu).
struct RowsLaunch {
  RowsLayout L;
  RowsSums s;  // lanes and row blocks; the vectors are the caller's to set
  int mode;
  int64_t blocks;  // CTAs
};
// Picks shape and layout for k columns over n_rows rows (n_sectors > 0: the batched kernel's
// tables); false when the tables do not fit.
// max_threads 0: the matvec kernels' own.
bool rows_plan(const MatvecProblem& p, int col, int k, int64_t n_rows, int n_sectors, RowsLaunch* out,
               int max_threads = 0);
// Launches a plan of this scan mode (rowkernel.cuh).
template <int MODE>
int launch_rows_mode(const MatvecProblem& p, const RowsLaunch& q, int col, int* d_err, const uint64_t* binom,
                     cudaStream_t st);

}  // namespace lsg
