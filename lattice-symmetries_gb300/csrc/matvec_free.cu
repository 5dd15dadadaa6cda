// matvec_free.cu -- y = H x without a permutation group (no symmetries, or spin inversion only): all states of
// a fixed particle number, of fixed (N_up, N_down), or of no constraint.
//
// Index.  Such bases are complete, so a state's index is its rank, and the rank of a state of fixed
// weight splits into a part of its low bits and a part of its high bits (the weight of the low bits
// follows from the high ones): index = rank_hi[state >> split] + rank_lo[state & mask], two table
// reads (in shared memory up to 26 bits) in place of a walk over the set bits through a binomial
// table or a search.  (N_up, N_down) has the same form with one table per species.
//
// Rows.  One thread per row and column.  A thread first tests the term slots (two exclusive patterns
// per slot, DeviceRowTerms) into a bit mask and then takes its set bits, four gathers at a time, so
// that lanes with other matches do not idle on a term that is not theirs; all columns of a row
// share a warp.
//
// The FP64 pipe (1 FMA per element for real vectors, 2 or 4 per complex column) and the loads bound
// it.  Measured (GB300, one thread per row with a binomial walk or a search per element, every column on
// its own -> here): 24 spins, weight 12 (2.7e6 rows), one real vector 1345 -> 178 us; 12-site
// Hubbard, 6 + 6 fermions (8.5e5 rows), 4 complex columns 1380 -> 261 us.
#include <algorithm>

#include "matvec_launch.cuh"
#include "rowsums.cuh"

namespace lsg {

extern const uint64_t* device_binomials();

constexpr int kFreeThreads = 512;
constexpr size_t kFreeSmem = 112 * 1024;  // two CTAs per SM

struct FreeLayout {
  int T, n_slots, n_diag_blocks, signs, tables_in_smem;
  uint32_t off_tlo, off_thi, off_coef, off_sm, off_sl1, off_sl2, off_st, off_ti, off_ts, off_tx, off_dm, off_dr, off_ds,
      off_db, off_dv;
  uint32_t total;
  int cols, rows_per_warp;
};

// Ranks of the low and high parts of a state.  species = 0: states of weight h, split bits low;
// 1: low part of weight lo_weight, high part of weight h with n_lo low states each.
__global__ void k_rank_tables(int split, int high_bits, int h, int species, int64_t n_lo,
                              const uint64_t* __restrict__ binom /*65x65*/, uint32_t* __restrict__ lo,
                              uint32_t* __restrict__ hi) {
  const int64_t n_low = (int64_t)1 << split, n_high = (int64_t)1 << high_bits;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_low + n_high;
       i += (int64_t)gridDim.x * blockDim.x) {
    const bool high = i >= n_low;
    uint64_t v = (uint64_t)(high ? i - n_low : i);
    const bool shifted = high && species == 0;
    int k = shifted ? h - __popcll(v) : 0;  // set bits below
    const int base = shifted ? split : 0;
    uint64_t r = 0;
    for (; v != 0 && k >= 0; v &= v - 1) {
      const int c = base + __ffsll((long long)v) - 1;
      ++k;
      if (c > 0 && k <= c) r += __ldg(binom + c * 65 + k);
    }
    if (high && species == 1) r *= (uint64_t)n_lo;
    (high ? hi[i - n_low] : lo[i]) = (uint32_t)r;
  }
}

int launch_rank_tables(int split, int high_bits, int h, int species, int64_t n_lo, uint32_t* d_lo, uint32_t* d_hi,
                       cudaStream_t s) {

  const uint64_t* binom = device_binomials();
  if (binom == nullptr) return LS_GPU_ERR_CUDA;
  const int64_t n = ((int64_t)1 << split) + ((int64_t)1 << high_bits);
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 8);
  k_rank_tables<<<blocks, 256, 0, s>>>(split, high_bits, h, species, n_lo, binom, d_lo, d_hi);
  return cuda_ok(cudaGetLastError(), "k_rank_tables") ? 0 : LS_GPU_ERR_CUDA;
}

template <typename State, bool INV, int COL>
__global__ void __launch_bounds__(kFreeThreads, 2)
    k_matvec_free(const MatvecProblem p, const FreeLayout L, const double* __restrict__ x_, int64_t ldx,
                  double* __restrict__ y_, int64_t ldy, int* __restrict__ err) {
  using Col = Column<COL>;
  using V = typename Col::V;
  using C = typename Col::C;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, nt = blockDim.x;
  auto states = [&](uint32_t off, const uint64_t* src, int n) {
    State* dst = (State*)(smem + off);
    for (int i = tid; i < n; i += nt) dst[i] = (State)__ldg(src + i);
  };
  auto words = [&](uint32_t off, const uint32_t* src, int n) {
    uint32_t* dst = (uint32_t*)(smem + off);
    for (int i = tid; i < n; i += nt) dst[i] = __ldg(src + i);
  };
  const int split = p.index.rank_split, high_bits = p.group.n_bits - split;
  if (L.tables_in_smem) {
    words(L.off_tlo, p.index.rank_lo, 1 << split);
    words(L.off_thi, p.index.rank_hi, 1 << high_bits);
  }
  states(L.off_sm, p.off.rows.sm, L.n_slots);
  states(L.off_sl1, p.off.rows.sl1, L.n_slots);
  states(L.off_sl2, p.off.rows.sl2, L.n_slots);
  words(L.off_st, p.off.rows.st, L.n_slots);
  words(L.off_ti, p.off.rows.tinfo, L.T);
  states(L.off_ts, p.off.s, L.T);
  states(L.off_tx, p.off.x, L.T);
  states(L.off_dm, p.diag.rows.sm, 32 * L.n_diag_blocks);
  states(L.off_dr, p.diag.rows.sl1, 32 * L.n_diag_blocks);
  states(L.off_ds, p.diag.rows.sl2, 32 * L.n_diag_blocks);
  uint2* db = (uint2*)(smem + L.off_db);
  for (int i = tid; i < L.n_diag_blocks; i += nt)
    db[i] = make_uint2(__ldg(p.diag.rows.st + i), __ldg(p.diag.rows.tinfo + i));
  stage_d2((double2*)(smem + L.off_dv), p.diag.rows.cval, p.diag.rows.n_cls);
  C* coef = (C*)(smem + L.off_coef);
  for (int i = tid; i < p.off.rows.n_cls; i += nt) {
    const double2 v = __ldg(p.off.rows.cval + i);
    if constexpr (COL == kColComplex) coef[i] = v;
    else coef[i] = v.x;
  }
  __syncthreads();
  const State* sm = (const State*)(smem + L.off_sm);
  const State* sl1 = (const State*)(smem + L.off_sl1);
  const State* sl2 = (const State*)(smem + L.off_sl2);
  const uint32_t* st = (const uint32_t*)(smem + L.off_st);
  const uint32_t* ti = (const uint32_t*)(smem + L.off_ti);
  const State* ts = (const State*)(smem + L.off_ts);
  const State* tx = (const State*)(smem + L.off_tx);
  const uint32_t* lo = L.tables_in_smem ? (const uint32_t*)(smem + L.off_tlo) : p.index.rank_lo;
  const uint32_t* hi = L.tables_in_smem ? (const uint32_t*)(smem + L.off_thi) : p.index.rank_hi;
  const State low_mask = (State)(((uint64_t)1 << split) - 1), flip = (State)p.group.flip;
  const uint32_t inversion_sign = p.group.spin_inversion == -1 ? 1u : 0u;
  const bool identity = p.index.identity != 0;
  const V* __restrict__ x = reinterpret_cast<const V*>(x_);
  V* __restrict__ y = reinterpret_cast<V*>(y_);

  const int lane = tid & 31, c = lane % L.cols, rl = lane / L.cols;
  if (rl >= L.rows_per_warp) return;
  const int64_t warps = ((int64_t)gridDim.x * nt) >> 5;
  for (int64_t row = (((int64_t)blockIdx.x * nt + tid) >> 5) * L.rows_per_warp + rl; row < p.n_rows;
       row += warps * L.rows_per_warp) {
    const State a = identity ? (State)row : (State)__ldg(p.index.reps + row);
    V acc = Col::zero();
    for (int s0 = 0; s0 < L.n_slots; s0 += 32) {
      const int n = min(32, L.n_slots - s0);
      uint32_t first = 0, any = 0;  // slots whose first / some pattern matches
      for (int i = 0; i < n; ++i) {
        const State v = a & sm[s0 + i];
        if (v == sl1[s0 + i]) first |= 1u << i;
        if (v == sl2[s0 + i]) any |= 1u << i;
      }
      any |= first;
      while (any != 0) {
        V xv[4];
        C cf[4];
        uint32_t ok = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          xv[u] = Col::zero();
          if (any != 0) {
            const int i = __ffs(any) - 1;
            any &= any - 1;
            const uint32_t t12 = st[s0 + i];
            const uint32_t t = ((first >> i) & 1u) ? t12 & 0xffffu : t12 >> 16;
            const uint32_t info = ti[t];
            State b = a ^ tx[t];
            uint32_t neg = info >> 31;
            if (L.signs) neg ^= (uint32_t)popc_state((State)(b & ts[t]));
            if ((info & kRowTermNeedsCheck) && !constraint_ok(p.constraint, b)) {
              atomicOr(err, 1);
              continue;
            }
            if (INV) {
              const State f = b ^ flip;
              if (f < b) {
                b = f;
                neg ^= inversion_sign;
              }
            }
            const uint64_t j = identity ? (uint64_t)b : (uint64_t)(hi[b >> split] + lo[b & low_mask]);
            xv[u] = __ldg(x + j * (uint64_t)ldx + c);
            cf[u] = flip_sign(coef[(info >> 16) & 0xffu], neg << 31);
            ok |= 1u << u;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if ((ok >> u) & 1u) Col::mac(acc, cf[u], xv[u]);
      }
    }
    double dre = 0.0, dim = 0.0;
    int count = 0;
    for (int b = 0; b < L.n_diag_blocks; ++b) {
      const uint2 info = db[b];  // {signs, class | last block of it << 31}
      const State* m = (const State*)(smem + L.off_dm) + 32 * b;
      const State* r = (const State*)(smem + L.off_dr) + 32 * b;
      const State* s = (const State*)(smem + L.off_ds) + 32 * b;
      for (int i = 0; i < (int)((info.y >> 16) & 0x3fu); ++i) {
        const int odd = (popc_state((State)(a & s[i])) ^ (int)(info.x >> i)) & 1;
        if ((a & m[i]) == r[i]) count += 1 - 2 * odd;
      }
      if (info.y >> 31) {
        const double2 v = ((const double2*)(smem + L.off_dv))[info.y & 0xffffu];
        dre = fma((double)count, v.x, dre);
        dim = fma((double)count, v.y, dim);
        count = 0;
      }
    }
    const V xi = __ldg(x + row * ldx + c);
    if constexpr (COL == kColReal) {
      y[row * ldy + c] = acc + dre * xi;
    } else {
      acc.x += dre * xi.x;
      acc.y += dre * xi.y;
      if (dim != 0.0) {
        acc.x -= dim * xi.y;
        acc.y += dim * xi.x;
      }
      y[row * ldy + c] = acc;
    }
  }
}

static bool free_layout(const MatvecProblem& p, FreeLayout* out) {
  FreeLayout L{};
  const DeviceRowTerms &t = p.off.rows, &d = p.diag.rows;
  if (!t.ok || !d.ok || p.group.n_bits > 63) return false;
  if (!p.index.identity && p.index.rank_lo == nullptr) return false;
  if ((size_t)p.off.n * 20 > kFreeSmem || (size_t)d.slot_blocks * 32 * 12 > kFreeSmem) return false;
  const size_t state = p.group.n_bits <= 32 ? 4 : 8;
  uint32_t o = 0;
  auto take = [&](size_t bytes) {
    const uint32_t at = o;
    o += (uint32_t)((bytes + 15) & ~(size_t)15);
    return at;
  };
  L.T = p.off.n;
  L.n_slots = t.n_slots;
  L.n_diag_blocks = d.slot_blocks;
  L.signs = t.any_sign;
  L.off_coef = take((size_t)t.n_cls * 16);
  L.off_sm = take(L.n_slots * state);
  L.off_sl1 = take(L.n_slots * state);
  L.off_sl2 = take(L.n_slots * state);
  L.off_st = take((size_t)L.n_slots * 4);
  L.off_ti = take((size_t)L.T * 4);
  L.off_ts = take(L.T * state);
  L.off_tx = take(L.T * state);
  L.off_dm = take(32 * L.n_diag_blocks * state);
  L.off_dr = take(32 * L.n_diag_blocks * state);
  L.off_ds = take(32 * L.n_diag_blocks * state);
  L.off_db = take((size_t)L.n_diag_blocks * 8);
  L.off_dv = take((size_t)d.n_cls * 16);
  if (!p.index.identity) {
    const size_t tables = 4 * (((size_t)1 << p.index.rank_split) + ((size_t)1 << (p.group.n_bits - p.index.rank_split)));
    L.tables_in_smem = o + tables <= kFreeSmem;
    if (L.tables_in_smem) {
      L.off_tlo = take((size_t)4 << p.index.rank_split);
      L.off_thi = take((size_t)4 << (p.group.n_bits - p.index.rank_split));
    }
  }
  L.total = o;
  *out = L;
  return o <= kFreeSmem;
}

bool free_fits(const MatvecProblem& p) {
  FreeLayout L;
  return p.projection != 2 && p.nnz_counter == nullptr && free_layout(p, &L);
}

int launch_free(const MatvecProblem& p, Scalar sc, int k, const double* d_x, int64_t ldx, double* d_y, int64_t ldy,
                int* d_err, cudaStream_t s) {
  FreeLayout L;
  if (!free_layout(p, &L)) return LS_GPU_ERR_INVALID;
  const bool cplx = sc == Scalar::Complex, inv = p.projection == 1, narrow = p.group.n_bits <= 32;
  const int words = cplx ? 2 : 1;
  auto go = [&](auto kern) -> int {
    if (!ensure_smem_limit((const void*)kern, L.total)) return LS_GPU_ERR_CUDA;
    for (int done = 0; done < k; done += L.cols) {
      // columns of one launch: a row's columns are lanes of one warp
      L.cols = std::min(k - done, 16);
      L.rows_per_warp = 32 / L.cols;
      const int64_t rows_per_cta = (int64_t)L.rows_per_warp * (kFreeThreads / 32);
      const int64_t blocks = std::min<int64_t>((p.n_rows + rows_per_cta - 1) / rows_per_cta, (int64_t)num_sms() * 2);
      kern<<<(unsigned)std::max<int64_t>(1, blocks), kFreeThreads, L.total, s>>>(
          p, L, d_x + (size_t)done * words, ldx, d_y + (size_t)done * words, ldy, d_err);
      if (!cuda_ok(cudaGetLastError(), "k_matvec_free")) return LS_GPU_ERR_CUDA;
    }
    return 0;
  };
  auto with_col = [&](auto tag, auto itag) -> int {
    using State = decltype(tag);
    constexpr bool I = decltype(itag)::value;
    if (!cplx) return go(k_matvec_free<State, I, kColReal>);
    return p.real_elements ? go(k_matvec_free<State, I, kColPair>) : go(k_matvec_free<State, I, kColComplex>);
  };
  auto with_inv = [&](auto tag) -> int {
    return inv ? with_col(tag, std::true_type{}) : with_col(tag, std::false_type{});
  };
  return narrow ? with_inv(uint32_t{}) : with_inv(uint64_t{});
}

}  // namespace lsg
