// matvec_free.cu -- y = H x without a permutation group (no symmetries, or spin inversion only): all states of
// a fixed particle number, of fixed (N_up, N_down), or of no constraint.
//
// Index.  Such bases are complete, so a state's index is its rank, and the rank of a state of fixed
// weight splits into a part of its low bits and a part of its high bits (the weight of the low bits
// follows from the high ones): index = rank_hi[state >> split] + rank_lo[state & mask], two table
// reads (in shared memory up to 26 bits) in place of a walk over the set bits through a binomial
// table or a search.  (N_up, N_down) has the same form with one table per species.
//
// Rows.  One thread per row and column.  A thread first matches the term slots (two exclusive patterns
// per slot, DeviceRowTerms) into a bit mask, 32 slots at once: the state's bit at the first (second)
// site of every slot is an XOR of table words over the state's nibbles, and so are the parities of
// 32 diagonal terms.  (Slots on more than two sites are tested one by one.)  It then takes the mask's
// set bits, four gathers at a time, so that lanes with other matches do not idle on a term that is
// not theirs.  The bits are taken from
// the top: neighbouring rows agree in their high sites, so their lanes meet the same terms there and
// read neighbouring entries of x.  All columns of a row share a warp.
//
// The FP64 pipe (1 FMA per element for real vectors, 2 or 4 per complex column) and the loads bound
// it.  Measured (GB300, one thread per row with a binomial walk or a search per element, every column on
// its own -> here): 24 spins, weight 12 (2.7e6 rows), one real vector 1345 -> 122 us (178 us
// with slots and diagonal terms tested one by one); 12-site Hubbard, 6 + 6 fermions (8.5e5 rows), 4
// complex columns 1380 -> 250 us.
#include <algorithm>

#include "matvec_launch.cuh"
#include "rowsums.cuh"

namespace lsg {

extern const uint64_t* device_binomials();

constexpr int kFreeThreads = 512;
constexpr size_t kFreeSmem = 112 * 1024;  // two CTAs per SM

// A slot as the kernel reads it: mask, the two patterns, their terms (first | second << 16).
template <typename State>
struct alignas(sizeof(State) == 4 ? 16 : 32) FreeSlot {
  State m, l1, l2;
  uint32_t terms;
};
template <typename State>
struct alignas(2 * sizeof(State)) FreeTerm {
  State x;
  uint32_t info;
};

// 32 slots at once: the bits that the two patterns want at the slots' first and second sites.
struct FreeWant {
  uint32_t first1, second1, first2, second2;  // pattern 1, pattern 2
  uint32_t valid;
};

struct FreeLayout {
  int T, n_slots, n_diag_blocks, signs, checks, planes, tables_in_smem;
  int nibbles;
  uint32_t off_tlo, off_thi, off_coef, off_slots, off_terms, off_ts, off_want, off_first, off_second, off_parity, off_dm, off_dr, off_ds, off_db, off_dv;
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

// Sets *bad unless state i of a caller's set has rank i, the basis' weights and no bit beyond the basis.
__global__ void k_check_ranks(const uint64_t* __restrict__ reps, int64_t n, DeviceConstraint constraint, int split,
                              int n_bits, const uint32_t* __restrict__ lo, const uint32_t* __restrict__ hi,
                              int* __restrict__ bad) {
  const uint64_t low_mask = ((uint64_t)1 << split) - 1;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t a = __ldg(reps + i);
    if ((a >> n_bits) != 0 || !constraint_ok(constraint, a) || hi[a >> split] + lo[a & low_mask] != (uint32_t)i)
      *bad = 1;
  }
}

int launch_check_ranks(int split, int n_bits, const DeviceConstraint& constraint, const uint64_t* d_reps, int64_t n,
                       const uint32_t* d_lo, const uint32_t* d_hi, int* d_bad, cudaStream_t s) {
  const int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 8);
  k_check_ranks<<<blocks, 256, 0, s>>>(d_reps, n, constraint, split, n_bits, d_lo, d_hi, d_bad);
  return cuda_ok(cudaGetLastError(), "k_check_ranks") ? 0 : LS_GPU_ERR_CUDA;
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
  FreeSlot<State>* slots = (FreeSlot<State>*)(smem + L.off_slots);
  for (int i = tid; i < L.n_slots; i += nt)
    slots[i] = {(State)__ldg(p.off.rows.sm + i), (State)__ldg(p.off.rows.sl1 + i), (State)__ldg(p.off.rows.sl2 + i),
                __ldg(p.off.rows.st + i)};
  FreeTerm<State>* terms = (FreeTerm<State>*)(smem + L.off_terms);
  for (int i = tid; i < L.T; i += nt) terms[i] = {(State)__ldg(p.off.x + i), __ldg(p.off.rows.tinfo + i)};
  states(L.off_ts, p.off.s, L.T);
  const int slot_blocks = (L.n_slots + 31) / 32;
  uint32_t* first_lut = (uint32_t*)(smem + L.off_first);    // [block][nibble][16]
  uint32_t* second_lut = (uint32_t*)(smem + L.off_second);
  uint32_t* parity_lut = (uint32_t*)(smem + L.off_parity);  // [diagonal block][nibble][16]
  FreeWant* want = (FreeWant*)(smem + L.off_want);
  const int per_block = 16 * L.nibbles;
  states(L.off_dm, p.diag.rows.sm, 32 * L.n_diag_blocks);
  states(L.off_dr, p.diag.rows.sl1, 32 * L.n_diag_blocks);
  states(L.off_ds, p.diag.rows.sl2, 32 * L.n_diag_blocks);
  uint2* db = (uint2*)(smem + L.off_db);
  for (int i = tid; i < L.n_diag_blocks; i += nt)
    db[i] = make_uint2(__ldg(p.diag.rows.st + i), __ldg(p.diag.rows.tinfo + i));
  stage_d2((double2*)(smem + L.off_dv), p.diag.rows.cval, p.diag.rows.n_cls);
  C* coef = (C*)(smem + L.off_coef);  // per term, with its sign
  for (int i = tid; i < L.T; i += nt) {
    const uint32_t info = __ldg(p.off.rows.tinfo + i);
    const double2 v = flip_sign(__ldg(p.off.rows.cval + ((info >> 16) & 0xffu)), info & 0x80000000u);
    if constexpr (COL == kColComplex) coef[i] = v;
    else coef[i] = v.x;
  }
  __syncthreads();
  const State* ds = (const State*)(smem + L.off_ds);
  if (L.planes) {
    for (int i = tid; i < slot_blocks * per_block; i += nt) {
      const int blk = i / per_block, at = (i - blk * per_block) >> 4;
      const State v = (State)((uint64_t)(i & 15) << (4 * at));
      uint32_t f = 0, g = 0;
      for (int k = 32 * blk; k < min(32 * blk + 32, L.n_slots); ++k) {
        const State m = slots[k].m;
        const State lowest = m & (0 - m);
        if (v & lowest) f |= 1u << (k & 31);
        const State highest = m ^ lowest ? m ^ lowest : m;  // one-site slots: the same site
        if (v & highest) g |= 1u << (k & 31);
      }
      first_lut[i] = f;
      second_lut[i] = g;
    }
    for (int blk = tid; blk < slot_blocks; blk += nt) {
      FreeWant w{0, 0, 0, 0, 0};
      for (int k = 32 * blk; k < min(32 * blk + 32, L.n_slots); ++k) {
        const State m = slots[k].m, l1 = slots[k].l1, l2 = slots[k].l2;
        const State lowest = m & (0 - m), highest = m ^ lowest ? m ^ lowest : m;
        const uint32_t bit = 1u << (k & 31);
        w.valid |= bit;
        if (l1 & lowest) w.first1 |= bit;
        if (l1 & highest) w.second1 |= bit;
        if (l2 & lowest) w.first2 |= bit;
        if (l2 & highest) w.second2 |= bit;
      }
      want[blk] = w;
    }
  }
  for (int i = tid; i < L.n_diag_blocks * per_block; i += nt) {
    const int blk = i / per_block, at = (i - blk * per_block) >> 4;
    const State v = (State)((uint64_t)(i & 15) << (4 * at));
    uint32_t f = 0;
    for (int k = 0; k < 32; ++k)
      if (popc_state((State)(v & ds[32 * blk + k])) & 1) f |= 1u << k;
    parity_lut[i] = f;
  }
  __syncthreads();
  const State* ts = (const State*)(smem + L.off_ts);
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
    for (int s0 = 32 * (slot_blocks - 1); s0 >= 0; s0 -= 32) {  // none without off-diagonal terms
      uint32_t first = 0, any = 0;  // slots whose first / some pattern matches
      if (L.planes) {
        const uint32_t* fl = first_lut + (s0 >> 5) * per_block;
        const uint32_t* sl = second_lut + (s0 >> 5) * per_block;
        uint32_t f = 0, g = 0;
        State left = a;
        for (int k = 0; k < L.nibbles; ++k, left >>= 4) {
          f ^= fl[16 * k + (int)(left & 15)];
          g ^= sl[16 * k + (int)(left & 15)];
        }
        const FreeWant w = want[s0 >> 5];
        first = ~(f ^ w.first1) & ~(g ^ w.second1) & w.valid;
        any = ~(f ^ w.first2) & ~(g ^ w.second2) & w.valid;
      } else {
        const int n = min(32, L.n_slots - s0);
        for (int i = 0; i < n; ++i) {
          const FreeSlot<State> q = slots[s0 + i];
          const State v = a & q.m;
          if (v == q.l1) first |= 1u << i;
          if (v == q.l2) any |= 1u << i;
        }
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
            const int i = 31 - __clz(any);
            any ^= 1u << i;
            const uint32_t t12 = slots[s0 + i].terms;
            const uint32_t t = ((first >> i) & 1u) ? t12 & 0xffffu : t12 >> 16;
            const FreeTerm<State> term = terms[t];
            State b = a ^ term.x;
            uint32_t neg = 0;
            if (L.signs) neg = (uint32_t)popc_state((State)(b & ts[t]));
            if (L.checks && (term.info & kRowTermNeedsCheck) && !constraint_ok(p.constraint, b)) {
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
            cf[u] = coef[t];
            if (L.signs || INV) cf[u] = flip_sign(cf[u], neg << 31);
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
      const uint32_t valid = 0xffffffffu >> (32 - ((info.y >> 16) & 0x3fu));
      uint32_t odd = info.x;
      State left = a;
      for (int k = 0; k < L.nibbles; ++k, left >>= 4) odd ^= parity_lut[b * per_block + 16 * k + (int)(left & 15)];
      uint32_t hit = valid;
      if (!((info.y >> 30) & 1u)) {  // some term of the block has a mask
        const State* m = (const State*)(smem + L.off_dm) + 32 * b;
        const State* r = (const State*)(smem + L.off_dr) + 32 * b;
        for (int i = 0; i < 32; ++i)
          if ((a & m[i]) != r[i]) hit &= ~(1u << i);
      }
      count += __popc(hit) - 2 * __popc(hit & odd);
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
  if ((size_t)p.off.n * 40 > 2 * kFreeSmem || (size_t)t.slot_blocks * 32 * 40 > 2 * kFreeSmem || (size_t)d.slot_blocks * 32 * 12 > kFreeSmem) return false;
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
  L.off_coef = take((size_t)L.T * 16);
  L.off_slots = take((size_t)L.n_slots * state * 4);
  L.off_terms = take((size_t)L.T * state * 2);
  L.off_ts = take(L.T * state);
  L.nibbles = (p.group.n_bits + 3) / 4;
  L.planes = t.two_site;
  L.checks = t.any_check;
  const size_t lut = L.planes ? (size_t)t.slot_blocks * L.nibbles * 64 : 0;
  L.off_want = take((size_t)t.slot_blocks * sizeof(FreeWant));
  L.off_first = take(lut);
  L.off_second = take(lut);
  L.off_parity = take((size_t)L.n_diag_blocks * L.nibbles * 64);
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
