// couplings.cu -- per-coupling inner products out[c] = <g, H_c x> = sum_i conj(g_i) (H_c x)_i for an
// operator H = sum_c H_c whose terms carry coupling ids (the backward pass of H(theta) x with
// respect to the coupling constants theta_c, since d/dtheta_c Re<g, H(theta) x> = Re out[c]).
//
// One pass over the rows, the same orbit scan as the packed matvec (one warp per row): every
// element's contribution conj(g_i) / n_i * v_t (-1)^popcount(beta & s_t) conj(chi) n_j x_j goes to
// the accumulator of its term's coupling instead of to y_i.  Per-lane sums are reduced per block,
// the block partials by one more small kernel in a fixed order (deterministic).
//
// k_coupling_rows does the same on the row-group orbit scan (one lane per element, rowgroup.cuh),
// where its tables fit and the rows are not few: a lane keeps one sum per coupling over its row's elements, with
// x_j n_j from a prescaled copy and coefficients from the (class, element) table, and multiplies by
// conj(g_i) / n_i once per row.  Alike terms of different couplings (Heisenberg and DM on a bond)
// are one element: the lane then sums per class, and the class sums count for each coupling with the
// class' coefficient at the very end.  28-site ladder, 1.43e6 rows, 3 couplings: 7.1 ms with one
// warp per row (k_coupling_products), 2.3 ms with one lane per element, 1.8 ms with alike terms
// merged (FP64 pipe 75 %: every element was added to every sum under a predicate), 1.4 ms with the
// element's sum picked by selects and multiply-adds at the rows' ends.
#include <type_traits>

#include "matvec_launch.cuh"
#include "rowsums.cuh"

namespace lsg {

extern const uint64_t* device_binomials();
constexpr int kMaxCouplings = 4;

template <int GPL, bool INV>
__global__ void __launch_bounds__(256, 2)
    k_coupling_products(const MatvecProblem p, const PackedLayout L, size_t off_cpl, int nc,
                        const double* __restrict__ g, const double* __restrict__ x,
                        double2* __restrict__ partial, int* __restrict__ err,
                        const uint64_t* __restrict__ binom) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr unsigned FULL = 0xffffffffu;
  const PackedTables T = stage_packed(p, L, smem, true);
  int32_t* cpl_off = (int32_t*)(smem + off_cpl);
  int32_t* cpl_diag = cpl_off + p.off.n;
  for (int i = threadIdx.x; i < p.off.n + p.diag.n; i += blockDim.x)
    cpl_off[i] = i < p.off.n ? p.off.coupling[i] : p.diag.coupling[i - p.off.n];
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const int nbits = p.group.n_bits;
  const int SH = 64 - nbits;
  const uint64_t lowmask = (1ull << SH) - 1;
  RowScan<GPL, INV> scan;
  scan.rec = T.rec;
  scan.gw = T.ga + (threadIdx.x >> 5) * 32 * rec_stride(GPL);  // this warp's g.a records
  scan.keys = scan_keys(nbits);
  scan.lane = lane;
  const double2* X = reinterpret_cast<const double2*>(x);
  const double2* Gv = reinterpret_cast<const double2*>(g);
  const DeviceIndex& ix = p.index;

  double2 tot[kMaxCouplings];
#pragma unroll
  for (int c = 0; c < kMaxCouplings; ++c) tot[c] = make_double2(0.0, 0.0);
  auto add = [&](int cid, double re, double im) {
#pragma unroll
    for (int c = 0; c < kMaxCouplings; ++c)
      if (c == cid) {
        tot[c].x += re;
        tot[c].y += im;
      }
  };

  const int64_t warp_id = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = warp_id; row < p.n_rows; row += n_warps) {
    const uint64_t a = __ldg(ix.reps + row);
    const double inv_na = __ldg(ix.inv_norms + row);
    if (inv_na == 0.0) continue;  // zero-norm representative: zero row
    const double2 gi = __ldg(Gv + row);
    const double2 xi = __ldg(X + row);
    const C2 gx = cmul_conj_b(C2{xi.x, xi.y}, C2{gi.x, gi.y});  // conj(g_i) x_i
    const C2 w{gi.x * inv_na, -gi.y * inv_na};                   // conj(g_i) / n_i

    for (int t = lane; t < T.nd; t += 32) {
      if ((a & T.dm[t]) == T.dr[t]) {
        double2 v = T.dv[t];
        if (__popcll(a & T.ds[t]) & 1) v = make_double2(-v.x, -v.y);
        const C2 val = cmul(C2{v.x, v.y}, gx);
        add(cpl_diag[t], val.re, val.im);
      }
    }

    scan.init(a);

    // the owning lane of each element keeps its key and term; coefficient, sign and coupling
    // are read at the flush
    uint64_t my_key = ~0ull;
    int my_t = 0;
    int nslot = 0;
    auto flush = [&]() {
      if (lane < nslot) {
        const uint64_t rep = my_key >> SH;
        const uint32_t idx = (uint32_t)(my_key & lowmask);
        const int64_t j = mv_index_lookup(ix, rep, binom);
        const double nj = j >= 0 ? __ldg(ix.norms + j) : 0.0;
        if (nj != 0.0) {
          double2 my_c = T.tv[my_t];
          if (__popcll((a ^ T.tx[my_t]) & T.ts[my_t]) & 1) my_c = make_double2(-my_c.x, -my_c.y);
          const int my_cid = cpl_off[my_t];
          double2 chi = T.ch[idx >> 1];
          if (INV && (idx & 1) && p.group.spin_inversion == -1) chi = make_double2(-chi.x, -chi.y);
          const C2 f = cmul_conj_b(C2{my_c.x * nj, my_c.y * nj}, C2{chi.x, chi.y});
          const double2 xv = __ldg(X + j);
          const C2 val = cmul(w, cmul(f, C2{xv.x, xv.y}));
          add(my_cid, val.re, val.im);
        }
      }
    };

    const int nt = T.nt;
    for (int t0 = 0; t0 < nt; t0 += 32) {
      const int tt = t0 + lane;
      const bool hit = tt < nt && (a & T.tm[tt]) == T.tl[tt];
      unsigned mask = __ballot_sync(FULL, hit);
      while (mask != 0) {
        const int t = t0 + __ffs(mask) - 1;
        mask &= mask - 1;
        const uint64_t xt = T.tx[t];
        const uint32_t info = T.ti[t];
        if (info & kTermNeedsCheck) {
          if (!constraint_ok(p.constraint, a ^ xt)) {
            if (lane == 0) atomicOr(err, 1);
            continue;
          }
        }
        const uint64_t key = (((info >> 16) & 0xffu) == 2u)
                                 ? scan.two_site((int)(info & 0xffu), (int)((info >> 8) & 0xffu))
                                 : scan.general(xt);
        if (lane == nslot) {
          my_key = key;
          my_t = t;
        }
        if (++nslot == 32) {
          flush();
          nslot = 0;
        }
      }
    }
    if (nslot > 0) flush();
  }

  // block reduction: lanes -> warps (shuffles) -> block (shared memory, fixed order)
  __shared__ double2 wsum[32][kMaxCouplings];
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < kMaxCouplings; ++c) {
    double re = tot[c].x, im = tot[c].y;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      re += __shfl_xor_sync(FULL, re, d);
      im += __shfl_xor_sync(FULL, im, d);
    }
    if (lane == 0) wsum[warp][c] = make_double2(re, im);
  }
  __syncthreads();
  if (threadIdx.x < nc) {
    double2 s = make_double2(0.0, 0.0);
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      s.x += wsum[w][threadIdx.x].x;
      s.y += wsum[w][threadIdx.x].y;
    }
    partial[(size_t)blockIdx.x * nc + threadIdx.x] = s;
  }
}

// out[c] = sum over the blocks' partials: a warp per coupling, lanes over the blocks, then a fixed
// tree (deterministic).
__global__ void k_sum_partials(const double2* __restrict__ partial, int n_blocks, int nc, double2* __restrict__ out) {
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (c >= nc) return;
  double2 s = make_double2(0.0, 0.0);
  for (int b = lane; b < n_blocks; b += 32) {
    const double2 v = partial[(size_t)b * nc + c];
    s.x += v.x;
    s.y += v.y;
  }
  s.x = warp_sum(s.x);
  s.y = warp_sum(s.y);
  if (lane == 0) out[c] = s;
}

constexpr int kCouplingThreads = 512;  // per-coupling sums in registers: up to 128 per thread

template <int MODE, bool INV>
__global__ void __launch_bounds__(kCouplingThreads, 1)
    k_coupling_rows(const MatvecProblem p, const RowsLayout L, const RowsSums s, int nc, const double2* __restrict__ gv,
                    double2* __restrict__ partial, int* __restrict__ err, const uint64_t* __restrict__ binom) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Group = RowGroup<MODE, INV, false, false>;
  __shared__ uint8_t class_of_off[64], class_of_diag[64];  // the sums that the classes go to
  if (threadIdx.x < 64) {
    class_of_off[threadIdx.x] = threadIdx.x < p.off.rows.n_cls ? (uint8_t)p.off.rows.coupling[threadIdx.x] : 0;
    class_of_diag[threadIdx.x] = threadIdx.x < p.diag.rows.n_cls ? (uint8_t)p.diag.rows.coupling[threadIdx.x] : 0;
  }
  Group::stage(L, p, smem);
  double2* coef = reinterpret_cast<double2*>(smem + L.off_coef);
  stage_coefficients<kColComplex>(L, p.off.rows, p.group.chars, coef);
  __syncthreads();
  Group g(L, p, smem);
  const double2* __restrict__ xs = reinterpret_cast<const double2*>(s.xs);
  const double2* __restrict__ x = reinterpret_cast<const double2*>(s.x);
  const int lane = g.lane;
  const int n_sums = p.off.rows.merged ? p.off.rows.n_cls : nc;
  double2 tot[kMaxCouplings], dtot[kMaxCouplings];
#pragma unroll
  for (int c = 0; c < kMaxCouplings; ++c) tot[c] = dtot[c] = make_double2(0.0, 0.0);
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t b = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; b < s.n_blocks; b += n_warps) {
    const int64_t begin = b * s.rows_per_block, end = min(begin + s.rows_per_block, p.n_rows);
    g.restart();
    for (int64_t row0 = begin; row0 < end; row0 += L.R) {
      g.load_rows(p.index, row0, (int)min((int64_t)L.R, end - row0));
      double2 acc[kMaxCouplings];
#pragma unroll
      for (int c = 0; c < kMaxCouplings; ++c) acc[c] = make_double2(0.0, 0.0);
      g.resolve(p.index, err, binom, [&](const auto& j, const auto& w, const auto& term) {
        constexpr int E = sizeof(j) / sizeof(j[0]);
        double2 xv[E];
#pragma unroll
        for (int e = 0; e < E; ++e) xv[e] = j[e] != Group::kAbsent ? __ldg(xs + j[e]) : make_double2(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          // the element's sum is picked and put back by selects: a multiply-add per component, where
          // an addition to each sum under a predicate took the FP64 pipe for all of them
          const int of_term = class_of_off[(g.template tab<uint32_t>(L.off_ti)[term[e]] >> 16) & 0xffu];
          const int cid = j[e] != Group::kAbsent ? of_term : kMaxCouplings;
          double2 v = acc[0];
#pragma unroll
          for (int c = 1; c < kMaxCouplings; ++c) v = c == cid ? acc[c] : v;
          Column<kColComplex>::mac(v, flip_sign(coef[w[e] & 0x7fffffffu], w[e] & 0x80000000u), xv[e]);
#pragma unroll
          for (int c = 0; c < kMaxCouplings; ++c) acc[c] = c == cid ? v : acc[c];
        }
      });
      // this lane's row: conj(g_i) / n_i times its sums
      const int r = lane >> L.lane_shift;
      const double inv = __shfl_sync(0xffffffffu, g.inv_l, r);
      if (r < g.nr && inv != 0.0) {
        const double2 gi = __ldg(gv + row0 + r);
        const double2 wi = make_double2(gi.x * inv, -gi.y * inv);
#pragma unroll
        for (int c = 0; c < kMaxCouplings; ++c)
          if (c < n_sums) Column<kColComplex>::mac(tot[c], wi, acc[c]);
      }
      // the diagonal: lane r holds row r's counts
      double2 d[kMaxCouplings];
#pragma unroll
      for (int c = 0; c < kMaxCouplings; ++c) d[c] = make_double2(0.0, 0.0);
      g.diagonal_counts([&](uint32_t cls, int n) {
        const double2 v = g.template tab<double2>(L.off_dv)[cls];
        const int cid = class_of_diag[cls];
#pragma unroll
        for (int c = 0; c < kMaxCouplings; ++c)
          if (c == cid) d[c] = make_double2(fma((double)n, v.x, d[c].x), fma((double)n, v.y, d[c].y));
      });
      if (lane < g.nr && g.inv_l != 0.0) {
        const double2 gi = __ldg(gv + row0 + lane), xi = __ldg(x + row0 + lane);
        const C2 gx = cmul_conj_b(C2{xi.x, xi.y}, C2{gi.x, gi.y});  // conj(g_i) x_i
#pragma unroll
        for (int c = 0; c < kMaxCouplings; ++c)
          if (c < nc) Column<kColComplex>::mac(dtot[c], d[c], make_double2(gx.re, gx.im));
      }
    }
  }
  // off-diagonal sums per class or coupling, diagonal sums per coupling
  __shared__ double2 wsum[kCouplingThreads / 32][kMaxCouplings], dsum[kCouplingThreads / 32][kMaxCouplings];
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < kMaxCouplings; ++c) {
    const double re = warp_sum(tot[c].x), im = warp_sum(tot[c].y);
    const double dre = warp_sum(dtot[c].x), dim = warp_sum(dtot[c].y);
    if (lane == 0) {
      wsum[warp][c] = make_double2(re, im);
      dsum[warp][c] = make_double2(dre, dim);
    }
  }
  __syncthreads();
  if (threadIdx.x < nc) {
    C2 t{0.0, 0.0};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      if (!p.off.rows.merged) {
        t.re += wsum[w][threadIdx.x].x;
        t.im += wsum[w][threadIdx.x].y;
      } else {
        for (int c = 0; c < p.off.rows.n_cls; ++c) {
          const double2 v = p.off.rows.cvec[c * nc + threadIdx.x];
          const C2 f = cmul(C2{v.x, v.y}, C2{wsum[w][c].x, wsum[w][c].y});
          t.re += f.re;
          t.im += f.im;
        }
      }
      t.re += dsum[w][threadIdx.x].x;
      t.im += dsum[w][threadIdx.x].y;
    }
    partial[(size_t)blockIdx.x * nc + threadIdx.x] = make_double2(t.re, t.im);
  }
}

// Returns 1 when there is no memory for the prescaled copy of x or the tables do not fit (nothing launched).
static int launch_coupling_rows(const MatvecProblem& p, int nc, const double* d_g, const double* d_x, double* d_out,
                                int* d_err, const uint64_t* binom, cudaStream_t st) {
  RowsLaunch q{};
  if (!rows_plan(p, kColComplex, 1, p.n_rows, 0, &q, kCouplingThreads)) return 1;
  double2* partial = (double2*)scratch((size_t)q.blocks * nc * sizeof(double2), 6);
  if (partial == nullptr) return LS_GPU_ERR_CUDA;
  double* d_xs = prescaled_copy(p, 2, 1, d_x, 1, 1, st);
  if (d_xs == nullptr) return 1;
  q.s.x = d_x;
  q.s.xs = d_xs;
  q.s.ldx = q.s.ldxs = 1;
  auto go = [&](auto kern) -> int {
    StageScope stage("couplings.kernel", st);
    if (!ensure_smem_limit((const void*)kern, q.L.total)) return LS_GPU_ERR_CUDA;
    kern<<<(unsigned)q.blocks, q.L.threads, q.L.total, st>>>(p, q.L, q.s, nc, reinterpret_cast<const double2*>(d_g),
                                                             partial, d_err, binom);
    if (!cuda_ok(cudaGetLastError(), "k_coupling_rows")) return LS_GPU_ERR_CUDA;
    k_sum_partials<<<1, 32 * kMaxCouplings, 0, st>>>(partial, (int)q.blocks, nc, reinterpret_cast<double2*>(d_out));
    return cuda_ok(cudaGetLastError(), "k_sum_partials") ? 0 : LS_GPU_ERR_CUDA;
  };
  const bool inv = p.group.spin_inversion != 0;
  int rc;
  switch (q.mode) {  // groups of at most 128 elements
    case kModeN32: rc = inv ? go(k_coupling_rows<kModeN32, true>) : go(k_coupling_rows<kModeN32, false>); break;
    case 2: rc = inv ? go(k_coupling_rows<2, true>) : go(k_coupling_rows<2, false>); break;
    case 5: rc = inv ? go(k_coupling_rows<5, true>) : go(k_coupling_rows<5, false>); break;
    default: rc = fail(LS_GPU_ERR_INVALID, "coupling products: at most 128 group elements");
  }
  cudaFreeAsync(d_xs, st);
  return rc;
}

int coupling_products_allowed(const MatvecProblem& p, int nc) {
  if (nc < 1 || nc > kMaxCouplings)
    return fail(LS_GPU_ERR_INVALID, "the fused coupling kernel handles 1 to 4 couplings");
  if (p.projection != 2 || p.group.gpl < 1 || p.group.gpl > 4 || p.group.onehot_packed == nullptr)
    return fail(LS_GPU_ERR_INVALID, "the fused coupling kernel needs a basis with lattice symmetries of at most "
                                    "128 elements");
  if (p.group.fermionic) return fail(LS_GPU_ERR_INVALID, "the fused coupling kernel has no fermionic signs");
  return 0;
}

int launch_coupling_products(const MatvecProblem& p, int nc, const double* d_g, const double* d_x, double* d_out,
                             int* d_err, cudaStream_t s) {
  const int allowed = coupling_products_allowed(p, nc);
  if (allowed != 0) return allowed;
  if (p.off.coupling == nullptr) return fail(LS_GPU_ERR_INVALID, "operator terms carry no coupling ids");
  const uint64_t* binom = device_binomials();
  if (binom == nullptr) return LS_GPU_ERR_CUDA;
  const PackedLayout L = make_packed_layout(p, 0, 256);
  const size_t off_cpl = (L.total + 15) & ~(size_t)15;
  const size_t smem = off_cpl + (size_t)(p.off.n + p.diag.n) * 4;
  // Few rows (one per warp of a CTA per SM) stay with a warp per row, which needs no scaled copy and fills smaller
  // tables: us per call from Python, warp per row / row groups, ladders of 12 and 16 sites (84 and 820
  // rows) 115 / 157, 125 / 156, 20 sites (9278 rows) 299 / 171; 6x6 translations, 1649 rows, 153 / 155.
  const bool few = p.n_rows <= (int64_t)num_sms() * 8 && smem <= kMaxDynamicSmem;
  if (p.n_rows > 0 && p.index.norms != nullptr && !few && rows_fit(p, 0)) {
    const int rc = launch_coupling_rows(p, nc, d_g, d_x, d_out, d_err, binom, s);
    if (rc != 1) return rc;
  }
  if (smem > kMaxDynamicSmem) return fail(LS_GPU_ERR_INVALID, "term tables too large for shared memory");
  const int blocks = std::max(1, std::min(num_sms() * 8, (int)((p.n_rows + 7) / 8)));
  double2* partial = (double2*)scratch((size_t)blocks * nc * sizeof(double2), 6);
  if (partial == nullptr) return LS_GPU_ERR_CUDA;
  auto go = [&](auto kern) -> int {
    StageScope stage("couplings.kernel", s);
    if (!ensure_smem_limit((const void*)kern, smem)) return LS_GPU_ERR_CUDA;
    kern<<<blocks, 256, smem, s>>>(p, L, off_cpl, nc, d_g, d_x, partial, d_err, binom);
    if (!cuda_ok(cudaGetLastError(), "k_coupling_products")) return LS_GPU_ERR_CUDA;
    k_sum_partials<<<1, 32 * kMaxCouplings, 0, s>>>(partial, blocks, nc, reinterpret_cast<double2*>(d_out));
    return cuda_ok(cudaGetLastError(), "k_sum_partials") ? 0 : LS_GPU_ERR_CUDA;
  };
  const bool inv = p.group.spin_inversion != 0;
  switch (p.group.gpl) {
    case 1: return inv ? go(k_coupling_products<1, true>) : go(k_coupling_products<1, false>);
    case 2: return inv ? go(k_coupling_products<2, true>) : go(k_coupling_products<2, false>);
    case 3: return inv ? go(k_coupling_products<3, true>) : go(k_coupling_products<3, false>);
    case 4: return inv ? go(k_coupling_products<4, true>) : go(k_coupling_products<4, false>);
    default: return LS_GPU_ERR_INVALID;
  }
}

}  // namespace lsg
