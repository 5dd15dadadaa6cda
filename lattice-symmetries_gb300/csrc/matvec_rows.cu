// matvec_rows.cu -- y = H x from the row-group orbit scan (rowgroup.cuh, rowsums.cuh): projected bases, real
// or complex vectors, up to 16 complex or 32 real columns per launch.  The choice of mode and shape,
// and the kernels of the N32 mode; those of the bit planes are in matvec_rows_w*.cu.
#include <algorithm>
#include <cmath>

#include "rowkernel.cuh"

namespace lsg {

// Planes of the bit-plane scan (of `words` words): enough for about 2^-4 ties per target, log2 |G| + 4
// bits at half filling.  Away from half filling a bit says less: on average its entropy, but the smallest
// images of a dilute orbit begin with zeros, which say -log2(1 - f) each; the mean of the two serves
// best where the patterns' table leaves room for it (half the shared memory; with 16 words on the 6x6
// torus under C6v it does not: 7 up 711 / 1492).  us for one real column, entropy alone / mean:
// 6x6 torus, 288 images, 7 of 36 spins up 194 / 148, 8 up 436 / 343; 7x7 translations, 6 of 49 up
// 726 / 529; 48-site chain, 5 up 511 / 383.
static int rows_planes(const MatvecProblem& p, int words) {
  const int n = p.group.n_bits, inv = p.group.spin_inversion != 0 ? 1 : 0;
  double f = 0.5;
  if (p.constraint.kind == 1) f = (double)p.constraint.w0 / n;
  if (p.constraint.kind == 2) f = (double)(p.constraint.w0 + p.constraint.w1) / n;
  const double entropy = f <= 0.0 || f >= 1.0 ? 0.0 : -(f * std::log2(f) + (1.0 - f) * std::log2(1.0 - f));
  auto planes = [&](double bits) {
    const double want = std::log2((double)std::max(p.group.n_elems, 1)) / std::max(bits, 0.2) + 4.0;
    return std::max(1, std::min({(int)std::ceil(want), n - inv, 32}));
  };
  const int least = planes(entropy);
  if (f <= 0.0 || f >= 0.5) return least;
  const int room = (int)(kMaxDynamicSmem / 2 / ((size_t)std::max(p.off.rows.n_pat, 1) * words * 4));
  return std::max(least, std::min(planes(0.5 * (entropy - std::log2(1.0 - f))), room));
}

// Dynamic shared memory of a row-group kernel (the coupling products keep 2.2 KB more, statically).
constexpr size_t kRowsSmem = kMaxDynamicSmem - 4096;

// Shared memory that leaves 60 KB of L1 for the gathers instead of 28 KB.  One column scatters its
// reads of x and of the index: 6x6 torus, 4 rows per warp, 20 warps within this 73.5 ms, 24 warps
// beyond it 80.5 ms (18 and 22 warps, which load the schedulers unevenly, 80.8 and 83.3 ms).
constexpr size_t kRowsSmemL1 = 194 * 1024;

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
  const int n = p.group.n_bits, inv = p.group.spin_inversion != 0 ? 1 : 0;
  if (mode == kModeN32) {
    L.words = (L.G + 7) / 8 * 8;
  } else {
    L.planes = rows_planes(p, mode);
    L.nlow = n - inv - L.planes;
    L.nlow_pad = (L.nlow + 3) / 4 * 4;
    const int pw = L.nlow_pad / 4 + 1;  // and the top bit's source
    L.perm_stride = 4 * (pw % 2 ? pw : pw + 1);
    L.words = L.planes * mode;
  }
  L.stride = L.words | 1;  // odd: patterns (and rows) next to each other fall into different banks
  L.site_words = (L.words + 31) / 32 * 32;
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
  L.off_perm = take((size_t)L.G * L.perm_stride);
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
  L.w_sets = take(mode == kModeN32 ? 0 : (size_t)mode * 128);
  L.warp_bytes = o;
  L.total = L.off_warp + (uint32_t)warps * L.warp_bytes;
  *out = L;
  return L.total <= kRowsSmem;
}

// The scan modes, and which of them `p` can run.
constexpr int kRowModes[] = {kModeN32, 2, 5, 9, 16};
static bool rows_mode_allowed(const MatvecProblem& p, int mode) {
  const int n = p.group.n_bits, W = (p.group.n_elems + 31) / 32;
  if (p.group.n_elems < 1 || !p.off.rows.ok || !p.diag.rows.ok) return false;
  if (p.group.fermionic && (p.group.gpl < 1 || p.group.gpl > 4)) return false;  // as the packed kernels
  if (mode == kModeN32) return n <= 32;
  if (n < 2 || n > 63 || W > mode) return false;
  for (const int m : kRowModes)
    if (m != kModeN32 && m >= W) return m == mode;  // the smallest that holds the group
  return false;
}

// About the instructions of one target's scan (32 targets at a time): the line between N32 and bit
// planes.  150 elements on 25 sites: 137 us by N32, 125 by planes; 128 elements of the 4x4 Hubbard
// model 2362 and 2764 us; 56 images of the 28-site chain 1544 and 1581 us; 28 elements of the ladder
// 4.4 and 6.2 ms a training step.  Two species make many ties
// among the top bits, which cost bit planes a round each.
static double rows_scan_cost(const MatvecProblem& p, int mode) {
  const int inv = p.group.spin_inversion != 0 ? 1 : 0;
  if (mode == kModeN32) return (p.group.n_elems + 7) / 8 * 8 * (3.5 + inv) + 60.0;
  const int planes = rows_planes(p, mode);
  return planes * (4.5 * mode + 5.0) + (p.constraint.kind == 2 ? 8.0 : 2.5) * (30.0 + 4.0 * (p.group.n_bits - planes));
}

constexpr int64_t kLeastWarps = 4;

bool rows_fit(const MatvecProblem& p, int n_sectors) {
  RowsLayout L;
  if (p.projection != 2) return false;
  for (const int m : kRowModes)
    if (rows_mode_allowed(p, m) && rows_layout(p, m, n_sectors > 0 || p.real_elements == 0, true, n_sectors, (int)kLeastWarps, 1, &L)) return true;
  return false;
}

// The modes that p can run, N32 and the group's bit planes, the cheaper scan first; their number.
static int rows_modes(const MatvecProblem& p, int (&modes)[2]) {
  int n = 0;
  for (const int m : kRowModes)
    if (rows_mode_allowed(p, m)) modes[n++] = m;
  if (n == 2 && rows_scan_cost(p, modes[1]) < rows_scan_cost(p, modes[0])) std::swap(modes[0], modes[1]);
  return n;
}

// Few rows: at most about one per warp of the packed kernels, which then take no longer than a row's
// latency, while here the tables of every CTA and the ties of a lane's elements do.  us of one product
// (k columns in one launch), a warp per row / a lane per element: 6x6 torus, 288 images, 3 up (40 rows),
// one real column 28 / 91, 6 up (7278 rows) 58 / 76; C6v, 432 images, 5 up (964 rows), 16 complex
// columns 68 / 210; 48-site chain, 4 up (4060 rows), one column 26 / 42; 4D hypercube, 384 images,
// 58 rows 42 / 97; 4x4 Hubbard, 128 images, 2 + 2 (2506 rows), 16 columns 30 / 40.
// Not so
//  - up to 32 bits for one column (24 sites, 48 images: 25 / 20) or a dozen rows (4x4 torus, 10 rows 20.5 / 18);
//  - for small groups (48 sites, 3 images, 5776 rows: 36 / 24) or one column of many terms (36 sites, all
//    pairs, 4 up: 94 / 65);
//  - where slots of the packed kernels are empty: they repeat element 0 and tie with it (216 images
//    on 6x6, 9212 rows, 165 / 98; 5x5, 150 images, 98 rows 55 / 26).
// slots: of the packed kernels, or 0 where only the kernel without shared tables could run (one column).
bool rows_few(const MatvecProblem& p, int k, int slots) {
  const int64_t sms = num_sms(), n = p.n_rows;
  const int G = p.group.n_elems;
  const bool wide = p.group.n_bits > 32, full = G == slots;
  if (n > 48 * sms || (k == 1 && (p.off.rows.n_slots > 256 || (!wide && G <= 32 * 9)))) return false;
  int modes[2];
  if (rows_modes(p, modes) == 0) return false;
  if (slots == 0) return modes[0] != kModeN32 && k == 1 && n <= 16 * sms;
  if (modes[0] == 16) return n <= (full ? 48 : 32) * sms;
  if (!wide) return k > 1 && G > 64 && full && n * G > 12288 && n <= 32 * sms;
  if (G <= 32) return false;
  if (G <= 128) return n <= 32 * sms;
  return n <= (full ? 48 : 4) * sms;
}

// Shape for p (rows_fit): the cheapest number of rows per warp among those that leave enough warps
// their area.
static bool rows_shape(const MatvecProblem& p, bool complex_elements, bool keep, int64_t n_rows, int n_sectors,
                       int max_warps, int sms, int* mode, RowsLayout* L) {
  int modes[2];
  const int n_modes = rows_modes(p, modes);
  for (int k = 0; k < n_modes; ++k) {
    const int m = modes[k];
    RowsLayout t[4];
    int warps[4];
    for (int i = 0; i < 4; ++i) {
      rows_layout(p, m, complex_elements, keep, n_sectors, 1, 8 >> i, &t[i]);
      auto fit = [&](size_t limit) -> int {
        const int64_t room = (int64_t)limit - t[i].off_warp;
        const int w = t[i].warp_bytes == 0 || room < 0 ? 0 : (int)std::min<int64_t>(max_warps, room / t[i].warp_bytes);
        return w >= 8 ? w / 4 * 4 : w;  // whole warps per scheduler
      };
      warps[i] = fit(kRowsSmem);
      if (!keep && fit(kRowsSmemL1) >= 20) warps[i] = fit(kRowsSmemL1);
    }
    for (const int enough : {keep ? 24 : 20, 16, 8, (int)kLeastWarps}) {
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
  // ... and enough of them to fill the tables in a few passes
  const int64_t staged = (int64_t)L.n_pat * L.words + (int64_t)p.group.n_bits * L.G;
  const int64_t per_sm = std::max<int64_t>({kLeastWarps, (groups + sms - 1) / sms, staged / 256});
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

static bool launch_plan(const MatvecProblem& p, Scalar sc, int k, RowsLaunch* q, int* col) {
  const bool cplx = sc == Scalar::Complex;
  *col = cplx ? (p.real_elements ? kColPair : kColComplex) : (k == 1 ? kColReal : kColPair);
  q->s.real_cols = (!cplx && *col == kColPair) ? k : 0;
  return rows_plan(p, *col, k, p.n_rows, 0, q);
}

int rows_mode(const MatvecProblem& p, Scalar sc, int k) {
  RowsLaunch q{};
  int col = 0;
  return launch_plan(p, sc, k, &q, &col) ? q.mode : -1;
}

int launch_rows(const MatvecProblem& p, Scalar sc, int k, const double* d_x, int64_t ldx, double* d_y, int64_t ldy,
                int* d_err, const uint64_t* binom, cudaStream_t st) {
  RowsLaunch q{};
  RowsSums& s = q.s;
  int col = 0;
  if (!launch_plan(p, sc, k, &q, &col)) return fail(LS_GPU_ERR_INVALID, "row-group tables do not fit in shared memory");
  s.x = d_x;
  s.xs = p.xs != nullptr ? p.xs : d_x;
  s.norms = p.xs != nullptr ? nullptr : p.index.norms;
  s.y = d_y;
  s.ldx = ldx;
  s.ldxs = p.xs != nullptr ? p.ldxs : ldx;
  s.ldy = ldy;
  switch (q.mode) {
    case kModeN32: return launch_rows_mode<kModeN32>(p, q, col, d_err, binom, st);
    case 2: return launch_rows_mode<2>(p, q, col, d_err, binom, st);
    case 5: return launch_rows_mode<5>(p, q, col, d_err, binom, st);
    case 9: return launch_rows_mode<9>(p, q, col, d_err, binom, st);
    default: return launch_rows_mode<16>(p, q, col, d_err, binom, st);
  }
}

template int launch_rows_mode<kModeN32>(const MatvecProblem&, const RowsLaunch&, int, int*, const uint64_t*, cudaStream_t);

}  // namespace lsg
