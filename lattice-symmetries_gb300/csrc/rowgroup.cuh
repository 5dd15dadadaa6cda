// rowgroup.cuh -- the orbit scan with one lane per generated element (bases with lattice
// symmetries).
//
// A warp takes R consecutive rows at a time.  Per group of rows it
//   1. keeps g.a of every group element for each row in shared memory (the rows are sorted, so a
//      row's images follow from the previous row's by the few bits that changed),
//   2. lists the matching terms of all rows (one ballot per 32 term slots and row),
//   3. resolves them, one element (KEEP = false: two) per lane at a time: the lane walks the group elements,
//      forms the candidates g.a ^ g.x from the row's images and the image of the element's flip
//      pattern (a table over the distinct patterns), keeps the minimum and the element that
//      reached it, and looks the representatives up,
//   4. hands every resolved element {column index, coefficient word} to the caller.
//
// What bounds it and why this split.  With one warp per element every element costs the warp-wide
// minimum, the tie pass, the term decoding and the bookkeeping of 32 lanes (~100 warp
// instructions, whatever the group's size); with one lane per element these are shared by 32
// elements and the scan is left with two 32-bit shared-memory loads, an XOR and half a
// three-input minimum (with spin inversion also half a maximum) per group element and 32
// elements.  Lanes take elements in one of two ways.  KEEP = false (one column): 32 / R lanes share
// a row and sum their own elements in registers; a lane's two elements read the row's images once.
// KEEP = true (several columns): the elements of all R rows are dealt to the lanes in the order of
// the term slots, so that no lane idles (short rows filled only 70 % of the lanes the other way)
// and neighbouring lanes read neighbouring patterns (few bank conflicts), and go to shared memory.
//
// Measured (GB300, warp per row -> lane per element): T x C6 on 25 sites, 150 elements, 34.7e3 rows, 5
// complex columns 1328 -> 125 us (the ragged block also scans once instead of twice; 137 us with N32);
// 28-site chain, 56 images, 16 columns 3609 -> 1540 us; 4x4 Hubbard, 128 elements, 8 columns 6724 ->
// 2358 us; 6x6 torus, 576 images, one column 169.1 -> 73.5 ms (85.2 ms with prefix minima instead of
// bit planes).
//
// Modes.  N32 (states of at most 32 bits): candidates are whole states, so their minimum is the
// representative; the scan remembers the chunk of 8 elements that first reached it and a second
// look at that chunk finds the element.
// Bit planes (any width; large groups): for each of the top positions of the image one bit per
// group element, 32 elements to a word -- linear over XOR like the images themselves, so the same
// row and pattern tables hold them.  A lane keeps the set of elements that can still be minimal (W
// words in registers) and goes down the positions: where some of them have a 0 there, those stay.
// With spin inversion the planes are taken relative to the top position's, which flips every image
// to its smaller form.  That is one XOR-AND, half an OR and a select per word and position, for about
// log2 |G| + 4 positions (13 x 9 words for 288 elements, where a minimum over 16-bit prefixes
// took 144 words at three operations and half-word bookkeeping); the one or two elements left are
// compared by their remaining bits, gathered through a byte table of source positions.
//
// The order of the tie-break (lowest element, unflipped first) is that of the packed kernels.
#pragma once

#include "matvec_impl.cuh"

namespace lsg {

// Scan modes: N32, or bit planes of W words per position (W the mode's value).
constexpr int kModeN32 = 0;
// Elements that a lane takes at a time (6x6 torus, one column: 2 against 1 is 85.2 against 86.4 ms; 4x4
// Hubbard, 8 columns: 1 / 2 / 4 at a time 2444 / 2534 / 3600 us); the sets of two elements on planes
// of 16 words do not fit the registers.
template <int MODE, bool KEEP>
constexpr int kLaneElements = KEEP || MODE > 9 ? 1 : 2;

// Shared-memory layout and shape of a row-group kernel (bytes from the start of dynamic shared
// memory; w_* relative to a warp's area).
struct RowsLayout {
  int threads, R, lanes_per_row, lane_shift, cap, T, n_slots, slot_blocks, n_pat, n_diag_blocks;
  int G, words, stride, site_words;  // words of g-images per row / pattern, their padded strides
  int planes, nlow, nlow_pad, perm_stride;  // bit planes: positions, bits below them, rounded up to 4, bytes
                                            // of an element's source positions
  uint32_t off_site, off_img, off_perm, off_coef, off_sm, off_sl1, off_sl2, off_st, off_ti, off_ts, off_xm;
  uint32_t off_dm, off_dr, off_ds, off_db, off_dv, off_fs, off_sectors, off_first, off_warp;
  uint32_t warp_bytes, w_ent, w_list, w_a, w_sets;  // w_list: KEEP the elements' positions in scan order
  uint32_t total;
};

__device__ __forceinline__ uint64_t shfl_u64(uint64_t v, int src) {
  return ((uint64_t)__shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src) << 32) |
         __shfl_sync(0xffffffffu, (uint32_t)v, src);
}

// States as the tables hold them: 32-bit words where they fit.
template <int MODE>
struct StateWord {
  using T = uint64_t;
};
template <>
struct StateWord<kModeN32> {
  using T = uint32_t;
};
__device__ __forceinline__ uint32_t shfl_state(uint32_t v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ uint64_t shfl_state(uint64_t v, int src) { return shfl_u64(v, src); }
__device__ __forceinline__ int popc_state(uint32_t v) { return __popc(v); }
__device__ __forceinline__ int popc_state(uint64_t v) { return __popcll(v); }
__device__ __forceinline__ int low_bit(uint32_t v) { return __ffs(v) - 1; }
__device__ __forceinline__ int low_bit(uint64_t v) { return __ffsll((long long)v) - 1; }

// One warp's view of the tables and its own area.
template <int MODE, bool INV, bool FERMI, bool KEEP>
struct RowGroup {
  static constexpr unsigned FULL = 0xffffffffu;
  using State = typename StateWord<MODE>::T;
  static constexpr uint32_t kAbsent = 0xffffffffu;  // column index of an element outside the basis

  const RowsLayout& L;
  const MatvecProblem& p;
  unsigned char* smem;
  uint32_t* ga;       // [R][stride]
  uint16_t* list;     // [R][cap]: the terms of each row's elements; KEEP: positions in entries, in scan order
  uint2* entries;     // KEEP: [R][cap], {term | row << 16, -} when listed, {column, coefficient word} resolved
  State* rows;        // [R] row states
  uint32_t* sets;     // bit planes: [W][32] the lanes' sets of minimal elements
  uint32_t img_s, ga_s;
  int lane;
  State prev;         // state whose images are in row `prev_row` of ga
  int prev_row;
  bool minus;         // the spin inversion's character is -1
  // per group of rows: lane r < nr holds row r's state, inverse norm and number of elements
  State a_l;
  double inv_l;
  int cnt_l;
  int nr;
  int total;          // KEEP: elements of all rows

  __device__ __forceinline__ RowGroup(const RowsLayout& L_, const MatvecProblem& p_, unsigned char* s)
      : L(L_), p(p_), smem(s) {
    unsigned char* w = s + L.off_warp + (threadIdx.x >> 5) * L.warp_bytes;
    ga = (uint32_t*)w;
    entries = (uint2*)(w + L.w_ent);
    list = (uint16_t*)(w + L.w_list);
    rows = (State*)(w + L.w_a);
    sets = (uint32_t*)(w + L.w_sets) + (threadIdx.x & 31);
    img_s = (uint32_t)__cvta_generic_to_shared(s + L.off_img);
    ga_s = (uint32_t)__cvta_generic_to_shared(ga);
    lane = threadIdx.x & 31;
    prev = 0;
    prev_row = -1;
    minus = p.group.spin_inversion == -1;
  }

  template <typename T>
  __device__ __forceinline__ const T* tab(uint32_t off) const {
    return reinterpret_cast<const T*>(smem + off);
  }

  // Fills the block's tables; the caller synchronises the block afterwards.
  __device__ __forceinline__ static void stage(const RowsLayout& L, const MatvecProblem& p, unsigned char* smem) {
    const int G = L.G, nb = p.group.n_bits;
    const int tid = threadIdx.x, nt = blockDim.x;
    uint32_t* site = (uint32_t*)(smem + L.off_site);
    if constexpr (MODE == kModeN32) {
#pragma unroll 4
      for (int i = tid; i < nb * L.site_words; i += nt) {
        const int b = i / L.site_words, w = i - b * L.site_words;
        site[i] = w < L.words ? (uint32_t)__ldg(p.group.onehot + b * G + (w < G ? w : 0)) : 0u;
      }
    } else {
      // word w of plane q: which of 32 elements move site b to the plane's position (or, with spin
      // inversion, to the top).  A warp reads the 32 images once and ballots plane by plane.
      const int ln = tid & 31, top = nb - 1;
#pragma unroll 2
      for (int i = tid >> 5; i < nb * MODE; i += nt >> 5) {
        const int b = i / MODE, w = i - b * MODE, g = 32 * w + ln;
        const uint64_t image = g < G ? __ldg(p.group.onehot + b * G + g) : 0ull;
        for (int q = 0; q < L.planes; ++q) {
          const uint32_t bit = (uint32_t)(image >> (top - q - (INV ? 1 : 0))) ^ (INV ? (uint32_t)(image >> top) : 0u);
          const unsigned v = __ballot_sync(FULL, bit & 1u);
          if (ln == 0) site[b * L.site_words + q * MODE + w] = v;
        }
      }
      for (int i = tid; i < nb * (L.site_words - L.words); i += nt) {
        const int pad = L.site_words - L.words, b = i / pad;
        site[b * L.site_words + L.words + i - b * pad] = 0u;
      }
    }
    if constexpr (MODE != kModeN32) {
      // source positions of an element's low bits, most significant first, after bits that are zero
      // in every state (position 63)
      unsigned char* perm = smem + L.off_perm;
      // and, last, of its top bit
      const int pad = L.nlow_pad - L.nlow;
      for (int i = tid; i < G * pad; i += nt) perm[(i / pad) * L.perm_stride + i % pad] = 63;
      for (int i = tid; i < nb * G; i += nt) {
        const int b = i / G, g = i - b * G;
        const int to = __ffsll((long long)__ldg(p.group.onehot + i)) - 1;
        if (to < L.nlow) perm[g * L.perm_stride + (L.nlow_pad - 1 - to)] = (unsigned char)b;
        if (to == nb - 1) perm[g * L.perm_stride + L.nlow_pad] = (unsigned char)b;
      }
    }
    auto states = [&](uint32_t off, const uint64_t* src, int n) {
      State* dst = (State*)(smem + off);
      for (int i = tid; i < n; i += nt) dst[i] = (State)__ldg(src + i);
    };
    states(L.off_sm, p.off.rows.sm, 32 * L.slot_blocks);
    states(L.off_sl1, p.off.rows.sl1, 32 * L.slot_blocks);
    states(L.off_sl2, p.off.rows.sl2, 32 * L.slot_blocks);
    uint32_t* st = (uint32_t*)(smem + L.off_st);
    for (int i = tid; i < 32 * L.slot_blocks; i += nt) st[i] = __ldg(p.off.rows.st + i);
    uint32_t* ti = (uint32_t*)(smem + L.off_ti);
    for (int i = tid; i < L.T; i += nt) ti[i] = __ldg(p.off.rows.tinfo + i);
    states(L.off_ts, p.off.s, L.T);
    states(L.off_xm, p.off.rows.xmask, L.n_pat);
    states(L.off_dm, p.diag.rows.sm, 32 * L.n_diag_blocks);
    states(L.off_dr, p.diag.rows.sl1, 32 * L.n_diag_blocks);
    states(L.off_ds, p.diag.rows.sl2, 32 * L.n_diag_blocks);
    uint2* db = (uint2*)(smem + L.off_db);
    for (int i = tid; i < L.n_diag_blocks; i += nt)
      db[i] = make_uint2(__ldg(p.diag.rows.st + i), __ldg(p.diag.rows.tinfo + i));
    stage_d2((double2*)(smem + L.off_dv), p.diag.rows.cval, p.diag.rows.n_cls);
    if constexpr (FERMI) states(L.off_fs, p.group.fsign_packed, nb * 32 * p.group.gpl);
    __syncthreads();
    // images of the flip patterns, from those of their sites
    uint32_t* img = (uint32_t*)(smem + L.off_img);
    const State* xm = (const State*)(smem + L.off_xm);
    for (int i = tid; i < L.n_pat * L.words; i += nt) {
      const int x = i / L.words, w = i - x * L.words;
      uint32_t v = 0;
      for (State m = xm[x]; m != 0; m &= m - 1) v ^= site[low_bit(m) * L.site_words + w];
      img[x * L.stride + w] = v;
    }
  }

  // (-1)^n of group element g on the occupied orbitals of `state`: the reversed pairs
  // sum_k popcount(state & L_g[k]) over occupied k have the parity of state & XOR_k L_g[k].
  __device__ __forceinline__ uint32_t fermion_sign(uint32_t g, State state) const {
    const State* l = tab<State>(L.off_fs) + g;
    const int stride = 32 * p.group.gpl;
    State crossed = 0;
    for (State m = state; m != 0; m &= m - 1) crossed ^= l[low_bit(m) * stride];
    return (uint32_t)popc_state((State)(state & crossed));
  }

  // Forgets the images of earlier rows (before a block of rows that does not follow them).
  __device__ __forceinline__ void restart() {
    prev = 0;
    prev_row = -1;
  }

  // Steps 1 and 2 for the rows [row0, row0 + n).
  __device__ __forceinline__ void load_rows(const DeviceIndex& ix, int64_t row0, int n) {
    nr = n;
    __syncwarp();  // the previous group's readers are done
    a_l = lane < nr ? (State)__ldg(ix.reps + row0 + lane) : (State)0;
    inv_l = lane < nr ? __ldg(ix.inv_norms + row0 + lane) : 0.0;
    cnt_l = 0;
    if (lane < nr) rows[lane] = a_l;
    const uint32_t site_s = (uint32_t)__cvta_generic_to_shared(smem + L.off_site) + 4u * (uint32_t)lane;
    const uint32_t row_bytes = 4u * (uint32_t)L.site_words;
#pragma unroll 1
    for (int r = 0; r < nr; ++r) {
      const State a = shfl_state(a_l, r);
      const State diff = a ^ prev;
      // four words per lane at a time; site rows are padded to whole warps, image rows are not
      for (int w0 = 0; w0 < L.words; w0 += 128) {
        const int left = L.words - w0;  // uniform
        const int wl = w0 + lane;
        uint32_t v[4] = {0, 0, 0, 0};
        if (prev_row >= 0) {
          const uint32_t* g = ga + prev_row * L.stride + wl;
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = lane + 32 * k < left ? g[32 * k] : 0u;
        }
        const uint32_t base = site_s + 4u * (uint32_t)w0;
        
#pragma unroll 1
        for (State d = diff; d != 0;) {
          const uint32_t s0 = base + (uint32_t)low_bit(d) * row_bytes;
          d &= d - 1;
          const bool pair = d != 0;  // uniform
          const uint32_t s1 = base + (pair ? (uint32_t)low_bit(d) : 0u) * row_bytes;
          d &= pair ? d - 1 : (State)0;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (32 * k < left) v[k] ^= lds_u32(s0 + 128 * k) ^ (pair ? lds_u32(s1 + 128 * k) : 0u);
        }
        uint32_t* g = ga + r * L.stride + wl;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (lane + 32 * k < left) g[32 * k] = v[k];
      }
      prev = a;
      prev_row = r;
    }
    // zero-norm rows take no part (their outputs are zero)
    const unsigned live = __ballot_sync(FULL, inv_l != 0.0);
    const unsigned below = (1u << lane) - 1u;
    total = 0;
    for (int b = 0; b < L.slot_blocks; ++b) {
      const State m = tab<State>(L.off_sm)[32 * b + lane];
      const State l1 = tab<State>(L.off_sl1)[32 * b + lane], l2 = tab<State>(L.off_sl2)[32 * b + lane];
      const uint32_t t12 = tab<uint32_t>(L.off_st)[32 * b + lane];
#pragma unroll 1
      for (int r = 0; r < nr; ++r) {
        const State x = shfl_state(a_l, r) & m;
        const bool h1 = x == l1, h2 = x == l2;
        const bool hit = (h1 || h2) && ((live >> r) & 1u);
        const unsigned hits = __ballot_sync(FULL, hit);
        const int before = __shfl_sync(FULL, cnt_l, r);
        if (hit) {
          const int rank = __popc(hits & below), at = r * L.cap + before + rank;
          const uint32_t t = h1 ? t12 & 0xffffu : t12 >> 16;
          if constexpr (KEEP) {
            entries[at].x = t | ((uint32_t)r << 16);
            list[total + rank] = (uint16_t)at;
          } else {
            list[at] = (uint16_t)t;
          }
        }
        if (lane == r) cnt_l += __popc(hits);
        if (KEEP) total += __popc(hits);
      }
    }
    __syncwarp();
  }

  // What pass 1 leaves for pass 2 of an element.  N32: the minimum and the word of its first chunk;
  // bit planes: the top bits of the minimum and the elements that have them.
  struct Found {
    uint32_t best, at;
    uint32_t set[MODE == kModeN32 ? 1 : MODE];
  };

  // Pass 1 for E elements: images of their rows at gp (one row without KEEP), of their patterns at ip.
  template <int E>
  __device__ __forceinline__ void first_pass(const uint32_t (&gp)[E], const uint32_t (&ip)[E], Found (&found)[E]) const {
    if constexpr (MODE == kModeN32) {
      const uint32_t flip = (uint32_t)p.group.flip;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        found[e].best = 0xffffffffu;
        found[e].at = 0;
      }
      for (uint32_t c = 0; c < (uint32_t)L.words; c += 8) {
        uint32_t a[8];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if (KEEP || e == 0) {
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = lds_u32_volatile(gp[e] + 4 * (c + k));
          }
          uint32_t h[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) h[k] = a[k] ^ lds_u32(ip[e] + 4 * (c + k));
          uint32_t mn = h[0], mx = h[0];
#pragma unroll
          for (int k = 1; k < 8; ++k) {
            mn = min(mn, h[k]);
            if (INV) mx = max(mx, h[k]);
          }
          if (INV) mn = min(mn, flip ^ mx);
          if (mn < found[e].best) {
            found[e].best = mn;
            found[e].at = c;
          }
        }
      }
    } else {
      constexpr int W = MODE;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        found[e].best = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int left = L.G - 32 * w;
          found[e].set[w] = left >= 32 ? ~0u : (left > 0 ? (1u << left) - 1u : 0u);
        }
      }
#pragma unroll 1  // (the instruction cache)
      for (int q = 0; q < L.planes; ++q) {
        uint32_t a[W];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if (KEEP || e == 0) {
#pragma unroll
            for (int w = 0; w < W; ++w) a[w] = lds_u32_volatile(gp[e] + 4 * (q * W + w));
          }
          uint32_t z[W], any = 0;  // the elements with a 0 here
#pragma unroll
          for (int w = 0; w < W; ++w) {
            z[w] = found[e].set[w] & ~(a[w] ^ lds_u32(ip[e] + 4 * (q * W + w)));
            any |= z[w];
          }
#pragma unroll
          for (int w = 0; w < W; ++w) found[e].set[w] = any != 0 ? z[w] : found[e].set[w];
          found[e].best = 2 * found[e].best + (any != 0 ? 0u : 1u);
        }
      }
    }
  }

  // The representative of one element and its key 2 * group element + flipped, from pass 1.
  __device__ __forceinline__ uint64_t second_pass(uint32_t gp, uint32_t ip, const Found& found, uint64_t beta,
                                                  uint32_t* key) const {
    if constexpr (MODE == kModeN32) {
      const uint32_t flip = (uint32_t)p.group.flip;
      const uint32_t at = found.at;
      uint32_t k0 = 0;
#pragma unroll
      for (int k = 7; k >= 0; --k) {
        const uint32_t h = lds_u32_volatile(gp + 4 * (at + k)) ^ lds_u32(ip + 4 * (at + k));
        if (INV && (h ^ flip) == found.best) k0 = 2 * k + 1;
        if (h == found.best) k0 = 2 * k;
      }
      *key = 2 * at + k0;
      return found.best;
    } else {
      // the remaining elements compared by their low bits (6x6 torus, 13 planes: 1.15 per target,
      // the slowest of 32 lanes has 2.5)
      uint32_t words = 0;  // of the set that are not empty
#pragma unroll
      for (int w = 0; w < MODE; ++w) {
        sets[32 * w] = found.set[w];
        if (found.set[w] != 0) words |= 1u << w;
      }
      uint32_t word = 0, base = 0, win = 0;
      uint64_t low = ~0ull;
      const uint32_t perm_s = (uint32_t)__cvta_generic_to_shared(smem + L.off_perm);
#pragma unroll 1
      do {
        if (word == 0 && words != 0) {
          base = (uint32_t)__ffs(words) - 1;
          words &= words - 1;
          word = sets[32 * base];
        }
        if (word != 0) {
          const uint32_t g = 32 * base + (uint32_t)__ffs(word) - 1;
          word &= word - 1;
          const uint32_t ps = perm_s + g * (uint32_t)L.perm_stride;
          uint32_t hi = 0, lo = 0;  // the low bits, most significant first
          int b = 0;
#pragma unroll 1
          for (; b < L.nlow_pad - 32; b += 4) {
            const uint32_t src = lds_u32(ps + b);
#pragma unroll
            for (int i = 0; i < 4; ++i) hi = 2 * hi + ((uint32_t)(beta >> __byte_perm(src, 0, 0x4440 + i)) & 1u);
          }
#pragma unroll 1
          for (; b < L.nlow_pad; b += 4) {
            const uint32_t src = lds_u32(ps + b);
#pragma unroll
            for (int i = 0; i < 4; ++i) lo = 2 * lo + ((uint32_t)(beta >> __byte_perm(src, 0, 0x4440 + i)) & 1u);
          }
          uint64_t v = ((uint64_t)hi << 32) | lo;
          uint32_t flipped = 0;
          if (INV) {
            flipped = (uint32_t)(beta >> (lds_u32(ps + L.nlow_pad) & 0xffu)) & 1u;
            if (flipped) v ^= (1ull << L.nlow) - 1;
          }
          // elements ascend: the first of equal images stays
          if (v < low) {
            low = v;
            win = 2 * g + flipped;
          }
        }
      } while (__any_sync(FULL, (word | words) != 0));
      *key = win;
      return ((uint64_t)found.best << L.nlow) | low;
    }
  }

  // Column indices of E representatives (kAbsent: not in the basis or !ok), the lookups side by side.
  template <int E>
  __device__ __forceinline__ void lookup(const DeviceIndex& ix, const uint64_t (&rep)[E], const bool (&ok)[E],
                                         uint32_t (&j)[E], const uint64_t* __restrict__ binom) const {
    if (ix.suffix16 != nullptr && !ix.identity && !ix.combinadic) {
      uint32_t n[E];
      uint32_t longest = 0;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const bool in = ok[e] && rep[e] <= ix.max_state;
        const uint64_t b = in ? rep[e] >> ix.shift : 0ull;
        j[e] = __ldg(ix.offsets + b);
        n[e] = __ldg(ix.offsets + b + 1);
        n[e] = in ? n[e] - j[e] : 0u;
      }
      const uint32_t low = (1u << ix.shift) - 1u;
#pragma unroll
      for (int e = 0; e < E; ++e) longest = max(longest, n[e]);
#pragma unroll 1
      while (longest > 1) {
        longest = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if (n[e] > 1) {
            const uint32_t half = n[e] >> 1;
            if (__ldg(ix.suffix16 + (size_t)j[e] + half) <= ((uint32_t)rep[e] & low)) j[e] += half;
            n[e] -= half;
          }
          longest = max(longest, n[e]);
        }
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const bool there = n[e] != 0 && __ldg(ix.suffix16 + (size_t)(n[e] != 0 ? j[e] : 0u)) == ((uint32_t)rep[e] & low);
        if (!there) j[e] = kAbsent;
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int64_t i = ok[e] ? mv_index_lookup(ix, rep[e], binom) : -1;
        j[e] = i >= 0 ? (uint32_t)i : kAbsent;
      }
    }
  }

  // Resolves E elements of this lane: terms term[e] of rows row[e] (one row without KEEP), where
  // ok[e]; columns (kAbsent for elements outside the basis or !ok) and coefficient words in j and w.
  template <int E>
  __device__ __forceinline__ void resolve_some(const DeviceIndex& ix, const uint32_t (&row)[E],
                                               const uint32_t (&term)[E], bool (&ok)[E], uint32_t (&j)[E],
                                               uint32_t (&w)[E], int* __restrict__ err,
                                               const uint64_t* __restrict__ binom) {
    const uint32_t stride = 4u * (uint32_t)L.stride;
    uint32_t gp[E], ip[E];
    Found found[E];
    uint64_t rep[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      gp[e] = ga_s + row[e] * stride;
      ip[e] = img_s + (tab<uint32_t>(L.off_ti)[term[e]] & 0xffffu) * stride;
    }
    first_pass<E>(gp, ip, found);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint32_t info = tab<uint32_t>(L.off_ti)[term[e]];
      const State beta = rows[row[e]] ^ tab<State>(L.off_xm)[info & 0xffffu];
      uint32_t key;
      rep[e] = second_pass(gp[e], ip[e], found[e], beta, &key);
      if (ok[e] && (info & kRowTermNeedsCheck) && !constraint_ok(p.constraint, beta)) {
        ok[e] = false;
        atomicOr(err, 1);
      }
      uint32_t g = key >> 1;
      if (g >= (uint32_t)L.G) g = 0;  // padding repeats element 0
      uint32_t neg = (uint32_t)popc_state((State)(beta & tab<State>(L.off_ts)[term[e]])) ^ (info >> 31);
      if (INV && minus) neg ^= key;
      if constexpr (FERMI) neg ^= fermion_sign(g, beta);
      w[e] = (((info >> 16) & 0xffu) * (uint32_t)L.G + g) | (neg << 31);
    }
    lookup<E>(ix, rep, ok, j, binom);
  }

  // Step 3 without KEEP: take(columns, coefficient words, terms) for the elements of this lane's row
  // lane >> lane_shift.
  template <typename Take>
  __device__ __forceinline__ void resolve(const DeviceIndex& ix, int* __restrict__ err,
                                          const uint64_t* __restrict__ binom, Take&& take) {
    constexpr int E = kLaneElements<MODE, KEEP>;
    const int r = lane >> L.lane_shift, sub = lane & (L.lanes_per_row - 1);
    const int cnt = __shfl_sync(FULL, cnt_l, r);
    const int most = (int)__reduce_max_sync(FULL, (unsigned)cnt);
    for (int s = 0; s < most; s += E * L.lanes_per_row) {
      uint32_t row[E], term[E], j[E], w[E];
      bool ok[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int i = s + sub + e * L.lanes_per_row;
        row[e] = (uint32_t)min(r, nr - 1);
        ok[e] = i < cnt;
        term[e] = ok[e] ? list[r * L.cap + i] : 0u;
      }
      resolve_some<E>(ix, row, term, ok, j, w, err, binom);
      take(j, w, term);
    }
  }

  // Step 3 with KEEP: the resolved elements replace the listed ones in entries.
  __device__ __forceinline__ void resolve(const DeviceIndex& ix, int* __restrict__ err,
                                          const uint64_t* __restrict__ binom) {
    constexpr int E = kLaneElements<MODE, KEEP>;
    for (int s = 0; s < total; s += 32 * E) {
      uint32_t at[E], row[E], term[E], j[E], w[E];
      bool ok[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int i = s + lane + 32 * e;
        ok[e] = i < total;
        at[e] = list[min(i, total - 1)];
        const uint32_t v = entries[at[e]].x;
        row[e] = v >> 16;
        term[e] = v & 0xffffu;
      }
      __syncwarp();  // a clamped lane reads an element that its owner replaces
      resolve_some<E>(ix, row, term, ok, j, w, err, binom);
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (ok[e] || s + lane + 32 * e < total) entries[at[e]] = make_uint2(j[e], w[e]);
      __syncwarp();
    }
  }

  // Signed counts of the diagonal terms, class by class: each(class, count) with lane r < nr holding
  // row r's count.
  template <typename Each>
  __device__ __forceinline__ void diagonal_counts(Each&& each) const {
    int n_l = 0;
    for (int b = 0; b < L.n_diag_blocks; ++b) {
      const State m = tab<State>(L.off_dm)[32 * b + lane], k = tab<State>(L.off_dr)[32 * b + lane];
      const State s = tab<State>(L.off_ds)[32 * b + lane];
      const uint2 info = tab<uint2>(L.off_db)[b];  // {signs of the 32 terms, class | last block of it << 31}
#pragma unroll 1
      for (int r = 0; r < nr; ++r) {
        const State a = shfl_state(a_l, r);
        const bool hit = (a & m) == k;
        const bool odd = popc_state((State)(a & s)) & 1;
        const unsigned hits = __ballot_sync(FULL, hit);
        const unsigned minus_hits = (__ballot_sync(FULL, odd) ^ info.x) & hits;
        if (lane == r) n_l += __popc(hits) - 2 * __popc(minus_hits);
      }
      if (info.y >> 31) {
        each(info.y & 0xffffu, n_l);
        n_l = 0;
      }
    }
  }

  // The diagonal elements: lane r < nr returns row r's.
  __device__ __forceinline__ double2 diagonal() const {
    double2 d = make_double2(0.0, 0.0);
    diagonal_counts([&](uint32_t cls, int n) {
      const double2 v = tab<double2>(L.off_dv)[cls];
      d.x = fma((double)n, v.x, d.x);
      d.y = fma((double)n, v.y, d.y);
    });
    return d;
  }
};

}  // namespace lsg
