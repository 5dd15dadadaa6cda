// rowgroup.cuh -- the orbit scan with one lane per generated element (bases with lattice
// symmetries).
//
// A warp takes R consecutive rows at a time.  Per group of rows it
//   1. keeps g.a of every group element for each row in shared memory (the rows are sorted, so a
//      row's images follow from the previous row's by the few bits that changed),
//   2. lists the matching terms of all rows (one ballot per 32 term slots and row),
//   3. resolves 32 elements at a time, one per lane: the lane walks the group elements, forms the
//      candidates g.a ^ g.x from the row's images and the image of the term's flip pattern (a
//      table over the distinct patterns), keeps their minimum and the element that reached it,
//      and looks the representative up; the element becomes {column index, coefficient word},
//   4. hands the resolved elements, row by row, to the caller (sums over right-hand sides, inner
//      products).
//
// What bounds it and why this split.  With one warp per element every element costs the warp-wide
// minimum, the tie pass, the term decoding and the bookkeeping of 32 lanes (~100 warp
// instructions, whatever the group's size); with one lane per element these are shared by 32
// elements and the scan is left with two 32-bit shared-memory loads, an XOR and half a
// three-input minimum (with spin inversion also half a maximum) per group element and 32
// elements.
//
// Measured (GB300, warp per row before -> lane per element): T x C6 on 25 sites, 150 elements, 34.7e3
// rows, 5 complex columns 1330 -> 154 us (the ragged block also scans once instead of twice);
// 28-site chain, 56 images, 16 columns 3614 -> 1697 us; 4x4 Hubbard, 128 elements, 8 columns
// 6735 -> 2967 us; 6x6 torus, 576 images, one column 169.8 -> 120.6 ms.
//
// Modes.  N32 (states of at most 32 bits): candidates are whole states, so their minimum is the
// representative; the scan remembers the chunk of 8 elements that first reached it and a second
// look at that chunk finds the element.  P16 (any width from 17 bits; used when the N32 tables do
// not fit or the group is large): candidates are the top 16 bits of the states, two elements per
// 32-bit word, so that loads, XORs and minima cover two elements each; the chunks of 16 elements
// that reach the minimal prefix are kept as a bit mask and their matching elements (usually one)
// are compared by their remaining bits, gathered through a byte table of source positions.
//
// The order of the tie-break (lowest element, unflipped first) is that of the packed kernels.
#pragma once

#include "matvec_impl.cuh"

namespace lsg {

constexpr int kModeN32 = 0, kModeP16 = 1;

// Shared-memory layout and shape of a row-group kernel (bytes from the start of dynamic shared
// memory; w_* relative to a warp's area).
struct RowsLayout {
  int threads, R, cap, T, n_slots, slot_blocks, n_pat, n_diag_blocks;
  int G, words, stride, site_words;  // words of g-images per row / pattern, their padded strides
  int nlow, perm_stride;             // P16: bits below the 16-bit prefix, bytes per element
  uint32_t off_site, off_img, off_perm, off_coef, off_sm, off_sl1, off_sl2, off_st, off_ti, off_ts, off_xm;
  uint32_t off_dm, off_dr, off_ds, off_db, off_dv, off_fs, off_warp;
  uint32_t warp_bytes, w_ent, w_ord, w_a;
  uint32_t total;
};

__device__ __forceinline__ uint32_t vmin2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t vmax2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint64_t shfl_u64(uint64_t v, int src) {
  return ((uint64_t)__shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src) << 32) |
         __shfl_sync(0xffffffffu, (uint32_t)v, src);
}

// One warp's view of the tables and its own area.
template <int MODE, bool INV, bool FERMI>
struct RowGroup {
  static constexpr unsigned FULL = 0xffffffffu;
  static constexpr uint32_t kAbsent = 0xffffffffu;  // column index of an element outside the basis

  const RowsLayout& L;
  const MatvecProblem& p;
  unsigned char* smem;
  uint32_t* ga;       // [R][stride]
  uint2* entries;     // [R][cap]: {t | row << 16, -} when listed, {column, coefficient word} resolved
  uint16_t* order;    // listed elements in scan order (positions in entries)
  uint64_t* rows;     // [R] row states
  uint32_t img_s, ga_s;
  int lane;
  uint64_t prev;      // state whose images are in row `prev_row` of ga
  int prev_row;
  // per group of rows: lane r < nr holds row r's state, inverse norm and number of elements
  uint64_t a_l;
  double inv_l;
  int cnt_l;
  int nr;

  __device__ __forceinline__ RowGroup(const RowsLayout& L_, const MatvecProblem& p_, unsigned char* s)
      : L(L_), p(p_), smem(s) {
    unsigned char* w = s + L.off_warp + (threadIdx.x >> 5) * L.warp_bytes;
    ga = (uint32_t*)w;
    entries = (uint2*)(w + L.w_ent);
    order = (uint16_t*)(w + L.w_ord);
    rows = (uint64_t*)(w + L.w_a);
    img_s = (uint32_t)__cvta_generic_to_shared(s + L.off_img);
    ga_s = (uint32_t)__cvta_generic_to_shared(ga);
    lane = threadIdx.x & 31;
    prev = 0;
    prev_row = -1;
  }

  template <typename T>
  __device__ __forceinline__ const T* tab(uint32_t off) const {
    return reinterpret_cast<const T*>(smem + off);
  }

  // Fills the block's tables; the caller synchronises the block afterwards.
  __device__ __forceinline__ static void stage(const RowsLayout& L, const MatvecProblem& p, unsigned char* smem) {
    const int G = L.G, nb = p.group.n_bits;
    const int tid = threadIdx.x, nt = blockDim.x;
    auto word = [&](uint64_t x, int w) -> uint32_t {  // word w of the images of the bits of x
      if constexpr (MODE == kModeN32) {
        const int g = w < G ? w : 0;
        uint64_t v = 0;
        for (; x != 0; x &= x - 1) v ^= __ldg(p.group.onehot + (__ffsll((long long)x) - 1) * G + g);
        return (uint32_t)v;
      } else {
        const int g0 = 2 * w < G ? 2 * w : 0, g1 = 2 * w + 1 < G ? 2 * w + 1 : 0;
        uint64_t v0 = 0, v1 = 0;
        for (; x != 0; x &= x - 1) {
          const uint64_t* r = p.group.onehot + (__ffsll((long long)x) - 1) * G;
          v0 ^= __ldg(r + g0);
          v1 ^= __ldg(r + g1);
        }
        return (uint32_t)(v0 >> (nb - 16)) | ((uint32_t)(v1 >> (nb - 16)) << 16);
      }
    };
    uint32_t* site = (uint32_t*)(smem + L.off_site);
    for (int i = tid; i < nb * L.site_words; i += nt) {
      const int b = i / L.site_words, w = i - b * L.site_words;
      site[i] = w < L.words ? word(1ull << b, w) : 0u;
    }
    uint32_t* img = (uint32_t*)(smem + L.off_img);
    for (int i = tid; i < L.n_pat * L.words; i += nt) {
      const int x = i / L.words, w = i - x * L.words;
      img[x * L.stride + w] = word(__ldg(p.off.rows.xmask + x), w);
    }
    if constexpr (MODE == kModeP16) {
      unsigned char* perm = smem + L.off_perm;
      for (int i = tid; i < nb * G; i += nt) {
        const int b = i / G, g = i - b * G;
        const int to = __ffsll((long long)__ldg(p.group.onehot + i)) - 1;
        if (to < L.nlow) perm[g * L.perm_stride + (L.nlow - 1 - to)] = (unsigned char)b;
      }
    }
    stage_u64((uint64_t*)(smem + L.off_sm), p.off.rows.sm, 32 * L.slot_blocks);
    stage_u64((uint64_t*)(smem + L.off_sl1), p.off.rows.sl1, 32 * L.slot_blocks);
    stage_u64((uint64_t*)(smem + L.off_sl2), p.off.rows.sl2, 32 * L.slot_blocks);
    uint32_t* st = (uint32_t*)(smem + L.off_st);
    for (int i = tid; i < 32 * L.slot_blocks; i += nt) st[i] = __ldg(p.off.rows.st + i);
    uint32_t* ti = (uint32_t*)(smem + L.off_ti);
    for (int i = tid; i < L.T; i += nt) ti[i] = __ldg(p.off.rows.tinfo + i);
    stage_u64((uint64_t*)(smem + L.off_ts), p.off.s, L.T);
    stage_u64((uint64_t*)(smem + L.off_xm), p.off.rows.xmask, L.n_pat);
    stage_u64((uint64_t*)(smem + L.off_dm), p.diag.rows.sm, 32 * L.n_diag_blocks);
    stage_u64((uint64_t*)(smem + L.off_dr), p.diag.rows.sl1, 32 * L.n_diag_blocks);
    stage_u64((uint64_t*)(smem + L.off_ds), p.diag.rows.sl2, 32 * L.n_diag_blocks);
    uint2* db = (uint2*)(smem + L.off_db);
    for (int i = tid; i < L.n_diag_blocks; i += nt)
      db[i] = make_uint2(__ldg(p.diag.rows.st + i), __ldg(p.diag.rows.tinfo + i));
    stage_d2((double2*)(smem + L.off_dv), p.diag.rows.cval, p.diag.rows.n_cls);
    if constexpr (FERMI) stage_u64((uint64_t*)(smem + L.off_fs), p.group.fsign_packed, nb * 32 * p.group.gpl);
  }

  // Forgets the images of earlier rows (before a block of rows that does not follow them).
  __device__ __forceinline__ void restart() {
    prev = 0;
    prev_row = -1;
  }

  // Steps 1 and 2 for the rows [row0, row0 + n).  Returns the number of listed elements.
  __device__ __forceinline__ int load_rows(const DeviceIndex& ix, int64_t row0, int n) {
    nr = n;
    __syncwarp();  // the previous group's readers are done
    a_l = lane < nr ? __ldg(ix.reps + row0 + lane) : 0ull;
    inv_l = lane < nr ? __ldg(ix.inv_norms + row0 + lane) : 0.0;
    cnt_l = 0;
    if (lane < nr) rows[lane] = a_l;
    const uint32_t site_s = (uint32_t)__cvta_generic_to_shared(smem + L.off_site);
    for (int r = 0; r < nr; ++r) {
      const uint64_t a = shfl_u64(a_l, r);
      const uint64_t diff = a ^ prev;
      for (int w0 = lane; w0 < L.words; w0 += 96) {
        // three words per lane at a time; site rows are padded to whole warps, image rows are not
        const bool in1 = w0 + 32 < L.words, in2 = w0 + 64 < L.words;
        uint32_t v0 = 0, v1 = 0, v2 = 0;
        if (prev_row >= 0) {
          const uint32_t* g = ga + prev_row * L.stride + w0;
          v0 = g[0];
          v1 = in1 ? g[32] : 0u;
          v2 = in2 ? g[64] : 0u;
        }
        const uint32_t base = site_s + 4u * (uint32_t)w0;
        for (uint64_t d = diff; d != 0; d &= d - 1) {
          const uint32_t s = base + (uint32_t)(__ffsll((long long)d) - 1) * (uint32_t)(4 * L.site_words);
          v0 ^= lds_u32(s);
          if (in1) v1 ^= lds_u32(s + 128);
          if (in2) v2 ^= lds_u32(s + 256);
        }
        uint32_t* g = ga + r * L.stride + w0;
        g[0] = v0;
        if (in1) g[32] = v1;
        if (in2) g[64] = v2;
      }
      prev = a;
      prev_row = r;
    }
    // zero-norm rows take no part (their outputs are zero)
    const unsigned live = __ballot_sync(FULL, inv_l != 0.0);
    int total = 0;
    const unsigned below = (1u << lane) - 1u;
    for (int b = 0; b < L.slot_blocks; ++b) {
      const uint64_t m = tab<uint64_t>(L.off_sm)[32 * b + lane];
      const uint64_t l1 = tab<uint64_t>(L.off_sl1)[32 * b + lane], l2 = tab<uint64_t>(L.off_sl2)[32 * b + lane];
      const uint32_t t12 = tab<uint32_t>(L.off_st)[32 * b + lane];
      for (int r = 0; r < nr; ++r) {
        uint64_t x;
        bool h1, h2;
        if constexpr (MODE == kModeN32) {
          const uint32_t v = __shfl_sync(FULL, (uint32_t)a_l, r) & (uint32_t)m;
          h1 = v == (uint32_t)l1 && (l1 >> 32) == 0;
          h2 = v == (uint32_t)l2 && (l2 >> 32) == 0;
        } else {
          x = shfl_u64(a_l, r) & m;
          h1 = x == l1;
          h2 = x == l2;
        }
        const bool hit = (h1 || h2) && ((live >> r) & 1u);
        const unsigned hits = __ballot_sync(FULL, hit);
        const int before = __shfl_sync(FULL, cnt_l, r);
        if (hit) {
          const int rank = __popc(hits & below);
          const int at = r * L.cap + before + rank;
          entries[at] = make_uint2((h1 ? t12 & 0xffffu : t12 >> 16) | ((uint32_t)r << 16), 0u);
          order[total + rank] = (uint16_t)at;
        }
        const int c = __popc(hits);
        if (lane == r) cnt_l += c;
        total += c;
      }
    }
    __syncwarp();
    return total;
  }

  // The candidate minimum over the group for the element whose row images start at shared address
  // gp and pattern images at ip.  beta is the generated state.  Returns the representative; *key
  // is 2 * element + flipped.
  __device__ __forceinline__ uint64_t scan(uint32_t gp, uint32_t ip, uint64_t beta, uint32_t* key) const {
    if constexpr (MODE == kModeN32) {
      const uint32_t flip = (uint32_t)p.group.flip;
      uint32_t best = 0xffffffffu, at = 0;
      for (int c = 0; c < L.words; c += 8) {
        uint32_t mn = 0xffffffffu, mx = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t h = lds_u32_volatile(gp + 4 * (c + k)) ^ lds_u32(ip + 4 * (c + k));
          mn = min(mn, h);
          if (INV) mx = max(mx, h);
        }
        const uint32_t m = INV ? min(mn, flip ^ mx) : mn;
        if (m < best) {
          best = m;
          at = (uint32_t)c;
        }
      }
      uint32_t k0 = 0;
#pragma unroll
      for (int k = 7; k >= 0; --k) {
        const uint32_t h = lds_u32_volatile(gp + 4 * (at + k)) ^ lds_u32(ip + 4 * (at + k));
        if (INV && (h ^ flip) == best) k0 = 2 * k + 1;
        if (h == best) k0 = 2 * k;
      }
      *key = 2 * at + k0;
      return best;
    } else {
      uint32_t best = 0x10000u, mask = 0, bit = 1;
      for (int c = 0; c < L.words; c += 8, bit <<= 1) {
        uint32_t mn = 0xffffffffu, mx = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t h = lds_u32_volatile(gp + 4 * (c + k)) ^ lds_u32(ip + 4 * (c + k));
          mn = vmin2(mn, h);
          if (INV) mx = vmax2(mx, h);
        }
        if (INV) mn = vmin2(mn, ~mx);
        const uint32_t m = min(mn & 0xffffu, mn >> 16);
        mask = m < best ? bit : (m == best ? mask | bit : mask);
        best = min(best, m);
      }
      // the elements of the marked chunks that reach the prefix, compared by their low bits
      const uint32_t two = best | (best << 16);
      uint32_t found = 0;  // bit 4 k + 2 half + flipped of the chunk at `at`
      uint32_t at = 0, win = 0;
      uint64_t low = ~0ull;
      const uint64_t low_ones = (1ull << L.nlow) - 1;
      const uint32_t perm_s = (uint32_t)__cvta_generic_to_shared(smem + L.off_perm);
      do {
        if (found == 0 && mask != 0) {
          at = (uint32_t)(__ffs(mask) - 1) * 8u;
          mask &= mask - 1;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t d = lds_u32_volatile(gp + 4 * (at + k)) ^ lds_u32(ip + 4 * (at + k)) ^ two;
            if ((d & 0xffffu) == 0u) found |= 1u << (4 * k);
            if ((d >> 16) == 0u) found |= 4u << (4 * k);
            if (INV) {
              if ((d & 0xffffu) == 0xffffu) found |= 2u << (4 * k);
              if ((d >> 16) == 0xffffu) found |= 8u << (4 * k);
            }
          }
        }
        if (found != 0) {
          const uint32_t f = (uint32_t)__ffs(found) - 1;
          found &= found - 1;
          const uint32_t g = 2 * at + (f >> 1);
          const uint32_t ps = perm_s + (g < (uint32_t)L.G ? g : 0u) * (uint32_t)L.perm_stride;
          uint64_t v = 0;
          for (int b = 0; b < L.nlow; b += 4) {
            const uint32_t src = lds_u32(ps + b);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (b + i < L.nlow) v = 2 * v + ((beta >> ((src >> (8 * i)) & 0xffu)) & 1ull);
          }
          if (f & 1u) v ^= low_ones;
          if (v < low) {
            low = v;
            win = 2 * g + (f & 1u);
          }
        }
      } while (__any_sync(FULL, (found | mask) != 0));
      *key = win;
      return ((uint64_t)best << L.nlow) | low;
    }
  }

  // Step 3 for the listed elements (total as returned by load_rows).
  __device__ __forceinline__ void resolve(const DeviceIndex& ix, int total, int* __restrict__ err,
                                          const uint64_t* __restrict__ binom) {
    for (int w = 0; w < total; w += 32) {
      const int at = order[min(w + lane, total - 1)];
      const bool mine = w + lane < total;
      const uint32_t e = entries[at].x;
      const int t = (int)(e & 0xffffu), r = (int)(e >> 16);
      const uint32_t info = tab<uint32_t>(L.off_ti)[t];
      const uint32_t pat = info & 0xffffu;
      const uint64_t beta = rows[r] ^ tab<uint64_t>(L.off_xm)[pat];
      const uint32_t stride = 4u * (uint32_t)L.stride;
      uint32_t key;
      const uint64_t rep = scan(ga_s + (uint32_t)r * stride, img_s + pat * stride, beta, &key);
      if (mine) {
        bool ok = true;
        if (info & kRowTermNeedsCheck) {
          ok = constraint_ok(p.constraint, beta);
          if (!ok) atomicOr(err, 1);
        }
        const int64_t j = ok ? mv_index_lookup(ix, rep, binom) : -1;
        uint32_t g = key >> 1;
        if (g >= (uint32_t)L.G) g = 0;  // padding repeats element 0
        uint32_t neg = (uint32_t)__popcll(beta & tab<uint64_t>(L.off_ts)[t]) ^ (info >> 31);
        if (INV && p.group.spin_inversion == -1) neg ^= key;
        if constexpr (FERMI) neg ^= (uint32_t)fermion_parity(tab<uint64_t>(L.off_fs) + g, 32 * p.group.gpl, beta);
        const uint32_t cls = (info >> 16) & 0xffu;
        entries[at] = make_uint2(j >= 0 ? (uint32_t)j : kAbsent, (cls * (uint32_t)L.G + g) | (neg << 31));
      }
    }
    __syncwarp();
  }

  // The diagonal elements: lane r < nr returns row r's.
  __device__ __forceinline__ double2 diagonal() const {
    double2 d = make_double2(0.0, 0.0);
    int n_l = 0;
    for (int b = 0; b < L.n_diag_blocks; ++b) {
      const uint64_t m = tab<uint64_t>(L.off_dm)[32 * b + lane], k = tab<uint64_t>(L.off_dr)[32 * b + lane];
      const uint64_t s = tab<uint64_t>(L.off_ds)[32 * b + lane];
      const uint2 info = tab<uint2>(L.off_db)[b];  // {signs of the 32 terms, class | last block of it << 31}
      for (int r = 0; r < nr; ++r) {
        bool hit, odd;
        if constexpr (MODE == kModeN32) {
          const uint32_t a = __shfl_sync(FULL, (uint32_t)a_l, r);
          hit = (a & (uint32_t)m) == (uint32_t)k && (k >> 32) == 0;
          odd = __popc(a & (uint32_t)s) & 1;
        } else {
          const uint64_t a = shfl_u64(a_l, r);
          hit = (a & m) == k;
          odd = __popcll(a & s) & 1;
        }
        const unsigned hits = __ballot_sync(FULL, hit);
        const unsigned minus = (__ballot_sync(FULL, odd) ^ info.x) & hits;
        if (lane == r) n_l += __popc(hits) - 2 * __popc(minus);
      }
      if (info.y >> 31) {
        const double2 v = tab<double2>(L.off_dv)[info.y & 0xffffu];
        d.x = fma((double)n_l, v.x, d.x);
        d.y = fma((double)n_l, v.y, d.y);
        n_l = 0;
      }
    }
    return d;
  }
};

}  // namespace lsg
