// ranks.h -- which bases without a permutation group have two-table ranks (matvec_free.cu), and the
// tables' shape.  Host code only.
#pragma once

#include <cstdint>

namespace lsg {

struct RankTables {
  int split = 0, high_bits = 0;  // low and high bits of a state
  int h = 0;                     // weight of the state; two species: of its high bits
  int species = 0;               // 1: the two halves have a weight each
  int64_t n_low = 0;             // species: states of the low half
  int64_t states = 0;            // of the complete basis
};

// n over k, saturated at 2^62.
inline uint64_t rank_binomial(int n, int k) {
  if (k < 0 || k > n) return 0;
  unsigned __int128 b = 1;
  for (int i = 1; i <= k; ++i) {
    b = b * (unsigned)(n - k + i) / (unsigned)i;  // exact: a binomial at every step
    if (b >> 62) return (uint64_t)1 << 62;
  }
  return (uint64_t)b;
}

// `bits` bits in all, `weight` of them set; up >= 0: two halves of which the low one has `up` set.
// inversion: only the states below their complement.  False where the tables would be too large (more
// than 40 bits: 8 MB) or a rank would not fit their 32-bit words.
inline bool rank_tables_for(int bits, int weight, int up, bool inversion, RankTables* t) {
  if (bits < 1 || bits > 40 || weight < 0 || weight > bits) return false;
  *t = RankTables{};
  if (up >= 0) {
    t->species = 1;
    t->split = t->high_bits = bits / 2;
    t->h = weight - up;
    const uint64_t low = rank_binomial(t->split, up), high = rank_binomial(t->high_bits, t->h);
    t->n_low = (int64_t)low;
    t->states = (int64_t)(low * high);  // each at most 20 over 10
  } else {
    t->split = (bits + 1) / 2;
    t->high_bits = bits - t->split;
    t->h = weight;
    t->states = (int64_t)(rank_binomial(bits, weight) / (inversion ? 2 : 1));
  }
  return t->states > 0 && t->states <= (int64_t)1 << 32;
}

}  // namespace lsg
