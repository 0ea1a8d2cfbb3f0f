// Local states of a sector key, last site first, without 64-bit divisions.
//
// The sites are grouped from the last one backwards into chunks whose
// dimensions multiply to at most 2^31 (a chunk never crosses the words of a
// two-word key).  A chunk's value is split off its word with one quotient by
// the chunk's space: the f64 estimate word * (1 / space) corrected twice by
// the exact remainder.  Inside a chunk every value is below 2^31, where with
// l = ceil(log2 d) and m = ceil(2^(31 + l) / d) < 2^32
//   floor(x / d) = (x m) >> (31 + l)
// (Granlund, Montgomery, "Division by invariant integers using
// multiplication", 1994, theorem 4.2: m d - 2^(31 + l) < d <= 2^l).  A digit
// is then a multiply-high, a shift and a multiply-subtract instead of the two
// 64-bit divisions of key_digit.
#pragma once
#include "keys.cuh"
#include "internal.cuh"

namespace edg {

constexpr int kMaxChunks = 8;

// Passed to kernels by value.  Position p counts sites from the last one.
struct DigitPlan {
  int n_sites;
  int key_words;
  uint64_t chunk_at;              // bit p: position p starts a new chunk
  uint64_t word_at;               // bit p: position p starts the high word
  uint32_t d[EDG_MAX_SITES];      // dimension at position p
  uint32_t magic[EDG_MAX_SITES];  // ceil(2^(31 + l) / d), l = ceil(log2 d)
  uint32_t shift[EDG_MAX_SITES];  // l - 1 (unused for d = 1)
  uint32_t space[kMaxChunks];     // product of a chunk's dimensions (0: the word's last chunk, taken whole)
  double inv[kMaxChunks];         // 1 / space
};

// Plan of local dimensions d_s (n_hi: sites of the high word, two-word keys);
// on the host, or by one thread of a CTA whose caller has the dimensions in
// device memory only.  False when a dimension is below 1 or a word needs too many chunks.
template <typename Int>
__host__ __device__ inline bool make_digit_plan(DigitPlan* p, const Int* dims, int n_sites, int key_words, int n_hi) {
  *p = DigitPlan{};
  p->n_sites = n_sites;
  p->key_words = key_words == 2 ? 2 : 1;
  const int split = p->key_words == 2 ? n_hi : 0;
  int chunk = -1;
  uint64_t prod = 0;
  for (int pos = 0; pos < n_sites; ++pos) {
    const int s = n_sites - 1 - pos;
    const int64_t d = (int64_t)dims[s];
    if (d < 1 || d > 65536) return false;
    const bool new_word = pos == 0 || (p->key_words == 2 && s == split - 1);
    if (new_word && pos > 0) p->word_at |= 1ull << pos;
    if (new_word || prod * (uint64_t)d > (1ull << 31)) {
      if (!new_word) {  // the chunk before this one ends inside the word
        p->space[chunk] = (uint32_t)prod;
        p->inv[chunk] = 1.0 / (double)prod;
      }
      if (++chunk >= kMaxChunks) return false;
      p->chunk_at |= 1ull << pos;
      prod = 1;
    }
    prod *= (uint64_t)d;
    p->d[pos] = (uint32_t)d;
    int l = 0;
    while ((1ll << l) < d) ++l;
    p->magic[pos] = (uint32_t)((((uint64_t)1 << (31 + l)) + (uint64_t)d - 1) / (uint64_t)d);
    p->shift[pos] = (uint32_t)(l > 0 ? l - 1 : 0);
  }
  return true;
}

// floor(x / space) with remainder, space <= 2^31, x < 2^63.  The first
// estimate is off by less than 2^11 (f64 rounding of x and of the product),
// the second by at most one.
__device__ __forceinline__ uint64_t split_chunk(uint64_t x, uint32_t space, double inv, uint32_t* rem) {
  uint64_t q = (uint64_t)((double)x * inv);
  int64_t r = (int64_t)(x - q * space);
  const int64_t c = (int64_t)floor((double)r * inv);
  q += (uint64_t)c;
  r -= c * (int64_t)space;
  if (r < 0) {
    r += space;
    --q;
  } else if (r >= (int64_t)space) {
    r -= space;
    ++q;
  }
  *rem = (uint32_t)r;
  return q;
}

// Calls use(p, digit) for the positions p = 0 .. n_sites - 1 (site
// n_sites - 1 - p) of a key; NS >= n_sites bounds the unrolled loop, so use()
// may index registers with p.
template <int NS, typename K, typename F>
__device__ __forceinline__ void for_each_digit(const DigitPlan& P, K key, F use) {
  uint64_t word = key_lo(key);
  uint32_t x = 0;
  int chunk = -1;
#pragma unroll
  for (int p = 0; p < NS; ++p) {
    if (p < P.n_sites) {
      if ((P.chunk_at >> p) & 1ull) {
        if (sizeof(K) == 16 && ((P.word_at >> p) & 1ull)) word = key_hi(key);
        ++chunk;
        if (P.space[chunk] != 0)
          word = split_chunk(word, P.space[chunk], P.inv[chunk], &x);
        else
          x = (uint32_t)word;
      }
      const uint32_t d = P.d[p];
      const uint32_t q = d > 1 ? __umulhi(P.magic[p], x) >> P.shift[p] : x;
      use(p, (int)(x - q * d));
      x = q;
    }
  }
}

}  // namespace edg
