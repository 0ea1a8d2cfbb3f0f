// Sector Hamiltonian assembly.
//
// For every off-diagonal term instance (a product of up to EDG_MAX_OPS site
// operators) a row (bra state) enumerates the product of the local transitions
// of its bra states, forms the ket key as bra_key + sum_j (ket_j - bra_j) *
// stride_j, finds the ket row by a bucketed search and emits (col, coef * prod
// amp).  This is the n-body triplet builder of edlgt/symmetries/
// sym_qmb_operations.py:297-562 with the configuration copy replaced by key
// arithmetic.  Diagonal terms use only the operator diagonal and drop |op_cc|
// < 1e-10 exactly like localbody_data_par (sym_qmb_operations.py:565-602).
// Each row's entries are then sorted by column and duplicates are summed,
// which yields the canonical (summed) matrix of edlgt/modeling/
// qmb_hamiltonian.py:196-199.  Kernels are templated on the key type (one
// word, or two words past 63 bits of key space: keys.cuh).
//
// Three kernels, one lane a row, digits in shared memory:
//   count_k  rows -> entry bounds;
//   fill_k   entries.  A row has transitions in about a quarter of the
//            instances, so a table per (site, state) holds the instances whose
//            factor there has any, as bits, and the row's instances are the
//            AND over its sites.  A lane takes four entries at a time: their
//            kets' searches run together (four independent chains of L2 reads
//            instead of one), then each is inserted into the row's window in
//            shared memory in column order.  The windows of a warp's rows are
//            one contiguous range of the output, written with coalesced
//            stores.  They are the final matrix when no row has duplicates or
//            entries on the diagonal (flags[1] stays 0: every 1D chain and 2D
//            lattice of the models), and no compaction follows.
//   diag_k   diagonal terms.
// Bound by instructions (two issued per cycle and SM, nine thousand per 32 rows
// of 13 entries): SU(2) L = 14 ring, 1,232,454 rows, 16,056,880 entries, 0.71 ms
// and 0.11 for the bounds.  With one thread per row walking every instance and
// sorting its window in global memory, and a compaction behind it, the same
// took 1.20 + 0.35 ms and 0.14.
#include "digits.cuh"
#include "lookup.cuh"

namespace {

constexpr double kOpTol = 1e-10;  // OP_TOL of the reference
constexpr int kThreads = 256;

struct Real {
  double v;
  __device__ static Real zero() { return {0.0}; }
  __device__ static Real load(const double* p, int64_t i) { return {p[i]}; }
  __device__ void store(double* p, int64_t i) const { p[i] = v; }
  __device__ Real operator*(const Real& o) const { return {v * o.v}; }
  __device__ Real& operator+=(const Real& o) { v += o.v; return *this; }
  __device__ double abs() const { return fabs(v); }
  __device__ static Real from(double re, double) { return {re}; }
};

struct Cplx {
  double re, im;
  __device__ static Cplx zero() { return {0.0, 0.0}; }
  __device__ static Cplx load(const double* p, int64_t i) { return {p[2 * i], p[2 * i + 1]}; }
  __device__ void store(double* p, int64_t i) const { p[2 * i] = re; p[2 * i + 1] = im; }
  __device__ Cplx operator*(const Cplx& o) const { return {re * o.re - im * o.im, re * o.im + im * o.re}; }
  __device__ Cplx& operator+=(const Cplx& o) { re += o.re; im += o.im; return *this; }
  __device__ double abs() const { return hypot(re, im); }
  __device__ static Cplx from(double re, double im) { return {re, im}; }
};

constexpr int kWarps = kThreads / 32;
constexpr int kWindow = 512;           // entries of a warp's windows
constexpr int kTableCap = 24 * 1024;   // bytes of a table kept in shared memory

// What fill_k and count_k read per instance, in shared memory where it fits
// (the same values through either pointer).
struct Tables {
  const int32_t* nops;    // [n_terms]
  const int32_t* site;    // [n_terms][EDG_MAX_OPS]
  const int32_t* table;   // [n_terms][EDG_MAX_OPS]
  const uint32_t* mask;   // [n_words][n_sites][dmax], or NULL: not staged
  const double* amp;
  const uint8_t* ket;
  int n_words;
};

// Bytes of the parts of a launch's shared memory, in this order: a warp's
// windows (fill_k), digits, instance records, instance masks, amplitudes, kets.
struct Parts {
  int windows, digits, terms, mask, amp, ket;
  __host__ __device__ int total() const { return windows + digits + terms + mask + amp + ket; }
};

__device__ __forceinline__ Tables stage_tables(const edg_assembly& a, const Parts& p, unsigned char* sm, int n_tables,
                                               int width) {
  Tables T{a.term_nops, a.term_site, a.term_table, nullptr, a.t_amp, a.t_ket, (a.n_terms + 31) / 32};
  const int n = a.n_terms, dm = a.dmax, ns = a.n_sites;
  unsigned char* at = sm + p.windows + p.digits;
  if (p.terms) {
    int32_t* t = reinterpret_cast<int32_t*>(at);
    for (int k = threadIdx.x; k < n * (1 + 2 * EDG_MAX_OPS); k += kThreads)
      t[k] = k < n ? a.term_nops[k] : k < n * (1 + EDG_MAX_OPS) ? a.term_site[k - n]
                                                                : a.term_table[k - n * (1 + EDG_MAX_OPS)];
    T.nops = t;
    T.site = t + n;
    T.table = t + n * (1 + EDG_MAX_OPS);
  }
  at += p.terms;
  uint32_t* mk = reinterpret_cast<uint32_t*>(at);
  if (p.mask)
    for (int k = threadIdx.x; k < T.n_words * ns * dm; k += kThreads) {
      const int left = n - 32 * (k / (ns * dm));  // instances of this word
      mk[k] = left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u;
    }
  at += p.mask;
  if (p.amp) {
    double* t = reinterpret_cast<double*>(at);
    for (int k = threadIdx.x; k < n_tables * dm * dm * width; k += kThreads) t[k] = a.t_amp[k];
    T.amp = t;
  }
  at += p.amp;
  if (p.ket) {
    for (int k = threadIdx.x; k < n_tables * dm * dm; k += kThreads) at[k] = a.t_ket[k];
    T.ket = at;
  }
  __syncthreads();
  if (p.mask) {
    // clear an instance's bit at (site, state) where its factor has no transition
    for (int k = threadIdx.x; k < n * EDG_MAX_OPS * dm; k += kThreads) {
      const int c = k % dm, j = k / dm % EDG_MAX_OPS, i = k / (dm * EDG_MAX_OPS);
      if (j < T.nops[i] && __ldg(a.t_count + T.table[i * EDG_MAX_OPS + j] * dm + c) == 0)
        atomicAnd(mk + ((i / 32) * ns + T.site[i * EDG_MAX_OPS + j]) * dm + c, ~(1u << (i & 31)));
    }
    T.mask = mk;
    __syncthreads();
  }
  return T;
}

// Digits of a row into dig[site * 32 + lane].
template <int NS, typename K>
__device__ __forceinline__ void stage_digits(const edg::DigitPlan& P, K key, uint8_t* dig, int lane) {
  const int ns = P.n_sites;
  edg::for_each_digit<NS>(P, key, [&](int p, int c) { dig[(ns - 1 - p) * 32 + lane] = (uint8_t)c; });
}

// Walks a row's entries in generation order: instances ascending, the
// combinations of an instance's transitions with the last factor fastest.
struct Walk {
  const edg_assembly& a;
  const Tables& T;
  const uint8_t* dig;  // this lane's digits, stride 32
  int word = -1, k = 0, nops = 0;
  uint32_t bits = 0;
  int cnt[EDG_MAX_OPS], idx[EDG_MAX_OPS];  // transitions of each factor, and the current one
  int ent[EDG_MAX_OPS];                    // each factor's (table, bra) row

  __device__ Walk(const edg_assembly& a_, const Tables& T_, const uint8_t* d) : a(a_), T(T_), dig(d) {}

  __device__ __forceinline__ uint32_t mask_of(int w) const {
    const int ns = a.n_sites, dm = a.dmax;
    if (T.mask != nullptr) {
      const uint32_t* m = T.mask + w * ns * dm;
      uint32_t v = 0xFFFFFFFFu;
      for (int s = 0; s < ns; ++s) v &= m[s * dm + dig[s * 32]];
      return v;
    }
    uint32_t v = 0u;
    for (int b = 0; b < 32 && 32 * w + b < a.n_terms; ++b) {
      const int i = 32 * w + b;
      bool any = true;
      for (int j = 0; j < T.nops[i]; ++j)
        any = any && __ldg(a.t_count + T.table[i * EDG_MAX_OPS + j] * dm + dig[T.site[i * EDG_MAX_OPS + j] * 32]) != 0;
      v |= any ? 1u << b : 0u;
    }
    return v;
  }
  // The next instance with transitions on this row.
  __device__ __forceinline__ bool next_term() {
    while (bits == 0u) {
      if (++word >= T.n_words) return false;
      bits = mask_of(word);
    }
    k = 32 * word + __ffs(bits) - 1;
    bits &= bits - 1u;
    nops = T.nops[k];
#pragma unroll
    for (int j = 0; j < EDG_MAX_OPS; ++j) {
      cnt[j] = 1;
      idx[j] = 0;
      if (j < nops) {
        ent[j] = T.table[k * EDG_MAX_OPS + j] * a.dmax + dig[T.site[k * EDG_MAX_OPS + j] * 32];
        cnt[j] = __ldg(a.t_count + ent[j]);
      }
    }
    return true;
  }
  __device__ __forceinline__ bool next() {
    if (word >= 0) {
      // mixed-radix increment; factors beyond nops have one transition
#pragma unroll
      for (int j = EDG_MAX_OPS - 1; j >= 0; --j) {
        if (idx[j] + 1 < cnt[j]) {
          ++idx[j];
          return true;
        }
        idx[j] = 0;
      }
    }
    return next_term();
  }
  template <typename V, typename K>
  __device__ __forceinline__ void entry(K key, K* ket_key, V* amp) const {
    K kk = key;
    V v = V::load(a.term_coef, k);
#pragma unroll
    for (int j = 0; j < EDG_MAX_OPS; ++j)
      if (j < nops) {
        const int e = ent[j] * a.dmax + idx[j];
        const int site = T.site[k * EDG_MAX_OPS + j];
        v = v * V::load(T.amp, e);
        kk += edg::key_step<K>((int64_t)((int)T.ket[e] - (int)dig[site * 32]) * (int64_t)a.strides[site], site,
                               a.sector.n_hi);
      }
    *ket_key = kk;
    *amp = v;
  }
};

template <typename K, int NS>
__global__ void __launch_bounds__(kThreads) count_k(const __grid_constant__ edg_assembly a,
                                                    const __grid_constant__ edg::DigitPlan P, const Parts parts,
                                                    int64_t* __restrict__ row_bound) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint8_t* const dig = sm_raw + warp * 32 * P.n_sites;
  const Tables T = stage_tables(a, parts, sm_raw, 0, 0);
  for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < a.sector.n; r += (int64_t)gridDim.x * kThreads) {
    stage_digits<NS>(P, edg::ld_key<K>(a.sector.keys, r), dig, lane);  // own lane's bytes only
    Walk w(a, T, dig + lane);
    int64_t total = 0;
    while (w.next_term()) total += (int64_t)w.cnt[0] * w.cnt[1] * ((int64_t)w.cnt[2] * w.cnt[3]);
    row_bound[r] = total;
  }
}

// Rows of NB keys in the sorted sector (-1: not a sector state), the searches
// of find_key side by side; `have` bit b: key b is asked for.
template <int NB, typename K>
__device__ __forceinline__ void find_rows(const edg_lookup_table& t, const K (&q)[NB], unsigned have, int32_t (&row)[NB]) {
  int32_t lo[NB], hi[NB], end[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    lo[b] = hi[b] = 0;
    if ((have >> b) & 1u) {
      uint64_t bucket;
      bool inside;
      if constexpr (sizeof(K) == 8) {
        bucket = q[b] >> t.shift;
        inside = bucket < (uint64_t)t.n_buckets;
      } else {
        const edg::u128 w = edg::key_dense(q[b], t.lo_space) >> t.shift;
        inside = w < (edg::u128)(uint64_t)t.n_buckets;
        bucket = (uint64_t)w;
      }
      if (inside) {
        lo[b] = (int32_t)__ldg(t.bucket_start + bucket);
        hi[b] = (int32_t)__ldg(t.bucket_start + bucket + 1);
      }
    }
    end[b] = hi[b];
  }
  bool more = true;
  while (more) {
    more = false;
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (lo[b] < hi[b]) {
        const int32_t mid = lo[b] + (hi[b] - lo[b]) / 2;
        if (edg::ld_key<K>(t.keys, mid) < q[b])
          lo[b] = mid + 1;
        else
          hi[b] = mid;
        more |= lo[b] < hi[b];
      }
  }
#pragma unroll
  for (int b = 0; b < NB; ++b) row[b] = lo[b] < end[b] && edg::ld_key<K>(t.keys, lo[b]) == q[b] ? lo[b] : -1;
}

// A row's entries into its window of cap entries (col, val; shared or global
// memory), sorted by column with duplicates added in generation order; returns
// how many.  Columns left of the diagonal grow from the window's start, those
// right of it from its end: with the instances in the order of their leading
// sites the first list arrives almost ascending and the second almost
// descending, so an insertion hardly moves anything (one list with every
// entry compared from its end took a third of the kernel's instructions).
template <typename V, typename K>
__device__ __forceinline__ int fill_row(const edg_assembly& a, const Tables& T, const uint8_t* dig, K key,
                                        int64_t r, int cap, int32_t* col, double* val, V* d, bool* present,
                                        int32_t* __restrict__ err) {
  constexpr int NB = sizeof(K) == 8 ? 4 : 2;  // searches in flight
  Walk w(a, T, dig);
  int left = 0, right = cap;  // [0, left) and [right, cap) are filled
  bool more = true;
  // Entries queue up in registers, the oldest at the highest index; the loops
  // over them rotate the queue instead of unrolling, which keeps the kernel
  // inside the instruction cache (four copies of the walk and the insertion
  // spent a third of their cycles waiting for instructions).
  K key_b[NB];
  V amp_b[NB];
  int32_t row_b[NB];
  while (more) {
    unsigned have = 0u;
#pragma unroll 1
    for (int b = 0; b < NB; ++b) {
      more = w.next();
      if (!more) break;
#pragma unroll
      for (int q = NB - 1; q > 0; --q) {
        key_b[q] = key_b[q - 1];
        amp_b[q] = amp_b[q - 1];
      }
      w.template entry<V, K>(key, &key_b[0], &amp_b[0]);
      have = (have << 1) | 1u;
    }
    find_rows<NB, K>(a.sector, key_b, have, row_b);
#pragma unroll 1
    for (int b = 0; b < NB; ++b) {
      const int32_t c = row_b[NB - 1];
      const V v = amp_b[NB - 1];
      const bool on = (have >> (NB - 1)) & 1u;
#pragma unroll
      for (int q = NB - 1; q > 0; --q) {
        row_b[q] = row_b[q - 1];
        amp_b[q] = amp_b[q - 1];
      }
      have <<= 1;
      if (!on) continue;
      if (c < 0) {
        atomicExch(err, EDG_ERR_MISSING_KET);
      } else if (c == (int32_t)r) {
        *d += v;
        *present = true;
      } else if (c < (int32_t)r) {
        int j = left;
        while (j > 0 && col[j - 1] > c) --j;
        if (j > 0 && col[j - 1] == c) {
          V t = V::load(val, j - 1);
          t += v;
          t.store(val, j - 1);
        } else {
          for (int i = left; i > j; --i) {
            col[i] = col[i - 1];
            V::load(val, i - 1).store(val, i);
          }
          col[j] = c;
          v.store(val, j);
          ++left;
        }
      } else {
        int j = right;
        while (j < cap && col[j] < c) ++j;
        if (j < cap && col[j] == c) {
          V t = V::load(val, j);
          t += v;
          t.store(val, j);
        } else {
          --right;
          for (int i = right; i < j - 1; ++i) {
            col[i] = col[i + 1];
            V::load(val, i + 1).store(val, i);
          }
          col[j - 1] = c;
          v.store(val, j - 1);
        }
      }
    }
  }
  const int n = left + cap - right;
  if (left < right)  // fewer entries than the bound: close the gap
    for (int i = left; i < n; ++i) {
      col[i] = col[right + i - left];
      V::load(val, right + i - left).store(val, i);
    }
  return n;
}

// *err: EDG_ERR_MISSING_KET when a ket lies outside the sector; *merged (if
// not NULL): some row has fewer entries than its bound.  diag, diag_present
// come in with the diagonal terms (from_diag) or are written from zero.
template <typename V, typename K, int NS>
__global__ void __launch_bounds__(kThreads, 2) fill_k(const __grid_constant__ edg_assembly a,
                                                   const __grid_constant__ edg::DigitPlan P, const Parts parts,
                                                   int n_tables, int from_diag, const int64_t* __restrict__ offsets,
                                                   int32_t* __restrict__ tcols, double* __restrict__ tvals,
                                                   int64_t* __restrict__ row_nnz, double* __restrict__ diag,
                                                   uint8_t* __restrict__ diag_present, int32_t* __restrict__ err,
                                                   int32_t* __restrict__ merged) {
  constexpr int W = sizeof(V) / sizeof(double);
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* const sval = reinterpret_cast<double*>(sm_raw) + warp * kWindow * W;
  int32_t* const scol = reinterpret_cast<int32_t*>(sm_raw + sizeof(V) * kWindow * kWarps) + warp * kWindow;
  uint8_t* const dig = sm_raw + parts.windows + warp * 32 * P.n_sites;
  const Tables T = stage_tables(a, parts, sm_raw, n_tables, W);
  const int64_t n_rows = a.sector.n, n_tiles = (n_rows + 31) / 32;
  for (int64_t t = blockIdx.x * (int64_t)kWarps + warp; t < n_tiles; t += (int64_t)gridDim.x * kWarps) {
    const int64_t r0 = t * 32, r = r0 + lane;
    const bool live = r < n_rows;
    const int64_t beg = offsets[live ? r : n_rows], end = live ? offsets[r + 1] : beg;
    const K key = live ? edg::ld_key<K>(a.sector.keys, r) : K(0);
    if (live) stage_digits<NS>(P, key, dig, lane);
    // as many rows at a time as have their windows in shared memory
    for (int first = 0; first < 32 && r0 + first < n_rows;) {
      const int64_t base = __shfl_sync(0xffffffffu, beg, first);
      const unsigned fits = __ballot_sync(0xffffffffu, live && lane >= first && end - base <= kWindow) >> first;
      const int rows = fits == 0xFFFFFFFFu ? 32 : __ffs(~fits) - 1;
      const bool staged = rows > 0;  // else one row longer than the windows, in global memory
      const int n_here = staged ? rows : 1;
      const bool mine = lane >= first && lane < first + n_here && live;
      int64_t m = 0;
      if (mine) {
        V d = from_diag ? V::load(diag, r) : V::zero();
        bool present = from_diag && diag_present[r] != 0;
        int32_t* col = staged ? scol + (beg - base) : tcols + beg;
        double* val = staged ? sval + (beg - base) * W : tvals + beg * W;
        m = fill_row<V, K>(a, T, dig + lane, key, r, (int)(end - beg), col, val, &d, &present, err);
        row_nnz[r] = m;
        d.store(diag, r);
        diag_present[r] = present ? 1 : 0;
        if (merged != nullptr && m != end - beg) atomicExch(merged, 1);
      }
      __syncwarp();
      if (staged) {
        const int64_t total = __shfl_sync(0xffffffffu, end, first + n_here - 1) - base;
        // (gaps after shortened rows are copied as they are: nobody reads them)
        for (int e = lane; e < (int)total; e += 32) tcols[base + e] = scol[e];
        for (int e = lane; e < (int)total * W; e += 32) tvals[base * W + e] = sval[e];
        __syncwarp();
      }
      first += n_here;
    }
  }
}

// diag[r] = (base[r] + sum of the diagonal terms) + extra; base may be NULL.
// A term counts where |op_cc| >= 1e-10; a row is present when a term counts,
// when base_present says so, or always when there is an extra.
template <typename V, typename K, int NS>
__global__ void __launch_bounds__(kThreads) diag_k(const __grid_constant__ edg_assembly a,
                                                   const __grid_constant__ edg::DigitPlan P, int in_smem,
                                                   const double* __restrict__ base,
                                                   const uint8_t* __restrict__ base_present, int has_extra, double ex_re,
                                                   double ex_im, double* __restrict__ diag,
                                                   uint8_t* __restrict__ diag_present) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  constexpr int W = sizeof(V) / sizeof(double);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dm = a.dmax, nd = a.n_dterms;
  uint8_t* const dig = sm_raw + warp * 32 * P.n_sites;
  double* const sd = reinterpret_cast<double*>(sm_raw + ((kThreads * P.n_sites + 15) & ~15));
  const double* td = a.dterm_diag;
  if (in_smem) {
    for (int64_t k = threadIdx.x; k < (int64_t)nd * dm * W; k += kThreads) sd[k] = a.dterm_diag[k];
    td = sd;
  }
  __syncthreads();
  for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < a.sector.n; r += (int64_t)gridDim.x * kThreads) {
    stage_digits<NS>(P, edg::ld_key<K>(a.sector.keys, r), dig, lane);
    V d = V::zero();
    bool present = has_extra != 0 || (base_present != nullptr && base_present[r] != 0);
    for (int k = 0; k < nd; ++k) {
      const V v = V::load(td, (int64_t)k * dm + dig[__ldg(a.dterm_site + k) * 32 + lane]);
      if (v.abs() >= kOpTol) {
        present = true;
        d += V::load(a.dterm_coef, k) * v;
      }
    }
    if (base != nullptr) {
      V b = V::load(base, r);
      b += d;
      d = b;
    }
    if (has_extra) d += V::from(ex_re, ex_im);
    d.store(diag, r);
    diag_present[r] = present ? 1 : 0;
  }
}

template <int W>
__global__ void __launch_bounds__(kThreads) compact_k(int64_t n_rows, const int64_t* __restrict__ offsets,
                                                      const int32_t* __restrict__ tcols, const double* __restrict__ tvals,
                                                      const int64_t* __restrict__ rowptr, int32_t* __restrict__ cols,
                                                      double* __restrict__ vals) {
  // one warp per row: coalesced copy of the merged window
  const int lane = threadIdx.x & 31;
  int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = warp; r < n_rows; r += nwarps) {
    int64_t src = offsets[r], dst = rowptr[r], m = rowptr[r + 1] - dst;
    for (int64_t i = lane; i < m; i += 32) {
      cols[dst + i] = tcols[src + i];
#pragma unroll
      for (int w = 0; w < W; ++w) vals[(dst + i) * W + w] = tvals[(src + i) * W + w];
    }
  }
}

int check_assembly(const edg_assembly* a, const char* who) {
  EDG_REQUIRE(a != nullptr, "%s: null description", who);
  EDG_REQUIRE(a->n_sites > 0 && a->n_sites <= EDG_MAX_SITES, "%s: n_sites out of range", who);
  EDG_REQUIRE(a->dmax > 0 && a->dmax <= 255, "%s: dmax out of range", who);
  EDG_REQUIRE(a->sector.n >= 0 && a->sector.n < (int64_t(1) << 31), "%s: sector too large for int32 columns", who);
  EDG_REQUIRE(a->n_terms >= 0 && a->n_dterms >= 0, "%s: negative term count", who);
  EDG_REQUIRE(a->sector.key_words >= 0 && a->sector.key_words <= 2, "%s: key_words must be 1 or 2", who);
  EDG_REQUIRE(a->sector.key_words != 2 ||
                  (a->sector.n_hi > 0 && a->sector.n_hi < a->n_sites &&
                   (reinterpret_cast<uintptr_t>(a->sector.keys) & 15) == 0),
              "%s: two-word keys need 0 < n_hi < n_sites and 16-byte aligned keys", who);
  return EDG_OK;
}

}  // namespace

namespace {

// Launch shape shared by the kernels: the digit plan and the shared-memory
// parts.
struct Setup {
  edg::DigitPlan P;
  Parts parts;
  bool wide, many;  // two-word keys; more than 16 sites
};

constexpr int kDiagCap = 64 * 1024;                     // diagonals kept in shared memory
constexpr int kMostDigits = kThreads * EDG_MAX_SITES;  // digits of a CTA's rows

inline int round16(int64_t b) { return (int)((b + 15) & ~int64_t(15)); }

int make_setup(const edg_assembly* a, const char* who, Setup* s) {
  s->wide = a->sector.key_words == 2;
  s->many = a->n_sites > 16;
  EDG_REQUIRE(edg::make_digit_plan(&s->P, a->loc_dims, a->n_sites, a->sector.key_words, a->sector.n_hi),
              "%s: bad local dimensions", who);
  s->parts = Parts{};
  s->parts.digits = round16((int64_t)kThreads * a->n_sites);
  const int64_t terms = (int64_t)a->n_terms * (1 + 2 * EDG_MAX_OPS) * 4;
  const int64_t mask = (int64_t)((a->n_terms + 31) / 32) * a->n_sites * a->dmax * 4;
  if (terms <= kTableCap) s->parts.terms = round16(terms);
  if (mask <= kTableCap) s->parts.mask = round16(mask);
  return EDG_OK;
}

// n_tables: tables whose amplitudes and kets are staged where they fit (0:
// unknown, read from global memory).
template <typename V, typename K, int NS>
int launch_fill(const edg_assembly* a, const Setup& s, int n_tables, int from_diag, const int64_t* offsets,
                int32_t* cols, double* vals, int64_t* row_nnz, double* diag, uint8_t* present, int32_t* err,
                int32_t* merged, cudaStream_t stream) {
  Parts p = s.parts;
  p.windows = (int)((sizeof(V) + 4) * kWindow * kWarps);
  const int64_t e = (int64_t)n_tables * a->dmax * a->dmax;
  if (e * (int64_t)(sizeof(V) + 1) <= kTableCap) {
    p.amp = round16(e * (int64_t)sizeof(V));
    p.ket = round16(e);
  }
  auto kern = fill_k<V, K, NS>;
  cudaError_t ce = edg::allow_smem(kern, p.windows + kMostDigits + 3 * kTableCap + 32);
  int occ = 1;
  if (ce == cudaSuccess) ce = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, p.total());
  if (ce != cudaSuccess) return edg::cuda_status(ce, "edg_assemble_fill");
  kern<<<edg::grid_for(a->sector.n, kThreads, occ > 0 ? occ : 1), kThreads, p.total(), stream>>>(
      *a, s.P, p, n_tables, from_diag, offsets, cols, vals, row_nnz, diag, present, err, merged);
  return EDG_OK;
}

template <typename V, typename K, int NS>
int launch_diag(const edg_assembly* a, const Setup& s, const double* base, const uint8_t* base_present, int has_extra,
                double re, double im, double* diag, uint8_t* present, cudaStream_t stream) {
  const size_t table = (size_t)a->n_dterms * a->dmax * sizeof(V);
  const int in_smem = table <= (size_t)kDiagCap;
  const size_t smem = s.parts.digits + (in_smem ? table : 0);
  auto kern = diag_k<V, K, NS>;
  cudaError_t e = edg::allow_smem(kern, kMostDigits + kDiagCap);
  if (e != cudaSuccess) return edg::cuda_status(e, "edg_assemble_diag");
  kern<<<edg::grid_for(a->sector.n, kThreads, 16), kThreads, smem, stream>>>(
      *a, s.P, in_smem, base, base_present, has_extra, re, im, diag, present);
  return EDG_OK;
}

// The kernel instance of an assembly: value type, key type, site bound.
#define EDG_ASM_DISPATCH(FN, ...)                                                      \
  (a->complex_values                                                                   \
       ? (s.wide ? FN<Cplx, edg::u128, EDG_MAX_SITES>(__VA_ARGS__)                     \
                 : s.many ? FN<Cplx, uint64_t, EDG_MAX_SITES>(__VA_ARGS__)             \
                          : FN<Cplx, uint64_t, 16>(__VA_ARGS__))                       \
       : (s.wide ? FN<Real, edg::u128, EDG_MAX_SITES>(__VA_ARGS__)                     \
                 : s.many ? FN<Real, uint64_t, EDG_MAX_SITES>(__VA_ARGS__)             \
                          : FN<Real, uint64_t, 16>(__VA_ARGS__)))

int run_diag(const edg_assembly* a, const Setup& s, const double* base, const uint8_t* base_present, int has_extra,
             double re, double im, double* diag, uint8_t* present, cudaStream_t stream) {
  return EDG_ASM_DISPATCH(launch_diag, a, s, base, base_present, has_extra, re, im, diag, present, stream);
}

int run_fill(const edg_assembly* a, int n_tables, const int64_t* offsets, int32_t* cols, double* vals, int64_t* row_nnz,
             double* diag, uint8_t* present, int32_t* err, int32_t* merged, cudaStream_t stream) {
  Setup s;
  int st = make_setup(a, "edg_assemble_fill", &s);
  if (st) return st;
  if (a->n_dterms > 0 || a->n_terms == 0) {
    st = run_diag(a, s, nullptr, nullptr, 0, 0.0, 0.0, diag, present, stream);
    if (st) return st;
  }
  if (a->n_terms == 0) {
    cudaError_t e = cudaMemsetAsync(row_nnz, 0, sizeof(int64_t) * (size_t)a->sector.n, stream);
    return e == cudaSuccess ? EDG_OK : edg::cuda_status(e, "edg_assemble_fill");
  }
  return EDG_ASM_DISPATCH(launch_fill, a, s, n_tables, a->n_dterms > 0 ? 1 : 0, offsets, cols, vals, row_nnz, diag, present,
                          err, merged, stream);
}

}  // namespace

extern "C" int edg_assemble_count(const edg_assembly* a, int64_t* row_bound, cudaStream_t stream) {
  int st = check_assembly(a, "edg_assemble_count");
  if (st) return st;
  if (a->sector.n == 0) return EDG_OK;
  Setup s;
  if ((st = make_setup(a, "edg_assemble_count", &s))) return st;
  auto kern = s.wide ? count_k<edg::u128, EDG_MAX_SITES> : s.many ? count_k<uint64_t, EDG_MAX_SITES>
                                                                  : count_k<uint64_t, 16>;
  cudaError_t e = edg::allow_smem(kern, kMostDigits + 2 * kTableCap);
  if (e != cudaSuccess) return edg::cuda_status(e, "edg_assemble_count");
  kern<<<edg::grid_for(a->sector.n, kThreads, 8), kThreads, s.parts.total(), stream>>>(*a, s.P, s.parts, row_bound);
  EDG_CHECK_LAUNCH("edg_assemble_count");
  return EDG_OK;
}

extern "C" int edg_assemble_fill(const edg_assembly* a, const int64_t* offsets, int32_t* tmp_cols, double* tmp_vals,
                                 int64_t* row_nnz, double* diag, uint8_t* diag_present, int32_t* error_flag,
                                 cudaStream_t stream) {
  int st = check_assembly(a, "edg_assemble_fill");
  if (st) return st;
  if (a->sector.n == 0) return EDG_OK;
  st = run_fill(a, 0, offsets, tmp_cols, tmp_vals, row_nnz, diag, diag_present, error_flag, nullptr, stream);
  if (st) return st;
  EDG_CHECK_LAUNCH("edg_assemble_fill");
  return EDG_OK;
}

extern "C" int edg_assemble_rows(const edg_assembly* a, int32_t n_tables, const int64_t* offsets, int32_t* cols, double* vals,
                                 int64_t* row_nnz, double* diag, uint8_t* diag_present, int32_t* flags,
                                 cudaStream_t stream) {
  int st = check_assembly(a, "edg_assemble_rows");
  if (st) return st;
  EDG_REQUIRE(n_tables >= 0 && flags != nullptr, "edg_assemble_rows: bad arguments");
  if (a->sector.n == 0) return EDG_OK;
  st = run_fill(a, n_tables, offsets, cols, vals, row_nnz, diag, diag_present, flags, flags + 1, stream);
  if (st) return st;
  EDG_CHECK_LAUNCH("edg_assemble_rows");
  return EDG_OK;
}

extern "C" int edg_assemble_diag(const edg_assembly* a, const double* base, const uint8_t* base_present,
                                 int32_t has_extra, double extra_re, double extra_im, double* diag,
                                 uint8_t* diag_present, cudaStream_t stream) {
  int st = check_assembly(a, "edg_assemble_diag");
  if (st) return st;
  if (a->sector.n == 0) return EDG_OK;
  EDG_REQUIRE((base == nullptr) == (base_present == nullptr), "edg_assemble_diag: base needs its presence flags");
  Setup s;
  if ((st = make_setup(a, "edg_assemble_diag", &s))) return st;
  st = run_diag(a, s, base, base_present, has_extra, extra_re, extra_im, diag, diag_present, stream);
  if (st) return st;
  EDG_CHECK_LAUNCH("edg_assemble_diag");
  return EDG_OK;
}

extern "C" int edg_assemble_compact(int64_t n_rows, int32_t complex_values, const int64_t* offsets,
                                    const int32_t* tmp_cols, const double* tmp_vals, const int64_t* rowptr,
                                    int32_t* cols, double* vals, cudaStream_t stream) {
  EDG_REQUIRE(n_rows >= 0, "edg_assemble_compact: negative size");
  if (n_rows == 0) return EDG_OK;
  unsigned grid = edg::grid_for(n_rows * 32, kThreads);
  if (complex_values)
    compact_k<2><<<grid, kThreads, 0, stream>>>(n_rows, offsets, tmp_cols, tmp_vals, rowptr, cols, vals);
  else
    compact_k<1><<<grid, kThreads, 0, stream>>>(n_rows, offsets, tmp_cols, tmp_vals, rowptr, cols, vals);
  EDG_CHECK_LAUNCH("edg_assemble_compact");
  return EDG_OK;
}
