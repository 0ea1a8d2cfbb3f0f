// Matrix-free Z_n lattice gauge theory with staggered fermions: zero-momentum
// basis construction and the batched matvec.
//
// Basis.  The Gauss-law sector is indexed densely (gidx = colex rank of the
// occupied-site set * zn^n_cot + cotree fields as base-zn digits), so a
// configuration is decoded from its index by peeling the spanning tree from
// the leaves (every tree field follows from the Gauss law at its child site)
// and encoded with two small tables (cotree digits per key byte, colex rank
// per occupation pattern).  The representatives of the translation orbits
// are marked in a bitmap over gidx (one thread per 64-bit word, no atomics),
// counted, scanned and written out in gidx order; then every orbit member's
// gidx gets, in a 4-byte orbit table, the row of its representative, the
// stabiliser size and the fermionic sign of the translation that maps the
// representative onto it.  This replaces the reference's translation table
// found by binary search and its projector B
// (edlgt/symmetries/translational_sym.py:567-819).
//
// Matvec.  One thread per representative row (persistent grid): the diagonal
// from the key; the Gauss index of each hopping and plaquette image from the
// row's own, its entry in the orbit table (4 bytes), and the x row that the
// entry names (nvec interleaved instances, one 32-byte sector for 8 f32
// instances).  Element: amplitude * sign *
// sqrt(|Stab r'| / |Stab r|), the zero-momentum projection of
// nbody_data_momentum (translational_sym.py:1394-1969) done on the fly.
#include <type_traits>

#include "internal.cuh"

namespace {

template <int ZN>
struct Zn {
  static constexpr int kBits = ZN == 2 ? 1 : 2;
  static constexpr uint64_t kMask = (1ull << kBits) - 1;
  __device__ static __forceinline__ int field(uint64_t key, int l) { return (int)((key >> (kBits * l)) & kMask); }
  __device__ static __forceinline__ int mod(int v) {
    v %= ZN;
    return v < 0 ? v + ZN : v;
  }
};

// Key of T(config): the lane array (one lane per row of sites) rotated by
// whole rows, then every lane rotated by whole sites; the same on the
// occupation bits.
__device__ __forceinline__ uint64_t translate_key(const edg_zn_translation& T, uint64_t key, int F, int N, int lane_f,
                                                  int lx) {
  const uint64_t fmask = (F == 64) ? ~0ull : ((1ull << F) - 1);
  const uint32_t mmask = (uint32_t)((1u << N) - 1);
  uint64_t f = key & fmask;
  uint32_t m = (uint32_t)(key >> F) & mmask;
  if (T.sf) f = ((f << T.sf) | (f >> (F - T.sf))) & fmask;
  if (T.sx) f = ((f << T.sx) & T.hif) | ((f >> (lane_f - T.sx)) & T.lof);
  if (T.sm) m = ((m << T.sm) | (m >> (N - T.sm))) & mmask;
  if (T.smx) m = ((m << T.smx) & T.him) | ((m >> (lx - T.smx)) & T.lom);
  return f | ((uint64_t)m << F);
}

// Parity (1 = negative) of the reordering T makes among occupied sites: rows
// that wrap in y pass every fermion of the rows that do not; inside a row the
// wrapping sites pass the staying ones.
__device__ __forceinline__ int translate_sign(const edg_zn_translation& T, uint32_t occ, int lx, int ly) {
  int par = (__popc(occ & T.ylow) & __popc(occ & T.yhigh)) & 1;
  if (T.smx) {
    for (int y = 0; y < ly; ++y) {
      const uint32_t row = occ >> (lx * y);
      par ^= (__popc(row & T.xhead) & __popc(row & T.xtail)) & 1;
    }
  }
  return par;
}

// Configuration of Gauss index g.
template <int ZN>
__device__ uint64_t decode(const edg_zn_lattice& L, uint64_t g) {
  using Z = Zn<ZN>;
  const uint64_t r = g / (uint64_t)L.pow_cot;
  uint32_t d = (uint32_t)(g - r * (uint64_t)L.pow_cot);
  const uint32_t occ = L.rank_occ[r];
  uint64_t key = (uint64_t)occ << L.field_bits;
  for (int c = 0; c < L.n_cot; ++c) {
    const uint32_t e = d % ZN;
    d /= ZN;
    key |= (uint64_t)e << (Z::kBits * L.cot_link[c]);
  }
  for (int k = 0; k < L.n_sites - 1; ++k) {
    const int v = L.peel_site[k];
    int s = (int)((occ >> v) & 1u) - (int)((L.odd_mask >> v) & 1u);
#pragma unroll
    for (int o = 0; o < 3; ++o) s -= L.peel_osign[k][o] * Z::field(key, L.peel_other[k][o]);
    key |= (uint64_t)Z::mod(L.peel_sign[k] * s) << (Z::kBits * L.peel_link[k]);
  }
  return key;
}

__device__ __forceinline__ int lane_bits(const edg_zn_lattice& L) { return 2 * L.link_bits * L.lx; }

// True when key is the smallest key of its orbit and no stabiliser element
// maps it onto minus itself.
__device__ bool is_rep(const edg_zn_lattice& L, uint64_t key) {
  const uint32_t occ = (uint32_t)(key >> L.field_bits);
  const int lf = lane_bits(L);
  for (int g = 1; g < L.n_group; ++g) {
    const uint64_t k2 = translate_key(L.group[g], key, L.field_bits, L.n_sites, lf, L.lx);
    if (k2 < key) return false;
    if (k2 == key && translate_sign(L.group[g], occ, L.lx, L.ly)) return false;
  }
  return true;
}

template <int ZN>
__global__ void __launch_bounds__(256) zn_mark_k(const __grid_constant__ edg_zn_lattice L, uint64_t* __restrict__ bitmap,
                                                 int64_t* __restrict__ counts, int64_t n_words) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (int64_t)gridDim.x * blockDim.x) {
    uint64_t bits = 0;
    const uint64_t g0 = (uint64_t)w * 64;
    for (int j = 0; j < 64; ++j) {
      const uint64_t g = g0 + j;
      if (g >= (uint64_t)L.n_gauss) break;
      if (is_rep(L, decode<ZN>(L, g))) bits |= 1ull << j;
    }
    bitmap[w] = bits;
    counts[w] = __popcll(bits);
  }
}

template <int ZN>
__global__ void __launch_bounds__(256) zn_fill_k(const __grid_constant__ edg_zn_lattice L, const uint64_t* __restrict__ bitmap,
                                                 const int64_t* __restrict__ offsets, uint64_t* __restrict__ keys,
                                                 int64_t n_words) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (int64_t)gridDim.x * blockDim.x) {
    uint64_t bits = bitmap[w];
    int64_t o = offsets[w];
    while (bits) {
      const int j = __ffsll((long long)bits) - 1;
      bits &= bits - 1;
      keys[o++] = decode<ZN>(L, (uint64_t)w * 64 + j);
    }
  }
}

// Gauss index from the two lookup tables (held in shared memory by the callers).
__device__ __forceinline__ uint64_t gauss_index(const uint64_t* __restrict__ lut, const uint32_t* __restrict__ rank,
                                                uint64_t key, int F, int n_chunks, uint64_t pow_cot) {
  uint64_t g = (uint64_t)rank[(uint32_t)(key >> F)] * pow_cot;
  for (int k = 0; k < n_chunks; ++k) g += lut[k * 256 + (int)((key >> (8 * k)) & 255u)];
  return g;
}

__device__ void load_tables(const edg_zn_lattice& L, uint64_t* lut, uint32_t* rank) {
  const int n_chunks = (L.field_bits + 7) / 8;
  for (int i = threadIdx.x; i < n_chunks * 256; i += blockDim.x) lut[i] = L.chunk_lut[i];
  for (int i = threadIdx.x; i < (1 << L.n_sites); i += blockDim.x) rank[i] = L.occ_rank[i];
  __syncthreads();
}

__global__ void __launch_bounds__(256) zn_orbit_k(const __grid_constant__ edg_zn_lattice L, const uint64_t* __restrict__ keys, int64_t n_rows,
                                                  uint32_t* __restrict__ orbit) {
  extern __shared__ uint64_t zsm[];
  const int n_chunks = (L.field_bits + 7) / 8;
  uint64_t* lut = zsm;
  uint32_t* rank = (uint32_t*)(zsm + n_chunks * 256);
  load_tables(L, lut, rank);
  const int lf = lane_bits(L);
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t key = keys[r];
    const uint32_t occ = (uint32_t)(key >> L.field_bits);
    int stab = 0;
    for (int g = 0; g < L.n_group; ++g)
      stab += translate_key(L.group[g], key, L.field_bits, L.n_sites, lf, L.lx) == key;
    int dv = 0;
    while (dv < L.n_div - 1 && L.divisors[dv] != stab) ++dv;
    const uint32_t base = (uint32_t)r | ((uint32_t)dv << 28);
    for (int g = 0; g < L.n_group; ++g) {
      const uint64_t k2 = translate_key(L.group[g], key, L.field_bits, L.n_sites, lf, L.lx);
      const uint32_t sg = (uint32_t)translate_sign(L.group[g], occ, L.lx, L.ly);
      orbit[gauss_index(lut, rank, k2, L.field_bits, n_chunks, (uint64_t)L.pow_cot)] = base | (sg << 31);
    }
  }
}

// ---------------------------------------------------------------- matvec
// Policy of data that is read once in a long while: first to leave L2, not
// kept in L1.
__device__ __forceinline__ uint64_t once_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// One x row (the nvec interleaved instances of a column) in 16-byte loads, or
// in 32-byte ones (WIDE), which fetch a whole sector a lane.
template <typename T, int NV, bool WIDE, bool ONCE>
__device__ __forceinline__ void load_row(const T* __restrict__ p, T (&v)[NV], uint64_t policy) {
  constexpr int kBytes = WIDE ? 32 : (NV * sizeof(T) >= 16 ? 16 : sizeof(T));
  constexpr int kVec = kBytes / sizeof(T);
  static_assert(NV % kVec == 0);
#pragma unroll
  for (int i = 0; i < NV; i += kVec) {
    if constexpr (sizeof(T) == 4 && kVec == 8) {
      if constexpr (ONCE)
        asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;"
            : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3]), "=f"(v[i + 4]), "=f"(v[i + 5]),
              "=f"(v[i + 6]), "=f"(v[i + 7])
            : "l"(p + i), "l"(policy));
      else
        asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
            : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3]), "=f"(v[i + 4]), "=f"(v[i + 5]),
              "=f"(v[i + 6]), "=f"(v[i + 7])
            : "l"(p + i));
    } else if constexpr (sizeof(T) == 4 && kVec == 4) {
      if constexpr (ONCE)
        asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
            : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3])
            : "l"(p + i), "l"(policy));
      else
        asm("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
            : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3])
            : "l"(p + i));
    } else if constexpr (sizeof(T) == 8 && kVec == 4) {
      if constexpr (ONCE)
        asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f64 {%0, %1, %2, %3}, [%4], %5;"
            : "=d"(v[i]), "=d"(v[i + 1]), "=d"(v[i + 2]), "=d"(v[i + 3])
            : "l"(p + i), "l"(policy));
      else
        asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
            : "=d"(v[i]), "=d"(v[i + 1]), "=d"(v[i + 2]), "=d"(v[i + 3])
            : "l"(p + i));
    } else if constexpr (sizeof(T) == 8 && kVec == 2) {
      if constexpr (ONCE)
        asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
            : "=d"(v[i]), "=d"(v[i + 1])
            : "l"(p + i), "l"(policy));
      else
        asm("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v[i]), "=d"(v[i + 1]) : "l"(p + i));
    } else {
      v[i] = __ldg(p + i);
    }
  }
}

template <typename T, int NV, bool WIDE>
__device__ __forceinline__ void store_row(T* __restrict__ p, const T (&v)[NV]) {
#pragma unroll
  for (int i = 0; i < NV; i += WIDE ? 32 / (int)sizeof(T) : 1) {
    if constexpr (WIDE && sizeof(T) == 4)
      asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + i), "f"(v[i]), "f"(v[i + 1]),
                   "f"(v[i + 2]), "f"(v[i + 3]), "f"(v[i + 4]), "f"(v[i + 5]), "f"(v[i + 6]), "f"(v[i + 7])
                   : "memory");
    else if constexpr (WIDE)
      asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p + i), "d"(v[i]), "d"(v[i + 1]), "d"(v[i + 2]),
                   "d"(v[i + 3])
                   : "memory");
    else
      p[i] = v[i];
  }
}

// Asynchronous copy of one orbit entry to shared memory.
__device__ __forceinline__ void copy_entry(uint32_t* to, const uint32_t* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}

// Sum of E^2 over the links of a key.
template <int ZN>
__device__ __forceinline__ double field_energy(const edg_zn_lattice& L, uint64_t key) {
  const uint64_t f = key & (~0ull >> (64 - L.field_bits));
  if constexpr (ZN == 2) {
    const int n1 = __popcll(f);
    return (double)(L.n_links - n1) * L.esq[0] + (double)n1 * L.esq[1];
  } else {
    const uint64_t low = 0x5555555555555555ull;
    const int n3 = ZN == 4 ? __popcll(f & (f >> 1) & low) : 0;
    const int n1 = __popcll(f & low) - n3, n2 = __popcll((f >> 1) & low) - n3;
    return (double)(L.n_links - n1 - n2 - n3) * L.esq[0] + (double)n1 * L.esq[1] + (double)n2 * L.esq[2] +
           (double)n3 * L.esq[3];
  }
}

constexpr int kMvThreads = 256;

// What a row's images need of the lattice, a link or a plaquette at a time.
// Raising the field of link l adds step[l] to a configuration's cotree index
// (its Gauss index within one occupation), less zn step[l] from the top value;
// lowering is the opposite; step is zero for a tree link, whose field is no
// digit.  The index of an image is so the row's own plus a constant and one
// term for each field that wraps (mod 2^32; pow_cot is below), not a fresh
// encoding from the tables.  Masks are over links, one bit each.
struct alignas(16) ZnLink {
  uint32_t pair, tail;     // occupation bits of both sites, of the tail
  uint32_t between, sign;  // Jordan-Wigner mask, 1 for eta < 0
  uint32_t mask, step, turn, unused;  // turn = zn step
};
struct alignas(16) ZnPlaq {
  uint32_t m0, m1, m2, m3;  // links raised, raised, lowered, lowered by U_p
  uint32_t t0, t1, t2, t3;  // their turns
  uint32_t step, unused[3]; // steps of the raised less those of the lowered
};
struct ZnTables {
  ZnLink link[2 * EDG_ZN_MAX_SITES];
  ZnPlaq plaq[EDG_ZN_MAX_SITES];
};

ZnTables make_tables(const edg_zn_lattice* L) {
  ZnTables t{};
  uint32_t w = 1;
  for (int c = 0; c < L->n_cot; ++c, w *= (uint32_t)L->zn) t.link[L->cot_link[c]].step = w;
  for (int l = 0; l < L->n_links; ++l) {
    ZnLink& k = t.link[l];
    k.tail = 1u << L->link_tail[l];
    k.pair = k.tail | (1u << L->link_head[l]);
    k.between = L->link_between[l];
    k.sign = L->link_eta[l] < 0 ? 1u : 0u;
    k.mask = 1u << l;
    k.turn = (uint32_t)L->zn * k.step;
  }
  for (int p = 0; p < L->n_sites; ++p) {
    ZnPlaq& k = t.plaq[p];
    const ZnLink* l[4];
    for (int i = 0; i < 4; ++i) l[i] = &t.link[L->plaq[p][i]];
    k.m0 = l[0]->mask, k.m1 = l[1]->mask, k.m2 = l[2]->mask, k.m3 = l[3]->mask;
    k.t0 = l[0]->turn, k.t1 = l[1]->turn, k.t2 = l[2]->turn, k.t3 = l[3]->turn;
    k.step = l[0]->step + l[1]->step - l[2]->step - l[3]->step;
  }
  return t;
}

// The even bits of a word, closed up.
__device__ __forceinline__ uint32_t even_bits(uint64_t v) {
  v &= 0x5555555555555555ull;
  v = (v | v >> 1) & 0x3333333333333333ull;
  v = (v | v >> 2) & 0x0F0F0F0F0F0F0F0Full;
  v = (v | v >> 4) & 0x00FF00FF00FF00FFull;
  v = (v | v >> 8) & 0x0000FFFF0000FFFFull;
  return (uint32_t)(v | v >> 16);
}

// Links of a key at the top value and at zero, one bit a link.
template <int ZN>
__device__ __forceinline__ uint32_t top_links(uint64_t key) {
  if constexpr (ZN == 2) return (uint32_t)key;
  if constexpr (ZN == 3) return even_bits(key >> 1);
  return even_bits(key & (key >> 1));
}
template <int ZN>
__device__ __forceinline__ uint32_t zero_links(uint64_t key) {
  if constexpr (ZN == 2) return ~(uint32_t)key;
  return even_bits(~(key | (key >> 1)));
}

// CTAs an SM and bytes of x rows a thread has in flight together.  Rows of a
// whole sector or more: 128 bytes at two CTAs; at three the 245,518,920-row
// product gets slower (8 f32: 67.9 ms against 55.3, 4 f64: 61.6 against 51.3),
// since the plaquette rows that more threads read leave L2 sooner, where
// 4,592,128 rows gain less (0.645 ms against 0.655, 0.493 against 0.568).
// Narrower rows: three CTAs (4 f32: 48.5 ms against 50.5, 0.423 against 0.525).
template <typename T, int NV>
constexpr int ctas_of() { return NV * sizeof(T) >= 32 ? 2 : 3; }
template <typename T, int NV>
constexpr int group_of() {
  constexpr int g = (NV * sizeof(T) >= 32 ? 128 : 64) / (NV * (int)sizeof(T));
  return g > 8 ? 8 : g;
}

// A thread owns row r.  First the orbit entries of all its images are copied to
// its slots of shared memory (asynchronously: no registers, and no image waits
// for another); then the x rows they name are gathered group by group, hops
// before plaquettes.  slots: [n_links + 2 n_sites][kMvThreads].
// What bounds it, over the rows of one occupation in turn: plaquettes stay
// within that occupation's rows (51 MB of 8 f32 instances on 4 x 3 Z_3), which
// L2 holds; the rows a hop names are spread over another occupation's and come
// from DRAM, half of each 64-byte access unused (225 GB read for 17.7 GB of x,
// y and keys).  Their loads pass L1 by and leave L2 first: 68.6 ms without
// that, 55.3 with it (8 f32, 245,518,920 rows).  Below one sector a row the
// instructions of the index arithmetic bound it (1 f32: 33 ms).  Encoding every
// image from the tables and one orbit load before each group of four x rows:
// 105 ms and 60.
// WIDE: x and y rows in 32-byte accesses (both 32-byte aligned): a 16-byte load
// asks for every sector twice.
template <int ZN, typename T, int NV, bool WIDE>
__global__ void __launch_bounds__(kMvThreads, ctas_of<T, NV>()) zn_matvec_k(const __grid_constant__ edg_zn_lattice L,
                                                          const __grid_constant__ ZnTables tab, const edg_zn_basis B,
                                                          const double* __restrict__ coup, const T* __restrict__ x,
                                                          T* __restrict__ y) {
  constexpr int kGroup = group_of<T, NV>();
  extern __shared__ uint32_t slots[];
  __shared__ double c_t[NV], c_m[NV], c_e[NV], c_b[NV];
  __shared__ double sq_div[8], isq_div[8];
  __shared__ ZnTables S;
  for (int i = threadIdx.x; i < (int)(sizeof(ZnTables) / 16); i += kMvThreads)
    reinterpret_cast<uint4*>(&S)[i] = reinterpret_cast<const uint4*>(&tab)[i];
  if (threadIdx.x < NV) {
    c_t[threadIdx.x] = -coup[4 * threadIdx.x + 0];
    c_m[threadIdx.x] = coup[4 * threadIdx.x + 1];
    c_e[threadIdx.x] = coup[4 * threadIdx.x + 2];
    c_b[threadIdx.x] = coup[4 * threadIdx.x + 3];
  }
  if (threadIdx.x < 8) {
    const double d = threadIdx.x < L.n_div ? (double)L.divisors[threadIdx.x] : 1.0;
    sq_div[threadIdx.x] = sqrt(d);
    isq_div[threadIdx.x] = 1.0 / sqrt(d);
  }
  __syncthreads();
  const int F = L.field_bits, n_chunks = (F + 7) / 8;
  const uint64_t pc = (uint64_t)L.pow_cot;
  uint32_t* const mine = slots + threadIdx.x;
  const uint64_t policy = once_policy();
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < B.n_rows; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t key = __ldcs((const unsigned long long*)B.keys + r);
    const uint32_t occ = (uint32_t)(key >> F);
    int n_hop = 0;
    uint32_t neg = 0;  // signs of the hops, by slot
    uint32_t self;
    {
      uint32_t dig = 0;
      for (int k = 0; k < n_chunks; ++k) dig += (uint32_t)__ldg(L.chunk_lut + k * 256 + (int)((key >> (8 * k)) & 255u));
      const uint32_t* const own = B.orbit + (uint64_t)__ldg(L.occ_rank + occ) * pc;
      self = own[dig];
      const uint32_t top = top_links<ZN>(key), zero = zero_links<ZN>(key);
      // hopping: c^dag_tail U c_head (tail empty, head full) and its conjugate
#pragma unroll 4
      for (int l = 0; l < L.n_links; ++l) {
        const ZnLink k = S.link[l];
        const uint32_t at = occ & k.pair;
        if (at != 0 && at != k.pair) {
          const bool up = (at & k.tail) == 0;
          const uint32_t d = ((up ? top : zero) & k.mask) ? k.step - k.turn : k.step;
          neg |= ((__popc(occ & k.between) ^ k.sign) & 1u) << n_hop;
          copy_entry(mine + n_hop * kMvThreads,
                     B.orbit + (uint64_t)__ldg(L.occ_rank + (occ ^ k.pair)) * pc + (uint32_t)(up ? dig + d : dig - d));
          ++n_hop;
        }
      }
      // plaquettes U_p and U_p^dag
#pragma unroll 2
      for (int p = 0; p < L.n_sites; ++p) {
        const ZnPlaq k = S.plaq[p];
        uint32_t a = dig + k.step, b = dig - k.step;
        if (top & k.m0) a -= k.t0;
        if (top & k.m1) a -= k.t1;
        if (zero & k.m2) a += k.t2;
        if (zero & k.m3) a += k.t3;
        if (zero & k.m0) b += k.t0;
        if (zero & k.m1) b += k.t1;
        if (top & k.m2) b -= k.t2;
        if (top & k.m3) b -= k.t3;
        uint32_t* const to = mine + (L.n_links + 2 * p) * kMvThreads;
        copy_entry(to, own + a);
        copy_entry(to + kMvThreads, own + b);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    double sum[NV], out[NV];
    auto gather = [&](auto hops, const uint32_t* list, int n) {
      // a multiple of four images for the plaquettes: no partial group up to there
      constexpr bool kFull = !decltype(hops)::value && kGroup <= 4;
#pragma unroll
      for (int v = 0; v < NV; ++v) sum[v] = 0.0;
      for (int i0 = 0; i0 < n; i0 += kGroup, list += kGroup * kMvThreads) {
        uint32_t e[kGroup];
        T xv[kGroup][NV];
#pragma unroll
        for (int c = 0; c < kGroup; ++c) {
          e[c] = kFull || i0 + c < n ? list[c * kMvThreads] : 0xFFFFFFFFu;
          if (e[c] != 0xFFFFFFFFu) load_row<T, NV, WIDE, decltype(hops)::value>(x + (int64_t)(e[c] & 0x0FFFFFFFu) * NV, xv[c], policy);
        }
#pragma unroll
        for (int c = 0; c < kGroup; ++c)
          if (e[c] != 0xFFFFFFFFu) {
            uint32_t sg = e[c];
            if constexpr (decltype(hops)::value) sg ^= neg << (31 - c);
            const double s = sq_div[(e[c] >> 28) & 7u];
            const double a = __hiloint2double(__double2hiint(s) ^ (int)(sg & 0x80000000u), __double2loint(s));
#pragma unroll
            for (int v = 0; v < NV; ++v) sum[v] = fma(a, (double)xv[c][v], sum[v]);
          }
        if constexpr (decltype(hops)::value) neg >>= kGroup;
      }
    };
    const double inv_s = isq_div[(self >> 28) & 7u];
    gather(std::true_type{}, mine, n_hop);
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = c_t[v] * (inv_s * sum[v]);
    gather(std::false_type{}, mine + L.n_links * kMvThreads, 2 * L.n_sites);
    const double esq = field_energy<ZN>(L, key);
    const double mass = (double)(__popc(occ & L.even_mask) - __popc(occ & ~L.even_mask));
    T xr[NV];
    load_row<T, NV, WIDE, false>(x + r * NV, xr, policy);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double d = c_e[v] * esq + c_m[v] * mass;
      xr[v] = (T)(fma(d, (double)xr[v], fma(c_b[v], inv_s * sum[v], out[v])));
    }
    store_row<T, NV, WIDE>(y + r * NV, xr);
  }
}

int check_lattice(const edg_zn_lattice* L, const char* where) {
  EDG_REQUIRE(L != nullptr, "%s: null lattice", where);
  EDG_REQUIRE(L->zn >= 2 && L->zn <= 4, "%s: zn must be 2, 3 or 4", where);
  EDG_REQUIRE(L->link_bits == (L->zn == 2 ? 1 : 2), "%s: link_bits must be %d", where, L->zn == 2 ? 1 : 2);
  EDG_REQUIRE(L->n_sites >= 4 && L->n_sites <= EDG_ZN_MAX_SITES && L->n_sites == L->lx * L->ly,
              "%s: need 4 <= lx * ly <= %d", where, EDG_ZN_MAX_SITES);
  EDG_REQUIRE(L->lx % 2 == 0 && L->ly >= 2, "%s: need lx even and ly >= 2", where);
  EDG_REQUIRE(L->n_links == 2 * L->n_sites && L->field_bits == L->link_bits * L->n_links &&
                  L->field_bits + L->n_sites <= 64,
              "%s: inconsistent link/field sizes", where);
  EDG_REQUIRE(L->n_group >= 1 && L->n_group <= EDG_ZN_MAX_GROUP, "%s: n_group must be 1..%d", where, EDG_ZN_MAX_GROUP);
  EDG_REQUIRE(L->n_div >= 1 && L->n_div <= 8, "%s: n_div must be 1..8", where);
  EDG_REQUIRE(L->n_gauss > 0 && L->n_gauss <= 0xFFFFFFFFll, "%s: Gauss index range must fit 32 bits", where);
  EDG_REQUIRE(L->pow_cot > 0 && L->pow_cot <= 0xFFFFFFFFll && L->n_gauss % L->pow_cot == 0,
              "%s: bad pow_cot", where);
  EDG_REQUIRE(L->n_cot == L->n_links - L->n_sites + 1, "%s: n_cot must be links - sites + 1", where);
  EDG_REQUIRE(L->chunk_lut != nullptr && L->occ_rank != nullptr && L->rank_occ != nullptr,
              "%s: null lookup table", where);
  return EDG_OK;
}

size_t table_smem(const edg_zn_lattice* L) {
  return sizeof(uint64_t) * 256 * (size_t)((L->field_bits + 7) / 8) + sizeof(uint32_t) * ((size_t)1 << L->n_sites);
}

// most: of any lattice (table_smem and a row's slots grow with its sites).
constexpr size_t kMostTables = sizeof(uint64_t) * 256 * 8 + (sizeof(uint32_t) << EDG_ZN_MAX_SITES);
constexpr size_t kMostSlots = sizeof(uint32_t) * kMvThreads * 4 * EDG_ZN_MAX_SITES;

template <typename K>
int set_smem(K kernel, size_t smem, size_t most, const char* where) {
  if (smem > 40 * 1024) {  // 48 KB less the kernels' own static arrays
    cudaError_t e = edg::allow_smem(kernel, most);
    if (e != cudaSuccess) return edg::cuda_status(e, where);
  }
  return EDG_OK;
}

// Persistent grid: resident CTAs per SM times the SM count.
template <typename K>
unsigned persistent_grid(K kernel, int threads, size_t smem, int64_t n_items) {
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return edg::grid_for(n_items, threads, per_sm);
}

template <int ZN, typename T, int NV, bool WIDE>
int launch_matvec(const edg_zn_lattice* L, const edg_zn_basis* B, const double* coup, const void* x, void* y,
                  cudaStream_t stream) {
  if constexpr (!WIDE && NV * sizeof(T) % 32 == 0) {
    if ((((uintptr_t)x | (uintptr_t)y) & 31u) == 0) return launch_matvec<ZN, T, NV, true>(L, B, coup, x, y, stream);
  }
  const size_t smem = sizeof(uint32_t) * kMvThreads * (size_t)(L->n_links + 2 * L->n_sites);
  auto kern = zn_matvec_k<ZN, T, NV, WIDE>;
  int st = set_smem(kern, smem, kMostSlots, "edg_zn_matvec");
  if (st != EDG_OK) return st;
  const unsigned grid = persistent_grid(kern, kMvThreads, smem, B->n_rows);
  kern<<<grid, kMvThreads, smem, stream>>>(*L, make_tables(L), *B, coup, (const T*)x, (T*)y);
  EDG_CHECK_LAUNCH("edg_zn_matvec");
  return EDG_OK;
}

template <int ZN>
int dispatch_matvec(const edg_zn_lattice* L, const edg_zn_basis* B, const double* coup, int nvec, int dtype,
                    const void* x, void* y, cudaStream_t s) {
#define EDG_ZN_MV(NV)                                                           \
  case NV:                                                                      \
    return dtype == 0 ? launch_matvec<ZN, double, NV, false>(L, B, coup, x, y, s)      \
                      : launch_matvec<ZN, float, NV, false>(L, B, coup, x, y, s);
  switch (nvec) {
    EDG_ZN_MV(1)
    EDG_ZN_MV(2)
    EDG_ZN_MV(4)
    EDG_ZN_MV(8)
  }
#undef EDG_ZN_MV
  edg::set_error("edg_zn_matvec: nvec must be 1, 2, 4 or 8");
  return EDG_ERR_ARG;
}

}  // namespace

extern "C" int64_t edg_zn_bitmap_words(const edg_zn_lattice* L) {
  if (L == nullptr || L->n_gauss <= 0) return -1;
  return (L->n_gauss + 63) / 64;
}

extern "C" int edg_zn_mark(const edg_zn_lattice* L, uint64_t* bitmap, int64_t* counts, cudaStream_t stream) {
  int st = check_lattice(L, "edg_zn_mark");
  if (st != EDG_OK) return st;
  EDG_REQUIRE(bitmap != nullptr && counts != nullptr, "edg_zn_mark: null output");
  const int64_t words = (L->n_gauss + 63) / 64;
  const unsigned grid = edg::grid_for(words, 256);
  switch (L->zn) {
    case 2: zn_mark_k<2><<<grid, 256, 0, stream>>>(*L, bitmap, counts, words); break;
    case 3: zn_mark_k<3><<<grid, 256, 0, stream>>>(*L, bitmap, counts, words); break;
    default: zn_mark_k<4><<<grid, 256, 0, stream>>>(*L, bitmap, counts, words); break;
  }
  EDG_CHECK_LAUNCH("edg_zn_mark");
  return EDG_OK;
}

extern "C" int edg_zn_fill(const edg_zn_lattice* L, const uint64_t* bitmap, const int64_t* offsets, uint64_t* keys,
                           cudaStream_t stream) {
  int st = check_lattice(L, "edg_zn_fill");
  if (st != EDG_OK) return st;
  EDG_REQUIRE(bitmap != nullptr && offsets != nullptr && keys != nullptr, "edg_zn_fill: null argument");
  const int64_t words = (L->n_gauss + 63) / 64;
  const unsigned grid = edg::grid_for(words, 256);
  switch (L->zn) {
    case 2: zn_fill_k<2><<<grid, 256, 0, stream>>>(*L, bitmap, offsets, keys, words); break;
    case 3: zn_fill_k<3><<<grid, 256, 0, stream>>>(*L, bitmap, offsets, keys, words); break;
    default: zn_fill_k<4><<<grid, 256, 0, stream>>>(*L, bitmap, offsets, keys, words); break;
  }
  EDG_CHECK_LAUNCH("edg_zn_fill");
  return EDG_OK;
}

extern "C" int edg_zn_orbit_table(const edg_zn_lattice* L, const uint64_t* keys, int64_t n_rows, uint32_t* orbit,
                                  cudaStream_t stream) {
  int st = check_lattice(L, "edg_zn_orbit_table");
  if (st != EDG_OK) return st;
  EDG_REQUIRE(keys != nullptr && orbit != nullptr, "edg_zn_orbit_table: null argument");
  EDG_REQUIRE(n_rows >= 0 && n_rows < 0x0FFFFFFFll, "edg_zn_orbit_table: n_rows must be below 2^28 - 1");
  cudaError_t e = cudaMemsetAsync(orbit, 0xFF, sizeof(uint32_t) * (size_t)L->n_gauss, stream);
  if (e != cudaSuccess) return edg::cuda_status(e, "edg_zn_orbit_table: memset");
  if (n_rows == 0) return EDG_OK;
  const size_t smem = table_smem(L);
  st = set_smem(zn_orbit_k, smem, kMostTables, "edg_zn_orbit_table");
  if (st != EDG_OK) return st;
  const unsigned grid = persistent_grid(zn_orbit_k, 256, smem, n_rows);
  zn_orbit_k<<<grid, 256, smem, stream>>>(*L, keys, n_rows, orbit);
  EDG_CHECK_LAUNCH("edg_zn_orbit_table");
  return EDG_OK;
}

extern "C" int edg_zn_matvec(const edg_zn_lattice* L, const edg_zn_basis* B, const double* couplings, int32_t nvec,
                             int32_t dtype, const void* x, void* y, cudaStream_t stream) {
  int st = check_lattice(L, "edg_zn_matvec");
  if (st != EDG_OK) return st;
  EDG_REQUIRE(B != nullptr && couplings != nullptr && x != nullptr && y != nullptr, "edg_zn_matvec: null argument");
  EDG_REQUIRE(dtype == 0 || dtype == 1, "edg_zn_matvec: dtype must be 0 (f64) or 1 (f32)");
  EDG_REQUIRE(B->n_rows >= 0 && B->n_rows < 0x0FFFFFFFll, "edg_zn_matvec: n_rows must be below 2^28 - 1");
  EDG_REQUIRE(B->keys != nullptr && B->orbit != nullptr, "edg_zn_matvec: null basis arrays");
  EDG_REQUIRE(((uintptr_t)x & 15u) == 0, "edg_zn_matvec: x must be 16-byte aligned");
  if (B->n_rows == 0) return EDG_OK;
  switch (L->zn) {
    case 2: return dispatch_matvec<2>(L, B, couplings, nvec, dtype, x, y, stream);
    case 3: return dispatch_matvec<3>(L, B, couplings, nvec, dtype, x, y, stream);
    default: return dispatch_matvec<4>(L, B, couplings, nvec, dtype, x, y, stream);
  }
}
