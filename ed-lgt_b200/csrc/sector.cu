// Symmetry-sector enumeration on packed keys of one or two 64-bit words.
//
// One level = one site.  Candidate i of level `depth` is (parent p = i / d,
// state c = i % d) with d = loc_dims[depth]; it survives when
//   * the state is allowed on that site (string constraints),
//   * every global U(1) sum can still reach its target (branch and bound with
//     the remaining min/max) or, at the last site, equals it; Z2 parities are
//     checked at the last site,
//   * every link pair and n-body constraint whose last site is `depth` holds.
// Survivors are written in candidate order, which keeps parents in order and
// states ascending: the final level is sorted by key, i.e. lexicographically
// (the order produced by edlgt/symmetries/symmetry_sector.py:785-967).
// Digits of earlier sites are decoded from the parent key.  Kernels are
// templated on the key type (keys.cuh): uint64_t, or a 128-bit pair of words
// when the key space exceeds 63 bits.
//
// Two forms.  While a level has at most `cap` prefixes, all levels run inside
// one cooperative launch (levels_coop_k): the sizes stay on the device, so
// there is no host round trip per level.  A level that would not fit is left
// to the per-level pair of launches (level_count, level_fill), whose caller
// reads its size and allocates it.
#include "gridbar.cuh"
#include "internal.cuh"
#include "keys.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;
constexpr int kMaxGlob = 4;

template <typename K>
__device__ __forceinline__ int digit_of(const edg_sector_tables& t, K key, int site) {
  return edg::key_digit(key, site, t.n_hi, t.strides[site], (uint64_t)t.loc_dims[site]);
}

// Evaluates candidate (parent_key, parent sums, state c) at `depth`.
template <typename K>
__device__ __forceinline__ bool candidate_ok(const edg_sector_tables& t, int depth, K pkey,
                                             const int32_t* __restrict__ psums, int c, int32_t* nsums) {
  const int n = t.n_sites, dm = t.dmax;
  if (!t.site_allowed[depth * dm + c]) return false;
  const bool last = depth == n - 1;
  for (int g = 0; g < t.n_glob; ++g) {
    int32_t v = t.glob_val[((int64_t)g * n + depth) * dm + c];
    int32_t prev = psums ? psums[g] : 0;
    if (t.glob_type == 0) {
      int32_t s = prev + v;
      nsums[g] = s;
      int32_t target = t.glob_target[g];
      if (last) {
        if (s != target) return false;
      } else {
        if (target < s + t.glob_rem_min[g * (n + 1) + depth + 1]) return false;
        if (target > s + t.glob_rem_max[g * (n + 1) + depth + 1]) return false;
      }
    } else {
      int32_t s = prev ^ v;
      nsums[g] = s;
      if (last && s != t.glob_target[g]) return false;
    }
  }
  for (int p = t.pair_start[depth]; p < t.pair_start[depth + 1]; ++p) {
    int s0 = t.pair_s0[p], s1 = t.pair_s1[p], dir = t.pair_dir[p];
    int c0 = s0 == depth ? c : digit_of(t, pkey, s0);
    int c1 = s1 == depth ? c : digit_of(t, pkey, s1);
    int32_t v = t.link_val[(((int64_t)dir * 2 + 0) * n + s0) * dm + c0] +
                t.link_val[(((int64_t)dir * 2 + 1) * n + s1) * dm + c1];
    if (v != t.link_target[dir]) return false;
  }
  if (t.nb_start != nullptr) {
    for (int a = t.nb_start[depth]; a < t.nb_start[depth + 1]; ++a) {
      int id = t.nb_id[a];
      int32_t acc = 0;
      for (int q = t.nb_site_start[id]; q < t.nb_site_start[id + 1]; ++q) {
        int s = t.nb_sites[q];
        int cs = s == depth ? c : digit_of(t, pkey, s);
        int32_t v = t.nb_val[((int64_t)id * n + s) * dm + cs];
        acc = t.nbody_type == 0 ? acc + v : (acc ^ v);
      }
      if (acc != t.nb_target[id]) return false;
    }
  }
  return true;
}

struct Level {
  int depth;
  int d;
  int n_glob;
  const uint64_t* prev_keys;
  const int32_t* prev_sums;
  int64_t n_cand;
};

template <typename K>
__device__ __forceinline__ bool eval_candidate(const edg_sector_tables& t, const Level& L, int64_t i, K* key_out,
                                               int32_t* sums_out) {
  if (i >= L.n_cand) return false;
  int64_t p = i / L.d;
  int c = (int)(i - p * L.d);
  K pkey = L.depth == 0 ? K(0) : edg::ld_key<K>(L.prev_keys, p);
  const int32_t* ps = (L.depth == 0 || L.n_glob == 0) ? nullptr : L.prev_sums + p * L.n_glob;
  bool ok = candidate_ok(t, L.depth, pkey, ps, c, sums_out);
  *key_out = pkey + edg::key_step<K>((int64_t)c * (int64_t)t.strides[L.depth], L.depth, t.n_hi);
  return ok;
}

template <typename K>
__global__ void __launch_bounds__(kThreads) level_count(edg_sector_tables t, Level L, int64_t* __restrict__ block_counts) {
  int64_t base = (int64_t)blockIdx.x * kTile;
  int local = 0;
  K key;
  int32_t sums[kMaxGlob];
#pragma unroll 1
  for (int it = 0; it < kItems; ++it) {
    int64_t i = base + (int64_t)it * kThreads + threadIdx.x;
    local += eval_candidate(t, L, i, &key, sums) ? 1 : 0;
  }
  // block reduction of per-thread counts
  __shared__ int warp_tot[kThreads / 32];
  int v = local;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < kThreads / 32; ++w) s += warp_tot[w];
    block_counts[blockIdx.x] = s;
  }
}

template <typename K>
__global__ void __launch_bounds__(kThreads) level_fill(edg_sector_tables t, Level L, const int64_t* __restrict__ block_offsets,
                                                       uint64_t* __restrict__ next_keys, int32_t* __restrict__ next_sums) {
  __shared__ int warp_cnt[kThreads / 32];
  __shared__ int64_t running;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) running = block_offsets[blockIdx.x];
  __syncthreads();
  int64_t base = (int64_t)blockIdx.x * kTile;
#pragma unroll 1
  for (int it = 0; it < kItems; ++it) {
    int64_t i = base + (int64_t)it * kThreads + threadIdx.x;
    K key = 0;
    int32_t sums[kMaxGlob];
    bool ok = eval_candidate(t, L, i, &key, sums);
    unsigned ballot = __ballot_sync(0xffffffffu, ok);
    if (lane == 0) warp_cnt[warp] = __popc(ballot);
    __syncthreads();
    int64_t pos = running;
    for (int w = 0; w < warp; ++w) pos += warp_cnt[w];
    pos += __popc(ballot & ((1u << lane) - 1u));
    if (ok) {
      edg::st_key(next_keys, pos, key);
      for (int g = 0; g < L.n_glob; ++g) next_sums[pos * L.n_glob + g] = sums[g];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = 0;
      for (int w = 0; w < kThreads / 32; ++w) s += warp_cnt[w];
      running += s;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// All levels in one cooperative launch.  Per level every CTA owns an equal run
// of parents.  A thread decides all children of a parent at once: the digits
// its constraints need are decoded once per parent instead of once per child,
// by multiplications with reciprocals (64-bit divisions were most of a level's
// time), and the surviving children are bits of a mask kept in shared memory.
// After one grid-wide wait the CTAs know their output offsets and write the
// children from the masks (each level is evaluated once); a second wait
// publishes the level.  Bound by the two waits and the latency of a few
// dependent loads, about 4 us a level, until levels have 10^5 prefixes.
// ---------------------------------------------------------------------------
constexpr int kCoopThreads = 512;
constexpr int kCoopSmem = 200 * 1024;
constexpr int kHead = 72;  // int64 words: level sizes [64] | levels done | prefixes | buffer | error | barrier

struct Coop {
  uint64_t* keys[2];
  int32_t* sums[2];
  int64_t* head;
  int64_t* counts;  // [2][grid]
  int64_t cap;
};

// floor(x / y) for x < 2^63, y < 2^62, inv = 1 / y: the f64 estimate, then its
// remainder divided the same way, then a correction by one.
__device__ __forceinline__ uint64_t fast_div(uint64_t x, uint64_t y, double inv) {
  uint64_t q = (uint64_t)((double)x * inv);
  int64_t r = (int64_t)(x - q * y);
  const int64_t c = (int64_t)floor((double)r * inv);
  q += (uint64_t)c;
  r -= c * (int64_t)y;
  if (r < 0) --q;
  if (r >= (int64_t)y) ++q;
  return q;
}

template <typename K, typename M>
__global__ void __launch_bounds__(kCoopThreads, 1) levels_coop_k(const __grid_constant__ edg_sector_tables t,
                                                                 const Coop C) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  M* const masks = reinterpret_cast<M*>(sm_raw);
  __shared__ double inv_stride[EDG_MAX_SITES], inv_dim[EDG_MAX_SITES];
  __shared__ int64_t red[2][kCoopThreads / 32];
  __shared__ int64_t tot[2];
  __shared__ int wsum[kCoopThreads / 32];
  __shared__ uint32_t allowed_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)gridDim.x, n = t.n_sites, dm = t.dmax, ng = t.n_glob;
  int* const err = reinterpret_cast<int*>(C.head + 67);
  edg::GridSync gs{reinterpret_cast<unsigned*>(C.head + 68), err};
  for (int s = tid; s < n; s += kCoopThreads) {
    inv_stride[s] = 1.0 / (double)t.strides[s];
    inv_dim[s] = 1.0 / (double)t.loc_dims[s];
  }
  auto digit = [&](K key, int s) -> int {
    const uint64_t d = (uint64_t)t.loc_dims[s];
    const uint64_t q = fast_div(edg::key_word(key, s, t.n_hi), t.strides[s], inv_stride[s]);
    return (int)(q - fast_div(q, d, inv_dim[s]) * d);
  };
  int64_t n_prev = 1;
  int cur = 0, depth = 0;
  for (; depth < n; ++depth) {
    const int d = t.loc_dims[depth];
    if (d > (int)sizeof(M) * 8) break;
    const bool last = depth == n - 1;
    if (tid == 0) {
      uint32_t m = 0u;
      for (int c = 0; c < d; ++c) m |= t.site_allowed[depth * dm + c] ? 1u << c : 0u;
      allowed_s = m;
    }
    __syncthreads();
    const int64_t p0 = n_prev * blockIdx.x / G, p1 = n_prev * (blockIdx.x + 1) / G;
    const uint64_t* const pk = C.keys[cur];
    const int32_t* const ps = C.sums[cur];
    // ---- which children of each parent survive ----
    int64_t mine = 0;
    for (int64_t p = p0 + tid; p < p1; p += kCoopThreads) {
      K key = K(0);
      if (depth > 0) {
        if constexpr (sizeof(K) == 8)
          key = pk[p];
        else
          key = ((K)pk[2 * p + 1] << 64) | (K)pk[2 * p];
      }
      uint32_t m = allowed_s;
      for (int g = 0; g < ng; ++g) {
        const int32_t prev = depth > 0 ? ps[p * ng + g] : 0;
        const int32_t* val = t.glob_val + ((int64_t)g * n + depth) * dm;
        const int32_t target = t.glob_target[g];
        if (t.glob_type == 0) {
          const int32_t lo = last ? 0 : t.glob_rem_min[g * (n + 1) + depth + 1];
          const int32_t hi = last ? 0 : t.glob_rem_max[g * (n + 1) + depth + 1];
          for (uint32_t b = m; b; b &= b - 1u) {
            const int c = __ffs(b) - 1;
            const int32_t s = prev + __ldg(val + c);
            if (target < s + lo || target > s + hi) m &= ~(1u << c);
          }
        } else if (last) {
          for (uint32_t b = m; b; b &= b - 1u) {
            const int c = __ffs(b) - 1;
            if ((prev ^ __ldg(val + c)) != target) m &= ~(1u << c);
          }
        }
      }
      for (int q = t.pair_start[depth]; q < t.pair_start[depth + 1] && m; ++q) {
        const int s0 = t.pair_s0[q], s1 = t.pair_s1[q], dir = t.pair_dir[q];
        const int32_t* v0 = t.link_val + (((int64_t)dir * 2 + 0) * n + s0) * dm;
        const int32_t* v1 = t.link_val + (((int64_t)dir * 2 + 1) * n + s1) * dm;
        const int32_t target = t.link_target[dir];
        const int32_t f0 = s0 == depth ? 0 : __ldg(v0 + digit(key, s0));
        const int32_t f1 = s1 == depth ? 0 : __ldg(v1 + digit(key, s1));
        for (uint32_t b = m; b; b &= b - 1u) {
          const int c = __ffs(b) - 1;
          const int32_t v = (s0 == depth ? __ldg(v0 + c) : f0) + (s1 == depth ? __ldg(v1 + c) : f1);
          if (v != target) m &= ~(1u << c);
        }
      }
      if (t.nb_start != nullptr) {
        for (int q = t.nb_start[depth]; q < t.nb_start[depth + 1] && m; ++q) {
          const int id = t.nb_id[q];
          const int32_t* val = t.nb_val + (int64_t)id * n * dm;
          int32_t acc = 0;
          int here = 0;  // factors on this level's site
          for (int e = t.nb_site_start[id]; e < t.nb_site_start[id + 1]; ++e) {
            const int s = t.nb_sites[e];
            if (s == depth) {
              ++here;
              continue;
            }
            const int32_t v = __ldg(val + (int64_t)s * dm + digit(key, s));
            acc = t.nbody_type == 0 ? acc + v : (acc ^ v);
          }
          for (uint32_t b = m; b; b &= b - 1u) {
            const int c = __ffs(b) - 1;
            const int32_t v = __ldg(val + (int64_t)depth * dm + c);
            const int32_t x = t.nbody_type == 0 ? acc + here * v : ((here & 1) ? acc ^ v : acc);
            if (x != t.nb_target[id]) m &= ~(1u << c);
          }
        }
      }
      masks[p - p0] = (M)m;
      mine += __popc(m);
    }
    // ---- offsets of the CTAs ----
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane == 0) red[0][warp] = mine;
    __syncthreads();
    int64_t* const cnt = C.counts + (int64_t)(depth & 1) * G;
    if (tid == 0) {
      int64_t a = 0;
      for (int w = 0; w < kCoopThreads / 32; ++w) a += red[0][w];
      cnt[blockIdx.x] = a;
    }
    if (!gs.wait()) return;
    int64_t below = 0, all = 0;
    for (int b = tid; b < G; b += kCoopThreads) {
      const int64_t v = __ldcg(cnt + b);
      all += v;
      below += b < (int)blockIdx.x ? v : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      all += __shfl_xor_sync(0xffffffffu, all, o);
      below += __shfl_xor_sync(0xffffffffu, below, o);
    }
    if (lane == 0) {
      red[0][warp] = all;
      red[1][warp] = below;
    }
    __syncthreads();
    if (tid < 2) {
      int64_t a = 0;
      for (int w = 0; w < kCoopThreads / 32; ++w) a += red[tid][w];
      tot[tid] = a;
    }
    __syncthreads();
    const int64_t total = tot[0];
    int64_t base = tot[1];
    if (total > C.cap) break;  // too many prefixes: the caller goes on from this level
    // ---- children in order ----
    uint64_t* const nk = C.keys[cur ^ 1];
    int32_t* const nsum = C.sums[cur ^ 1];
    const int64_t stride = (int64_t)t.strides[depth];
    for (int64_t q0 = p0; q0 < p1; q0 += kCoopThreads) {
      const int64_t p = q0 + tid;
      const uint32_t m = p < p1 ? (uint32_t)masks[p - p0] : 0u;
      const int c0 = __popc(m);
      int inc = c0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (lane == 31) wsum[warp] = inc;
      __syncthreads();
      int before = 0, here = 0;
      for (int w = 0; w < kCoopThreads / 32; ++w) {
        before += w < warp ? wsum[w] : 0;
        here += wsum[w];
      }
      if (m) {
        K key = K(0);
        if (depth > 0) {
          if constexpr (sizeof(K) == 8)
            key = pk[p];
          else
            key = ((K)pk[2 * p + 1] << 64) | (K)pk[2 * p];
        }
        int64_t at = base + before + inc - c0;
        for (uint32_t b = m; b; b &= b - 1u, ++at) {
          const int c = __ffs(b) - 1;
          const K kk = key + edg::key_step<K>((int64_t)c * stride, depth, t.n_hi);
          edg::st_key(nk, at, kk);
          for (int g = 0; g < ng; ++g) {
            const int32_t prev = depth > 0 ? ps[p * ng + g] : 0;
            const int32_t v = __ldg(t.glob_val + ((int64_t)g * n + depth) * dm + c);
            nsum[at * ng + g] = t.glob_type == 0 ? prev + v : (prev ^ v);
          }
        }
      }
      base += here;
      __syncthreads();
    }
    if (blockIdx.x == 0 && tid == 0) C.head[depth] = total;
    cur ^= 1;
    n_prev = total;
    if (!gs.wait()) return;
    if (total == 0) {
      ++depth;
      break;
    }
  }
  if (blockIdx.x == 0 && tid == 0) {
    C.head[64] = depth;
    C.head[65] = n_prev;
    C.head[66] = cur;
  }
}

int check_tables(const edg_sector_tables* t, int32_t depth, int64_t n_prev, const char* who) {
  EDG_REQUIRE(t != nullptr, "%s: null tables", who);
  EDG_REQUIRE(t->n_sites > 0 && t->n_sites <= EDG_MAX_SITES, "%s: n_sites out of range", who);
  EDG_REQUIRE(depth >= 0 && depth < t->n_sites, "%s: depth %d out of range", who, depth);
  EDG_REQUIRE(t->n_glob >= 0 && t->n_glob <= kMaxGlob, "%s: at most %d global symmetries", who, kMaxGlob);
  EDG_REQUIRE(n_prev >= 0, "%s: negative parent count", who);
  EDG_REQUIRE(depth == 0 ? n_prev == 1 : true, "%s: level 0 expands one empty parent", who);
  EDG_REQUIRE(t->key_words == 0 || t->key_words == 1 || t->key_words == 2, "%s: key_words must be 1 or 2", who);
  EDG_REQUIRE(t->key_words != 2 || (t->n_hi > 0 && t->n_hi < t->n_sites), "%s: n_hi out of range", who);
  return EDG_OK;
}

}  // namespace

extern "C" int64_t edg_sector_levels_work_elems(void) { return kHead + 2 * edg::kSmCount; }

extern "C" int64_t edg_sector_levels_cap(const edg_sector_tables* t) {
  if (t == nullptr || t->n_sites < 1 || t->n_sites > EDG_MAX_SITES) return -1;
  int d = 1;
  for (int s = 0; s < t->n_sites; ++s) d = t->loc_dims[s] > d ? t->loc_dims[s] : d;
  const int bytes = d <= 8 ? 1 : d <= 16 ? 2 : 4;
  return (int64_t)edg::kSmCount * (kCoopSmem / bytes - 1);
}

extern "C" int edg_sector_levels(const edg_sector_tables* t, uint64_t* keys0, uint64_t* keys1, int32_t* sums0,
                                 int32_t* sums1, int64_t cap, int64_t* work, cudaStream_t stream) {
  int st = check_tables(t, 0, 1, "edg_sector_levels");
  if (st) return st;
  EDG_REQUIRE(keys0 && keys1 && sums0 && sums1 && work, "edg_sector_levels: null pointer");
  EDG_REQUIRE(cap >= 1 && cap <= edg_sector_levels_cap(t), "edg_sector_levels: cap out of range");
  EDG_REQUIRE(t->key_words != 2 || ((reinterpret_cast<uintptr_t>(keys0) | reinterpret_cast<uintptr_t>(keys1)) & 15) == 0,
              "edg_sector_levels: two-word keys must be 16-byte aligned");
  int dmx = 1;
  for (int s = 0; s < t->n_sites; ++s) {
    EDG_REQUIRE(t->loc_dims[s] > 0 && t->loc_dims[s] <= t->dmax, "edg_sector_levels: bad local dimension");
    dmx = t->loc_dims[s] > dmx ? t->loc_dims[s] : dmx;
  }
  const bool wide = t->key_words == 2;
  const int bytes = dmx <= 8 ? 1 : dmx <= 16 ? 2 : 4;
  const void* kern =
      wide ? (bytes == 1 ? (const void*)levels_coop_k<edg::u128, uint8_t>
                         : bytes == 2 ? (const void*)levels_coop_k<edg::u128, uint16_t>
                                      : (const void*)levels_coop_k<edg::u128, uint32_t>)
           : (bytes == 1 ? (const void*)levels_coop_k<uint64_t, uint8_t>
                         : bytes == 2 ? (const void*)levels_coop_k<uint64_t, uint16_t>
                                      : (const void*)levels_coop_k<uint64_t, uint32_t>);
  int dev = 0, n_sm = 0, coop = 0, occ = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  const int64_t grid = n_sm < edg::kSmCount ? n_sm : edg::kSmCount;
  const int64_t smem = ((cap + grid - 1) / grid + 1) * bytes;  // masks of a CTA's parents
  if (e == cudaSuccess) e = edg::allow_smem(kern, kCoopSmem);
  if (e == cudaSuccess && smem <= kCoopSmem)  // (more on a device with fewer SMs: a run of parents is longer)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kCoopThreads, (size_t)smem);
  if (e == cudaSuccess) e = cudaMemsetAsync(work, 0, kHead * sizeof(int64_t), stream);
  if (e != cudaSuccess) return edg::cuda_status(e, "edg_sector_levels");
  if (!coop || occ < 1) {  // nothing done: the caller runs every level itself
    const int64_t none[3] = {0, 1, 0};
    e = cudaMemcpyAsync(work + 64, none, sizeof(none), cudaMemcpyHostToDevice, stream);
    return e == cudaSuccess ? EDG_OK : edg::cuda_status(e, "edg_sector_levels");
  }
  Coop c{{keys0, keys1}, {sums0, sums1}, work, work + kHead, cap};
  edg_sector_tables tab = *t;
  void* args[] = {&tab, &c};
  e = cudaLaunchCooperativeKernel(kern, dim3((unsigned)grid), dim3(kCoopThreads), args, (size_t)smem, stream);
  return e == cudaSuccess ? EDG_OK : edg::cuda_status(e, "edg_sector_levels");
}

extern "C" int64_t edg_sector_level_blocks(int64_t n_candidates) {
  return edg::ceil_div(n_candidates > 0 ? n_candidates : 1, kTile);
}

extern "C" int edg_sector_level_count(const edg_sector_tables* t, int32_t depth, const uint64_t* prev_keys,
                                      const int32_t* prev_sums, int64_t n_prev, int64_t* block_offsets,
                                      int64_t* scratch, cudaStream_t stream) {
  int st = check_tables(t, depth, n_prev, "edg_sector_level_count");
  if (st) return st;
  int d = t->loc_dims[depth];
  EDG_REQUIRE(d > 0 && d <= t->dmax, "edg_sector_level_count: bad local dimension");
  EDG_REQUIRE(t->key_words != 2 || depth == 0 || (reinterpret_cast<uintptr_t>(prev_keys) & 15) == 0,
              "edg_sector_level_count: two-word keys must be 16-byte aligned");
  Level L{depth, d, t->n_glob, prev_keys, prev_sums, n_prev * (int64_t)d};
  int64_t nb = edg_sector_level_blocks(L.n_cand);
  if (t->key_words == 2)
    level_count<edg::u128><<<(unsigned)nb, kThreads, 0, stream>>>(*t, L, block_offsets);
  else
    level_count<uint64_t><<<(unsigned)nb, kThreads, 0, stream>>>(*t, L, block_offsets);
  EDG_CHECK_LAUNCH("edg_sector_level_count");
  return edg_scan_i64(block_offsets, block_offsets, nb, scratch, stream);
}

extern "C" int edg_sector_level_fill(const edg_sector_tables* t, int32_t depth, const uint64_t* prev_keys,
                                     const int32_t* prev_sums, int64_t n_prev, const int64_t* block_offsets,
                                     uint64_t* next_keys, int32_t* next_sums, cudaStream_t stream) {
  int st = check_tables(t, depth, n_prev, "edg_sector_level_fill");
  if (st) return st;
  int d = t->loc_dims[depth];
  EDG_REQUIRE(d > 0 && d <= t->dmax, "edg_sector_level_fill: bad local dimension");
  EDG_REQUIRE(t->key_words != 2 || ((depth == 0 || (reinterpret_cast<uintptr_t>(prev_keys) & 15) == 0) &&
                                     (reinterpret_cast<uintptr_t>(next_keys) & 15) == 0),
              "edg_sector_level_fill: two-word keys must be 16-byte aligned");
  Level L{depth, d, t->n_glob, prev_keys, prev_sums, n_prev * (int64_t)d};
  int64_t nb = edg_sector_level_blocks(L.n_cand);
  if (t->key_words == 2)
    level_fill<edg::u128><<<(unsigned)nb, kThreads, 0, stream>>>(*t, L, block_offsets, next_keys, next_sums);
  else
    level_fill<uint64_t><<<(unsigned)nb, kThreads, 0, stream>>>(*t, L, block_offsets, next_keys, next_sums);
  EDG_CHECK_LAUNCH("edg_sector_level_fill");
  return EDG_OK;
}

// ---------------------------------------------------------------------------
// key <-> configuration conversion
// ---------------------------------------------------------------------------
namespace {

__global__ void keys_to_configs_k(const uint64_t* __restrict__ keys, int64_t n, int n_sites,
                                  const int32_t* __restrict__ loc_dims, uint16_t* __restrict__ configs) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t k = keys[i];
    for (int s = n_sites - 1; s >= 0; --s) {
      uint64_t d = (uint64_t)loc_dims[s];
      configs[i * n_sites + s] = (uint16_t)(k % d);
      k /= d;
    }
  }
}

__global__ void configs_to_keys_k(const uint16_t* __restrict__ configs, int64_t n, int n_sites,
                                  const uint64_t* __restrict__ strides, uint64_t* __restrict__ keys) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t k = 0;
    for (int s = 0; s < n_sites; ++s) k += (uint64_t)configs[i * n_sites + s] * strides[s];
    keys[i] = k;
  }
}

// Two-word keys: digits of sites [n_hi, n) from the low word, of [0, n_hi)
// from the high word.
__global__ void keys_to_configs_wide_k(const uint64_t* __restrict__ keys, int64_t n, int n_sites, int n_hi,
                                       const int32_t* __restrict__ loc_dims, uint16_t* __restrict__ configs) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t lo = keys[2 * i], hi = keys[2 * i + 1];
    for (int s = n_sites - 1; s >= n_hi; --s) {
      uint64_t d = (uint64_t)loc_dims[s];
      configs[i * n_sites + s] = (uint16_t)(lo % d);
      lo /= d;
    }
    for (int s = n_hi - 1; s >= 0; --s) {
      uint64_t d = (uint64_t)loc_dims[s];
      configs[i * n_sites + s] = (uint16_t)(hi % d);
      hi /= d;
    }
  }
}

__global__ void configs_to_keys_wide_k(const uint16_t* __restrict__ configs, int64_t n, int n_sites, int n_hi,
                                       const uint64_t* __restrict__ strides, uint64_t* __restrict__ keys) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t hi = 0, lo = 0;
    for (int s = 0; s < n_hi; ++s) hi += (uint64_t)configs[i * n_sites + s] * strides[s];
    for (int s = n_hi; s < n_sites; ++s) lo += (uint64_t)configs[i * n_sites + s] * strides[s];
    keys[2 * i] = lo;
    keys[2 * i + 1] = hi;
  }
}

}  // namespace

extern "C" int edg_keys_to_configs_wide(const uint64_t* keys, int64_t n, int32_t n_sites, int32_t n_hi,
                                        const int32_t* loc_dims, uint16_t* configs, cudaStream_t stream) {
  EDG_REQUIRE(n >= 0 && n_sites > 1 && n_sites <= EDG_MAX_SITES && n_hi > 0 && n_hi < n_sites,
              "edg_keys_to_configs_wide: bad sizes");
  if (n == 0) return EDG_OK;
  keys_to_configs_wide_k<<<edg::grid_for(n, 256), 256, 0, stream>>>(keys, n, n_sites, n_hi, loc_dims, configs);
  EDG_CHECK_LAUNCH("edg_keys_to_configs_wide");
  return EDG_OK;
}

extern "C" int edg_configs_to_keys_wide(const uint16_t* configs, int64_t n, int32_t n_sites, int32_t n_hi,
                                        const uint64_t* strides, uint64_t* keys, cudaStream_t stream) {
  EDG_REQUIRE(n >= 0 && n_sites > 1 && n_sites <= EDG_MAX_SITES && n_hi > 0 && n_hi < n_sites,
              "edg_configs_to_keys_wide: bad sizes");
  if (n == 0) return EDG_OK;
  configs_to_keys_wide_k<<<edg::grid_for(n, 256), 256, 0, stream>>>(configs, n, n_sites, n_hi, strides, keys);
  EDG_CHECK_LAUNCH("edg_configs_to_keys_wide");
  return EDG_OK;
}

extern "C" int edg_keys_to_configs(const uint64_t* keys, int64_t n, int32_t n_sites, const int32_t* loc_dims,
                                   uint16_t* configs, cudaStream_t stream) {
  EDG_REQUIRE(n >= 0 && n_sites > 0 && n_sites <= EDG_MAX_SITES, "edg_keys_to_configs: bad sizes");
  if (n == 0) return EDG_OK;
  keys_to_configs_k<<<edg::grid_for(n, 256), 256, 0, stream>>>(keys, n, n_sites, loc_dims, configs);
  EDG_CHECK_LAUNCH("edg_keys_to_configs");
  return EDG_OK;
}

extern "C" int edg_configs_to_keys(const uint16_t* configs, int64_t n, int32_t n_sites, const uint64_t* strides,
                                   uint64_t* keys, cudaStream_t stream) {
  EDG_REQUIRE(n >= 0 && n_sites > 0 && n_sites <= EDG_MAX_SITES, "edg_configs_to_keys: bad sizes");
  if (n == 0) return EDG_OK;
  configs_to_keys_k<<<edg::grid_for(n, 256), 256, 0, stream>>>(configs, n, n_sites, strides, keys);
  EDG_CHECK_LAUNCH("edg_configs_to_keys");
  return EDG_OK;
}
