// Grid-wide barrier of a cooperative launch (every CTA resident).
#pragma once
#include "reorth_bulk.cuh"
#include "edgpu.h"
#include "internal.cuh"

namespace edg {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits (thread 0) until *bar, which only grows, has reached target.  A wait
// longer than 1 s writes EDG_ERR_TIMEOUT to *err; once *err is set no CTA
// waits any more.
__device__ __forceinline__ void grid_wait(const unsigned* bar, unsigned target, int* err) {
  if ((int)(ld_acquire_u32(bar) - target) >= 0) return;
  const uint64_t t0 = bulk::now_ns();
  for (unsigned spins = 1; (int)(ld_acquire_u32(bar) - target) < 0; ++spins) {
    if ((spins & 255u) == 0) {
      if (*(volatile int*)err) break;
      if (bulk::now_ns() - t0 > 1000000000ull) {
        atomicExch(err, EDG_ERR_TIMEOUT);
        break;
      }
    }
  }
}

// One barrier: every CTA adds one to *bar (a multiple of the grid before the
// barrier) and waits for the next multiple.  Arrivals are counted, not reset:
// a counter that the last CTA resets before it releases the others costs two
// more trips to L2 (3 us a barrier against 1.3 us).  Every thread gets false
// once a wait has run out.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, int* err) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned old = atomicAdd(bar, 1u);
    grid_wait(bar, (old / gridDim.x + 1u) * gridDim.x, err);
    __threadfence();
    ok_s = *(volatile int*)err == 0;
  }
  __syncthreads();
  return ok_s != 0;
}

// The barriers of one launch whose counter was zero before it: the target is
// known, so the arrival need not come back before the wait starts.
struct GridSync {
  unsigned* bar;
  int* err;
  unsigned target = 0;
  __device__ __forceinline__ bool wait() {
    __shared__ int ok_s;
    __syncthreads();
    if (gridDim.x == 1) return true;
    target += gridDim.x;
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
      grid_wait(bar, target, err);
      ok_s = *(volatile int*)err == 0;
    }
    __syncthreads();
    return ok_s != 0;
  }
};

// A lane's share of the sum of n values, stride apart, that other CTAs wrote:
// every 32nd, N of them in flight.  A plain loop asks for a few at a time and
// for its remainder one by one, an L2 round trip each.
template <int N>
__device__ __forceinline__ double lane_share(const double* p, int64_t stride, int n) {
  double a = 0.0;
  for (int b = threadIdx.x & 31; b < n; b += 32 * N) {
    double v[N];
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = b + 32 * k < n ? __ldcg(p + (b + 32 * k) * stride) : 0.0;
#pragma unroll
    for (int k = 0; k < N; ++k) a += v[k];
  }
  return a;
}

__device__ __forceinline__ double warp_sum(double a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// CTAs of a small cooperative solve of n rows: one up to 256 rows, where no CTA
// waits for another (a Krylov step at 182 rows 145 us, with three CTAs 198; an
// f64 ground state at 141 rows 0.54 ms, 0.62); past that at least 128 rows a
// CTA, at most one an SM.  Fewer rows a CTA mean more partials in every sum
// (Krylov step at 12,292 rows: 291 us with 83 rows a CTA, 267 with 128, 274
// with 256; f64 ground state at 8,953 rows: 1.13 ms with 64, 1.11 with 128,
// 1.22 with 256).
inline int64_t coop_ctas(int64_t n, int n_sm) {
  if (n <= 256) return 1;
  const int64_t g = (n + 127) / 128, most = n_sm < kSmCount ? n_sm : kSmCount;
  return g < most ? g : most;
}

// Whether a small cooperative solve's product suits its few threads (512 an SM
// against 1,024 to 2,048 of the passes): at most `total` entries, and `per_cta`
// a CTA.  See the callers' figures.
inline bool coop_entries(int64_t nnz, int64_t n, int64_t total, int64_t per_cta) {
  return nnz <= total && nnz <= per_cta * coop_ctas(n, kSmCount);
}

}  // namespace edg
