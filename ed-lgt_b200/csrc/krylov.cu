// Krylov time evolution psi <- exp(-i H dt) psi for a Hermitian sector
// Hamiltonian (real form or complex), with complex Krylov vectors stored in
// complex64 or complex128 and every inner product, the Lanczos recurrence and
// the small exponential in double precision.
//
// One step: v_0 = psi/|psi|; m Lanczos steps w = H v_j, orthogonalised against
// the basis (one classical Gram-Schmidt pass over all previous vectors, or
// two; or against v_{j-1}, v_j only), alpha_j = Re<v_j, w>, beta_{j+1} = |w|;
// then c = |psi| exp(-i T dt) e_1 for the m x m tridiagonal T (Taylor series
// over substeps on the device, exact to double precision) and psi = V c.  A
// breakdown (beta = 0) leaves zero vectors whose block of T decouples from
// e_1, so the step needs no host synchronisation.  Replaces scipy's
// expm_multiply as called by QMB_hamiltonian.time_evolution
// (edlgt/modeling/qmb_hamiltonian.py:334-426).
//
// The basis is stored unnormalised, u_i = beta_i v_i: the update pass writes
// u_{j+1} in the vectors' type while it sums |u_{j+1}|^2, and the factors
// 1 / beta_i go into the coefficients of later passes.  A normalised basis
// needs the updated w written in f64 and a further pass that reads it back
// (40 B a row of a complex64 basis).
//
// Two forms, chosen by the number of rows and entries (one_launch):
//   * large sectors: matvec, dots, coefficients, update as launches over all
//     rows; for the local recurrence on the packed layout the dots are summed
//     in the matvec's epilogue (packed.cu) and a step is two launches;
//   * small sectors (krylov_coop_k): the whole time step is one cooperative
//     launch.  There the rows are a few hundred per SM, every launch costs
//     more than its work, and what is left is two grid-wide waits a step.
#include "gridbar.cuh"
#include "spmv.cuh"

#include <type_traits>

#include <cmath>

namespace {

constexpr int kThreads = 256;
constexpr int kMaxM = 64;
constexpr int kMaxOrth = 14000;  // vectors of edg_krylov_orth (update_k's shared coefficients)
constexpr int64_t kCoopMaxRows = 1024 * edg::kSmCount;  // see krylov_coop_k

template <typename T>
__device__ __forceinline__ edg::cd ldc(const T* p, int64_t i);
template <>
__device__ __forceinline__ edg::cd ldc<float2>(const float2* p, int64_t i) {
  float2 v = p[i];
  return {(double)v.x, (double)v.y};
}
template <>
__device__ __forceinline__ edg::cd ldc<double2>(const double2* p, int64_t i) {
  double2 v = p[i];
  return {v.x, v.y};
}
template <typename T>
__device__ __forceinline__ void stc(T* p, int64_t i, double re, double im);
template <>
__device__ __forceinline__ void stc<float2>(float2* p, int64_t i, double re, double im) {
  p[i] = make_float2((float)re, (float)im);
}
template <>
__device__ __forceinline__ void stc<double2>(double2* p, int64_t i, double re, double im) {
  p[i] = make_double2(re, im);
}

constexpr int kWarps = kThreads / 32;

// Totals of NV doubles per thread over the block, in every thread of warp 0.
template <int NV>
__device__ __forceinline__ void block_totals(double (&v)[NV], double* red /*[kWarps][NV]*/) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if (lane == 0) red[warp * NV + q] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double a = lane < nw ? red[lane * NV + q] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      v[q] = a;
    }
  }
  __syncthreads();
}

// Thread 0 of the last CTA to arrive gets true, with part[0 .. gridDim.x)
// summed in a fixed order in *total; `mine` is this CTA's partial (thread 0).
__device__ __forceinline__ bool last_cta_sum(double mine, double* part, unsigned* ticket, double* total) {
  __shared__ int last;
  if (threadIdx.x == 0) {
    part[blockIdx.x] = mine;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return false;
  __threadfence();
  double a = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) a += __ldcg(part + b);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (threadIdx.x == 0) *ticket = 0u;
  *total = a;
  return threadIdx.x == 0;
}

// |psi|
template <typename T>
__global__ void __launch_bounds__(kThreads) norm_k(const T* __restrict__ x, int64_t n, double* __restrict__ part,
                                                   unsigned* __restrict__ ticket, double* __restrict__ out) {
  __shared__ double red[kWarps];
  double a[1] = {0.0};
  for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < n; r += (int64_t)gridDim.x * kThreads) {
    edg::cd v = ldc<T>(x, r);
    a[0] = fma(v.re, v.re, fma(v.im, v.im, a[0]));
  }
  block_totals<1>(a, red);
  double t;
  if (last_cta_sum(a[0], part, ticket, &t)) out[0] = sqrt(t);
}

// u_0 = psi / |psi| (a zero psi gives zeros); beta[0] = |u_0|
template <typename T>
__global__ void scale_k(const T* __restrict__ src, int64_t n, const double* __restrict__ s, T* __restrict__ dst,
                        double* __restrict__ beta) {
  const double inv = s[0] > 0.0 ? 1.0 / s[0] : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) beta[0] = s[0] > 0.0 ? 1.0 : 0.0;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    edg::cd v = ldc<T>(src, r);
    stc<T>(dst, r, v.re * inv, v.im * inv);
  }
}

// Resident CTAs per SM of the two passes over the basis, and their grids: a
// grid of more CTAs than are resident ends in a part-filled wave.  Rows are
// taken grid-stride, so that at any time the grid reads one window of each
// vector: with a contiguous chunk of rows per CTA the dots of 26 complex64
// vectors (848,614 rows) took 151 us, here 56 (update pass 45).
template <typename T>
constexpr int dot_ctas() { return sizeof(T) == 8 ? 3 : 2; }
constexpr int kUpdateCtas = 3;
template <typename T>
constexpr int local_ctas() { return sizeof(T) == 8 ? 6 : 4; }
constexpr int kTile = 8;  // vectors per dots tile (w is read once per tile)

// partial[b][i] = sum over the CTA's rows of conj(u_i[r]) w[r], ilo <= i <= j
template <typename T>
__global__ void __launch_bounds__(kThreads, dot_ctas<T>()) dots_k(const T* __restrict__ V, int64_t n, int64_t ldv, int ilo, int j,
                                                   const double2* __restrict__ w, double2* __restrict__ partial,
                                                   int ld_i) {
  __shared__ double red[kWarps * kTile * 2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i0 = ilo + (int)blockIdx.y * kTile; i0 <= j; i0 += (int)gridDim.y * kTile) {
    double re[kTile], im[kTile];
#pragma unroll
    for (int t = 0; t < kTile; ++t) re[t] = im[t] = 0.0;
    const T* Vi = V + (int64_t)i0 * ldv;
    const int nt = min(kTile, j + 1 - i0);
    for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < n; r += (int64_t)gridDim.x * kThreads) {
      const double2 wr = w[r];
      T x[kTile];
#pragma unroll
      for (int t = 0; t < kTile; ++t)
        if (t < nt) x[t] = Vi[(int64_t)t * ldv + r];
#pragma unroll
      for (int t = 0; t < kTile; ++t)
        if (t < nt) {
          re[t] = fma((double)x[t].x, wr.x, fma((double)x[t].y, wr.y, re[t]));
          im[t] = fma((double)x[t].x, wr.y, fma(-(double)x[t].y, wr.x, im[t]));
        }
    }
#pragma unroll
    for (int t = 0; t < kTile; ++t) {
      double a = re[t], b = im[t];
      for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
      }
      if (lane == 0) {
        red[(warp * kTile + t) * 2] = a;
        red[(warp * kTile + t) * 2 + 1] = b;
      }
    }
    __syncthreads();
    if (threadIdx.x < nt) {
      double a = 0.0, b = 0.0;
      for (int wi = 0; wi < kWarps; ++wi) {
        a += red[(wi * kTile + threadIdx.x) * 2];
        b += red[(wi * kTile + threadIdx.x) * 2 + 1];
      }
      partial[(int64_t)blockIdx.x * ld_i + i0 + threadIdx.x] = make_double2(a, b);
    }
    __syncthreads();
  }
}

// Coefficients of the update from the dots: coef[i - ilo] = <v_i, w> / beta_i
// with w = ws * (the vector the dots were taken of), coef[j + 1 - ilo] = ws;
// ws = 1 / beta_j for the product itself (pass 0), 1 for a vector already
// updated.  alpha_j = Re <v_j, w>, added to in a second pass.
__global__ void __launch_bounds__(kThreads) coef_k(const double2* __restrict__ partial, int nb, int ld_i, int ilo,
                                                   int j, int pass, const double* __restrict__ beta,
                                                   double2* __restrict__ coef, double* __restrict__ alpha) {
  __shared__ double red[kWarps * 2];
  const int i = ilo + blockIdx.x;
  double a[2] = {0.0, 0.0};
  for (int q = threadIdx.x; q < nb; q += kThreads) {
    const double2 p = partial[(int64_t)q * ld_i + i];
    a[0] += p.x;
    a[1] += p.y;
  }
  block_totals<2>(a, red);
  if (threadIdx.x == 0) {
    const double bj = beta[j], bi = beta[i];
    const double si = bi > 0.0 ? 1.0 / bi : 0.0;
    const double ws = pass > 0 ? 1.0 : (bj > 0.0 ? 1.0 / bj : 0.0);
    const double hr = si * (ws * a[0]), hi = si * (ws * a[1]);
    coef[i - ilo] = make_double2(si * hr, si * hi);
    if (i == j) {
      coef[j + 1 - ilo] = make_double2(ws, 0.0);
      alpha[j] = pass > 0 ? alpha[j] + hr : hr;
    }
  }
}

// x = ws w - sum_{i} coef_i u_i over ilo <= i <= j; written to out (the next
// Krylov vector, in T) with beta_{j+1} = |x|, or back to w (a pass that
// another one follows).
template <typename T>
__global__ void __launch_bounds__(kThreads, kUpdateCtas) update_k(const T* __restrict__ V, int64_t n, int64_t ldv, int ilo, int j,
                                                     const double2* __restrict__ coef, double2* __restrict__ w,
                                                     T* __restrict__ out, double* __restrict__ part,
                                                     unsigned* __restrict__ ticket, double* __restrict__ beta) {
  constexpr int kGroup = 8;  // vectors loaded together
  extern __shared__ __align__(16) double2 hs[];  // [j + 2 - ilo]
  __shared__ double red[kWarps];
  const int nv = j + 1 - ilo;
  for (int t = threadIdx.x; t <= nv; t += kThreads) hs[t] = coef[t];
  __syncthreads();
  const double ws = hs[nv].x;
  const T* Vi = V + (int64_t)ilo * ldv;
  double a[1] = {0.0};
  for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < n; r += (int64_t)gridDim.x * kThreads) {
    const double2 x = w[r];
    double sr = 0.0, si = 0.0;
    for (int i0 = 0; i0 < nv; i0 += kGroup) {
      T v[kGroup];
#pragma unroll
      for (int t = 0; t < kGroup; ++t)
        if (i0 + t < nv) v[t] = Vi[(int64_t)(i0 + t) * ldv + r];
#pragma unroll
      for (int t = 0; t < kGroup; ++t)
        if (i0 + t < nv) {
          const double2 h = hs[i0 + t];
          sr = fma((double)v[t].x, h.x, fma(-(double)v[t].y, h.y, sr));
          si = fma((double)v[t].x, h.y, fma((double)v[t].y, h.x, si));
        }
    }
    const double2 y = make_double2(fma(ws, x.x, -sr), fma(ws, x.y, -si));
    if (out != nullptr)
      stc<T>(out, r, y.x, y.y);
    else
      w[r] = y;
    a[0] = fma(y.x, y.x, fma(y.y, y.y, a[0]));
  }
  if (out == nullptr) return;
  block_totals<1>(a, red);
  double t;
  if (last_cta_sum(a[0], part, ticket, &t)) beta[j + 1] = sqrt(t);
}

// The update of the local recurrence, whose coefficients the product has left
// in coef = {c_{j-1}, c_j, 1 / beta_j}: u_{j+1} = w / beta_j - c_{j-1} u_{j-1} -
// c_j u_j (prev NULL at j = 0) and beta_{j+1}.  A stream of three vectors in
// and one out: what bounds it is how many loads are in flight, so a thread
// takes kRows rows at a time and the registers leave room for four or six CTAs
// an SM (7,133,222 complex64 rows: 84 us with the general update kernel, here
// 51 us = 5.6 TB/s).
template <typename T>
__global__ void __launch_bounds__(kThreads, local_ctas<T>()) update_local_k(
    const T* __restrict__ prev, const T* __restrict__ cur, int64_t n, const double2* __restrict__ coef,
    const double2* __restrict__ w, T* __restrict__ out, double* __restrict__ part, unsigned* __restrict__ ticket,
    double* __restrict__ beta_next) {
  constexpr int kRows = 2;
  __shared__ double red[kWarps];
  const double2 cp = coef[0], cc = coef[1];
  const double ws = coef[2].x;
  const int64_t step = (int64_t)gridDim.x * kThreads;
  double a[1] = {0.0};
  for (int64_t r0 = blockIdx.x * (int64_t)kThreads + threadIdx.x; r0 < n; r0 += kRows * step) {
    T p[kRows], c[kRows];
    double2 x[kRows];
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int64_t r = r0 + q * step;
      if (r < n) {
        x[q] = __ldcs(w + r);  // read once
        c[q] = cur[r];
        if (prev != nullptr) p[q] = prev[r];
      }
    }
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int64_t r = r0 + q * step;
      if (r < n) {
        const double vr = (double)c[q].x, vi = (double)c[q].y;
        double sr = fma(vr, cc.x, -vi * cc.y), si = fma(vr, cc.y, vi * cc.x);
        if (prev != nullptr) {
          const double pr = (double)p[q].x, pi = (double)p[q].y;
          sr = fma(pr, cp.x, fma(-pi, cp.y, sr));
          si = fma(pr, cp.y, fma(pi, cp.x, si));
        }
        const double yr = fma(ws, x[q].x, -sr), yi = fma(ws, x[q].y, -si);
        stc<T>(out, r, yr, yi);
        a[0] = fma(yr, yr, fma(yi, yi, a[0]));
      }
    }
  }
  block_totals<1>(a, red);
  double t;
  if (last_cta_sum(a[0], part, ticket, &t)) *beta_next = sqrt(t);
}

// Scaled coefficients c = b0 exp(-i T dt) e_1 of the Krylov vectors, T =
// tridiag(beta[1..m-1], alpha[0..m-1]), by one warp (lane L holds rows 2L and
// 2L + 1, so a product with T is two exchanges with the neighbours).
// exp(-i T dt) is applied as ceil(|dt| |T|_inf) substeps, each a Taylor
// series of kTerms terms: |tau T| <= 1, so what is left out is below 1 / 21!
// = 2e-20.  Returns |beta_m e_m^T exp(-i T dt) e_1| b0 (a posteriori error
// estimate).  One thread doing the same chain serially took 0.66 ms a step at
// m = 30 (all of its vectors in local memory); the warp takes 0.01 ms.
__device__ __forceinline__ double warp_expm(const double* alpha, const double* beta, int m, double dt, double b0,
                                            double2* c) {
  constexpr int kTerms = 20;
  const int lane = threadIdx.x & 31, i0 = 2 * lane, i1 = i0 + 1;
  const double a0 = i0 < m ? alpha[i0] : 0.0, a1 = i1 < m ? alpha[i1] : 0.0;
  const double bl = i0 > 0 && i0 < m ? beta[i0] : 0.0;  // couples i0 - 1, i0
  const double bm = i1 < m ? beta[i1] : 0.0;            // couples i0, i1
  const double br = i1 + 1 < m ? beta[i1 + 1] : 0.0;    // couples i1, i1 + 1
  double nrm = fmax(fabs(a0) + fabs(bl) + fabs(bm), fabs(a1) + fabs(bm) + fabs(br));
  bool bad = !(nrm < 1e300);  // NaN or infinite entries: fmax alone would lose them
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
  const double h = fabs(dt) * nrm;
  bad = __any_sync(0xffffffffu, bad || !(h < 1e9));  // no substep count: the result is NaN
  const int reps = bad ? 0 : (h > 1.0 ? (int)ceil(h) : 1);
  const double tau = dt / (double)(reps > 0 ? reps : 1);
  double v0r = lane == 0 ? 1.0 : 0.0, v0i = 0.0, v1r = 0.0, v1i = 0.0;
  for (int rep = 0; rep < reps; ++rep) {
    double t0r = v0r, t0i = v0i, t1r = v1r, t1i = v1i;
#pragma unroll
    for (int k = 1; k <= kTerms; ++k) {
      const double lr = __shfl_up_sync(0xffffffffu, t1r, 1), li = __shfl_up_sync(0xffffffffu, t1i, 1);
      const double rr = __shfl_down_sync(0xffffffffu, t0r, 1), ri = __shfl_down_sync(0xffffffffu, t0i, 1);
      // the end lanes keep their own value, which their zero coupling drops
      const double x0r = fma(a0, t0r, fma(bl, lr, bm * t1r)), x0i = fma(a0, t0i, fma(bl, li, bm * t1i));
      const double x1r = fma(a1, t1r, fma(bm, t0r, br * rr)), x1i = fma(a1, t1i, fma(bm, t0i, br * ri));
      const double f = tau * (1.0 / k);  // t <- (-i tau T) t / k
      t0r = f * x0i;
      t0i = -f * x0r;
      t1r = f * x1i;
      t1i = -f * x1r;
      v0r += t0r;
      v0i += t0i;
      v1r += t1r;
      v1i += t1i;
    }
  }
  if (bad) v0r = v0i = v1r = v1i = nan("");
  // the vectors are stored as beta_i v_i
  if (i0 < m) {
    const double s = beta[i0] > 0.0 ? b0 / beta[i0] : 0.0;
    c[i0] = make_double2(s * v0r, s * v0i);
  }
  if (i1 < m) {
    const double s = beta[i1] > 0.0 ? b0 / beta[i1] : 0.0;
    c[i1] = make_double2(s * v1r, s * v1i);
  }
  const double last = (m - 1) & 1 ? hypot(v1r, v1i) : hypot(v0r, v0i);
  return fabs(beta[m]) * __shfl_sync(0xffffffffu, last, (m - 1) >> 1) * b0;
}

__global__ void __launch_bounds__(32) small_expm_k(const double* __restrict__ alpha, const double* __restrict__ beta,
                                                   int m, double dt, const double* __restrict__ beta0,
                                                   double2* __restrict__ c, double* __restrict__ err) {
  const double e = warp_expm(alpha, beta, m, dt, beta0[0], c);
  if (threadIdx.x == 0) err[0] = e;
}

// psi[r] = sum_{i<m} c_i u_i[r]
template <typename T>
__global__ void combine_k(const T* __restrict__ V, int64_t n, int64_t ldv, int m, const double2* __restrict__ c,
                          T* __restrict__ psi) {
  __shared__ double2 cs[kMaxM];
  for (int t = threadIdx.x; t < m; t += blockDim.x) cs[t] = c[t];
  __syncthreads();
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    double a = 0.0, b = 0.0;
#pragma unroll 8
    for (int i = 0; i < m; ++i) {
      edg::cd v = ldc<T>(V, (int64_t)i * ldv + r);
      a = fma(v.re, cs[i].x, fma(-v.im, cs[i].y, a));
      b = fma(v.re, cs[i].y, fma(v.im, cs[i].x, b));
    }
    stc<T>(psi, r, a, b);
  }
}

// ---------------------------------------------------------------------------
// A whole time step as one cooperative launch (small sectors).  CTA b owns
// the rows [n b / G, n (b + 1) / G): their row of w, of the matrix and of the
// basis stay in its shared memory where they fit, and only the gathers of
// u_j, the dots partials and the next vector go through L2.  Per Krylov step
// two grid-wide waits: for the dots, and for the norm with the next vector.
// Bound by those waits and the dependent L2 reads between them: the partials of
// a sum are asked for together, and those of the norm while the product runs
// (12,292 rows: 0.31 ms without, 0.29 with, 0.27 on fewer CTAs).  A step of dt = 0.05 (m = 30, full reorthogonalisation,
// complex128, static-pair SU(2) chains; launches per pass before):
//   n = 182: 0.14 ms (1.48), 12,292: 0.27 ms (1.69), 101,613: 0.61 ms (1.87).
// The line (kCoopRows rows per SM) lies where the matrix and the basis no
// longer fit shared memory: at 101,613 rows the passes below take 0.96 ms, at
// 848,614 rows this form takes 6.6 ms and the passes 4.2.
// ---------------------------------------------------------------------------
constexpr int kCoopThreads = 512;
constexpr int kCoopWarps = kCoopThreads / 32;
constexpr int kCoopSmem = 200 * 1024;  // dynamic shared memory of a CTA (one per SM)
constexpr int kCoopRows = 1024;        // most rows of a CTA
constexpr int kMvLanes = 4;            // lanes per row of the product

template <typename T, typename SV>
struct CoopArgs {
  const int64_t* rowptr;
  const int32_t* cols;
  const SV* vals;
  const SV* diag;
  T* V;  // [m + 1][ldv]: written and read by this launch
  T* psi;
  double2* partial;  // [2][G][kMaxM + 1]
  double* npart;     // [2][G]
  unsigned* bar;
  int* err;
  int32_t* status;
  double* err_out;
  int64_t n, ldv;
  double dt;
  int m, reorth;
};

template <typename SV>
__device__ __forceinline__ void load_diag(const SV* __restrict__ d, int64_t r, edg::cd& o) {
  if constexpr (edg::Store<SV>::cplx)
    o = edg::cd{(double)d[r].x, (double)d[r].y};
  else
    o.re = (double)d[r];
}

template <typename T, typename SV>
__global__ void __launch_bounds__(kCoopThreads, 1) krylov_coop_k(const CoopArgs<T, SV> A) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ double2 hs[kMaxM + 1];
  __shared__ double al[kMaxM], be[kMaxM + 2];
  __shared__ double red[kCoopWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)gridDim.x, m = A.m;
  const int64_t r0 = A.n * blockIdx.x / G, r1 = A.n * (blockIdx.x + 1) / G;
  const int rows = (int)(r1 - r0);
  // shared memory: w | row offsets | matrix rows | basis rows
  double2* const w = reinterpret_cast<double2*>(sm);
  int64_t off = (int64_t)rows * 16;
  int32_t* const rp = reinterpret_cast<int32_t*>(sm + off);
  off = (off + (int64_t)(rows + 1) * 4 + 15) & ~int64_t(15);
  const int64_t e0 = A.rowptr[r0], ne = A.rowptr[r1] - e0;
  for (int r = tid; r <= rows; r += kCoopThreads) rp[r] = (int32_t)(A.rowptr[r0 + r] - e0);
  const SV* vals = A.vals + e0;
  const int32_t* cols = A.cols + e0;
  if (off + ne * (int64_t)(sizeof(SV) + 4) + 16 <= kCoopSmem) {
    SV* sv = reinterpret_cast<SV*>(sm + off);
    int32_t* sc = reinterpret_cast<int32_t*>(sv + ne);
    for (int64_t e = tid; e < ne; e += kCoopThreads) {
      sv[e] = vals[e];
      sc[e] = cols[e];
    }
    vals = sv;
    cols = sc;
    off = (off + ne * (int64_t)(sizeof(SV) + 4) + 15) & ~int64_t(15);
  }
  T* own = A.V + r0;  // this CTA's rows of the basis and their row stride
  int64_t ld = A.ldv;
  const bool basis_here = off + (int64_t)rows * (m + 1) * (int64_t)sizeof(T) <= kCoopSmem;
  if (basis_here) {
    own = reinterpret_cast<T*>(sm + off);
    ld = rows;
  }
  edg::GridSync gs{A.bar, A.err};
  // one value per thread to this CTA's partial, and a grid-wide wait
  unsigned waits = 0;  // parity of the norm partials' buffer
  auto post_sum = [&](double a) -> bool {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) red[warp] = a;
    __syncthreads();
    ++waits;
    if (tid == 0) {
      double t = 0.0;
      for (int q = 0; q < kCoopWarps; ++q) t += red[q];
      A.npart[(int64_t)(waits & 1) * G + blockIdx.x] = t;
    }
    return gs.wait();
  };
  // the partials of the last post_sum (a warp's loads, all in flight), and
  // their sum
  constexpr int kPer = (edg::kSmCount + 31) / 32;
  double np[kPer];
  auto load_sum = [&] {
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      np[k] = lane + 32 * k < G ? __ldcg(A.npart + (int64_t)(waits & 1) * G + lane + 32 * k) : 0.0;
  };
  auto take_sum = [&] {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) t += np[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  };
  auto give_up = [&] {
    if (tid == 0 && A.status != nullptr) atomicExch(A.status, EDG_ERR_TIMEOUT);
  };
  // ---- u_0 = psi / |psi| ----
  double a = 0.0;
  for (int r = tid; r < rows; r += kCoopThreads) {
    const edg::cd x = ldc<T>(A.psi, r0 + r);
    a = fma(x.re, x.re, fma(x.im, x.im, a));
  }
  if (!post_sum(a)) return give_up();
  load_sum();
  const double b0 = sqrt(take_sum()), inv0 = b0 > 0.0 ? 1.0 / b0 : 0.0;
  if (tid == 0) be[0] = b0 > 0.0 ? 1.0 : 0.0;
  for (int r = tid; r < rows; r += kCoopThreads) {
    const edg::cd x = ldc<T>(A.psi, r0 + r);
    stc<T>(A.V, r0 + r, x.re * inv0, x.im * inv0);
    if (basis_here) stc<T>(own, r, x.re * inv0, x.im * inv0);
  }
  if (!gs.wait()) return give_up();
  for (int j = 0; j < m; ++j) {
    // ---- w = H u_j on this CTA's rows; |u_j| meanwhile ----
    if (j > 0 && warp == 0) load_sum();
    {
      const T* u = A.V + (int64_t)j * A.ldv;
      const int part = tid & (kMvLanes - 1);
      const int n_it = (rows + kCoopThreads / kMvLanes - 1) / (kCoopThreads / kMvLanes);
      for (int it = 0; it < n_it; ++it) {
        const int r = it * (kCoopThreads / kMvLanes) + tid / kMvLanes;
        edg::cd acc{0.0, 0.0};
        T xr{};
        edg::cd dr{0.0, 0.0};
        if (r < rows && part == 0) {
          xr = u[r0 + r];
          load_diag(A.diag, r0 + r, dr);
        }
        if (r < rows) {
          constexpr int U = 4;  // gathers in flight per lane
          const int end = rp[r + 1];
          for (int p0 = rp[r] + part; p0 < end; p0 += U * kMvLanes) {
            T x[U];
            SV v[U];
#pragma unroll
            for (int k = 0; k < U; ++k)
              if (p0 + k * kMvLanes < end) {
                x[k] = u[cols[p0 + k * kMvLanes]];
                v[k] = vals[p0 + k * kMvLanes];
              }
#pragma unroll
            for (int k = 0; k < U; ++k)
              if (p0 + k * kMvLanes < end) {
                const edg::cd xk{(double)x[k].x, (double)x[k].y};
                if constexpr (edg::Store<SV>::cplx)
                  edg::fma_acc(acc, edg::cd{(double)v[k].x, (double)v[k].y}, xk);
                else
                  edg::fma_acc(acc, (double)v[k], xk);
              }
          }
        }
#pragma unroll
        for (int o = kMvLanes / 2; o > 0; o >>= 1) {
          acc.re += __shfl_xor_sync(0xffffffffu, acc.re, o, kMvLanes);
          acc.im += __shfl_xor_sync(0xffffffffu, acc.im, o, kMvLanes);
        }
        if (r < rows && part == 0) {
          if constexpr (edg::Store<SV>::cplx)
            edg::fma_acc(acc, dr, edg::cd{(double)xr.x, (double)xr.y});
          else
            edg::fma_acc(acc, dr.re, edg::cd{(double)xr.x, (double)xr.y});
          w[r] = make_double2(acc.re, acc.im);
        }
      }
    }
    if (j > 0 && warp == 0) {
      const double t = take_sum();
      if (lane == 0) be[j] = sqrt(t);
    }
    const int passes = A.reorth == 0 ? 1 : A.reorth;
    const int ilo = A.reorth == 0 ? (j > 0 ? j - 1 : 0) : 0;
    for (int pass = 0; pass < passes; ++pass) {
      __syncthreads();
      // ---- dots of this CTA's rows, a warp per vector ----
      double2* P = A.partial + (int64_t)pass * G * (kMaxM + 1);
      for (int i = ilo + warp; i <= j; i += kCoopWarps) {
        double gr = 0.0, gi = 0.0;
        const T* ui = own + (int64_t)i * ld;
#pragma unroll 4
        for (int r = lane; r < rows; r += 32) {
          const edg::cd x = ldc<T>(ui, r);
          const double2 y = w[r];
          gr = fma(x.re, y.x, fma(x.im, y.y, gr));
          gi = fma(x.re, y.y, fma(-x.im, y.x, gi));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          gr += __shfl_xor_sync(0xffffffffu, gr, o);
          gi += __shfl_xor_sync(0xffffffffu, gi, o);
        }
        if (lane == 0) P[(int64_t)blockIdx.x * (kMaxM + 1) + i] = make_double2(gr, gi);
      }
      if (!gs.wait()) return give_up();
      // the product was not divided by beta_j: the first pass does
      const double ws = pass > 0 ? 1.0 : (be[j] > 0.0 ? 1.0 / be[j] : 0.0);
      for (int i0 = ilo + warp; i0 <= j; i0 += 2 * kCoopWarps) {
        double2 p[2][kPer];  // two vectors' partials in flight
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int k = 0; k < kPer; ++k)
            p[h][k] = i0 + h * kCoopWarps <= j && lane + 32 * k < G
                          ? __ldcg(P + (int64_t)(lane + 32 * k) * (kMaxM + 1) + i0 + h * kCoopWarps)
                          : make_double2(0.0, 0.0);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double gr = 0.0, gi = 0.0;
#pragma unroll
          for (int k = 0; k < kPer; ++k) {
            gr += p[h][k].x;
            gi += p[h][k].y;
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            gr += __shfl_xor_sync(0xffffffffu, gr, o);
            gi += __shfl_xor_sync(0xffffffffu, gi, o);
          }
          const int i = i0 + h * kCoopWarps;
          if (lane == 0 && i <= j) {
            const double si = be[i] > 0.0 ? 1.0 / be[i] : 0.0;
            gr *= ws, gi *= ws;
            hs[i] = make_double2(si * (si * gr), si * (si * gi));
            if (i == j) al[j] = pass > 0 ? al[j] + si * gr : si * gr;
          }
        }
      }
      __syncthreads();
      // ---- w -= sum_i coef_i u_i; after the last pass it is u_{j+1} ----
      const bool last = pass + 1 == passes;
      double nrm = 0.0;
      for (int r = tid; r < rows; r += kCoopThreads) {
        double sr = 0.0, si = 0.0;
#pragma unroll 8
        for (int i = ilo; i <= j; ++i) {
          const edg::cd x = ldc<T>(own, (int64_t)i * ld + r);
          sr = fma(x.re, hs[i].x, fma(-x.im, hs[i].y, sr));
          si = fma(x.re, hs[i].y, fma(x.im, hs[i].x, si));
        }
        const double2 y = make_double2(fma(ws, w[r].x, -sr), fma(ws, w[r].y, -si));
        if (last) {
          stc<T>(A.V, (int64_t)(j + 1) * A.ldv + r0 + r, y.x, y.y);
          if (basis_here) stc<T>(own, (int64_t)(j + 1) * ld + r, y.x, y.y);
          nrm = fma(y.x, y.x, fma(y.y, y.y, nrm));
        } else {
          w[r] = y;
        }
      }
      if (last && !post_sum(nrm)) return give_up();
    }
  }
  // ---- psi = V c: every CTA forms the coefficients itself ----
  if (warp == 0) {
    load_sum();
    const double t = take_sum();
    if (lane == 0) be[m] = sqrt(t);
    __syncwarp();
    const double e = warp_expm(al, be, m, A.dt, b0, hs);
    if (lane == 0 && blockIdx.x == 0) A.err_out[0] = e;
  }
  __syncthreads();
  for (int r = tid; r < rows; r += kCoopThreads) {
    double x = 0.0, y = 0.0;
#pragma unroll 8
    for (int i = 0; i < m; ++i) {
      const edg::cd v = ldc<T>(own, (int64_t)i * ld + r);
      x = fma(v.re, hs[i].x, fma(-v.im, hs[i].y, x));
      y = fma(v.re, hs[i].y, fma(v.im, hs[i].x, y));
    }
    stc<T>(A.psi, r0 + r, x, y);
  }
}

struct KLayout {
  int64_t V, w, partial, normp, alpha, beta, coef, c, misc, sync, total;
  int64_t ldv;
};

inline int64_t al(int64_t x) { return (x + 255) & ~int64_t(255); }

constexpr int kDotBlocks = edg::kSmCount * 4;

KLayout klayout(const edg_krylov_problem* p) {
  KLayout L{};
  const int64_t n = p->n_rows;
  const int esz = p->vec_dtype == 2 ? 16 : 8;
  L.ldv = (n + 15) & ~int64_t(15);  // a vector starts on its own cache line
  int64_t o = 0;
  L.V = o; o = al(o + (int64_t)(p->m + 1) * L.ldv * esz);
  L.w = o; o = al(o + n * 16);
  L.partial = o; o = al(o + (int64_t)kDotBlocks * (kMaxM + 1) * 16);
  L.normp = o; o = al(o + (int64_t)edg::kSmCount * 8 * 8);
  L.alpha = o; o = al(o + (kMaxM + 1) * 8);
  L.beta = o; o = al(o + (kMaxM + 2) * 8);
  L.coef = o; o = al(o + (kMaxM + 2) * 16);
  L.c = o; o = al(o + (kMaxM + 1) * 16);
  L.misc = o; o = al(o + 8 * 8);  // [0] beta0, [1] err
  L.sync = o; o = al(o + 8 * 4);  // tickets (2) | error word | - | grid barrier
  L.total = o;
  return L;
}

// Whether a step may run as krylov_coop_k: few enough rows and entries, the CSR
// arrays at hand, which that kernel reads whatever layout is passed beside them
// (a problem may come with its packed layout alone), and a way to report a
// grid-wide wait that ran out (the problem's status word, or a result the call
// waits for).  The lines on the entries lie where columns are random, the worst
// case for its gathers (m = 30, passes / one launch): complex128 100,000 rows
// 0.763 / 0.743 ms at 2.0M entries and 0.887 / 1.264 at 3.0M, complex64 60,000
// rows 0.982 / 0.903 at 3.0M and 1.063 / 1.404 at 4.0M; on a few CTAs (complex
// matrix, 1,000 rows) 0.744 / 0.654 at 27,000 a CTA and 0.819 / 0.945 at 49,000.
// With neighbouring columns the one launch still gains there (150,000 rows, 3.0M
// entries: 1.13 times) and loses past 4M.
bool one_launch(const edg_krylov_problem* p, bool reports) {
  const bool csr = p->cols != nullptr && p->vals != nullptr, diagonal = p->nnz == 0 && p->pk_words == nullptr;
  return reports && p->n_rows <= kCoopMaxRows && (csr || diagonal) &&
         edg::coop_entries(p->nnz, p->n_rows, p->vec_dtype == 2 ? 2000000 : 3000000, 27000);
}

template <typename T, typename SV>
int run_step(const edg_krylov_problem* p, T* psi, double dt, char* ws, double* err_out, cudaStream_t s) {
  const KLayout L = klayout(p);
  const int64_t n = p->n_rows, ldv = L.ldv;
  const int m = p->m;
  T* V = (T*)(ws + L.V);
  double2* w = (double2*)(ws + L.w);
  double2* partial = (double2*)(ws + L.partial);
  double* normp = (double*)(ws + L.normp);
  double* alpha = (double*)(ws + L.alpha);
  double* beta = (double*)(ws + L.beta);
  double2* coef = (double2*)(ws + L.coef);
  double2* c = (double2*)(ws + L.c);
  double* misc = (double*)(ws + L.misc);
  unsigned* tickets = (unsigned*)(ws + L.sync);
  int* err_word = (int*)(tickets + 2);
  unsigned* bar = tickets + 4;  // grid barrier of the cooperative form
  cudaError_t e = cudaMemsetAsync(tickets, 0, 8 * sizeof(int), s);
  if (e != cudaSuccess) return edg::cuda_status(e, "krylov");
  bool done = false;
  if (one_launch(p, p->status != nullptr || err_out != nullptr)) {
    int dev = 0, n_sm = 0, coop = 0, occ = 0;
    auto kern = krylov_coop_k<T, SV>;
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (e == cudaSuccess) e = edg::allow_smem(kern, kCoopSmem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kCoopThreads, kCoopSmem);
    if (e != cudaSuccess) return edg::cuda_status(e, "edg_krylov_step: set-up");
    const int64_t g = edg::coop_ctas(n, n_sm);
    if (coop && occ >= 1 && (n + g - 1) / g <= kCoopRows) {
      CoopArgs<T, SV> a{p->rowptr, p->cols, (const SV*)p->vals, (const SV*)p->diag, V, psi, partial, normp, bar,
                        err_word, p->status, misc + 1, n, ldv, dt, m, p->reorth_passes};
      void* args[] = {&a};
      e = cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)g), dim3(kCoopThreads), args, kCoopSmem, s);
      if (e != cudaSuccess) return edg::cuda_status(e, "edg_krylov_step: cooperative launch");
      done = true;
    }
  }
  if (!done) {
    const unsigned gn = edg::grid_for(n, kThreads);
    const unsigned gu = edg::grid_for(n, kThreads, kUpdateCtas);
    const int nb = (int)edg::grid_for(n, kThreads, dot_ctas<T>());
    const unsigned gv = edg::grid_for(n, 256);
    norm_k<T><<<gn, kThreads, 0, s>>>(psi, n, normp, tickets, misc);  // beta0
    scale_k<T><<<gv, 256, 0, s>>>(psi, n, misc, V, beta);
    for (int j = 0; j < m; ++j) {
      const T* vj = V + (int64_t)j * ldv;
      // reorth_passes = 0: local recurrence (against v_{j-1}, v_j only);
      // 1 or 2: classical Gram-Schmidt over the whole basis, once or twice
      const int passes = p->reorth_passes == 0 ? 1 : p->reorth_passes;
      const int ilo = p->reorth_passes == 0 ? (j > 0 ? j - 1 : 0) : 0;
      int st;
      bool dots_done = false;
      if constexpr (std::is_same<SV, double>::value || std::is_same<SV, float>::value) {
        if (p->pk_words != nullptr && p->reorth_passes == 0) {
          // the coefficients come out of the product
          const edg::KrylovStep step{j > 0 ? (const void*)(vj - ldv) : nullptr, (double*)partial, tickets, beta,
                                     alpha, coef, j};
          st = edg::launch_packed_krylov<SV>(n, p->pk_tile_off, p->pk_words, (const SV*)p->pk_table, p->pk_count,
                                             p->pk_colbits, (const SV*)p->diag, (const SV*)vj, (double*)w, step,
                                             p->status, s);
          dots_done = true;
        } else if (p->pk_words != nullptr) {  // (re, im) as two interleaved right-hand sides
          st = edg::launch_packed_spmv<SV>(2, 2, n, p->pk_tile_off, p->pk_words, (const SV*)p->pk_table, p->pk_count,
                                           p->pk_colbits, (const SV*)p->diag, (const SV*)vj, (double*)w, 0, nullptr,
                                           p->status, s, 1);
        } else {
          st = edg::launch_spmv<SV, T, double2>(1, n, p->nnz, p->rowptr, p->cols, (const SV*)p->vals,
                                                (const SV*)p->diag, vj, w, s, 0, p->spmv_group);
        }
      } else {
        st = edg::launch_spmv<SV, T, double2>(1, n, p->nnz, p->rowptr, p->cols, (const SV*)p->vals,
                                              (const SV*)p->diag, vj, w, s, 0, p->spmv_group);
      }
      if (st) return st;
      if (dots_done) {
        update_local_k<T><<<edg::grid_for(n, kThreads, local_ctas<T>()), kThreads, 0, s>>>(
            j > 0 ? vj - ldv : nullptr, vj, n, coef, w, V + (int64_t)(j + 1) * ldv, normp, tickets + 1, beta + j + 1);
        if ((e = cudaGetLastError()) != cudaSuccess) return edg::cuda_status(e, "edg_krylov_step: lanczos");
        continue;
      }
      for (int pass = 0; pass < passes; ++pass) {
        const bool last = pass + 1 == passes;
        dots_k<T><<<nb, kThreads, 0, s>>>(V, n, ldv, ilo, j, w, partial, kMaxM + 1);
        coef_k<<<j + 1 - ilo, kThreads, 0, s>>>(partial, nb, kMaxM + 1, ilo, j, pass, beta, coef, alpha);
        update_k<T><<<gu, kThreads, (j + 2 - ilo) * sizeof(double2), s>>>(V, n, ldv, ilo, j, coef, w,
                                            last ? V + (int64_t)(j + 1) * ldv : nullptr, normp, tickets + 1, beta);
      }
      if ((e = cudaGetLastError()) != cudaSuccess) return edg::cuda_status(e, "edg_krylov_step: lanczos");
    }
    small_expm_k<<<1, 32, 0, s>>>(alpha, beta, m, dt, misc, c, misc + 1);
    combine_k<T><<<gv, 256, 0, s>>>(V, n, ldv, m, c, psi);
    if ((e = cudaGetLastError()) != cudaSuccess) return edg::cuda_status(e, "edg_krylov_step: combine");
  }
  if (err_out) {
    int waits = 0;
    e = cudaMemcpyAsync(err_out, misc + 1, sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&waits, err_word, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return edg::cuda_status(e, "edg_krylov_step: error estimate");
    if (waits != 0) {
      *err_out = nan("");
      edg::set_error("edg_krylov_step: a grid-wide wait ran out");
      return EDG_ERR_TIMEOUT;
    }
  }
  return EDG_OK;
}

int check_k(const edg_krylov_problem* p) {
  EDG_REQUIRE(p != nullptr, "edg_krylov: null problem");
  EDG_REQUIRE(p->vec_dtype == 2 || p->vec_dtype == 3, "edg_krylov: vec_dtype must be 2 (c128) or 3 (c64)");
  EDG_REQUIRE(p->mat_dtype >= 0 && p->mat_dtype <= 3, "edg_krylov: bad mat_dtype");
  EDG_REQUIRE((p->mat_dtype == 0 || p->mat_dtype == 2) == (p->vec_dtype == 2),
              "edg_krylov: matrix and vectors must share the precision (f64/c128 or f32/c64)");
  EDG_REQUIRE(p->m >= 1 && p->m <= kMaxM, "edg_krylov: m must be 1..%d", kMaxM);
  EDG_REQUIRE(p->reorth_passes >= 0 && p->reorth_passes <= 2, "edg_krylov: reorth_passes must be 0..2");
  EDG_REQUIRE(p->n_rows > 0 && p->rowptr && p->diag, "edg_krylov: empty matrix");
  EDG_REQUIRE(p->pk_words == nullptr ||
                  ((p->mat_dtype == 0 || p->mat_dtype == 1) && p->pk_tile_off && p->pk_table && p->pk_count >= 1 &&
                   p->pk_count <= EDG_PACK_MAX_VALUES && p->pk_colbits >= 1 && p->pk_colbits <= 31 &&
                   p->n_rows < ((int64_t)1 << p->pk_colbits)),
              "edg_krylov: a packed layout needs a real matrix (mat_dtype 0 or 1) and a complete layout");
  EDG_REQUIRE(p->nnz == 0 || (p->cols && p->vals) || p->pk_words,
              "edg_krylov: off-diagonal entries without CSR arrays or a packed layout");
  return EDG_OK;
}

}  // namespace

// One Lanczos step for a caller that applies its own product (the projected
// matvec of a momentum sector): the same three kernels a pass as the steps
// above, with everything the host would read kept on the device.  What bounds
// a short step is the host: 12,329 momentum states (147,578 sector rows), 55
// steps with library products and two reads a step took 12.9 ms, here 4.2, of
// which the nine kernels a step take 2.6.
extern "C" int64_t edg_krylov_orth_bytes(int32_t max_vectors) {
  if (max_vectors < 1 || max_vectors > kMaxOrth) return -1;
  return al((int64_t)edg::kSmCount * 2 * (max_vectors + 1) * 16) + al((int64_t)edg::kSmCount * 8 * 8) +
         al((int64_t)(max_vectors + 2) * 16) + 256;
}

extern "C" int edg_krylov_orth(int64_t n, int64_t ldv, double* V, int32_t j, double* w, int32_t passes, double* alpha,
                               double* beta, int32_t max_vectors, void* work, int64_t work_bytes,
                               cudaStream_t stream) {
  EDG_REQUIRE(n > 0 && ldv >= n && V && w && alpha && beta && work, "edg_krylov_orth: null argument or bad size");
  EDG_REQUIRE(max_vectors >= 1 && max_vectors <= kMaxOrth && j >= 0 && j < max_vectors,
              "edg_krylov_orth: j must lie in [0, max_vectors), max_vectors in [1, %d]", kMaxOrth);
  EDG_REQUIRE(passes == 1 || passes == 2, "edg_krylov_orth: passes must be 1 or 2");
  EDG_REQUIRE(work_bytes >= edg_krylov_orth_bytes(max_vectors), "edg_krylov_orth: workspace too small");
  EDG_REQUIRE(((reinterpret_cast<uintptr_t>(V) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(work)) &
               15) == 0,
              "edg_krylov_orth: pointers must be 16-byte aligned");
  char* ws = (char*)work;
  const int ld_i = max_vectors + 1;
  double2* partial = (double2*)ws;
  ws += al((int64_t)edg::kSmCount * 2 * ld_i * 16);
  double* normp = (double*)ws;
  ws += al((int64_t)edg::kSmCount * 8 * 8);
  double2* coef = (double2*)ws;
  ws += al((int64_t)(max_vectors + 2) * 16);
  unsigned* ticket = (unsigned*)ws;
  const double2* basis = (const double2*)V;
  const int nb = (int)edg::grid_for(n, kThreads, dot_ctas<double2>());
  // few rows: tiles of vectors side by side, up to two CTAs an SM (12,329 rows,
  // 49 CTAs a tile: 7.3 us a pass one after the other, here 3.7)
  const int tiles = j / kTile + 1, room = 2 * edg::kSmCount / nb;
  const unsigned ny = (unsigned)(room < 1 ? 1 : (room < tiles ? room : tiles));
  const unsigned gu = edg::grid_for(n, kThreads, kUpdateCtas);
  if (j == 0) {
    cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof(unsigned), stream);
    if (e != cudaSuccess) return edg::cuda_status(e, "edg_krylov_orth");
  }
  if ((j + 2) * sizeof(double2) > 40 * 1024) {  // above the limit a kernel has without asking
    cudaError_t e = edg::allow_smem(update_k<double2>, (kMaxOrth + 1) * sizeof(double2));
    if (e != cudaSuccess) return edg::cuda_status(e, "edg_krylov_orth");
  }
  for (int pass = 0; pass < passes; ++pass) {
    dots_k<double2><<<dim3(nb, ny), kThreads, 0, stream>>>(basis, n, ldv, 0, j, (const double2*)w, partial, ld_i);
    coef_k<<<j + 1, kThreads, 0, stream>>>(partial, nb, ld_i, 0, j, pass, beta, coef, alpha);
    update_k<double2><<<gu, kThreads, (j + 2) * sizeof(double2), stream>>>(
        basis, n, ldv, 0, j, coef, (double2*)w, pass + 1 == passes ? (double2*)V + (int64_t)(j + 1) * ldv : nullptr,
        normp, ticket, beta);
  }
  EDG_CHECK_LAUNCH("edg_krylov_orth");
  return EDG_OK;
}

extern "C" int64_t edg_krylov_workspace_bytes(const edg_krylov_problem* p) {
  if (check_k(p)) return -1;
  return klayout(p).total;
}

extern "C" int edg_krylov_one_launch(const edg_krylov_problem* p) {
  if (check_k(p)) return -1;
  return one_launch(p, p->status != nullptr) ? 1 : 0;
}

extern "C" int edg_krylov_step(const edg_krylov_problem* p, void* psi, double dt, void* workspace,
                               int64_t workspace_bytes, double* err_out, cudaStream_t stream) {
  int st = check_k(p);
  if (st) return st;
  EDG_REQUIRE(psi != nullptr && workspace != nullptr && workspace_bytes >= klayout(p).total,
              "edg_krylov_step: workspace too small");
  const bool c128 = p->vec_dtype == 2;
  (void)c128;
  switch (p->mat_dtype) {
    case 0: return run_step<double2, double>(p, (double2*)psi, dt, (char*)workspace, err_out, stream);
    case 2: return run_step<double2, double2>(p, (double2*)psi, dt, (char*)workspace, err_out, stream);
    case 1: return run_step<float2, float>(p, (float2*)psi, dt, (char*)workspace, err_out, stream);
    default: return run_step<float2, float2>(p, (float2*)psi, dt, (char*)workspace, err_out, stream);
  }
}
