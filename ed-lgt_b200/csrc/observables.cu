// Diagonal (local) observables: out[s] += sum_r |psi_r|^2 * diag[s][c_s(r)] for
// every site s at once.  This is LocalTerm.get_expval in a symmetry sector
// (edlgt/modeling/local_term.py:119-237 with exp_val_data,
// edlgt/modeling/qmb_state.py:631-654): local terms only keep the operator
// diagonal, so an expectation value is a weighted reduction over the basis.
//
// One thread takes rows grid-stride, decodes each key (digits.cuh) and adds
// |psi_r|^2 diag[s][c] to one f64 register per site, the diagonals in shared
// memory (lanes read a few neighbouring entries: no bank conflicts).  Bound by
// the instructions per digit: SU(2) L = 16 (7,133,222 rows, 16 sites,
// complex128) 0.144 ms; with 64-bit divisions and sums in local memory 0.333.
#include "digits.cuh"

namespace {

constexpr int kThreads = 256;

template <int PT>
__device__ __forceinline__ double prob(const void* psi, int64_t r, int64_t stride) {
  if (PT == 0) {
    double a = ((const double*)psi)[r * stride];
    return a * a;
  } else if (PT == 1) {
    double a = ((const float*)psi)[r * stride];
    return a * a;
  } else if (PT == 2) {
    double2 a = ((const double2*)psi)[r * stride];
    return a.x * a.x + a.y * a.y;
  } else {
    float2 a = ((const float2*)psi)[r * stride];
    return (double)a.x * a.x + (double)a.y * a.y;
  }
}

constexpr int kTableCap = 40 * 1024;  // diagonals larger than this stay in global memory

// CTAs whose accumulators fit an SM's registers (one wave of them is launched)
constexpr int ctas_for(int ns) { return ns <= 16 ? 3 : ns <= 32 ? 2 : 1; }

// NS >= n_sites sites accumulated in registers.
template <int PT, int NS, typename K>
__global__ void __launch_bounds__(kThreads, ctas_for(NS)) local_expval_k(const __grid_constant__ edg::DigitPlan P,
                                                           const uint64_t* __restrict__ keys, int64_t n,
                                                           const void* __restrict__ psi, int64_t psi_stride,
                                                           const double* __restrict__ diag, int dmax, int in_smem,
                                                           double* __restrict__ out) {
  extern __shared__ __align__(16) double tab[];  // [n_sites][dmax]
  __shared__ double acc[EDG_MAX_SITES];
  const int ns = P.n_sites;
  for (int s = threadIdx.x; s < ns; s += kThreads) acc[s] = 0.0;
  if (in_smem)
    for (int k = threadIdx.x; k < ns * dmax; k += kThreads) tab[k] = diag[k];
  __syncthreads();
  const double* const d = in_smem ? tab : diag;
  double loc[NS];
#pragma unroll
  for (int p = 0; p < NS; ++p) loc[p] = 0.0;
  for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < n; r += (int64_t)gridDim.x * kThreads) {
    const double p2 = prob<PT>(psi, r, psi_stride);
    edg::for_each_digit<NS>(P, edg::ld_key<K>(keys, r),
                            [&](int p, int c) { loc[p] = fma(p2, d[(ns - 1 - p) * dmax + c], loc[p]); });
  }
#pragma unroll
  for (int p = 0; p < NS; ++p) {
    double v = loc[p];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (p < ns && (threadIdx.x & 31) == 0) atomicAdd(&acc[ns - 1 - p], v);
  }
  __syncthreads();
  for (int s = threadIdx.x; s < ns; s += kThreads) atomicAdd(out + s, acc[s]);
}

template <int PT, int NS, typename K>
void launch(const edg::DigitPlan& P, const uint64_t* keys, int64_t n, const void* psi, int64_t stride,
            const double* diag, int dmax, double* out, cudaStream_t s) {
  const size_t table = sizeof(double) * (size_t)P.n_sites * dmax;
  const int in_smem = table <= (size_t)kTableCap;
  const unsigned g = edg::grid_for(n, kThreads, ctas_for(NS));
  local_expval_k<PT, NS, K><<<g, kThreads, in_smem ? table : 0, s>>>(P, keys, n, psi, stride, diag, dmax, in_smem,
                                                                     out);
}

template <int NS, typename K>
void launch_pt(int pt, const edg::DigitPlan& P, const uint64_t* keys, int64_t n, const void* psi, int64_t stride,
               const double* diag, int dmax, double* out, cudaStream_t s) {
  switch (pt) {
    case 0: launch<0, NS, K>(P, keys, n, psi, stride, diag, dmax, out, s); break;
    case 1: launch<1, NS, K>(P, keys, n, psi, stride, diag, dmax, out, s); break;
    case 2: launch<2, NS, K>(P, keys, n, psi, stride, diag, dmax, out, s); break;
    default: launch<3, NS, K>(P, keys, n, psi, stride, diag, dmax, out, s); break;
  }
}

template <int W>
int local_expval(const uint64_t* keys, int64_t n, int32_t n_hi, const edg_site_dims* dims, int32_t n_sites,
                 const void* psi, int32_t psi_dtype, int64_t psi_stride, const double* diag, int32_t dmax, double* out,
                 cudaStream_t stream) {
  EDG_REQUIRE(dims != nullptr && n >= 0 && n_sites > 0 && n_sites <= EDG_MAX_SITES && dmax > 0 && psi_stride >= 1,
              "edg_local_expval: bad arguments");
  EDG_REQUIRE(W == 1 || (n_hi > 0 && n_hi < n_sites), "edg_local_expval_wide: n_hi out of range");
  EDG_REQUIRE(psi_dtype >= 0 && psi_dtype <= 3, "edg_local_expval: psi_dtype must be 0..3");
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double) * n_sites, stream);
  if (e != cudaSuccess) return edg::cuda_status(e, "edg_local_expval: reset");
  if (n == 0) return EDG_OK;
  EDG_REQUIRE(W == 1 || (reinterpret_cast<uintptr_t>(keys) & 15) == 0,
              "edg_local_expval_wide: two-word keys must be 16-byte aligned");
  edg::DigitPlan P;
  EDG_REQUIRE(edg::make_digit_plan(&P, dims->d, n_sites, W, n_hi), "edg_local_expval: bad local dimensions");
  using K = typename edg::KeyOf<W>::type;
  if (n_sites <= 16)
    launch_pt<16, K>(psi_dtype, P, keys, n, psi, psi_stride, diag, dmax, out, stream);
  else if (n_sites <= 32)
    launch_pt<32, K>(psi_dtype, P, keys, n, psi, psi_stride, diag, dmax, out, stream);
  else
    launch_pt<EDG_MAX_SITES, K>(psi_dtype, P, keys, n, psi, psi_stride, diag, dmax, out, stream);
  EDG_CHECK_LAUNCH("edg_local_expval");
  return EDG_OK;
}

}  // namespace

extern "C" int edg_local_expval(const uint64_t* keys, int64_t n, const edg_site_dims* dims, int32_t n_sites,
                                const void* psi, int32_t psi_dtype, int64_t psi_stride, const double* diag,
                                int32_t dmax, double* out, cudaStream_t stream) {
  return local_expval<1>(keys, n, 0, dims, n_sites, psi, psi_dtype, psi_stride, diag, dmax, out, stream);
}

extern "C" int edg_local_expval_wide(const uint64_t* keys, int64_t n, int32_t n_hi, const edg_site_dims* dims,
                                     int32_t n_sites, const void* psi, int32_t psi_dtype, int64_t psi_stride,
                                     const double* diag, int32_t dmax, double* out, cudaStream_t stream) {
  return local_expval<2>(keys, n, n_hi, dims, n_sites, psi, psi_dtype, psi_stride, diag, dmax, out, stream);
}
