// Gauge phases of the real form: the assembled matrix is D^dagger H D with
// D = diag(i^e(r)), e(r) = sum_s w[s][c_s(r)] (edgpu/modeling/assembly.py), so
// a vector moves between the two bases by one phase per row.
//
// One thread per row decodes its key (digits.cuh) and sums the exponents from
// a shared-memory table; the phase itself is a swap and a sign, exact.  Moves 8
// (key) + s_psi bytes in and 16 out a row, and is bound by the instructions of
// the decode: on the 7,133,222-state sector of the L = 16 static pair 122 us for
// a float32 vector (200 MB) and 129 us for a complex128 one (285 MB), a third of
// the copy rate at most.  It replaces a decode of the whole configuration table
// to the host, its upload as int64 and a gather per site: 235 ms a call with the
// table already decoded.
#include "digits.cuh"

namespace {

constexpr int kThreads = 256;

template <int PT>
__device__ __forceinline__ double2 load(const void* psi, int64_t i) {
  if (PT == 0) return make_double2(((const double*)psi)[i], 0.0);
  if (PT == 1) return make_double2((double)((const float*)psi)[i], 0.0);
  if (PT == 2) return ((const double2*)psi)[i];
  if (PT == 3) {
    const float2 a = ((const float2*)psi)[i];
    return make_double2((double)a.x, (double)a.y);
  }
  return make_double2(1.0, 0.0);
}

// out[r] = i^{e(r)} psi[r] (sign = 1) or i^{-e(r)} psi[r] (sign = 3, modulo
// 4); PT = 4: the phase itself.
template <int PT, int NS, typename K>
__global__ void __launch_bounds__(kThreads) gauge_k(const __grid_constant__ edg::DigitPlan P,
                                                    const uint64_t* __restrict__ keys, int64_t n,
                                                    const uint8_t* __restrict__ weights, int dmax, int sign,
                                                    const void* __restrict__ psi, int64_t stride,
                                                    double2* __restrict__ out) {
  extern __shared__ uint8_t tab[];  // [n_sites][dmax], position order
  for (int k = threadIdx.x; k < P.n_sites * dmax; k += kThreads) {
    const int p = k / dmax;
    tab[k] = weights[(P.n_sites - 1 - p) * dmax + (k - p * dmax)];
  }
  __syncthreads();
  for (int64_t r = blockIdx.x * (int64_t)kThreads + threadIdx.x; r < n; r += (int64_t)gridDim.x * kThreads) {
    const double2 a = load<PT>(psi, r * stride);
    int e = 0;
    edg::for_each_digit<NS>(P, edg::ld_key<K>(keys, r), [&](int p, int c) { e += c < dmax ? tab[p * dmax + c] : 0; });
    e = (e * sign) & 3;
    const double re = (e & 1) ? a.y : a.x, im = (e & 1) ? a.x : a.y;
    out[r] = make_double2((e == 1 || e == 2) ? -re : re, e >= 2 ? -im : im);
  }
}

template <int NS, typename K>
void launch(int pt, unsigned grid, size_t smem, cudaStream_t s, const edg::DigitPlan& P, const uint64_t* keys,
            int64_t n, const uint8_t* w, int dmax, int sign, const void* psi, int64_t stride, double2* out) {
  switch (pt) {
    case 0: gauge_k<0, NS, K><<<grid, kThreads, smem, s>>>(P, keys, n, w, dmax, sign, psi, stride, out); break;
    case 1: gauge_k<1, NS, K><<<grid, kThreads, smem, s>>>(P, keys, n, w, dmax, sign, psi, stride, out); break;
    case 2: gauge_k<2, NS, K><<<grid, kThreads, smem, s>>>(P, keys, n, w, dmax, sign, psi, stride, out); break;
    case 3: gauge_k<3, NS, K><<<grid, kThreads, smem, s>>>(P, keys, n, w, dmax, sign, psi, stride, out); break;
    default: gauge_k<4, NS, K><<<grid, kThreads, smem, s>>>(P, keys, n, w, dmax, sign, psi, stride, out); break;
  }
}

}  // namespace

extern "C" int edg_gauge_apply(const uint64_t* keys, int64_t n, int32_t key_words, int32_t n_hi,
                               const edg_site_dims* dims, int32_t n_sites, const uint8_t* weights, int32_t dmax,
                               int32_t conj, const void* psi, int32_t psi_dtype, int64_t psi_stride, void* out,
                               cudaStream_t stream) {
  EDG_REQUIRE(dims != nullptr && n >= 0 && n_sites > 0 && n_sites <= EDG_MAX_SITES && dmax > 0 && dmax <= 256 &&
                  psi_stride >= 1,
              "edg_gauge_apply: bad sizes");
  EDG_REQUIRE(key_words <= 1 || (key_words == 2 && n_hi > 0 && n_hi < n_sites &&
                                 (reinterpret_cast<uintptr_t>(keys) & 15) == 0),
              "edg_gauge_apply: two-word keys need 0 < n_hi < n_sites and 16-byte aligned keys");
  EDG_REQUIRE(psi_dtype >= 0 && psi_dtype <= 3, "edg_gauge_apply: psi_dtype must be 0..3");
  if (n == 0) return EDG_OK;
  EDG_REQUIRE(keys != nullptr && weights != nullptr && out != nullptr && (reinterpret_cast<uintptr_t>(out) & 15) == 0,
              "edg_gauge_apply: null argument, or an output that is not 16-byte aligned");
  edg::DigitPlan P;
  EDG_REQUIRE(edg::make_digit_plan(&P, dims->d, n_sites, key_words, n_hi), "edg_gauge_apply: bad local dimensions");
  const unsigned grid = edg::grid_for(n, kThreads);
  const size_t smem = (size_t)n_sites * dmax;  // at most 64 x 256 bytes
  const int pt = psi == nullptr ? 4 : psi_dtype;
  const int sign = conj ? 3 : 1;
  double2* o = (double2*)out;
  if (key_words == 2)
    launch<EDG_MAX_SITES, edg::u128>(pt, grid, smem, stream, P, keys, n, weights, dmax, sign, psi, psi_stride, o);
  else if (n_sites <= 16)
    launch<16, uint64_t>(pt, grid, smem, stream, P, keys, n, weights, dmax, sign, psi, psi_stride, o);
  else
    launch<EDG_MAX_SITES, uint64_t>(pt, grid, smem, stream, P, keys, n, weights, dmax, sign, psi, psi_stride, o);
  EDG_CHECK_LAUNCH("edg_gauge_apply");
  return EDG_OK;
}
