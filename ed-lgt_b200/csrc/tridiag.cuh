// Device tridiagonal eigen-solve shared by the Lanczos drivers: the k lowest
// eigenpairs of T = tridiag(b[1..m-1], a[0..m-1], b[1..m-1]) computed by the
// calling CTA (NT = blockDim.x threads): multisection on Sturm counts
// (NT points per round) for the eigenvalues, then inverse iteration
// with a pivoted tridiagonal LU (thread 0) for the eigenvectors.
//
// The whole solve is a serial chain, so what it costs is the latency of a
// step.  The Sturm counts run on the leading minors p_i = (a_i - x) p_{i-1} -
// b_i^2 p_{i-2} of T scaled by a power of two (exact) below norm 1: one
// multiply-add per row on the chain, where the quotients p_i / p_{i-1} need a
// division; both are rescaled by powers of two every fourth row.  The factors
// and vectors stay in shared memory up to kTriSmem rows, the pivots are kept
// as reciprocals.  With quotients, factors in global memory and a serial search
// of the counts the checks of a solve (two pairs, 53 rows at its end) took
// 0.63 ms, now 0.37; those of a three-problem sweep 0.46 and 0.30.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace edg {

constexpr int kTriThreads = 256;
constexpr int kTriSmem = 256;  // rows kept in shared memory

// Eigenvalues of the scaled T below x: sign changes of the leading minors.
__device__ inline int sturm_count(const double* d, const double* e2, int m, double x) {
  constexpr double kBig = 0x1p300, kSmall = 0x1p-300;
  double p0 = 1.0, p1 = d[0] - x;
  if (p1 == 0.0) p1 = -kSmall;
  int cnt = p1 < 0.0;
  for (int i0 = 1; i0 < m; i0 += 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + q;
      if (i < m) {
        double p2 = fma(d[i] - x, p1, -(e2[i] * p0));
        if (p2 == 0.0) p2 = -p1 * kSmall;  // counted as a pivot just below zero
        cnt += (p2 < 0.0) != (p1 < 0.0);
        p0 = p1;
        p1 = p2;
      }
    }
    // |d - x| <= 2 and e2 <= 1: four rows grow by less than 3^4
    const double big = fmax(fabs(p0), fabs(p1));
    const double f = big < kSmall ? kBig : big > kBig ? kSmall : 1.0;
    p0 *= f;
    p1 *= f;
  }
  return cnt;
}

// What a convergence check needs of the coefficients al[0..m-1], be[1..m]
// (be[0] couples nothing and is not read: callers need not set it): the
// dimension mv at which the recurrence ends (the first i >= 1 with |be[i]| <=
// 1e-12 max(|al| + |be|), else m) and whether it ends there.  For the calling
// CTA (NT threads); every thread gets both.
template <int NT = kTriThreads>
__device__ inline int ritz_dimension(const double* al, const double* be, int m, bool* ends) {
  __shared__ double mx[NT / 32];
  __shared__ int first_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double scale = 0.0;
  for (int i = tid; i < m; i += NT) scale = fmax(scale, fabs(al[i]) + (i > 0 ? fabs(be[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) scale = fmax(scale, __shfl_xor_sync(0xffffffffu, scale, o));
  if (lane == 0) mx[warp] = scale;
  if (tid == 0) first_s = m + 1;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) scale = fmax(scale, mx[w]);
  const double thr = 1e-12 * fmax(scale, 1e-300);
  for (int i = 1 + tid; i <= m; i += NT)
    if (fabs(be[i]) <= thr) atomicMin(&first_s, i);
  __syncthreads();
  const int first = first_s;
  __syncthreads();
  *ends = first <= m;
  return first <= m ? first : m;
}

// k lowest eigenpairs of the tridiagonal (a[0..m-1], bb[1..m-1]) for the
// calling CTA.  evals_out[q] (q < k), evecs_out[q * ldv + i] (i < m, may be
// null), wk: 6*m doubles of scratch (used beyond kTriSmem rows).
template <int NT = kTriThreads>
__device__ inline void tridiag_body(const double* a, const double* bb, int m, int k, double* evals_out,
                                    double* evecs_out, int ldv, double* wk) {
  __shared__ double sh[7][kTriSmem];
  __shared__ int piv_sh[kTriSmem];
  __shared__ double ext[2][NT / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool small = m <= kTriSmem;
  // scaled diagonal and squared off-diagonal, later the factors l and u2
  double* const x1 = small ? sh[0] : wk;
  double* const x2 = small ? sh[1] : wk + m;
  const double* A = a;
  const double* B = bb;
  // Gershgorin interval
  double gl = 1e300, gu = -1e300;
  for (int i = tid; i < m; i += NT) {
    const double ai = a[i], bi = i > 0 ? bb[i] : 0.0, bn = i + 1 < m ? bb[i + 1] : 0.0;
    const double off = fabs(bi) + fabs(bn);
    gl = fmin(gl, ai - off);
    gu = fmax(gu, ai + off);
    if (small) {
      sh[2][i] = ai;
      sh[3][i] = bi;
    }
  }
  if (small) {
    A = sh[2];
    B = sh[3];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, o));
    gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, o));
  }
  if (lane == 0) {
    ext[0][warp] = gl;
    ext[1][warp] = gu;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    gl = fmin(gl, ext[0][w]);
    gu = fmax(gu, ext[1][w]);
  }
  const double span = fmax(fabs(gl), fabs(gu));
  gl = gl - 2.0 * span * 1e-15 - 1e-300;
  gu = gu + 2.0 * span * 1e-15 + 1e-300;
  // power of two that brings the norm into [1/4, 1/2): exponent field 2044 -
  // that of span (spans outside 2^+-1000 are left alone)
  const int ef = (__double2hiint(span) >> 20) & 0x7ff;
  const double is = ef > 23 && ef < 2023 ? __hiloint2double((2044 - ef) << 20, 0) : 1.0;
  for (int i = tid; i < m; i += NT) {
    const double e = (i > 0 ? B[i] : 0.0) * is;
    x1[i] = A[i] * is;
    x2[i] = e * e;
  }
  __syncthreads();
  for (int e = 0; e < k && e < m; ++e) {
    double lo = gl, hi = gu;  // the same in every thread
    for (int round = 0; round < 12; ++round) {
      if (!(hi - lo > 2.2e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300)) break;
      // NT interior points; the first with count >= e + 1 bounds
      // eigenvalue e from above
      auto point = [&](int t) { return lo + (hi - lo) * (double)(t + 1) / (double)(NT + 1); };
      const int below = __syncthreads_count(sturm_count(x1, x2, m, point(tid) * is) < e + 1);
      const double nlo = below > 0 ? point(below - 1) : lo, nhi = below < NT ? point(below) : hi;
      lo = nlo;
      hi = nhi;
    }
    if (tid == 0) evals_out[e] = 0.5 * (lo + hi);
  }
  __syncthreads();
  // inverse iteration for eigenvectors (thread 0; m is small)
  if (tid == 0 && evecs_out != nullptr) {
    double* dl = x1;  // LU factors of T - theta, reciprocal pivots
    double* du2 = x2;
    double* rd = small ? sh[4] : wk + 2 * m;
    double* du = small ? sh[5] : wk + 3 * m;
    int* piv = small ? piv_sh : (int*)(wk + 5 * m);
    double scale = 0.0;
    for (int i = 0; i < m; ++i) scale = fmax(scale, fabs(A[i]) + (i > 0 ? fabs(B[i]) : 0.0));
    const double eps_shift = 2.2e-16 * fmax(scale, 1e-300);
    for (int e = 0; e < k && e < m; ++e) {
      const double theta = evals_out[e];
      double* const out = evecs_out + (int64_t)e * ldv;
      double* const s = small ? sh[6] : out;
      // factor (T - theta I) with partial pivoting (dgttrf); d, u: row i of
      // what is left, before its elimination step
      double d = A[0] - theta, u = m > 1 ? B[1] : 0.0;
      for (int i = 0; i < m - 1; ++i) {
        const double l = B[i + 1], dn = A[i + 1] - theta, un = i + 2 < m ? B[i + 2] : 0.0;
        if (fabs(d) >= fabs(l)) {
          if (d == 0.0) d = eps_shift;
          const double r = 1.0 / d, f = l * r;
          piv[i] = i;
          rd[i] = r;
          dl[i] = f;
          du[i] = u;
          du2[i] = 0.0;
          d = dn - f * u;
          u = un;
        } else {
          const double r = 1.0 / l, f = d * r;
          piv[i] = i + 1;
          rd[i] = r;
          dl[i] = f;
          du[i] = dn;
          du2[i] = un;
          d = u - f * dn;
          u = -f * un;
        }
      }
      if (d == 0.0) d = eps_shift;
      rd[m - 1] = 1.0 / d;
      for (int i = 0; i < m; ++i) s[i] = 1.0 / sqrt((double)m) * (1.0 + 0.01 * (double)((i * 7 + e * 3) % 5));
      for (int it = 0; it < 3; ++it) {
        // solve L U x = P s, the running entries in registers
        double cur = s[0];
        for (int i = 0; i < m - 1; ++i) {
          const double nx = s[i + 1];
          if (piv[i] == i) {
            s[i] = cur;
            cur = nx - dl[i] * cur;
          } else {
            s[i] = nx;
            cur = cur - dl[i] * nx;
          }
        }
        double y1 = cur * rd[m - 1], y2 = 0.0, nn = 0.0;
        s[m - 1] = y1;
        for (int i = m - 2; i >= 0; --i) {
          const double y = (s[i] - du[i] * y1 - du2[i] * y2) * rd[i];
          s[i] = y;
          y2 = y1;
          y1 = y;
        }
        // orthogonalise against earlier eigenvectors (near-degenerate pairs)
        for (int f = 0; f < e; ++f) {
          const double* sf = evecs_out + (int64_t)f * ldv;
          double p = 0.0;
          for (int i = 0; i < m; ++i) p += sf[i] * s[i];
          for (int i = 0; i < m; ++i) s[i] -= p * sf[i];
        }
        for (int i = 0; i < m; ++i) nn += s[i] * s[i];
        nn = 1.0 / sqrt(nn);
        for (int i = 0; i < m; ++i) s[i] *= nn;
      }
      // sign convention: largest component positive
      int imax = 0;
      for (int i = 1; i < m; ++i)
        if (fabs(s[i]) > fabs(s[imax])) imax = i;
      const double sg = s[imax] < 0.0 ? -1.0 : 1.0;
      for (int i = 0; i < m; ++i) out[i] = sg * s[i];
    }
  }
}

}  // namespace edg
