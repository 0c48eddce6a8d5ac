// Fourier modes of the constant-coefficient finite-difference operators (device code):
// their symbols and the small dense solves of the BDF preconditioners.
#pragma once
#include <cuda_runtime.h>

#include "fft_line.cuh"
#include "internal.h"

namespace rdcu {

// Symbol of operator g of the table at multi-index nidx.
__device__ __forceinline__ double2 lin_symbol(const LinTable& t, int g, const int* nidx) {
  const int nax = t.op[g].nax, a = t.op[g].ax0, b = t.op[g].ax1;
  if (nax == 0) return make_double2(1.0, 0.0);
  const double sa = t.sinv[t.off[a] + nidx[a]];
  if (nax == 1) return make_double2(0.0, sa * t.idx[a]);
  if (a == b) {
    const double ca = t.cosv[t.off[a] + nidx[a]];
    return make_double2((2.0 * ca - 2.0) * t.idx[a] * t.idx[a], 0.0);
  }
  const double sb = t.sinv[t.off[b] + nidx[b]];
  return make_double2(-2.0 * sa * sb * t.idx[a] * t.idx[b], 0.0);
}

// x = (I + alpha L(k))^-1 r at one mode, n <= NF <= kMaxPrecFields, by Gaussian elimination
// with partial pivoting, or Cramer's rule where it does; a (numerically) singular mode is
// passed through unchanged.
// The operators and their coefficients come with the kernel's parameters (constant memory):
// reading the entry list from global memory, entry by entry, was a third of k_mid_solve's
// time.
template <int NF>
__device__ __forceinline__ void mode_solve(const LinTable& t, const int* nidx, double2* v, int n) {
  static_assert(NF <= kMaxPrecFields, "mode solves of at most kMaxPrecFields fields");
  if constexpr (NF == 2) {
    // real symbols (diffusion and reaction terms): one or two real unknowns by Cramer's rule,
    // with one division (the general elimination takes three, and the pivot search:
    // k_mid_solve of 256 x 256 took 9.6 us with it, 8.4 us so)
    if (t.real) {
      const double al = t.alpha_dev ? *t.alpha_dev : t.alpha;
      double m00 = 1.0, m01 = 0.0, m10 = 0.0, m11 = 1.0;
#pragma unroll 2
      for (int g = 0; g < t.nops; ++g) {
        const double sy = al * lin_symbol(t, g, nidx).x;
        m00 += sy * t.coef[g][0][0];
        m01 += sy * t.coef[g][0][1];
        m10 += sy * t.coef[g][1][0];
        m11 += sy * t.coef[g][1][1];
      }
      if (n == 1) m01 = m10 = 0.0, m11 = 1.0;
      const double det = m00 * m11 - m01 * m10;
      if (!(det * det > 1e-300)) return;
      const double inv = 1.0 / det;
      const double2 b0 = v[0], b1 = n == 2 ? v[1] : make_double2(0.0, 0.0);
      v[0] = make_double2(inv * (m11 * b0.x - m01 * b1.x), inv * (m11 * b0.y - m01 * b1.y));
      if (n == 2) v[1] = make_double2(inv * (m00 * b1.x - m10 * b0.x), inv * (m00 * b1.y - m10 * b0.y));
      return;
    }
  }
  double2 A[NF][NF];
  double2 b[NF];
#pragma unroll
  for (int i = 0; i < NF; ++i) {
#pragma unroll
    for (int j = 0; j < NF; ++j) A[i][j] = make_double2(i == j ? 1.0 : 0.0, 0.0);
    b[i] = i < n ? v[i] : make_double2(0.0, 0.0);
  }
  const double alpha = t.alpha_dev ? *t.alpha_dev : t.alpha;
#pragma unroll 2
  for (int g = 0; g < t.nops; ++g) {
    const double2 sy = lin_symbol(t, g, nidx);
#pragma unroll
    for (int i = 0; i < NF; ++i)
#pragma unroll
      for (int j = 0; j < NF; ++j) {
        const double cf = alpha * t.coef[g][i][j];
        A[i][j].x += cf * sy.x;
        A[i][j].y += cf * sy.y;
      }
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < NF; ++k) {
    if (k >= n) break;
    // pivot
    int p = k;
    double best = A[k][k].x * A[k][k].x + A[k][k].y * A[k][k].y;
#pragma unroll
    for (int i = k + 1; i < NF; ++i) {
      if (i >= n) break;
      const double m2 = A[i][k].x * A[i][k].x + A[i][k].y * A[i][k].y;
      if (m2 > best) { best = m2; p = i; }
    }
    if (!(best > 1e-300)) { ok = false; break; }
#pragma unroll
    for (int i = 0; i < NF; ++i)
      if (i == p && p != k) {
#pragma unroll
        for (int j = 0; j < NF; ++j) { const double2 tmp = A[k][j]; A[k][j] = A[i][j]; A[i][j] = tmp; }
        const double2 tb = b[k]; b[k] = b[i]; b[i] = tb;
      }
    const double2 piv = A[k][k];
    const double inv = 1.0 / (piv.x * piv.x + piv.y * piv.y);
    const double2 ip = make_double2(piv.x * inv, -piv.y * inv);
#pragma unroll
    for (int i = k + 1; i < NF; ++i) {
      if (i >= n) break;
      const double2 f = c_mul(A[i][k], ip);
#pragma unroll
      for (int j = k; j < NF; ++j) A[i][j] = c_sub(A[i][j], c_mul(f, A[k][j]));
      b[i] = c_sub(b[i], c_mul(f, b[k]));
    }
  }
  if (!ok) return;
#pragma unroll
  for (int k = NF - 1; k >= 0; --k) {
    if (k >= n) continue;
    double2 acc = b[k];
#pragma unroll
    for (int j = k + 1; j < NF; ++j)
      if (j < n) acc = c_sub(acc, c_mul(A[k][j], b[j]));
    const double2 piv = A[k][k];
    const double inv = 1.0 / (piv.x * piv.x + piv.y * piv.y);
    b[k] = c_mul(acc, make_double2(piv.x * inv, -piv.y * inv));
  }
#pragma unroll
  for (int i = 0; i < NF; ++i)
    if (i < n) v[i] = b[i];
}

}  // namespace rdcu
