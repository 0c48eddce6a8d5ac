// Preconditioner of one-dimensional stiff problems: z = (I + alpha J_lin)^-1 r, J_lin the
// constant-coefficient linear part of the finite-difference Jacobian, which the FFT
// diagonalises (modes.cuh).
//
// One kernel of one CTA: the fields go into shared memory as complex lines (two real
// fields per line), the forward transform, the n x n solve of every mode pair (k, N - k)
// in place, the inverse transform and the store.  A line of up to 8192 complex values is
// 128 KB, so the data cross global memory once; the transforms' exchanges and FP64 work on
// the one SM bound it (about 17k cycles of each at 8192 points).  Against the three
// launches of the general passes it saves two launches, and it reaches lines that those
// passes cannot hold (above 4096 points, which ran without a preconditioner).
#include <algorithm>
#include <cmath>

#include "fft_line.cuh"
#include "modes.cuh"
#include "prec1d.h"

namespace rdcu {
namespace {

// A thread stages up to 16 values per stage, so that 8192 values need at most 745 threads
// whatever the radix (11 leaves the fewest values per thread).
constexpr int kLineElems = 16;
constexpr int kLineThreads = 768;

struct LinePrecArgs {
  int n, N, np;
  LinePlan plan;
  const double2* tw;
  const double* r;
  double* z;
  LinTable lin;
};

template <int RS, int NF>
__global__ void __launch_bounds__(kLineThreads, 1) k_prec_line(const __grid_constant__ LinePrecArgs a) {
  extern __shared__ double2 buf[];
  const int n = a.n, N = a.N, np = a.np, T = blockDim.x, tid = threadIdx.x;
  for (int p = 0; p < np; ++p) {
    const double* r0 = a.r + (long long)(2 * p) * N;
    const bool two = 2 * p + 1 < n;
    for (int x = tid; x < N; x += T) buf[p * N + x] = make_double2(r0[x], two ? r0[N + x] : 0.0);
  }
  __syncthreads();
  fft_lines<RS, false, kLineElems>(buf, N, np, a.plan, a.tw);
  for (int k = tid; k <= N / 2; k += T) {
    const int km = k == 0 ? 0 : N - k;
    double2 v[NF];
#pragma unroll
    for (int p = 0; p < (NF + 1) / 2; ++p) {
      if (p < np) {
        const double2 Z = buf[p * N + k], Zm = buf[p * N + km];
        v[2 * p] = make_double2(0.5 * (Z.x + Zm.x), 0.5 * (Z.y - Zm.y));
        v[2 * p + 1] = make_double2(0.5 * (Z.y + Zm.y), -0.5 * (Z.x - Zm.x));
      }
    }
    const int nidx[3] = {k, 0, 0};
    mode_solve<NF>(a.lin, nidx, v, n);
#pragma unroll
    for (int p = 0; p < (NF + 1) / 2; ++p) {
      if (p < np) {
        double2 A = v[2 * p], B = 2 * p + 1 < n ? v[2 * p + 1] : make_double2(0.0, 0.0);
        if (k == km) {  // the real modes of real fields
          A.y = 0.0;
          B.y = 0.0;
        }
        buf[p * N + km] = make_double2(A.x + B.y, B.x - A.y);
        buf[p * N + k] = make_double2(A.x - B.y, A.y + B.x);
      }
    }
  }
  __syncthreads();
  fft_lines<RS, true, kLineElems>(buf, N, np, a.plan, a.tw);
  for (int p = 0; p < np; ++p) {
    double* z0 = a.z + (long long)(2 * p) * N;
    const bool two = 2 * p + 1 < n;
    for (int x = tid; x < N; x += T) {
      const double2 v = buf[p * N + x];
      z0[x] = v.x;
      if (two) z0[N + x] = v.y;
    }
  }
}

template <typename F>
void by_kind(const LinePlan& p, int n, F&& f) {
  if (plan_is_pow2(p)) {
    if (n <= 2)
      f(k_prec_line<kRadixPow2, 2>);
    else
      f(k_prec_line<kRadixPow2, kMaxPrecFields>);
  } else {
    if (n <= 2)
      f(k_prec_line<kRadixAll, 2>);
    else
      f(k_prec_line<kRadixAll, kMaxPrecFields>);
  }
}

template <typename T>
bool put(T** dst, const std::vector<T>& v, size_t* bytes) {
  const size_t b = std::max<size_t>(1, v.size()) * sizeof(T);
  if (cudaMalloc((void**)dst, b) != cudaSuccess) return false;
  *bytes += b;
  return v.empty() || cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess;
}

}  // namespace

bool LinePrecond::init(int n, int N, double L, const std::vector<LinEntry>& lin) {
  release();
  const int np = (n + 1) / 2;
  if (n < 1 || n > kMaxPrecFields || (long long)np * N > kLinePrecElems) return false;
  if (!make_line_plan(N, &plan_, kLinePrecElems)) return false;
  n_ = n;
  N_ = N;
  dx_ = L / N;
  // the threads that hold every line of a stage at its radix
  int per = kLineElems;
  for (int s = 0; s < plan_.nstages; ++s) {
    const int R = plan_.radix[s];
    per = std::min(per, R >= kLineElems ? R : kLineElems / R * R);
  }
  block_ = std::max(128, ((np * N + per - 1) / per + 31) / 32 * 32);
  // the roots of unity, half of them computed (the others are their conjugates), serve the
  // transforms and the operators' symbols
  std::vector<double2> tw(N);
  std::vector<double> sv(N), cv(N);
  for (int m = 0; 2 * m <= N; ++m) {
    const long double th = 2.0L * 3.141592653589793238462643383279502884L * m / N;
    const double c = 4LL * m == N ? 0.0 : (double)cosl(th), sn = 2 * m == N ? 0.0 : (double)sinl(th);
    for (int q : {m, (N - m) % N}) {
      cv[q] = c;
      sv[q] = q == m ? sn : -sn;
      tw[q] = make_double2(c, -sv[q]);
    }
  }
  nlin_ = (int)lin.size();
  bool ok = put(&tw_, tw, &device_bytes) && put(&lin_, lin, &device_bytes) && put(&sinv_, sv, &device_bytes) &&
            put(&cosv_, cv, &device_bytes);
  by_kind(plan_, n_, [&](auto kern) {
    ok = ok && cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kLinePrecElems * (int)sizeof(double2)) == cudaSuccess;
  });
  if (!ok) {
    cudaGetLastError();
    release();
  }
  return ok;
}

void LinePrecond::release() {
  void* p[] = {tw_, lin_, sinv_, cosv_};
  for (void* q : p)
    if (q) cudaFree(q);
  tw_ = nullptr;
  lin_ = nullptr;
  sinv_ = nullptr;
  cosv_ = nullptr;
  device_bytes = 0;
}

cudaError_t LinePrecond::apply(const double* r, double* z, const double* alpha_dev, cudaStream_t st) const {
  LinePrecArgs a{};
  a.n = n_;
  a.N = N_;
  a.np = (n_ + 1) / 2;
  a.plan = plan_;
  a.tw = tw_;
  a.r = r;
  a.z = z;
  a.lin.n = n_;
  a.lin.nent = nlin_;
  a.lin.ndim = 1;
  a.lin.ent = lin_;
  a.lin.sinv = sinv_;
  a.lin.cosv = cosv_;
  a.lin.alpha_dev = alpha_dev;
  for (int d = 0; d < 3; ++d) {
    a.lin.Ns[d] = d == 0 ? N_ : 1;
    a.lin.dx[d] = d == 0 ? dx_ : 1.0;
  }
  const size_t smem = (size_t)a.np * N_ * sizeof(double2);
  by_kind(plan_, n_, [&](auto kern) { kern<<<1, block_, smem, st>>>(a); });
  return cudaGetLastError();
}

}  // namespace rdcu
