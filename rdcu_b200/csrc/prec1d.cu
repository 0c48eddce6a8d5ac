// Preconditioner of one-dimensional stiff problems: z = (I + alpha J_lin)^-1 r, J_lin the
// constant-coefficient linear part of the finite-difference Jacobian, which the FFT
// diagonalises (modes.cuh).
//
// One kernel, one thread-block cluster.  Two real fields form a complex line of N = C Q
// points; CTA r of the cluster of C holds the points r + C q and transforms them over q,
//     F_r[a] = sum_q x[r + C q] W_Q^(q a),
// then the C-point DFTs across the cluster, read from its CTAs through distributed shared
// memory, give the spectrum,
//     X[a + Q b] = sum_r W_C^(r b) W_N^(r a) F_r[a],   a < Q, b < C.
// The mode k = a + Q b and its mirror N - k come from a and Q - a, so a CTA that takes the
// pairs (a, Q - a) solves its modes alone and sends the results back the same way; the
// inverse transform ends on the CTA's own points.  Two cluster barriers in all.
//
// The data (at most 64 KB per CTA) cross global memory once; what is left is the latency
// of a short transform: with one CTA for the whole line, 8192 points took 80 us (FP64 work
// and exchanges of 8192 points on one SM), with eight 17.6 us (19.2
// with the general elimination for each mode).  The general passes take
// three launches and hold no line above 4096 points.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "fft_line.cuh"
#include "modes.cuh"
#include "prec1d.h"

namespace rdcu {
namespace {

namespace cg = cooperative_groups;

constexpr int kLineThreads = 512;
constexpr int kLineElems = kLineThreads * kStageElems;  // values of a CTA's part of the lines

struct LinePrecArgs {
  int n, N, Q, np;
  LinePlan plan;      // of Q
  const double2* tw;  // exp(-2 pi i t / N)
  const double* r;
  double* z;
  LinTable lin;
};

__host__ __device__ constexpr int pairs_of(int Q, int C) { return (Q / 2 + 1 + C - 1) / C; }
__host__ __device__ constexpr size_t line_smem(int Q, int C, int np) {
  return ((size_t)Q + (size_t)np * Q + (size_t)np * pairs_of(Q, C) * 2 * C) * sizeof(double2);
}

// Forward or inverse transforms of the CTA's part of the lines (LX: their length when it is
// known at compile time).
template <int LX, bool INV>
__device__ __forceinline__ void part_fft(double2* buf, int Q, int np, const LinePlan& p, const double2* tw) {
  if constexpr (LX > 0)
    fft_pow2_t<LX, INV>(buf, LX, np, tw, true);
  else
    fft_lines<kRadixAll, INV>(buf, Q, np, p, tw);
}

template <int C, int LX, int NF>
__global__ void __launch_bounds__(LX > 0 ? 256 : kLineThreads, 1) k_prec_line(const __grid_constant__ LinePrecArgs a) {
  extern __shared__ double2 sm[];
  const int n = a.n, N = a.N, Q = LX > 0 ? LX : a.Q, np = a.np, T = blockDim.x, tid = threadIdx.x;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = C > 1 ? (int)cl.block_rank() : 0;
  double2* tw = sm;
  double2* buf = tw + Q;       // the CTA's points of every line
  double2* X = buf + np * Q;   // its modes: [line][pair][side][b]
  const int nI = Q / 2 + 1, nP = pairs_of(Q, C);
  for (int t = tid; t < Q; t += T) tw[LX > 0 ? swz8(t) : t] = a.tw[t * C];
  chain_wait();
  for (int p = 0; p < np; ++p) {
    const double* r0 = a.r + (long long)(2 * p) * N + rank;
    const bool two = 2 * p + 1 < n;
    for (int q = tid; q < Q; q += T) buf[p * Q + q] = make_double2(r0[(long long)q * C], two ? r0[N + (long long)q * C] : 0.0);
  }
  __syncthreads();
  part_fft<LX, false>(buf, Q, np, a.plan, tw);
  if (C > 1) cl.sync();
  // pair i = rank + C ii covers a = i (side 0) and a = Q - i (side 1, unless it is i itself)
  const int ntask = np * nP * 2;
  auto task = [&](int e, int* p, int* i, int* av) {
    *p = e / (nP * 2);
    const int w = e - *p * nP * 2;
    *i = rank + C * (w >> 1);
    *av = (w & 1) ? Q - *i : *i;
    return *i < nI && !((w & 1) && (*i == 0 || 2 * *i == Q));
  };
  for (int e = tid; e < ntask; e += T) {
    int p, i, av;
    if (!task(e, &p, &i, &av)) continue;
    double2 v[C];
#pragma unroll
    for (int r = 0; r < C; ++r) {
      const double2* src = C > 1 ? cl.map_shared_rank(buf, r) : buf;
      v[r] = src[p * Q + av];
      if (r > 0) v[r] = c_mul(v[r], __ldg(&a.tw[r * av]));
    }
    if constexpr (C > 1) Dft<C, false>::run(v);
#pragma unroll
    for (int b = 0; b < C; ++b) X[e * C + b] = v[b];
  }
  __syncthreads();
  for (int e = tid; e < nP * C; e += T) {
    const int ii = e / C, b = e - ii * C;
    const int i = rank + C * ii;
    if (i >= nI) continue;
    // the mirror of k = i + Q b
    int side = 1, bm = C - 1 - b;
    if (i == 0 || 2 * i == Q) {
      side = 0;
      if (i == 0) bm = b == 0 ? 0 : C - b;
      if (b > bm) continue;  // done with its mirror
    }
    double2* x0 = X + ii * 2 * C + b;
    double2* xm = X + (ii * 2 + side) * C + bm;
    const int stride = nP * 2 * C;
    double2 v[NF];
#pragma unroll
    for (int p = 0; p < (NF + 1) / 2; ++p) {
      if (p < np) {
        const double2 Z = x0[p * stride], Zm = xm[p * stride];
        v[2 * p] = make_double2(0.5 * (Z.x + Zm.x), 0.5 * (Z.y - Zm.y));
        v[2 * p + 1] = make_double2(0.5 * (Z.y + Zm.y), -0.5 * (Z.x - Zm.x));
      }
    }
    const int nidx[3] = {i + Q * b, 0, 0};
    mode_solve<NF>(a.lin, nidx, v, n);
#pragma unroll
    for (int p = 0; p < (NF + 1) / 2; ++p) {
      if (p < np) {
        double2 A = v[2 * p], B = 2 * p + 1 < n ? v[2 * p + 1] : make_double2(0.0, 0.0);
        if (x0 == xm) {  // the real modes of real fields
          A.y = 0.0;
          B.y = 0.0;
        }
        xm[p * stride] = make_double2(A.x + B.y, B.x - A.y);
        x0[p * stride] = make_double2(A.x - B.y, A.y + B.x);
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < ntask; e += T) {
    int p, i, av;
    if (!task(e, &p, &i, &av)) continue;
    double2 v[C];
#pragma unroll
    for (int b = 0; b < C; ++b) v[b] = X[e * C + b];
    if constexpr (C > 1) Dft<C, true>::run(v);
#pragma unroll
    for (int r = 0; r < C; ++r) {
      if (r > 0) v[r] = c_mul(v[r], tw_get<true>(a.tw, r * av));
      double2* dst = C > 1 ? cl.map_shared_rank(buf, r) : buf;
      dst[p * Q + av] = v[r];
    }
  }
  if (C > 1)
    cl.sync();
  else
    __syncthreads();
  part_fft<LX, true>(buf, Q, np, a.plan, tw);
  for (int p = 0; p < np; ++p) {
    double* z0 = a.z + (long long)(2 * p) * N + rank;
    const bool two = 2 * p + 1 < n;
    for (int q = tid; q < Q; q += T) {
      const double2 v = buf[p * Q + q];
      z0[(long long)q * C] = v.x;
      if (two) z0[N + (long long)q * C] = v.y;
    }
  }
}

using LineKernel = void (*)(LinePrecArgs);

template <int C>
LineKernel kernel_of(int Q, int n) {
  // power-of-two lines end at 1024 points per CTA up to 8192 in all
  if constexpr (C == 1 || C == 2 || C == 4 || C == 8)
    if (Q == 1024) return n <= 2 ? k_prec_line<C, 1024, 2> : k_prec_line<C, 1024, kMaxPrecFields>;
  return n <= 2 ? k_prec_line<C, 0, 2> : k_prec_line<C, 0, kMaxPrecFields>;
}

LineKernel kernel_of(int C, int Q, int n) {
  switch (C) {
    case 8: return kernel_of<8>(Q, n);
    case 7: return kernel_of<7>(Q, n);
    case 6: return kernel_of<6>(Q, n);
    case 5: return kernel_of<5>(Q, n);
    case 4: return kernel_of<4>(Q, n);
    case 3: return kernel_of<3>(Q, n);
    case 2: return kernel_of<2>(Q, n);
    default: return kernel_of<1>(Q, n);
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
  if (n < 1 || n > kMaxPrecFields || N < 1 || N > 8 * kLineElems) return false;
  // The cluster: the smallest divisor of N that leaves a CTA at most 1024 values (a few
  // radix stages; a cluster barrier costs as much as one), else the largest up to 8.
  C_ = 1;
  for (int c = 8; c >= 1; --c) {
    if (N % c) continue;
    if (C_ == 1 || np * (N / c) <= 1024) C_ = c;
  }
  const int Q = N / C_;
  if (np * Q > kLineElems || !make_line_plan(Q, &plan_)) return false;
  n_ = n;
  N_ = N;
  dx_ = L / N;
  // the threads that hold every line of a stage at its radix
  int per = kStageElems;
  for (int s = 0; s < plan_.nstages; ++s) {
    const int R = plan_.radix[s];
    per = std::min(per, R >= kStageElems ? R : kStageElems / R * R);
  }
  block_ = std::max(128, ((np * Q + per - 1) / per + 31) / 32 * 32);
  if (block_ > kLineThreads) return false;
  block_ = std::max(block_, 256);  // the mode solves use them
  // the roots of unity, half of them computed (the others are their conjugates), serve the
  // transforms and the operators' symbols
  std::vector<double2> tw(N);
  std::vector<double> sv(N), cv(N);
  for (int m = 0; 2 * m <= N; ++m) {
    const long double th = 2.0L * 3.141592653589793238462643383279502884L * m / N;
    long double sl, cl;
    sincosl(th, &sl, &cl);
    const double c = 4LL * m == N ? 0.0 : (double)cl, sn = 2 * m == N ? 0.0 : (double)sl;
    for (int q : {m, (N - m) % N}) {
      cv[q] = c;
      sv[q] = q == m ? sn : -sn;
      tw[q] = make_double2(c, -sv[q]);
    }
  }
  set_lin_ops(lin, &lin_);
  bool ok = put(&tw_, tw, &device_bytes) && put(&sinv_, sv, &device_bytes) &&
            put(&cosv_, cv, &device_bytes);
  size_t limit = 0;
  ok = ok && opt_in_smem((const void*)kernel_of(C_, Q, n_), &limit) && line_smem(Q, C_, np) <= limit;
  if (!ok) {
    cudaGetLastError();
    release();
  }
  return ok;
}

void LinePrecond::release() {
  void* p[] = {tw_, sinv_, cosv_};
  for (void* q : p)
    if (q) cudaFree(q);
  tw_ = nullptr;
  sinv_ = nullptr;
  cosv_ = nullptr;
  device_bytes = 0;
}

cudaError_t LinePrecond::apply(const double* r, double* z, const double* alpha_dev, cudaStream_t st) const {
  LinePrecArgs a{};
  a.n = n_;
  a.N = N_;
  a.Q = N_ / C_;
  a.np = (n_ + 1) / 2;
  a.plan = plan_;
  a.tw = tw_;
  a.r = r;
  a.z = z;
  a.lin = lin_;
  a.lin.n = n_;
  a.lin.ndim = 1;
  a.lin.sinv = sinv_;
  a.lin.cosv = cosv_;
  a.lin.alpha_dev = alpha_dev;
  for (int d = 0; d < 3; ++d) {
    a.lin.Ns[d] = d == 0 ? N_ : 1;
    a.lin.idx[d] = d == 0 ? 1.0 / dx_ : 1.0;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C_);
  cfg.blockDim = dim3(block_);
  cfg.dynamicSmemBytes = line_smem(a.Q, C_, a.np);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C_;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel_of(C_, N_ / C_, n_), a);
}

}  // namespace rdcu
