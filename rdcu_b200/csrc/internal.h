// Internal types of librdcu (not part of the C ABI).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/rdcu.h"

namespace rdcu {

// ----------------------------------------------------------------------------- FFT plans
constexpr int kMaxStages = 16;
constexpr int kMaxLine = 4096;  // longest complex line one CTA transforms in shared memory

// Division of 0 <= n < 2^31 by an invariant d >= 1 with a multiply and a shift
// (Granlund & Montgomery, "Division by invariant integers using multiplication",
// PLDI 1994): s = ceil(log2 d), m = ceil(2^(31+s) / d) < 2^32, q = (n*m) >> (31+s).
// Exact because the rounding error of m is below d and n*error < 2^(31+s).
struct FastDiv {
  unsigned m;
  int s;
};
inline FastDiv make_fastdiv(unsigned d) {
  if (d == 0) d = 1;  // the tile width of a pass that the grid does not have
  int s = 0;
  while ((1ull << s) < d) ++s;
  const unsigned long long num = 1ull << (31 + s);
  FastDiv f;
  f.m = (unsigned)((num + d - 1) / d);
  f.s = s;
  return f;
}
// make_fastdiv for a divisor known at compile time
__host__ __device__ constexpr FastDiv make_fastdiv_c(unsigned d) {
  int s = 0;
  while ((1ull << s) < d) ++s;
  const unsigned long long num = 1ull << (31 + s);
  return FastDiv{(unsigned)((num + d - 1) / d), s};
}
#ifdef __CUDACC__
__device__ __forceinline__ int fdiv(int n, FastDiv f) {
  return (int)(((unsigned long long)(unsigned)n * f.m) >> (31 + f.s));
}
#endif

// Mixed-radix Stockham plan for one complex line length.
struct LinePlan {
  int L;
  int nstages;
  int radix[kMaxStages];
  FastDiv div_m[kMaxStages];   // L / radix[s] (butterflies per line at stage s)
  FastDiv div_ns[kMaxStages];  // span Ns before stage s
};

// Stage radices of a line of L points; n = 0 when L has a prime factor above 13 (n = 0 also
// for L = 1, which needs no stage).  Powers of two: 8s, then 4 or 2 (the register kernels' sequence).
// Other lengths: as few radices up to 16 as possible, since every stage is a trip through
// shared memory and two barriers, and as even as possible, since the smallest one sets the
// number of threads (100 = 10 x 10, 80 = 8 x 10 rather than 5 x 16); in the order of
// gcd(R, 8): the first stage's stores go R elements apart, which is free of bank
// conflicts for odd R.
struct RadixSeq {
  int n;
  int r[kMaxStages];
};
__host__ __device__ constexpr RadixSeq radix_seq(int L) {
  RadixSeq q{};
  int rem = L;
  if ((L & (L - 1)) == 0) {
    while (rem > 1) {
      const int R = rem % 8 == 0 ? 8 : rem;
      q.r[q.n++] = R;
      rem /= R;
    }
    return q;
  }
  // all but the last three factors: the largest divisors; then the most even split into
  // as few factors as possible
  while (rem > 16 * 16 * 16) {
    int R = 16;
    while (R > 1 && rem % R != 0) --R;
    if (R == 1) return RadixSeq{};
    q.r[q.n++] = R;
    rem /= R;
  }
  int best[3] = {0, 0, 0};
  if (rem <= 16) {
    best[0] = rem;
  } else {
    for (int a = 16; a >= 2 && !best[0]; --a)  // two factors a >= b, the smallest a
      if (rem % a == 0 && rem / a <= a)
        for (int c = a; c >= 2; --c)
          if (rem % c == 0 && rem / c <= c) {
            best[0] = c;
            best[1] = rem / c;
          }
    if (!best[0])
      for (int a = 16; a >= 2; --a)  // three factors a >= b >= c, the largest c
        if (rem % a == 0)
          for (int b = a; b >= 2; --b)
            if (rem / a % b == 0 && rem / a / b <= b && rem / a / b > best[2]) {
              best[0] = a;
              best[1] = b;
              best[2] = rem / a / b;
            }
  }
  if (!best[0]) {  // no three factors up to 16: the largest divisors one by one
    while (rem > 1) {
      int R = 16;
      while (R > 1 && rem % R != 0) --R;
      if (R == 1) return RadixSeq{};
      q.r[q.n++] = R;
      rem /= R;
    }
  } else {
    for (int i = 0; i < 3; ++i)
      if (best[i] > 1) q.r[q.n++] = best[i];
  }
  for (int i = 1; i < q.n; ++i)  // stable insertion sort
    for (int k = i; k > 0; --k) {
      const int a = q.r[k - 1] % 8 == 0 ? 8 : q.r[k - 1] % 4 == 0 ? 4 : q.r[k - 1] % 2 == 0 ? 2 : 1;
      const int b = q.r[k] % 8 == 0 ? 8 : q.r[k] % 4 == 0 ? 4 : q.r[k] % 2 == 0 ? 2 : 1;
      if (a <= b) break;
      const int t = q.r[k];
      q.r[k] = q.r[k - 1];
      q.r[k - 1] = t;
    }
  return q;
}

bool make_line_plan(int L, LinePlan* p);
// exp(-2 pi i t / L) for t < L, rounded from long double.
void make_twiddles(int L, std::vector<double2>& tw);

// ----------------------------------------------------------------------------- spectra
// One entry of an inverse-transform channel: coef * Mpart(k) * U_src(k), where
// Mpart is the real-part (part 0) or imaginary-part (part 1) multiplier of the
// derivative operator on axes ax0 (and ax1) -- see spectral.cu.
struct ChanEntry {
  int src;   // source field
  int nax;   // 0: identity, 1: d_ax0, 2: d_ax0 d_ax1
  int ax0, ax1;
  int part;  // 0: Re of the reference's complex Y block, 1: Im
  int pad;
  double coef;
};

struct ChanTable {
  int nch;
  const int* off;         // [nch+1] entry ranges
  const ChanEntry* ent;
  const double* kv;       // wavenumbers, axis a at kv + kv_off[a]
  int kv_off[3];
  int Ns[3];
  int ndim;
  int kv_total;  // sum of Ns over the axes (length of kv)
};

// Dictionary terms left after folding the linear derivative terms into channels.
struct DictTerm {
  int field;
  int nf;   // factors
  int off;  // first factor
  int pad;
  double C;
};
struct DictFactor {
  int q;    // quantity: < n physical field, else channel q-n
  int eta;  // integer power (never 0: zero powers are dropped, pow(x,0) == 1)
};
struct DictTable {
  int n;
  int nterms;
  const DictTerm* terms;      // grouped by field, reference order kept within a field
  const DictFactor* fac;
  const int* field_begin;     // [n+1]
  const int* fold;            // [n] channel holding the folded linear part, -1 if none
  int nfac;                   // number of factors (fac length)
  // Dense form when every term is a product of fields of total degree <= 3 in poly_nf
  // (= n <= 3) fields: f_i = fold_i + sum_m poly[i * poly_count + m] * monomial_m (Mono
  // order); poly_nf = 0 otherwise.
  const double* poly;
  int poly_nf, poly_count;
};

// Monomials of total degree <= 3 in NF variables, in a fixed order: monomial 0 is 1 and
// monomial m > 0 is monomial parent(m) times variable var(m).
template <int NF>
struct Mono;
template <>
struct Mono<1> {
  static constexpr int count = 4;
  __host__ __device__ static constexpr int parent(int m) { return m - 1; }
  __host__ __device__ static constexpr int var(int) { return 0; }
};
template <>
struct Mono<2> {
  static constexpr int count = 10;  // 1 u v uu uv vv uuu uuv uvv vvv
  __host__ __device__ static constexpr int parent(int m) {
    return m == 1 || m == 2 ? 0 : m == 3 || m == 4 ? 1 : m == 5 ? 2 : m == 6 || m == 7 ? 3 : m == 8 ? 4 : 5;
  }
  __host__ __device__ static constexpr int var(int m) { return m == 1 || m == 3 || m == 6 ? 0 : 1; }
};
template <>
struct Mono<3> {
  static constexpr int count = 20;
  __host__ __device__ static constexpr int parent(int m) {
    constexpr int p[20] = {-1, 0, 0, 0, 1, 1, 1, 2, 2, 3, 4, 4, 4, 5, 5, 6, 7, 7, 8, 9};
    return p[m];
  }
  __host__ __device__ static constexpr int var(int m) {
    constexpr int v[20] = {-1, 0, 1, 2, 0, 1, 2, 1, 2, 2, 0, 1, 2, 1, 2, 2, 1, 2, 2, 2};
    return v[m];
  }
};

// Exponent vectors (up to 3 variables) of the Mono<nf> monomials.
inline std::vector<std::array<int, 3>> mono_exponents(int nf) {
  std::vector<std::array<int, 3>> ex;
  auto build = [&](auto mn) {
    using MN = decltype(mn);
    ex.assign(MN::count, {0, 0, 0});
    for (int m = 1; m < MN::count; ++m) {
      ex[m] = ex[MN::parent(m)];
      ex[m][MN::var(m)] += 1;
    }
  };
  if (nf == 1) build(Mono<1>{});
  if (nf == 2) build(Mono<2>{});
  if (nf == 3) build(Mono<3>{});
  return ex;
}

// Constant-coefficient linear part of the finite-difference Jacobian, one entry per
// linear term: row field, source field, FD operator, coefficient.  Its symbol at
// wavenumber theta_a = 2 pi m_a / N_a is exact for the reference's stencils:
// identity 1; d_a -> i sin(theta_a)/dx_a; d_a d_a -> (2 cos(theta_a) - 2)/dx_a^2;
// d_a d_b -> -2 sin(theta_a) sin(theta_b)/(dx_a dx_b) (the reference's 0.5 factor).
struct LinEntry {
  int row, src, nax, ax0, ax1, pad;
  double coef;
};
constexpr int kMaxPrecFields = 4;  // per-mode dense solve size of the preconditioner

// The linear entries by operator (identity, d_a, d_a d_b): J_lin = sum_g symbol_g C_g.
constexpr int kMaxLinOps = 13;
struct LinTable {
  int n, nops, ndim;
  int real;  // every symbol is real (no first derivative)
  struct {
    int nax, ax0, ax1;
  } op[kMaxLinOps];
  double coef[kMaxLinOps][kMaxPrecFields][kMaxPrecFields];
  const double* sinv;  // sin(2 pi m / N_a) at sinv + off[a]
  const double* cosv;
  int off[3];
  int Ns[3];
  double idx[3];       // 1 / dx
  double alpha;        // preconditioner of I + alpha * J_lin
  const double* alpha_dev;  // when set, alpha is read from here (device-resident solves)
};
// Fills the operators and coefficients of t from the entries.
void set_lin_ops(const std::vector<LinEntry>& lin, LinTable* t);

// ----------------------------------------------------------------------------- DP45
enum StopReason { kStopNone = 0, kStopDone = 1, kStopOutput = 2, kStopLog = 3, kStopChunk = 4 };

// Device-resident DP45 controller state.  Kernels of one attempt read the buffer
// slots from here, so a step sequence can run (and be captured in a CUDA graph)
// without host round trips.
struct DP45Ctl {
  double t, h, hmin, hmax, t1;
  double t_last;        // start of the last accepted step
  double err_norm;      // last RMS error norm
  double atol, rtol;
  long long n_attempts, n_accepted;
  int running;          // kernels of an attempt return at once when 0
  int stop_reason;
  int accepted;         // last attempt accepted
  int fixed;
  int check_t1;         // solve mode: stop at t >= t1 or h <= hmin
  int y_slot, yn_slot, yl_slot;    // which ybuf is y, the stage state / y_new, y_last
  int k1_buf, k7_buf;              // kbuf index of logical k1 and k7 (FSAL swap)
  int last_k1_buf, last_k7_buf;    // mapping of the last accepted step (dense output)
  int log_count, log_cap;
  int eval_i, n_eval;
  int max_attempts;     // per launch sequence
  int attempts_this_launch;
  int nparts;           // error partial sums written by the stage-7 epilogue
  int pipe_err;         // nonzero: a pass on TMA tiles gave up waiting for its copies
};

struct DP45Bufs {
  double* ybuf[3];
  double* kbuf[7];
};

// Sets the message rdcu_last_error(NULL) returns on this thread (api.cu).
void set_thread_error(const std::string& msg);

// Allows a kernel the largest dynamic shared memory the device grants next to its static
// shared memory (*limit, in bytes).  The limit belongs to the function, whatever handle
// launches it: set to one handle's size, it would fail the launches of another that needs
// more.
inline bool opt_in_smem(const void* func, size_t* limit = nullptr) {
  cudaFuncAttributes fa;
  if (cudaFuncGetAttributes(&fa, func) != cudaSuccess) return false;
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return false;
  const int dyn = optin - (int)fa.sharedSizeBytes;
  if (limit) *limit = (size_t)std::max(0, dyn);
  return cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) == cudaSuccess;
}

#ifdef __CUDACC__
// Programmatic dependent launch: waits for the kernels this one depends on (no effect in a
// launch without the attribute), then lets the next kernel of the chain start its own
// prologue.  Before the wait a kernel reads only what no kernel of the chain writes.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch of a kernel of a chain: with `chain`, its prologue may overlap the kernel before it
// on the stream (which must be one that calls chain_wait(), or finish first).
template <typename... KA, typename... A>
inline cudaError_t launch_chain(bool chain, void (*kern)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chain ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}
#endif

}  // namespace rdcu
