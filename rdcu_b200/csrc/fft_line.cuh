// Shared-memory FP64 Stockham FFT over a batch of complex lines (device code).
//
// Method: the Stockham autosort formulation (Van Loan, "Computational Frameworks for
// the Fast Fourier Transform", SIAM 1992, ch. 1.7) with mixed radices 2..16.  Stage s with radix R and span Ns (product of earlier radices) maps butterfly
// j of a line of length L (m = L/R butterflies) as
//     in:  x[j + r*m] * w^(r * (j mod Ns) * L/(Ns*R)),   r < R
//     out: y[(j/Ns)*Ns*R + (j mod Ns) + r*Ns]  = R-point DFT of the inputs,
// which leaves the result in natural order.  Twiddles w^t = exp(-2 pi i t/L) come from
// a table in shared memory.  Each stage stages its butterflies in registers, so one
// buffer suffices (two barriers per stage).
#pragma once
#include <cuda_runtime.h>

#include "internal.h"

namespace rdcu {

__device__ __forceinline__ double2 c_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 c_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 c_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ double2 c_rot(double2 a) {
  return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ double2 tw_get(const double2* tw, int t) {
  double2 w = tw[t];
  if (INV) w.y = -w.y;
  return w;
}

// 16-byte asynchronous global->shared copy (zero-filled when pred is false; the source
// address is then not read).  Completion: cp_async_wait_all() and a barrier.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
// W = 4, 8 or 16 bytes, both addresses W-byte aligned
template <int W>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
  if constexpr (W == 16) {
    cp_async16(smem, gmem, true);
  } else {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(W) : "memory");
  }
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
// commit the copies issued so far as a group; wait until at most one group is pending
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// cos and sin of 2 pi k / R, k = 1..(R-1)/2, for the odd radices, and of 2 pi k / 9 and
// 2 pi k / 16: correctly rounded from the definition.  In constant memory, where the FP64
// instructions read them as operands: as literals the compiler moves those of every radix
// out of the stage loop and spills them.
static __constant__ double c_root3[2] = {-0.5, 0.86602540378443864676};
static __constant__ double c_root5[4] = {0.30901699437494742410, -0.80901699437494742410, 0.95105651629515357212,
                                         0.58778525229247312917};
static __constant__ double c_root7[6] = {0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624,
                                         0.78183148246802980871, 0.97492791218182360702,  0.43388373911755812048};
static __constant__ double c_root11[10] = {0.84125353283118116886,  0.41541501300188642553,  -0.14231483827328514044,
                                           -0.65486073394528506406, -0.95949297361449738989, 0.54064081745559758211,
                                           0.90963199535451837141,  0.98982144188093273238,  0.75574957435425828377,
                                           0.28173255684142969771};
static __constant__ double c_root13[12] = {
    0.88545602565320989590,  0.56806474673115580251,  0.12053668025532305335, -0.35460488704253562597,
    -0.74851074817110109863, -0.97094181742605202716, 0.46472317204376854566, 0.82298386589365639458,
    0.99270887409805399280,  0.93501624268541482344,  0.66312265824079520238, 0.23931566428755776715};
// W_9^e = (c_w9[2 e], -c_w9[2 e + 1]), e <= 4, and W_16^e likewise, e <= 9
static __constant__ double c_w9[10] = {1.0, 0.0, 0.76604444311897803520, 0.64278760968653932632,
                                       0.17364817766693034885, 0.98480775301220805937, -0.5, 0.86602540378443864676,
                                       -0.93969262078590838405, 0.34202014332566873304};
static __constant__ double c_w16[20] = {
    1.0, 0.0, 0.92387953251128675613, 0.38268343236508977173, 0.70710678118654752440, 0.70710678118654752440,
    0.38268343236508977173, 0.92387953251128675613, 0.0, 1.0, -0.38268343236508977173, 0.92387953251128675613,
    -0.70710678118654752440, 0.70710678118654752440, -0.92387953251128675613, 0.38268343236508977173, -1.0, 0.0,
    -0.92387953251128675613, -0.38268343236508977173};
template <int R>
__device__ __forceinline__ double root_cos(int k) {
  return R == 3 ? c_root3[k - 1] : R == 5 ? c_root5[k - 1] : R == 7 ? c_root7[k - 1] : R == 11 ? c_root11[k - 1] : c_root13[k - 1];
}
template <int R>
__device__ __forceinline__ double root_sin(int k) {
  return R == 3 ? c_root3[k] : R == 5 ? c_root5[k + 1] : R == 7 ? c_root7[k + 2] : R == 11 ? c_root11[k + 4] : c_root13[k + 5];
}

// In-register R-point DFT of v (forward: exp(-2 pi i rk/R); inverse: conjugate).  Odd
// primes: the sums and differences of the inputs r and R - r take the cosines and sines
// of the definition, (R-1)^2 real-by-complex products and no table reads (a 5-point DFT
// by complex products with table entries took 20 products and 20 shared-memory reads).
template <int R, bool INV>
struct Dft {
  static_assert(R == 3 || R == 5 || R == 7 || R == 11 || R == 13, "odd primes");
  __device__ __forceinline__ static void run(double2 (&v)[R]) {
    constexpr int H = (R - 1) / 2;
    double2 a[H], b[H];  // per output pair (k, R - k): cosine and sine sums
    const double2 v0 = v[0];
    double2 sum = v0;
#pragma unroll
    for (int k = 0; k < H; ++k) {
      a[k] = v0;
      b[k] = make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      const double2 p = c_add(v[r], v[R - r]), m = c_sub(v[r], v[R - r]);
      sum = c_add(sum, p);
#pragma unroll
      for (int k = 1; k <= H; ++k) {
        const int t = (r * k) % R;
        const double c = root_cos<R>(t <= H ? t : R - t);
        const double s = t <= H ? root_sin<R>(t) : -root_sin<R>(R - t);
        a[k - 1].x += c * p.x;
        a[k - 1].y += c * p.y;
        b[k - 1].x += s * m.x;
        b[k - 1].y += s * m.y;
      }
    }
    v[0] = sum;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      const double2 ib = c_rot<INV>(b[k - 1]);  // -i b forward, +i b inverse
      v[k] = c_add(a[k - 1], ib);
      v[R - k] = c_sub(a[k - 1], ib);
    }
  }
};

template <bool INV>
struct Dft<2, INV> {
  __device__ __forceinline__ static void run(double2 (&v)[2]) {
    double2 a = v[0], b = v[1];
    v[0] = c_add(a, b);
    v[1] = c_sub(a, b);
  }
};

template <bool INV>
struct Dft<4, INV> {
  __device__ __forceinline__ static void run(double2 (&v)[4]) {
    double2 t0 = c_add(v[0], v[2]), t1 = c_sub(v[0], v[2]);
    double2 t2 = c_add(v[1], v[3]), t3 = c_rot<INV>(c_sub(v[1], v[3]));
    v[0] = c_add(t0, t2);
    v[2] = c_sub(t0, t2);
    v[1] = c_add(t1, t3);
    v[3] = c_sub(t1, t3);
  }
};

template <bool INV>
struct Dft<8, INV> {
  __device__ __forceinline__ static void run(double2 (&v)[8]) {
    // X[k] = E[k] + W^k O[k], X[k+4] = E[k] - W^k O[k]; E, O = 4-point DFTs of the
    // even and odd inputs; W = exp(-+ 2 pi i / 8).
    double2 e[4] = {v[0], v[2], v[4], v[6]};
    double2 o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, INV>::run(e);
    Dft<4, INV>::run(o);
    const double s = 0.70710678118654752440;  // sqrt(1/2)
    // W^1 = s(1 -+ i), W^2 = -+ i, W^3 = s(-1 -+ i)
    double2 w1o = INV ? make_double2(s * (o[1].x - o[1].y), s * (o[1].x + o[1].y))
                      : make_double2(s * (o[1].x + o[1].y), s * (o[1].y - o[1].x));
    double2 w2o = c_rot<INV>(o[2]);
    double2 w3o = INV ? make_double2(-s * (o[3].x + o[3].y), s * (o[3].x - o[3].y))
                      : make_double2(s * (o[3].y - o[3].x), -s * (o[3].x + o[3].y));
    v[0] = c_add(e[0], o[0]);
    v[4] = c_sub(e[0], o[0]);
    v[1] = c_add(e[1], w1o);
    v[5] = c_sub(e[1], w1o);
    v[2] = c_add(e[2], w2o);
    v[6] = c_sub(e[2], w2o);
    v[3] = c_add(e[3], w3o);
    v[7] = c_sub(e[3], w3o);
  }
};

// N1 N2-point DFT of coprime factors without twiddles (I. J. Good, "The interaction
// algorithm and practical Fourier analysis", J. R. Stat. Soc. B 20, 1958): with inputs
// n = (N2 n1 + N1 n2) mod N, output k is output (k mod N1, k mod N2) of the 2D DFT.
template <int N1, int N2, bool INV>
struct DftCoprime {
  __device__ __forceinline__ static void run(double2 (&v)[N1 * N2]) {
    constexpr int N = N1 * N2;
    double2 t[N2][N1];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) t[n2][n1] = v[(N2 * n1 + N1 * n2) % N];
      Dft<N1, INV>::run(t[n2]);
    }
    double2 u[N1][N2];
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) {
#pragma unroll
      for (int n2 = 0; n2 < N2; ++n2) u[k1][n2] = t[n2][k1];
      Dft<N2, INV>::run(u[k1]);
    }
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = u[k % N1][k % N2];
  }
};
#define RDCU_DFT_COPRIME(R, N1, N2)                                                        \
  template <bool INV>                                                                      \
  struct Dft<R, INV> {                                                                     \
    __device__ __forceinline__ static void run(double2 (&v)[R]) {     \
      DftCoprime<N1, N2, INV>::run(v);                                                     \
    }                                                                                      \
  }
RDCU_DFT_COPRIME(6, 2, 3);
RDCU_DFT_COPRIME(10, 2, 5);
RDCU_DFT_COPRIME(12, 4, 3);
RDCU_DFT_COPRIME(14, 2, 7);
RDCU_DFT_COPRIME(15, 3, 5);
#undef RDCU_DFT_COPRIME

// R x R points in two steps: X[k1 + R k2] = sum_n2 W^(n2 k1) W_R^(n2 k2) sum_n1 x[R n1 + n2] W_R^(n1 k1)
template <bool INV>
struct Dft<9, INV> {
  __device__ __forceinline__ static void run(double2 (&v)[9]) {
    double2 t[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 3; ++n1) t[n2][n1] = v[3 * n1 + n2];
      Dft<3, INV>::run(t[n2]);
#pragma unroll
      for (int k1 = 1; k1 < 3; ++k1)
        if (n2 > 0) t[n2][k1] = c_mul(t[n2][k1], make_double2(c_w9[2 * n2 * k1], INV ? c_w9[2 * n2 * k1 + 1] : -c_w9[2 * n2 * k1 + 1]));
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      double2 u[3] = {t[0][k1], t[1][k1], t[2][k1]};
      Dft<3, INV>::run(u);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = u[k2];
    }
  }
};
template <bool INV>
struct Dft<16, INV> {
  __device__ __forceinline__ static void run(double2 (&v)[16]) {
    double2 t[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) t[n2][n1] = v[4 * n1 + n2];
      Dft<4, INV>::run(t[n2]);
#pragma unroll
      for (int k1 = 1; k1 < 4; ++k1) {
        if (n2 == 0) continue;
        const int e = n2 * k1;
        t[n2][k1] = e == 4 ? c_rot<INV>(t[n2][k1]) : c_mul(t[n2][k1], make_double2(c_w16[2 * e], INV ? c_w16[2 * e + 1] : -c_w16[2 * e + 1]));
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      double2 u[4] = {t[0][k1], t[1][k1], t[2][k1], t[3][k1]};
      Dft<4, INV>::run(u);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = u[k2];
    }
  }
};

// Complex values a thread holds per stage (register budget of the staging), and the
// largest block of an FFT pass (kMaxBlock x 128 registers fills the register file).
constexpr int kStageElems = 8;
constexpr int kMaxBlock = 512;

// Position of line element i under the swizzle of a radix-8 first stage: the low three
// bits are XORed with the 8-element block index, so the eight consecutive outputs of a
// butterfly land in eight different bank groups across a quarter warp.
__device__ __forceinline__ int swz8(int i) { return i ^ ((i >> 3) & 7); }

// One Stockham stage over nlines lines (stride LS) held in shared memory `buf`.
// Requires blockDim.x * QMAX >= nlines*L/R; the caller sizes the block for that.  QMAX,
// the butterflies of a thread, fills at most kStageElems values by default.
// POW2: L and Ns are powers of two (index arithmetic by shifts); otherwise the
// plan's precomputed invariant divisors are used.
// SWZ: bit 0 writes the outputs at swz8 positions (a first stage, Ns = 1, R = 8: its
// stride-8 stores otherwise put a quarter warp on one bank group); bit 1 reads the
// inputs from swz8 positions (the stage after it).  twz: the twiddle table is stored at
// swz8 positions (the span-8 stage reads twiddles r*kk*L/64 for kk = 0..7, which
// otherwise share a bank group).  Values are unchanged.
// SWZ < 0: the flags swz instead (lines of a multiple of 8 points only).
template <int R, bool INV, bool POW2, int SWZ = 0, int QMAX = (R >= kStageElems ? 1 : kStageElems / R)>
__device__ __forceinline__ void stockham_stage(double2* buf, int LS, int nlines, int L, int Ns, FastDiv dm,
                                               FastDiv dns, const double2* tw, bool twz = false, int swz = 0) {
  const bool swz_in = SWZ < 0 ? (swz & 2) != 0 : (SWZ & 2) != 0;
  const bool swz_out = SWZ < 0 ? (swz & 1) != 0 : (SWZ & 1) != 0;
  const int m = L / R;
  const int nb = nlines * m;
  const int T = blockDim.x;
  const int tstride = L / (Ns * R);
  const int lm = POW2 ? __ffs(m) - 1 : 0;
  const int lns = POW2 ? __ffs(Ns) - 1 : 0;
  double2 v[QMAX][R];
  int dst[QMAX], dbase[QMAX];
#pragma unroll
  for (int q = 0; q < QMAX; ++q) {
    const int g = threadIdx.x + q * T;
    dst[q] = -1;
    dbase[q] = 0;
    if (g < nb) {
      const int line = POW2 ? (g >> lm) : fdiv(g, dm);
      const int j = g - line * m;
      const int jd = POW2 ? (j >> lns) : fdiv(j, dns);
      const int kk = j - jd * Ns;
      const double2* src = buf + line * LS;
      const int tstep = kk * tstride;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        double2 x = src[swz_in ? swz8(j + r * m) : j + r * m];
        if (r > 0 && tstep != 0) x = c_mul(x, tw_get<INV>(tw, twz ? swz8(r * tstep) : r * tstep));
        v[q][r] = x;
      }
      Dft<R, INV>::run(v[q]);
      dbase[q] = line * LS;
      dst[q] = jd * Ns * R + kk;
    } else {
      // defined on every path: a value that looks live around the stage loop keeps its
      // registers in every other radix's stage too
#pragma unroll
      for (int r = 0; r < R; ++r) v[q][r] = make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < QMAX; ++q) {
    if (dst[q] >= 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) buf[dbase[q] + (swz_out ? swz8(dst[q] + r * Ns) : dst[q] + r * Ns)] = v[q][r];
    }
  }
  __syncthreads();
}

// Radix sets a kernel is compiled for: power-of-two lengths use radices 8, 4, 2 only
// (no register spills); any other supported length uses the general set.
constexpr int kRadixPow2 = 0;
constexpr int kRadixAll = 1;
// radices up to 10 only: kernels of this set fit 80 registers where the full set takes 128
// (and spills), which is half as many warps again for passes bound by latency
constexpr int kRadixMid = 2;
// the full set with ceil(8 / R) butterflies per thread, at least kStageElems values whatever
// the radix: kMaxBlock threads then transform any kMaxBlock * kStageElems values.  For the
// tiles whose radix-3, -5, -6 or -7 stages have more butterflies than the full set's block
// (4000 = 16 x 10 x 5 x 5 points: 800 in a stage).  For all lengths it would cost up to 8%
// (2D attempts, 300 x 330: 194 -> 210 us; 2000 x 1000: 1.34 -> 1.44 ms).
constexpr int kRadixWide = 3;

inline bool plan_is_pow2(const LinePlan& p) {
  for (int s = 0; s < p.nstages; ++s)
    if (p.radix[s] != 2 && p.radix[s] != 4 && p.radix[s] != 8) return false;
  return true;
}

inline bool plan_is_mid(const LinePlan& p) {
  for (int s = 0; s < p.nstages; ++s)
    if (p.radix[s] > 10) return false;
  return true;
}

// Full transform of nlines lines.  All threads of the block must call it; the data
// must be visible (a barrier before the call).  Returns after a barrier.  The stages are
// inlined: calls cost the saved registers of every thread and stage (the first stage's
// outputs are swizzled for the second where its radix is even, see radix_seq).
template <int RS, bool INV>
__device__ __forceinline__ void fft_lines(double2* buf, int LS, int nlines, const LinePlan& p, const double2* tw) {
  int Ns = 1;
  const bool sw = p.nstages > 1 && (p.L & 7) == 0 && (p.radix[0] & 1) == 0;
#pragma unroll 1
  for (int s = 0; s < p.nstages; ++s) {
    // (opaque to the compiler, which otherwise hoists every radix's L / R multiples out of
    // the loop and spills them)
    int L = p.L;
    asm volatile("" : "+r"(L));
    const int R = p.radix[s];
    const FastDiv dm = p.div_m[s], dns = p.div_ns[s];
    const int swz = sw ? (s == 0 ? 1 : s == 1 ? 2 : 0) : 0;
#define RDCU_STAGE(K, P2)                                                                          \
  case K:                                                                                         \
    stockham_stage<K, INV, P2, -1, RS == kRadixWide ? (kStageElems + K - 1) / K                    \
                                   : K >= kStageElems ? 1 : kStageElems / K>(                      \
        buf, LS, nlines, L, Ns, dm, dns, tw, false, swz);                                          \
    break;
    if (RS == kRadixPow2) {
      switch (R) {
        RDCU_STAGE(8, true)
        RDCU_STAGE(4, true)
        RDCU_STAGE(2, true)
        default: break;
      }
    } else if (RS == kRadixMid) {
      switch (R) {
        RDCU_STAGE(2, false)
        RDCU_STAGE(3, false)
        RDCU_STAGE(4, false)
        RDCU_STAGE(5, false)
        RDCU_STAGE(6, false)
        RDCU_STAGE(7, false)
        RDCU_STAGE(8, false)
        RDCU_STAGE(9, false)
        RDCU_STAGE(10, false)
        default: break;
      }
    } else {
      switch (R) {
        RDCU_STAGE(2, false)
        RDCU_STAGE(3, false)
        RDCU_STAGE(4, false)
        RDCU_STAGE(5, false)
        RDCU_STAGE(6, false)
        RDCU_STAGE(7, false)
        RDCU_STAGE(8, false)
        RDCU_STAGE(9, false)
        RDCU_STAGE(10, false)
        RDCU_STAGE(11, false)
        RDCU_STAGE(12, false)
        RDCU_STAGE(13, false)
        RDCU_STAGE(14, false)
        RDCU_STAGE(15, false)
        RDCU_STAGE(16, false)
        default: break;  // plans only contain the radices above
      }
    }
#undef RDCU_STAGE
    Ns *= R;
  }
}

// The same transform for a power-of-two length L known at compile time: the stage
// sequence of make_line_plan (radix 8 while 8 divides what is left, then 4 or 2) with
// every length, span and stride a constant.  Bitwise equal to fft_lines on that plan.
template <int L, bool INV, int NS = 1>
__device__ __forceinline__ void fft_pow2_t(double2* buf, int LS, int nlines, const double2* tw, bool twz) {
  if constexpr (NS < L) {
    constexpr int REM = L / NS;
    constexpr int R = (REM % 8 == 0) ? 8 : REM;  // REM is 8^a times 1, 2 or 4
    static_assert(R == 2 || R == 4 || R == 8, "power-of-two lengths only");
    // a radix-8 first stage writes swizzled when a second stage reads it back
    constexpr int SWZ = (NS == 1 && R == 8 && L > 8) ? 1 : (NS == 8 ? 2 : 0);
    stockham_stage<R, INV, true, SWZ>(buf, LS, nlines, L, NS, FastDiv{}, FastDiv{}, tw, twz);
    fft_pow2_t<L, INV, NS * R>(buf, LS, nlines, tw, twz);
  }
}

// The transform for any supported length L known at compile time (the plan's stage
// sequence, constant spans and divisors; bitwise equal to fft_lines on that plan).
// Twiddles are read plainly.
template <int L, bool INV, int S = 0, int NS = 1>
__device__ __forceinline__ void fft_fixed_t(double2* buf, int LS, int nlines, const double2* tw) {
  constexpr RadixSeq seq = radix_seq(L);
  if constexpr (S < seq.n) {
    constexpr int R = seq.r[S];
    constexpr bool SW = seq.n > 1 && L % 8 == 0 && seq.r[0] % 2 == 0;
    constexpr int SWZ = SW ? (S == 0 ? 1 : S == 1 ? 2 : 0) : 0;
    stockham_stage<R, INV, false, SWZ>(buf, LS, nlines, L, NS, make_fastdiv_c(L / R), make_fastdiv_c(NS), tw);
    fft_fixed_t<L, INV, S + 1, NS * R>(buf, LS, nlines, tw);
  }
}

}  // namespace rdcu
