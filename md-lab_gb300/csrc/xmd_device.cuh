// xmd_device.cuh -- device helpers shared by the kernels of xmd_kernels.cu
// and the persistent ensemble kernel (xmd_ensemble.cu): minimum image, warp
// and block reductions, the thermostat chain update, cycle springs, the
// extended-range arithmetic of the exchange recursions, the exchange spring
// gradients, trap forces, and the FP32 pair and phase arithmetic of the
// mixed form.  Everything here is inline device code or a constant.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstddef>
#include <cstdint>
#include <type_traits>

#include "xmd_ewald_tables.h"
#include "xmd_kernels.cuh"

namespace xk {

#define FULL 0xffffffffu

__device__ inline size_t dtri(int n) { return (size_t)n * (n - 1) / 2; }

// Nearest image of a difference a in a box of side L: md_simulation_x.c:70-81
// with md_periodic_image_count_x (:858-865) shift a + L/2 into [0, L] by
// whole boxes and subtract L/2 again; a - L rint(a/L) is the same image in
// three FP64 operations instead of eight (ties at exactly L/2 aside, the
// results differ in the last bits only).
__device__ inline double min_image(double a, double L, double invL) { return fma(-L, rint(a * invL), a); }

__device__ inline double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  return v;
}
__device__ inline double warp_min(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    double t = __shfl_xor_sync(FULL, v, o);
    v = t < v ? t : v;
  }
  return v;
}

// block-wide reductions; buf needs 33 doubles and must not be reused by the
// caller until one more __syncthreads() has passed.
__device__ inline double block_sum(double v, double *buf) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) buf[w] = v;
  __syncthreads();
  if (w == 0) {
    double t = lane < nw ? buf[lane] : 0.0;
    t = warp_sum(t);
    if (lane == 0) buf[32] = t;
  }
  __syncthreads();
  return buf[32];
}
__device__ inline double block_min(double v, double init, double *buf) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_min(v);
  if (lane == 0) buf[w] = v;
  __syncthreads();
  if (w == 0) {
    double t = lane < nw ? buf[lane] : init;
    t = warp_min(t);
    if (lane == 0) buf[32] = t < init ? t : init;
  }
  __syncthreads();
  return buf[32];
}

// Thermostat update of one chain.  v[], F[], mass[] are the chain's DOFs
// (ndof of them, counted as cfv DOFs in the kinetic term); half = 1 is
// md_update_nhc_VV3_1_x (kick, chain, drift, chain), half = 2 is
// md_update_nhc_VV3_2_x (kick, chain).
template <int L>
struct ChainState {
  double th[L], vt[L], Q[L];
  double iQ[L];  // 1/Q (one-DOF chains): multiplications instead of FP64 divisions
};

// md_simulation_x.c:599-613; INV: divide by multiplying with the stored 1/Q
// (a double division is a multi-instruction sequence on the slow FP64 pipe)
template <int L, bool INV = false>
__device__ inline void chain_forces(const ChainState<L> &c, double kin, double cfv, double kT,
                                    double *nhf) {
  nhf[0] = INV ? (kin - cfv * kT) * c.iQ[0] : (kin - cfv * kT) / c.Q[0];
#pragma unroll
  for (int j = 1; j < L; ++j) {
    const double num = c.Q[j - 1] * c.vt[j - 1] * c.vt[j - 1] - kT;
    nhf[j] = INV ? num * c.iQ[j] : num / c.Q[j];
  }
}


// exp(r) 2^62 for |r| < 1/2 on the integer pipe: the Taylor series through
// r^13/13! by Horner's rule on 64-bit fixed-point numbers, the terms from r^8
// on, 1 + r/9 (1 + r/10 (...)) times r^8/8!, with 32 bits (their rounding and
// the first omitted term are below 1e-17 of the result for |r| <= 0.35, a
// tenth of a double's half ulp).  About 110 integer instructions, where
// thirteen FP64 multiply-adds hold the FP64 pipe for 830 cycles a warp.
__device__ __forceinline__ long long exp_q62(double r) {
  const long long b = __double_as_longlong(r);
  const int sh = (int)((b >> 52) & 0x7ff) - 1011;  // |r| = sig 2^(sh - 64)
  const long long sig = (b & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
  long long R = sh >= 0 ? sig << min(sh, 10) : sig >> min(-sh, 63);
  R = b < 0 ? -R : R;  // r 2^64
  const int r32 = (int)(R >> 32);
  constexpr unsigned ONE = 1u << 30;
  unsigned t = ONE + __mulhi(r32, (int)__umulhi(ONE, 330382099u));  // 2^32 / 13
  t = ONE + __mulhi(r32, (int)__umulhi(t, 357913941u));             // 2^32 / 12
  t = ONE + __mulhi(r32, (int)__umulhi(t, 390451572u));
  t = ONE + __mulhi(r32, (int)__umulhi(t, 429496729u));
  t = ONE + __mulhi(r32, (int)__umulhi(t, 477218588u));  // 2^32 / 9
  constexpr unsigned long long C8 = 114377133393536ULL;  // 2^62 / 8!
  long long p = (long long)__umul64hi(C8 << 16, (unsigned long long)t << 18);
  p = 915017067148291LL + __mul64hi(R, p);  // 2^62 / 7!
  p = 6405119470038039LL + __mul64hi(R, p);
  p = 38430716820228233LL + __mul64hi(R, p);
  p = 192153584101141163LL + __mul64hi(R, p);
  p = 768614336404564651LL + __mul64hi(R, p);
  p = (1LL << 61) + __mul64hi(R, p);
  p = (1LL << 62) + __mul64hi(R, p);
  return (1LL << 62) + __mul64hi(R, p);
}
// p 2^-62 rounded to a double, 2^60 <= p < 2^63
__device__ __forceinline__ double q62_double(long long p) {
  const int z = __clzll(p);  // 1..3
  const unsigned long long m = ((unsigned long long)p << (z - 1)) + (1ULL << 9);  // half an ulp of bit 10 added
  return __longlong_as_double((long long)((m >> 10) + ((unsigned long long)(1023 - z) << 52)));
}

// exp(x) for the thermostat factors exp(-h v_eta / 4) and exp(-h v_eta / 2):
// on the integer pipe for |x| < 1/4, the usual case with a small step,
// otherwise exp().  The range test reads the bit pattern, off the FP64 pipe.
__device__ inline double nhc_exp(double x) {
  if ((__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFLL) < 0x3FD0000000000000LL)  // |x| < 2^-2
    return q62_double(exp_q62(x));
  return exp(x);
}

template <int L>
__device__ inline void chain_odd(ChainState<L> &c, double h, const double *nhf) {
  constexpr int M2 = L / 2;
  // exp(-h x / 2) is taken as exp(-h x / 4)^2 (one FP64 exp instead of two,
  // equal to rounding); the last member has no successor, both factors are 1
#pragma unroll
  for (int j = 1; j <= M2; ++j) {
    if (j == M2) {
      c.vt[2 * j - 1] = c.vt[2 * j - 1] + 0.5 * h * nhf[2 * j - 1];
    } else {
      const double e = nhc_exp(-0.25 * h * c.vt[2 * j]);
      c.vt[2 * j - 1] = c.vt[2 * j - 1] * (e * e) + 0.5 * h * nhf[2 * j - 1] * e;
    }
  }
}

template <int D>
__device__ inline double spring2(Geo g, const double *x, int ja, int la, int jb, int lb,
                                 int image) {
  double s = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    double t = x[sidx(ja, d, la, D, g.Ns)] - x[sidx(jb, d, lb, D, g.Ns)];
    if (image) t = min_image(t, g.box[d], g.inv_box[d]);
    s += t * t;
  }
  return s;
}

// spring between bead P of particle a and bead 1 of particle b (0-based),
// weighted by the mass of the bead-P end as in the reference.
template <int D>
__device__ inline double link(Geo g, const double *x, const double *m, double w2, int a, int b,
                              int image) {
  const int jP = g.P - 1;
  return 0.5 * m[(size_t)jP * g.Ns + a] * w2 * spring2<D>(g, x, jP, a, 0, b, image);
}

// exclusive prefix sums out[c] = in[0] + ... + in[c-1] (c = 0..n) by the
// block, in a fixed order (contiguous runs per thread, then the run totals
// scanned over the block): every block that calls it gets the same numbers
__device__ inline void block_exclusive_prefix(const double *__restrict__ in, int n, double *out) {
  __shared__ double wsum[32];
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int a = min(n, (int)threadIdx.x * per), b = min(n, a + per);
  double run = 0.0;
  for (int c = a; c < b; ++c) run += in[c];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double inc = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(FULL, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  if (w == 0) {
    double v = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(FULL, v, o);
      if (lane >= o) v += t;
    }
    wsum[lane] = v;
  }
  __syncthreads();
  double pre = (w > 0 ? wsum[w - 1] : 0.0) + (inc - run);
  for (int c = a; c < b; ++c) {
    out[c] = pre;
    pre += in[c];
  }
  if (threadIdx.x == blockDim.x - 1) out[n] = pre;
}

// One DOF of the fast-chain thermostat step (slot s = (j D + d) Ns + l,
// l < N): md_update_nhc_VV3_1_x (half 1) or _VV3_2_x (half 2) for the DOF
// and its own chain.
template <int D, int L>
__device__ inline void nhc_slot(const Geo &g, int half, size_t s, int l, double *__restrict__ x,
                                double *__restrict__ v, double *__restrict__ f, const double *__restrict__ fex,
                                const double *__restrict__ m, double *__restrict__ th, double *__restrict__ vt,
                                const double *__restrict__ Q, const double *__restrict__ iQ, double kT, double h) {
  const size_t S = g.slots();
  const int j = (int)(s / ((size_t)D * g.Ns));
  constexpr int M2 = L / 2;
  ChainState<L> c;
#pragma unroll
  for (int i = 0; i < L; ++i) {
    c.th[i] = th[i * S + s];
    c.vt[i] = vt[i * S + s];
    c.Q[i] = Q[i * S + s];
    c.iQ[i] = iQ[i * S + s];
  }
  const double mass = m[(size_t)j * g.Ns + l];
  double vv = v[s];
  double F = f[s];
  if (fex) {  // the pending exchange forces, as add_into would add them
    F += fex[s];
    f[s] = F;
  }
  double nhf[L];
  if (half == 1) chain_forces<L, true>(c, mass * vv * vv, 1.0, kT, nhf);
  // thermostatted half kick: md_simulation_x.c:674-678
  const double ek = nhc_exp(-0.25 * h * c.vt[0]);
  vv = vv * (ek * ek) + 0.5 * h * F * ek;
#pragma unroll
  for (int k = 1; k <= M2; ++k) c.th[2 * k - 2] = c.th[2 * k - 2] + h * c.vt[2 * k - 2] / 2;
  if (half == 2) chain_forces<L, true>(c, mass * vv * vv, 1.0, kT, nhf);
  chain_odd<L>(c, h, nhf);
  if (half == 1) {
    x[s] = x[s] + h * vv;  // drift: md_simulation_x.c:684-689
#pragma unroll
    for (int k = 1; k <= M2; ++k) c.th[2 * k - 1] = c.th[2 * k - 1] + h * c.vt[2 * k - 1];
    chain_forces<L, true>(c, mass * vv * vv, 1.0, kT, nhf);
#pragma unroll
    for (int k = 1; k <= M2; ++k)
      {
        const double e = nhc_exp(-0.5 * h * c.vt[2 * k - 1]);
        c.vt[2 * k - 2] = c.vt[2 * k - 2] * (e * e) + h * nhf[2 * k - 2] * e;
      }
  }
  v[s] = vv;
#pragma unroll
  for (int i = 0; i < L; ++i) {
    th[i * S + s] = c.th[i];
    vt[i * S + s] = c.vt[i];
  }
}



// ln 2 split so that e * LN2_HI is exact for |e| < 2^21 (32 significant bits)
constexpr double LN2_HI = 0.6931471803691238, LN2_LO = 1.9082149292705877e-10;
constexpr double LOG2E = 1.4426950408889634;

struct Ext {
  double m;  // mantissa (0 or a normal number of moderate size)
  int e;     // value = m * 2^e
};

// exp(x) for any finite x as 2^e exp(r), |r| <= ln2/2: exp(r) 2^62 from the
// integer pipe, the reduction in FP64.  The series reads r's bits, so an x that
// is infinite or no number is told by its own exponent, EXP_BAD; from 2^30 on e
// is held to +-2^29.
constexpr int EXP_BAD = 0x7fffffff;
__device__ __forceinline__ long long exp_reduced(double x, int &e) {
  constexpr double MAGIC = 6755399441055744.0;  // 1.5 2^52: adding rounds to an integer, in the low word
  const double tq = fma(x, LOG2E, MAGIC), q = tq - MAGIC;
  double r = fma(-q, LN2_HI, x);
  r = fma(-q, LN2_LO, r);
  const int hi = __double2hiint(x) & 0x7fffffff;
  e = __double2loint(tq);
  if (hi >= 0x41d00000)  // |x| >= 2^30
    e = hi >= 0x7ff00000 ? EXP_BAD : x < 0 ? -(1 << 29) : 1 << 29;
  return exp_q62(r);
}
__device__ inline Ext ext_exp(double x) {
  Ext w;
  w.m = q62_double(exp_reduced(x, w.e));
  if (w.e == EXP_BAD) w = {x - x, 0};  // (not a number)
  return w;
}

// exp(x) as ext_exp forms it, the power of two put into the exponent field by
// integer arithmetic; results near or beyond the ends of the normal range
// (|x| > 700) and anything that is no finite number are left to exp()
__device__ inline double exp_fast(double x) {
  int e;
  const double m = q62_double(exp_reduced(x, e));
  if (e <= -1020 || e >= 1020) return exp(x);
  return __longlong_as_double(__double_as_longlong(m) + ((long long)e << 52));
}

// m * 2^d for d <= 0 (0 once the result would drop below the subnormals)
__device__ inline double scale_down(double m, int d) {
  if (d >= -1022) return m * __longlong_as_double((long long)(d + 1023) << 52);
  if (d < -1100) return 0.0;
  return m * 0x1p-1022 * __longlong_as_double((long long)(d + 1022 + 1023) << 52);
}

// acc += t in extended range
__device__ inline void ext_add(double &am, int &ae, double tm, int te) {
  if (tm == 0.0) return;
  if (am == 0.0) {
    am = tm;
    ae = te;
  } else if (te > ae) {
    am = scale_down(am, ae - te) + tm;
    ae = te;
  } else {
    am += scale_down(tm, te - ae);
  }
}

__device__ inline void ext_norm(double &m, int &e) {
  if (m == 0.0) return;
  int k;
  m = frexp(m, &k);
  e += k;
}

// ---- extended range on the integer pipe --------------------------------
// A non-negative number m 2^(e-62) with a 62-bit integer mantissa (2^61 <= m
// < 2^62, or m = 0 with e = XI_NONE): nine bits more than a double's, and no
// FP64 instruction, which on GB300 holds its pipe for 64 cycles a warp.  The
// unsigned solves and the diagonal blocks' inverses work on these: a product or
// a sum of two drops less than 2^-60 of its value, a warp's sum rounds to 2^-57
// of its largest term.  G is within 3 to 5e-16 of 128-bit recursions' (N = 512 and
// 1000; 5 to 8e-16 when warp sums dropped five bits of every lane, 7e-15 in FP64
// with sums of 57 bits).
// A number that is none (from an infinite or NaN energy) is one of exponent
// XI_BAD: products hold exponents to it, sums take the largest, so that whatever
// contains it has an exponent above XI_TOP, which no number reaches (weights
// are at most xi^N), and becomes NaN where it leaves these forms; a zero times it
// is a zero still, whose exponent stays far below any number's.
struct XI {
  long long m;
  int e;
};
constexpr int XI_NONE = -(1 << 30) + (1 << 25), XI_BAD = 1 << 28, XI_TOP = 1 << 26;

// v 2^e of a non-negative double v
__device__ __forceinline__ XI xi_from(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)(b >> 52);
  XI r{((b & 0xFFFFFFFFFFFFFLL) | (1LL << 52)) << 9, e + ex - 1022};
  if (ex == 0) r = {0, XI_NONE};
  return r;
}
// exp(x)
__device__ __forceinline__ XI xi_exp(double x) {
  int e;
  const long long p = exp_reduced(x, e);  // 0.70 .. 1.42 times 2^62
  if (e >= XI_BAD || e <= -(1 << 29)) return {1LL << 61, min(e, XI_BAD)};
  return p >= (1LL << 62) ? XI{p >> 1, e + 1} : XI{p, e};
}
// rounded to a double (to zero below 2^-1074; e up to 1024, or above XI_TOP)
__device__ __forceinline__ double xi_double(XI a) {
  if (a.e > XI_TOP) return __longlong_as_double(0x7ff8000000000000LL);
  const bool low = a.e < -1020;
  const int e = low ? a.e + 200 : a.e;
  if (a.m == 0 || e < -1020) return 0.0;
  const double v = __longlong_as_double(((a.m + 256) >> 9) + ((long long)(e + 1021) << 52));
  return low ? v * 0x1p-200 : v;
}
// ln of a non-zero number: y = logf of the mantissa taken to [0.7, 1.42), then
// one Newton step against exp on the integer pipe; a handful of FP64
// instructions where log() takes about sixty
__device__ __forceinline__ double xi_log(XI a) {
  const bool up = a.m < 0x2D413CCCFE779800LL;  // sqrt(1/2) 2^62: double the mantissa
  const unsigned long long f = (unsigned long long)a.m << (up ? 2 : 1);  // mantissa 2^63
  const int e = up ? a.e - 1 : a.e;
  const float y = logf((float)(unsigned)(f >> 32) * 0x1p-31f);
  const unsigned long long p = (unsigned long long)exp_q62(-(double)y);  // e^-y 2^62
  const long long z = (long long)__umul64hi(f, p << 1) - (1LL << 62);    // (m e^-y - 1) 2^62, about 1e-7
  const double d = (double)z * 0x1p-62;
  return fma((double)e, LN2_HI, fma((double)e, LN2_LO, fma(-0.5 * d, d, d)) + (double)y);
}
__device__ __forceinline__ XI xi_mul(XI a, XI b) {
  XI r{(long long)__umul64hi((unsigned long long)a.m << 2, (unsigned long long)b.m), __viaddmin_s32(a.e, b.e, XI_BAD)};
  if (r.m < (1LL << 61)) r.m <<= 1, r.e -= 1;
  return r;
}
__device__ __forceinline__ XI xi_add(XI a, XI b) {
  XI r;
  r.e = a.e > b.e ? a.e : b.e;
  r.m = (a.m >> min(r.e - a.e, 63)) + (b.m >> min(r.e - b.e, 63));
  if (r.m >= (1LL << 62)) r.m >>= 1, r.e += 1;
  return r;
}
__device__ __forceinline__ XI xi_shfl(XI a, int src) {
  return {__shfl_sync(FULL, a.m, src), __shfl_sync(FULL, a.e, src)};
}
// the warp's sum in every lane: aligned to the largest exponent, in parts of 21,
// 21 and 20 bits (a warp-wide integer reduction is one 32-bit instruction), and
// rounded once, to a 2^-57th of the largest term (32 terms need five bits more)
__device__ __forceinline__ XI xi_warp_sum(XI a) {
  const int em = __reduce_max_sync(FULL, a.e);
  const long long q = a.m >> min(em - a.e, 63);
  const unsigned p0 = __reduce_add_sync(FULL, (unsigned)q & 0x1fffffu);
  const unsigned p1 = __reduce_add_sync(FULL, (unsigned)(q >> 21) & 0x1fffffu);
  const unsigned p2 = __reduce_add_sync(FULL, (unsigned)(q >> 42));
  const long long low = (long long)p0 + ((long long)p1 << 21);
  const long long t = ((long long)p2 << 37) + ((low + 16) >> 5);  // below 2^62
  if (t == 0) return {0, XI_NONE};
  const int sh = __clzll(t) - 2;
  return {t << sh, em + 5 - sh};
}

// packed lower triangle: row i (1..N), column j (0..i-1) at tri(i) + j
__device__ inline size_t moff(int i, int j) { return (size_t)i * (i - 1) / 2 + j; }

// Both weight triangles in one launch: block (row, direction), threads
// along the row.  Forward row n: M_{n,j} = exp(-beta ENk[n][n-j] + (n-j-1)
// ln xi - ln n); backward row i <-> u = N-i+1, column j <-> l = N-j:
// exp(-beta ENk[l][i-j] + (i-j-1) ln xi - ln l).  ln xi and the table
// lnn[l] = ln l come from the host.
// sgn = -1 gives the weights of a negative xi' (|xi'| in vi and lnvi): the
// mantissa of every term with odd k - 1 changes sign.
// both = 1 (first = 0, both directions): the two triangles hold the same
// numbers, M_{l,l-k} = M'_{N-l+k,N-l}, so block l takes row l of ENk and
// writes each weight into both (one exponential per entry).
// INT: the mantissas are XI's 62-bit integers (unsigned weights), else doubles.
template <bool INT>
__device__ inline void weights_row(int N, double beta, double vi, double lnvi, const double *__restrict__ ENk,
                                   const double *__restrict__ lnn, double *__restrict__ Mf, int *__restrict__ Ef,
                                   double *__restrict__ Mb, int *__restrict__ Eb, int first, int sgn, int both,
                                   int row, int dir, int t0, int nt) {
  double *Mm = dir ? Mb : Mf;
  int *Me = dir ? Eb : Ef;
  for (int j = t0; j < row; j += nt) {
    const int k = row - j;
    const int l = dir ? N - j : row;
    const bool on = vi != 0.0 || k == 1;
    const double x = on ? -beta * ENk[dtri(l) + k - 1] + (k - 1) * lnvi - lnn[l] : 0.0;
    double m;
    int e;
    if (INT) {
      const XI w = on ? xi_exp(x) : XI{0, XI_NONE};
      m = __longlong_as_double(w.m);
      e = w.e;
    } else {
      const Ext w = on ? ext_exp(x) : Ext{0.0, 0};
      m = sgn < 0 && ((k - 1) & 1) ? -w.m : w.m;
      e = w.e;
    }
    Mm[moff(row, j)] = m;
    Me[moff(row, j)] = e;
    if (both) {
      Mb[moff(N - row + k, N - row)] = m;
      Eb[moff(N - row + k, N - row)] = e;
    }
  }
}

// X_0 = 1, X_i = sum_{j<i} M_{i,j} X_j (i = 1..N); out_i = -ln(X_i)/beta written
// to out[i] (forward) or out[N-i] (backward).  One block, 16 warps.
constexpr int TS_WARPS = 16, TS_CHUNK = 32;

// v * 2^d for a non-negative double v and d <= 0, by integer arithmetic on
// the exponent field (the FP64 pipe is the scarce resource); results below
// the normal range are flushed to 0 (they are below 2^-1021 of the sum
// they enter)
__device__ inline double scale2(double v, int d) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)((b >> 52) & 0x7ff);
  const long long r = b + ((long long)d << 52);
  return __longlong_as_double((ex == 0 || ex + d <= 0) ? 0LL : r);  // selects, no branch
}

// normalise a non-negative extended value to a mantissa in [0.5, 1)
__device__ inline void norm2(double &m, int &e) {
  const long long b = __double_as_longlong(m);
  const int ex = (int)((b >> 52) & 0x7ff);
  const bool z = ex == 0;  // zero (values here are never subnormal) stays zero
  e = z ? e : e + ex - 1022;
  m = __longlong_as_double(z ? 0LL : ((b & ~(0x7ffLL << 52)) | (1022LL << 52)));
}

// Block b solves direction first + b (0 forward, 1 backward) with the
// weights (Mm[dir], Me[dir]) into out[dir]: launched with two blocks, the
// forward and backward recursions run side by side on two SMs.
struct TriJob {
  const double *Mm[2];
  const int *Me[2];
  double *out[2];
  double *sign;  // optional: sign of X_i (signed weights), forward direction only
  // unsigned weights, [chunk][32][32] XI mantissas and exponents each: the
  // inverses B of the diagonal blocks, and W = B U with U the chunk's weights
  // against the chunk before it
  double *Bm[2];
  int *Be[2];
  double *Wm[2];
  int *We[2];
  double *Sm[2];  // partial sums of the cluster solve of very long systems
  // optional: the unknowns X_0..X_N as XI (unsigned solves) and, last, 1/X_N,
  // kept for the connection probabilities
  long long *Xm[2];
  int *Xe[2];
};

// Extended-range dot product of row i of the weights with the unknowns over
// columns [j0, j1), reduced over the warp: (am, E) with value am 2^E.  One
// pass: each lane keeps a running (am, E) and rescales when a larger term
// exponent arrives; loads are issued four columns per lane at a time.  Zero
// weights (xi = 0 beyond k = 1) are skipped by their bit pattern.  E is
// EXT_NONE while a lane has no term.
constexpr int EXT_NONE = -2147483647;

// Warp sums of extended-range terms are taken in 64-bit fixed point on the
// integer pipe: a warp-wide FP64 add holds GB300's FP64 pipe for many cycles,
// and a five-level reduction of doubles cost more than the dot products
// around it.  fx(v, d, FB): v * 2^d (d <= 0) as a signed integer with FB
// fractional bits, built from the bit pattern (truncated); the caller keeps
// 32 |v| 2^FB below 2^63.
__device__ inline long long fx(double v, int d, int FB) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)((b >> 52) & 0x7ff);
  const long long sig = (b & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
  const int sh = ex - 1075 + FB + d;
  const long long q = sh >= 0 ? (sig << sh) : (sh > -63 ? (sig >> -sh) : 0LL);
  return ex == 0 ? 0LL : (b < 0 ? -q : q);
}
// q * 2^-FB as a double (truncated to 53 bits), by integer arithmetic
__device__ inline double fx_to_double(long long q, int FB) {
  if (q == 0) return 0.0;
  const bool neg = q < 0;
  const unsigned long long u = neg ? (unsigned long long)(-q) : (unsigned long long)q;
  const int top = 63 - __clzll((long long)u);
  const unsigned long long m = top > 52 ? (u >> (top - 52)) : (u << (52 - top));
  const long long bits = ((long long)(neg ? 1 : 0) << 63) | ((long long)(top - FB + 1023) << 52) |
                         (long long)(m & 0xFFFFFFFFFFFFFULL);
  return __longlong_as_double(bits);
}
__device__ inline long long warp_sum_ll(long long q) {
#pragma unroll
  for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(FULL, q, o);
  return q;
}
// warp sum of arbitrary finite doubles on the integer pipe: every lane's
// value in 57-bit fixed point relative to the largest lane's binade, summed
// exactly, rounded once (truncation) to 53 bits; the result reaches every lane
__device__ inline double warp_sum_fx(double v) {
  const int ex = (int)((__double_as_longlong(v) >> 52) & 0x7ff);
  int em = ex;
#pragma unroll
  for (int o = 16; o; o >>= 1) em = max(em, __shfl_xor_sync(FULL, em, o));
  if (em == 0) return 0.0;  // all zero (subnormals do not occur in these sums)
  const long long q = warp_sum_ll(fx(v, 1022 - em, 57));
  if (q == 0) return 0.0;
  const double r = fx_to_double(q, 57);  // value 2^(1022 - em) too large
  return __longlong_as_double(__double_as_longlong(r) + ((long long)(em - 1022) << 52));
}

constexpr int XD_SLOTS = 4;  // columns per lane per pass (loads in flight against L2 latency)
__device__ inline void ext_dot(const double *__restrict__ mr, const int *__restrict__ er, const double *Xm,
                               const int *Xe, int j0, int j1, int lane, double &am_out, int &E_out) {
  double am = 0.0;
  int E = EXT_NONE;
  for (int jb = j0 + lane; jb - lane < j1; jb += 32 * XD_SLOTS) {
    double mv[XD_SLOTS], xv[XD_SLOTS];
    int ev[XD_SLOTS], xe[XD_SLOTS];
#pragma unroll
    for (int u = 0; u < XD_SLOTS; ++u) {
      const int j = jb + 32 * u;
      const bool ok = j < j1;
      mv[u] = ok ? mr[j] : 0.0;
      ev[u] = ok ? er[j] : 0;
      xv[u] = ok ? Xm[j] : 0.0;
      xe[u] = ok ? Xe[j] : 0;
    }
#pragma unroll
    for (int u = 0; u < XD_SLOTS; ++u) {
      if (jb - lane + 32 * u >= j1) break;  // warp-uniform: no lane has this slot
      const bool nz = __double_as_longlong(mv[u]) != 0;
      const int te = ev[u] + xe[u];
      const int ne = (nz && (E == EXT_NONE || te > E)) ? te : E;
      const double a2 = scale2(am, E == EXT_NONE ? 0 : E - ne);
      const double t2 = fma(mv[u], scale2(xv[u], nz ? te - ne : 0), a2);
      am = nz ? t2 : am;
      E = ne;
    }
  }
  // each lane's sum normalised to a mantissa below 1, so that 57 fractional
  // bits keep the 32-lane sum below 2^62 and resolve it to 2^-51 of itself
  if (E != EXT_NONE) norm2(am, E);
  if (__double_as_longlong(am) == 0) E = EXT_NONE;
  int Em = E;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const int oe = __shfl_xor_sync(FULL, Em, o);
    Em = (Em == EXT_NONE || (oe != EXT_NONE && oe > Em)) ? oe : Em;
  }
  const long long q = warp_sum_ll(E == EXT_NONE ? 0LL : fx(am, E - Em, 57));
  am_out = fx_to_double(q, 57);
  E_out = Em;
}

// (pm, pe) += (am, E), both non-negative extended-range values; normalised
__device__ inline void ext_acc(double &pm, int &pe, double am, int E) {
  if (__double_as_longlong(am) != 0 && E != EXT_NONE) {
    if (__double_as_longlong(pm) == 0) {
      pm = am;
      pe = E;
    } else {
      const int mx = pe > E ? pe : E;
      pm = scale2(pm, pe - mx) + scale2(am, E - mx);
      pe = mx;
    }
  }
  norm2(pm, pe);
}

// The chunks of TS_CHUNK rows are solved in order by warp 0.  Row i's sum
// over the unknowns of earlier chunks is split: the part over all but the
// previous chunk is computed by warps 1.. while warp 0 is still solving that
// previous chunk (so it costs no time on the sequential path); the previous
// chunk's 32 columns are added by all warps between the two solves.  The
// weights the sequential steps need (the chunk's own triangle and the
// 32 x 32 block of the previous chunk's columns) are staged in shared memory
// by warps 1.. one chunk ahead, so the sequential path reads no global memory.
constexpr int TS_LD = TS_CHUNK + 1;  // padded row of the staged blocks

// (sum, E) of the warp's non-negative extended terms (pm, pe), nz marking
// lanes with a term; E = EXT_NONE when none has
__device__ inline void ext_warp_sum(bool nz, double pm, int pe, double &sum, int &E) {
  if (nz) norm2(pm, pe);  // mantissa below 1 (see ext_dot)
  int Em = nz ? pe : EXT_NONE;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const int oe = __shfl_xor_sync(FULL, Em, o);
    Em = (Em == EXT_NONE || (oe != EXT_NONE && oe > Em)) ? oe : Em;
  }
  sum = fx_to_double(warp_sum_ll(nz ? fx(pm, pe - Em, 57) : 0LL), 57);
  E = Em;
}

// weight M_{i,j} of direction dir (0 forward, 1 backward) from ENk, the same
// number weights_row stores
__device__ inline XI weight_at(int N, double beta, double vi, double lnvi, const double *__restrict__ ENk,
                               const double *__restrict__ lnn, int dir, int i, int j) {
  const int k = i - j, l = dir ? N - j : i;
  if (vi == 0.0 && k != 1) return {0, XI_NONE};
  return xi_exp(-beta * ENk[dtri(l) + k - 1] + (k - 1) * lnvi - lnn[l]);
}

// One column of B(c) = (I - A)^-1 or W(c) = (I - A)^-1 U for direction dir,
// by a warp: the forward substitution from right-hand side b (lane r holds row
// r; a unit vector, or U's column).  The chunk's block A[r][t] =
// M_{i0+r, i0+t} (t < r) is staged in Am/Ae as XI (zero elsewhere).  Step t
// takes the finished row t to the later rows: one shuffle and one integer
// multiply-add a step, where a sum over the lanes for each row took ten
// shuffles and FP64 products.
__device__ __forceinline__ XI block_solve_column(XI b, int t0, int rows, const long long (*Am)[TS_LD],
                                                 const int (*Ae)[TS_LD]) {
  const int lane = threadIdx.x & 31;
  for (int t = t0; t + 1 < rows; ++t) {
    const XI x = xi_shfl(b, t);
    if (lane > t) b = xi_add(b, xi_mul({Am[lane][t], Ae[lane][t]}, x));
  }
  return b;
}
__device__ inline void block_inv_column(int N, const TriJob &job, int dir, int c, int s,
                                        const long long (*Am)[TS_LD], const int (*Ae)[TS_LD]) {
  const int lane = threadIdx.x & 31;
  const XI b = block_solve_column(lane == s ? XI{1LL << 61, 1} : XI{0, XI_NONE}, s, min(TS_CHUNK, N - c * TS_CHUNK),
                                  Am, Ae);
  const size_t o = (size_t)c * TS_CHUNK * TS_CHUNK + lane * TS_CHUNK + s;
  ((long long *)job.Bm[dir])[o] = b.m;
  job.Be[dir][o] = b.e;
}

// one column of W(c) likewise, c >= 1
__device__ inline void block_w_column(int N, double beta, double vi, double lnvi, const double *__restrict__ ENk,
                                      const double *__restrict__ lnn, const TriJob &job, int dir, int c, int s,
                                      const long long (*Am)[TS_LD], const int (*Ae)[TS_LD]) {
  const int lane = threadIdx.x & 31, i0 = 1 + c * TS_CHUNK;
  XI u{0, XI_NONE};
  if (i0 + lane <= N) u = weight_at(N, beta, vi, lnvi, ENk, lnn, dir, i0 + lane, i0 - TS_CHUNK + s);
  u = block_solve_column(u, 0, min(TS_CHUNK, N - c * TS_CHUNK), Am, Ae);
  const size_t o = (size_t)c * TS_CHUNK * TS_CHUNK + lane * TS_CHUNK + s;
  ((long long *)job.Wm[dir])[o] = u.m;
  job.We[dir][o] = u.e;
}

// gradient of the two springs at bead (ja, la) towards (jn, ln) and (jp, lp):
// m w2 (x - x_n) + m w2 (x - x_p), md_pimd_x.c:2344-2367
template <int D>
__device__ inline void grad2(Geo g, const double *x, double mw2, int ja, int la, int jn, int ln,
                             int jp, int lp, int image, double *gr) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const double xa = x[sidx(ja, d, la, D, g.Ns)];
    double a = xa - x[sidx(jn, d, ln, D, g.Ns)];
    double c = xa - x[sidx(jp, d, lp, D, g.Ns)];
    if (image) {
      a = min_image(a, g.box[d], g.inv_box[d]);
      c = min_image(c, g.box[d], g.inv_box[d]);
    }
    gr[d] = mw2 * a + mw2 * c;
  }
}

__device__ inline double trap_f(const TrapPrm &p, int d, double xv) {
  if (p.kind == TRAP_HARMONIC) return -p.w * p.w * (xv - p.c[d]);
  if (p.kind == TRAP_NEG_HARMONIC) return -(-p.w * p.w * (xv - p.c[d]));
  return -p.w2[d] * p.w2[d] * (xv - p.c[d]);
}

// a column's nx and its largest kept |nz| share the int4's x field
__host__ __device__ inline int col_nx(const int4 &c) { return c.x & 255; }
__host__ __device__ inline int col_nz(const int4 &c) { return c.x >> 8; }

struct Kahan {
  float s = 0.f, c = 0.f;
  __device__ inline void add(float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ inline double value() const { return (double)s - (double)c; }
};

// double-float accumulator: hi + lo with error-free TwoSum per addition
struct DF {
  float hi = 0.f, lo = 0.f;
  __device__ inline void add(float v) {
    const float s = hi + v;
    const float bp = s - hi;
    const float e = (hi - (s - bp)) + (v - bp);
    hi = s;
    lo += e;
  }
  __device__ inline double value() const { return (double)hi + (double)lo; }
};

// Real-space images farther than EW32_XCUT / alpha are left out of the FP32
// form: there h(x) = erfc(x) + 2x exp(-x^2)/sqrt(pi) < 1e-5, and for the
// electron gas at alpha L = 5.6 the dropped images change the largest force
// component by 4e-8 of itself (against 2e-12 at 4.6 and the FP32 form's own
// 6e-6 from rounding the positions), while the images per pair fall from
// 2.32 to 1.11.
constexpr float EW32_XCUT = 3.6f;

// The approximate unit's operations without the code around them for
// subnormal numbers, which cannot matter here: 1/R^3 overflows for such an R^2,
// and the other arguments are within [1, 3] and above -19.
__device__ __forceinline__ float rsqrt_ftz(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float rcp_ftz(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float ex2_ftz(float v) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// h(alpha R) / R^3 in FP32 without tables: h(x) = exp(-x^2) (2x/sqrt(pi) +
// erfcx(x)), erfcx(x) ~ t P(t), t = 1/(1 + x/2) (fit in xmd_ewald_tables.h,
// relative error 2e-8 on [0, 4.7]); 1/R from rsqrt, exp from ex2
__device__ __forceinline__ float ew_h32(float R2, float alpha) {
  const float cc[EW32_DEG + 1] = EW32_ERFCX_INIT;
  const float ri = rsqrt_ftz(R2);
  const float x = alpha * (R2 * ri);
  const float t = rcp_ftz(fmaf((float)EW32_C, x, 1.f));
  float q = cc[EW32_DEG];
#pragma unroll
  for (int k = EW32_DEG - 1; k >= 0; --k) q = fmaf(q, t, cc[k]);
  const float e = ex2_ftz(-x * x * 1.4426950408889634f);
  return e * fmaf(x, 1.1283791670955126f, q * t) * (ri * ri * ri);
}

// constants of the FP32 pair kernel, prepared on the host so that the
// kernel issues no FP64 instruction (on GB300 the FP64 pipe is 58x slower
// and also serves conversions and divisions of doubles)
struct P32 {
  float L[3], iL[3];
  float igs2, gpre;  // Gaussian: 1/s^2 and (g / (pi s^2)) (2 / s^2)
  float qs;          // Coulomb / Ewald strength
  float alpha, rc2;  // Ewald: splitting, FP32 cut-off squared
  int kmax;          // Ewald: 0 = 8-image search, else |k_d| <= kmax
  int single;        // Ewald: no image shifted along two axes lies inside the cut-off
  int nsum;          // Ewald: the reference's image cube |n_d| <= nsum
  int uniform;       // all beads of the system have one mass (1/m = im0)
  float im0;
};

// the FP32 pair kernel's constants for a system and potential (host)
P32 make_p32(const Geo &g, const PairPrm &p);

template <int D, int KIND, bool SINGLE>
__device__ inline void pair_eval32(const P32 &q, const float *dx, float *F) {
  if (KIND == PAIR_GAUSSIAN || KIND == PAIR_PERIODIC_GAUSSIAN) {
    float t[D], r2 = 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      t[d] = dx[d];
      if (KIND == PAIR_PERIODIC_GAUSSIAN) t[d] = t[d] - q.L[d] * rintf(t[d] * q.iL[d]);
      r2 = fmaf(t[d], t[d], r2);
    }
    const float mult = q.gpre * __expf(-r2 * q.igs2);
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] = mult * t[d];
  } else if (KIND == PAIR_COULOMB || KIND == PAIR_PERIODIC_COULOMB) {
    float t[D], r2 = 0.f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      t[d] = dx[d];
      if (KIND == PAIR_PERIODIC_COULOMB) t[d] = t[d] - q.L[d] * rintf(t[d] * q.iL[d]);
      r2 = fmaf(t[d], t[d], r2);
    }
    const float ri = rsqrtf(r2);
    const float mult = q.qs * ri * ri * ri;
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] = mult * t[d];
  } else if (KIND == PAIR_EWALD_REAL) {
    // Minimum image m = dx - r L (r = rint(dx/L)); images t = m - k L.
    // Images beyond rc32 (alpha rc32 <= EW32_XCUT) are left out.  When rc32
    // is at most the smallest box length only the 8 images with k_d in
    // {0, sign(m_d)} can lie inside it (any other has a component of length
    // >= L); otherwise all 27 with |k_d| <= kmax are tried.  The reference's
    // cube |r_d + k_d| <= nsum matters only for nsum < 2.
    float m[3], sg[3], r[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      r[d] = rintf(dx[d] * q.iL[d]);
      m[d] = fmaf(-r[d], q.L[d], dx[d]);
      sg[d] = m[d] < 0.f ? -1.f : 1.f;
    }
    const float ns = (float)q.nsum;
    float F0 = 0.f, F1 = 0.f, F2 = 0.f;
    if (SINGLE) {
      // A component shifted by a box edge is at least half the edge long, so
      // below sqrt(L_d^2 + L_e^2) / 2 (0.707 L; alpha L > 5.1) only the minimum
      // image and the three shifted along one axis are left: the first is
      // evaluated by every lane together, the others, 0.23 a pair at alpha L =
      // 5.6, as many rounds as the busiest lane has (see k_pair_tiles32 for
      // what this gives).
      const float R0 = fmaf(m[2], m[2], fmaf(m[1], m[1], m[0] * m[0]));
      bool in = R0 < q.rc2;
      unsigned mask = 0u;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (R0 + q.L[d] * fmaf(-2.f, fabsf(m[d]), q.L[d]) < q.rc2) mask |= 1u << d;
      if (q.nsum < 2) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (!(fabsf(r[d]) <= ns)) in = false, mask &= 1u << d;
          if (!(fabsf(r[d] + sg[d]) <= ns)) mask &= ~(1u << d);
        }
      }
      const float mult0 = in ? ew_h32(R0, q.alpha) : 0.f;
      F0 = m[0] * mult0;
      F1 = m[1] * mult0;
      F2 = m[2] * mult0;
      while (mask) {
        const unsigned low = mask & (0u - mask);
        mask ^= low;
        const float t0 = (low & 1) ? m[0] - copysignf(q.L[0], m[0]) : m[0];
        const float t1 = (low & 2) ? m[1] - copysignf(q.L[1], m[1]) : m[1];
        const float t2 = (low & 4) ? m[2] - copysignf(q.L[2], m[2]) : m[2];
        const float mult = ew_h32(fmaf(t2, t2, fmaf(t1, t1, t0 * t0)), q.alpha);
        F0 = fmaf(t0, mult, F0);
        F1 = fmaf(t1, mult, F1);
        F2 = fmaf(t2, mult, F2);
      }
    } else if (q.kmax == 0) {
      // With a_d = |m_d| the shifted component has length L_d - a_d, so an
      // image's squared distance is |m|^2 plus dl_d = L_d (L_d - 2 a_d) for
      // each shifted axis: the 8 candidates are tested with a few adds.  The
      // accepted ones (2.3 per pair on average at alpha L = 5.6) are then
      // evaluated lowest bit first, so the warp runs as many rounds as its
      // busiest lane has images instead of one round per candidate.
      const float R0 = fmaf(m[2], m[2], fmaf(m[1], m[1], m[0] * m[0]));
      float dl[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) dl[d] = q.L[d] * fmaf(-2.f, fabsf(m[d]), q.L[d]);
      unsigned mask = 0u;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float R2 = R0 + ((c & 1) ? dl[0] : 0.f) + ((c & 2) ? dl[1] : 0.f) + ((c & 4) ? dl[2] : 0.f);
        bool ok = R2 < q.rc2;
        if (q.nsum < 2)
          ok = ok && fabsf(r[0] + ((c & 1) ? sg[0] : 0.f)) <= ns && fabsf(r[1] + ((c & 2) ? sg[1] : 0.f)) <= ns &&
               fabsf(r[2] + ((c & 4) ? sg[2] : 0.f)) <= ns;
        mask |= ok ? 1u << c : 0u;
      }
      while (mask) {
        const int c = __ffs(mask) - 1;
        mask &= mask - 1;
        const float t0 = (c & 1) ? fmaf(-sg[0], q.L[0], m[0]) : m[0];
        const float t1 = (c & 2) ? fmaf(-sg[1], q.L[1], m[1]) : m[1];
        const float t2 = (c & 4) ? fmaf(-sg[2], q.L[2], m[2]) : m[2];
        const float R2 = fmaf(t2, t2, fmaf(t1, t1, t0 * t0));
        const float mult = ew_h32(R2, q.alpha);
        F0 = fmaf(t0, mult, F0);
        F1 = fmaf(t1, mult, F1);
        F2 = fmaf(t2, mult, F2);
      }
    } else {
      for (int k0 = -q.kmax; k0 <= q.kmax; ++k0) {
        const float f0 = (float)k0;
        if (fabsf(r[0] + f0) > ns) continue;
        const float t0 = fmaf(-f0, q.L[0], m[0]);
        for (int k1 = -q.kmax; k1 <= q.kmax; ++k1) {
          const float f1 = (float)k1;
          if (fabsf(r[1] + f1) > ns) continue;
          const float t1 = fmaf(-f1, q.L[1], m[1]);
          for (int k2 = -q.kmax; k2 <= q.kmax; ++k2) {
            const float f2 = (float)k2;
            if (fabsf(r[2] + f2) > ns) continue;
            const float t2 = fmaf(-f2, q.L[2], m[2]);
            const float R2 = fmaf(t2, t2, fmaf(t1, t1, t0 * t0));
            if (R2 >= q.rc2) continue;
            const float mult = ew_h32(R2, q.alpha);
            F0 = fmaf(t0, mult, F0);
            F1 = fmaf(t1, mult, F1);
            F2 = fmaf(t2, mult, F2);
          }
        }
      }
    }
    F[0] = q.qs * F0;
    if (D > 1) F[1] = q.qs * F1;
    if (D > 2) F[2] = q.qs * F2;
  }
}

__device__ inline float2 cmulf(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}


// the solve's job for weight scratch rs_f / rs_b (rec_scratch_doubles(N)
// each) and outputs VBN / tmpV (host)
TriJob tri_job(int N, double *rs_f, double *rs_b, double *VBN, double *tmpV);

// out[] = -ln X / beta and the kept unknowns of a solve from X_0..X_N, entries
// i0, i0 + step, ...
__device__ inline void tri_solve_out(int N, double beta, const TriJob &job, int backward, const long long *Xm,
                                     const int *Xe, int i0, int step) {
  double *__restrict__ out = job.out[backward];
  const double ib = 1.0 / beta;
  for (int i = i0; i <= N; i += step) {
    const XI x{Xm[i], Xe[i]};
    if (i > 0) {
      // the quotient, corrected by its residual
      const double lnx = x.e > XI_TOP ? xi_double(x) : xi_log(x), q = -lnx * ib;
      out[backward ? N - i : i] = fma(-fma(q, beta, lnx), ib, q);
    } else {
      out[backward ? N : 0] = 0.0;
    }
    if (job.Xm[backward]) {
      job.Xm[backward][i] = x.m;
      job.Xe[backward][i] = x.e;
      if (i == N) {
        // 1 / (m 2^(e-62)) = (1 / mantissa in [1/2, 1)) 2^-e
        XI v = xi_from(1.0 / __longlong_as_double(((x.m + 256) >> 9) + (1021LL << 52)), -x.e);
        if (x.e > XI_TOP) v.e = XI_BAD;
        job.Xm[backward][N + 1] = v.m;
        job.Xe[backward][N + 1] = v.e;
      }
    }
  }
}

// row i's sum over the unknowns 0 <= j < j1, by the warp
__device__ inline XI xi_dot(const long long *__restrict__ Mm, const int *__restrict__ Me, const long long *Xm,
                            const int *Xe, int i, int j1, int lane) {
  XI a{0, XI_NONE};
  for (int j = lane; j < j1; j += 32) a = xi_add(a, xi_mul({Mm[moff(i, j)], Me[moff(i, j)]}, {Xm[j], Xe[j]}));
  return xi_warp_sum(a);
}

// a + m x for a normalised x; the product may miss one bit of 62
__device__ __forceinline__ XI xi_mul_add(XI a, XI m, XI x) {
  return xi_add(a, {(long long)__umul64hi((unsigned long long)x.m << 2, (unsigned long long)m.m),
                    __viaddmin_s32(m.e, x.e, XI_BAD)});
}

// The block solve of direction `backward` by the calling thread block (any
// whole number of warps; rows of a chunk go round-robin over the warps, each
// row's sums inside one warp, so the result does not depend on the count).
// viaw: by the products W, X_c = B_c P_c + W_c X_{c-1}, with the sums in the order
// of the cluster solve (k_tri_solve_c), whose bits it then gives.
// sh: (8 + 4) (N + 1 + 2 TS_CHUNK + 2 TS_CHUNK TS_LD) bytes of shared memory.
__device__ inline void tri_solve_b_dev(int N, double beta, const TriJob &job, int backward, double *sh,
                                       bool viaw = false) {
  const long long *__restrict__ Mm = (const long long *)job.Mm[backward];
  const int *__restrict__ Me = job.Me[backward];
  const long long *__restrict__ Bgm = (const long long *)job.Bm[backward];
  const int *__restrict__ Bge = job.Be[backward];
  const long long *__restrict__ Wgm = (const long long *)job.Wm[backward];
  const int *__restrict__ Wge = job.We[backward];
  long long *Um = (long long *)sh;          // [TS_CHUNK][TS_LD] next chunk vs the chunk before it (viaw: its W block)
  long long *Bsm = Um + TS_CHUNK * TS_LD;   // [TS_CHUNK][TS_LD] the chunk's B block
  long long *Pm = Bsm + TS_CHUNK * TS_LD;   // [TS_CHUNK] sums over the unknowns before the previous chunk
  long long *Rm = Pm + TS_CHUNK;            // [TS_CHUNK] right-hand sides of the chunk
  long long *Xm = Rm + TS_CHUNK;            // N+1
  int *Ue = (int *)(Xm + N + 1);            // [TS_CHUNK][TS_LD]
  int *Bse = Ue + TS_CHUNK * TS_LD;         // [TS_CHUNK][TS_LD]
  int *Pe = Bse + TS_CHUNK * TS_LD;         // [TS_CHUNK]
  int *Re = Pe + TS_CHUNK;                  // [TS_CHUNK]
  int *Xe = Re + TS_CHUNK;                  // N+1
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // stage chunk n0's B block and its rows' weights against columns c0..c0+31, or W
  auto stage = [&](int n0, int c0) {
    const int cc = (n0 - 1) / TS_CHUNK;
    for (int q = threadIdx.x; q < TS_CHUNK * TS_CHUNK; q += blockDim.x) {
      const int r = q / TS_CHUNK, k = q % TS_CHUNK, i = n0 + r, o = r * TS_LD + k;
      const bool in = i <= N;
      const bool un = in && c0 >= 0;
      const size_t uo = viaw ? (size_t)cc * TS_CHUNK * TS_CHUNK + q : un ? moff(i, c0 + k) : 0;
      Um[o] = un ? (viaw ? Wgm : Mm)[uo] : 0;
      Ue[o] = un ? (viaw ? Wge : Me)[uo] : XI_NONE;
      Bsm[o] = in ? Bgm[(size_t)cc * TS_CHUNK * TS_CHUNK + q] : 0;
      Bse[o] = in ? Bge[(size_t)cc * TS_CHUNK * TS_CHUNK + q] : XI_NONE;
    }
  };
  if (threadIdx.x == 0) {
    Xm[0] = 1LL << 61;  // X_0 = 1
    Xe[0] = 1;
  }
  stage(1, -1);
  // chunk 0: its rows against column 0
  for (int r = threadIdx.x; r < TS_CHUNK; r += blockDim.x) {
    Pm[r] = 1 + r <= N ? Mm[moff(1 + r, 0)] : 0;
    Pe[r] = 1 + r <= N ? Me[moff(1 + r, 0)] : XI_NONE;
  }
  __syncthreads();
  for (int i0 = 1, c = 0; i0 <= N; i0 += TS_CHUNK, ++c) {
    // U: right-hand sides (viaw: B_c P_c)
    for (int r = w; r < TS_CHUNK; r += nw) {
      const int o = r * TS_LD + lane;
      XI p{Pm[r], Pe[r]};
      if (viaw) {
        p = xi_warp_sum(xi_mul({Bsm[o], Bse[o]}, {Pm[lane], Pe[lane]}));
      } else if (c > 0) {
        const int col = i0 - TS_CHUNK + lane;
        p = xi_add(p, xi_warp_sum(xi_mul({Um[o], Ue[o]}, {Xm[col], Xe[col]})));
      }
      if (lane == 0) {
        Rm[r] = p.m;
        Re[r] = p.e;
      }
    }
    __syncthreads();
    // B: the chunk's unknowns
    for (int r = w; r < TS_CHUNK; r += nw) {
      const int i = i0 + r, o = r * TS_LD + lane, col = i0 - TS_CHUNK + lane;
      if (i > N) break;  // warp-uniform
      XI x;
      if (!viaw)
        x = xi_warp_sum(xi_mul({Bsm[o], Bse[o]}, {Rm[lane], Re[lane]}));
      else if (c > 0)
        x = xi_add({Rm[r], Re[r]}, xi_warp_sum(xi_mul({Um[o], Ue[o]}, {Xm[col], Xe[col]})));
      else
        x = {Rm[r], Re[r]};
      if (lane == 0) {
        Xm[i] = x.m;
        Xe[i] = x.e;
      }
    }
    __syncthreads();
    // next chunk: its weights against this chunk, its B block, and its rows'
    // sums over the unknowns before this chunk
    const int n0 = i0 + TS_CHUNK;
    if (n0 > N) break;
    stage(n0, i0);
    for (int r = w; r < TS_CHUNK; r += nw) {
      const int i = n0 + r;
      XI p{0, XI_NONE};
      if (i <= N && !viaw) {
        p = xi_dot(Mm, Me, Xm, Xe, i, i0, lane);
      } else if (i <= N) {
        if (lane == 0) p = {Mm[moff(i, 0)], Me[moff(i, 0)]};
        for (int j = 1 + lane; j < i0; j += TS_CHUNK) {
          const size_t q = moff(i, j);
          p = xi_mul_add(p, {Mm[q], Me[q]}, {Xm[j], Xe[j]});
        }
        p = xi_warp_sum(p);
      }
      if (lane == 0) {
        Pm[r] = p.m;
        Pe[r] = p.e;
      }
    }
    __syncthreads();
  }
  tri_solve_out(N, beta, job, backward, Xm, Xe, threadIdx.x, blockDim.x);
}


// particle l's interior springs, E_l^(1) and the increment gl[l]: one warp
template <int D>
__device__ inline void eint_particle(const Geo &g, const double *__restrict__ x, const double *__restrict__ m,
                                     double w2, int image, double *Eint, double *ENk, double *gl, int l, int lane) {
  double res = 0;
  for (int j = lane; j + 1 < g.P; j += 32)
    res += 0.5 * m[(size_t)j * g.Ns + l] * w2 * spring2<D>(g, x, j, l, j + 1, l, image);
  res = warp_sum(res);
  // lane 0: the closing spring of l (E_l^(1)); lane 1: the link to l+1 (the
  // increment of the prefix sums), both in one pass
  if (lane < 2) {
    const int b = lane == 0 ? l : (l + 1 < g.N ? l + 1 : l);
    const double lk = link<D>(g, x, m, w2, l, b, image);
    if (lane == 0) {
      Eint[l] = res;
      ENk[dtri(l + 1)] = res + lk;
    } else if (l + 1 < g.N) {
      gl[l] = res + lk;
    }
  }
}

// E_l^(k) (1-based row l, cycle length k >= 2) from the prefix sums G
template <int D>
__device__ inline void enk_entry(const Geo &g, const double *__restrict__ x, const double *__restrict__ m, double w2,
                                 int image, const double *__restrict__ Eint, const double *G, double *__restrict__ ENk,
                                 int l, int k) {
  ENk[dtri(l) + k - 1] = Eint[l - 1] + ((G[l - 1] - G[l - k]) + link<D>(g, x, m, w2, l - 1, l - k, image));
}

// the ring springs' force on interior bead j (1..P-2) of particle l, as the
// acceleration the step stores in f: the reference divides the gradient
// m w2 (2x - x_n - x_p) (md_pimd_x.c:2344-2367) by the bead's mass m, which
// cancels, so w2 (x - x_n) + w2 (x - x_p) is taken directly (equal to
// rounding; no FP64 division, the GPU's slowest FP64 operation)
template <int D>
__device__ inline void spring_interior_bead(const Geo &g, const double *__restrict__ x, double w2, int image,
                                            double *__restrict__ f, int j, int l) {
  double gr[D];
  grad2<D>(g, x, w2, j, l, j + 1, l, j - 1, l, image, gr);
#pragma unroll
  for (int d = 0; d < D; ++d) f[sidx(j, d, l, D, g.Ns)] = -gr[d];
}

// X'_{N-l} / X_N of row l (1-based) of G
__device__ inline XI g_ext_row(int N, const TriJob &job, int l) {
  return xi_mul({job.Xm[1][N - l], job.Xe[1][N - l]}, {job.Xm[0][N + 1], job.Xe[0][N + 1]});
}
// G[l][j] (1-based) = M_{l,j-1} X_{j-1} X'_{N-l} / X_N, and 1 - X_l X'_{N-l} / X_N
// for j = l + 1, from the recursions' numbers; q: X'_{N-l} / X_N
__device__ inline double g_ext_elem(const TriJob &job, XI q, int l, int j) {
  if (j > l + 1) return 0.0;
  if (j == l + 1) return 1 - xi_double(xi_mul({job.Xm[0][l], job.Xe[0][l]}, q));
  const size_t o = moff(l, j - 1);
  const XI w{((const long long *)job.Mm[0])[o], job.Me[0][o]};
  return xi_double(xi_mul(xi_mul(w, {job.Xm[0][j - 1], job.Xe[0][j - 1]}), q));
}

// FP32 phase factor e^{2 pi i x/L} of slot t (D = 3): the fraction of x/L in
// FP64 (exact), the sine and cosine of the reduced angle in FP32.  The sums
// form the harmonics where they use them (phase32_next): a slice's eleven rows
// a coordinate are ten times the reads, and cost more than nine products.
__device__ inline float2 phase32_slot(const Geo &g, const double *__restrict__ x, size_t t) {
  const int l = (int)(t % g.Ns), d = (int)(t / g.Ns) % 3;
  float s1 = 0.f, c1 = 1.f;
  if (l < g.N) {
    double u = x[t] * g.inv_box[d];
    u -= rint(u);  // in [-1/2, 1/2]
    sincospif((float)(2.0 * u), &s1, &c1);
  }
  return make_float2(c1, s1);
}
__device__ __forceinline__ float2 phase32_next(float2 e, float2 e1) {
  return make_float2(fmaf(e.x, e1.x, __fmul_rn(-e.y, e1.y)), fmaf(e.x, e1.y, __fmul_rn(e.y, e1.x)));
}

constexpr int P32_UNROLL = 2;  // steps of the single-shift Ewald tiles evaluated side by side

// tile job wi (slice wi / jobs, tile pair I <= J) of the FP32 pair forces,
// one warp: per-tile sums into out (see k_pair_tiles32)
template <int D, int KIND>
__device__ inline void pair_tile32_job(const Geo &g, const P32 &q, const float *__restrict__ x,
                                       const float *__restrict__ im, float *__restrict__ out, int T, int jobs, int wi,
                                       int lane) {
  const int j = wi / jobs;
  int job = wi % jobs, I = 0;
  while (job >= T - I) {
    job -= T - I;
    ++I;
  }
  const int J = I + job;
  const int a = I * 32 + lane, b0 = J * 32 + lane;
  const bool va = a < g.N, vb = b0 < g.N;
  float xa[D], xb[D], fa[D], fb[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    xa[d] = va ? x[sidx(j, d, a, D, g.Ns)] : 0.f;
    xb[d] = vb ? x[sidx(j, d, b0, D, g.Ns)] : 0.f;
    fa[d] = fb[d] = 0.f;
  }
  // a diagonal tile visits each pair once in 16 steps (the last by half the lanes)
  const bool diag = I == J;
  const int src = (lane + 1) & 31, s0 = diag ? 1 : 0, s1 = diag ? 16 : 31;
  const float ima = !q.uniform && va ? im[(size_t)j * g.Ns + a] : 1.f;
  float imb = !q.uniform && vb ? im[(size_t)j * g.Ns + b0] : 1.f;
  if (diag) {
#pragma unroll
    for (int d = 0; d < D; ++d) xb[d] = __shfl_sync(FULL, xb[d], src);
    imb = __shfl_sync(FULL, imb, src);
  }
  auto step = [&](int s, auto single) {
    const int bi = J * 32 + ((lane + s) & 31);
    if (va && bi < g.N && !(diag && s == 16 && lane >= 16)) {
      float dx[D], F[D];
#pragma unroll
      for (int d = 0; d < D; ++d) dx[d] = xa[d] - xb[d];
      pair_eval32<D, KIND, decltype(single)::value>(q, dx, F);
      // the reference divides by the mass of the higher-index particle; with
      // one mass for all the sums are multiplied by its inverse
      if (!q.uniform) {
        const float inv = a > bi ? ima : imb;
#pragma unroll
        for (int d = 0; d < D; ++d) F[d] *= inv;
      }
#pragma unroll
      for (int d = 0; d < D; ++d) {
        fa[d] += F[d];
        fb[d] -= F[d];
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xb[d] = __shfl_sync(FULL, xb[d], src);
      fb[d] = __shfl_sync(FULL, fb[d], src);
    }
    if (!q.uniform) imb = __shfl_sync(FULL, imb, src);
  };
  if (KIND == PAIR_EWALD_REAL && q.single) {
#pragma unroll P32_UNROLL
    for (int s = s0; s <= s1; ++s) step(s, std::true_type{});
  } else {
    for (int s = s0; s <= s1; ++s) step(s, std::false_type{});
  }
  const int home = (lane - s1 - 1) & 31;  // b's sums are s1 + 1 lanes away
#pragma unroll
  for (int d = 0; d < D; ++d) {
    fb[d] = __shfl_sync(FULL, fb[d], home);
    if (q.uniform) fa[d] *= q.im0, fb[d] *= q.im0;
  }
  if (I == J) {
    if (va) {
#pragma unroll
      for (int d = 0; d < D; ++d) out[(((size_t)I * g.P + j) * D + d) * g.Ns + a] = fa[d] + fb[d];
    }
  } else {
    if (va) {
#pragma unroll
      for (int d = 0; d < D; ++d) out[(((size_t)J * g.P + j) * D + d) * g.Ns + a] = fa[d];
    }
    if (vb) {
#pragma unroll
      for (int d = 0; d < D; ++d) out[(((size_t)I * g.P + j) * D + d) * g.Ns + b0] = fb[d];
    }
  }
}

// ---- exchange spring forces of the end beads -----------------------------
// Bead 1 of l meets bead P of every q with weight G[q][l], bead P of l meets
// bead 1 of every q with weight G[l][q] (md_pimd_x.c:2674-2717): the same
// spring vector c = xP_l - x1_q with the weight G[l][q] serves bead P of l and,
// negated, bead 1 of q, so a 32 x 32 tile of the lower triangle serves both.  A
// warp takes one of `parts` equal parts of a tile's rows l, a column q a lane
// (the weights' rows and G's are then read and written whole sectors at a
// time), forms G there and stores it (FROM_G: reads it).  The columns' sums stay
// in the lanes; the rows' are added across them by halving exchanges, R rows
// of (weight, weighted vector) at once: one addition a value instead of five.
// Bound by the FP64 pipe where there are many tiles, by its latency where few.
// The ring's own spring at an end bead does not depend on the partner: it is
// weighted once, by the summed weights.  G is zero above the superdiagonal; an
// element (l, l+1) in the next tile's first column goes to a corner entry.
// scr: columns [T * parts][D+1][Ns] (slot: row tile and part), rows [T][D+1][Ns]
// (slot: column tile), then corners [T][D+1].
__host__ __device__ inline int exch_parts(int N) { return N <= 128 ? 8 : 4; }
__host__ __device__ inline int exch_jobs(int N) {
  const int T = (N + 31) / 32;
  return T * (T + 1) / 2 * exch_parts(N);
}
template <int D, int R, bool FROM_G>
__device__ inline void exch_tile_rows(const Geo &g, const double *__restrict__ x, int image, const TriJob &tj,
                                      double *__restrict__ G, double *__restrict__ scr, int LT, int QT, int part,
                                      int parts, int lane) {
  constexpr int CP = D == 1 ? 2 : 4, NV = R * CP;  // padded components of a row's sums; their number
  static_assert(NV <= 32, "a row batch's sums fill at most one value a lane");
  const int N = g.N, T = (N + 31) / 32, q = QT * 32 + lane;
  const bool vq = q < N;
  double x1[D], a1[D + 1];
#pragma unroll
  for (int d = 0; d < D; ++d) x1[d] = vq ? x[sidx(0, d, q, D, g.Ns)] : 0.0;
#pragma unroll
  for (int d = 0; d <= D; ++d) a1[d] = 0.0;
  double *rows = scr + (size_t)T * parts * (D + 1) * g.Ns;
  for (int l0 = LT * 32 + part * 32 / parts; l0 < LT * 32 + (part + 1) * 32 / parts; l0 += R) {
    double w[R], v[NV];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int l = l0 + r;
      w[r] = 0.0;
      if (l < N && vq && q <= l + 1)
        w[r] = FROM_G ? G[(size_t)l * N + q] : g_ext_elem(tj, g_ext_row(N, tj, l + 1), l + 1, q + 1);
    }
    if (!FROM_G) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (l0 + r < N && vq && q <= l0 + r + 1) G[(size_t)(l0 + r) * N + q] = w[r];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int l = l0 + r < N ? l0 + r : N - 1;
#pragma unroll
      for (int d = 0; d < CP - 1; ++d) {
        v[r * CP + d] = 0.0;
        if (d < D) {
          double c = x[sidx(g.P - 1, d, l, D, g.Ns)] - x1[d];
          if (image) c = min_image(c, g.box[d], g.inv_box[d]);
          c *= w[r];
          v[r * CP + d] = c;
          a1[d] -= c;
        }
      }
      v[r * CP + CP - 1] = w[r];
      a1[D] += w[r];
    }
#pragma unroll
    for (int h = NV / 2, off = 16; h > 0; h /= 2, off /= 2) {
      const bool up = lane & off;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const double keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
        v[i] = keep + __shfl_xor_sync(FULL, send, off);
      }
    }
#pragma unroll
    for (int off = 16 / NV; off > 0; off /= 2) v[0] += __shfl_xor_sync(FULL, v[0], off);
    const int i = lane / (32 / NV), l = l0 + i / CP, d = i % CP == CP - 1 ? D : i % CP;
    if (lane % (32 / NV) == 0 && l < N && (i % CP == CP - 1 || d < D))
      rows[((size_t)QT * (D + 1) + d) * g.Ns + l] = v[0];
  }
  if (vq) {
#pragma unroll
    for (int d = 0; d <= D; ++d) scr[((size_t)(LT * parts + part) * (D + 1) + d) * g.Ns + q] = a1[d];
  }
  const int l = LT * 32 + 31;
  if (LT == QT && part == 0 && lane == 31 && l + 1 < N) {
    double *o = G + (size_t)l * N + l + 1;
    const double w = FROM_G ? *o : g_ext_elem(tj, g_ext_row(N, tj, l + 1), l + 1, l + 2);
    if (!FROM_G) *o = w;
    double *co = rows + (size_t)T * (D + 1) * g.Ns + (size_t)LT * (D + 1);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      double c = x[sidx(g.P - 1, d, l, D, g.Ns)] - x[sidx(0, d, l + 1, D, g.Ns)];
      if (image) c = min_image(c, g.box[d], g.inv_box[d]);
      co[d] = c * w;
    }
    co[D] = w;
  }
}
template <int D, bool FROM_G>
__device__ inline void exch_tile_job(const Geo &g, const double *__restrict__ x, int image, const TriJob &tj,
                                     double *__restrict__ G, double *__restrict__ scr, int job, int lane) {
  const int parts = exch_parts(g.N), part = job % parts;
  int LT = 0, QT = job / parts;
  while (QT > LT) QT -= ++LT;
  if (parts == 8)
    exch_tile_rows<D, 4, FROM_G>(g, x, image, tj, G, scr, LT, QT, part, parts, lane);
  else
    exch_tile_rows<D, 8, FROM_G>(g, x, image, tj, G, scr, LT, QT, part, parts, lane);
}

// Share y of EX_Y of the sums of an end bead's (side 0 bead 1, side 1 bead P)
// partial entries: of the weighted vectors' coordinate d in .x, of the weights
// in .y.  exch_end_value adds the shares in order; the entries of a long
// system are many and each a trip to L2, so its kernel takes a thread a share.
constexpr int EX_Y = 8;
template <int D>
__device__ inline double2 exch_end_share(const Geo &g, const double *__restrict__ scr, int side, int d, int l, int y) {
  const int T = (g.N + 31) / 32, parts = exch_parts(g.N), t = l / 32;
  const size_t row = (size_t)(D + 1) * g.Ns;
  const double *base = scr + (side ? (size_t)T * parts * row : 0);
  const int a = side ? 0 : t * parts, b = side ? t + 1 : T * parts;
  double2 s = make_double2(0, 0);
#pragma unroll 4
  for (int k = a + y; k < b; k += EX_Y) {
    s.x += base[k * row + (size_t)d * g.Ns + l];
    s.y += base[k * row + (size_t)D * g.Ns + l];
  }
  return s;
}
// the spring vector of end bead `side` (0: bead 1, 1: bead P) along its own
// ring, coordinate d
__device__ inline double exch_own_spring(const Geo &g, const double *__restrict__ x, int image, int side, int d, int l) {
  const int j = side ? g.P - 1 : 0, jn = side ? g.P - 2 : 1;
  const double r = x[sidx(j, d, l, g.D, g.Ns)] - x[sidx(jn, d, l, g.D, g.Ns)];
  return image ? min_image(r, g.box[d], g.inv_box[d]) : r;
}
// the exchange force on the end bead, as the acceleration the step stores
// (the bead's mass cancels, as in spring_interior_bead); r: exch_own_spring
template <int D>
__device__ inline double exch_end_value(const Geo &g, double r, double w2, const double *__restrict__ scr, int side,
                                        int d, int l, const double2 *share, int stride) {
  const int T = (g.N + 31) / 32, t = (l + side) / 32;
  double S = 0, W = 0;
#pragma unroll
  for (int y = 0; y < EX_Y; ++y) {
    S += share[y * stride].x;
    W += share[y * stride].y;
  }
  if (((l + side) & 31) == 0 && t > 0 && l + side < g.N) {
    const double *co = scr + ((size_t)T * (exch_parts(g.N) + 1) * g.Ns + t - 1) * (D + 1);
    S += side ? co[d] : -co[d];
    W += co[D];
  }
  return -w2 * (W * r + S);
}

// ---- FP32 reciprocal sums (mixed form) ------------------------------------
// Both kernels' bodies for a block of SK_W warps, shared with the persistent
// ensemble step, whose results are the same bits: the order of every sum
// depends on N, the columns and SK_W alone.
constexpr int SK_NG = 8;                // harmonics of one structure-factor item
static_assert(SK_NG % 2 == 0, "z factors are read two at a time, 16 bytes aligned");
constexpr int SK_W = 8, SK_T = 32 * SK_W;
constexpr int SK_CH = 128;              // particles staged at a time
constexpr int SK_NC = 4 * SK_NG + 2;    // sums of one item

// staged phase factors of one particle, in float2: z harmonics 1.., x and y
// harmonics 0..; the stride is an odd number of 16-byte units, so that lanes
// writing 16 bytes each of different particles meet different banks
__host__ __device__ inline int sk32_z(int ns) { return (ns + 1) & ~1; }
__host__ __device__ inline int sk32_x(int ns) { return (ns + 2) & ~1; }
__host__ __device__ inline int sk32_stride(int ns) {
  const int s = sk32_z(ns) + 2 * sk32_x(ns);
  return s / 2 % 2 ? s : s + 2;
}
__host__ __device__ inline size_t sk32_smem(int ns) {
  const size_t a = sizeof(float2) * SK_CH * sk32_stride(ns), b = sizeof(float2) * SK_W / 2 * SK_NC * 32;
  return a > b ? a : b;
}

// a + b and a - b of two double-float values, rounded to FP32 (TwoSum of
// the high parts, the low parts added to its error)
__device__ inline float df_sum(const DF &a, const DF &b) {
  const float s = a.hi + b.hi, bp = s - a.hi;
  const float e = (a.hi - (s - bp)) + (b.hi - bp);
  return s + ((e + a.lo) + b.lo);
}
__device__ inline float df_diff(const DF &a, const DF &b) {
  const float s = a.hi - b.hi, bp = s - a.hi;
  const float e = (a.hi - (s - bp)) + (-b.hi - bp);
  return s + ((e + a.lo) - b.lo);
}

// Structure factors of 32 items of slice j and from them their entries of the
// force tables, T[column][0..ns]: W(0), then (A, B) = W(n) +- W(-n) with
// W = c(n) conj(S(n)).  Item i: column i's harmonics nz = 0..SK_NG for
// i < ncol, above that column i - ncol's further ones (the nlong columns that
// have them; columns are sorted longest first).  An item is a lane, the warps
// take every SK_W-th particle: the particle's z factors are then read at one
// address, its x and y factors at different banks, and a column's
// exp(i(x + y)) is formed once for its harmonics.  Each product is added in
// FP32, at most SK_CH / SK_W = 16 particles at a time (an error of ~1e-7 of a
// term, the size of the phase factors' own rounding), each partial sum in
// double-float.  Bound by FP32 issue, four multiply-adds a harmonic, at 60 to
// 70% of the issue slots.  37 us and no tables kernel (8 us) at N = 512, P = 64,
// |n| <= 10, against 72 with a thread per four harmonics of a column, whose
// lanes read scattered rows of staged harmonics; items of 6, 8 and 10 harmonics
// 38, 37 and 42 us (blocks an SM: 3, 2, 2), in the ensemble step 509, 492, 507.
// sh: sk32_smem(ns) bytes; every thread of the block calls.
__device__ inline void sk32_group(const Geo &g, int ns, int ncol, int nlong, const int4 *__restrict__ cols,
                                  const float *__restrict__ coef32, const float2 *__restrict__ ph1,
                                  float4 *__restrict__ T, int j, int group, float2 *sh) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, item = group * 32 + lane;
  const bool live = item < ncol + nlong, more = item >= ncol;
  const int ci = live ? (more ? item - ncol : item) : 0, n0 = more ? SK_NG : 0;
  const int4 c = cols[ci];
  const int top = live ? min(col_nz(c) - n0, SK_NG) : 0;
  const int zs = sk32_z(ns), xs = sk32_x(ns), stride = sk32_stride(ns);
  const int ox = zs + col_nx(c), oy = zs + xs + abs(c.y);
  const float sy = c.y < 0 ? -1.f : 1.f;
  float h[SK_NC], lo[SK_NC];  // s0 (re, im), then per harmonic P (re, im), Q (re, im)
#pragma unroll
  for (int k = 0; k < SK_NC; ++k) h[k] = lo[k] = 0.f;
  auto flush = [&](int k) {
    DF a{h[k], 0.f};
    a.add(lo[k]);
    h[k] = a.hi;
    lo[k] = a.lo;
  };
  // a thread's first factors of a chunk, read while the one before is summed
  constexpr int NQ = (3 * SK_CH + SK_T - 1) / SK_T;
  float2 first[NQ];
  auto fetch = [&](int l0) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int q = tid + k * SK_T, li = l0 + q % SK_CH, d = q / SK_CH;
      if (d < 3 && li < g.N) first[k] = ph1[((size_t)j * 3 + d) * g.Ns + li];
    }
  };
  fetch(0);
  for (int l0 = 0; l0 < g.N; l0 += SK_CH) {
    const int cnt = min(g.N - l0, SK_CH);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const int q = tid + k * SK_T, li = q % SK_CH, d = q / SK_CH;
      if (d >= 3 || li >= cnt) continue;
      const float2 e1 = first[k];
      float2 e = d == 2 ? e1 : make_float2(1.f, 0.f);
      float4 *o = (float4 *)(sh + li * stride + (d == 2 ? 0 : zs + d * xs));
      for (int n = d == 2 ? 1 : 0; n <= ns; n += 2) {
        const float2 f = phase32_next(e, e1);
        *o++ = make_float4(e.x, e.y, f.x, f.y);
        e = phase32_next(f, e1);
      }
    }
    fetch(l0 + SK_CH);
    __syncthreads();
    if (l0 > 0) {
#pragma unroll
      for (int k = 0; k < SK_NC; ++k)
        if (k < 2 + 4 * top) flush(k);
    }
    if (live) {
#pragma unroll 2
      for (int li = w; li < cnt; li += SK_W) {
        const float2 *row = sh + li * stride;
        const float2 ex = row[ox], ey = row[oy];
        const float yi = sy * ey.y;
        const float er = fmaf(ex.x, ey.x, __fmul_rn(-ex.y, yi)), ei = fmaf(ex.x, yi, __fmul_rn(ex.y, ey.x));
        lo[0] = __fadd_rn(lo[0], er);
        lo[1] = __fadd_rn(lo[1], ei);
#pragma unroll
        for (int u = 0; u < SK_NG; u += 2) {
          if (u >= top) break;
          const float4 z = *(const float4 *)(row + n0 + u);
          float *a = lo + 2 + 4 * u;
          a[0] = fmaf(er, z.x, a[0]);
          a[1] = fmaf(ei, z.x, a[1]);
          a[2] = fmaf(er, z.y, a[2]);
          a[3] = fmaf(ei, z.y, a[3]);
          a[4] = fmaf(er, z.z, a[4]);
          a[5] = fmaf(ei, z.z, a[5]);
          a[6] = fmaf(er, z.w, a[6]);
          a[7] = fmaf(ei, z.w, a[7]);
        }
      }
    }
  }
  // the warps' sums meet in shared memory, the upper half's in the lower half's
  // first; warp u mod SK_W finishes harmonic u of each item
  constexpr int HW = SK_W / 2;
  float2 *mine = sh + (w % HW) * SK_NC * 32 + lane;
  __syncthreads();
  if (w >= HW) {
#pragma unroll
    for (int k = 0; k < SK_NC; ++k)
      if (k < 2 + 4 * top) mine[k * 32] = make_float2(h[k], lo[k]);
  }
  __syncthreads();
  if (w < HW) {
#pragma unroll
    for (int k = 0; k < SK_NC; ++k)
      if (k < 2 + 4 * top) {
        const float2 p = mine[k * 32];
        DF a{h[k], lo[k]};
        a.add(p.x);
        mine[k * 32] = make_float2(a.hi, __fadd_rn(a.lo, p.y));
      }
  }
  __syncthreads();
  for (int u = w; u <= top; u += SK_W) {
    if (!live || (more && u == 0)) continue;
    DF v[4];
    const int k0 = u == 0 ? 0 : 4 * u - 2, nk = u == 0 ? 2 : 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= nk) break;
#pragma unroll
      for (int i = 0; i < HW; ++i) {
        const float2 p = sh[(i * SK_NC + k0 + k) * 32 + lane];
        v[k].add(p.x);
        v[k].add(p.y);
      }
    }
    float4 *o = T + ((size_t)j * ncol + ci) * (ns + 1);
    const float *cf = coef32 + c.w - c.z;  // cf[nz], nz >= c.z
    if (u == 0) {
      const float c0 = c.z <= 0 ? cf[0] : 0.f;
      o[0] = make_float4(c0 * (v[0].hi + v[0].lo), -c0 * (v[1].hi + v[1].lo), 0.f, 0.f);
    } else {
      // S(+-n) = (P_r -+ Q_i, P_i +- Q_r)
      const int n = n0 + u;
      const float cp = cf[n], cm = c.z < 0 ? cf[-n] : 0.f;
      const float pr = __fmul_rn(cp, df_diff(v[0], v[3])), pi = __fmul_rn(-cp, df_sum(v[1], v[2]));
      const float mr = __fmul_rn(cm, df_sum(v[0], v[3])), mi = __fmul_rn(-cm, df_diff(v[1], v[2]));
      o[n] = make_float4(__fadd_rn(pr, mr), __fadd_rn(pi, mi), __fsub_rn(pr, mr), __fsub_rn(pi, mi));
      // the forces take harmonics two at a time
      if (n == col_nz(c) && n % 2 && n < ns) o[n + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}
__host__ __device__ inline int sk32_groups(int ncol, int nlong) { return (ncol + nlong + 31) / 32; }

// a column as the forces read it: rows of its x and y factors, nzmax, unused;
// nx, ny, sign of ny
struct RecipCol {
  int ox, oy, nz, pad;
  float fx, fy, sy, pad2;
};
__device__ inline RecipCol recip_col32(int4 c, int ns) {
  return {col_nx(c) * 32, (ns + 1 + abs(c.y)) * 32, col_nz(c), 0, (float)col_nx(c), (float)c.y, c.y < 0 ? -1.f : 1.f, 0.f};
}

// the FP32 pair tiles' partial sums of slot s, in double
__device__ inline double pair_sum32(const Geo &g, const float *__restrict__ part, int T, size_t s) {
  const size_t S = g.slots();
  double acc = 0;
#pragma unroll 4
  for (int t = 0; t < T; ++t) acc += (double)part[(size_t)t * S + s];
  return acc;
}

// Reciprocal forces on 32 particles of slice j, one a lane, by a block of SK_W warps: warp w sums columns w, w + SK_W, ..., so that
// the lanes read each table entry at one address; Kahan sums, the warps' added
// in double-float.  sc, sT: columns (recip_col32) and force tables, of all columns
// or (PARTS, cap < ncol) of cap at a time, a multiple of SK_W, which stage(c0, n)
// brings there; pxy: [2][ns+1][32]
// float2, red: [SK_W][3][32] float2, of these warps alone (red may lie over
// sT).  The real space's tile sums (part, T tiles, pscale) are added here too:
// their loads pass beside other blocks' sums, and the reciprocal forces' own
// trip to f serves both.  NSM: the largest ns.  Bound by FP32 issue, eight multiply-adds a
// harmonic: 36 us at N = 512, P = 64, |n| <= 10, 57 with two threads a particle,
// each on half the columns with its own reads of the tables.
template <int NSM, bool PARTS, class Stage>
__device__ inline void recip_tile32(const Geo &g, int ns, int ncol, int cap, Stage stage, const RecipCol *sc,
                                    const float4 *sT, float2 *pxy, float2 *red, const float2 *__restrict__ ph1,
                                    double scale, double *__restrict__ f, int j, int l0, int w, int lane,
                                    const float *__restrict__ part, int T, double pscale) {
  const int l = min(l0 + lane, g.N - 1);  // lanes past the end repeat the last particle
  const float2 *p1 = ph1 + (size_t)j * 3 * g.Ns + l;
  if (w < 2) {
    const float2 e1 = p1[(size_t)w * g.Ns];
    float2 e = make_float2(1.f, 0.f);
    for (int n = 0; n <= ns; ++n) {
      pxy[(w * (ns + 1) + n) * 32 + lane] = e;
      e = phase32_next(e, e1);
    }
  }
  float2 ez[NSM], nz[NSM];  // e^{i n z}, and n times it
  ez[0] = nz[0] = p1[(size_t)2 * g.Ns];
#pragma unroll
  for (int n = 1; n < NSM; ++n) {
    ez[n] = phase32_next(ez[n - 1], ez[0]);
    nz[n] = make_float2(__fmul_rn((float)(n + 1), ez[n].x), __fmul_rn((float)(n + 1), ez[n].y));
  }
  __syncthreads();
  Kahan F[3];
  auto column = [&](int ci) {
    const RecipCol c = sc[ci];
    const float4 *t = sT + ci * (ns + 1);
    const float2 vx = pxy[c.ox + lane], vy = pxy[c.oy + lane];
    const float yi = c.sy * vy.y;
    const float er = fmaf(vx.x, vy.x, __fmul_rn(-vx.y, yi)), ei = fmaf(vx.x, yi, __fmul_rn(vx.y, vy.x));
    const float4 w0 = t[0];
    float ur = w0.x, ui = w0.y, vr = 0.f, vi = 0.f;
#pragma unroll
    for (int n = 0; n < NSM; ++n) {  // harmonic n + 1; an odd nzmax below ns is followed by a zero entry
      if (n % 2 == 0 ? n >= c.nz : n >= ns) break;
      const float4 ab = t[n + 1];
      ur = fmaf(ez[n].x, ab.x, fmaf(-ez[n].y, ab.w, ur));
      ui = fmaf(ez[n].x, ab.y, fmaf(ez[n].y, ab.z, ui));
      vr = fmaf(nz[n].x, ab.z, fmaf(-nz[n].y, ab.y, vr));
      vi = fmaf(nz[n].x, ab.w, fmaf(nz[n].y, ab.x, vi));
    }
    const float Tm = fmaf(er, ui, __fmul_rn(ei, ur));
    F[0].add(__fmul_rn(c.fx, Tm));
    F[1].add(__fmul_rn(c.fy, Tm));
    F[2].add(fmaf(er, vi, __fmul_rn(ei, vr)));
  };
  if (PARTS && cap < ncol) {
    for (int c0 = 0; c0 < ncol; c0 += cap) {
      const int n = min(cap, ncol - c0);
      if (c0 > 0) __syncthreads();  // the part before is no longer read
      stage(c0, n);
      __syncthreads();
      for (int ci = w; ci < n; ci += SK_W) column(ci);
    }
  } else {
    for (int ci = w; ci < ncol; ci += SK_W) column(ci);
  }
  __syncthreads();  // the tables are no longer read
#pragma unroll
  for (int d = 0; d < 3; ++d) red[(w * 3 + d) * 32 + lane] = make_float2(F[d].s, -F[d].c);
  __syncthreads();
  if (w < 3 && l0 + lane < g.N) {
    DF s;
    for (int i = 0; i < SK_W; ++i) {
      const float2 p = red[(i * 3 + w) * 32 + lane];
      s.add(p.x);
      s.add(p.y);
    }
    const double ib = w == 0 ? g.inv_box[0] : (w == 1 ? g.inv_box[1] : g.inv_box[2]);
    const size_t o = sidx(j, w, l, 3, g.Ns);
    f[o] = (f[o] + scale * s.value() * ib) + pair_sum32(g, part, T, o) * pscale;
  }
}

}  // namespace xk
