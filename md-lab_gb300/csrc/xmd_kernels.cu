// xmd_kernels.cu -- sm_103a kernels of the PIMD force-and-integrate step.
//
// FP64 throughout (the "plain" form that reproduces MD-Lab's _nocl build to
// 1e-10).  On GB300 the FP64 pipe runs at 1/58 of the FP32 rate (measured:
// 1.2 TFLOP/s DFMA), so every kernel is organised to spend as few FP64
// instructions as the reference's arithmetic allows: pair forces use
// Newton's third law with warp-rotation tiles (one evaluation per pair, no
// atomics), the Ewald reciprocal sum goes through per-slice structure factors
// with per-axis phase factors (O(N K) instead of O(N^2 K)), and reductions
// are warp shuffles with a fixed summation order (results are bitwise
// reproducible run to run).
//
// Reference counterparts (MD-Lab file:line) are cited at each kernel.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <string>
#include <vector>

#include "xmd_ewald_tables.h"
#include "xmd_device.cuh"
#include "xmd_kernels.cuh"

namespace xk {

static std::atomic<uint64_t> g_launches{0};
uint64_t launch_count() { return g_launches.load(); }

// ---- live per-kernel timing (CUDA events on the launching stream) ----
static bool g_prof = false;
struct ProfRec {
  const char *name;
  cudaEvent_t a, b;
};
static std::vector<ProfRec> g_prof_recs;

void profile_enable(bool on) { g_prof = on; }
bool profiling() { return g_prof; }

// sums the recorded launches per kernel name: returns "name ms launches;..."
std::string profile_report() {
  std::vector<std::pair<std::string, std::pair<double, int>>> acc;
  for (auto &r : g_prof_recs) {
    cudaEventSynchronize(r.b);
    float ms = 0;
    cudaEventElapsedTime(&ms, r.a, r.b);
    bool found = false;
    for (auto &e : acc)
      if (e.first == r.name) {
        e.second.first += ms;
        e.second.second += 1;
        found = true;
      }
    if (!found) acc.push_back({r.name, {ms, 1}});
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  g_prof_recs.clear();
  std::string out;
  char buf[256];
  for (auto &e : acc) {
    snprintf(buf, sizeof buf, "%s %.6f %d;", e.first.c_str(), e.second.first, e.second.second);
    out += buf;
  }
  return out;
}

Prof::Prof(const char *n, cudaStream_t s) : name(n), st(s) {
  if (!g_prof) return;
  cudaStreamCaptureStatus cs;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) return;
  cudaEventCreate(&a);
  cudaEventRecord(a, st);
}
Prof::~Prof() {
  if (!a) return;
  cudaEvent_t b;
  cudaEventCreate(&b);
  cudaEventRecord(b, st);
  g_prof_recs.push_back({name, a, b});
}

cudaError_t launched() {
  g_launches.fetch_add(1);
  return cudaGetLastError();
}

static inline int cdiv(size_t a, int b) { return (int)((a + b - 1) / b); }

#define DISPATCH_D(Dv, ...)                 \
  switch (Dv) {                             \
    case 1: {                               \
      constexpr int D = 1;                  \
      __VA_ARGS__;                          \
    } break;                                \
    case 2: {                               \
      constexpr int D = 2;                  \
      __VA_ARGS__;                          \
    } break;                                \
    case 3: {                               \
      constexpr int D = 3;                  \
      __VA_ARGS__;                          \
    } break;                                \
    default:                                \
      return cudaErrorInvalidValue;         \
  }

// ===================================================================
// layout conversion
// ===================================================================

// The records are moved through shared memory a block at a time, so that
// the reads (writes) of the record array are contiguous 8-byte words across
// the block: the array may be the page-locked host array itself, read or
// written by the kernel over the CPU-GPU link.
// n 8-byte words from src to dst, both 16-byte aligned, by the block's
// threads in 16-byte pieces, several loads in flight a thread (the source or
// destination may be host memory across the CPU-GPU link)
__device__ inline void block_copy_words(double *__restrict__ dst, const double *__restrict__ src, int n, int nthr) {
  const int n2 = n >> 1;
  const double2 *s2 = (const double2 *)src;
  double2 *d2 = (double2 *)dst;
#pragma unroll 4
  for (int q = threadIdx.x; q < n2; q += nthr) d2[q] = s2[q];
  if ((n & 1) && threadIdx.x == 0) dst[n - 1] = src[n - 1];
}

constexpr int CONV_T = 256;  // particle records per block
constexpr int CHAIN_T = 128;  // chain records per block (L <= 8: at most 25.6 KB staged)

template <int D>
// mass_flag (optional) is cleared when a record's mass differs from the
// first record's (bit pattern)
__global__ void __launch_bounds__(CONV_T) k_aos_to_soa(Geo g, const double *__restrict__ aos, double *x, double *v,
                                                       double *f, double *m, int *mass_flag) {
  constexpr int RW = 1 + 3 * D;
  __shared__ __align__(16) double sm[CONV_T * RW];
  const int b0 = blockIdx.x * CONV_T, nb = min(CONV_T, g.N * g.P - b0);
  block_copy_words(sm, aos + (size_t)b0 * RW, nb * RW, CONV_T);
  __syncthreads();
  if ((int)threadIdx.x >= nb) return;
  const int b = b0 + threadIdx.x, l = b / g.P, j = b % g.P;
  const double *r = sm + threadIdx.x * RW;
  if (mass_flag && __double_as_longlong(r[0]) != __double_as_longlong(aos[0])) atomicAnd(mass_flag, 0);
  m[(size_t)j * g.Ns + l] = r[0];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const size_t s = sidx(j, d, l, D, g.Ns);
    x[s] = r[1 + d];
    v[s] = r[1 + D + d];
    f[s] = r[1 + 2 * D + d];
  }
}

template <int D>
__global__ void __launch_bounds__(CONV_T) k_soa_to_aos(Geo g, double *__restrict__ aos, const double *x,
                                                       const double *v, const double *f, const double *m) {
  constexpr int RW = 1 + 3 * D;
  __shared__ __align__(16) double sm[CONV_T * RW];
  const int b0 = blockIdx.x * CONV_T, nb = min(CONV_T, g.N * g.P - b0);
  if ((int)threadIdx.x < nb) {
    const int b = b0 + threadIdx.x, l = b / g.P, j = b % g.P;
    double *r = sm + threadIdx.x * RW;
    r[0] = m[(size_t)j * g.Ns + l];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const size_t s = sidx(j, d, l, D, g.Ns);
      r[1 + d] = x[s];
      r[1 + D + d] = v[s];
      r[1 + 2 * D + d] = f[s];
    }
  }
  __syncthreads();
  block_copy_words(aos + (size_t)b0 * RW, sm, nb * RW, CONV_T);
}

cudaError_t aos_to_soa(const Geo &g, const double *aos, double *x, double *v, double *f,
                       double *m, cudaStream_t st, int *mass_flag) {
  const int n = g.N * g.P;
  {
    XK_PROF("aos_to_soa");
    DISPATCH_D(g.D, k_aos_to_soa<D><<<cdiv(n, CONV_T), CONV_T, 0, st>>>(g, aos, x, v, f, m, mass_flag));
  }
  return XK_LAUNCHED();
}

cudaError_t soa_to_aos(const Geo &g, double *aos, const double *x, const double *v,
                       const double *f, const double *m, cudaStream_t st) {
  const int n = g.N * g.P;
  {
    XK_PROF("soa_to_aos");
    DISPATCH_D(g.D, k_soa_to_aos<D><<<cdiv(n, CONV_T), CONV_T, 0, st>>>(g, aos, x, v, f, m));
  }
  return XK_LAUNCHED();
}

// chain record: int f at offset 0, then theta[L], vtheta[L], Q[L] (doubles)
// starting at offset 8.  Fast chains go to slot order, grouped chains keep
// the chain order.
template <int D>
// f_flag (optional, upload) is cleared when a record's f differs from 1
__global__ void __launch_bounds__(CHAIN_T) k_chains(Geo g, int L, int nf, bool fast, bool to_dev, unsigned char *rec,
                                                   size_t rb, double *th, double *vt, double *Q, const int *cf,
                                                   double *iQ, int all_iq, int *f_flag) {
  // records staged as 8-byte words (rb is a multiple of 8), see k_aos_to_soa;
  // a block's records start 16-byte aligned (CHAIN_T rb is a multiple of 16)
  extern __shared__ __align__(16) double csm[];
  const int rw = (int)(rb / 8);
  const int c0 = blockIdx.x * CHAIN_T, nb = min(CHAIN_T, nf - c0);
  double *words = (double *)(rec + (size_t)c0 * rb);
  if (to_dev) {
    block_copy_words(csm, words, nb * rw, CHAIN_T);
    __syncthreads();
  }
  const int c = c0 + threadIdx.x;
  if ((int)threadIdx.x < nb) {
    size_t slot, stride;
    if (fast) {
      const int b = c / D, d = c % D;
      const int l = b / g.P, j = b % g.P;
      slot = sidx(j, d, l, D, g.Ns);
      stride = g.slots();
    } else {
      slot = c;
      stride = nf;
    }
    double *r = csm + threadIdx.x * rw + 1;
    if (to_dev && f_flag && *(const int *)(csm + threadIdx.x * rw) != 1) atomicAnd(f_flag, 0);
    if (!to_dev) {
      // whole records go back: f (1 for one-DOF chains, else as uploaded), zero padding
      int *fi = (int *)(csm + threadIdx.x * rw);
      fi[0] = fast ? 1 : cf[c];
      fi[1] = 0;
    }
    for (int i = 0; i < L; ++i) {
      if (to_dev) {
        th[i * stride + slot] = r[i];
        vt[i * stride + slot] = r[L + i];
        // 1/Q only where Q changed (a re-upload of the same chains divides
        // nothing)
        const double q = r[2 * L + i];
        if (iQ && (all_iq || q != Q[i * stride + slot])) iQ[i * stride + slot] = q != 0.0 ? 1.0 / q : 0.0;
        Q[i * stride + slot] = q;
      } else {
        r[i] = th[i * stride + slot];
        r[L + i] = vt[i * stride + slot];
        r[2 * L + i] = Q[i * stride + slot];
      }
    }
  }
  if (!to_dev) {
    __syncthreads();
    block_copy_words(words, csm, nb * rw, CHAIN_T);
  }
}

cudaError_t chains_to_dev(const Geo &g, int L, int nf, bool fast, const unsigned char *rec,
                          size_t rb, double *th, double *vt, double *Q, double *iQ, bool all_iq, cudaStream_t st,
                          int *f_flag) {
  {
    XK_PROF("chains");
    DISPATCH_D(g.D, k_chains<D><<<cdiv(nf, CHAIN_T), CHAIN_T, CHAIN_T * rb, st>>>(
                        g, L, nf, fast, true, (unsigned char *)rec, rb, th, vt, Q, nullptr, iQ, all_iq ? 1 : 0,
                        f_flag));
  }
  return XK_LAUNCHED();
}

cudaError_t chains_to_host(const Geo &g, int L, int nf, bool fast, unsigned char *rec, size_t rb,
                           const double *th, const double *vt, const double *Q, const int *cf,
                           cudaStream_t st) {
  if (!fast && !cf) return cudaErrorInvalidValue;
  {
    XK_PROF("chains");
    DISPATCH_D(g.D, k_chains<D><<<cdiv(nf, CHAIN_T), CHAIN_T, CHAIN_T * rb, st>>>(
                        g, L, nf, fast, false, rec, rb, (double *)th, (double *)vt, (double *)Q, cf, nullptr, 0,
                        nullptr));
  }
  return XK_LAUNCHED();
}

// ===================================================================
// Nose-Hoover chains, "VV3" splitting: md_simulation_x.c:599-792
// ===================================================================


template <int D, int L>
__global__ void __launch_bounds__(256) k_nhc_fast(Geo g, int half, double *__restrict__ x,
                                                  double *__restrict__ v,
                                                  double *__restrict__ f, const double *__restrict__ fex,
                                                  const double *__restrict__ m,
                                                  double *__restrict__ th, double *__restrict__ vt,
                                                  const double *__restrict__ Q, const double *__restrict__ iQ,
                                                  double kT, double h) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.slots()) return;
  const int l = (int)(s % g.Ns);
  if (l >= g.N) return;
  nhc_slot<D, L>(g, half, s, l, x, v, f, fex, m, th, vt, Q, iQ, kT, h);
}

// chains over several DOFs (reference numbering dof = bead*D + d,
// bead = l*P + j); one thread per chain, DOFs in the reference's order.
template <int D, int L>
__global__ void k_nhc_grouped(Geo g, int half, int nf, const int *__restrict__ cf,
                              const int *__restrict__ c0, const int *__restrict__ c2,
                              double *__restrict__ x, double *__restrict__ v,
                              const double *__restrict__ f, const double *__restrict__ m,
                              double *__restrict__ th, double *__restrict__ vt,
                              const double *__restrict__ Q, double kT, double h) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  constexpr int M2 = L / 2;
  ChainState<L> c;
#pragma unroll
  for (int k = 0; k < L; ++k) {
    c.th[k] = th[(size_t)k * nf + i];
    c.vt[k] = vt[(size_t)k * nf + i];
    c.Q[k] = Q[(size_t)k * nf + i];
  }
  const int f0 = c0[i], f2 = c2[i];
  const double cfv = cf[i];
  auto slot = [&](int dof) {
    const int b = dof / D, d = dof % D;
    return sidx(b % g.P, d, b / g.P, D, g.Ns);
  };
  auto mass = [&](int dof) {
    const int b = dof / D;
    return m[(size_t)(b % g.P) * g.Ns + b / g.P];
  };
  auto kinetic = [&]() {
    double sum = 0;
    for (int q = 0; q < f2; ++q) {
      const size_t s = slot(f0 + q);
      sum += mass(f0 + q) * v[s] * v[s];
    }
    return sum;
  };
  double nhf[L];
  if (half == 1) chain_forces<L>(c, kinetic(), cfv, kT, nhf);
  const double e2 = nhc_exp(-0.25 * h * c.vt[0]), e1 = e2 * e2;
  for (int q = 0; q < f2; ++q) {
    const size_t s = slot(f0 + q);
    v[s] = v[s] * e1 + 0.5 * h * f[s] * e2;
  }
#pragma unroll
  for (int k = 1; k <= M2; ++k) c.th[2 * k - 2] = c.th[2 * k - 2] + h * c.vt[2 * k - 2] / 2;
  if (half == 2) chain_forces<L>(c, kinetic(), cfv, kT, nhf);
  chain_odd<L>(c, h, nhf);
  if (half == 1) {
    for (int q = 0; q < f2; ++q) {
      const size_t s = slot(f0 + q);
      x[s] = x[s] + h * v[s];
    }
#pragma unroll
    for (int k = 1; k <= M2; ++k) c.th[2 * k - 1] = c.th[2 * k - 1] + h * c.vt[2 * k - 1];
    chain_forces<L>(c, kinetic(), cfv, kT, nhf);
#pragma unroll
    for (int k = 1; k <= M2; ++k)
      {
        const double e = nhc_exp(-0.5 * h * c.vt[2 * k - 1]);
        c.vt[2 * k - 2] = c.vt[2 * k - 2] * (e * e) + h * nhf[2 * k - 2] * e;
      }
  }
#pragma unroll
  for (int k = 0; k < L; ++k) {
    th[(size_t)k * nf + i] = c.th[k];
    vt[(size_t)k * nf + i] = c.vt[k];
  }
}

#define DISPATCH_L(Lv, ...)           \
  switch (Lv) {                       \
    case 2: {                         \
      constexpr int LL = 2;           \
      __VA_ARGS__;                    \
    } break;                          \
    case 4: {                         \
      constexpr int LL = 4;           \
      __VA_ARGS__;                    \
    } break;                          \
    case 6: {                         \
      constexpr int LL = 6;           \
      __VA_ARGS__;                    \
    } break;                          \
    case 8: {                         \
      constexpr int LL = 8;           \
      __VA_ARGS__;                    \
    } break;                          \
    default:                          \
      return cudaErrorInvalidValue;   \
  }

cudaError_t nhc_vv3(const Geo &g, int half, const Chains &c, double *x, double *v,
                    double *f, const double *m, double kT, double h, cudaStream_t st, const double *fex) {
  if (c.fast) {
    const size_t S = g.slots();
    {
      XK_PROF("nhc_fast");
      DISPATCH_D(g.D, DISPATCH_L(c.L, k_nhc_fast<D, LL><<<cdiv(S, 256), 256, 0, st>>>(
                                          g, half, x, v, f, fex, m, c.th, c.vt, c.Q, c.iQ, kT, h)));
    }
  } else {
    if (fex) {
      cudaError_t e = add_into(f, fex, g.slots(), st);
      if (e != cudaSuccess) return e;
    }
    {
      XK_PROF("nhc_grouped");
      DISPATCH_D(g.D, DISPATCH_L(c.L, k_nhc_grouped<D, LL><<<cdiv(c.nf, 128), 128, 0, st>>>(
                                          g, half, c.nf, c.cf, c.c0, c.c2, x, v, f, m, c.th,
                                          c.vt, c.Q, kT, h)));
    }
  }
  return XK_LAUNCHED();
}

// md_simulation_x.c:846-853
__global__ void k_wrap(Geo g, double *x) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.slots()) return;
  if ((int)(s % g.Ns) >= g.N) return;
  const int d = (int)((s / g.Ns) % g.D);
  const double L = g.box[d];
  double a = x[s];
  if (a < 0)
    a += L;
  else if (a > L)
    a -= L;
  x[s] = a;
}

cudaError_t wrap_box(const Geo &g, double *x, cudaStream_t st) {
  {
    XK_PROF("wrap");
    k_wrap<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, x);
  }
  return XK_LAUNCHED();
}

cudaError_t zero(double *p, size_t n, cudaStream_t st) {
  return cudaMemsetAsync(p, 0, n * sizeof(double), st);
}

__global__ void k_set_value(double *p, double v) { *p = v; }

cudaError_t set_value(double *p, double v, cudaStream_t st) {
  k_set_value<<<1, 1, 0, st>>>(p, v);
  return cudaGetLastError();
}

// ===================================================================
// cycle spring energies E_l^(k): md_pimd_x.c:1969-2210 (CPU :2086-2207)
// ===================================================================


// interior ring springs of particle l and the closing spring P -> 1: one
// warp per particle, lanes over the beads, fixed-order warp sum.  Also
// gl[l] = Eint[l] + link(l, l+1) (l < N-1), the increments whose prefix
// sums k_enk_direct needs.
template <int D>
__global__ void k_eint(Geo g, const double *__restrict__ x, const double *__restrict__ m,
                       double w2, int image, double *Eint, double *ENk, double *gl) {
  const int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (l >= g.N) return;
  eint_particle<D>(g, x, m, w2, image, Eint, ENk, gl, l, threadIdx.x & 31);
}


// the prefix sums of the N-1 ENk increments into gl[N ..] (one block), for
// systems too large to hold them in each k_enk_direct block
__global__ void __launch_bounds__(1024) k_gscan(int N, double *__restrict__ gl) {
  block_exclusive_prefix(gl, N - 1, gl + N);
}

// E_l^(k) for k = 2..l (1-based row l) in closed form.
// The reference's recursion adds, for k = 2..l with c = l-k+1,
//   Eint[c] + link(c, c+1) + link(l, c) - link(l, c+1),
// and the link(l, .) terms telescope, so
//   E_l^(k) = Eint[l] + (G[l-1] - G[l-k]) + link(l, l-k+1),
// G the prefix sums of Eint[c] + link(c, c+1): every entry independent, one
// spring each (no N x N table of springs, no scan along the row).
// With own_g, every block scans the increments itself into shared memory
// (N doubles): a separate scan launch on the sequential path costs more than
// the repeated scan.
template <int D>
__global__ void __launch_bounds__(256) k_enk_direct(Geo g, const double *__restrict__ x,
                                                    const double *__restrict__ m, double w2, int image,
                                                    const double *__restrict__ Eint,
                                                    const double *__restrict__ gl, double *__restrict__ ENk,
                                                    int own_g) {
  extern __shared__ double Gs[];
  const double *G = gl + g.N;
  if (own_g) {
    block_exclusive_prefix(gl, g.N - 1, Gs);
    __syncthreads();
    G = Gs;
  }
  // rows l1 and N+2-l1 (l1-1 and N+1-l1 entries, N together) share a block
  const int l1 = blockIdx.x + 2, l2 = g.N - blockIdx.x;
  const int n1 = l1 - 1, n = n1 + (l2 > l1 ? l2 - 1 : 0);
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int l = e < n1 ? l1 : l2, k = 2 + (e < n1 ? e : e - n1);  // 1-based row, cycle length
    enk_entry<D>(g, x, m, w2, image, Eint, G, ENk, l, k);
  }
}

cudaError_t fill_enk(const Geo &g, const double *x, const double *m, double w2, int image,
                     double *Eint, double *ENk, double *gl, cudaStream_t st) {
  {
    XK_PROF("eint");
    DISPATCH_D(g.D, k_eint<D><<<cdiv((size_t)g.N * 32, 64), 64, 0, st>>>(g, x, m, w2, image, Eint, ENk, gl));
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess || g.N < 2) return e;
  const bool own_g = g.N <= 6000;  // N doubles of shared memory a block (within 48 KB)
  if (!own_g) {
    {
      XK_PROF("gscan");
      k_gscan<<<1, 1024, 0, st>>>(g.N, gl);
    }
    e = XK_LAUNCHED();
    if (e != cudaSuccess) return e;
  }
  {
    XK_PROF("enk_direct");
    DISPATCH_D(g.D, k_enk_direct<D><<<g.N / 2, 256, own_g ? sizeof(double) * g.N : 0, st>>>(
                        g, x, m, w2, image, Eint, gl, ENk, own_g ? 1 : 0));
  }
  return XK_LAUNCHED();
}

// virial cross term 1/2 m w2 (x_a - x_b).(x_a - x_c) for beads a, b, c:
// md_pimd_x.c:4376-4421
template <int D>
__device__ inline double cross(Geo g, const double *x, const double *m, double w2, int ja, int la,
                               int jb, int lb, int jc, int lc, int image) {
  double r = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const double xa = x[sidx(ja, d, la, D, g.Ns)];
    double t = xa - x[sidx(jb, d, lb, D, g.Ns)];
    double u = xa - x[sidx(jc, d, lc, D, g.Ns)];
    if (image) {
      t = min_image(t, g.box[d], g.inv_box[d]);
      u = min_image(u, g.box[d], g.inv_box[d]);
    }
    r += 0.5 * m[(size_t)ja * g.Ns + la] * w2 * t * u;
  }
  return r;
}

// ENk2 of the virial estimator, md_pimd_x.c:4423-4556 (CPU :4521-4553): row l,
// k = 1..l.  With t_a(b) = 1/2 m_a w2 (x_a1 - x_bP).(x_a1 - x_b1) the reference
// starts a row at t_l(l) and adds, for k = 2..l with c = l-k+1,
//   t_l(c) - t_l(c+1) + t_c(c+1);
// the t_l terms telescope, so
//   ENk2[l][k] = t_l(s) + H[l-1] - H[s-1],   s = l-k+1,
// H the prefix sums of t_c(c+1).  The t_c(c+1) have either sign, so H is kept
// with its rounding errors (two doubles): differences of it are good to the
// last bit of the result, not of H.
// Bound: FP64 pipe, one term of D minimum images an entry (three, and a scan
// of FP64 sums along each row, in a kernel of a warp a row).  A sampling pass of 128
// electrons and 32 beads: 288 -> 262 us.

// H[c], c = 0..N-1: high parts, then low parts (one block)
template <int D>
__global__ void __launch_bounds__(1024) k_enk2_prefix(Geo g, const double *__restrict__ x,
                                                      const double *__restrict__ m, double w2, int image,
                                                      double *H) {
  __shared__ double wh[32], wl[32];
  const int n = g.N - 1, per = (n + blockDim.x - 1) / blockDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int a = min(n, (int)threadIdx.x * per), b = min(n, a + per);
  // (h, l) += (t, tl): the rounding error of the high parts' sum joins the low parts
  auto add = [](double &h, double &l, double t, double tl) {
    const double s = h + t, v = s - h;
    l += tl + ((h - (s - v)) + (t - v));
    h = s;
  };
  auto warp_scan = [&](double &h, double &l) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(FULL, h, o), tl = __shfl_up_sync(FULL, l, o);
      if (lane >= o) add(h, l, t, tl);
    }
  };
  double h = 0.0, l = 0.0;
  for (int c = a; c < b; ++c) {
    const double t = cross<D>(g, x, m, w2, 0, c, g.P - 1, c + 1, 0, c + 1, image);
    H[c + 1] = t;
    add(h, l, t, 0.0);
  }
  warp_scan(h, l);
  if (lane == 31) {
    wh[w] = h;
    wl[w] = l;
  }
  __syncthreads();
  const int nw = blockDim.x >> 5;
  if (w == 0 && nw > 1) {
    double th = lane < nw ? wh[lane] : 0.0, tl = lane < nw ? wl[lane] : 0.0;
    warp_scan(th, tl);
    wh[lane] = th;
    wl[lane] = tl;
  }
  __syncthreads();
  // the sum before this thread's run
  h = __shfl_up_sync(FULL, h, 1);
  l = __shfl_up_sync(FULL, l, 1);
  if (lane == 0) h = l = 0.0;
  if (w > 0) add(h, l, wh[w - 1], wl[w - 1]);
  if (threadIdx.x == 0) H[0] = H[g.N] = 0.0;
  for (int c = a; c < b; ++c) {
    add(h, l, H[c + 1], 0.0);
    H[c + 1] = h;
    H[g.N + c + 1] = l;
  }
}

template <int D>
__global__ void __launch_bounds__(128) k_enk2_direct(Geo g, const double *__restrict__ x,
                                                     const double *__restrict__ m, double w2, int image,
                                                     const double *__restrict__ H, double *__restrict__ ENk2) {
  // rows l1 and N+1-l1 (N+1 entries together) share a block
  const int l1 = blockIdx.x + 1, l2 = g.N - blockIdx.x, n = l1 + (l2 > l1 ? l2 : 0);
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int l = e < l1 ? l1 : l2, k = 1 + (e < l1 ? e : e - l1), s = l - k + 1;
    const double t = cross<D>(g, x, m, w2, 0, l - 1, g.P - 1, s - 1, 0, s - 1, image);
    const double h = H[l - 1] - H[s - 1], lo = H[g.N + l - 1] - H[g.N + s - 1];
    ENk2[dtri(l) + k - 1] = t + (h + lo);
  }
}

// cubic-path table of md_pimd_fill_ENk2_x (md_pimd_x.c:3959-3987, CPU
// :4049-4054): for the cycle over particles l = N2-k+1..N2, each bead P is
// followed by bead 1 of the next particle in the cycle (b) and
//   ENk2[N2][k] = sum_l 1/2 m_b w2 (x_b - x_{l,P}).(x_b - x_{l,1}).
// For l < N2 the term depends on l alone (b = l+1), so a row is a scan over
// k of those terms plus the closing term of l = N2 (b = N2-k+1).
template <int D>
__global__ void k_enk2_cubic_rows(Geo g, const double *__restrict__ x, const double *__restrict__ m,
                                  double w2, int image, double *__restrict__ ENk2) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int n = w + 1;  // 1-based N2
  if (n > g.N) return;
  const int jP = g.P - 1;
  double carry = 0;
  for (int k0 = 1; k0 <= n; k0 += 32) {
    const int k = k0 + lane;
    double inc = 0, close = 0;
    if (k <= n) {
      if (k >= 2) {
        const int l = n - k + 1;  // 1-based, l < n: b = l+1
        inc = cross<D>(g, x, m, w2, 0, l, jP, l - 1, 0, l - 1, image);
      }
      const int b = n - k + 1;  // closing bead of l = n
      close = cross<D>(g, x, m, w2, 0, b - 1, jP, n - 1, 0, n - 1, image);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += t;
    }
    const double e = carry + inc;
    if (k <= n) ENk2[dtri(n) + k - 1] = e + close;
    carry = __shfl_sync(FULL, e, 31);
  }
}

cudaError_t fill_enk2_cubic(const Geo &g, const double *x, const double *m, double w2, int image,
                            double *ENk2, cudaStream_t st) {
  const size_t thr = (size_t)g.N * 32;
  {
    XK_PROF("enk2_cubic_rows");
    DISPATCH_D(g.D, k_enk2_cubic_rows<D><<<cdiv(thr, 256), 256, 0, st>>>(g, x, m, w2, image, ENk2));
  }
  return XK_LAUNCHED();
}

cudaError_t fill_enk2(const Geo &g, const double *x, const double *m, double w2, int image,
                      double *ENk2, double *H, cudaStream_t st) {
  {
    XK_PROF("enk2_prefix");
    const int T = std::min(1024, std::max(32, (g.N - 1 + 31) / 32 * 32));
    DISPATCH_D(g.D, k_enk2_prefix<D><<<1, T, 0, st>>>(g, x, m, w2, image, H));
  }
  const cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  {
    XK_PROF("enk2_direct");
    DISPATCH_D(g.D, k_enk2_direct<D><<<(g.N + 1) / 2, 128, 0, st>>>(g, x, m, w2, image, H, ENk2));
  }
  return XK_LAUNCHED();
}

// ===================================================================
// exchange recursions (single persistent block each)
// ===================================================================

// ---- linear-solve form ----------------------------------------------
// With Z_n = exp(-beta V_n) the forward recursion is linear:
//   Z_0 = 1,  Z_n = sum_{k=1..n} M_{n,n-k} Z_{n-k},
//   M_{n,j} = xi^(k-1) exp(-beta E_n^(k)) / n            (k = n - j),
// and V_n = -ln(Z_n)/beta; this is the reference's log-sum-exp recursion
// without the shift.  The backward recursion is the same system after the
// index map i = N-u+1 (X_i = exp(-beta tmpV_{u-1})), j = N-l, k = i-j:
//   M'_{i,j} = xi^(k-1) exp(-beta E_l^(k)) / l.
// Z spans far more than the FP64 exponent range (beta V_n ~ 100 n), so every
// weight and unknown is kept in extended range: an FP64 mantissa and an int
// power of two.  All weights (N^2/2 exponentials) are computed in parallel
// over the GPU; one block then solves the unit lower-triangular system in
// chunks of 32 rows: the contribution of the already known unknowns to the
// chunk is a parallel extended-range dot product per row, and the chunk
// itself is a 32-step warp-synchronous substitution.  No exponential or
// logarithm sits on the sequential chain, which matters because a dependent
// FP64 operation costs ~64 cycles on this GPU.
//
// For xi = 0 only k = 1 enters (M_{i,i-1}), as in the reference's branch.


__global__ void __launch_bounds__(128) k_weights(int N, double beta, double vi, double lnvi,
                                                 const double *__restrict__ ENk, const double *__restrict__ lnn,
                                                 double *__restrict__ Mf, int *__restrict__ Ef,
                                                 double *__restrict__ Mb, int *__restrict__ Eb, int first, int sgn,
                                                 int both) {
  weights_row<false>(N, beta, vi, lnvi, ENk, lnn, Mf, Ef, Mb, Eb, first, sgn, both, blockIdx.x + 1, first + blockIdx.y,
              threadIdx.x, blockDim.x);
}

static cudaError_t weights(int N, double beta, double vi, const double *ENk, const double *lnn, double *rs_f,
                           double *rs_b, int first, int count, cudaStream_t st, int sgn = 1) {
  const double lnvi = vi != 0.0 ? log(vi) : 0.0;
  const int both = count == 2 ? 1 : 0;  // first = 0
  dim3 grid(N, both ? 1 : count);
  {
    XK_PROF("weights");
    k_weights<<<grid, 128, 0, st>>>(N, beta, vi, lnvi, ENk, lnn, rs_f, rs_f ? (int *)(rs_f + ntri(N)) : nullptr,
                                    rs_b, rs_b ? (int *)(rs_b + ntri(N)) : nullptr, first, sgn, both);
  }
  return XK_LAUNCHED();
}


__global__ void __launch_bounds__(TS_WARPS * 32) k_tri_solve(int N, double beta, TriJob job, int first) {
  const int backward = first + blockIdx.x;
  const double *__restrict__ Mm = job.Mm[backward];
  const int *__restrict__ Me = job.Me[backward];
  double *__restrict__ out = job.out[backward];
  extern __shared__ double sh[];
  double *Wm = sh;                              // [2][TS_CHUNK][TS_LD] the chunk's triangle
  double *Um = Wm + 2 * TS_CHUNK * TS_LD;       // [2][TS_CHUNK][TS_LD] previous chunk's columns
  double *Pm = Um + 2 * TS_CHUNK * TS_LD;       // [2][TS_CHUNK] partial sums (double buffer)
  double *Xm = Pm + 2 * TS_CHUNK;               // N+1
  int *We = (int *)(Xm + N + 1);                // [2][TS_CHUNK][TS_LD]
  int *Ue = We + 2 * TS_CHUNK * TS_LD;          // [2][TS_CHUNK][TS_LD]
  int *Pe = Ue + 2 * TS_CHUNK * TS_LD;          // [2][TS_CHUNK]
  int *Xe = Pe + 2 * TS_CHUNK;                  // N+1
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // weights of chunk starting at n0 (triangle) and its block against the
  // columns c0 .. c0+31 (c0 < 0: none) into buffer nb; threads t0, t0+stride..
  auto stage = [&](int n0, int c0, int nb, int t0, int stride) {
    for (int q = t0; q < 2 * TS_CHUNK * TS_CHUNK; q += stride) {
      const int which = q / (TS_CHUNK * TS_CHUNK), rs = q % (TS_CHUNK * TS_CHUNK);
      const int r = rs / TS_CHUNK, c = rs % TS_CHUNK, i = n0 + r;
      const size_t o = ((size_t)nb * TS_CHUNK + r) * TS_LD + c;
      if (which == 0) {
        const bool in = i <= N && c < r;
        Wm[o] = in ? Mm[moff(i, n0 + c)] : 0.0;
        We[o] = in ? Me[moff(i, n0 + c)] : 0;
      } else {
        const bool in = i <= N && c0 >= 0;
        Um[o] = in ? Mm[moff(i, c0 + c)] : 0.0;
        Ue[o] = in ? Me[moff(i, c0 + c)] : 0;
      }
    }
  };
  if (threadIdx.x == 0) {
    Xm[0] = 0.5;
    Xe[0] = 1;
  }
  stage(1, -1, 0, threadIdx.x, blockDim.x);
  __syncthreads();
  // chunk 0: its rows against column 0
  for (int r = w; r < TS_CHUNK; r += TS_WARPS) {
    const int i = 1 + r;
    double am = 0.0;
    int E = 0;
    if (i <= N) ext_dot(Mm + moff(i, 0), Me + moff(i, 0), Xm, Xe, 0, 1, lane, am, E);
    if (lane == 0) {
      double pm = 0.0;
      int pe = 0;
      if (i <= N) ext_acc(pm, pe, am, E);
      Pm[r] = pm;
      Pe[r] = pe;
    }
  }
  __syncthreads();
  for (int i0 = 1, c = 0; i0 <= N; i0 += TS_CHUNK, ++c) {
    const int buf = c & 1;
    double *Pmc = Pm + buf * TS_CHUNK;
    int *Pec = Pe + buf * TS_CHUNK;
    // the previous chunk's columns [i0 - 32, i0), one per lane, from the
    // staged block
    if (c > 0) {
      const int col = i0 - TS_CHUNK + lane;
      for (int r = w; r < TS_CHUNK; r += TS_WARPS) {
        if (i0 + r > N) continue;  // warp-uniform
        const size_t o = ((size_t)buf * TS_CHUNK + r) * TS_LD + lane;
        const double mv = Um[o];
        const bool nz = __double_as_longlong(mv) != 0;
        const int te = nz ? Ue[o] + Xe[col] : EXT_NONE;
        int E = te;
#pragma unroll
        for (int o2 = 16; o2; o2 >>= 1) {
          const int oe = __shfl_xor_sync(FULL, E, o2);
          E = oe > E ? oe : E;
        }
        double am = nz ? mv * scale2(Xm[col], nz ? te - E : 0) : 0.0;
        am = warp_sum(am);
        if (lane == 0) {
          double pm = Pmc[r];
          int pe = Pec[r];
          ext_acc(pm, pe, am, E);
          Pmc[r] = pm;
          Pec[r] = pe;
        }
      }
      __syncthreads();
    }
    if (w == 0) {
      // lane r owns row i0+r; each step publishes one unknown and every
      // later row adds its term (exponent arithmetic and one FMA on the
      // sequential chain)
      const int i = i0 + lane;
      const bool own = i <= N;
      double am = own ? Pmc[lane] : 0.0;
      int ae = own ? Pec[lane] : 0;
      double mm[TS_CHUNK];
      int me[TS_CHUNK];
      const size_t ro = ((size_t)buf * TS_CHUNK + lane) * TS_LD;
#pragma unroll
      for (int s = 0; s < TS_CHUNK; ++s) {
        mm[s] = Wm[ro + s];
        me[s] = We[ro + s];
      }
#pragma unroll
      for (int s = 0; s < TS_CHUNK; ++s) {
        if (lane == s) {
          norm2(am, ae);
          if (own) {
            Xm[i] = am;
            Xe[i] = ae;
          }
        }
        const double xm = __shfl_sync(FULL, am, s);
        const int xe = __shfl_sync(FULL, ae, s);
        // later rows add their term; a larger term exponent sets the scale
        // (straight-line code with selects: no divergence on the chain)
        const bool upd = lane > s && __double_as_longlong(mm[s]) != 0;
        const int te = me[s] + xe;
        const int ne = (upd && te > ae) ? te : ae;
        const double t2 = fma(mm[s], scale2(xm, upd ? te - ne : 0), scale2(am, ae - ne));
        am = upd ? t2 : am;
        ae = ne;
      }
    } else {
      // next chunk: stage its weights, and its rows against the columns
      // solved before this chunk
      const int n0 = i0 + TS_CHUNK;
      if (n0 <= N) stage(n0, i0, buf ^ 1, threadIdx.x - 32, blockDim.x - 32);
      for (int r = w - 1; r < TS_CHUNK; r += TS_WARPS - 1) {
        const int i = n0 + r;
        if (i > N) break;  // warp-uniform; later rows are out of range too
        double am;
        int E;
        ext_dot(Mm + moff(i, 0), Me + moff(i, 0), Xm, Xe, 0, i0, lane, am, E);
        if (lane == 0) {
          double pm = 0.0;
          int pe = 0;
          ext_acc(pm, pe, am, E);
          Pm[(buf ^ 1) * TS_CHUNK + r] = pm;
          Pe[(buf ^ 1) * TS_CHUNK + r] = pe;
        }
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x + 1; i <= N; i += blockDim.x) {
    const double lnx = log(fabs(Xm[i])) + Xe[i] * LN2_HI + Xe[i] * LN2_LO;
    out[backward ? N - i : i] = -lnx / beta;
    if (job.sign && !backward) job.sign[i] = Xm[i] < 0.0 ? -1.0 : 1.0;
  }
  if (threadIdx.x == 0) {
    out[backward ? N : 0] = 0.0;
    if (job.sign && !backward) job.sign[0] = 1.0;
  }
}

// slots of the cluster solve's summing blocks (k_tri_solve_c)
__host__ __device__ inline int tsc_slots(int nch, int CL) { return (nch - 1 + CL - 2) / (CL - 1); }
// doubles of partial sums in memory for one direction of the SLOTS = 0 variant
static size_t tsc_sums(int N) {
  const int nch = (N + TS_CHUNK - 1) / TS_CHUNK;
  return nch <= 29 ? 0 : (size_t)7 * tsc_slots(nch, 8) * TS_CHUNK * 32 * 3 / 2;
}

// one direction's scratch: weights (mantissas, then exponents as ints), the
// diagonal blocks' inverses B and the products W (mantissas, exponents), the
// unknowns X_0..X_N and 1/X_N (mantissas, exponents), and the partial sums of the
// cluster solve's memory variant
size_t rec_scratch_doubles(int N) {
  const size_t nch = (N + TS_CHUNK - 1) / TS_CHUNK;
  return ntri(N) + (ntri(N) + 1) / 2 + 1 + nch * TS_CHUNK * TS_CHUNK * 3 + (size_t)(N + 2) + (N + 3) / 2 + tsc_sums(N);
}

// directions first .. first + count - 1 of job
// ---- block-inverse form (unsigned weights) ----------------------------
// Within chunk c (rows i0 .. i0+31) the system reads X = R + A X with A the
// strictly lower 32 x 32 block of the weights and R the rows' sums over all
// earlier unknowns, so X = B R with B = (I - A)^-1 = I + A + A^2 + ...  B
// depends only on the weights: k_weights_inv computes it for every chunk at
// once (a warp per column, all chunks in parallel over the GPU), and the
// solve then replaces the 32-step substitution by a 32-term product per row,
// done by all warps.  With non-negative weights every term is non-negative,
// so the extended-range sums have no cancellation.


// Weights and the diagonal-block inverses in one launch, so that the
// inverses (latency-bound: a chain of 31 steps per column) run beside
// the weight rows instead of after them: blocks 0..N-1 are k_weights' rows,
// the rest take four columns of one chunk's B (groups 0..7 of the chunk) or W
// (8..15, for the cluster solve) each and evaluate the blocks they need from
// ENk themselves.
__global__ void __launch_bounds__(128) k_weights_inv(int N, double beta, double vi, double lnvi,
                                                     const double *__restrict__ ENk,
                                                     const double *__restrict__ lnn, TriJob job, int first,
                                                     int both, int groups) {
  __shared__ long long Am[TS_CHUNK][TS_LD];
  __shared__ int Ae[TS_CHUNK][TS_LD];
  if ((int)blockIdx.x < N) {
    weights_row<true>(N, beta, vi, lnvi, ENk, lnn, (double *)job.Mm[0], (int *)job.Me[0], (double *)job.Mm[1],
                (int *)job.Me[1], first, 1, both, blockIdx.x + 1, first, threadIdx.x,
                blockDim.x);
    return;
  }
  const int nch = (N + TS_CHUNK - 1) / TS_CHUNK;
  const int b = blockIdx.x - N, dir = first + b / (nch * groups), c = b / groups % nch, q = b % groups;
  const bool inv = q < 8;
  if (!inv && c == 0) return;  // no chunk before the first
  const int s0 = (q & 7) << 2, s = s0 + (threadIdx.x >> 5), t0 = inv ? s0 : 0;
  const int i0 = 1 + c * TS_CHUNK;
  // column s of B reads the block's entries t >= s only
  for (int e = threadIdx.x; e < TS_CHUNK * TS_CHUNK; e += blockDim.x) {
    const int r = e / TS_CHUNK, t = e % TS_CHUNK;
    XI a{0, XI_NONE};
    if (t < r && t >= t0 && i0 + r <= N) a = weight_at(N, beta, vi, lnvi, ENk, lnn, dir, i0 + r, i0 + t);
    Am[r][t] = a.m;
    Ae[r][t] = a.e;
  }
  __syncthreads();
  if (inv) {
    block_inv_column(N, job, dir, c, s, Am, Ae);
    return;
  }
  block_w_column(N, beta, vi, lnvi, ENk, lnn, job, dir, c, s, Am, Ae);
}

// One block per direction, 16 warps, three phases per chunk c:
//   U: R_r = (row r's sum over the unknowns before chunk c-1) + (its terms
//      over chunk c-1's 32 unknowns), one warp per row;
//   B: X_{i0+r} = sum_s B[r][s] R_s, one warp per row;
//   next: chunk c+1's weights against chunk c and its B block are staged in
//      shared memory, and its rows' sums over the unknowns before chunk c
//      are taken (the long dot products, split over the warps).
constexpr int TSB_WARPS = 32;  // one warp per row of a chunk in every phase

__global__ void __launch_bounds__(TSB_WARPS * 32) k_tri_solve_b(int N, double beta, TriJob job, int first) {
  extern __shared__ double sh[];
  tri_solve_b_dev(N, beta, job, first + blockIdx.x, sh);
}

// The solve spread over a thread-block cluster: one cluster of CL blocks per
// direction.  With P_c the rows' sums of chunk c over the unknowns before
// chunk c-1,
//   X_c = B_c (P_c + U_c X_{c-1}) = Y_c + W_c X_{c-1},   Y_c = B_c P_c,
// so block 0's chain is one 32 x 32 product a chunk.  The other blocks own
// the later rows' running sums (chunk k >= 1 belongs to block
// 1 + (k-1) mod (CL-1), its slot (k-1) / (CL-1)): in iteration c each adds
// chunk c-1's unknowns, which block 0 wrote into its shared memory, to the
// rows of its chunks after c, one column a lane; the owner of chunk c+1 does
// that chunk's rows first, adds up their lanes, forms Y_{c+1} and writes it
// into block 0's shared memory.  Every block arrives at the iteration's
// cluster barrier as soon as the others need nothing more of it: the bulk of
// the sums runs between a block's arrival and its wait, with the next
// weights' loads in flight.
// Bound: the chain of N/32 chunks, each a product, a warp sum, a remote store
// and a cluster barrier (about 1800 cycles), and in long systems the integer
// instructions of the sums, which is why a row's partial sums stay in
// registers (SLOTS > 0) and the weights come as XI.
// Variants: 8 blocks up to 7 SLOTS + 1 = 29 chunks (N = 928; more blocks would
// only take SMs from the pair forces beside them), 16 with 8 slots up to 121
// chunks; beyond, or where 16 blocks do not fit, 8 with the partial sums in
// memory (SLOTS = 0).
constexpr int TSC_WARPS = 16;  // warps per block; warp w takes rows w and w + 16 of a chunk
constexpr int TSC_HB = 8;      // SLOTS = 0: rows whose weights a summing warp loads at a time

static size_t tsc_smem(int N) { return (sizeof(long long) + sizeof(int)) * (size_t)(N + 1 + 3 * TS_CHUNK) + 16; }
template <int CL, int SLOTS>
__global__ void __launch_bounds__(TSC_WARPS * 32) k_tri_solve_c(int N, double beta, TriJob job, int first) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int backward = first + blockIdx.y;
  const long long *__restrict__ Mm = (const long long *)job.Mm[backward];
  const int *__restrict__ Me = job.Me[backward];
  const long long *__restrict__ Bgm = (const long long *)job.Bm[backward];
  const int *__restrict__ Bge = job.Be[backward];
  const long long *__restrict__ Wgm = (const long long *)job.Wm[backward];
  const int *__restrict__ Wge = job.We[backward];
  const int nch = (N + TS_CHUNK - 1) / TS_CHUNK;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int CC = TS_CHUNK * TS_CHUNK;
  extern __shared__ double sh[];
  // block 0: Y [2][TS_CHUNK], X_0..X_N; the others: the last unknowns
  // [2][TS_CHUNK], a chunk's completed row sums [TS_CHUNK]
  long long *Ym = (long long *)sh, *Xm = Ym + 2 * TS_CHUNK, *Hxm = Ym, *Hpm = Xm;
  int *Ye = (int *)(Ym + N + 1 + 3 * TS_CHUNK), *Xe = Ye + 2 * TS_CHUNK, *Hxe = Ye, *Hpe = Xe;
  // two rows a warp of the 32 x 32 block of a chunk, a column a lane
  struct Rows {
    long long m[2];
    int e[2];
  };
  auto load_block = [&](const long long *m, const int *e, int c) {
    Rows b{{0, 0}, {XI_NONE, XI_NONE}};
    if (c < nch)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const size_t o = (size_t)c * CC + (w + h * TSC_WARPS) * TS_CHUNK + lane;
        b.m[h] = m[o];
        b.e[h] = e[o];
      }
    return b;
  };
  // summing blocks: this warp's row h of slot t
  auto row_of = [&](int t, int h) { return 1 + (rank + t * (CL - 1)) * TS_CHUNK + w + h * TSC_WARPS; };
  auto weight = [&](int i, int j0) {  // row i's weight against column j0 + lane
    const size_t o = moff(i, j0 + lane);
    return i <= N ? XI{Mm[o], Me[o]} : XI{0, XI_NONE};
  };
  constexpr int R = SLOTS > 0 ? 2 * SLOTS : 1;
  XI acc[R], nxt[R];
  const int slots = tsc_slots(nch, CL);
  long long *Sm = nullptr;  // SLOTS = 0: partial sums [slots][TS_CHUNK][32] in memory, of this block
  int *Se = nullptr;
  Rows blk{{0, 0}, {XI_NONE, XI_NONE}};
  if (rank == 0) {
    if (threadIdx.x == 0) {
      Xm[0] = 1LL << 61;  // X_0 = 1
      Xe[0] = 1;
    }
    // Y_0 = B_0 times the first rows' weights against X_0
    const XI p = 1 + lane <= N ? XI{Mm[moff(1 + lane, 0)], Me[moff(1 + lane, 0)]} : XI{0, XI_NONE};
    const Rows b = load_block(Bgm, Bge, 0);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const XI y = xi_warp_sum(xi_mul({b.m[h], b.e[h]}, p));
      if (lane == 0) {
        Ym[w + h * TSC_WARPS] = y.m;
        Ye[w + h * TSC_WARPS] = y.e;
      }
    }
  } else {
    // the rows' sums start with their weights against X_0, in lane 0
    auto start = [&](int t, int h) {
      const int i = row_of(t, h);
      return lane == 0 && i <= N ? XI{Mm[moff(i, 0)], Me[moff(i, 0)]} : XI{0, XI_NONE};
    };
    if (SLOTS > 0) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        acc[q] = start(q / 2, q & 1);
        nxt[q] = {0, XI_NONE};
      }
    } else {
      const size_t per = (size_t)slots * TS_CHUNK * 32;
      Sm = (long long *)job.Sm[backward] + (rank - 1) * per;
      Se = (int *)((long long *)job.Sm[backward] + (CL - 1) * per) + (rank - 1) * per;
      for (int q = 0; q < 2 * slots; ++q) {
        const XI a = start(q / 2, q & 1);
        const size_t o = ((size_t)(q / 2) * TS_CHUNK + w + (q & 1) * TSC_WARPS) * 32 + lane;
        Sm[o] = a.m;
        Se[o] = a.e;
      }
    }
    if (rank == 1) blk = load_block(Bgm, Bge, 1);  // chunk 1's owner
  }
  Rows blk2 = rank == 0 ? load_block(Wgm, Wge, 1) : blk;
  cl.sync();  // every block has started and holds its initial sums
  for (int c = 0; c < nch; ++c) {
    const int i0 = 1 + c * TS_CHUNK, buf = c & 1;
    if (rank == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = w + h * TSC_WARPS, i = i0 + r;
        const XI y{Ym[buf * TS_CHUNK + r], Ye[buf * TS_CHUNK + r]};
        const XI v = c > 0 ? XI{Xm[i0 - TS_CHUNK + lane], Xe[i0 - TS_CHUNK + lane]} : XI{0, XI_NONE};
        const XI x = xi_add(y, xi_warp_sum(xi_mul({blk.m[h], blk.e[h]}, v)));
        if (i > N) continue;
        if (lane == 0) {
          Xm[i] = x.m;
          Xe[i] = x.e;
        } else if (lane < CL) {
          *cl.map_shared_rank(Hxm + buf * TS_CHUNK + r, lane) = x.m;
          *cl.map_shared_rank(Hxe + buf * TS_CHUNK + r, lane) = x.e;
        }
      }
      cl.barrier_arrive();
      blk = blk2;  // W_{c+1}, loaded an iteration ago
      blk2 = load_block(Wgm, Wge, c + 2);
    } else {
      // chunk c-1's unknowns, columns j0 on
      const int j0 = i0 - TS_CHUNK;
      XI x{0, XI_NONE};
      if (c >= 1) x = {Hxm[(buf ^ 1) * TS_CHUNK + lane], Hxe[(buf ^ 1) * TS_CHUNK + lane]};
      // the owner of chunk c+1 completes that chunk's rows, now over the
      // unknowns before chunk c, and hands Y_{c+1} to block 0
      const int kn = c + 1, tn = (kn - 1) / (CL - 1);
      const bool owner = kn < nch && kn - tn * (CL - 1) == rank;
      // first slot whose chunk comes after c
      const int t0 = c + 1 > rank ? (c + 1 - rank + CL - 2) / (CL - 1) : 0;
      if (owner) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          XI p{0, XI_NONE};
          if (SLOTS > 0) {
#pragma unroll
            for (int t = 0; t < SLOTS; ++t)
              if (t == tn) p = xi_mul_add(acc[2 * t + h], nxt[2 * t + h], x);
          } else {
            const size_t o = ((size_t)tn * TS_CHUNK + w + h * TSC_WARPS) * 32 + lane;
            p = {Sm[o], Se[o]};
            if (c >= 1) p = xi_mul_add(p, weight(row_of(tn, h), j0), x);
          }
          p = xi_warp_sum(p);
          if (lane == 0) {
            Hpm[w + h * TSC_WARPS] = p.m;
            Hpe[w + h * TSC_WARPS] = p.e;
          }
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const XI y = xi_warp_sum(xi_mul({blk.m[h], blk.e[h]}, {Hpm[lane], Hpe[lane]}));
          if (lane == 0) {
            *cl.map_shared_rank(Ym + (kn & 1) * TS_CHUNK + w + h * TSC_WARPS, 0) = y.m;
            *cl.map_shared_rank(Ye + (kn & 1) * TS_CHUNK + w + h * TSC_WARPS, 0) = y.e;
          }
        }
      }
      cl.barrier_arrive();
      if (SLOTS > 0) {
#pragma unroll
        for (int q = 0; q < R; ++q) {
          if (q / 2 < t0) continue;
          if (c >= 1) acc[q] = xi_mul_add(acc[q], nxt[q], x);
          nxt[q] = weight(row_of(q / 2, q & 1), i0);
        }
      } else if (c >= 1) {
        for (int qb = 2 * (owner ? t0 + 1 : t0); qb < 2 * slots; qb += TSC_HB) {
          XI m[TSC_HB];
#pragma unroll
          for (int u = 0; u < TSC_HB; ++u)
            m[u] = qb + u < 2 * slots ? weight(row_of((qb + u) / 2, u & 1), j0) : XI{0, XI_NONE};
#pragma unroll
          for (int u = 0; u < TSC_HB; ++u) {
            const int q = qb + u;
            if (q >= 2 * slots) break;
            const size_t o = ((size_t)(q / 2) * TS_CHUNK + w + (q & 1) * TSC_WARPS) * 32 + lane;
            const XI a = xi_mul_add({Sm[o], Se[o]}, m[u], x);
            Sm[o] = a.m;
            Se[o] = a.e;
          }
        }
      }
      const int k2 = c + 2, t2 = (k2 - 1) / (CL - 1);
      if (k2 < nch && k2 - t2 * (CL - 1) == rank) blk = load_block(Bgm, Bge, k2);
    }
    cl.barrier_wait();
  }
  // V_B = -ln X / beta: the unknowns dealt over the blocks, read from block 0
  tri_solve_out(N, beta, job, backward, cl.map_shared_rank(Xm, 0), cl.map_shared_rank(Xe, 0),
                threadIdx.x * CL + rank, CL * blockDim.x);
  cl.sync();  // block 0's shared memory is read until here
}

// the variant for N that fits this device: 0 none, 1 eight blocks, 2 sixteen,
// 3 eight with the sums in memory
struct ClusterKernel {
  void (*fn)(int, double, TriJob, int);
  int cl;
};
static const ClusterKernel g_cluster_kernels[4] = {
    {nullptr, 0}, {k_tri_solve_c<8, 4>, 8}, {k_tri_solve_c<16, 8>, 16}, {k_tri_solve_c<8, 0>, 8}};

static void cluster_config(const ClusterKernel &k, int N, int count, cudaStream_t st, cudaLaunchConfig_t &cfg,
                           cudaLaunchAttribute &attr) {
  cfg = {};
  cfg.gridDim = dim3(k.cl, count);
  cfg.blockDim = dim3(TSC_WARPS * 32);
  cfg.dynamicSmemBytes = tsc_smem(N);
  cfg.stream = st;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = k.cl;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
}

// whether two clusters of the variant fit at once with N's shared memory (the
// largest that did and the smallest that did not are kept)
static bool cluster_fits(int v, int N) {
  static std::mutex mu;
  static size_t good[4] = {0, 0, 0, 0}, bad[4] = {~(size_t)0, ~(size_t)0, ~(size_t)0, ~(size_t)0};
  const size_t smem = tsc_smem(N);
  std::lock_guard<std::mutex> lk(mu);
  if (smem <= good[v]) return true;
  if (smem >= bad[v]) return false;
  const ClusterKernel &k = g_cluster_kernels[v];
  int n = 0;
  cudaError_t e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess && k.cl > 8) e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(k, N, 2, nullptr, cfg, attr);
    e = cudaOccupancyMaxActiveClusters(&n, (const void *)k.fn, &cfg);
  }
  if (e != cudaSuccess) cudaGetLastError();
  if (e == cudaSuccess && n >= 2) {
    good[v] = smem;
    return true;
  }
  bad[v] = smem;
  return false;
}
static int cluster_variant(int N) {
  const int nch = (N + TS_CHUNK - 1) / TS_CHUNK;
  if (nch <= 29) return cluster_fits(1, N) ? 1 : 0;
  if (nch <= 121 && cluster_fits(2, N)) return 2;
  return cluster_fits(3, N) ? 3 : 0;
}

// Which kernel solves the unsigned recursions: SOLVE_AUTO picks by size
// (a choice recorded for this N by set_solve_choice, else the cluster from
// five chunks on), SOLVE_BLOCK forces k_tri_solve_b, SOLVE_CLUSTER forces
// k_tri_solve_c.  Both give the same unknowns to rounding.
static std::atomic<int> g_solve_force{SOLVE_AUTO};
static std::mutex g_solve_mu;
static std::vector<std::pair<int, int>> g_solve_choice;  // (N, path)

void set_solve_path(int path) { g_solve_force = path; }
int solve_path() { return g_solve_force; }
void set_solve_choice(int N, int path) {
  std::lock_guard<std::mutex> lk(g_solve_mu);
  for (auto &c : g_solve_choice)
    if (c.first == N) {
      c.second = path;
      return;
    }
  g_solve_choice.emplace_back(N, path);
}
int solve_choice(int N) {
  const int forced = g_solve_force;
  if (forced != SOLVE_AUTO) return forced;
  {
    std::lock_guard<std::mutex> lk(g_solve_mu);
    for (const auto &c : g_solve_choice)
      if (c.first == N) return c.second;
  }
  // the cluster pays off from five chunks on; below that (and in ensembles
  // of small systems) one block per direction leaves the SMs to the other
  // systems
  return (N + TS_CHUNK - 1) / TS_CHUNK > 4 ? SOLVE_CLUSTER : SOLVE_BLOCK;
}

// the cluster variant that the unsigned solve of N takes (0: the block solve);
// *bad: the cluster was forced, but none fits
static int takes_cluster(int N, bool *bad) {
  const bool want = solve_choice(N) == SOLVE_CLUSTER;
  const int v = want ? cluster_variant(N) : 0;
  *bad = want && !v && g_solve_force == SOLVE_CLUSTER;
  return v;
}

bool solve_by_cluster(int N) {
  bool bad;
  return takes_cluster(N, &bad) != 0;
}

static cudaError_t tri_solve(int N, double beta, const TriJob &job, int first, int count, cudaStream_t st,
                             int cluster = 0) {
  if (!job.sign) {
    // unsigned weights: the block solve (the diagonal-block inverses came
    // with the weights, k_weights_inv)
    if (cluster) {
      {
        XK_PROF(count == 2 ? "vb_tv_solve" : (first ? "tv_solve" : "vb_solve"));
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        const ClusterKernel &k = g_cluster_kernels[cluster];
        cluster_config(k, N, count, st, cfg, attr);
        const cudaError_t e = cudaLaunchKernelEx(&cfg, k.fn, N, beta, job, first);
        if (e != cudaSuccess) return e;
      }
      return XK_LAUNCHED();
    }
    const size_t smem = (sizeof(double) + sizeof(int)) * (N + 1 + 2 * TS_CHUNK + 2 * TS_CHUNK * TS_LD) + 16;
    static bool opted_b = false;
    if (!opted_b) {
      cudaError_t ea = cudaFuncSetAttribute(k_tri_solve_b, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (ea != cudaSuccess) return ea;
      opted_b = true;
    }
    {
      XK_PROF(count == 2 ? "vb_tv_solve" : (first ? "tv_solve" : "vb_solve"));
      k_tri_solve_b<<<count, TSB_WARPS * 32, smem, st>>>(N, beta, job, first);
    }
    return XK_LAUNCHED();
  }
  const size_t smem = (sizeof(double) + sizeof(int)) * (N + 1 + 2 * TS_CHUNK + 4 * TS_CHUNK * TS_LD) + 16;
  static bool opted = false;
  if (!opted) {
    cudaError_t ea = cudaFuncSetAttribute(k_tri_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (ea != cudaSuccess) return ea;
    opted = true;
  }
  {
    XK_PROF(count == 2 ? "vb_tv_solve" : (first ? "tv_solve" : "vb_solve"));
    k_tri_solve<<<count, TS_WARPS * 32, smem, st>>>(N, beta, job, first);
  }
  return XK_LAUNCHED();
}

TriJob tri_job(int N, double *rs_f, double *rs_b, double *VBN, double *tmpV) {
  TriJob j{};
  const size_t boff = ntri(N) + (ntri(N) + 1) / 2 + 1;
  const size_t nb = (size_t)((N + TS_CHUNK - 1) / TS_CHUNK) * TS_CHUNK * TS_CHUNK;
  double *rs[2] = {rs_f, rs_b};
  for (int d = 0; d < 2; ++d) {
    if (!rs[d]) continue;
    double *b = rs[d] + boff;
    j.Bm[d] = b;
    j.Be[d] = (int *)(b + nb);
    j.Wm[d] = b + nb + nb / 2;
    j.We[d] = (int *)(j.Wm[d] + nb);
    j.Xm[d] = (long long *)(j.Wm[d] + nb + nb / 2);
    j.Xe[d] = (int *)(j.Xm[d] + N + 2);
    j.Sm[d] = (double *)j.Xm[d] + N + 2 + (N + 3) / 2;
  }
  j.Mm[0] = rs_f;
  j.Me[0] = (const int *)(rs_f + ntri(N));
  j.out[0] = VBN;
  j.Mm[1] = rs_b;
  j.Me[1] = (const int *)(rs_b + ntri(N));
  j.out[1] = tmpV;
  return j;
}

// unsigned weights of directions first .. first + count - 1 with their
// diagonal blocks' inverses (count = 2: first = 0), then the solve
static cudaError_t weights_solve(int N, double beta, double vi, const double *ENk, const double *lnn,
                                 const TriJob &job, int first, int count, cudaStream_t st) {
  const double lnvi = vi != 0.0 ? log(vi) : 0.0;
  bool bad;
  const int cluster = takes_cluster(N, &bad);
  if (bad) return cudaErrorInvalidConfiguration;
  const int groups = cluster ? 16 : 8, nch = (N + TS_CHUNK - 1) / TS_CHUNK;  // four columns of B or W a block
  {
    XK_PROF("weights");
    k_weights_inv<<<N + count * nch * groups, 128, 0, st>>>(N, beta, vi, lnvi, ENk, lnn, job, first,
                                                           count == 2 ? 1 : 0, groups);
  }
  const cudaError_t e = XK_LAUNCHED();
  return e == cudaSuccess ? tri_solve(N, beta, job, first, count, st, cluster) : e;
}

cudaError_t fill_vb(int N, double beta, double vi, const double *ENk, const double *lnn, double *VBN, double *rs,
                    cudaStream_t st) {
  return weights_solve(N, beta, vi, ENk, lnn, tri_job(N, rs, nullptr, VBN, nullptr), 0, 1, st);
}

cudaError_t back_vb(int N, double beta, double vi, const double *ENk, const double *lnn, double *tmpV, double *rs,
                    cudaStream_t st) {
  return weights_solve(N, beta, vi, ENk, lnn, tri_job(N, nullptr, rs, nullptr, tmpV), 1, 1, st);
}

cudaError_t fill_vb_tv(int N, double beta, double vi, const double *ENk, const double *lnn, double *VBN,
                       double *tmpV, double *rs_f, double *rs_b, cudaStream_t st) {
  return weights_solve(N, beta, vi, ENk, lnn, tri_job(N, rs_f, rs_b, VBN, tmpV), 0, 2, st);
}

cudaError_t fill_vb_signed(int N, double beta, double vi2, const double *ENk, const double *lnn, double *V2,
                           double *sign, double *rs, cudaStream_t st) {
  cudaError_t e = weights(N, beta, fabs(vi2), ENk, lnn, rs, nullptr, 0, 1, st, vi2 < 0 ? -1 : 1);
  if (e != cudaSuccess) return e;
  TriJob j = tri_job(N, rs, nullptr, V2, nullptr);
  j.sign = sign;
  return tri_solve(N, beta, j, 0, 1, st);
}

// connection probabilities G[l][j]: md_pimd_x.c:2660-2673
// G[l][j] (md_pimd_x.c:2588-2620); ln xi comes from the host and 1/l from
// a host table, so an element costs one exponential (exp_fast) on the FP64
// pipe.  The exponent is a difference of numbers of size beta V_B^(N) (up to
// ~1e5 at N = 512), so its rounding sets G's relative accuracy; it is summed
// in the reference's order, ((V_B^(j-1) + E) + tmpV[l]) - V_B^(N), so that the
// two round alike.
__global__ void k_fill_g(int N, double beta, double vi, double lnvi, const double *__restrict__ ENk,
                         const double *__restrict__ VBN, const double *__restrict__ tmpV,
                         const double *__restrict__ invl, double *__restrict__ G) {
  const int l = blockIdx.y + 1;  // 1-based row
  const double tv = tmpV[l], vn = VBN[N];
  for (int j = blockIdx.x * blockDim.x + threadIdx.x + 1; j <= N; j += gridDim.x * blockDim.x) {
    double gv;
    if (j > l + 1)
      gv = 0;
    else if (j == l + 1)
      gv = 1 - exp(-beta * ((VBN[l] + tv) - vn));
    else if (vi == 0.0 && l - j != 0)
      gv = 0;
    else if (vi == 0.0)
      gv = exp_fast(-beta * (((VBN[j - 1] + ENk[dtri(l) + l - j]) + tv) - vn)) * invl[l];
    else
      gv = exp_fast(__dadd_rn(__dmul_rn(-beta, ((VBN[j - 1] + ENk[dtri(l) + l - j]) + tv) - vn),
                              __dmul_rn((double)(l - j), lnvi))) *
           invl[l];
    G[(size_t)(l - 1) * N + (j - 1)] = gv;
  }
}

cudaError_t fill_g(int N, double beta, double vi, const double *ENk, const double *VBN,
                   const double *tmpV, const double *lnn, double *G, cudaStream_t st) {
  const double lnvi = vi != 0.0 ? log(vi) : 0.0;
  dim3 grid((N + 255) / 256, N);
  {
    XK_PROF("fill_g");
    k_fill_g<<<grid, 256, 0, st>>>(N, beta, vi, lnvi, ENk, VBN, tmpV, lnn + N + 1, G);
  }
  return XK_LAUNCHED();
}

// The same G from the extended-range numbers the recursions already hold.
// With Z_n = exp(-beta V_B^(n)) = X_n of the forward solve, exp(-beta tmpV[l])
// = X'_{N-l} of the backward one, and the weight M_{l,j-1} = xi^(l-j)/l
// exp(-beta E_l^(l-j+1)) of the forward triangle,
//   G[l][j] = M_{l,j-1} X_{j-1} X'_{N-l} / X_N        (j <= l)
//   G[l][l+1] = 1 - X_l X'_{N-l} / X_N
// a product of four numbers each held to a few ulps, where the reference's
// exp(-beta(V_B^(j-1) + E + tmpV[l] - V_B^(N))) loses beta V_B^(N) ulps to the
// cancellation inside the exponent (up to ~1e-10 relative at N = 512); k_exch
// below forms it where the springs need it.

// ===================================================================
// exchange-weighted spring forces: md_pimd_x.c:2674-2717
// ===================================================================


// One launch for G and the springs that do not wait for its sums: warps of
// the first `nt` blocks take the tile parts of exch_tile_job (four a block: one
// a scheduler, spread over the SMs), the threads of the others the interior
// beads j = 2..P-1 (1-based).  With k_exch_finish two launches where G, a fill
// of f, the interior, the ends (each spring vector formed once a side) and
// their sums were five: 34 us against 48 (sums of launches timed apart, with
// some 4 us a launch) at N = 512, P = 64, a whole step of N = 64, P = 64 51 us
// against 57; at N = 1600 the FP64 pipe bounds both, 71 and 70 us.  R = 8 rows
// a batch and four parts a tile: two parts 65 us, four 58 at N = 1600.
constexpr int EX_W = 4;
template <int D, bool FROM_G>
__global__ void __launch_bounds__(32 * EX_W) k_exch(Geo g, const double *__restrict__ x, double w2, int image,
                                                    TriJob tj, double *__restrict__ G, double *__restrict__ f,
                                                    double *__restrict__ scr, int nt, int jobs) {
  if ((int)blockIdx.x < nt) {
    const int job = blockIdx.x * EX_W + (threadIdx.x >> 5);
    if (job < jobs) exch_tile_job<D, FROM_G>(g, x, image, tj, G, scr, job, threadIdx.x & 31);
    return;
  }
  const size_t t = (size_t)(blockIdx.x - nt) * blockDim.x + threadIdx.x;
  const int l = (int)(t % g.Ns), j = (int)(t / g.Ns) + 1;  // 0-based bead index 1..P-2
  if (j >= g.P - 1) return;
  if (l < g.N) {
    spring_interior_bead<D>(g, x, w2, image, f, j, l);
  } else {
    for (int d = 0; d < D; ++d) f[sidx(j, d, l, D, g.Ns)] = 0.0;
  }
}

// the end beads, from the tiles' partial sums: 32 x EX_Y threads take 32 beads'
// sums in one coordinate
template <int D>
__global__ void __launch_bounds__(32 * EX_Y) k_exch_finish(Geo g, const double *__restrict__ x, double w2, int image,
                                                           const double *__restrict__ scr, double *__restrict__ f) {
  __shared__ double2 share[EX_Y][32];
  const int t = blockIdx.x * 32 + threadIdx.x, l = t % g.Ns, side = t / g.Ns, d = blockIdx.y;
  if (side < 2 && l < g.N) share[threadIdx.y][threadIdx.x] = exch_end_share<D>(g, scr, side, d, l, threadIdx.y);
  __syncthreads();
  if (threadIdx.y != 0 || side >= 2) return;
  f[sidx(side ? g.P - 1 : 0, d, l, D, g.Ns)] =
      l < g.N ? exch_end_value<D>(g, exch_own_spring(g, x, image, side, d, l), w2, scr, side, d, l,
                                  &share[0][threadIdx.x], 32)
              : 0.0;
}

size_t exch_scratch_doubles(const Geo &g) {
  const size_t T = (g.N + 31) / 32;
  return (T * (exch_parts(g.N) + 1) * g.Ns + T) * (g.D + 1);
}

cudaError_t exch_force(const Geo &g, const double *x, double w2, int image, const double *rs_f, const double *rs_b,
                       double *G, double *f, double *scratch, cudaStream_t st) {
  const int jobs = exch_jobs(g.N), nt = cdiv(jobs, EX_W);
  const int ni = g.P > 2 ? cdiv((size_t)(g.P - 2) * g.Ns, 32 * EX_W) : 0;
  {
    XK_PROF("exch_ends");
    if (rs_f) {
      const TriJob tj = tri_job(g.N, (double *)rs_f, (double *)rs_b, nullptr, nullptr);
      DISPATCH_D(g.D, (k_exch<D, false><<<nt + ni, 32 * EX_W, 0, st>>>(g, x, w2, image, tj, G, f, scratch, nt, jobs)));
    } else {
      DISPATCH_D(g.D, (k_exch<D, true><<<nt + ni, 32 * EX_W, 0, st>>>(g, x, w2, image, TriJob{}, G, f, scratch, nt, jobs)));
    }
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  {
    XK_PROF("exch_finish");
    DISPATCH_D(g.D, k_exch_finish<D><<<dim3(cdiv(2 * g.Ns, 32), g.D), dim3(32, EX_Y), 0, st>>>(g, x, w2, image, scratch, f));
  }
  return XK_LAUNCHED();
}

// ===================================================================
// trap: md_pimd_x.c:1297-1391 (CPU :1370-1389), md_simulation_x.c:127-159
// ===================================================================


// f += V'(x) / P, the 1/P from the host (a product instead of an FP64
// division per DOF; equal to rounding)
__global__ void k_trap_force(Geo g, TrapPrm p, const double *__restrict__ x,
                             double *__restrict__ f, double invP) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.slots() || (int)(s % g.Ns) >= g.N) return;
  const int d = (int)((s / g.Ns) % g.D);
  f[s] += trap_f(p, d, x[s]) * invP;
}

cudaError_t trap_force(const Geo &g, const TrapPrm &p, const double *x, double *f,
                       cudaStream_t st) {
  {
    XK_PROF("trap_force");
    k_trap_force<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, p, x, f, 1.0 / g.P);
  }
  return XK_LAUNCHED();
}

// deterministic final reduction of per-block partial sums into *acc
__global__ void k_reduce_into(const double *__restrict__ part, int n, double scale, double add,
                              double *acc) {
  __shared__ double buf[33];
  double s = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
  s = block_sum(s, buf);
  if (threadIdx.x == 0) *acc += s * scale + add;
}

static cudaError_t reduce_into(const double *part, int n, double scale, double add, double *acc,
                               cudaStream_t st) {
  {
    XK_PROF("reduce_into");
    k_reduce_into<<<1, 256, 0, st>>>(part, n, scale, add, acc);
  }
  return XK_LAUNCHED();
}

// md_statistics_x.c:322-338 energies
template <int D>
__global__ void k_trap_energy(Geo g, TrapPrm p, const double *__restrict__ x,
                              const double *__restrict__ m, double *part) {
  __shared__ double buf[33];
  double e = 0;
  for (size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x; b < (size_t)g.N * g.P;
       b += (size_t)gridDim.x * blockDim.x) {
    const int l = (int)(b % g.N), j = (int)(b / g.N);
    const double mm = m[(size_t)j * g.Ns + l];
    if (p.kind == TRAP_HARMONIC_2) {
      double r = 0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double t = x[sidx(j, d, l, D, g.Ns)] - p.c[d];
        r += 0.5 * mm * p.w2[d] * p.w2[d] * t * t;
      }
      e += r;
    } else {
      double r2 = 0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double t = x[sidx(j, d, l, D, g.Ns)] - p.c[d];
        r2 += t * t;
      }
      const double v = 0.5 * mm * p.w * p.w * r2;
      e += p.kind == TRAP_HARMONIC ? v : -v;
    }
  }
  e = block_sum(e, buf);
  if (threadIdx.x == 0) part[blockIdx.x] = e;
}

cudaError_t trap_energy(const Geo &g, const TrapPrm &p, const double *x, const double *m,
                        double *acc, double *scratch, cudaStream_t st) {
  int nb = cdiv((size_t)g.N * g.P, 256);
  if (nb > 304) nb = 304;
  {
    XK_PROF("trap_energy");
    DISPATCH_D(g.D, k_trap_energy<D><<<nb, 256, 0, st>>>(g, p, x, m, scratch));
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  return reduce_into(scratch, nb, 1.0 / g.P, 0.0, acc, st);
}

// ===================================================================
// pair forces and energies per bead slice: md_pimd_x.c:1527-1677
// (CPU :1650-1675) and :1679-1824, potentials md_simulation_x.c:166-293,
// md_statistics_x.c:340-396.
//
// One warp evaluates a 32 x 32 tile (I, J), I <= J, of one slice: lane i
// keeps particle a = 32I + i; the partner data (position, mass, reaction
// force) rotates through the lanes, so every unordered pair is evaluated
// once and both forces are kept in registers.  Each particle's force from
// the tiles of partner block t lands in scratch slot t exactly once; the
// finishing kernel sums the slots in a fixed order and adds (sum)/P.
// ===================================================================

__constant__ double c_ew_h[EW_NINT][EW_DEG + 1] = EW_H_INIT;
constexpr size_t EW_TAB_BYTES = sizeof(double) * 2 * EW_NINT * (EW_DEG + 1);
__constant__ double c_ew_erfc[EW_NINT][EW_DEG + 1] = EW_ERFC_INIT;

// Force F(dx) (times the pair's strength, before the 1/m and 1/P factors)
// and, with want_e, the pair energy.  The Ewald kind is warp-collective: all
// lanes call it, `active` says whether the lane's pair counts.
// per-warp queue of accepted Ewald images (shared memory)
constexpr int EW_TAKE = 4;  // images per lane per batch
struct EwWarp {
  double cm[32][9];          // each lane's candidate components m_d - k L_d
  double val[32 * EW_TAKE];  // evaluated factor per queue item
  unsigned take[32];         // each lane's images in this batch (bit = k code)
  int base[32];              // first queue item of each lane
};

// Ewald forces (not energies) come back without the strength p.qs, which
// the kernels fold into the inverse masses: F the FP64 images' sum, G the
// FP32 sum of the far images (alpha R >= p.xsplit).
template <int D, int KIND, bool ENERGY_TAB>
__device__ inline void pair_eval(const PairPrm &p, const Geo &g, const double *dx, const float *dxf,
                                 double *F, double &E, bool want_e, const double *tabs, bool active,
                                 EwWarp *ws, int lane, float *G = nullptr) {
  if (KIND == PAIR_GAUSSIAN || KIND == PAIR_PERIODIC_GAUSSIAN) {
    double t[D], r2 = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      t[d] = dx[d];
      if (KIND == PAIR_PERIODIC_GAUSSIAN) t[d] = min_image(t[d], g.box[d], g.inv_box[d]);
      r2 += t[d] * t[d];
    }
    // r^2 / s^2 by the reciprocal and one residual step (a correctly rounded
    // quotient without an FP64 division), the exponential on the integer
    // pipe: about 15 FP64 instructions a pair where exp() and four divisions
    // took over a hundred
    const double q = r2 * p.is2;
    double a = fma(fma(-q, p.s * p.s, r2), p.is2, q);
    if ((__double2hiint(a) & 0x7ff00000) == 0x7ff00000) a = q;  // r^2 or s^2 beyond the range: no residual
    const double ex = exp_fast(-a);
    const double mult = p.g2 * ex;
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] = mult * t[d];
    if (want_e) E = p.g0 * ex;
  } else if (KIND == PAIR_COULOMB || KIND == PAIR_PERIODIC_COULOMB) {
    double t[D], r2 = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      t[d] = dx[d];
      if (KIND == PAIR_PERIODIC_COULOMB) t[d] = min_image(t[d], g.box[d], g.inv_box[d]);
      r2 += t[d] * t[d];
    }
    const double r = sqrt(r2);
    const double mult = p.qs / (r2 * r);
#pragma unroll
    for (int d = 0; d < D; ++d) F[d] = mult * t[d];
    if (want_e) E = p.qs / r;
  } else if (KIND == PAIR_EWALD_REAL) {
    // Real-space images of the partner inside the reference's cube
    // |n_i| <= nsum (md_simulation_x.c:281-292) whose distance is below
    // rcut.  dx is first reduced to its minimum image m = dx - s L, so the
    // candidates are n = s + k with |k_d| <= 1.  The candidates are culled
    // on the FP32 pipe into a bit mask (with a 1e-4 margin; the FP64 test
    // below decides), then evaluated in warp-wide rounds, one accepted image
    // per lane per round, so that the FP64 pipe runs with full warps.  Per
    // image the factor (erfc(x) + 2x exp(-x^2)/sqrt(pi)) / R^3, x = alpha R,
    // comes from the piecewise polynomial EW_H (no FP64 erfc or exp), 1/R
    // from rsqrt.  On this GPU FP64 comparisons and int <-> double
    // conversions share the slow FP64 pipe, so rounding to integers uses
    // the 1.5 * 2^52 addition and the cut-off test compares bit patterns.
    // Forces only: images at alpha R >= p.xsplit (55% of those inside rcut
    // at alpha rcut = 5.2, xsplit = 4) go to the FP32 pipe instead,
    // through ew_h32, and their sum joins the FP64 one per pair.
    constexpr double MAGIC = 6755399441055744.0;  // 1.5 * 2^52
    const double *tab = ENERGY_TAB ? tabs + EW_NINT * (EW_DEG + 1) : tabs;
    const long long rc2_bits = __double_as_longlong(p.rc2);
    double mm[3];
    int sh[3];
    unsigned mask = 0u, far = 0u;
    // FP32 minimum image (from the FP32 positions): the culling, and the far
    // images' evaluation
    const float L0 = p.boxf[0], L1 = p.boxf[1], L2 = p.boxf[2];
    float m0 = 0.f, m1 = 0.f, m2 = 0.f;
    if (active) {
      if (ENERGY_TAB) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double tq = fma(dx[d], g.inv_box[d], MAGIC);  // MAGIC + rint(dx/L)
          sh[d] = __double2loint(tq);
          mm[d] = fma(-(tq - MAGIC), g.box[d], dx[d]);
        }
      } else {
        // forces: the shift from the FP32 separation (near a half box either
        // image is a valid centre: the candidates reach one box further
        // either way, and alpha rcut <= 5.2 keeps rcut below 1.35 L), and
        // m = dx - s L by one FP64 addition of -L, 0 or L
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          sh[d] = __float2int_rn(dxf[d] * p.iboxf[d]);
          double sel = 0.0;
          if (sh[d] == 1) {
            sel = -g.box[d];
          } else if (sh[d] == -1) {
            sel = g.box[d];
          } else if (sh[d] != 0) {
            sel = -(double)sh[d] * g.box[d];
          }
          mm[d] = dx[d] + sel;
        }
      }
      m0 = fmaf(-(float)sh[0], L0, dxf[0]);
      m1 = fmaf(-(float)sh[1], L1, dxf[1]);
      m2 = fmaf(-(float)sh[2], L2, dxf[2]);
#pragma unroll
      for (int c = 0; c < 27; ++c) {
        const int k0 = c / 9 - 1, k1 = (c / 3) % 3 - 1, k2 = c % 3 - 1;
        const float t0 = fmaf(-(float)k0, L0, m0), t1 = fmaf(-(float)k1, L1, m1), t2 = fmaf(-(float)k2, L2, m2);
        const float r2 = fmaf(t2, t2, fmaf(t1, t1, t0 * t0));
        const bool in_cube = abs(sh[0] + k0) <= p.nsum && abs(sh[1] + k1) <= p.nsum && abs(sh[2] + k2) <= p.nsum;
        if (!ENERGY_TAB && r2 >= p.xs2f) {
          // a far image (alpha R >= xsplit): FP32, cut at rcut in FP32
          if (r2 < p.rcf2 && in_cube) far |= 1u << c;
        } else if (r2 < p.rcf2_cull && in_cube) {
          mask |= 1u << c;
        }
      }
    }
    // far images on the FP32 pipe, each lane its own (their h(alpha R) is
    // below 5.2e-7, so FP32's relative error of a few 1e-6 leaves a few
    // 1e-13 of the force in all)
    if (!ENERGY_TAB) {
      float G0 = 0.f, G1 = 0.f, G2 = 0.f;
      unsigned fr = far;
      while (fr) {
        const int c = __ffs(fr) - 1;
        fr &= fr - 1;
        const float t0 = fmaf(-(float)(c / 9 - 1), L0, m0);
        const float t1 = fmaf(-(float)((c / 3) % 3 - 1), L1, m1);
        const float t2 = fmaf(-(float)(c % 3 - 1), L2, m2);
        const float v = ew_h32(fmaf(t2, t2, fmaf(t1, t1, t0 * t0)), p.alphaf);
        G0 = fmaf(t0, v, G0);
        G1 = fmaf(t1, v, G1);
        G2 = fmaf(t2, v, G2);
      }
      G[0] = G0, G[1] = G1, G[2] = G2;
    }
    double F0 = 0, F1 = 0, F2 = 0, e = 0;
    // the three candidate components per axis, m - k L for k = -1, 0, 1
    double cm[9];
    if (mask) {
      cm[0] = mm[0] + g.box[0], cm[1] = mm[0], cm[2] = mm[0] - g.box[0];
      cm[3] = mm[1] + g.box[1], cm[4] = mm[1], cm[5] = mm[1] - g.box[1];
      cm[6] = mm[2] + g.box[2], cm[7] = mm[2], cm[8] = mm[2] - g.box[2];
#pragma unroll
      for (int q = 0; q < 9; ++q) ws->cm[lane][q] = cm[q];
    }
    // Accepted images are evaluated as one queue per warp: batches of up to
    // four images per lane, every lane evaluating consecutive queue items, so
    // that the FP64 pipe runs with (nearly) full warps whatever the number of
    // images of each lane's pair.  The owner lane then accumulates its own.
    unsigned rem = mask;
    while (__any_sync(FULL, rem != 0u)) {
      unsigned take = 0u, t = rem;
#pragma unroll
      for (int i = 0; i < EW_TAKE; ++i) {
        const unsigned b = t & (0u - t);
        take |= b;
        t ^= b;
      }
      rem ^= take;
      const int cnt = __popc(take);
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      const int base = incl - cnt, total = __shfl_sync(FULL, incl, 31);
      ws->take[lane] = take;
      ws->base[lane] = base;
      __syncwarp();
      for (int round = 0; round < total; round += 32) {
        const int q = round + lane;
        if (q >= total) continue;
        int o = 0;
#pragma unroll
        for (int st = 16; st; st >>= 1)
          if (ws->base[o + st] <= q) o += st;
        unsigned b = ws->take[o];
        for (int r = q - ws->base[o]; r > 0; --r) b &= b - 1;
        const int c = __ffs(b) - 1;
        const int q0 = c / 9, q1 = (c / 3) % 3, q2 = c % 3;
        const double t0 = ws->cm[o][q0], t1 = ws->cm[o][3 + q1], t2 = ws->cm[o][6 + q2];
        const double R2 = fma(t2, t2, fma(t1, t1, t0 * t0));
        double val = 0.0;
        if (__double_as_longlong(R2) < rc2_bits) {
          const double rinv = rsqrt(R2);
          const double xr = p.alpha * (R2 * rinv);
          const double tq = fma(xr, EW_INV_W, MAGIC);  // MAGIC + rint(x/w): interval index
          int iv = __double2loint(tq);
          iv = iv < EW_NINT - 1 ? iv : EW_NINT - 1;
          const double u = fma(xr, 2 * EW_INV_W, fma(-2.0, tq, 2 * MAGIC));  // 2 (x/w - iv)
          const double *cf = tab + iv * (EW_DEG + 1);
          double hv = cf[EW_DEG];
#pragma unroll
          for (int qq = EW_DEG - 1; qq >= 0; --qq) hv = fma(hv, u, cf[qq]);
          val = ENERGY_TAB ? hv * rinv : hv * (rinv * rinv * rinv);
        }
        ws->val[q] = val;
      }
      __syncwarp();
      unsigned b = take;
      for (int i = 0; i < cnt; ++i) {
        const int c = __ffs(b) - 1;
        b &= b - 1;
        const double val = ws->val[base + i];
        if (ENERGY_TAB) {
          e += val;
        } else {
          const int q0 = c / 9, q1 = (c / 3) % 3, q2 = c % 3;
          const double t0 = q0 == 0 ? cm[0] : (q0 == 1 ? cm[1] : cm[2]);
          const double t1 = q1 == 0 ? cm[3] : (q1 == 1 ? cm[4] : cm[5]);
          const double t2 = q2 == 0 ? cm[6] : (q2 == 1 ? cm[7] : cm[8]);
          F0 = fma(t0, val, F0);
          F1 = fma(t1, val, F1);
          F2 = fma(t2, val, F2);
        }
      }
      __syncwarp();
    }
    F[0] = F0;
    if (D > 1) F[1] = F1;
    if (D > 2) F[2] = F2;
    if (want_e) E = p.qs * e;
  }
}

// The Gaussian and Coulomb kinds: a warp takes one of `split` equal parts of a
// 32 x 32 tile's rotation steps (lane l meets bead (l + s) mod 32 of the other
// tile in step s; tiles on the diagonal visit each pair once, steps 1..16),
// so that a small system still gives every SM sub-partition a warp: the
// kernel is bound by the FP64 instructions' latency there, 64 cycles each in
// a dependent chain.  Partials go to slot t * split + part of the other tile
// t (of its own tile on the diagonal), summed by k_pair_finish.
template <int D, int KIND, bool ENERGY>
__global__ void __launch_bounds__(256) k_pair_split(Geo g, PairPrm p, const double *__restrict__ x,
                                                    const double *__restrict__ m, double *__restrict__ out, int T,
                                                    int jobs, int split) {
  const int lane = threadIdx.x & 31, nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int w = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; w < jobs * g.P * split; w += nwarps) {
    const int part = w % split, j = w / split / jobs;
    int job = w / split % jobs, I = 0;
    while (job >= T - I) {
      job -= T - I;
      ++I;
    }
    const int J = I + job;
    const bool diag = I == J;
    const int a = I * 32 + lane, b = J * 32 + lane, nb = min(32, g.N - J * 32);
    const bool va = a < g.N, vb = lane < nb;
    double xa[D], xb[D], fa[D], fb[D], ea = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xa[d] = va ? x[sidx(j, d, a, D, g.Ns)] : 0.0;
      xb[d] = vb ? x[sidx(j, d, b, D, g.Ns)] : 0.0;
      fa[d] = fb[d] = 0.0;
    }
    const double ima = !ENERGY && va ? 1.0 / m[(size_t)j * g.Ns + a] : 1.0;
    const double imb = !ENERGY && vb ? 1.0 / m[(size_t)j * g.Ns + b] : 1.0;
    const int s0 = diag ? 1 + part * 16 / split : part * 32 / split;
    const int s1 = diag ? 1 + (part + 1) * 16 / split : (part + 1) * 32 / split;
    for (int s = s0; s < s1; ++s) {
      if (diag && s >= nb && s + nb <= 32) continue;  // no pair of the tile's nb beads in this step
      const int from = (lane + s) & 31, back = (lane - s) & 31;
      const bool act = va && from < nb && !(diag && s == 16 && lane >= 16);
      double dx[D], F[D], E = 0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        dx[d] = xa[d] - __shfl_sync(FULL, xb[d], from);
        F[d] = 0;
      }
      const double im2 = __shfl_sync(FULL, imb, from);
      if (act) pair_eval<D, KIND, ENERGY>(p, g, dx, nullptr, F, E, ENERGY, nullptr, true, nullptr, lane);
      if constexpr (ENERGY) {
        ea += E;
      } else {
        // the reference divides by the mass of the higher-index particle
        const double inv = a > J * 32 + from ? ima : im2;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          F[d] *= inv;
          fa[d] += F[d];
          fb[d] -= __shfl_sync(FULL, F[d], back);
        }
      }
    }
    if constexpr (ENERGY) {
      ea = warp_sum(ea);
      if (lane == 0) out[w] = ea;
    } else {
      // slot layout: out[((t*P + j)*D + d)*Ns + l]
#pragma unroll
      for (int d = 0; d < D; ++d) {
        if (va) out[(((size_t)(J * split + part) * g.P + j) * D + d) * g.Ns + a] = diag ? fa[d] + fb[d] : fa[d];
        if (vb && !diag) out[(((size_t)(I * split + part) * g.P + j) * D + d) * g.Ns + b] = fb[d];
      }
    }
  }
}

constexpr int PAIR_SPLIT_MAX = 8;
// parts of a tile: enough that every SM sub-partition has two warps (of 152 SMs,
// not the device's: the parts set the order of the sums)
static int pair_split(const Geo &g, int jobs) {
  int split = 1;
  while (split < PAIR_SPLIT_MAX && (size_t)jobs * g.P * split < 2 * 4 * 152) split *= 2;
  return split;
}

// real-space Ewald (3D): a warp per tile, partner data rotated through the lanes
template <bool ENERGY>
__global__ void __launch_bounds__(256, 2) k_pair_tiles(Geo g, PairPrm p,
                                                    const double *__restrict__ x,
                                                    const double *__restrict__ m,
                                                    double *__restrict__ out, int T, int jobs) {
  constexpr int D = 3, KIND = PAIR_EWALD_REAL;
  // Ewald polynomial tables staged in shared memory (lanes index them freely)
  extern __shared__ double stab[];  // the two tables (EW_TAB_BYTES of dynamic shared memory)
  {
    for (int i = threadIdx.x; i < 2 * EW_NINT * (EW_DEG + 1); i += blockDim.x)
      stab[i] = i < EW_NINT * (EW_DEG + 1) ? (&c_ew_h[0][0])[i] : (&c_ew_erfc[0][0])[i - EW_NINT * (EW_DEG + 1)];
    __syncthreads();
  }
  __shared__ EwWarp ewq[8];
  EwWarp *ews = &ewq[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  // warps loop over the tile jobs (slice j, tile pair I <= J) round-robin, so
  // that a grid of resident blocks (pair_launch) stages the tables once.  The
  // warps are numbered across blocks first: the jobs of the last, partial
  // round spread over all blocks (and SMs) instead of filling the first ones.
  for (int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; warp < jobs * g.P; warp += nwarps) {
    const int j = warp / jobs;
    int job = warp % jobs, I = 0;
    while (job >= T - I) {
      job -= T - I;
      ++I;
    }
    const int J = I + job;
    const int a = I * 32 + lane, b0 = J * 32 + lane;
    const bool va = a < g.N, vb = b0 < g.N;
    double xa[D], xb[D], fa[D], fb[D];
    float xaf[D], xbf[D];  // FP32 copies for the Ewald image culling
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xa[d] = va ? x[sidx(j, d, a, D, g.Ns)] : 0.0;
      xb[d] = vb ? x[sidx(j, d, b0, D, g.Ns)] : 0.0;
      xaf[d] = (float)xa[d];
      xbf[d] = (float)xb[d];
      fa[d] = fb[d] = 0.0;
    }
    // inverse masses, so that each pair multiplies instead of dividing
    // (Ewald forces: times the strength, and FP32 copies for the far images)
    constexpr bool EWF = !ENERGY;
    const double ima = (!ENERGY && va) ? (EWF ? p.qs : 1.0) / m[(size_t)j * g.Ns + a] : 1.0;
    double imb = (!ENERGY && vb) ? (EWF ? p.qs : 1.0) / m[(size_t)j * g.Ns + b0] : 1.0;
    const float ima32 = EWF ? (float)ima : 0.f;
    float imb32 = EWF ? (float)imb : 0.f;
    float ga[3] = {0.f, 0.f, 0.f}, gb[3] = {0.f, 0.f, 0.f};  // far images' forces (FP32)
    double ea = 0;
    for (int s = 0; s < 32; ++s) {
      const int bi = J * 32 + ((lane + s) & 31);
      const bool act = va && bi < g.N && (I != J || a > bi);
      double dx[D], F[D], E = 0;
      float dxf[D], G[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int d = 0; d < D; ++d) {
        dx[d] = xa[d] - xb[d];
        dxf[d] = xaf[d] - xbf[d];
        F[d] = 0;
      }
      pair_eval<D, KIND, ENERGY>(p, g, dx, dxf, F, E, ENERGY, stab, act, ews, lane, G);
      if (act) {
        if (ENERGY) {
          ea += E;
        } else {
          // the reference divides by the mass of the higher-index particle
          const double inv = a > bi ? ima : imb;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            fa[d] += F[d] * inv;
            fb[d] -= F[d] * inv;
          }
          if (EWF) {
            const float inv32 = a > bi ? ima32 : imb32;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              ga[d] = fmaf(G[d], inv32, ga[d]);
              gb[d] = fmaf(-G[d], inv32, gb[d]);
            }
          }
        }
      }
      const int src = (lane + 1) & 31;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        xb[d] = __shfl_sync(FULL, xb[d], src);
        xbf[d] = __shfl_sync(FULL, xbf[d], src);
        if (!ENERGY) fb[d] = __shfl_sync(FULL, fb[d], src);
        if (EWF) gb[d] = __shfl_sync(FULL, gb[d], src);
      }
      if (!ENERGY) imb = __shfl_sync(FULL, imb, src);
      if (EWF) imb32 = __shfl_sync(FULL, imb32, src);
    }
    if (ENERGY) {
      ea = warp_sum(ea);
      if (lane == 0) out[warp] = ea;
      continue;
    }
    if (EWF) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        fa[d] += (double)ga[d];
        fb[d] += (double)gb[d];
      }
    }
    // slot layout: out[((t*P + j)*D + d)*Ns + l]
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
}

__global__ void k_pair_finish(Geo g, const double *__restrict__ part, int T, double scale,
                              double *__restrict__ f) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t S = g.slots();
  if (s >= S || (int)(s % g.Ns) >= g.N) return;
  double acc = 0;
  for (int t = 0; t < T; ++t) acc += part[(size_t)t * S + s];
  f[s] += acc * scale;
}

// ===================================================================
// two species: md_pimd_calc_pair_force_2_x / _energy_2_x (md_pimd_x.c:
// 3282-3632).  Every bead of species a meets every bead of species b in the
// same slice.  A warp takes the rectangular tile (a-tile I, b-tile J) of one
// slice; a's beads stay in the lanes and b's rotate through them with their
// accumulated forces, as in k_pair_tiles but without the triangle.  The
// reference's callback divides by a's mass and gives b -m_a F/(m_b P), so
// a gains F/(m_a P) and b loses F/(m_b P).  Partials go per partner tile:
//   outa[((J*P + j)*D + d)*Ns_a + l],  outb[((I*P + j)*D + d)*Ns_b + l]
// ===================================================================
template <int D, int KIND, bool ENERGY>
__global__ void __launch_bounds__(256, 2) k_pair_cross(Geo ga, Geo gb, PairPrm p, const double *__restrict__ xa,
                                                    const double *__restrict__ ma, const double *__restrict__ xb,
                                                    const double *__restrict__ mb, double *__restrict__ outa,
                                                    double *__restrict__ outb, int TA, int TB) {
  extern __shared__ double stab[];  // Ewald: the two tables (EW_TAB_BYTES of dynamic shared memory)
  if (KIND == PAIR_EWALD_REAL) {
    for (int i = threadIdx.x; i < 2 * EW_NINT * (EW_DEG + 1); i += blockDim.x)
      stab[i] = i < EW_NINT * (EW_DEG + 1) ? (&c_ew_h[0][0])[i] : (&c_ew_erfc[0][0])[i - EW_NINT * (EW_DEG + 1)];
    __syncthreads();
  }
  __shared__ EwWarp ewq[KIND == PAIR_EWALD_REAL ? 8 : 1];
  EwWarp *ews = &ewq[KIND == PAIR_EWALD_REAL ? (threadIdx.x >> 5) : 0];
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int jobs = TA * TB;
  // warps numbered across blocks first, as in k_pair_tiles
  for (int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; warp < jobs * ga.P; warp += nwarps) {
    const int j = warp / jobs, job = warp % jobs;
    const int I = job / TB, J = job % TB;
    const int a = I * 32 + lane, b0 = J * 32 + lane;
    const bool va = a < ga.N, vb = b0 < gb.N;
    double xa_[D], xb_[D], fa[D], fb[D];
    float xaf[D], xbf[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xa_[d] = va ? xa[sidx(j, d, a, D, ga.Ns)] : 0.0;
      xb_[d] = vb ? xb[sidx(j, d, b0, D, gb.Ns)] : 0.0;
      xaf[d] = (float)xa_[d];
      xbf[d] = (float)xb_[d];
      fa[d] = fb[d] = 0.0;
    }
    // inverse masses (Ewald forces: times the strength, and FP32 copies)
    constexpr bool EWF = KIND == PAIR_EWALD_REAL && !ENERGY;
    const double ima = (!ENERGY && va) ? (EWF ? p.qs : 1.0) / ma[(size_t)j * ga.Ns + a] : 1.0;
    double imb = (!ENERGY && vb) ? (EWF ? p.qs : 1.0) / mb[(size_t)j * gb.Ns + b0] : 1.0;
    const float ima32 = EWF ? (float)ima : 0.f;
    float imb32 = EWF ? (float)imb : 0.f;
    float gfa[3] = {0.f, 0.f, 0.f}, gfb[3] = {0.f, 0.f, 0.f};  // far images' forces (FP32)
    double ea = 0;
    for (int s = 0; s < 32; ++s) {
      const int bi = J * 32 + ((lane + s) & 31);
      const bool act = va && bi < gb.N;
      double dx[D], F[D], E = 0;
      float dxf[D], G[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int d = 0; d < D; ++d) {
        dx[d] = xa_[d] - xb_[d];
        dxf[d] = xaf[d] - xbf[d];
        F[d] = 0;
      }
      if (KIND == PAIR_EWALD_REAL) pair_eval<D, KIND, ENERGY>(p, ga, dx, dxf, F, E, ENERGY, stab, act, ews, lane, G);
      if (act) {
        if (KIND != PAIR_EWALD_REAL)
          pair_eval<D, KIND, ENERGY>(p, ga, dx, dxf, F, E, ENERGY, stab, true, nullptr, lane);
        if (ENERGY) {
          ea += E;
        } else {
#pragma unroll
          for (int d = 0; d < D; ++d) {
            fa[d] += F[d] * ima;
            fb[d] -= F[d] * imb;
          }
          if (EWF) {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              gfa[d] = fmaf(G[d], ima32, gfa[d]);
              gfb[d] = fmaf(-G[d], imb32, gfb[d]);
            }
          }
        }
      }
      const int src = (lane + 1) & 31;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        xb_[d] = __shfl_sync(FULL, xb_[d], src);
        if (KIND == PAIR_EWALD_REAL) xbf[d] = __shfl_sync(FULL, xbf[d], src);
        if (!ENERGY) fb[d] = __shfl_sync(FULL, fb[d], src);
        if (EWF) gfb[d] = __shfl_sync(FULL, gfb[d], src);
      }
      if (!ENERGY) imb = __shfl_sync(FULL, imb, src);
      if (EWF) imb32 = __shfl_sync(FULL, imb32, src);
    }
    if (ENERGY) {
      ea = warp_sum(ea);
      if (lane == 0) outa[warp] = ea;
      continue;
    }
    if (EWF) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        fa[d] += (double)gfa[d];
        fb[d] += (double)gfb[d];
      }
    }
    if (va) {
#pragma unroll
      for (int d = 0; d < D; ++d) outa[(((size_t)J * ga.P + j) * D + d) * ga.Ns + a] = fa[d];
    }
    if (vb) {
#pragma unroll
      for (int d = 0; d < D; ++d) outb[(((size_t)I * gb.P + j) * D + d) * gb.Ns + b0] = fb[d];
    }
  }
}

size_t pair_scratch_doubles(const Geo &g) {
  const int T = (g.N + 31) / 32;
  const size_t jobs = (size_t)T * (T + 1) / 2;
  // partial slots (doubles, or float2 in the FP32 form), then room for the
  // FP32 form's copies of the positions and inverse masses
  size_t a = (size_t)T * g.slots() + (g.slots() + (size_t)g.P * g.Ns + 1) / 2 + 1;
  const int split = pair_split(g, (int)jobs);
  if (a < (size_t)T * split * g.slots()) a = (size_t)T * split * g.slots();
  const size_t d = g.D == 3 ? (size_t)T * ewd_split(jobs * g.P) * g.slots() + 1 + ewd_pos_doubles(g) : 0;
  if (d > a) a = d;
  size_t b = jobs * g.P * split;
  return a > b ? a : b;
}

// resident blocks of a kernel of 256 threads (the persistent grid), or fewer
// when the warps needed run out
template <class K>
static int resident_grid(K kernel, size_t warps_needed, int &occ, int &sms, size_t dyn = 0) {
  if (!occ) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // static plus dynamic shared memory above 48 KB needs the opt-in
    if (dyn > 0) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, 256, dyn) != cudaSuccess || occ < 1) occ = 1;
    if (sms < 1) sms = 1;
  }
  const size_t need = (warps_needed + 7) / 8, full = (size_t)sms * occ;
  return (int)(need < full ? need : full);
}

// choices of the FP64 autotuner per system shape (what, kind, D, N, P)
static std::mutex g_tune64_mu;
static std::vector<std::pair<std::array<int, 5>, int>> g_tune64;

void set_tuning(int what, int kind, int D, int N, int P, int v) {
  std::lock_guard<std::mutex> lk(g_tune64_mu);
  for (auto &e : g_tune64)
    if (e.first == std::array<int, 5>{what, kind, D, N, P}) {
      e.second = v;
      return;
    }
  g_tune64.push_back({{what, kind, D, N, P}, v});
}

int tuning(int what, int kind, int D, int N, int P) {
  std::lock_guard<std::mutex> lk(g_tune64_mu);
  for (auto &e : g_tune64)
    if (e.first == std::array<int, 5>{what, kind, D, N, P}) return e.second;
  return 0;
}

// the FP64 Ewald tiles' persistent grid: blocks per SM as tuned for this
// shape (TUNE_PAIR64_BPS), else as many as stay resident
template <bool ENERGY>
static int pair_grid(size_t warps_needed, const Geo &g) {
  static int occ = 0, sms = 0;
  const int full = resident_grid(k_pair_tiles<ENERGY>, warps_needed, occ, sms, EW_TAB_BYTES);
  const int bps = tuning(TUNE_PAIR64_BPS, PAIR_EWALD_REAL, 3, g.N, g.P);
  if (bps > 0 && bps < occ) return full < sms * bps ? full : sms * bps;
  return full;
}

// the kernels' derived constants (PairPrm::rc2 ... g2), computed once per
// launch instead of per pair
PairPrm with_far_images(const PairPrm &p, const Geo &g) {
  PairPrm q = p;
  if (p.kind == PAIR_GAUSSIAN || p.kind == PAIR_PERIODIC_GAUSSIAN) {  // (the range enters squared: any sign)
    q.is2 = 1.0 / (p.s * p.s);
    q.g0 = p.g / (M_PI * p.s * p.s);
    q.g2 = q.g0 * 2 / (p.s * p.s);
  }
  q.rc2 = p.rcut * p.rcut;
  q.alphaf = (float)p.alpha;
  q.rcf2 = (float)q.rc2;
  q.rcf2_cull = (float)(q.rc2 * 1.0001);
  q.xs2f = FLT_MAX;
  if (p.xsplit > 0 && p.alpha > 0) q.xs2f = (float)((p.xsplit / p.alpha) * (p.xsplit / p.alpha));
  for (int d = 0; d < 3; ++d) {
    q.boxf[d] = (float)g.box[d];
    q.iboxf[d] = (float)g.inv_box[d];
  }
  return q;
}

template <int D, int KIND, bool ENERGY>
static void launch_split(const Geo &g, const PairPrm &p, const double *x, const double *m, double *out, int T, int jobs,
                         int split, cudaStream_t st) {
  static int occ = 0, sms = 0;
  const int full = resident_grid(k_pair_split<D, KIND, ENERGY>, (size_t)jobs * g.P * split, occ, sms);
  const int bps = tuning(TUNE_PAIR64_BPS, KIND, D, g.N, g.P);
  const int grid = bps > 0 && bps < occ && full > sms * bps ? sms * bps : full;
  k_pair_split<D, KIND, ENERGY><<<grid, 256, 0, st>>>(g, p, x, m, out, T, jobs, split);
}

// split: parts of a tile (all but Ewald)
template <int D, bool ENERGY>
static cudaError_t pair_launch(const Geo &g, const PairPrm &p_in, const double *x, const double *m,
                               double *out, int T, int jobs, int split, cudaStream_t st) {
  const PairPrm p = with_far_images(p_in, g);
  const size_t warps = (size_t)jobs * g.P;
  switch (p.kind) {
    case PAIR_GAUSSIAN: {
      XK_PROF("pair_tiles_gauss");
      launch_split<D, PAIR_GAUSSIAN, ENERGY>(g, p, x, m, out, T, jobs, split, st);
      break;
    }
    case PAIR_PERIODIC_GAUSSIAN: {
      XK_PROF("pair_tiles_pgauss");
      launch_split<D, PAIR_PERIODIC_GAUSSIAN, ENERGY>(g, p, x, m, out, T, jobs, split, st);
      break;
    }
    case PAIR_COULOMB: {
      XK_PROF("pair_tiles_coul");
      launch_split<D, PAIR_COULOMB, ENERGY>(g, p, x, m, out, T, jobs, split, st);
      break;
    }
    case PAIR_PERIODIC_COULOMB: {
      XK_PROF("pair_tiles_pcoul");
      launch_split<D, PAIR_PERIODIC_COULOMB, ENERGY>(g, p, x, m, out, T, jobs, split, st);
      break;
    }
    case PAIR_EWALD_REAL:
      if (D != 3) return cudaErrorInvalidValue;
      {
        XK_PROF("pair_tiles_ewald_real");
        k_pair_tiles<ENERGY><<<pair_grid<ENERGY>(warps, g), 256, EW_TAB_BYTES, st>>>(g, p, x, m, out, T, jobs);
      }
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return XK_LAUNCHED();
}

cudaError_t pair_force(const Geo &g, const PairPrm &p, const double *x, const double *m,
                       double *f, double *scratch, cudaStream_t st) {
  if (p.inv_mass > 0 && ewd_applies(g, p, false)) return ewd_force(g, p, x, f, scratch, st);
  const int T = (g.N + 31) / 32;
  const int jobs = T * (T + 1) / 2, split = p.kind == PAIR_EWALD_REAL ? 1 : pair_split(g, jobs);
  cudaError_t e;
  DISPATCH_D(g.D, e = (pair_launch<D, false>(g, p, x, m, scratch, T, jobs, split, st)));
  if (e != cudaSuccess) return e;
  {
    XK_PROF("pair_finish");
    k_pair_finish<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, scratch, T * split, 1.0 / g.P, f);
  }
  return XK_LAUNCHED();
}

cudaError_t pair_energy(const Geo &g, const PairPrm &p, const double *x, double *acc,
                        double *scratch, cudaStream_t st) {
  const int T = (g.N + 31) / 32;
  const int jobs = T * (T + 1) / 2;
  int split = 1;
  cudaError_t e;
  double unit = 1.0;
  if (ewd_applies(g, p, true)) {
    e = ewd_energy_tiles(g, p, x, scratch, &split, st);
    unit = p.qs * p.alpha;
  } else {
    if (p.kind != PAIR_EWALD_REAL) split = pair_split(g, jobs);
    DISPATCH_D(g.D, e = (pair_launch<D, true>(g, p, x, nullptr, scratch, T, jobs, split, st)));
  }
  if (e != cudaSuccess) return e;
  // the Ewald energy carries -pi/(alpha^2 V) per pair (md_statistics_x.c:385)
  double add = 0;
  if (p.kind == PAIR_EWALD_REAL) {
    const double V = g.box[0] * g.box[1] * g.box[2];
    add = -p.qs * M_PI / (p.alpha * p.alpha * V) * ((double)g.N * (g.N - 1) / 2);
  }
  return reduce_into(scratch, jobs * g.P * split, unit / g.P, add, acc, st);
}

size_t pair2_scratch_doubles(const Geo &ga, const Geo &gb) {
  const int TA = (ga.N + 31) / 32, TB = (gb.N + 31) / 32;
  size_t forces = (size_t)TB * ga.slots() + (size_t)TA * gb.slots();
  if (ga.D == 3) forces = forces * ewd_split((size_t)TA * TB * ga.P) + 1 + ewd_pos_doubles(ga) + ewd_pos_doubles(gb);
  const size_t energy = (size_t)TA * TB * ga.P;
  return forces > energy ? forces : energy;
}

template <int D, int KIND, bool ENERGY>
static cudaError_t cross_launch(const Geo &ga, const Geo &gb, const PairPrm &p, const double *xa, const double *ma,
                                const double *xb, const double *mb, double *outa, double *outb, int TA, int TB,
                                cudaStream_t st) {
  static int occ = 0, sms = 0;
  const size_t dyn = KIND == PAIR_EWALD_REAL ? EW_TAB_BYTES : 0;
  const int grid = resident_grid(k_pair_cross<D, KIND, ENERGY>, (size_t)TA * TB * ga.P, occ, sms, dyn);
  XK_PROF("pair_cross");
  k_pair_cross<D, KIND, ENERGY><<<grid, 256, dyn, st>>>(ga, gb, with_far_images(p, ga), xa, ma, xb, mb, outa, outb, TA,
                                                        TB);
  return XK_LAUNCHED();
}

template <int D, bool ENERGY>
static cudaError_t cross_dispatch(const Geo &ga, const Geo &gb, const PairPrm &p, const double *xa,
                                  const double *ma, const double *xb, const double *mb, double *outa,
                                  double *outb, int TA, int TB, cudaStream_t st) {
  switch (p.kind) {
    case PAIR_GAUSSIAN:
      return cross_launch<D, PAIR_GAUSSIAN, ENERGY>(ga, gb, p, xa, ma, xb, mb, outa, outb, TA, TB, st);
    case PAIR_PERIODIC_GAUSSIAN:
      return cross_launch<D, PAIR_PERIODIC_GAUSSIAN, ENERGY>(ga, gb, p, xa, ma, xb, mb, outa, outb, TA, TB, st);
    case PAIR_COULOMB:
      return cross_launch<D, PAIR_COULOMB, ENERGY>(ga, gb, p, xa, ma, xb, mb, outa, outb, TA, TB, st);
    case PAIR_PERIODIC_COULOMB:
      return cross_launch<D, PAIR_PERIODIC_COULOMB, ENERGY>(ga, gb, p, xa, ma, xb, mb, outa, outb, TA, TB, st);
    case PAIR_EWALD_REAL:
      if (D != 3) return cudaErrorInvalidValue;
      return cross_launch<D, PAIR_EWALD_REAL, ENERGY>(ga, gb, p, xa, ma, xb, mb, outa, outb, TA, TB, st);
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t pair_force_2(const Geo &ga, const Geo &gb, const PairPrm &p, const double *xa, const double *ma,
                         const double *xb, const double *mb, double *fa, double *fb, double *scratch,
                         cudaStream_t st, double inv_ma, double inv_mb) {
  if (ga.D != gb.D || ga.P != gb.P) return cudaErrorInvalidValue;
  if (inv_ma > 0 && inv_mb > 0 && ewd_applies(ga, p, false))
    return ewd_force_2(ga, gb, p, xa, inv_ma, xb, inv_mb, fa, fb, scratch, st);
  const int TA = (ga.N + 31) / 32, TB = (gb.N + 31) / 32;
  double *outa = scratch, *outb = scratch + (size_t)TB * ga.slots();
  cudaError_t e;
  DISPATCH_D(ga.D, e = (cross_dispatch<D, false>(ga, gb, p, xa, ma, xb, mb, outa, outb, TA, TB, st)));
  if (e != cudaSuccess) return e;
  {
    XK_PROF("pair_finish");
    k_pair_finish<<<cdiv(ga.slots(), 256), 256, 0, st>>>(ga, outa, TB, 1.0 / ga.P, fa);
  }
  e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  {
    XK_PROF("pair_finish");
    k_pair_finish<<<cdiv(gb.slots(), 256), 256, 0, st>>>(gb, outb, TA, 1.0 / gb.P, fb);
  }
  return XK_LAUNCHED();
}

cudaError_t pair_energy_2(const Geo &ga, const Geo &gb, const PairPrm &p, const double *xa, const double *xb,
                          double *acc, double *scratch, cudaStream_t st) {
  if (ga.D != gb.D || ga.P != gb.P) return cudaErrorInvalidValue;
  const int TA = (ga.N + 31) / 32, TB = (gb.N + 31) / 32;
  cudaError_t e;
  DISPATCH_D(ga.D, e = (cross_dispatch<D, true>(ga, gb, p, xa, nullptr, xb, nullptr, scratch, nullptr, TA, TB, st)));
  if (e != cudaSuccess) return e;
  // -pi/(alpha^2 V) per pair of the Ewald energy (md_statistics_x.c:385)
  double add = 0;
  if (p.kind == PAIR_EWALD_REAL) {
    const double V = ga.box[0] * ga.box[1] * ga.box[2];
    add = -p.qs * M_PI / (p.alpha * p.alpha * V) * ((double)ga.N * gb.N);
  }
  return reduce_into(scratch, TA * TB * ga.P, 1.0 / ga.P, add, acc, st);
}

// ===================================================================
// Ewald reciprocal space through structure factors (md_simulation_x.c:
// 259-280 force, md_statistics_x.c:364-385 energy).  For every wave vector
// n of the half cube H (|n_i| <= nsum, first non-zero component positive)
//   S_j(n) = sum_l exp(i 2 pi n.x_l / L)            (bead slice j)
//   F_a    = 4 pi/(m P) sum_{n in H} (n/L) c(n) Im(exp(i theta_a) S_j(n)*)
//   E_j    = sum_{n in H} c(n) (|S_j(n)|^2 - N)
// with c(n) = s exp(-pi^2 G^2/alpha^2)/(pi V G^2): the same sums as the
// reference's per-pair loops, regrouped (the l = l2 term of sin vanishes).
// Wave vectors are grouped in columns (nx, ny) with nz contiguous, so the
// phase exp(i(theta_x + theta_y)) is formed once per column.
// ===================================================================

struct Col {
  int nx, ny, nz0, off;
};

static std::vector<Col> columns(int ns) {
  std::vector<Col> c;
  int off = 0;
  for (int nx = 0; nx <= ns; ++nx)
    for (int ny = -ns; ny <= ns; ++ny) {
      if (nx == 0 && ny < 0) continue;
      const int nz0 = (nx == 0 && ny == 0) ? 1 : -ns;
      c.push_back({nx, ny, nz0, off});
      off += ns - nz0 + 1;
    }
  return c;
}

int recip_count(int ns) { return ((2 * ns + 1) * (2 * ns + 1) * (2 * ns + 1) - 1) / 2; }


size_t recip_phase_doubles(const Geo &g, int ns) { return (size_t)g.P * 3 * (ns + 1) * g.Ns * 2; }

// phase[((j*3 + d)*(ns+1) + n)*Ns + l] = exp(i 2 pi n x / L) as (re, im)
__global__ void k_phase(Geo g, int ns, const double *__restrict__ x, double2 *__restrict__ ph) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)g.P * 3 * g.Ns) return;
  const int l = (int)(t % g.Ns);
  const int jd = (int)(t / g.Ns);  // j*3 + d
  const int d = jd % 3;
  double s1 = 0, c1 = 1;
  if (l < g.N) sincospi(2.0 * x[t] * g.inv_box[d], &s1, &c1);
  double re = 1, im = 0;
  double2 *o = ph + (size_t)jd * (ns + 1) * g.Ns + l;
  o[0] = make_double2(1.0, 0.0);
  for (int n = 1; n <= ns; ++n) {
    const double r2 = re * c1 - im * s1, i2 = re * s1 + im * c1;
    re = r2;
    im = i2;
    o[(size_t)n * g.Ns] = make_double2(re, im);
  }
}

__device__ inline double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ inline double2 phase_at(const double2 *ph, const Geo &g, int ns, int j, int d, int n,
                                   int l) {
  const double2 v = ph[(((size_t)j * 3 + d) * (ns + 1) + (n < 0 ? -n : n)) * g.Ns + l];
  return n < 0 ? make_double2(v.x, -v.y) : v;
}

// Within a column the wave vectors +nz and -nz share cos(nz theta_z) and
// sin(nz theta_z): exp(i(theta_xy +- nz theta_z)) = e_xy (c +- i s).  Both
// kernels below work on such pairs, which roughly halves their FP64 work.

// S_j(n) for one column (nx, ny) and all its nz.  One thread per (slice,
// column) sums over the slice's particles, whose phase factors are staged in
// shared memory in chunks, so no cross-thread reduction is needed.  With
// P = sum e_xy c and Q = sum e_xy s:  S(+nz) = P + iQ,  S(-nz) = P - iQ.
// Block = COLS columns of one slice x GR particle groups.  For large slices
// (N >= 256) the 16 lanes of a column (adjacent in the warp) sum every 16th
// particle of each staged chunk and combine by four shuffles at the end, so
// that a slice's columns give 16 times as many warps to hide the FP64
// latency and the grid (12 blocks per slice at |n| <= 10) fills the SMs in
// even rounds; small slices keep one thread per column.
constexpr int SK_CHUNK = 64;
constexpr int SK_BIG_N = 256;  // slices of at least this many particles use 16 groups

template <int NS, int COLS, int GR>
__global__ void __launch_bounds__(COLS * GR, COLS * GR >= 256 ? 2 : 1) k_sk(Geo g, const double2 *__restrict__ ph,
                                                                       const int4 *__restrict__ cols, int ncol,
                                                                       double2 *__restrict__ S, int nk) {
  constexpr int SK_THREADS = COLS * GR, SK_GROUPS = GR;
  // staged phases of SK_CHUNK particles: x, y, z factors for n = 0..NS
  __shared__ double2 sp[3][NS + 1][SK_CHUNK];
  const int j = blockIdx.y;
  const int gq = threadIdx.x & (SK_GROUPS - 1);
  const int ci = blockIdx.x * COLS + threadIdx.x / SK_GROUPS;
  const bool live = ci < ncol;
  const int4 c = live ? cols[ci] : make_int4(0, 0, 1, 0);
  const int ax = col_nx(c), ay = c.y < 0 ? -c.y : c.y;
  const bool cy = c.y < 0;  // conjugate the y factor
  double s0r = 0, s0i = 0, P[NS][2], Q[NS][2];
#pragma unroll
  for (int n = 0; n < NS; ++n) P[n][0] = P[n][1] = Q[n][0] = Q[n][1] = 0.0;
  const double2 *base = ph + (size_t)j * 3 * (NS + 1) * g.Ns;
  for (int l0 = 0; l0 < g.N; l0 += SK_CHUNK) {
    const int cnt = g.N - l0 < SK_CHUNK ? g.N - l0 : SK_CHUNK;
    __syncthreads();
    for (int q = threadIdx.x; q < 3 * (NS + 1) * SK_CHUNK; q += SK_THREADS) {
      const int l = q % SK_CHUNK, row = q / SK_CHUNK;  // row = d*(NS+1) + n
      (&sp[0][0][0])[q] = l < cnt ? base[(size_t)row * g.Ns + l0 + l] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (!live) continue;
    for (int l = gq; l < cnt; l += SK_GROUPS) {
      const double2 ex = sp[0][ax][l];
      double2 ey = sp[1][ay][l];
      if (cy) ey.y = -ey.y;
      const double2 exy = cmul(ex, ey);
      s0r += exy.x;
      s0i += exy.y;
#pragma unroll
      for (int n = 1; n <= NS; ++n) {
        const double2 ez = sp[2][n][l];
        P[n - 1][0] = fma(exy.x, ez.x, P[n - 1][0]);
        P[n - 1][1] = fma(exy.y, ez.x, P[n - 1][1]);
        Q[n - 1][0] = fma(exy.x, ez.y, Q[n - 1][0]);
        Q[n - 1][1] = fma(exy.y, ez.y, Q[n - 1][1]);
      }
    }
  }
  // the column's lanes, pairwise in a fixed order
#pragma unroll
  for (int o = 1; o < SK_GROUPS; o <<= 1) {
    s0r += __shfl_xor_sync(FULL, s0r, o);
    s0i += __shfl_xor_sync(FULL, s0i, o);
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      P[n][0] += __shfl_xor_sync(FULL, P[n][0], o);
      P[n][1] += __shfl_xor_sync(FULL, P[n][1], o);
      Q[n][0] += __shfl_xor_sync(FULL, Q[n][0], o);
      Q[n][1] += __shfl_xor_sync(FULL, Q[n][1], o);
    }
  }
  if (!live || gq != 0) return;
  double2 *o = S + (size_t)j * nk + c.w - c.z;  // o[nz] for nz = c.z..NS
  if (c.z <= 0) o[0] = make_double2(s0r, s0i);
#pragma unroll
  for (int n = 1; n <= NS; ++n) {
    const double Pr = P[n - 1][0], Pi = P[n - 1][1], Qr = Q[n - 1][0], Qi = Q[n - 1][1];
    o[n] = make_double2(Pr - Qi, Pi + Qr);
    if (c.z < 0) o[-n] = make_double2(Pr + Qi, Pi - Qr);
  }
}

// force tables per (slice, column): W(nz) = c(n) conj(S(n)); slot 0 holds
// W(0), slots 4n-3 .. 4n hold A = W(+n) + W(-n), B = W(+n) - W(-n), n A
// and n B (W(-n) = 0 where -n is not in the half space: column (0, 0))
template <int NS>
__global__ void k_recip_tables(const int4 *__restrict__ cols, int ncol, const double2 *__restrict__ S,
                               const double *__restrict__ coef, int nk, double2 *__restrict__ T) {
  constexpr int NT = 4 * NS + 1;
  const int j = blockIdx.y;
  const int ci = blockIdx.x * blockDim.y + threadIdx.y;
  const int n = threadIdx.x;  // 0..NS
  if (ci >= ncol || n > NS) return;
  const int4 c = cols[ci];
  auto W = [&](int nz) {
    if (nz < c.z) return make_double2(0.0, 0.0);
    const int k = c.w + (nz - c.z);
    const double2 s = S[(size_t)j * nk + k];
    return make_double2(coef[k] * s.x, -coef[k] * s.y);
  };
  double2 *o = T + ((size_t)j * ncol + ci) * NT;
  if (n == 0) {
    o[0] = W(0);
  } else {
    const double2 wp = W(n), wm = W(-n);
    const double2 A = make_double2(wp.x + wm.x, wp.y + wm.y), B = make_double2(wp.x - wm.x, wp.y - wm.y);
    o[4 * n - 3] = A;
    o[4 * n - 2] = B;
    o[4 * n - 1] = make_double2(n * A.x, n * A.y);
    o[4 * n] = make_double2(n * B.x, n * B.y);
  }
}

// forces: block per (slice, 128 particles), the slice's tables in shared
// memory.  Per column, with U = sum_nz e_z(nz) W(nz) and V = sum_nz nz e_z W:
//   sum_nz c(n) Im(e^{i theta} conj S(n)) = Im(e_xy U),   z part Im(e_xy V),
// where for each pair +-nz:  e_z(+)W(+) + e_z(-)W(-) = c A + i s B  and
// nz (e_z(+)W(+) - e_z(-)W(-)) = nz (c B + i s A).
//
// WITH_E also writes the particle's share of the slice energy,
//   e[j*Ns + l] = sum_n c(n) Re(e^{i theta} conj S(n)) - e0 = Re(sum_col e_xy U) - e0,
// with e0 = sum_n c(n), so that sum_l e = sum_n c(n) (|S(n)|^2 - N).
// TPP > 1 (a few bead slices, as in the learned model's judgements): TPP
// consecutive threads share a particle, thread h taking columns h, h + TPP,
// ..., and their sums are added by a butterfly over the TPP lanes.
template <int NS, bool WITH_E = false, int TPP = 1>
__global__ void __launch_bounds__(128) k_recip_force(Geo g, const double2 *__restrict__ ph,
                                                     const int4 *__restrict__ cols, const int *__restrict__ toff,
                                                     int ncol, const double2 *__restrict__ T, double scale,
                                                     double *__restrict__ f, double *__restrict__ e = nullptr,
                                                     double e0 = 0.0) {
  constexpr int NT = 4 * NS + 1;
  // the slice's tables in shared memory, each column only up to its largest
  // kept |nz| (toff: compact offsets), so that two blocks fit on an SM
  extern __shared__ double sm[];
  double2 *sT = (double2 *)sm;
  const int j = blockIdx.y;
  const double2 *Tj = T + (size_t)j * ncol * NT;
  for (int ci = threadIdx.x >> 5; ci < ncol; ci += blockDim.x >> 5) {
    const int n = toff[ci + 1] - toff[ci];
    for (int q = threadIdx.x & 31; q < n; q += 32) sT[toff[ci] + q] = Tj[(size_t)ci * NT + q];
  }
  __syncthreads();
  const int l = blockIdx.x * (blockDim.x / TPP) + threadIdx.x / TPP, h = threadIdx.x % TPP;
  if (l >= g.N) return;  // (a particle's TPP lanes leave together)
  double2 ez[NS + 1];
  const double2 *pz = ph + (((size_t)j * 3 + 2) * (NS + 1)) * g.Ns + l;
#pragma unroll
  for (int n = 1; n <= NS; ++n) ez[n] = pz[(size_t)n * g.Ns];
  double Fx = 0, Fy = 0, Fz = 0, Er = 0;
  for (int ci = h; ci < ncol; ci += TPP) {
    const int4 c = cols[ci];
    const int nzc = col_nz(c);
    const double2 exy = cmul(phase_at(ph, g, NS, j, 0, col_nx(c), l), phase_at(ph, g, NS, j, 1, c.y, l));
    const double2 *t = sT + toff[ci];
    double Ur = t[0].x, Ui = t[0].y, Vr = 0, Vi = 0;
#pragma unroll
    for (int n = 1; n <= NS; ++n) {
      if (n > nzc) break;  // uniform: every thread walks the same column
      const double2 A = t[4 * n - 3], B = t[4 * n - 2], nA = t[4 * n - 1], nB = t[4 * n];
      const double cz = ez[n].x, sz = ez[n].y;
      Ur = fma(cz, A.x, fma(-sz, B.y, Ur));
      Ui = fma(cz, A.y, fma(sz, B.x, Ui));
      Vr = fma(cz, nB.x, fma(-sz, nA.y, Vr));
      Vi = fma(cz, nB.y, fma(sz, nA.x, Vi));
    }
    const double Tm = fma(exy.x, Ui, exy.y * Ur);  // Im(e_xy U)
    const double Zm = fma(exy.x, Vi, exy.y * Vr);  // Im(e_xy V)
    Fx = fma((double)col_nx(c), Tm, Fx);
    Fy = fma((double)c.y, Tm, Fy);
    Fz += Zm;
    if (WITH_E) Er += fma(exy.x, Ur, -exy.y * Ui);  // Re(e_xy U)
  }
  if (TPP > 1) {
    const unsigned gm = ((1u << TPP) - 1u) << ((threadIdx.x & 31) & ~(TPP - 1));
#pragma unroll
    for (int o = 1; o < TPP; o <<= 1) {
      Fx += __shfl_xor_sync(gm, Fx, o);
      Fy += __shfl_xor_sync(gm, Fy, o);
      Fz += __shfl_xor_sync(gm, Fz, o);
      if (WITH_E) Er += __shfl_xor_sync(gm, Er, o);
    }
    if (h != 0) return;
  }
  if (WITH_E) e[(size_t)j * g.Ns + l] = Er - e0;
  f[sidx(j, 0, l, 3, g.Ns)] += scale * Fx * g.inv_box[0];
  f[sidx(j, 1, l, 3, g.Ns)] += scale * Fy * g.inv_box[1];
  f[sidx(j, 2, l, 3, g.Ns)] += scale * Fz * g.inv_box[2];
}

__global__ void k_recip_energy(Geo g, const double2 *__restrict__ S, const double *__restrict__ coef,
                               int nk, double *part) {
  __shared__ double buf[33];
  const int j = blockIdx.x;
  double e = 0;
  for (int k = threadIdx.x; k < nk; k += blockDim.x) {
    const double ck = coef[k];
    if (__double_as_longlong(ck) == 0) continue;  // a dropped vector
    const double2 s = S[(size_t)j * nk + k];
    e += ck * (s.x * s.x + s.y * s.y - g.N);
  }
  e = block_sum(e, buf);
  if (threadIdx.x == 0) part[j] = e;
}

static int ncols(int ns) { return ns * (2 * ns + 1) + ns + 1; }
size_t recip_df_off(int ns) { return (5 * (size_t)ncols(ns) + 1 + 3) & ~(size_t)3; }

cudaError_t recip_setup(const Geo &g, int ns, double alpha, double qs, Recip &r,
                        cudaStream_t st) {
  // host-side tables: c(n) in the full column order, then the kept columns
  std::vector<Col> cols = columns(ns);
  const int nk = recip_count(ns);
  std::vector<double> coef(nk), wgt(nk);
  const double V = g.box[0] * g.box[1] * g.box[2];
  double wmax = 0;
  for (const Col &c : cols)
    for (int nz = c.nz0; nz <= ns; ++nz) {
      const double gx = c.nx / g.box[0], gy = c.ny / g.box[1], gz = nz / g.box[2];
      const double G = sqrt(gx * gx + gy * gy + gz * gz);
      const int k = c.off + nz - c.nz0;
      coef[k] = qs * pow(G, -2) * exp(-M_PI * M_PI * G * G / (alpha * alpha)) / (V * M_PI);
      wgt[k] = fabs(coef[k]) * G;  // weight of the vector in the forces
      wmax = wgt[k] > wmax ? wgt[k] : wmax;
    }
  // per column the largest |nz| whose vector is kept (+nz and -nz have the
  // same |G|); columns without one are left out, the rest sorted longest first
  std::vector<std::pair<int, int4>> kept;
  for (const Col &c : cols) {
    int nzmax = -1;
    for (int nz = c.nz0; nz <= ns; ++nz) {
      const int k = c.off + nz - c.nz0;
      if (wgt[k] >= RECIP_KEEP * wmax) {
        nzmax = abs(nz) > nzmax ? abs(nz) : nzmax;
      }
    }
    for (int nz = c.nz0; nz <= ns; ++nz)
      if (abs(nz) > nzmax) coef[c.off + nz - c.nz0] = 0.0;
    if (nzmax < 0 || (c.nz0 > 0 && nzmax < c.nz0)) continue;
    kept.push_back({nzmax, make_int4(c.nx | (nzmax << 8), c.ny, c.nz0, c.off)});
  }
  std::stable_sort(kept.begin(), kept.end(), [](const std::pair<int, int4> &a, const std::pair<int, int4> &b) {
    return a.first > b.first;
  });
  std::vector<int4> cd(kept.size());
  for (size_t i = 0; i < kept.size(); ++i) cd[i] = kept[i].second;
  // compact table offsets of the kept columns (4 nzmax + 1 entries each)
  std::vector<int> toff(kept.size() + 1, 0);
  for (size_t i = 0; i < kept.size(); ++i) toff[i + 1] = toff[i] + 4 * kept[i].first + 1;
  std::vector<int> dft;
  recip_df_tables(ns, cd, wgt, wmax, r, dft);
  r.nsum = ns;
  r.nk = nk;
  r.ncol = (int)cd.size();
  r.nlong = 0;
  for (const auto &k : kept) r.nlong += k.first > SK_NG;
  r.tsz = toff.back();
  r.csum = 0;
  for (double c : coef) r.csum += c;
  cudaError_t e = cudaMemcpyAsync(r.coef, coef.data(), sizeof(double) * nk, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  // an FP32 copy behind them for the mixed form's force tables
  std::vector<float> coef32(coef.begin(), coef.end());
  e = cudaMemcpyAsync(r.coef + nk, coef32.data(), sizeof(float) * nk, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  // and as FP32 pairs for the double-float ones
  std::vector<float2> pairs(nk);
  for (int k = 0; k < nk; ++k) pairs[k] = make_float2(coef32[k], (float)(coef[k] - (double)coef32[k]));
  e = cudaMemcpyAsync(r.coef + recip_coef_pairs_at(nk), pairs.data(), sizeof(float2) * nk, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  if (!cd.empty()) {
    e = cudaMemcpyAsync(r.kvec, cd.data(), sizeof(int4) * cd.size(), cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
  }
  e = cudaMemcpyAsync(r.kvec + 4 * (size_t)(ns * (2 * ns + 1) + ns + 1), toff.data(), sizeof(int) * toff.size(),
                      cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(r.kvec + recip_df_off(ns), dft.data(), sizeof(int) * dft.size(), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return e;
  // dropped vectors keep S = 0 (their c(n) = 0 multiplies them in the energies)
  if (r.S) {
    e = cudaMemsetAsync(r.S, 0, sizeof(double2) * (size_t)nk * g.P, st);
    if (e != cudaSuccess) return e;
  }
  return cudaStreamSynchronize(st);
}

// kvec: the kept columns (int4, longest first) and their compact table
// offsets, then, from recip_df_off (16-byte aligned), the double-float
// kernels' tables
size_t recip_cols_ints(int ns) { return recip_df_off(ns) + recip_df_ints(ns); }

// compact table offsets behind the column table in the same buffer
static const int *recip_toff(const Recip &r) {
  return r.kvec + 4 * (size_t)(r.nsum * (2 * r.nsum + 1) + r.nsum + 1);
}
#define DISPATCH_NS(nsv, ...)                                         \
  switch (nsv) {                                                      \
    case 1: { constexpr int NS = 1; __VA_ARGS__; } break;             \
    case 2: { constexpr int NS = 2; __VA_ARGS__; } break;             \
    case 3: { constexpr int NS = 3; __VA_ARGS__; } break;             \
    case 4: { constexpr int NS = 4; __VA_ARGS__; } break;             \
    case 5: { constexpr int NS = 5; __VA_ARGS__; } break;             \
    case 6: { constexpr int NS = 6; __VA_ARGS__; } break;             \
    case 7: { constexpr int NS = 7; __VA_ARGS__; } break;             \
    case 8: { constexpr int NS = 8; __VA_ARGS__; } break;             \
    case 9: { constexpr int NS = 9; __VA_ARGS__; } break;             \
    case 10: { constexpr int NS = 10; __VA_ARGS__; } break;           \
    case 11: { constexpr int NS = 11; __VA_ARGS__; } break;           \
    case 12: { constexpr int NS = 12; __VA_ARGS__; } break;           \
    default: return cudaErrorInvalidValue;                            \
  }

// FP64 structure factors of the kept columns
static cudaError_t structure_factors(const Geo &g, const Recip &r, const double *x, cudaStream_t st) {
  const int4 *cols = (const int4 *)r.kvec;
  const int nc = r.ncol;
  const size_t n = (size_t)g.P * 3 * g.Ns;
  {
    XK_PROF("phase");
    k_phase<<<cdiv(n, 256), 256, 0, st>>>(g, r.nsum, x, (double2 *)r.phase);
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  if (nc <= 0) return cudaSuccess;
  {
    XK_PROF("sk");
    int lay = tuning(TUNE_SK_LAYOUT, r.nsum, 3, g.N, g.P);
    if (lay == 0)
      lay = g.N < SK_BIG_N ? SK_64x1 : ((size_t)((nc + 15) / 16) * g.P < 2 * 152 ? SK_8x32 : SK_16x16);
    if (lay == SK_8x32) {
      // few slices (a judgement's): 8 columns of 32 lanes per block, twice
      // the blocks, each with half the work
      dim3 grid((nc + 7) / 8, g.P);
      DISPATCH_NS(r.nsum, (k_sk<NS, 8, 32><<<grid, 256, 0, st>>>(g, (const double2 *)r.phase,
                                                                 cols, nc, (double2 *)r.S, r.nk)));
    } else if (lay == SK_16x16) {
      dim3 grid((nc + 15) / 16, g.P);
      DISPATCH_NS(r.nsum, (k_sk<NS, 16, 16><<<grid, 256, 0, st>>>(g, (const double2 *)r.phase,
                                                                  cols, nc, (double2 *)r.S, r.nk)));
    } else {
      dim3 grid((nc + 63) / 64, g.P);
      DISPATCH_NS(r.nsum, (k_sk<NS, 64, 1><<<grid, 64, 0, st>>>(g, (const double2 *)r.phase,
                                                                cols, nc, (double2 *)r.S, r.nk)));
    }
  }
  return XK_LAUNCHED();
}

size_t recip_table_doubles(const Geo &g, int ns) { return (size_t)g.P * ncols(ns) * (4 * ns + 1) * 2; }

static cudaError_t recip_tables_of(const Geo &g, const Recip &r, cudaStream_t st) {
  const int nc = r.ncol;
  dim3 tgrid((nc + 7) / 8, g.P), tblk(r.nsum + 1, 8);
  DISPATCH_NS(r.nsum, {
    XK_PROF("recip_tables");
    k_recip_tables<NS><<<tgrid, tblk, 0, st>>>((const int4 *)r.kvec, nc, (const double2 *)r.S, r.coef, r.nk,
                                               (double2 *)r.T);
  });
  return XK_LAUNCHED();
}

static cudaError_t recip_force_from(const Geo &g, const Recip &own, const double *T_other, double scale, double *f,
                                    cudaStream_t st) {
  const int nc = own.ncol;
  const size_t smem = sizeof(double2) * own.tsz;
  dim3 grid((g.N + 127) / 128, g.P);
  DISPATCH_NS(own.nsum, {
    auto kf = k_recip_force<NS>;
    static bool opted = false;
    if (!opted) {
      cudaError_t ea = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (ea != cudaSuccess) return ea;
      opted = true;
    }
    XK_PROF("recip_force");
    kf<<<grid, 128, smem, st>>>(g, (const double2 *)own.phase, (const int4 *)own.kvec, recip_toff(own), nc,
                                (const double2 *)T_other, scale, f, nullptr, 0.0);
  });
  return XK_LAUNCHED();
}

cudaError_t recip_force(const Geo &g, const Recip &r, const double *x, double inv_mP, double *f,
                        cudaStream_t st, bool df) {
  if (g.D != 3) return cudaErrorInvalidValue;
  if (df) {
    cudaError_t e = recip_df_sk(g, r, x, st);
    if (e == cudaSuccess) e = recip_df_tables_of(g, r, st);
    if (e == cudaSuccess) e = recip_df_force_from(g, r, r.T, 4 * M_PI * inv_mP, f, st);
    return e;
  }
  cudaError_t e = structure_factors(g, r, x, st);
  if (e == cudaSuccess) e = recip_tables_of(g, r, st);
  if (e == cudaSuccess) e = recip_force_from(g, r, r.T, 4 * M_PI * inv_mP, f, st);
  return e;
}

cudaError_t recip_force_energy(const Geo &g, const Recip &r, const double *x, double scale, double *f,
                               double *e, cudaStream_t st) {
  if (g.D != 3) return cudaErrorInvalidValue;
  cudaError_t err = structure_factors(g, r, x, st);
  if (err != cudaSuccess) return err;
  const int nc = r.ncol;
  const double e0 = r.csum;
  const size_t smem = sizeof(double2) * r.tsz;
  dim3 tgrid((nc + 7) / 8, g.P), tblk(r.nsum + 1, 8);
  // blocks of 128 threads; with few bead slices (the learned model's
  // judgements) 4 or 16 threads share a particle's columns, so that the
  // grid still covers every SM twice
  int dev = 0, sms = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t parts = (size_t)g.N * g.P;
  const int tpp = parts * 1 >= (size_t)256 * sms ? 1 : (parts * 4 >= (size_t)256 * sms ? 4 : 16);
  const int ppb = 128 / tpp;
  dim3 grid((g.N + ppb - 1) / ppb, g.P);
  DISPATCH_NS(r.nsum, {
    {
      XK_PROF("recip_tables");
      k_recip_tables<NS><<<tgrid, tblk, 0, st>>>((const int4 *)r.kvec, nc, (const double2 *)r.S, r.coef,
                                                 r.nk, (double2 *)r.T);
    }
    auto kf = tpp == 1 ? k_recip_force<NS, true, 1> : (tpp == 4 ? k_recip_force<NS, true, 4> : k_recip_force<NS, true, 16>);
    static bool opted[3] = {false, false, false};
    const int oi = tpp == 1 ? 0 : (tpp == 4 ? 1 : 2);
    if (!opted[oi]) {
      cudaError_t ea = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (ea != cudaSuccess) return ea;
      opted[oi] = true;
    }
    {
      XK_PROF("recip_force_energy");
      kf<<<grid, 128, smem, st>>>(g, (const double2 *)r.phase, (const int4 *)r.kvec, recip_toff(r), nc,
                                  (const double2 *)r.T, 4 * M_PI * scale, f, e, e0);
    }
  });
  return XK_LAUNCHED();
}

cudaError_t recip_energy(const Geo &g, const Recip &r, const double *x, double *acc,
                         double *scratch, cudaStream_t st, bool df) {
  if (g.D != 3) return cudaErrorInvalidValue;
  if (df) {
    cudaError_t e = recip_df_sk(g, r, x, st);
    if (e == cudaSuccess) e = recip_df_energy(g, r, scratch, st);
    return e == cudaSuccess ? reduce_into(scratch, g.P, 1.0 / g.P, 0.0, acc, st) : e;
  }
  cudaError_t e = structure_factors(g, r, x, st);
  if (e != cudaSuccess) return e;
  {
    XK_PROF("recip_energy");
    k_recip_energy<<<g.P, 256, 0, st>>>(g, (const double2 *)r.S, r.coef, r.nk, scratch);
  }
  e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  return reduce_into(scratch, g.P, 1.0 / g.P, 0.0, acc, st);
}

// Two species (md_pimd_calc_pair_force_2_x with the Ewald callback): the
// reciprocal part of the cross pairs, regrouped like the one-species sums,
//   F_a = 4 pi/(m_a P) sum_{n in H} (n/L) c(n) Im(e^{i theta_a} S_b(n)*)
// and the same with a and b exchanged; there is no l = l2 term to drop.  The
// cross energy of slice j is sum_{n in H} 2 c(n) Re(S_a,j(n) S_b,j(n)*).
// Each species keeps its own phases, structure factors and tables (T from
// its own S); a's forces read b's tables and b's read a's.
static bool recip_pair_ok(const Geo &ga, const Recip &ra, const Geo &gb, const Recip &rb) {
  return ga.D == 3 && gb.D == 3 && ga.P == gb.P && ra.nsum == rb.nsum && ra.nk == rb.nk && ra.ncol == rb.ncol;
}

cudaError_t recip_force_2(const Geo &ga, const Recip &ra, const double *xa, double inv_mPa, double *fa,
                          const Geo &gb, const Recip &rb, const double *xb, double inv_mPb, double *fb,
                          cudaStream_t st, bool df) {
  if (!recip_pair_ok(ga, ra, gb, rb)) return cudaErrorInvalidValue;
  if (df) {
    cudaError_t e = recip_df_sk(ga, ra, xa, st);
    if (e == cudaSuccess) e = recip_df_sk(gb, rb, xb, st);
    if (e == cudaSuccess) e = recip_df_tables_of(ga, ra, st);
    if (e == cudaSuccess) e = recip_df_tables_of(gb, rb, st);
    if (e == cudaSuccess) e = recip_df_force_from(ga, ra, rb.T, 4 * M_PI * inv_mPa, fa, st);
    if (e == cudaSuccess) e = recip_df_force_from(gb, rb, ra.T, 4 * M_PI * inv_mPb, fb, st);
    return e;
  }
  cudaError_t e = structure_factors(ga, ra, xa, st);
  if (e == cudaSuccess) e = structure_factors(gb, rb, xb, st);
  if (e == cudaSuccess) e = recip_tables_of(ga, ra, st);
  if (e == cudaSuccess) e = recip_tables_of(gb, rb, st);
  if (e == cudaSuccess) e = recip_force_from(ga, ra, rb.T, 4 * M_PI * inv_mPa, fa, st);
  if (e == cudaSuccess) e = recip_force_from(gb, rb, ra.T, 4 * M_PI * inv_mPb, fb, st);
  return e;
}

__global__ void k_recip_energy_2(const double2 *__restrict__ Sa, const double2 *__restrict__ Sb,
                                 const double *__restrict__ coef, int nk, double *part) {
  __shared__ double buf[33];
  const int j = blockIdx.x;
  double e = 0;
  for (int k = threadIdx.x; k < nk; k += blockDim.x) {
    const double ck = coef[k];
    if (__double_as_longlong(ck) == 0) continue;  // a dropped vector
    const double2 a = Sa[(size_t)j * nk + k], b = Sb[(size_t)j * nk + k];
    e += 2 * ck * (a.x * b.x + a.y * b.y);
  }
  e = block_sum(e, buf);
  if (threadIdx.x == 0) part[j] = e;
}

cudaError_t recip_energy_2(const Geo &ga, const Recip &ra, const double *xa, const Geo &gb, const Recip &rb,
                           const double *xb, double *acc, double *scratch, cudaStream_t st) {
  if (!recip_pair_ok(ga, ra, gb, rb)) return cudaErrorInvalidValue;
  cudaError_t e = structure_factors(ga, ra, xa, st);
  if (e == cudaSuccess) e = structure_factors(gb, rb, xb, st);
  if (e != cudaSuccess) return e;
  {
    XK_PROF("recip_energy");
    k_recip_energy_2<<<ga.P, 256, 0, st>>>((const double2 *)ra.S, (const double2 *)rb.S, ra.coef, ra.nk, scratch);
  }
  e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  return reduce_into(scratch, ga.P, 1.0 / ga.P, 0.0, acc, st);
}

// ===================================================================
// static structure factor between two bead slices: md_pimd_x.c:5404-5448
// ===================================================================
// one block per wave vector q: cos and sin sums of q.x over the particles of
// slices ja and jb; out[q] = (C_a C_b + S_a S_b) / N
__global__ void k_sk_structure(Geo g, const double *__restrict__ x, int ja, int jb,
                               const double *__restrict__ qis, double *__restrict__ out) {
  __shared__ double buf[33];
  const int q = blockIdx.x;
  const double q0 = qis[3 * q], q1 = qis[3 * q + 1], q2 = qis[3 * q + 2];
  double ca = 0, sa = 0, cb = 0, sb = 0;
  for (int l = threadIdx.x; l < g.N; l += blockDim.x) {
    double s, c;
    sincos(q0 * x[sidx(ja, 0, l, 3, g.Ns)] + q1 * x[sidx(ja, 1, l, 3, g.Ns)] + q2 * x[sidx(ja, 2, l, 3, g.Ns)], &s, &c);
    ca += c;
    sa += s;
    sincos(q0 * x[sidx(jb, 0, l, 3, g.Ns)] + q1 * x[sidx(jb, 1, l, 3, g.Ns)] + q2 * x[sidx(jb, 2, l, 3, g.Ns)], &s, &c);
    cb += c;
    sb += s;
  }
  ca = block_sum(ca, buf);
  sa = block_sum(sa, buf);
  cb = block_sum(cb, buf);
  sb = block_sum(sb, buf);
  if (threadIdx.x == 0) out[q] = ca * cb / g.N + sa * sb / g.N;
}

cudaError_t sk_structure(const Geo &g, const double *x, int ja, int jb, const double *qis, int nq, double *out,
                         cudaStream_t st) {
  if (g.D != 3 || nq <= 0) return nq == 0 ? cudaSuccess : cudaErrorInvalidValue;
  {
    XK_PROF("sk_structure");
    k_sk_structure<<<nq, 128, 0, st>>>(g, x, ja, jb, qis, out);
  }
  return XK_LAUNCHED();
}

// ===================================================================
// estimators
// ===================================================================

// Primitive (md_pimd_x.c:1267-1293) and, with ENk2, virial
// (md_pimd_x.c:4288-4322) exchange estimators.  The reference's recursion
//   res[n] = sum_k (res[n-k] - E2[n][k]) w_{n,k} / sum_k w_{n,k},
//   w_{n,k} = exp((k-1) ln xi - beta (ENk[n][k] + VBN[n-k]) + m_n)
// is a unit lower-triangular system res = p res + c in the normalised
// weights p_{n,n-k} = w_{n,k} / sum_k w_{n,k} and c_n = -sum_k p_{n,n-k}
// E2[n][k].  The weights need only ENk and VBN, so they are computed for all
// rows at once (a warp per row); the solve then takes the chunked scheme of
// k_tri_solve in plain FP64 (the normalised weights are at most 1 and res
// is an energy: no extended range is needed).
__global__ void k_est_weights(int N, double beta, double vi, const double *__restrict__ ENk,
                              const double *__restrict__ VBN, const double *__restrict__ E2, double *__restrict__ Pw,
                              double *__restrict__ cvec) {
  const int lane = threadIdx.x & 31;
  const int n = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) + 1;
  if (n > N) return;
  const double *row = ENk + dtri(n), *row2 = E2 + dtri(n);
  double *prow = Pw + moff(n, 0);
  if (vi == 0.0) {
    // only k = 1 carries weight (md_pimd_x.c:1280): p = 1, the rest 0
    for (int j = lane; j < n; j += 32) prow[j] = j == n - 1 ? 1.0 : 0.0;
    if (lane == 0) cvec[n] = -row2[0];
    return;
  }
  const double lnvi = log(vi);
  double mloc = 1e10;
  for (int k = lane + 1; k <= n; k += 32) {
    const double t = -(k - 1) * lnvi + beta * (row[k - 1] + VBN[n - k]);
    mloc = t < mloc ? t : mloc;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const double t = __shfl_xor_sync(FULL, mloc, o);
    mloc = t < mloc ? t : mloc;
  }
  // each weight's exponential once: kept in the output row, normalised below
  double s1 = 0.0;
  for (int k = lane + 1; k <= n; k += 32) {
    const double w = exp((k - 1) * lnvi - beta * (row[k - 1] + VBN[n - k]) + mloc);
    prow[n - k] = w;
    s1 += w;
  }
  s1 = warp_sum_fx(s1);
  const double inv = 1.0 / s1;
  double cs = 0.0;
  for (int k = lane + 1; k <= n; k += 32) {
    const double pk = prow[n - k] * inv;
    prow[n - k] = pk;
    cs = fma(-pk, row2[k - 1], cs);
  }
  cs = warp_sum_fx(cs);
  if (lane == 0) cvec[n] = cs;
}

// x_0 = 0, x_i = c_i + sum_{j<i} Pw[moff(i, j)] x_j; adds x_N + add to *acc.
// Chunks of TS_CHUNK rows are substituted in order by warp 0 (one FMA and
// one shuffle per step on the sequential path) while the other warps stage
// the next chunk's weights in shared memory and sum its rows over all
// columns solved before the current chunk.
__global__ void __launch_bounds__(TS_WARPS * 32) k_lin_solve(int N, const double *__restrict__ Pw,
                                                             const double *__restrict__ cvec, double add,
                                                             double *acc) {
  extern __shared__ double sh[];
  double *W = sh;                              // [2][TS_CHUNK][TS_LD] the chunk's triangle
  double *U = W + 2 * TS_CHUNK * TS_LD;        // [2][TS_CHUNK][TS_LD] previous chunk's columns
  double *Ps = U + 2 * TS_CHUNK * TS_LD;       // [2][TS_CHUNK] partial sums (double buffer)
  double *X = Ps + 2 * TS_CHUNK;               // N+1
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto stage = [&](int n0, int c0, int nb, int t0, int stride) {
    for (int q = t0; q < 2 * TS_CHUNK * TS_CHUNK; q += stride) {
      const int which = q / (TS_CHUNK * TS_CHUNK), rs = q % (TS_CHUNK * TS_CHUNK);
      const int r = rs / TS_CHUNK, c = rs % TS_CHUNK, i = n0 + r;
      const size_t o = ((size_t)nb * TS_CHUNK + r) * TS_LD + c;
      if (which == 0)
        W[o] = (i <= N && c < r) ? Pw[moff(i, n0 + c)] : 0.0;
      else
        U[o] = (i <= N && c0 >= 0) ? Pw[moff(i, c0 + c)] : 0.0;
    }
  };
  if (threadIdx.x == 0) X[0] = 0.0;
  stage(1, -1, 0, threadIdx.x, blockDim.x);
  // chunk 0: column 0 holds x_0 = 0, so its rows start from c
  for (int r = threadIdx.x; r < TS_CHUNK; r += blockDim.x) Ps[r] = 1 + r <= N ? cvec[1 + r] : 0.0;
  __syncthreads();
  for (int i0 = 1, c = 0; i0 <= N; i0 += TS_CHUNK, ++c) {
    const int buf = c & 1;
    double *Psc = Ps + buf * TS_CHUNK;
    if (c > 0) {
      const int col = i0 - TS_CHUNK + lane;
      for (int r = w; r < TS_CHUNK; r += TS_WARPS) {
        if (i0 + r > N) continue;  // warp-uniform
        double v = U[((size_t)buf * TS_CHUNK + r) * TS_LD + lane] * X[col];
        v = warp_sum_fx(v);
        if (lane == 0) Psc[r] += v;
      }
      __syncthreads();
    }
    if (w == 0) {
      const int i = i0 + lane;
      const bool own = i <= N;
      double a = own ? Psc[lane] : 0.0;
      double mm[TS_CHUNK];
      const size_t ro = ((size_t)buf * TS_CHUNK + lane) * TS_LD;
#pragma unroll
      for (int s2 = 0; s2 < TS_CHUNK; ++s2) mm[s2] = W[ro + s2];
#pragma unroll
      for (int s2 = 0; s2 < TS_CHUNK; ++s2) {
        if (lane == s2 && own) X[i] = a;
        const double xs = __shfl_sync(FULL, a, s2);
        a = lane > s2 ? fma(mm[s2], xs, a) : a;
      }
    } else {
      const int n0 = i0 + TS_CHUNK;
      if (n0 <= N) stage(n0, i0, buf ^ 1, threadIdx.x - 32, blockDim.x - 32);
      for (int r = w - 1; r < TS_CHUNK; r += TS_WARPS - 1) {
        const int i = n0 + r;
        if (i > N) break;  // warp-uniform; later rows are out of range too
        const double *prow = Pw + moff(i, 0);
        double v0 = 0.0, v1 = 0.0;
        int j = lane;
        for (; j + 32 < i0; j += 64) {
          v0 = fma(prow[j], X[j], v0);
          v1 = fma(prow[j + 32], X[j + 32], v1);
        }
        if (j < i0) v0 = fma(prow[j], X[j], v0);
        const double v = warp_sum_fx(v0 + v1);
        if (lane == 0) Ps[(buf ^ 1) * TS_CHUNK + r] = cvec[i] + v;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *acc += X[N] + add;
}

size_t vbn_scratch_doubles(int N) { return ntri(N) + N + 2; }

// The same estimator from the cycle probabilities.  The recursion's res[N]
// is the expectation of -sum over cycles of E2 when cycles are drawn as the
// recursion draws them (last cycle of n particles has length k with
// probability p_{n,k}); the probability that the cycle j..l occurs is
// G[l][j] (j <= l), the connection probability of the exchange forces
// (md_pimd_x.c:2588-2620).  So
//   res[N] = -sum_l sum_{j<=l} G[l][j] E2[l][l-j+1],
// every term independent: row sums (a block per row), then one block adds
// the rows in order.
__global__ void __launch_bounds__(256) k_est_rows(int N, const double *__restrict__ G, const double *__restrict__ E2,
                                                  double *__restrict__ part) {
  __shared__ double buf[33];
  const int l = blockIdx.x + 1;
  const double *grow = G + (size_t)(l - 1) * N, *erow = E2 + dtri(l);
  double v = 0.0;
  for (int j = threadIdx.x + 1; j <= l; j += blockDim.x) v = fma(grow[j - 1], erow[l - j], v);
  v = block_sum(v, buf);
  if (threadIdx.x == 0) part[l - 1] = v;
}

__global__ void __launch_bounds__(1024) k_est_total(int N, const double *__restrict__ part, double add,
                                                    double *acc) {
  __shared__ double buf[33];
  double v = 0.0;
  for (int i = threadIdx.x; i < N; i += blockDim.x) v += part[i];
  v = block_sum(v, buf);
  if (threadIdx.x == 0) *acc += add - v;
}

cudaError_t vbn_energy(int N, double beta, double vi, double add, const double *ENk, const double *VBN,
                       const double *ENk2, double *acc, double *scratch, cudaStream_t st, const double *G) {
  if (G) {
    {
      XK_PROF("est_rows");
      k_est_rows<<<N, 256, 0, st>>>(N, G, ENk2 ? ENk2 : ENk, scratch);
    }
    cudaError_t e = XK_LAUNCHED();
    if (e != cudaSuccess) return e;
    {
      XK_PROF("est_total");
      k_est_total<<<1, 1024, 0, st>>>(N, scratch, add, acc);
    }
    return XK_LAUNCHED();
  }
  double *Pw = scratch, *cvec = scratch + ntri(N) + 1;
  {
    XK_PROF("est_weights");
    k_est_weights<<<cdiv((size_t)N * 32, 256), 256, 0, st>>>(N, beta, vi, ENk, VBN, ENk2 ? ENk2 : ENk, Pw, cvec);
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  const size_t smem = sizeof(double) * (N + 1 + 2 * TS_CHUNK + 4 * TS_CHUNK * TS_LD);
  static bool opted = false;
  if (!opted) {
    e = cudaFuncSetAttribute(k_lin_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    opted = true;
  }
  {
    XK_PROF("est_solve");
    k_lin_solve<<<1, TS_WARPS * 32, smem, st>>>(N, Pw, cvec, add, acc);
  }
  return XK_LAUNCHED();
}

// sum over beads j >= 2 of -(x_j - x_1).F m: md_pimd_x.c:4323-4345
template <int D>
__global__ void k_force_virial(Geo g, const double *__restrict__ x, const double *__restrict__ f,
                               const double *__restrict__ m, int image, double *part) {
  __shared__ double buf[33];
  double e = 0;
  const size_t nb = (size_t)(g.P - 1) * g.N;
  for (size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb;
       b += (size_t)gridDim.x * blockDim.x) {
    const int l = (int)(b % g.N), j = (int)(b / g.N) + 1;
    const double mm = m[(size_t)j * g.Ns + l];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      double t = x[sidx(j, d, l, D, g.Ns)] - x[sidx(0, d, l, D, g.Ns)];
      if (image) t = min_image(t, g.box[d], g.inv_box[d]);
      e += -t * f[sidx(j, d, l, D, g.Ns)] * mm;
    }
  }
  e = block_sum(e, buf);
  if (threadIdx.x == 0) part[blockIdx.x] = e;
}

cudaError_t force_virial(const Geo &g, const double *x, const double *f, const double *m,
                         int image, double *acc, double *scratch, cudaStream_t st) {
  int nb = cdiv((size_t)g.N * (g.P > 1 ? g.P - 1 : 1), 256);
  if (nb > 304) nb = 304;
  {
    XK_PROF("force_virial");
    DISPATCH_D(g.D, k_force_virial<D><<<nb, 256, 0, st>>>(g, x, f, m, image, scratch));
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  return reduce_into(scratch, nb, 0.5, 0.0, acc, st);
}

// -(x - c) . f m summed over all beads, c = L/2 (mode 0, md_pimd_x.c:3898-3922)
// or each particle's centroid (mode 1, :3923-3955, the centroid summed as the
// reference does, x_j / P in bead order).  One thread per particle.
template <int D>
__global__ void k_virial_about(Geo g, const double *__restrict__ x, const double *__restrict__ f,
                               const double *__restrict__ m, int mode, double *part) {
  __shared__ double buf[33];
  double e = 0;
  for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < g.N; l += gridDim.x * blockDim.x) {
    double c[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      c[d] = mode ? 0.0 : g.box[d] / 2;
      if (mode)
        for (int j = 0; j < g.P; ++j) c[d] += x[sidx(j, d, l, D, g.Ns)] / g.P;
    }
    for (int j = 0; j < g.P; ++j) {
      const double mm = m[(size_t)j * g.Ns + l];
#pragma unroll
      for (int d = 0; d < D; ++d) e += -(x[sidx(j, d, l, D, g.Ns)] - c[d]) * f[sidx(j, d, l, D, g.Ns)] * mm;
    }
  }
  e = block_sum(e, buf);
  if (threadIdx.x == 0) part[blockIdx.x] = e;
}

cudaError_t virial_about(const Geo &g, const double *x, const double *f, const double *m, int mode, double add,
                         double *acc, double *scratch, cudaStream_t st) {
  int nb = cdiv((size_t)g.N, 128);
  if (nb > 304) nb = 304;
  {
    XK_PROF("virial_about");
    DISPATCH_D(g.D, k_virial_about<D><<<nb, 128, 0, st>>>(g, x, f, m, mode, scratch));
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  return reduce_into(scratch, nb, 0.5, add, acc, st);
}

// md_simulation_x.c:858-865
__device__ inline int image_count(double x, double L) {
  const int c = (int)(fabs(x) / L);
  return x > L ? -c : (x < 0 ? c + 1 : 0);
}

// md_pimd_x.c:4350-4374: every bead of a ring polymer shifted by the image
// count of its first bead; one thread per (dimension, particle)
__global__ void k_polymer_wrap(Geo g, double *x) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.D * g.N) return;
  const int d = t / g.N, l = t % g.N;
  const double L = g.box[d];
  const int c = image_count(x[sidx(0, d, l, g.D, g.Ns)], L);
  if (c == 0) return;
  const double sh = __dmul_rn((double)c, L);
  for (int j = 0; j < g.P; ++j) {
    const size_t o = sidx(j, d, l, g.D, g.Ns);
    x[o] = __dadd_rn(x[o], sh);
  }
}

cudaError_t polymer_wrap(const Geo &g, double *x, cudaStream_t st) {
  {
    XK_PROF("polymer_wrap");
    k_polymer_wrap<<<cdiv((size_t)g.D * g.N, 128), 128, 0, st>>>(g, x);
  }
  return XK_LAUNCHED();
}

// md_pimd_x.c:3081-3108: histogram of the distances from bead 1 of l to bead
// jb of every other particle, bin (int)(r / incre) below `points`.  Every
// operation of the distance is the reference's, rounded alike (no fused
// multiply-add: md_minimum_image_x is a += L/2, a += L count, a - L/2), so
// each distance lands in the reference's bin.  Block (32 x 8): 32 first
// beads l, 8 warps over the partners; counts in shared memory, then added
// to the global histogram.
template <int D>
__global__ void k_pair_hist(Geo g, const double *__restrict__ x, int jb, int points, double incre, int image,
                            unsigned int *hist) {
  extern __shared__ unsigned int sh_hist[];
  for (int i = threadIdx.y * 32 + threadIdx.x; i < points; i += 256) sh_hist[i] = 0;
  __syncthreads();
  const int l = blockIdx.x * 32 + threadIdx.x;
  if (l < g.N) {
    double p1[D];
#pragma unroll
    for (int d = 0; d < D; ++d) p1[d] = x[sidx(0, d, l, D, g.Ns)];
    for (int q = blockIdx.y * 8 + threadIdx.y; q < g.N; q += gridDim.y * 8) {
      if (q == l) continue;
      double s2 = 0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        double a = __dsub_rn(p1[d], x[sidx(jb, d, q, D, g.Ns)]);
        if (image) {
          const double L = g.box[d], h = L / 2;
          a = __dadd_rn(a, h);
          a = __dadd_rn(a, __dmul_rn(L, (double)image_count(a, L)));
          a = __dsub_rn(a, h);
        }
        s2 = __dadd_rn(s2, __dmul_rn(a, a));
      }
      const int k = (int)__ddiv_rn(__dsqrt_rn(s2), incre);
      if (k < points) atomicAdd(&sh_hist[k], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.y * 32 + threadIdx.x; i < points; i += 256)
    if (sh_hist[i]) atomicAdd(&hist[i], sh_hist[i]);
}

cudaError_t pair_hist(const Geo &g, const double *x, int jb, int points, double rmax, int image, unsigned int *hist,
                      cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(unsigned int) * points, st);
  if (e != cudaSuccess) return e;
  const int bx = (g.N + 31) / 32;
  int by = (2 * 152 + bx - 1) / bx;
  const int maxy = (g.N + 7) / 8;
  if (by > maxy) by = maxy;
  if (by < 1) by = 1;
  const double incre = rmax / points;
  {
    XK_PROF("pair_hist");
    DISPATCH_D(g.D, (k_pair_hist<D><<<dim3(bx, by), dim3(32, 8), sizeof(unsigned int) * points, st>>>(
                        g, x, jb, points, incre, image, hist)));
  }
  return XK_LAUNCHED();
}

__global__ void k_add_into(double *__restrict__ f, const double *__restrict__ a, size_t n) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) f[t] += a[t];
}

cudaError_t add_into(double *f, const double *a, size_t n, cudaStream_t st) {
  {
    XK_PROF("add_exchange");
    k_add_into<<<cdiv(n, 256), 256, 0, st>>>(f, a, n);
  }
  return XK_LAUNCHED();
}

__global__ void k_add_scalar(double *acc, double v) { *acc += v; }

cudaError_t add_scalar(double *acc, double v, cudaStream_t st) {
  {
    XK_PROF("add_scalar");
    k_add_scalar<<<1, 1, 0, st>>>(acc, v);
  }
  return XK_LAUNCHED();
}

}  // namespace xk

namespace xk {

// ===================================================================
// FP64 pipe probe: eight independent FMA chains per thread, enough warps to
// fill every SM.  Gives the FP64 roofline denominator of this GPU.
// ===================================================================
__global__ void k_dfma_probe(double *out, int iters, double a, double b) {
  double x0 = threadIdx.x * 1e-3, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
  double x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

double fp64_peak_tflops(cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = sms * 8, threads = 256, iters = 2048;
  double *out = nullptr;
  if (cudaMallocAsync(&out, sizeof(double) * blocks * threads, st) != cudaSuccess) return -1;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  double best = 0;
  for (int rep = 0; rep < 3; ++rep) {
    cudaEventRecord(a, st);
    k_dfma_probe<<<blocks, threads, 0, st>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(b, st);
    cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    const double tf = 2.0 * 8 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12;
    if (tf > best) best = tf;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFreeAsync(out, st);
  cudaStreamSynchronize(st);
  return cudaGetLastError() == cudaSuccess ? best : -1;
}

// FP32 pipe probe, the same shape: the roofline denominator of the FP32
// kernels of the mixed and learned forms
__global__ void k_ffma_probe(float *out, int iters, float a, float b) {
  float x0 = threadIdx.x * 1e-3f, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
  float x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
    x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
  }
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

double fp32_peak_tflops(cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = sms * 8, threads = 256, iters = 65536;
  float *out = nullptr;
  if (cudaMallocAsync(&out, sizeof(float) * blocks * threads, st) != cudaSuccess) return -1;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  double best = 0;
  for (int rep = 0; rep < 3; ++rep) {
    cudaEventRecord(a, st);
    k_ffma_probe<<<blocks, threads, 0, st>>>(out, iters, 0.999999f, 1e-7f);
    cudaEventRecord(b, st);
    cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    const double tf = 2.0 * 8 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12;
    if (tf > best) best = tf;
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFreeAsync(out, st);
  cudaStreamSynchronize(st);
  return cudaGetLastError() == cudaSuccess ? best : -1;
}

}  // namespace xk

namespace xk {

// ===================================================================
// Pair forces without any allocation (md_gb300_pair_force_noalloc_x).
//
// For callers that may not allocate device memory, the per-tile partial
// forces of k_pair_split go to this fixed array instead of a buffer from
// the allocator.  It lives in every GPU that loads the library, until the
// process exits.  k_pair_split writes every element that k_pair_finish reads,
// so nothing in it has to start at zero; concurrent calls share it and
// therefore must not overlap on the GPU.
// ===================================================================
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_SCRATCH_DOUBLES];

constexpr int NOALLOC_MAX_DEVICES = 64;
static double *g_noalloc_addr[NOALLOC_MAX_DEVICES];
static std::mutex g_noalloc_mu;

size_t pair_force_noalloc_need(const Geo &g) {
  const int T = (g.N + 31) / 32;
  return (size_t)T * g.slots();
}

cudaError_t pair_force_noalloc(const Geo &g, const PairPrm &p, const double *x, const double *m,
                               double *f, cudaStream_t st) {
  if (p.kind == PAIR_EWALD_REAL) return cudaErrorNotSupported;
  if (pair_force_noalloc_need(g) > NOALLOC_SCRATCH_DOUBLES) return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
  double *scratch;
  {
    // set-up, once per device, with that device current: the array's
    // device address (its host-side name is not a device pointer)
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      void *a = nullptr;
      e = cudaGetSymbolAddress(&a, g_noalloc_scratch);
      if (e != cudaSuccess) return e;
      g_noalloc_addr[dev] = (double *)a;
    }
    scratch = g_noalloc_addr[dev];
  }
  const int T = (g.N + 31) / 32;
  const int jobs = T * (T + 1) / 2;
  const int nb = cdiv((size_t)jobs * g.P * 32, 256);
  const PairPrm q = with_far_images(p, g);
  switch (g.D * 16 + p.kind) {
#define XK_NOALLOC_CASE(DV, K)                                                                   \
  case DV * 16 + K:                                                                              \
    k_pair_split<DV, K, false><<<nb, 256, 0, st>>>(g, q, x, m, scratch, T, jobs, 1);             \
    break;
    XK_NOALLOC_CASE(1, PAIR_GAUSSIAN)
    XK_NOALLOC_CASE(1, PAIR_PERIODIC_GAUSSIAN)
    XK_NOALLOC_CASE(1, PAIR_COULOMB)
    XK_NOALLOC_CASE(1, PAIR_PERIODIC_COULOMB)
    XK_NOALLOC_CASE(2, PAIR_GAUSSIAN)
    XK_NOALLOC_CASE(2, PAIR_PERIODIC_GAUSSIAN)
    XK_NOALLOC_CASE(2, PAIR_COULOMB)
    XK_NOALLOC_CASE(2, PAIR_PERIODIC_COULOMB)
    XK_NOALLOC_CASE(3, PAIR_GAUSSIAN)
    XK_NOALLOC_CASE(3, PAIR_PERIODIC_GAUSSIAN)
    XK_NOALLOC_CASE(3, PAIR_COULOMB)
    XK_NOALLOC_CASE(3, PAIR_PERIODIC_COULOMB)
#undef XK_NOALLOC_CASE
    default:
      return cudaErrorNotSupported;
  }
  e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  k_pair_finish<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, scratch, T, 1.0 / g.P, f);
  return XK_LAUNCHED();
}

}  // namespace xk

namespace xk {

// ===================================================================
// Mixed-precision form: pair and real-space Ewald forces in FP32, each
// lane's sum over one 32 x 32 tile (at most 32 terms) in plain FP32 and the
// tile partials added in FP64 (k_pair_finish32); reciprocal space with FP32
// phase products summed in FP32 over 16 particles and those partial sums
// in double-float (an unevaluated sum of two FP32 numbers, ~48 significant
// bits), S(k) and the force tables in FP32, and each particle's sum over
// the wave-vector columns compensated (Kahan).  Positions and every
// estimator stay FP64; partial sums leave the FP32 kernels as doubles.
// Against the FP64 form the largest force error is ~1e-5 of the largest
// force at 512 electrons, 64 beads, set by the FP32 rounding of the pair
// separations rather than by the sums.
// ===================================================================


// same tile/rotation scheme as k_pair_tiles, on FP32 copies of the positions
// and inverse masses.  Each lane's sums within a tile have 32 terms at most,
// added in FP32 (rounding ~ sqrt(32) ulp of the partial, far below the
// rounding of the FP32 positions); the per-tile partials are added in double
// by k_pair_finish32.  With one mass for all beads (q.uniform) the inverse
// mass is applied to the partials instead of to every pair.
// Bound by instruction issue (200 a step before the last of the changes here,
// 78% of the slots).  Ewald at N = 512, P = 64, alpha L = 5.6: 83 us with eight
// candidates a pair and 32 steps on the diagonal, 69 with the minimum image
// and single shifts only, where no other can lie inside the cut-off, and 16
// steps, 65 with two steps unrolled, 59 without the subnormal handling of
// rsqrtf, division and __expf.
template <int D, int KIND>
__global__ void __launch_bounds__(256, 3) k_pair_tiles32(Geo g, P32 q, const float *__restrict__ x,
                                                      const float *__restrict__ im,
                                                      float *__restrict__ out, int T, int jobs) {
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  // persistent warps: tile jobs (slice j, tile pair I <= J) in round-robin,
  // warps numbered across blocks first (the last round spreads over all SMs)
  for (int wi = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; wi < jobs * g.P; wi += nwarps) {
    pair_tile32_job<D, KIND>(g, q, x, im, out, T, jobs, wi, lane);
  }
}

// FP32 copies of the positions and inverse masses for the FP32 pair kernel
// FP32 positions and (im32 non-null: beads of different masses) inverse
// masses; with one mass for all beads the tiles apply it to their sums and
// no division is taken here; ph1 (non-null, D = 3): first phase factors,
// ph1[(j*3 + d)*Ns + l]
__global__ void k_to32(Geo g, const double *__restrict__ x, const double *__restrict__ m, float *__restrict__ x32,
                       float *__restrict__ im32, float2 *__restrict__ ph1) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < g.slots()) x32[t] = (float)x[t];
  if (ph1 && t < g.slots()) ph1[t] = phase32_slot(g, x, t);
  if (im32 && t < (size_t)g.P * g.Ns) im32[t] = (float)(1.0 / m[t]);
}

// f += scale * sum over the T partial slots, in double
__global__ void k_pair_finish32(Geo g, const float *__restrict__ part, int T, double scale,
                                double *__restrict__ f) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.slots() || (int)(s % g.Ns) >= g.N) return;
  f[s] += pair_sum32(g, part, T, s) * scale;
}

// Tile shape of the FP32 pair kernel: warps (32 x 32 pair tiles) per block,
// by system shape.  Chosen by the autotuner (md_gb300_autotune_pair_x); 8
// unless tuned.  Results do not depend on it: every tile job writes its own
// partial-sum slots.
static std::mutex g_tune_mu;
static std::vector<std::pair<std::array<int, 4>, int>> g_tune;

void set_pair32_warps(int kind, int D, int N, int P, int warps) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  for (auto &e : g_tune)
    if (e.first == std::array<int, 4>{kind, D, N, P}) {
      e.second = warps;
      return;
    }
  g_tune.push_back({{kind, D, N, P}, warps});
}

int pair32_warps(int kind, int D, int N, int P) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  for (auto &e : g_tune)
    if (e.first == std::array<int, 4>{kind, D, N, P}) return e.second;
  return 8;
}

// persistent grid: as many blocks of `wpb` warps as the kernel keeps
// resident, or fewer when the jobs run out
template <int D, int K>
static cudaError_t launch_pair32(const Geo &g, const P32 &q, const float *x, const float *im, float *part, int T,
                                 int jobs, int wpb, cudaStream_t st) {
  static int occ[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
  }
  if (!occ[wpb]) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ[wpb], k_pair_tiles32<D, K>, wpb * 32, 0);
    if (e != cudaSuccess) return e;
    if (occ[wpb] < 1) occ[wpb] = 1;
  }
  const size_t need = ((size_t)jobs * g.P + wpb - 1) / wpb, full = (size_t)sms * occ[wpb];
  k_pair_tiles32<D, K><<<(int)(need < full ? need : full), wpb * 32, 0, st>>>(g, q, x, im, part, T, jobs);
  return cudaSuccess;
}

// the FP32 pair kernel's constants for a system and potential
P32 make_p32(const Geo &g, const PairPrm &p) {
  P32 q{};
  for (int d = 0; d < 3; ++d) {
    q.L[d] = (float)g.box[d];
    q.iL[d] = (float)g.inv_box[d];
  }
  q.igs2 = p.s != 0 ? (float)(1.0 / (p.s * p.s)) : 0.f;
  q.gpre = p.s != 0 ? (float)(p.g / (M_PI * p.s * p.s) * (2.0 / (p.s * p.s))) : 0.f;
  q.qs = (float)p.qs;
  q.alpha = (float)p.alpha;
  q.nsum = p.nsum;
  const double rc32 = p.alpha > 0 ? fmin(p.rcut, (double)EW32_XCUT / p.alpha) : 0.0;
  q.rc2 = (float)(rc32 * rc32);
  q.kmax = p.kmax[0] > p.kmax[1] ? (p.kmax[0] > p.kmax[2] ? p.kmax[0] : p.kmax[2])
                                 : (p.kmax[1] > p.kmax[2] ? p.kmax[1] : p.kmax[2]);
  if (p.kind == PAIR_EWALD_REAL && rc32 <= fmin(g.box[0], fmin(g.box[1], g.box[2]))) q.kmax = 0;
  if (q.kmax == 0 && p.kind == PAIR_EWALD_REAL) {
    // (1e-5: the FP32 rounding of the separations)
    double two = 1e300;
    for (int d = 0; d < 3; ++d) {
      const double e = g.box[(d + 1) % 3];
      two = fmin(two, (g.box[d] * g.box[d] + e * e) / 4);
    }
    q.single = rc32 * rc32 < two * (1 - 1e-5);
  }
  q.uniform = p.inv_mass > 0;
  q.im0 = (float)p.inv_mass;
  return q;
}

// scratch of the FP32 pair forces: T * slots float partials (room for twice
// that is reserved), then the FP32 positions and inverse masses
struct P32Bufs {
  int T;
  float *part, *x32, *im32;
};
static P32Bufs p32_bufs(const Geo &g, double *scratch) {
  const int T = (g.N + 31) / 32;
  float *x32 = (float *)(scratch + (size_t)T * g.slots());
  return {T, (float *)scratch, x32, x32 + g.slots()};
}
static cudaError_t pair_tiles32(const Geo &g, const PairPrm &p, const P32 &q, const P32Bufs &b, cudaStream_t st) {
  const int jobs = b.T * (b.T + 1) / 2;
  int wpb = pair32_warps(p.kind, g.D, g.N, g.P);
  if (wpb != 1 && wpb != 2 && wpb != 4 && wpb != 8) wpb = 8;
  cudaError_t le = cudaSuccess;
  XK_PROF(p.kind == PAIR_EWALD_REAL ? "pair_tiles32_ewald_real" : "pair_tiles32");
  switch (g.D * 16 + p.kind) {
#define XK_P32_CASE(DV, K) \
  case DV * 16 + K:        \
    le = launch_pair32<DV, K>(g, q, b.x32, b.im32, b.part, b.T, jobs, wpb, st); \
    break;
    XK_P32_CASE(1, PAIR_GAUSSIAN)
    XK_P32_CASE(1, PAIR_PERIODIC_GAUSSIAN)
    XK_P32_CASE(1, PAIR_COULOMB)
    XK_P32_CASE(1, PAIR_PERIODIC_COULOMB)
    XK_P32_CASE(2, PAIR_GAUSSIAN)
    XK_P32_CASE(2, PAIR_PERIODIC_GAUSSIAN)
    XK_P32_CASE(2, PAIR_COULOMB)
    XK_P32_CASE(2, PAIR_PERIODIC_COULOMB)
    XK_P32_CASE(3, PAIR_GAUSSIAN)
    XK_P32_CASE(3, PAIR_PERIODIC_GAUSSIAN)
    XK_P32_CASE(3, PAIR_COULOMB)
    XK_P32_CASE(3, PAIR_PERIODIC_COULOMB)
    XK_P32_CASE(3, PAIR_EWALD_REAL)
#undef XK_P32_CASE
    default:
      return cudaErrorInvalidValue;
  }
  return le != cudaSuccess ? le : XK_LAUNCHED();
}

cudaError_t pair_force32(const Geo &g, const PairPrm &p, const double *x, const double *m, double *f,
                         double *scratch, cudaStream_t st) {
  const P32 q = make_p32(g, p);
  const P32Bufs b = p32_bufs(g, scratch);
  {
    XK_PROF("to32");
    k_to32<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, x, m, b.x32, q.uniform ? nullptr : b.im32, nullptr);
  }
  cudaError_t e = XK_LAUNCHED();
  if (e == cudaSuccess) e = pair_tiles32(g, p, q, b, st);
  if (e != cudaSuccess) return e;
  {
    XK_PROF("pair_finish");
    k_pair_finish32<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, b.part, b.T, 1.0 / g.P, f);
  }
  return XK_LAUNCHED();
}

// ---- reciprocal space, mixed ----------------------------------------
// a block per (slice, 32 items), the longest items' blocks first
__global__ void __launch_bounds__(SK_T, 2) k_sk32(Geo g, int ns, int ncol, int nlong, const int4 *__restrict__ cols,
                                                  const float *__restrict__ coef32, const float2 *__restrict__ ph1,
                                                  float4 *__restrict__ T) {
  extern __shared__ __align__(16) float2 sk32_sh[];
  sk32_group(g, ns, ncol, nlong, cols, coef32, ph1, T, blockIdx.x, blockIdx.y, sk32_sh);
}

// a block per slice and 32 of its particles (recip_tile32); four blocks an SM
// (64 registers) or three (80) at N = 512, P = 64 36 us each, four better where
// the columns are few
template <int NS>
__global__ void __launch_bounds__(SK_T, 4) k_recip_force32(Geo g, int ncol, const int4 *__restrict__ cols,
                                                           const float2 *__restrict__ ph1,
                                                           const float4 *__restrict__ T, double scale,
                                                           double *__restrict__ f, const float *__restrict__ part,
                                                           int ntile, double pscale) {
  extern __shared__ __align__(16) float4 rf32_sh[];
  float4 *sT = rf32_sh;
  RecipCol *sc = (RecipCol *)(sT + ncol * (NS + 1));
  const int j = blockIdx.y;
  const float4 *Tj = T + (size_t)j * ncol * (NS + 1);
  for (int q = threadIdx.x; q < ncol * (NS + 1); q += SK_T) sT[q] = Tj[q];
  for (int q = threadIdx.x; q < ncol; q += SK_T) sc[q] = recip_col32(cols[q], NS);
  recip_tile32<NS, false>(g, NS, ncol, ncol, [](int, int) {}, sc, sT, (float2 *)(sc + ncol), (float2 *)rf32_sh, ph1,
                          scale, f, j, blockIdx.x * 32, threadIdx.x >> 5, threadIdx.x & 31, part, ntile, pscale);
}

// The mixed form's Ewald forces: FP32 positions and phases, real-space tiles,
// structure factors with their force tables, and the forces of both sums in
// four launches (separate copies, phases and a finishing kernel for the tiles
// were six: 199 us a step of N = 512, P = 64 then, 196 now).  The tiles, which fill
// the GPU, come after the structure factors: beside a learned residual, its own
// stream's chain then starts early (222 us a step with the tiles first, 211).  The tables use
// the FP64 form's buffer, the phases lie behind the FP64 ones.
cudaError_t ewald_force32(const Geo &g, const PairPrm &p, const Recip &r, const double *x, const double *m,
                          double inv_mP, double *f, double *scratch, cudaStream_t st) {
  if (g.D != 3) return cudaErrorInvalidValue;
  if (r.ncol <= 0) return pair_force32(g, p, x, m, f, scratch, st);
  const P32 q = make_p32(g, p);
  const P32Bufs b = p32_bufs(g, scratch);
  float2 *ph1 = (float2 *)(r.phase + recip_phase_doubles(g, r.nsum));
  {
    XK_PROF("to32");
    k_to32<<<cdiv(g.slots(), 256), 256, 0, st>>>(g, x, m, b.x32, q.uniform ? nullptr : b.im32, ph1);
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess) return e;
  {
    XK_PROF("sk32");
    static bool opted = false;
    if (!opted) {
      e = cudaFuncSetAttribute(k_sk32, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      opted = true;
    }
    k_sk32<<<dim3(g.P, sk32_groups(r.ncol, r.nlong)), SK_T, sk32_smem(r.nsum), st>>>(
        g, r.nsum, r.ncol, r.nlong, (const int4 *)r.kvec, (const float *)(r.coef + r.nk), ph1, (float4 *)r.T);
  }
  e = XK_LAUNCHED();
  if (e == cudaSuccess) e = pair_tiles32(g, p, q, b, st);
  if (e != cudaSuccess) return e;
  XK_PROF("recip_force32");
  DISPATCH_NS(r.nsum, {
    auto kf = k_recip_force32<NS>;
    static bool opted = false;
    if (!opted) {
      e = cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      if (e != cudaSuccess) return e;
      opted = true;
    }
    const size_t tab = (sizeof(float4) * (NS + 1) + sizeof(RecipCol)) * r.ncol + sizeof(float2) * 2 * (NS + 1) * 32;
    const size_t red = sizeof(float2) * SK_W * 3 * 32;
    kf<<<dim3((g.N + 31) / 32, g.P), SK_T, tab > red ? tab : red, st>>>(
        g, r.ncol, (const int4 *)r.kvec, ph1, (const float4 *)r.T, 4 * M_PI * inv_mP, f, b.part, b.T, 1.0 / g.P);
  });
  return XK_LAUNCHED();
}

}  // namespace xk
