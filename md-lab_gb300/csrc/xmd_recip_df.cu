// xmd_recip_df.cu -- the FP64 form's reciprocal-space Ewald sums in
// double-float arithmetic (xmd_df.cuh), and their small terms in FP32, in
// one set of kernels: phase factors, structure factors, force tables, forces.
//
// The sums are those of xmd_kernels.cu (columns of wave vectors (nx, ny)
// with +-nz pairs; recip_setup's kept vectors).  Vectors whose force weight
// |G| c(n) is at least RECIP_DF_SPLIT of the largest (at alpha L = 5.6 those
// with |n|^2 <= 52, a sphere) are summed in pairs of FP32 numbers with 48
// significant bits; the others, 70% of the kept ones at |n| <= 10, in FP32
// from the pairs' high parts, where a rounding of a few 1e-7 leaves below
// 1e-14 of the reciprocal force.  Why not FP64: a warp's FP64 instruction
// holds that pipe for 64 cycles, against about 12 FP32 instructions for a
// double-float multiply-add.
#include <algorithm>
#include <cmath>
#include <vector>

#include "xmd_df.cuh"
#include "xmd_kernels.cuh"

namespace xk {

constexpr unsigned ALL = 0xffffffffu;
static inline int cdivz(size_t a, int b) { return (int)((a + b - 1) / b); }

struct dfc {  // complex pair
  df r, i;
};
__device__ __forceinline__ dfc unpack(float4 v) { return {{v.x, v.z}, {v.y, v.w}}; }
__device__ __forceinline__ float4 pack(df r, df i) {
  r = df_norm(r), i = df_norm(i);
  return make_float4(r.h, i.h, r.l, i.l);
}
__device__ __forceinline__ dfc mul(dfc a, dfc b) {
  return {df_sub(df_mul(a.r, b.r), df_mul(a.i, b.i)), df_add(df_mul(a.r, b.i), df_mul(a.i, b.r))};
}
// acc += a b
__device__ __forceinline__ void fma_to(df &acc, df a, df b) {
  df p = two_prod(a.h, b.h);
  p.l = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l));
  const df s = two_sum(acc.h, p.h);
  acc.h = s.h;
  acc.l = __fadd_rn(acc.l, __fadd_rn(s.l, p.l));
}
__device__ __forceinline__ df neg(df a) { return {-a.h, -a.l}; }
// n a, n a small integer
__device__ __forceinline__ df times(float n, df a) {
  df p = two_prod(n, a.h);
  p.l = __fmaf_rn(n, a.l, p.l);
  return p;
}
__device__ __forceinline__ df shfl_xor(unsigned mask, df a, int o) {
  return {__shfl_xor_sync(mask, a.h, o), __shfl_xor_sync(mask, a.l, o)};
}

// column record: x = nx | nzmax << 8 | (nzs + 1) << 16, y = ny, z = first nz, w = offset of its first vector;
// harmonics |nz| <= nzs (nzs = -1: none) are double-float, the rest up to nzmax FP32
__host__ __device__ inline int dc_nx(int4 c) { return c.x & 255; }
__host__ __device__ inline int dc_nz(int4 c) { return (c.x >> 8) & 255; }
__host__ __device__ inline int dc_nzs(int4 c) { return (c.x >> 16) - 1; }

constexpr int DF_NG = 4;  // harmonics of one structure-factor item

// ints of the double-float tables: columns, table offsets, items
static int ncols_of(int ns) { return ns * (2 * ns + 1) + ns + 1; }
static size_t toff_at(int ns) { return 4 * (size_t)ncols_of(ns); }
static size_t items_at(int ns) { return toff_at(ns) + (((size_t)ncols_of(ns) + 1 + 3) & ~(size_t)3); }
size_t recip_df_ints(int ns) { return items_at(ns) + (size_t)ncols_of(ns) * ((ns + DF_NG - 1) / DF_NG); }

// Host tables from recip_setup's kept columns (x = nx | nzmax << 8) and the
// vectors' force weights.  Items (column, group of DF_NG harmonics): those
// with a double-float harmonic first, so that a warp's threads run one kind.
void recip_df_tables(int ns, const std::vector<int4> &kept, const std::vector<double> &wgt, double wmax, Recip &r,
                     std::vector<int> &out) {
  struct C {
    int nzs, nzmax;
    int4 c;
  };
  std::vector<C> cs;
  for (const int4 &k : kept) {
    const int nzmax = k.x >> 8;
    int nzs = -1;
    for (int nz = k.z < 0 ? 0 : k.z; nz <= nzmax; ++nz)
      if (wgt[k.w + nz - k.z] >= RECIP_DF_SPLIT * wmax) nzs = nz;
    cs.push_back({nzs, nzmax, make_int4((k.x & 255) | (nzmax << 8) | ((nzs + 1) << 16), k.y, k.z, k.w)});
  }
  std::stable_sort(cs.begin(), cs.end(), [](const C &a, const C &b) {
    return a.nzs != b.nzs ? a.nzs > b.nzs : a.nzmax > b.nzmax;
  });
  out.assign(recip_df_ints(ns), 0);
  std::vector<int> dfi, fpi;
  int off = 0;
  for (size_t i = 0; i < cs.size(); ++i) {
    const int4 c = cs[i].c;
    const int v[4] = {c.x, c.y, c.z, c.w};
    std::copy(v, v + 4, out.begin() + 4 * i);
    out[toff_at(ns) + i] = off;
    const int s = std::max(cs[i].nzs, 0);
    off += 1 + 4 * s + (cs[i].nzmax - s);
    for (int g = 0; g == 0 || g * DF_NG < cs[i].nzmax; ++g) {
      const bool d = g == 0 ? cs[i].nzs >= 0 : g * DF_NG + 1 <= cs[i].nzs;
      (d ? dfi : fpi).push_back((int)i | g << 16);
    }
  }
  out[toff_at(ns) + cs.size()] = off;
  // items of one harmonic group side by side: their threads read the same z factors
  auto by_group = [](int a, int b) { return (a >> 16) < (b >> 16); };
  std::stable_sort(dfi.begin(), dfi.end(), by_group);
  std::stable_sort(fpi.begin(), fpi.end(), by_group);
  std::copy(dfi.begin(), dfi.end(), out.begin() + items_at(ns));
  std::copy(fpi.begin(), fpi.end(), out.begin() + items_at(ns) + dfi.size());
  r.df_items = (int)dfi.size();
  r.items = (int)(dfi.size() + fpi.size());
  r.tdf = off;
}

// ph[((j*3 + d)*(ns+1) + n)*Ns + l] = exp(i 2 pi n x / L): the first harmonic
// in FP64 from the exact fraction of x/L, the others by double-float products
__global__ void __launch_bounds__(128) k_df_phase(Geo g, int ns, const double *__restrict__ x,
                                                  float4 *__restrict__ ph) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.P * 3 * g.Ns) return;
  const int l = t % g.Ns, jd = t / g.Ns, d = jd % 3;
  double s = 0, c = 1;
  if (l < g.N) {
    const double u = x[t] * g.inv_box[d];
    sincospi(2.0 * (u - rint(u)), &s, &c);
  }
  const float ch = (float)c, sh = (float)s;
  const dfc e = {{ch, (float)(c - ch)}, {sh, (float)(s - sh)}};
  float4 *o = ph + (size_t)jd * (ns + 1) * g.Ns + l;
  o[0] = make_float4(1.f, 0.f, 0.f, 0.f);
  dfc w = e;
  for (int n = 1; n <= ns; ++n) {
    const float4 v = pack(w.r, w.i);
    o[(size_t)n * g.Ns] = v;
    w = mul(unpack(v), e);
  }
}

// Structure factors: GR threads share an item (column and DF_NG harmonics)
// of a slice, particles interleaved; phases staged DF_CH particles at a
// time.  With P = sum e_xy cos(nz theta_z), Q = sum e_xy sin(nz theta_z):
// S(+nz) = P + iQ, S(-nz) = P - iQ.  The FP32 items add their products in
// FP32 over 16 particles and those sums in double-float.
// Bound: FP32 issue of the double-float items (about 230 instructions a
// particle and item).
constexpr int DF_CH = 64, DF_SK_T = 512, DF_GR = 8;
template <int NS>
__global__ void __launch_bounds__(DF_SK_T, 1)
    k_df_sk(int N, int Ns, const float4 *__restrict__ ph, const int4 *__restrict__ cols, const int *__restrict__ items,
            int ndf, int nitems, float4 *__restrict__ S, int nk) {
  constexpr int LD = DF_CH + 1;
  extern __shared__ __align__(16) float4 df_sp[];  // [3][NS + 1][LD]
  const int j = blockIdx.y, gq = threadIdx.x % DF_GR;
  const int it = blockIdx.x * (DF_SK_T / DF_GR) + threadIdx.x / DF_GR;
  const bool live = it < nitems, isdf = it < ndf;
  const int item = live ? items[it] : 0;
  const int4 c = cols[item & 0xffff];
  const int n0 = (item >> 16) * DF_NG, nzmax = live ? dc_nz(c) : 0;
  const float4 *px = df_sp + dc_nx(c) * LD, *py = df_sp + (NS + 1 + abs(c.y)) * LD, *pz = df_sp + 2 * (NS + 1) * LD;
  const float sy = c.y < 0 ? -1.f : 1.f;
  df s0r = {0.f, 0.f}, s0i = {0.f, 0.f}, Pr[DF_NG], Pi[DF_NG], Qr[DF_NG], Qi[DF_NG];
#pragma unroll
  for (int u = 0; u < DF_NG; ++u) Pr[u] = Pi[u] = Qr[u] = Qi[u] = {0.f, 0.f};
  const float4 *base = ph + (size_t)j * 3 * (NS + 1) * Ns;
  for (int l0 = 0; l0 < N; l0 += DF_CH) {
    const int cnt = N - l0 < DF_CH ? N - l0 : DF_CH;
    __syncthreads();
    for (int q = threadIdx.x; q < 3 * (NS + 1) * DF_CH; q += DF_SK_T) {
      const int l = q % DF_CH, row = q / DF_CH;
      if (l < cnt) df_sp[row * LD + l] = base[(size_t)row * Ns + l0 + l];
    }
    __syncthreads();
    if (!live) continue;
    if (isdf) {
      for (int l = gq; l < cnt; l += DF_GR) {
        const dfc ex = unpack(px[l]);
        dfc ey = unpack(py[l]);
        ey.i.h *= sy, ey.i.l *= sy;
        const dfc e = mul(ex, ey);
        s0r = df_add(s0r, e.r);
        s0i = df_add(s0i, e.i);
#pragma unroll
        for (int u = 0; u < DF_NG; ++u) {
          if (n0 + u + 1 > nzmax) break;
          const dfc ez = unpack(pz[(n0 + u + 1) * LD + l]);
          fma_to(Pr[u], e.r, ez.r);
          fma_to(Pi[u], e.i, ez.r);
          fma_to(Qr[u], e.r, ez.i);
          fma_to(Qi[u], e.i, ez.i);
        }
      }
    } else {
      // at most DF_CH / DF_GR = 8 terms a chunk, in FP32
      float a0 = 0.f, a1 = 0.f, p[DF_NG][4];
#pragma unroll
      for (int u = 0; u < DF_NG; ++u) p[u][0] = p[u][1] = p[u][2] = p[u][3] = 0.f;
      for (int l = gq; l < cnt; l += DF_GR) {
        const float4 ex = px[l], ey = py[l];
        const float yi = sy * ey.y;
        const float er = fmaf(ex.x, ey.x, -ex.y * yi), ei = fmaf(ex.x, yi, ex.y * ey.x);
        a0 += er;
        a1 += ei;
#pragma unroll
        for (int u = 0; u < DF_NG; ++u) {
          if (n0 + u + 1 > nzmax) break;
          const float4 ez = pz[(n0 + u + 1) * LD + l];
          p[u][0] = fmaf(er, ez.x, p[u][0]);
          p[u][1] = fmaf(ei, ez.x, p[u][1]);
          p[u][2] = fmaf(er, ez.y, p[u][2]);
          p[u][3] = fmaf(ei, ez.y, p[u][3]);
        }
      }
      s0r = df_add(s0r, {a0, 0.f});
      s0i = df_add(s0i, {a1, 0.f});
#pragma unroll
      for (int u = 0; u < DF_NG; ++u) {
        Pr[u] = df_add(Pr[u], {p[u][0], 0.f});
        Pi[u] = df_add(Pi[u], {p[u][1], 0.f});
        Qr[u] = df_add(Qr[u], {p[u][2], 0.f});
        Qi[u] = df_add(Qi[u], {p[u][3], 0.f});
      }
    }
  }
#pragma unroll
  for (int o = 1; o < DF_GR; o <<= 1) {
    s0r = df_add(s0r, shfl_xor(ALL, s0r, o));
    s0i = df_add(s0i, shfl_xor(ALL, s0i, o));
#pragma unroll
    for (int u = 0; u < DF_NG; ++u) {
      Pr[u] = df_add(Pr[u], shfl_xor(ALL, Pr[u], o));
      Pi[u] = df_add(Pi[u], shfl_xor(ALL, Pi[u], o));
      Qr[u] = df_add(Qr[u], shfl_xor(ALL, Qr[u], o));
      Qi[u] = df_add(Qi[u], shfl_xor(ALL, Qi[u], o));
    }
  }
  if (!live || gq != 0) return;
  float4 *o = S + (size_t)j * nk + c.w - c.z;  // o[nz]
  if (n0 == 0 && c.z <= 0) o[0] = pack(s0r, s0i);
#pragma unroll
  for (int u = 0; u < DF_NG; ++u) {
    const int n = n0 + u + 1;
    if (n > nzmax) break;
    o[n] = pack(df_sub(Pr[u], Qi[u]), df_add(Pi[u], Qr[u]));
    if (c.z < 0) o[-n] = pack(df_add(Pr[u], Qi[u]), df_sub(Pi[u], Qr[u]));
  }
}

__device__ __forceinline__ float4 pack64(double r, double i) {
  const float rh = (float)r, ih = (float)i;
  return make_float4(rh, ih, (float)(r - rh), (float)(i - ih));
}

// Force tables of a slice, compact: per column W(0), then A, B, n A, n B (as
// in k_recip_tables) per double-float harmonic, then (A, B) in FP32 per
// remaining one.
template <int NS>
__global__ void k_df_tables(const int4 *__restrict__ cols, const int *__restrict__ toff, int ncol,
                            const float4 *__restrict__ S, const double *__restrict__ coef, int nk, int tdf,
                            float4 *__restrict__ T) {
  const int j = blockIdx.y, ci = blockIdx.x * blockDim.y + threadIdx.y, n = threadIdx.x;
  if (ci >= ncol) return;
  const int4 c = cols[ci];
  if (n > dc_nz(c)) return;
  auto W = [&](int nz) {
    if (nz < c.z) return make_double2(0.0, 0.0);
    const int k = c.w + (nz - c.z);
    const float4 s = S[(size_t)j * nk + k];
    return make_double2(coef[k] * ((double)s.x + s.z), -coef[k] * ((double)s.y + s.w));
  };
  float4 *o = T + (size_t)j * tdf + toff[ci];
  const int nzs = dc_nzs(c) > 0 ? dc_nzs(c) : 0;
  if (n == 0) {
    const double2 w = W(0);
    o[0] = pack64(w.x, w.y);
    return;
  }
  const double2 wp = W(n), wm = W(-n);
  const double2 A = make_double2(wp.x + wm.x, wp.y + wm.y), B = make_double2(wp.x - wm.x, wp.y - wm.y);
  if (n <= nzs) {
    o[4 * n - 3] = pack64(A.x, A.y);
    o[4 * n - 2] = pack64(B.x, B.y);
    o[4 * n - 1] = pack64(n * A.x, n * A.y);
    o[4 * n] = pack64(n * B.x, n * B.y);
  } else {
    o[4 * nzs + (n - nzs)] = make_float4((float)A.x, (float)A.y, (float)B.x, (float)B.y);
  }
}

// Forces: TPP threads share a particle, thread h taking columns h, h + TPP,
// ... (sorted by length, so that neighbours run alike); tables, columns and
// the block's x and y phase factors in shared memory, the z factors in
// registers.  Per column, with U = sum_nz e_z W and V = sum_nz nz e_z W:
// F_x, F_y from Im(e_xy U), F_z from Im(e_xy V).
// Bound: FP32 issue (eight double-float multiply-adds a harmonic, 96
// instructions).
constexpr int DF_RF_T = 256;
template <int NS, int TPP>
__global__ void __launch_bounds__(DF_RF_T, 2)
    k_df_force(Geo g, const float4 *__restrict__ ph, const int4 *__restrict__ cols, const int *__restrict__ toff,
               int ncol, const float4 *__restrict__ T, int tdf, double scale, double *__restrict__ f) {
  constexpr int PPB = DF_RF_T / TPP;
  extern __shared__ __align__(16) float4 df_sm[];
  float4 *sT = df_sm, *pxy = df_sm + tdf;                // [tdf], [2 (NS + 1)][PPB]
  int4 *sc = (int4 *)(pxy + 2 * (NS + 1) * PPB);         // [ncol]
  int *so = (int *)(sc + ncol);                          // [ncol]
  const int j = blockIdx.y, l0 = blockIdx.x * PPB;
  const float4 *Tj = T + (size_t)j * tdf, *pj = ph + (size_t)j * 3 * (NS + 1) * g.Ns;
  for (int q = threadIdx.x; q < tdf; q += DF_RF_T) sT[q] = Tj[q];
  for (int q = threadIdx.x; q < ncol; q += DF_RF_T) sc[q] = cols[q], so[q] = toff[q];
  for (int q = threadIdx.x; q < 2 * (NS + 1) * PPB; q += DF_RF_T) {
    const int r = q / PPB, l = l0 + q % PPB;
    if (l < g.N) pxy[q] = pj[(size_t)r * g.Ns + l];
  }
  __syncthreads();
  const int li = threadIdx.x / TPP, h = threadIdx.x % TPP, l = l0 + li;
  if (l >= g.N) return;  // a particle's TPP lanes leave together
  dfc ez[NS];
#pragma unroll
  for (int n = 1; n <= NS; ++n) ez[n - 1] = unpack(pj[((size_t)2 * (NS + 1) + n) * g.Ns + l]);
  df F[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) F[d] = {0.f, 0.f};
  for (int ci = h; ci < ncol; ci += TPP) {
    const int4 c = sc[ci];
    const int nzs = dc_nzs(c), nzc = dc_nz(c);
    const float4 *t = sT + so[ci];
    const float4 vx = pxy[dc_nx(c) * PPB + li];
    float4 vy = pxy[(NS + 1 + abs(c.y)) * PPB + li];
    if (c.y < 0) vy.y = -vy.y, vy.w = -vy.w;
    const float4 w0 = t[0];
    // the FP32 harmonics
    float ur = 0.f, ui = 0.f, vr = 0.f, vi = 0.f;
    const float4 *tt = t + 3 * max(nzs, 0);
#pragma unroll
    for (int n = 1; n <= NS; ++n) {
      if (n > nzc) break;
      if (n <= nzs) continue;
      const float4 ab = tt[n];
      const float cz = ez[n - 1].r.h, sz = ez[n - 1].i.h;
      ur = fmaf(cz, ab.x, fmaf(-sz, ab.w, ur));
      ui = fmaf(cz, ab.y, fmaf(sz, ab.z, ui));
      vr = fmaf((float)n, fmaf(cz, ab.z, -sz * ab.y), vr);
      vi = fmaf((float)n, fmaf(cz, ab.w, sz * ab.x), vi);
    }
    if (nzs < 0) {
      ur += w0.x;
      ui += w0.y;
      const float er = fmaf(vx.x, vy.x, -vx.y * vy.y), ei = fmaf(vx.x, vy.y, vx.y * vy.x);
      const float Tm = fmaf(er, ui, ei * ur), Zm = fmaf(er, vi, ei * vr);
      F[0] = df_add(F[0], {(float)dc_nx(c) * Tm, 0.f});
      F[1] = df_add(F[1], {(float)c.y * Tm, 0.f});
      F[2] = df_add(F[2], {Zm, 0.f});
      continue;
    }
    const dfc e = mul(unpack(vx), unpack(vy));
    df Ur = {w0.x, w0.z}, Ui = {w0.y, w0.w}, Vr = {0.f, 0.f}, Vi = {0.f, 0.f};
#pragma unroll
    for (int n = 1; n <= NS; ++n) {
      if (n > nzs) break;
      const dfc A = unpack(t[4 * n - 3]), B = unpack(t[4 * n - 2]), nA = unpack(t[4 * n - 1]), nB = unpack(t[4 * n]);
      const df cz = ez[n - 1].r, sz = ez[n - 1].i, mz = neg(sz);
      fma_to(Ur, cz, A.r);
      fma_to(Ur, mz, B.i);
      fma_to(Ui, cz, A.i);
      fma_to(Ui, sz, B.r);
      fma_to(Vr, cz, nB.r);
      fma_to(Vr, mz, nA.i);
      fma_to(Vi, cz, nB.i);
      fma_to(Vi, sz, nA.r);
    }
    Ur = df_add(Ur, {ur, 0.f}), Ui = df_add(Ui, {ui, 0.f});
    Vr = df_add(Vr, {vr, 0.f}), Vi = df_add(Vi, {vi, 0.f});
    const df Tm = df_add(df_mul(e.r, Ui), df_mul(e.i, Ur));
    F[0] = df_add(F[0], times((float)dc_nx(c), Tm));
    F[1] = df_add(F[1], times((float)c.y, Tm));
    fma_to(F[2], e.r, Vi);
    fma_to(F[2], e.i, Vr);
  }
  const unsigned gm = TPP >= 32 ? ALL : ((1u << TPP) - 1u) << ((threadIdx.x & 31) & ~(TPP - 1));
#pragma unroll
  for (int o = 1; o < TPP; o <<= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) F[d] = df_add(F[d], shfl_xor(gm, F[d], o));
  if (h != 0) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) f[sidx(j, d, l, 3, g.Ns)] += scale * df_value(F[d]) * g.inv_box[d];
}

// slice energies sum_n c(n) (|S|^2 - N), and the cross form 2 c(n) Re(S_a S_b*)
__global__ void k_df_energy(int N, const float4 *__restrict__ Sa, const double *__restrict__ coef, int nk,
                            double *part) {
  __shared__ double buf[8];
  const int j = blockIdx.x;
  double e = 0;
  for (int k = threadIdx.x; k < nk; k += blockDim.x) {
    const double ck = coef[k];
    if (__double_as_longlong(ck) == 0) continue;  // a dropped vector
    const float4 s = Sa[(size_t)j * nk + k];
    const double re = (double)s.x + s.z, im = (double)s.y + s.w;
    e += ck * (re * re + im * im - N);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) e += __shfl_down_sync(ALL, e, o);
  if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)blockDim.x / 32; ++w) e += buf[w];
    part[j] = e;
  }
}

#define DF_NS(nsv, ...)                                  \
  switch (nsv) {                                         \
    case 1: { constexpr int NS = 1; __VA_ARGS__; } break;   \
    case 2: { constexpr int NS = 2; __VA_ARGS__; } break;   \
    case 3: { constexpr int NS = 3; __VA_ARGS__; } break;   \
    case 4: { constexpr int NS = 4; __VA_ARGS__; } break;   \
    case 5: { constexpr int NS = 5; __VA_ARGS__; } break;   \
    case 6: { constexpr int NS = 6; __VA_ARGS__; } break;   \
    case 7: { constexpr int NS = 7; __VA_ARGS__; } break;   \
    case 8: { constexpr int NS = 8; __VA_ARGS__; } break;   \
    case 9: { constexpr int NS = 9; __VA_ARGS__; } break;   \
    case 10: { constexpr int NS = 10; __VA_ARGS__; } break; \
    case 11: { constexpr int NS = 11; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;               \
  }

static const int *df_base(const Recip &r) { return r.kvec + recip_df_off(r.nsum); }
static const int4 *df_cols(const Recip &r) { return (const int4 *)df_base(r); }
static const int *df_toff(const Recip &r) { return df_base(r) + toff_at(r.nsum); }

template <int NS>
constexpr size_t sk_smem() {
  return sizeof(float4) * 3 * (NS + 1) * (DF_CH + 1);
}

cudaError_t recip_df_sk(const Geo &g, const Recip &r, const double *x, cudaStream_t st) {
  {
    XK_PROF("phase");
    k_df_phase<<<cdivz((size_t)g.P * 3 * g.Ns, 128), 128, 0, st>>>(g, r.nsum, x, (float4 *)r.phase);
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess || r.items <= 0) return e;
  XK_PROF("sk");
  const dim3 grid(cdivz(r.items, DF_SK_T / DF_GR), g.P);
  DF_NS(r.nsum, {
    static bool opted = false;
    if (!opted) {
      e = cudaFuncSetAttribute(k_df_sk<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sk_smem<NS>());
      if (e != cudaSuccess) return e;
      opted = true;
    }
    k_df_sk<NS><<<grid, DF_SK_T, sk_smem<NS>(), st>>>(g.N, g.Ns, (const float4 *)r.phase, df_cols(r),
                                                     df_base(r) + items_at(r.nsum), r.df_items, r.items, (float4 *)r.S,
                                                     r.nk);
  });
  return XK_LAUNCHED();
}

cudaError_t recip_df_tables_of(const Geo &g, const Recip &r, cudaStream_t st) {
  if (r.items <= 0) return cudaSuccess;
  XK_PROF("recip_tables");
  const dim3 grid((r.ncol + 7) / 8, g.P), blk(r.nsum + 1, 8);
  DF_NS(r.nsum, (k_df_tables<NS><<<grid, blk, 0, st>>>(df_cols(r), df_toff(r), r.ncol, (const float4 *)r.S, r.coef,
                                                       r.nk, r.tdf, (float4 *)r.T)));
  return XK_LAUNCHED();
}

template <int NS, int TPP>
static cudaError_t launch_force(const Geo &g, const Recip &r, const double *T, double scale, double *f,
                                cudaStream_t st) {
  static bool opted = false;
  if (!opted) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_df_force<NS, TPP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    opted = true;
  }
  constexpr int PPB = DF_RF_T / TPP;
  const size_t smem = sizeof(float4) * (r.tdf + 2 * (NS + 1) * PPB) + (sizeof(int4) + sizeof(int)) * r.ncol;
  k_df_force<NS, TPP><<<dim3((g.N + PPB - 1) / PPB, g.P), DF_RF_T, smem, st>>>(
      g, (const float4 *)r.phase, df_cols(r), df_toff(r), r.ncol, (const float4 *)T, r.tdf, scale, f);
  return XK_LAUNCHED();
}

// forces on g's particles (phases of r) from the tables T
cudaError_t recip_df_force_from(const Geo &g, const Recip &r, const double *T, double scale, double *f,
                                cudaStream_t st) {
  if (r.items <= 0) return cudaSuccess;
  XK_PROF("recip_force");
  // threads a particle: 4 once that fills the SMs with 16 warps each, else 16
  const bool big = (size_t)g.N * g.P * 4 >= (size_t)152 * 512;
  DF_NS(r.nsum, {
    return big ? launch_force<NS, 4>(g, r, T, scale, f, st) : launch_force<NS, 16>(g, r, T, scale, f, st);
  });
  return cudaSuccess;
}

cudaError_t recip_df_energy(const Geo &g, const Recip &r, double *part, cudaStream_t st) {
  XK_PROF("recip_energy");
  k_df_energy<<<g.P, 256, 0, st>>>(g.N, (const float4 *)r.S, r.coef, r.nk, part);
  return XK_LAUNCHED();
}

}  // namespace xk
