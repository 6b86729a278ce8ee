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

constexpr int DF_NG = 8;  // harmonics of one structure-factor item

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
// of a slice, particles interleaved; phases staged DF_CH particles at a time,
// the next chunk copied asynchronously while one is summed.  With
// P = sum e_xy cos(nz theta_z), Q = sum e_xy sin(nz theta_z):
// S(+nz) = P + iQ, S(-nz) = P - iQ.  FP32 harmonics add their products in
// FP32, 8 particles at a time, into the accumulator's low part, which then
// joins the high part exactly.
// Bound: FP32 issue of the double-float harmonics (48 instructions a
// particle and pair, 60 for e_xy).  Eight harmonics an item and not four:
// inside the sphere a column has at most seven, so e_xy is formed once a
// column, and no group is padded (142 -> 83 us at 512 x 64 with the
// asynchronous copies).  Blocks of the double-float items, the longest, start
// first.  Two blocks of 256 threads an SM and not one of 512, which left a
// third of the chip idle in the last round: 512 x 33, |n| <= 10, 82 -> 63 us;
// 700 x 20, |n| <= 9, 109 -> 80; 512 x 64 83 -> 82.
constexpr int DF_CH = 64, DF_SK_T = 256;

__device__ __forceinline__ void copy16(float4 *dst, const float4 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int NS, int GR>
__global__ void __launch_bounds__(DF_SK_T, 2)
    k_df_sk(int N, int Ns, const float4 *__restrict__ ph, const int4 *__restrict__ cols, const int *__restrict__ items,
            int ndf, int nitems, float4 *__restrict__ S, int nk) {
  constexpr int LD = DF_CH + 1, STAGE = 3 * (NS + 1) * LD, NG = NS < DF_NG ? NS : DF_NG;
  extern __shared__ __align__(16) float4 df_sp[];  // two stages of [3][NS + 1][LD]
  const int j = blockIdx.x, gq = threadIdx.x % GR;
  const int it = blockIdx.y * (DF_SK_T / GR) + threadIdx.x / GR;
  const bool live = it < nitems;
  const int item = live ? items[it] : 0;
  const int4 c = cols[item & 0xffff];
  const int n0 = (item >> 16) * DF_NG;
  const int top = live ? min(dc_nz(c) - n0, NG) : 0;           // harmonics of this item
  const int nd = live && it < ndf ? max(dc_nzs(c) - n0, 0) : -1;  // of those, double-float (-1: e_xy in FP32 too)
  const int ox = dc_nx(c) * LD, oy = (NS + 1 + abs(c.y)) * LD, oz = (2 * (NS + 1) + n0 + 1) * LD;
  const float sy = c.y < 0 ? -1.f : 1.f;
  df s0r = {0.f, 0.f}, s0i = {0.f, 0.f}, Pr[NG], Pi[NG], Qr[NG], Qi[NG];
#pragma unroll
  for (int u = 0; u < NG; ++u) Pr[u] = Pi[u] = Qr[u] = Qi[u] = {0.f, 0.f};
  const float4 *base = ph + (size_t)j * 3 * (NS + 1) * Ns;
  const int chunks = (N + DF_CH - 1) / DF_CH;
  auto stage = [&](int k) {
    float4 *to = df_sp + (k & 1) * STAGE;
    const int l0 = k * DF_CH, cnt = min(N - l0, DF_CH);
    for (int q = threadIdx.x; q < 3 * (NS + 1) * DF_CH; q += DF_SK_T) {
      const int l = q % DF_CH, row = q / DF_CH;
      if (l < cnt) copy16(to + row * LD + l, base + (size_t)row * Ns + l0 + l);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0);
  for (int k = 0; k < chunks; ++k) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // chunk k is there, and nobody reads the other stage any more
    if (k + 1 < chunks) stage(k + 1);
    if (!live) continue;
    const float4 *sp = df_sp + (k & 1) * STAGE;
    const int cnt = min(N - k * DF_CH, DF_CH);
    if (nd >= 0) {
      for (int l = gq; l < cnt; l += GR) {
        const dfc ex = unpack(sp[ox + l]);
        dfc ey = unpack(sp[oy + l]);
        ey.i.h *= sy, ey.i.l *= sy;
        const dfc e = mul(ex, ey);
        s0r = df_add(s0r, e.r);
        s0i = df_add(s0i, e.i);
#pragma unroll
        for (int u = 0; u < NG; ++u) {
          if (u >= top) break;
          const float4 v = sp[oz + u * LD + l];
          if (u < nd) {
            const dfc ez = unpack(v);
            fma_to(Pr[u], e.r, ez.r);
            fma_to(Pi[u], e.i, ez.r);
            fma_to(Qr[u], e.r, ez.i);
            fma_to(Qi[u], e.i, ez.i);
          } else {
            Pr[u].l = fmaf(e.r.h, v.x, Pr[u].l);
            Pi[u].l = fmaf(e.i.h, v.x, Pi[u].l);
            Qr[u].l = fmaf(e.r.h, v.y, Qr[u].l);
            Qi[u].l = fmaf(e.i.h, v.y, Qi[u].l);
          }
        }
      }
    } else {
      for (int l = gq; l < cnt; l += GR) {
        const float4 ex = sp[ox + l], ey = sp[oy + l];
        const float yi = sy * ey.y;
        const float er = fmaf(ex.x, ey.x, -ex.y * yi), ei = fmaf(ex.x, yi, ex.y * ey.x);
        s0r.l += er;
        s0i.l += ei;
#pragma unroll
        for (int u = 0; u < NG; ++u) {
          if (u >= top) break;
          const float4 v = sp[oz + u * LD + l];
          Pr[u].l = fmaf(er, v.x, Pr[u].l);
          Pi[u].l = fmaf(ei, v.x, Pi[u].l);
          Qr[u].l = fmaf(er, v.y, Qr[u].l);
          Qi[u].l = fmaf(ei, v.y, Qi[u].l);
        }
      }
      s0r = two_sum(s0r.h, s0r.l);
      s0i = two_sum(s0i.h, s0i.l);
    }
#pragma unroll
    for (int u = 0; u < NG; ++u) {
      if (u >= top) break;
      if (u < nd) continue;
      Pr[u] = two_sum(Pr[u].h, Pr[u].l);
      Pi[u] = two_sum(Pi[u].h, Pi[u].l);
      Qr[u] = two_sum(Qr[u].h, Qr[u].l);
      Qi[u] = two_sum(Qi[u].h, Qi[u].l);
    }
  }
#pragma unroll
  for (int o = 1; o < GR; o <<= 1) {
    s0r = df_add(s0r, shfl_xor(ALL, s0r, o));
    s0i = df_add(s0i, shfl_xor(ALL, s0i, o));
#pragma unroll
    for (int u = 0; u < NG; ++u) {
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
  for (int u = 0; u < NG; ++u) {
    if (u >= top) break;
    const int n = n0 + u + 1;
    o[n] = pack(df_sub(Pr[u], Qi[u]), df_add(Pi[u], Qr[u]));
    if (c.z < 0) o[-n] = pack(df_add(Pr[u], Qi[u]), df_sub(Pi[u], Qr[u]));
  }
}

// Force tables of a slice, compact: per column W(0), then A, B, n A, n B (as
// in k_recip_tables) per double-float harmonic, then (A, B) in FP32 per
// remaining one.  coef: c(n) as FP32 pairs.
template <int NS>
__global__ void __launch_bounds__(8 * (NS + 1))
    k_df_tables(const int4 *__restrict__ cols, const int *__restrict__ toff, int ncol, const float4 *__restrict__ S,
                const float2 *__restrict__ coef, int nk, int tdf, float4 *__restrict__ T) {
  const int j = blockIdx.y, ci = blockIdx.x * blockDim.y + threadIdx.y, n = threadIdx.x;
  if (ci >= ncol) return;
  const int4 c = cols[ci];
  if (n > dc_nz(c)) return;
  auto W = [&](int nz) -> dfc {  // c(n) conj(S(n))
    if (nz < c.z) return {{0.f, 0.f}, {0.f, 0.f}};
    const int k = c.w + (nz - c.z);
    const float2 ck = coef[k];
    const dfc s = unpack(S[(size_t)j * nk + k]);
    return {df_mul({ck.x, ck.y}, s.r), df_mul({-ck.x, -ck.y}, s.i)};
  };
  float4 *o = T + (size_t)j * tdf + toff[ci];
  const int nzs = max(dc_nzs(c), 0);
  if (n == 0) {
    const dfc w = W(0);
    o[0] = pack(w.r, w.i);
    return;
  }
  const dfc wp = W(n), wm = W(-n);
  const df Ar = df_add(wp.r, wm.r), Ai = df_add(wp.i, wm.i), Br = df_sub(wp.r, wm.r), Bi = df_sub(wp.i, wm.i);
  if (n <= nzs) {
    const float m = (float)n;
    o[4 * n - 3] = pack(Ar, Ai);
    o[4 * n - 2] = pack(Br, Bi);
    o[4 * n - 1] = pack(times(m, Ar), times(m, Ai));
    o[4 * n] = pack(times(m, Br), times(m, Bi));
  } else {
    o[4 * nzs + (n - nzs)] = make_float4(Ar.h + Ar.l, Ai.h + Ai.l, Br.h + Br.l, Bi.h + Bi.l);
  }
}

// Forces: a block of W warps has 32 particles of a slice, one a lane; warp w
// takes columns w, w + W, ..., so that its lanes run alike and read each
// table entry at one address, and the warps' sums meet in shared memory
// (4 or 16 lanes a particle, each on its own column, waited for their
// scattered table reads: 126 -> 98 us at 512 x 64, 29 -> 18 us at 128 x 32).
// Tables, columns and the particles' x and y phase factors are staged, the z
// factors in registers.  Per column, with U = sum_nz e_z W and
// V = sum_nz nz e_z W: F_x, F_y from Im(e_xy U), F_z from Im(e_xy V).
// Bound: FP32 issue (eight double-float multiply-adds a harmonic, 96
// instructions).
template <int NS, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
    k_df_force(Geo g, const float4 *__restrict__ ph, const int4 *__restrict__ cols, const int *__restrict__ toff,
               int ncol, const float4 *__restrict__ T, int tdf, double scale, double *__restrict__ f) {
  extern __shared__ __align__(16) float4 df_sm[];
  float4 *sT = df_sm, *pxy = df_sm + tdf;        // [tdf], [2 (NS + 1)][32]
  int4 *sc = (int4 *)(pxy + 2 * (NS + 1) * 32);  // [ncol]
  int *so = (int *)(sc + ncol);                  // [ncol]
  const int j = blockIdx.y, l0 = blockIdx.x * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float4 *Tj = T + (size_t)j * tdf, *pj = ph + (size_t)j * 3 * (NS + 1) * g.Ns;
  const int l = min(l0 + lane, g.N - 1);  // (lanes past the end repeat the last particle)
  for (int q = threadIdx.x; q < tdf; q += 32 * NW) copy16(sT + q, Tj + q);
  for (int r = w; r < 2 * (NS + 1); r += NW) copy16(pxy + r * 32 + lane, pj + (size_t)r * g.Ns + l);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int q = threadIdx.x; q < ncol; q += 32 * NW) sc[q] = cols[q], so[q] = toff[q];
  dfc ez[NS];
#pragma unroll
  for (int n = 1; n <= NS; ++n) ez[n - 1] = unpack(pj[((size_t)2 * (NS + 1) + n) * g.Ns + l]);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  df F[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) F[d] = {0.f, 0.f};
  for (int ci = w; ci < ncol; ci += NW) {
    const int4 c = sc[ci];
    const int nzs = dc_nzs(c), nzc = dc_nz(c);
    const float4 *t = sT + so[ci];
    const float4 vx = pxy[dc_nx(c) * 32 + lane];
    float4 vy = pxy[(NS + 1 + abs(c.y)) * 32 + lane];
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
  // the warps' sums, in order (the tables are no longer read)
  __syncthreads();
  float2 *sum = (float2 *)df_sm;  // [NW][3][32]
#pragma unroll
  for (int d = 0; d < 3; ++d) sum[(w * 3 + d) * 32 + lane] = make_float2(F[d].h, F[d].l);
  __syncthreads();
  if (w >= 3 || l0 + lane >= g.N) return;
  df t = {0.f, 0.f};
  for (int v = 0; v < NW; ++v) {
    const float2 p = sum[(v * 3 + w) * 32 + lane];
    t = df_add(t, {p.x, p.y});
  }
  const double ib = w == 0 ? g.inv_box[0] : (w == 1 ? g.inv_box[1] : g.inv_box[2]);
  f[sidx(j, w, l, 3, g.Ns)] += scale * df_value(t) * ib;
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
  return 2 * sizeof(float4) * 3 * (NS + 1) * (DF_CH + 1);
}

template <int NS, int GR>
static cudaError_t launch_sk(const Geo &g, const Recip &r, cudaStream_t st) {
  static bool opted = false;
  if (!opted) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_df_sk<NS, GR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sk_smem<NS>());
    if (e != cudaSuccess) return e;
    opted = true;
  }
  const dim3 grid(g.P, cdivz(r.items, DF_SK_T / GR));
  k_df_sk<NS, GR><<<grid, DF_SK_T, sk_smem<NS>(), st>>>(g.N, g.Ns, (const float4 *)r.phase, df_cols(r),
                                                       df_base(r) + items_at(r.nsum), r.df_items, r.items,
                                                       (float4 *)r.S, r.nk);
  return XK_LAUNCHED();
}

cudaError_t recip_df_sk(const Geo &g, const Recip &r, const double *x, cudaStream_t st) {
  {
    XK_PROF("phase");
    k_df_phase<<<cdivz((size_t)g.P * 3 * g.Ns, 128), 128, 0, st>>>(g, r.nsum, x, (float4 *)r.phase);
  }
  cudaError_t e = XK_LAUNCHED();
  if (e != cudaSuccess || r.items <= 0) return e;
  XK_PROF("sk");
  // 16 threads an item where 8 would give four SMs seven blocks at most (152
  // SMs by number: the threads set the order of the sums):
  // 700 x 20, |n| <= 9, 80 -> 53 us; 512 x 33, |n| <= 10 (264 blocks), 63 -> 55;
  // 128 x 32, |n| <= 8 (160), 22.0 -> 20.7; 200 x 48, |n| <= 9 (288), keeps 38 (43)
  const bool few = (size_t)g.P * cdivz(r.items, DF_SK_T / 8) * 4 <= 7 * 152;
  DF_NS(r.nsum, { return few ? launch_sk<NS, 16>(g, r, st) : launch_sk<NS, 8>(g, r, st); });
  return cudaSuccess;
}

cudaError_t recip_df_tables_of(const Geo &g, const Recip &r, cudaStream_t st) {
  if (r.items <= 0) return cudaSuccess;
  XK_PROF("recip_tables");
  const dim3 grid((r.ncol + 7) / 8, g.P), blk(r.nsum + 1, 8);
  DF_NS(r.nsum, (k_df_tables<NS><<<grid, blk, 0, st>>>(df_cols(r), df_toff(r), r.ncol, (const float4 *)r.S,
                                                       recip_coef_pairs(r), r.nk, r.tdf, (float4 *)r.T)));
  return XK_LAUNCHED();
}

template <int NS, int NW>
static cudaError_t launch_force(const Geo &g, const Recip &r, const double *T, double scale, double *f,
                                cudaStream_t st) {
  static bool opted = false;
  if (!opted) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_df_force<NS, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    opted = true;
  }
  size_t smem = sizeof(float4) * (r.tdf + 2 * (NS + 1) * 32) + (sizeof(int4) + sizeof(int)) * r.ncol;
  smem = std::max(smem, sizeof(float2) * 3 * 32 * NW);
  k_df_force<NS, NW><<<dim3((g.N + 31) / 32, g.P), 32 * NW, smem, st>>>(
      g, (const float4 *)r.phase, df_cols(r), df_toff(r), r.ncol, (const float4 *)T, r.tdf, scale, f);
  return XK_LAUNCHED();
}

// forces on g's particles (phases of r) from the tables T
cudaError_t recip_df_force_from(const Geo &g, const Recip &r, const double *T, double scale, double *f,
                                cudaStream_t st) {
  if (r.items <= 0) return cudaSuccess;
  XK_PROF("recip_force");
  // 16 warps a block when blocks of 8 would not give every SM two
  const bool few = (size_t)((g.N + 31) / 32) * g.P < 2 * 152;
  DF_NS(r.nsum, {
    return few ? launch_force<NS, 16>(g, r, T, scale, f, st) : launch_force<NS, 8>(g, r, T, scale, f, st);
  });
  return cudaSuccess;
}

cudaError_t recip_df_energy(const Geo &g, const Recip &r, double *part, cudaStream_t st) {
  XK_PROF("recip_energy");
  k_df_energy<<<g.P, 256, 0, st>>>(g.N, (const float4 *)r.S, r.coef, r.nk, part);
  return XK_LAUNCHED();
}

}  // namespace xk
