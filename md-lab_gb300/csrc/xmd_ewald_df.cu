// xmd_ewald_df.cu -- the FP64 form's Ewald sums in double-float arithmetic
// (xmd_df.cuh): FP32 pairs with about 48 significant bits on the FP32 pipe.
//
// The FP64 pipe holds a warp's instruction for 64 cycles on GB300, and the
// FP64 sums' results carry an error of about 1e-12 of a bead's force anyway
// (the cut-off); double-float rounding, about 1e-14, is far below that.  The
// strict form (every term FP64) and geometries these kernels do not take stay
// on the kernels of xmd_kernels.cu.
#include <cfloat>
#include <cmath>

#include "xmd_df.cuh"
#include "xmd_ewald_df_tables.h"
#include "xmd_ewald_tables.h"
#include "xmd_kernels.cuh"

namespace xk {

constexpr unsigned ALL = 0xffffffffu;
static inline int cdivz(size_t a, int b) { return (int)((a + b - 1) / b); }

__device__ __align__(16) const float g_ewd_h[EWD_H_NINT * 8] = EWD_H_INIT;
__device__ __align__(16) const float g_ewd_erfc[EWD_ERFC_NINT * 8] = EWD_ERFC_INIT;

// ===================================================================
// Real space.  Coordinates are scaled by alpha, wrapped into the box and
// kept as three FP32 limbs on fixed grids (x = h + m + l, h a multiple of
// G1 = 2^(e-23) with alpha L < 2^e, m of G2 = G1 2^-23, l with the scaling's
// own rounding error): differences of h and m, and their shift by the box
// edge, are exact, so a separation is good to 2^-48 of itself however close
// the two beads are.
// ===================================================================
struct EwdPrm {
  double box[3], inv_box[3], alpha;
  double magic1, magic2;     // 1.5 2^52 G1, 1.5 2^52 G2: adding and subtracting rounds to the grid
  float Lh[3], Lm[3], Ll[3]; // alpha L on the same grids
  float iL[3];               // 1 / (alpha L)
  float Ph[3], Pl[3];        // alpha L, its double and its square as pairs
  float Th[3], Tl[3], Sh[3], Sl[3];
  float rc2;                 // (alpha rcut)^2
  float nsum;
  int cube;                  // the reference's image cube always holds the candidates of wrapped beads (nsum >= 2)
};

static double grid_round(double v, double magic) {
  volatile double t = v + magic;
  return t - magic;
}

static EwdPrm make_ewd(const Geo &g, const PairPrm &p) {
  EwdPrm q{};
  double top = 0;
  for (int d = 0; d < 3; ++d) top = fmax(top, p.alpha * g.box[d]);
  int e = 0;
  frexp(top, &e);  // top < 2^e
  q.magic1 = ldexp(1.5, 52 + e - 23);
  q.magic2 = ldexp(1.5, 52 + e - 46);
  q.alpha = p.alpha;
  for (int d = 0; d < 3; ++d) {
    const double L = p.alpha * g.box[d];
    q.box[d] = g.box[d];
    q.inv_box[d] = g.inv_box[d];
    const double h = grid_round(L, q.magic1), m = grid_round(L - h, q.magic2);
    q.Lh[d] = (float)h;
    q.Lm[d] = (float)m;
    q.Ll[d] = (float)(L - h - m + fma(p.alpha, g.box[d], -L));
    q.iL[d] = (float)(1.0 / L);
    const df P = df_split(L), S = df_split(L * L);
    q.Ph[d] = P.h, q.Pl[d] = P.l;
    q.Th[d] = 2 * P.h, q.Tl[d] = 2 * P.l;
    q.Sh[d] = S.h;
    q.Sl[d] = (float)fma(L, L, -(double)S.h);
  }
  q.rc2 = (float)(p.alpha * p.alpha * p.rcut * p.rcut);
  q.nsum = (float)p.nsum;
  q.cube = p.nsum >= 2;
  return q;
}

// Forces: with rcut at most every box edge, only the 8 images with k_d in
// {0, sign(m_d)} around the minimum image m lie inside the cut-off (any
// other has a component of length >= L).  Energies keep a longer cut-off,
// 5.8 / alpha, and take the few images beyond (one component of length
// L + |m_d|, erfc below 1e-14) in FP32 when rcut is at most 1.05 L.
// alpha L above 64 would leave the grids too coarse; it is also far outside
// what a converged reciprocal sum with n_sum <= 11 can use.
bool ewd_applies(const Geo &g, const PairPrm &p, bool energy) {
  if (g.D != 3 || p.kind != PAIR_EWALD_REAL || !(p.alpha > 0) || !(p.xsplit > 0)) return false;
  double lo = g.box[0], hi = g.box[0];
  for (int d = 1; d < 3; ++d) lo = fmin(lo, g.box[d]), hi = fmax(hi, g.box[d]);
  const int nint = energy ? EWD_ERFC_NINT : EWD_H_NINT;
  return lo > 0 && p.rcut <= lo * (energy ? 1.05 : 1.0) && p.alpha * hi < 64.0 &&
         p.alpha * p.rcut * EWD_INV_W < nint - 2;
}

size_t ewd_pos_doubles(const Geo &g) { return (size_t)6 * g.P * g.Ns; }  // three float4 a bead

// pos[(k*P + j)*Ns + l], k = 0..2: (h0, h1, h2, m0), (m1, m2, l0, l1), (l2, n0, n1, n2) with n the box shift that
// wrapped the bead
__global__ void __launch_bounds__(128) k_ewd_split(EwdPrm q, int N, int Ns, int P, const double *__restrict__ x,
                                                   float4 *__restrict__ pos) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P * Ns) return;
  const int j = t / Ns, l = t % Ns;
  float h[3], m[3], lo[3], n[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double v = l < N ? x[((size_t)j * 3 + d) * Ns + l] : 0.0;
    const double s = floor(v * q.inv_box[d]);
    const double xw = fma(-s, q.box[d], v), y = q.alpha * xw, yl = fma(q.alpha, xw, -y);
    const double hd = __dadd_rn(__dadd_rn(y, q.magic1), -q.magic1);
    const double r = y - hd;
    const double md = __dadd_rn(__dadd_rn(r, q.magic2), -q.magic2);
    h[d] = (float)hd, m[d] = (float)md, lo[d] = (float)(r - md + yl), n[d] = (float)s;
  }
  const size_t S = (size_t)P * Ns;
  pos[t] = make_float4(h[0], h[1], h[2], m[0]);
  pos[S + t] = make_float4(m[1], m[2], lo[0], lo[1]);
  pos[2 * S + t] = make_float4(lo[2], n[0], n[1], n[2]);
}

// R^2 = (x)^2 in, h(x)/x^3 (forces) or erfc(x)/x (energies) out, x = alpha R.
// x = sqrt(R^2) and 1/x from an FP32 reciprocal square root, each refined once
// and corrected by its residual; h or erfc from the interval's row.
template <bool ENERGY>
__device__ __forceinline__ df ewd_image(df R, const float4 *__restrict__ tab) {
  float y = rsqrtf(R.h);
  y = __fmaf_rn(__fmul_rn(0.5f, y), __fmaf_rn(-__fmul_rn(R.h, y), y, 1.f), y);
  // a = 1 - R^2 y^2, about 1e-7
  const df yy = two_prod(y, y);
  const float a = __fmaf_rn(-R.l, yy.h, __fmaf_rn(-R.h, yy.l, __fmaf_rn(-R.h, yy.h, 1.f)));
  const float hy = 0.5f * y;
  float g = __fmul_rn(R.h, y);
  g = __fmaf_rn(__fadd_rn(__fmaf_rn(-g, g, R.h), R.l), hy, g);  // x to half an ulp
  const float t = __fmul_rn(__fadd_rn(__fmaf_rn(-g, g, R.h), R.l), hy);
  const float gl = __fmaf_rn(t, __fmaf_rn(hy, t, 0.5f * a), t);  // x = g + gl, 1/x = y (1 + a/2 + ...)
  const float tq = __fmaf_rn(g, EWD_INV_W, 12582912.f);  // 1.5 2^23: the interval in the low bits
  const int iv = min(__float_as_int(tq) & 0x7ff, (ENERGY ? EWD_ERFC_NINT : EWD_H_NINT) - 1);
  const float fi = __fsub_rn(tq, 12582912.f);
  const float uh = __fmaf_rn(g, 2 * EWD_INV_W, -2.f * fi), ul = 2 * EWD_INV_W * gl;
  const float4 ca = tab[2 * iv], cb = tab[2 * iv + 1];
  // Horner in pairs: c2 + u (c3 + c4 u), then c1 + u (.), then c0 + u (.)
  const float s3 = __fmaf_rn(uh, cb.w, cb.z);
  const float s2 = __fmaf_rn(ul, s3, __fmaf_rn(uh, s3, cb.y));
  df p = two_prod(uh, cb.x);
  float e = __fmaf_rn(ul, __fadd_rn(cb.x, s2), __fmaf_rn(uh, s2, p.l));
  df r = two_sum(ca.z, p.h);
  r.l = __fadd_rn(r.l, __fadd_rn(ca.w, e));
  p = two_prod(uh, r.h);
  e = __fmaf_rn(ul, __fadd_rn(r.h, r.l), __fmaf_rn(uh, r.l, p.l));
  df w = fast_two_sum(ca.x, p.h);
  w.l = __fadd_rn(w.l, __fadd_rn(ca.y, e));
  if constexpr (ENERGY) {
    // 1/x = y (1 - a)^(-1/2) = y + y (a/2 + 3 a^2/8)
    const float c = __fmul_rn(y, __fmul_rn(a, __fmaf_rn(0.375f, a, 0.5f)));
    return df_mul(w, {y, c});
  }
  // 1/x^3 = y^3 (1 - a)^(-3/2) = y^3 + y^3 (3 a/2 + 15 a^2/8)
  df y3 = two_prod(yy.h, y);
  y3.l = __fmaf_rn(yy.l, y, y3.l);
  y3.l = __fmaf_rn(y3.h, __fmul_rn(a, __fmaf_rn(1.875f, a, 1.5f)), y3.l);
  return df_mul(w, y3);
}

// erfc(x)/x in FP32 for the energies' images beyond L (a few 1e-15)
__device__ __forceinline__ float ewd_erfc32(float R2) {
  const float cc[EW32_DEG + 1] = EW32_ERFCX_INIT;
  const float ri = rsqrtf(R2), x = R2 * ri, t = __fdividef(1.f, fmaf((float)EW32_C, x, 1.f));
  float v = cc[EW32_DEG];
#pragma unroll
  for (int k = EW32_DEG - 1; k >= 0; --k) v = fmaf(v, t, cc[k]);
  return __expf(-R2) * v * t * ri;
}

struct EwdSide {
  const float4 *pos;
  int N, Ns;
};

constexpr int EWD_WARPS = 8;
struct EwdWarp {
  float4 b[3][32];  // the tile's partners
  float2 q[256];    // accepted images of one rotation step: R^2, then the factor
};
template <bool ENERGY>
constexpr size_t ewd_smem() {
  return sizeof(float4) * 2 * (ENERGY ? EWD_ERFC_NINT : EWD_H_NINT) + sizeof(EwdWarp) * EWD_WARPS;
}

// One warp per 32 x 32 tile of a slice, as in k_pair_tiles, or per part of its
// steps (ewd_split): a's beads in the lanes, b's rotating by, accumulated with
// Newton's third law, partials into slots summed by k_ewd_finish (no
// atomics).  Tiles on the diagonal visit each pair once (16 steps) and come
// last.
//
// Per step the lane's pair gives the squared lengths of its 8 candidates in
// pairs: |m|^2 plus A_d = L_d^2 - 2 L_d |m_d| per shifted axis.  Those inside
// the cut-off go to the warp's queue (ballots give each its place), so that
// the factor is evaluated with full warps whatever the lanes' counts; the
// owner then forms
//   F_d = sign(m_d) (|m_d| V - L_d V_d),   V = sum of all factors, V_d of
// those shifted along d.  Factors fall with distance, so the sums add the
// smaller to the larger (three-operation exact additions).
//
// Bound: FP32 issue, about 650 operations a pair and step.  Measured on the
// 512-electron, 64-bead gas (alpha L = 5.6, 3.35 images a pair, 8.4 M pairs):
// 257 us where the FP64 tiles took 1352 (256 x 256 cross pairs 145 and 667
// us); in parts 128 electrons, 32 beads take 24 us (51 with whole tiles, 218 in
// FP64) and their energies 24 (61 and 325).  The forces' error against 64-bit
// sums, set by the cut-off at alpha R = 5.2, is 3.6e-13 of the forces' norm
// (4.1e-13 with the FP64 tiles and their FP32 far images), 12 to 512 electrons
// alike.  Energies take three limbs: in two, images below the sum's last bit were lost and biased it by
// -5e-16 of the pair energies; now 0.6e-15 (128 electrons, 32 beads, rms of 16
// states) and 0.5e-15 (512, 64) of the energy against 64 bits, 1.3e-15 and
// 2.6e-15 with the FP64 tiles, for 3% more time.
template <bool CROSS, bool ENERGY>
__global__ void __launch_bounds__(32 * EWD_WARPS, 2)
    k_ewd_tiles(EwdPrm q, int P, EwdSide A, EwdSide B, float2 *__restrict__ outa, float2 *__restrict__ outb,
                double *__restrict__ eout, int TA, int TB, int split) {
  extern __shared__ __align__(16) float4 ewd_sm[];
  constexpr int NROW = 2 * (ENERGY ? EWD_ERFC_NINT : EWD_H_NINT);
  float4 *tab = ewd_sm;
  {
    const float4 *src = (const float4 *)(ENERGY ? g_ewd_erfc : g_ewd_h);
    for (int i = threadIdx.x; i < NROW; i += blockDim.x) tab[i] = src[i];
  }
  EwdWarp *ws = (EwdWarp *)(ewd_sm + NROW) + (threadIdx.x >> 5);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int nwarps = gridDim.x * EWD_WARPS;
  const int full = CROSS ? TA * TB : TA * (TA - 1) / 2;
  const int njobs = (full + (CROSS ? 0 : TA)) * P * split;
  for (int u = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; u < njobs; u += nwarps) {
    const int w = u / split, part = u % split;
    int j, I, J;
    const bool diag = !CROSS && w >= full * P;
    if (CROSS) {
      j = w / full;
      const int r = w % full;
      I = r / TB, J = r % TB;
    } else if (diag) {
      j = (w - full * P) / TA;
      I = J = (w - full * P) % TA;
    } else {
      j = w / full;
      int r = w % full;
      I = 0;
      while (r >= TA - 1 - I) {
        r -= TA - 1 - I;
        ++I;
      }
      J = I + 1 + r;
    }
    const int a = I * 32 + lane, b0 = J * 32 + lane;
    const bool va = a < A.N, vb = b0 < B.N;
    const size_t SA = (size_t)P * A.Ns, SB = (size_t)P * B.Ns;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 *pa = A.pos + (size_t)j * A.Ns + a, *pb = B.pos + (size_t)j * B.Ns + b0;
    const float4 a0 = va ? pa[0] : z4, a1 = va ? pa[SA] : z4, a2 = va ? pa[2 * SA] : z4;
    const float4 t0 = vb ? pb[0] : z4, t1 = vb ? pb[SB] : z4, t2 = vb ? pb[2 * SB] : z4;
    __syncwarp();  // the previous job's reads are done
    ws->b[0][lane] = t0;
    ws->b[1][lane] = t1;
    ws->b[2][lane] = t2;
    const bool wrapped =
        a2.y != 0.f || a2.z != 0.f || a2.w != 0.f || t2.y != 0.f || t2.z != 0.f || t2.w != 0.f;
    const bool test_cube = !q.cube || __any_sync(ALL, wrapped);
    __syncwarp();
    df fa[3], fb[3], en = {0.f, 0.f};
    float enc = 0.f;  // third limb of the energy: far images are smaller than the pair's last bit
#pragma unroll
    for (int d = 0; d < 3; ++d) fa[d] = fb[d] = {0.f, 0.f};
    const int steps = (diag ? 16 : 32) / split;
    const int s0 = (diag ? 1 : 0) + part * steps, s1 = s0 + steps - 1;
    for (int s = s0; s <= s1; ++s) {
      const int bl = (lane + s) & 31;
      const bool act = va && J * 32 + bl < B.N && !(diag && s == 16 && lane >= 16);
      const float4 b0v = ws->b[0][bl], b1v = ws->b[1][bl], b2v = ws->b[2][bl];
      const float dh[3] = {a0.x - b0v.x, a0.y - b0v.y, a0.z - b0v.z};
      const float dm[3] = {a0.w - b0v.w, a1.x - b1v.x, a1.y - b1v.y};
      const float dl[3] = {a1.z - b1v.z, a1.w - b1v.w, a2.x - b2v.x};
      df m[3];          // |minimum image|
      float sg[3], sh[3];
      df R0 = {0.f, 0.f}, Ad[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        sh[d] = rintf(dh[d] * q.iL[d]);
        const float h = __fmaf_rn(-sh[d], q.Lh[d], dh[d]), mm = __fmaf_rn(-sh[d], q.Lm[d], dm[d]);
        m[d] = fast_two_sum(h, mm);
        m[d].l = __fadd_rn(m[d].l, __fmaf_rn(-sh[d], q.Ll[d], dl[d]));
        sg[d] = m[d].h < 0.f ? -1.f : 1.f;
        m[d].h = fabsf(m[d].h);
        m[d].l *= sg[d];
        df sq = two_prod(m[d].h, m[d].h);
        sq.l = __fmaf_rn(2.f * m[d].h, m[d].l, sq.l);
        R0 = d == 0 ? sq : df_add(R0, sq);
        df p = two_prod(q.Th[d], m[d].h);
        p.l = __fmaf_rn(q.Tl[d], m[d].h, __fmaf_rn(q.Th[d], m[d].l, p.l));
        Ad[d] = fast_two_sum(q.Sh[d], -p.h);
        Ad[d].l = __fadd_rn(Ad[d].l, __fsub_rn(q.Sl[d], p.l));
      }
      unsigned okm = act ? 0xffu : 0u;
      if (test_cube) {
        // the reference's cube |n_d| <= nsum, n the image's whole shift
        const float na[3] = {a2.y - b2v.y, a2.z - b2v.z, a2.w - b2v.w};
        const unsigned bits[3] = {0xaau, 0xccu, 0xf0u};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float n = na[d] + sh[d];
          if (!(fabsf(n) <= q.nsum)) okm &= bits[d];
          if (!(fabsf(n + sg[d]) <= q.nsum)) okm &= ~bits[d];
        }
      }
      df R[8];
      R[0] = R0;
      R[1] = df_add(R0, Ad[0]);
      R[2] = df_add(R0, Ad[1]);
      R[3] = df_add(R[1], Ad[1]);
#pragma unroll
      for (int c = 0; c < 4; ++c) R[4 + c] = df_add(R[c], Ad[2]);
      int at[8], total = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const bool in = R[c].h < q.rc2 && ((okm >> c) & 1u);
        const unsigned ball = __ballot_sync(ALL, in);
        at[c] = in ? total + __popc(ball & lt) : -1;
        total += __popc(ball);
        if (in) ws->q[at[c]] = make_float2(R[c].h, R[c].l);
      }
      __syncwarp();
      for (int r = lane; r < total; r += 32) {
        const float2 v = ws->q[r];
        const df f = ewd_image<ENERGY>({v.x, v.y}, tab);
        if (ENERGY) {
          const df s0 = two_sum(en.h, f.h), s1 = two_sum(en.l, f.l), s2 = two_sum(s0.l, s1.h);
          en = fast_two_sum(s0.h, s2.h);
          enc = __fadd_rn(enc, __fadd_rn(s1.l, s2.l));
        } else {
          ws->q[r] = make_float2(f.h, f.l);
        }
      }
      __syncwarp();
      if constexpr (ENERGY) {
        // images with one component of length L + |m_d| inside the longer cut-off
        bool more = false;
#pragma unroll
        for (int d = 0; d < 3; ++d) more = more || R0.h + q.Sh[d] + q.Th[d] * m[d].h < q.rc2;
        if (act && more) {
#pragma unroll
          for (int d = 0; d < 3; ++d)
            for (int c = 0; c < 8; ++c) {
              if ((c >> d) & 1) continue;
              const float R2 = R0.h + q.Sh[d] + q.Th[d] * m[d].h + ((c & 1) ? Ad[0].h : 0.f) +
                               ((c & 2) ? Ad[1].h : 0.f) + ((c & 4) ? Ad[2].h : 0.f);
              const float na = d == 0 ? a2.y - b2v.y : (d == 1 ? a2.z - b2v.z : a2.w - b2v.w);
              if (R2 < q.rc2 && ((okm >> c) & 1u) && fabsf(na + sh[d] - sg[d]) <= q.nsum) enc += ewd_erfc32(R2);
            }
        }
      } else {
        df v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float2 t = at[c] >= 0 ? ws->q[at[c]] : make_float2(0.f, 0.f);
          v[c] = {t.x, t.y};
        }
        const df p0 = df_add_fast(v[0], v[1]), p1 = df_add_fast(v[2], v[3]);
        const df p2 = df_add_fast(v[4], v[5]), p3 = df_add_fast(v[6], v[7]);
        df V[3], Va;
        V[2] = df_add_fast(p2, p3);
        Va = df_add_fast(df_add_fast(p0, p1), V[2]);
        V[1] = df_add_fast(p1, p3);
        V[0] = df_add_fast(df_add_fast(v[1], v[3]), df_add_fast(v[5], v[7]));
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          df F = df_sub(df_mul(m[d], Va), df_mul({q.Ph[d], q.Pl[d]}, V[d]));
          F.h *= sg[d];
          F.l *= sg[d];
          fa[d] = df_norm(df_add(fa[d], F));
          fb[d] = df_norm(df_sub(fb[d], F));
          const int src = (lane + 1) & 31;
          fb[d].h = __shfl_sync(ALL, fb[d].h, src);
          fb[d].l = __shfl_sync(ALL, fb[d].l, src);
        }
        __syncwarp();  // the queue's reads are done
      }
    }
    if constexpr (ENERGY) {
      double e = df_value(en) + (double)enc;
#pragma unroll
      for (int o = 16; o; o >>= 1) e += __shfl_down_sync(ALL, e, o);
      if (lane == 0) eout[u] = e;
    } else {
      // b's sums back to their home lanes
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int src = (lane - s1 - 1) & 31;
        fb[d].h = __shfl_sync(ALL, fb[d].h, src);
        fb[d].l = __shfl_sync(ALL, fb[d].l, src);
      }
      if (diag) {
        if (va)
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const df f = df_norm(df_add(fa[d], fb[d]));
            outa[(((size_t)(I * split + part) * P + j) * 3 + d) * A.Ns + a] = make_float2(f.h, f.l);
          }
        continue;
      }
      float2 *ob = CROSS ? outb : outa;
      if (va)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const df f = df_norm(fa[d]);
          outa[(((size_t)(J * split + part) * P + j) * 3 + d) * A.Ns + a] = make_float2(f.h, f.l);
        }
      if (vb)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const df f = df_norm(fb[d]);
          ob[(((size_t)(I * split + part) * P + j) * 3 + d) * B.Ns + b0] = make_float2(f.h, f.l);
        }
    }
  }
}

// f += scale * sum over the T partial slots
__global__ void k_ewd_finish(int N, int Ns, size_t S, const float2 *__restrict__ part, int T, double scale,
                             double *__restrict__ f) {
  const size_t s = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S || (int)(s % Ns) >= N) return;
  df acc = {0.f, 0.f};
#pragma unroll 8
  for (int t = 0; t < T; ++t) {
    const float2 v = part[(size_t)t * S + s];
    acc = df_norm(df_add(acc, {v.x, v.y}));
  }
  f[s] += scale * df_value(acc);
}

// Parts of a tile's rotation steps.  With a warp a tile, 128 electrons and 32
// beads kept 320 of the 2432 warps that fit on 152 SMs.  So up to four parts
// until there are two rounds of warps (beyond, the last round costs less than
// the parts' slots of partials); eight only where four leave most SM
// sub-partitions idle.  The parts set the order of the sums, so the line counts
// 152 SMs and not the device's: the same system gives the same bits.  A step of
// N x P electrons (|n| <= 4) with whole tiles, and with 2, 4 and 8 parts, * taken: 16 x 4 63, 53* (8); 64 x 32 96, 64* (8);
// 128 x 32 109, 85, 80*, 87; 128 x 64 119, 106, 94*, 96; 200 x 48 160, 138,
// 133*, 134; 300 x 64 234, 222*, 221; 512 x 33 282, 281*, 280; 512 x 64 435*,
// 433; 256 + 256 x 64 614, 610* (2 a cross tile) us.
int ewd_split(size_t jobs) {
  if (jobs * 4 < 8 * 152) return 8;
  int split = 1;
  while (split < 4 && jobs * split < 2 * 2432) split *= 2;
  return split;
}

template <bool CROSS, bool ENERGY>
static cudaError_t launch_tiles(const EwdPrm &q, int P, const EwdSide &A, const EwdSide &B, float2 *oa, float2 *ob,
                                double *eo, int TA, int TB, int split, int bps, cudaStream_t st) {
  static int occ = 0, sms = 0;
  if (!occ) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_ewd_tiles<CROSS, ENERGY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ewd_smem<ENERGY>());
    int n = 0;
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_ewd_tiles<CROSS, ENERGY>, 32 * EWD_WARPS,
                                                        ewd_smem<ENERGY>());
    if (e != cudaSuccess) return e;
    occ = n > 0 ? n : 1;
  }
  const size_t jobs = (size_t)(CROSS ? TA * TB : TA * (TA + 1) / 2) * P * split;
  const size_t room = (size_t)sms * (bps > 0 && bps < occ ? bps : occ);
  // fewer jobs than warps: over as many SMs as there are jobs
  size_t grid = (jobs + EWD_WARPS - 1) / EWD_WARPS;
  if (grid < jobs && grid < (size_t)sms) grid = jobs < (size_t)sms ? jobs : sms;
  if (grid > room) grid = room;
  k_ewd_tiles<CROSS, ENERGY><<<(int)grid, 32 * EWD_WARPS, ewd_smem<ENERGY>(), st>>>(
      q, P, A, B, oa, ob, eo, TA, TB, split);
  return XK_LAUNCHED();
}

static cudaError_t split_positions(const Geo &g, const EwdPrm &q, const double *x, double *pos, cudaStream_t st) {
  XK_PROF("ewald_split");
  k_ewd_split<<<cdivz((size_t)g.P * g.Ns, 128), 128, 0, st>>>(q, g.N, g.Ns, g.P, x, (float4 *)pos);
  return XK_LAUNCHED();
}

static cudaError_t finish(const Geo &g, const float2 *part, int T, double scale, double *f, cudaStream_t st) {
  XK_PROF("pair_finish");
  k_ewd_finish<<<cdivz(g.slots(), 256), 256, 0, st>>>(g.N, g.Ns, g.slots(), part, T, scale, f);
  return XK_LAUNCHED();
}

// scratch: T slots of partials (8 bytes each), then the split positions
cudaError_t ewd_force(const Geo &g, const PairPrm &p, const double *x, double *f, double *scratch, cudaStream_t st) {
  const EwdPrm q = make_ewd(g, p);
  const int T = (g.N + 31) / 32, split = ewd_split((size_t)T * (T + 1) / 2 * g.P);
  double *pos = scratch + (((size_t)T * split * g.slots() + 1) & ~(size_t)1);
  cudaError_t e = split_positions(g, q, x, pos, st);
  if (e != cudaSuccess) return e;
  const EwdSide A{(const float4 *)pos, g.N, g.Ns};
  {
    XK_PROF("pair_tiles_ewald_real");
    e = launch_tiles<false, false>(q, g.P, A, A, (float2 *)scratch, nullptr, nullptr, T, T, split,
                                   tuning(TUNE_PAIR64_BPS, PAIR_EWALD_REAL, 3, g.N, g.P), st);
  }
  if (e != cudaSuccess) return e;
  // unit charges and scaled lengths inside: F = s alpha^2 / (m P) sum
  return finish(g, (const float2 *)scratch, T * split, p.qs * p.alpha * p.alpha * p.inv_mass / g.P, f, st);
}

// energies erfc(x)/x of the tiles' parts (jobs * P * *parts doubles, T (T + 1) / 2 jobs a slice)
cudaError_t ewd_energy_tiles(const Geo &g, const PairPrm &p, const double *x, double *scratch, int *parts,
                             cudaStream_t st) {
  const EwdPrm q = make_ewd(g, p);
  const int T = (g.N + 31) / 32, split = ewd_split((size_t)T * (T + 1) / 2 * g.P);
  double *pos = scratch + (((size_t)T * split * g.slots() + 1) & ~(size_t)1);
  cudaError_t e = split_positions(g, q, x, pos, st);
  if (e != cudaSuccess) return e;
  const EwdSide A{(const float4 *)pos, g.N, g.Ns};
  *parts = split;
  XK_PROF("pair_tiles_ewald_real");
  return launch_tiles<false, true>(q, g.P, A, A, nullptr, nullptr, scratch, T, T, split, 0, st);
}

cudaError_t ewd_force_2(const Geo &ga, const Geo &gb, const PairPrm &p, const double *xa, double inv_ma,
                        const double *xb, double inv_mb, double *fa, double *fb, double *scratch, cudaStream_t st) {
  const EwdPrm q = make_ewd(ga, p);
  const int TA = (ga.N + 31) / 32, TB = (gb.N + 31) / 32;
  const int split = ewd_split((size_t)TA * TB * ga.P);
  double *oa = scratch, *ob = oa + (size_t)TB * split * ga.slots();
  double *pa = scratch + ((((size_t)TB * ga.slots() + (size_t)TA * gb.slots()) * split + 1) & ~(size_t)1);
  double *pb = pa + ewd_pos_doubles(ga);
  cudaError_t e = split_positions(ga, q, xa, pa, st);
  if (e == cudaSuccess) e = split_positions(gb, q, xb, pb, st);
  if (e != cudaSuccess) return e;
  {
    XK_PROF("pair_cross");
    e = launch_tiles<true, false>(q, ga.P, {(const float4 *)pa, ga.N, ga.Ns}, {(const float4 *)pb, gb.N, gb.Ns},
                                  (float2 *)oa, (float2 *)ob, nullptr, TA, TB, split, 0, st);
  }
  if (e != cudaSuccess) return e;
  const double s = p.qs * p.alpha * p.alpha / ga.P;
  e = finish(ga, (const float2 *)oa, TB * split, s * inv_ma, fa, st);
  if (e != cudaSuccess) return e;
  return finish(gb, (const float2 *)ob, TA * split, s * inv_mb, fb, st);
}

}  // namespace xk
