// One-CTA building blocks of the batched layer kernel (k_batch.cu): a
// one-sided Jacobi on the columns of a matrix in shared memory or L2, and a
// small complex GEMM.
#pragma once

#include <cuda_runtime.h>

#include "qt_internal.cuh"

// ---------------------------------------------------------------------------
// rotation of one column pair
// ---------------------------------------------------------------------------

template <typename R>
struct cta_rotation {
  R c, s, er, ei;  // x_p' = c x_p - s e^{-i phi} x_q ;  x_q' = s e^{i phi} x_p + c x_q
  bool on;
};

// From the pair's sums aa = |x_p|^2, bb = |x_q|^2, gr + i gi = x_p^H x_q:
// rotate while the relative off-diagonal exceeds tol; the angle in FP64,
// rounded to the columns' precision.  What is fused is written out: the same
// bits wherever this is inlined.
template <typename R>
__device__ __forceinline__ cta_rotation<R> cta_angle64(R aa, R bb, R gr, R gi, double tol, double nu2) {
  cta_rotation<R> o;
  o.c = 1; o.s = 0; o.er = 1; o.ei = 0;
  const double ag = sqrt(fma((double)gr, (double)gr, __dmul_rn((double)gi, (double)gi)));
  o.on = (double)aa > nu2 && (double)bb > nu2 && ag > tol * sqrt((double)aa * bb);
  if (o.on) {
    const double zeta = ((double)bb - aa) / (2.0 * ag);
    const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0)));
    const double cs = 1.0 / sqrt(fma(t, t, 1.0));
    o.c = (R)cs;
    o.s = (R)(cs * t);
    o.er = (R)(gr / ag);
    o.ei = (R)(gi / ag);
  }
  return o;
}

// Unevaluated sums hi + lo of two floats (|lo| <= ulp(hi) / 2), good to about
// 2^-44; the error-free sum and product are Dekker's and Knuth's.  Rounded
// operations that the compiler may not fuse throughout: a product fused into
// the sum after it would no longer be the product whose error is kept.
struct ff { float h, l; };
__device__ __forceinline__ ff ff_fast(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ ff ff_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ ff ff_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, fmaf(a, b, -p)};
}
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
  ff p = ff_prod(a.h, b.h);
  p.l = fmaf(a.h, b.l, fmaf(a.l, b.h, p.l));
  return ff_fast(p.h, p.l);
}
__device__ __forceinline__ ff ff_sqrt(ff a) {  // one Newton step from the FP32 root
  const float r = sqrtf(a.h);
  return ff_fast(r, __fdividef(__fadd_rn(fmaf(-r, r, a.h), a.l), 2.f * r));
}
__device__ __forceinline__ ff ff_rcp(ff a) {  // Newton: i (1 + e + e^2), e = 1 - a i
  const float i = __frcp_rn(a.h);
  const float e = fmaf(-a.l, i, fmaf(-a.h, i, 1.f));
  return ff_fast(i, __fmul_rn(i, fmaf(e, e, e)));
}
__device__ __forceinline__ ff ff_one_plus(ff a) {
  ff s = ff_sum(1.f, a.h);
  return ff_fast(s.h, __fadd_rn(s.l, a.l));
}
// The float that a value within 2^-40 relative of v rounds to; *sure is
// cleared where two floats are possible.
__device__ __forceinline__ float ff_round(ff v, bool* sure) {
  const float d = __fmul_rn(fabsf(v.h), 9.0949470177e-13f);  // 2^-40
  const float up = __fadd_rn(v.h, __fadd_rn(v.l, d)), dn = __fadd_rn(v.h, __fsub_rn(v.l, d));
  *sure = *sure && up == dn;
  return up;
}

// The same rotation as cta_angle64 bit for bit, without FP64: in unevaluated
// FP32 pairs, whose 2^-42 leaves the rounded float the FP64 evaluation gives
// (2^-50 off the exact value) in all but one case in 10^4; those, sums
// outside [2^-100, 2^100], and pairs at the tolerance itself go to FP64.
// Why: a warp instruction occupies the SM's two FP64 lanes for 16 cycles, and
// the four roots and five quotients were 1700 such cycles for every pair,
// against 64 for the products and rotation of two columns of 64 rows.
__device__ __forceinline__ cta_rotation<float> cta_angle(float aa, float bb, float gr, float gi, double tol, float tol2,
                                                         double nu2, float nu2_dn) {
  cta_rotation<float> o;
  o.c = 1.f; o.s = 0.f; o.er = 1.f; o.ei = 0.f; o.on = false;
  // (double)aa > nu2 exactly when aa exceeds the largest float below nu2
  if (!(aa > nu2_dn && bb > nu2_dn)) return o;
  const float gm = fmaxf(fabsf(gr), fabsf(gi));
  const bool range = fminf(aa, bb) > 7.9e-31f && fmaxf(aa, bb) < 1.2e30f && gm > 7.9e-31f && tol2 > 1e-25f;
  if (!range) return cta_angle64<float>(aa, bb, gr, gi, tol, nu2);
  // common factor 2^-e: the larger of |gr|, |gi| into [1, 2)
  const float sc = __uint_as_float((254u << 23) - (__float_as_uint(gm) & 0x7f800000u));
  const float xr = __fmul_rn(gr, sc), xi = __fmul_rn(gi, sc), xa = __fmul_rn(aa, sc), xb = __fmul_rn(bb, sc);
  // (the smaller norm is above 1e-30 then, or these are no sums of two columns)
  if (fmaxf(xa, xb) > 1e30f || fminf(xa, xb) < 0.9e-30f) return cta_angle64<float>(aa, bb, gr, gi, tol, nu2);
  const ff p1 = ff_prod(xr, xr), p2 = ff_prod(xi, xi);
  ff p = ff_sum(p1.h, p2.h);
  p = ff_fast(p.h, __fadd_rn(p.l, __fadd_rn(p1.l, p2.l)));
  // |gamma|^2 against tol^2 aa bb, both to 1e-6; the factors first, so that nothing overflows
  const float ratio = __fdividef(p.h, xa) * __fdividef(1.f, xb);
  if (ratio < 0.9999f * tol2) return o;
  bool sure = ratio > 1.0001f * tol2;
  const ff ag = ff_sqrt(p), inv = ff_rcp(ag);
  ff er = ff_prod(xr, inv.h), ei = ff_prod(xi, inv.h);
  er = ff_fast(er.h, fmaf(xr, inv.l, er.l));
  ei = ff_fast(ei.h, fmaf(xi, inv.l, ei.l));
  const ff d = ff_sum(xb, -xa);
  ff z = ff_prod(d.h, inv.h);
  z = ff_fast(z.h, fmaf(d.h, inv.l, fmaf(d.l, inv.h, z.l)));
  const bool neg = z.h < 0.f || (z.h == 0.f && z.l < 0.f);
  z = {__fmul_rn(0.5f, neg ? -z.h : z.h), __fmul_rn(0.5f, neg ? -z.l : z.l)};
  sure = sure && z.h < 1e15f;
  const ff r = ff_sqrt(ff_one_plus(ff_mul(z, z)));
  ff g = ff_sum(z.h, r.h);
  g = ff_fast(g.h, __fadd_rn(g.l, __fadd_rn(z.l, r.l)));
  const ff t = ff_rcp(g);
  const ff q = ff_one_plus(ff_mul(t, t));
  // 1 / sqrt(q): y (1 + e / 2 + 3 e^2 / 8), e = 1 - q y^2
  const float y = rsqrtf(q.h);
  const ff y2 = ff_prod(y, y);
  const float e = __fsub_rn(fmaf(-q.h, y2.h, 1.f), fmaf(q.h, y2.l, __fmul_rn(q.l, y2.h)));
  const ff cs = ff_fast(y, __fmul_rn(__fmul_rn(y, e), fmaf(0.375f, e, 0.5f)));
  const ff sn = ff_mul(cs, t);
  o.c = ff_round(cs, &sure);
  o.s = ff_round(sn, &sure);
  o.s = neg ? -o.s : o.s;
  o.er = copysignf(ff_round(er, &sure), xr);  // (a sum of pairs loses the sign of a zero)
  o.ei = copysignf(ff_round(ei, &sure), xi);
  o.on = true;
  // a component of the phase so small that its error term would be denormal
  sure = sure && (xr == 0.f || fabsf(xr) > 1e-15f) && (xi == 0.f || fabsf(xi) > 1e-15f);
  if (!sure) return cta_angle64<float>(aa, bb, gr, gi, tol, nu2);
  return o;
}

template <typename R>
__device__ inline R cta_warp_sum(R v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// one-sided Jacobi
// ---------------------------------------------------------------------------

// Tournament (circle method) over n (even) players.
__device__ inline void cta_tourney(int r, int q, int n, int& a, int& b) {
  if (q == 0) { a = r % (n - 1); b = n - 1; }
  else { a = (r + q) % (n - 1); b = (r - q + (n - 1)) % (n - 1); }
}

// The sums of NP column pairs over the warp, each lane ending with sum
// (lane / (8 / NP)) in the order aa, bb, gr, gi of pair 0, of pair 1, ...
// Every step halves the values a lane carries, so 4 NP sums take 4 NP + 1 (or
// fewer) shuffles instead of 20 NP; a value is summed over the lanes in the
// same order as by cta_warp_sum.
template <int NP, typename R>
__device__ __forceinline__ R cta_pair_sums(R (&v)[4 * NP]) {
  const int lane = threadIdx.x & 31;
  int off = 16;
#pragma unroll
  for (int cnt = 4 * NP; cnt > 1; cnt >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < cnt / 2; i++) {
      const R send = up ? v[i] : v[i + cnt / 2];
      const R keep = up ? v[i + cnt / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  R s = v[0];
#pragma unroll
  for (; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}

template <int RPL, typename C>
__device__ __forceinline__ void cta_load_column(C (&x)[RPL], const C* X, int m) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < RPL; k++) x[k] = lane + 32 * k < m ? X[lane + 32 * k] : czero<C>();
}

// x_p' = c x_p - s e^{-i phi} x_q, x_q' = s e^{i phi} x_p + c x_q, every
// rounding written out: the products that are fused stay the same wherever
// this is inlined.
template <int RPL>
__device__ __forceinline__ void cta_store_rotated(const float2 (&xp)[RPL], const float2 (&xq)[RPL], float c, float s,
                                                  float er, float ei, float2* P, float2* Q, int m) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < RPL; k++) {
    if (lane + 32 * k < m) {
      const float2 u = xp[k], v = xq[k];
      P[lane + 32 * k] =
          make_float2(fmaf(c, u.x, -__fmul_rn(s, fmaf(er, v.x, __fmul_rn(ei, v.y)))),
                      fmaf(c, u.y, -__fmul_rn(s, fmaf(er, v.y, -__fmul_rn(ei, v.x)))));
      Q[lane + 32 * k] =
          make_float2(fmaf(c, v.x, __fmul_rn(s, fmaf(er, u.x, -__fmul_rn(ei, u.y)))),
                      fmaf(s, fmaf(ei, u.x, __fmul_rn(er, u.y)), __fmul_rn(c, v.y)));
    }
  }
}

// One round's pairs first .. first + NP - 1 (those below `pairs`) by one warp:
// both columns of each pair in registers from the sums to the rotation, the
// angles of all NP pairs evaluated at once by the lanes that hold their sums.
template <int NP, int RPL>
__device__ __forceinline__ bool cta_round_pairs(float2* X, int ld, int m, int n, int round, int first, double tol,
                                                float tol2, double nu2, float nu2_dn) {
  const int lane = threadIdx.x & 31, pairs = n / 2;
  float2 xp[NP][RPL], xq[NP][RPL];
  float2 *P[NP], *Q[NP];
  float v[4 * NP];
#pragma unroll
  for (int g = 0; g < NP; g++) {
    int a, b;
    cta_tourney(round, min(first + g, pairs - 1), n, a, b);
    P[g] = X + (size_t)ld * a;
    Q[g] = X + (size_t)ld * b;
    const int rows = first + g < pairs ? m : 0;
    cta_load_column<RPL>(xp[g], P[g], rows);
    cta_load_column<RPL>(xq[g], Q[g], rows);
  }
#pragma unroll
  for (int g = 0; g < NP; g++) {
    float aa = 0, bb = 0, gr = 0, gi = 0;
#pragma unroll
    for (int k = 0; k < RPL; k++) {
      const float2 u = xp[g][k], w = xq[g][k];
      aa = fmaf(u.x, u.x, fmaf(u.y, u.y, aa));
      bb = fmaf(w.x, w.x, fmaf(w.y, w.y, bb));
      gr = fmaf(u.x, w.x, fmaf(u.y, w.y, gr));
      gi = fmaf(u.x, w.y, fmaf(-u.y, w.x, gi));
    }
    v[4 * g] = aa; v[4 * g + 1] = bb; v[4 * g + 2] = gr; v[4 * g + 3] = gi;
  }
  const float s = cta_pair_sums<NP>(v);
  constexpr int ST = 8 / NP;
  const int base = lane & ~(4 * ST - 1);
  const float aa = __shfl_sync(0xffffffffu, s, base), bb = __shfl_sync(0xffffffffu, s, base + ST);
  const float gr = __shfl_sync(0xffffffffu, s, base + 2 * ST), gi = __shfl_sync(0xffffffffu, s, base + 3 * ST);
  const cta_rotation<float> o = cta_angle(aa, bb, gr, gi, tol, tol2, nu2, nu2_dn);
  const unsigned on = __ballot_sync(0xffffffffu, o.on);
  if (!on) return false;
#pragma unroll
  for (int g = 0; g < NP; g++) {
    const int src = 4 * ST * g;
    const float c = __shfl_sync(0xffffffffu, o.c, src), sn = __shfl_sync(0xffffffffu, o.s, src);
    const float er = __shfl_sync(0xffffffffu, o.er, src), ei = __shfl_sync(0xffffffffu, o.ei, src);
    if ((on >> src) & 1) cta_store_rotated<RPL>(xp[g], xq[g], c, sn, er, ei, P[g], Q[g], m);
  }
  return true;
}

// Jacobi on the n (even) columns of X (m <= 32 RPL rows, leading dimension
// ld; shared or global memory of this CTA alone): rounds of n / 2 disjoint
// pairs.  A pair is rotated while its relative off-diagonal exceeds tol;
// columns with |x|^2 <= nu2 are frozen.  A sweep that rotates nothing ends
// it.  Returns the sweeps run.  Every thread of the CTA calls it.
//
// What bounds it: the chain of a round (column loads, five levels of
// shuffles, the angle, the rotation, one barrier) times n - 1 rounds a sweep;
// with two or more CTAs on an SM their chains overlap.  A warp takes one pair
// at a time while there is a warp per pair, then two and four, whose chains
// overlap too.  Measured on 6240 updates of 200 Haar circuits (caps 16 to 64):
// 14.5 ms a replay, 160 ms with the angles in FP64 by every lane, the columns
// in L2 and the products untiled.
template <int NT, int RPL>
__device__ int cta_jacobi(float2* X, int ld, int m, int n, double tol, double nu2, int max_sweeps) {
  constexpr int W = NT / 32;
  // pairs a warp holds at once: 16 RPL registers for four
  constexpr int MAXP = NT <= 256 || RPL <= 2 ? 4 : NT == 512 ? (RPL <= 4 ? 4 : 2) : (RPL <= 4 ? 2 : 1);
  const int warp = threadIdx.x >> 5, pairs = n / 2;
  const float tol2 = (float)(tol * tol), nu2_dn = __double2float_rd(nu2);
  int sweeps = 0;
  if (n < 2) return 0;
  for (int sweep = 0; sweep < max_sweeps; sweep++) {
    bool rotated = false;
    for (int r = 0; r < n - 1; r++) {
      if (MAXP == 1 || pairs <= W) {
        for (int q = warp; q < pairs; q += W)
          rotated |= cta_round_pairs<1, RPL>(X, ld, m, n, r, q, tol, tol2, nu2, nu2_dn);
      } else if (MAXP == 2 || pairs <= 2 * W) {
        for (int q = 2 * warp; q < pairs; q += 2 * W)
          rotated |= cta_round_pairs<MAXP < 2 ? 1 : 2, RPL>(X, ld, m, n, r, q, tol, tol2, nu2, nu2_dn);
      } else {
        for (int q = 4 * warp; q < pairs; q += 4 * W)
          rotated |= cta_round_pairs<MAXP < 4 ? 1 : 4, RPL>(X, ld, m, n, r, q, tol, tol2, nu2, nu2_dn);
      }
      __syncthreads();
    }
    sweeps = sweep + 1;
    if (!__syncthreads_or(rotated)) break;
  }
  return sweeps;
}

// m <= 32 RMAX.
template <int NT, int RMAX>
__device__ int cta_jacobi_any(float2* X, int ld, int m, int n, double tol, double nu2, int max_sweeps) {
  if (m <= 32) return cta_jacobi<NT, 1>(X, ld, m, n, tol, nu2, max_sweeps);
  if constexpr (RMAX >= 2)
    if (m <= 64) return cta_jacobi<NT, 2>(X, ld, m, n, tol, nu2, max_sweeps);
  if constexpr (RMAX >= 4)
    if (m <= 128) return cta_jacobi<NT, 4>(X, ld, m, n, tol, nu2, max_sweeps);
  if constexpr (RMAX >= 8) return cta_jacobi<NT, 8>(X, ld, m, n, tol, nu2, max_sweeps);
  return 0;
}

// ---------------------------------------------------------------------------
// op(A) op(B) (M x N), one CTA, in the precision of C (operands widened as read)
// ---------------------------------------------------------------------------
//
// TILE x TILE outputs at a time, 16 deep, through shared memory (both
// operands read along their columns, so every global load is coalesced).
// conj_a: op(A) = A^H with A (K x M), its columns taken in the order perm_a
// where that is given; conj_b: op(B) = B^H with B (N x K).  store(r, c, value)
// takes the results.  sm: cta_gemm_smem<C>(TILE) bytes.
constexpr int CTA_GK = 16;
template <typename C>
constexpr size_t cta_gemm_smem(int tile) { return 2 * (size_t)CTA_GK * (tile + 1) * sizeof(C); }

template <int NT, int TILE, typename C, typename EA, typename EB, typename F>
__device__ void cta_gemm_tile(bool conj_a, bool conj_b, int M, int N, int K, const EA* A, int lda, const int* perm_a,
                              const EB* B, int ldb, void* sm, F store) {
  constexpr int TX = (NT <= 512 || TILE < 32) ? 16 : 32, TY = NT / TX;
  constexpr int RM = TILE / TX, RN = TILE / TY;
  static_assert(RM >= 1 && RN >= 1, "tile too small for the CTA");
  C (*As)[TILE + 1] = reinterpret_cast<C (*)[TILE + 1]>(sm);
  C (*Bs)[TILE + 1] = As + CTA_GK;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  for (int m0 = 0; m0 < M; m0 += TILE)
    for (int n0 = 0; n0 < N; n0 += TILE) {
      C acc[RM][RN];
#pragma unroll
      for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) acc[i][j] = czero<C>();
      for (int k0 = 0; k0 < K; k0 += CTA_GK) {
        for (int idx = threadIdx.x; idx < TILE * CTA_GK; idx += NT) {
          C v = czero<C>();
          const int mi = conj_a ? idx / CTA_GK : idx % TILE, ka = conj_a ? idx % CTA_GK : idx / TILE;
          if (m0 + mi < M && k0 + ka < K)
            v = conj_a ? cconj(ccast<C>(A[(k0 + ka) + (size_t)lda * (perm_a ? perm_a[m0 + mi] : m0 + mi)]))
                       : ccast<C>(A[(m0 + mi) + (size_t)lda * (k0 + ka)]);
          As[ka][mi] = v;
          v = czero<C>();
          const int ni = conj_b ? idx % TILE : idx / CTA_GK, kb = conj_b ? idx / TILE : idx % CTA_GK;
          if (n0 + ni < N && k0 + kb < K)
            v = conj_b ? cconj(ccast<C>(B[(n0 + ni) + (size_t)ldb * (k0 + kb)]))
                       : ccast<C>(B[(k0 + kb) + (size_t)ldb * (n0 + ni)]);
          Bs[kb][ni] = v;
        }
        __syncthreads();
        const int kl = min(CTA_GK, K - k0);
#pragma unroll 4
        for (int k = 0; k < kl; k++) {
          C a[RM], b[RN];
#pragma unroll
          for (int i = 0; i < RM; i++) a[i] = As[k][tx + TX * i];
#pragma unroll
          for (int j = 0; j < RN; j++) b[j] = Bs[k][ty + TY * j];
#pragma unroll
          for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < RN; j++) cfma(acc[i][j], a[i], b[j]);
        }
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) {
          const int r = m0 + tx + TX * i, c = n0 + ty + TY * j;
          if (r < M && c < N) store(r, c, acc[i][j]);
        }
    }
  __syncthreads();
}

// TMAX: the largest tile the caller's shared memory holds (32 or 64).  The
// 64-wide tile reads shared memory half as often per product; a product of
// at most 32 rows or columns would leave half of it empty.
template <int NT, int TMAX, typename C, typename EA, typename EB, typename F>
__device__ void cta_gemm(bool conj_a, bool conj_b, int M, int N, int K, const EA* A, int lda, const int* perm_a,
                         const EB* B, int ldb, void* sm, F store) {
  if constexpr (TMAX >= 64)
    if (M > 32 && N > 32)
      return cta_gemm_tile<NT, 64, C>(conj_a, conj_b, M, N, K, A, lda, perm_a, B, ldb, sm, store);
  cta_gemm_tile<NT, 32, C>(conj_a, conj_b, M, N, K, A, lda, perm_a, B, ldb, sm, store);
}
