// One-sided block Jacobi SVD (Hestenes).
//
// Replaces the dense LAPACK ?gesdd called by LinearAlgebra.svd at
// src/svd.jl:26-27 and in switch! (src/switch.jl:39): X (mm x nn,
// mm >= nn) is driven to orthogonal columns, X <- X V, so X = U diag(s) and
// the input equals U diag(s) V^H.
//
// Columns are split into blocks of JW = 8.  One sweep is a round-robin
// tournament over the blocks (circle method); a round processes every block
// pair (16 columns) at once: the pair's 16x16 Gram is formed, tested against
// `tol` (relative off-diagonals), diagonalised by a cyclic two-sided Jacobi
// (the pair solver) and the resulting unitary applied to the pair's columns
// of X (and rows of V).  A sweep in which no pair rotates ends the iteration.
// Round implementations:
//   FP32 storage, where the caller takes pairwise rotations (a sketched
//     matrix): jacobi_ring32_kernel -- one cooperative launch per sweep,
//     single column pairs rotated in the registers of a CTA that holds eight
//     columns, blocks of four columns passed between CTAs (see the comment
//     above that kernel);
//   FP32 storage otherwise: jacobi_sweep32_kernel -- one cooperative launch per
//     sweep, or for all sweeps where only a sweep without rotations ends them,
//     each round rebuilding its columns from the previous round's unitaries
//     (see the comment above that kernel);
//   FP32 storage, two launches per round: pair_eig32_kernel (Gram + test +
//     pair solver) and pair_apply32_kernel (rotation);
//   FP64 storage, default: pair_round64_kernel -- one launch per round, a
//     thread-block cluster holding the pair's rows in shared memory, the
//     rotation angles found in FP32 (see the comment above that kernel);
//   FP32 storage on request: pair_round_kernel, the same shape of round;
//   any storage: gram_kernel + eig_kernel + apply_kernel (partial Grams
//     over row chunks, FP64 pair solver, rotation).
// eig_kernel works on the FP64 Gram; the others on the scaled Gram (cosines) in
// FP32, see pair_eig_scaled below.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <functional>
#include <vector>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include <cooperative_groups.h>

#include <type_traits>

#include "qt_internal.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int JW = 8;        // columns per block
constexpr int JC = 2 * JW;   // columns per block pair
constexpr int JR = 64;       // rows per shared-memory slab
constexpr int NT = 256;      // threads per CTA
constexpr int MAX_INNER = 12;
constexpr int NGRAM = JC * JC;
static_assert(NT == NGRAM, "the round kernel maps one Gram entry to each thread");

__device__ inline void tournament(int r, int q, int n, int& a, int& b) {
  // circle method over n (even) players, round r, table q
  if (q == 0) { a = r % (n - 1); b = n - 1; }
  else { a = (r + q) % (n - 1); b = (r - q + (n - 1)) % (n - 1); }
  if (a > b) { const int t = a; a = b; b = t; }
}

__device__ inline void pair_columns(int round, int pair, int nb, int nn, int* col) {
  int bi, bj;
  tournament(round, pair, nb, bi, bj);
  if (threadIdx.x < JC) {
    const int c = threadIdx.x;
    const int gc = (c < JW) ? bi * JW + c : bj * JW + (c - JW);
    col[c] = (gc < nn) ? gc : -1;
  }
}

// partner of index y in inner round ir of the circle tournament over the 16
// columns of a pair (the pairing of tournament(ir, ., 16)): 15 meets ir, the
// others meet 2 ir - y (mod 15).  (Pairing the two blocks' columns first and
// each block's own after converged in more outer sweeps.)
__device__ inline int inner_partner(int ir, int y) {
  if (y == JC - 1) return ir;
  if (y == ir) return JC - 1;
  return (2 * ir - y + (JC - 1)) % (JC - 1);
}

template <typename T> struct acc_of;
template <> struct acc_of<double> { typedef double2 type; };
template <> struct acc_of<float> { typedef float2 type; };

// Partial Gram of one pair over rows [r_begin, r_end) -> part (16x16 double2).
template <typename TS, typename TG>
__global__ void __launch_bounds__(NT)
gram_kernel(const TS* __restrict__ X, int64_t ldx, int mm, int nn, int nb, int round, int rows_per_chunk,
            double2* __restrict__ parts) {
  typedef typename acc_of<TG>::type CG;
  __shared__ TS Xs[JR][JC + 1];
  __shared__ int col[JC];
  const int pair = blockIdx.x, chunk = blockIdx.y;
  pair_columns(round, pair, nb, nn, col);
  __syncthreads();
  const int t = threadIdx.x;
  int gi = -1, gj = -1;
  if (t < JC * (JC + 1) / 2) {
    int r = 0, rem = t;
    while (rem >= JC - r) { rem -= JC - r; r++; }
    gi = r; gj = r + rem;
  }
  CG acc = czero<CG>();
  const int r_begin = chunk * rows_per_chunk, r_end = min(mm, r_begin + rows_per_chunk);
  for (int r0 = r_begin; r0 < r_end; r0 += JR) {
    for (int idx = t; idx < JR * JC; idx += NT) {
      const int rr = idx % JR, c = idx / JR, gr = r0 + rr;
      TS v = czero<TS>();
      if (gr < r_end && col[c] >= 0) v = X[gr + ldx * col[c]];
      Xs[rr][c] = v;
    }
    __syncthreads();
    if (gi >= 0) {
      const int lim = min(JR, r_end - r0);
      for (int rr = 0; rr < lim; rr++) cfma_conj(acc, ccast<CG>(Xs[rr][gi]), ccast<CG>(Xs[rr][gj]));
    }
    __syncthreads();
  }
  double2* out = parts + ((size_t)pair * gridDim.y + chunk) * NGRAM;
  if (gi >= 0) {
    out[gi * JC + gj] = ccast<double2>(acc);
    out[gj * JC + gi] = cconj(ccast<double2>(acc));
  }
}

template <typename TS>
__device__ void apply_rows(TS* __restrict__ M, int64_t ld, int r_begin, int r_end, const int* col,
                           const typename cplx_of<typename real_of<TS>::type>::type (*Wt)[JC + 1],
                           TS (*Xs)[JC + 1]) {
  typedef typename real_of<TS>::type RS;
  typedef typename cplx_of<RS>::type CS;
  const int t = threadIdx.x;
  for (int r0 = r_begin; r0 < r_end; r0 += JR) {
    for (int idx = t; idx < JR * JC; idx += NT) {
      const int rr = idx % JR, c = idx / JR, gr = r0 + rr;
      TS v = czero<TS>();
      if (gr < r_end && col[c] >= 0) v = M[gr + ld * col[c]];
      Xs[rr][c] = v;
    }
    __syncthreads();
    for (int idx = t; idx < JR * JC; idx += NT) {
      const int c = idx % JC, rr = idx / JC, gr = r0 + rr;
      if (gr >= r_end || col[c] < 0) continue;
      CS acc = czero<CS>();
#pragma unroll
      for (int k = 0; k < JC; k++) cfma(acc, ccast<CS>(Xs[rr][k]), Wt[k][c]);
      M[gr + ld * col[c]] = ccast<TS>(acc);
    }
    __syncthreads();
  }
}

// Shared state of the 16x16 pair diagonalisation: the Gram and the rotation
// angles in FP64 (the relative accuracy of the small columns lives in the
// Gram's small entries, which an FP32 update would swamp with the rounding
// of the large ones); the accumulated unitary W in RW (the storage
// precision, in which it is applied).
template <typename RW>
struct pair_eig_shared {
  typedef typename cplx_of<RW>::type CW;
  double2 G[JC][JC + 1];  // the pair's Gram, driven to diagonal
  CW W[JC][JC + 1];       // accumulated unitary
  int rp[JC / 2], rq[JC / 2], ron[JC / 2];
  double rc[JC / 2], rt[JC / 2], ra[JC / 2], rb[JC / 2];
  double2 rse[JC / 2];    // s e^{i phi}
  int inner_rot;
};

// Cyclic two-sided Jacobi on sh.G (Hermitian 16x16, every thread of the CTA
// calls it), W accumulating the rotations.  Each 2x2 rotation uses the
// relative-accuracy formula: tan from zeta = (beta-alpha)/(2|gamma|), the
// smaller root.  Columns with |x|^2 <= nu2 are at the rounding level of X and
// are neither rotated nor tested.
template <typename RW>
__device__ int diagonalise_pair(pair_eig_shared<RW>& sh, const int* col, double tol_inner, double nu2) {
  typedef typename cplx_of<RW>::type CW;
  const int t = threadIdx.x;
  int sweep = 0;
  for (; sweep < MAX_INNER; sweep++) {
    __syncthreads();  // every thread has read inner_rot of the previous sweep
    if (t == 0) sh.inner_rot = 0;
    __syncthreads();
    for (int ir = 0; ir < JC - 1; ir++) {
      if (t < JC / 2) {
        int p, q;
        tournament(ir, t, JC, p, q);
        sh.rp[t] = p; sh.rq[t] = q; sh.ron[t] = 0;
        if (col[p] >= 0 && col[q] >= 0) {
          // the running diagonal is clamped at zero (see the update below)
          const double a = fmax(sh.G[p][p].x, 0.0), b = fmax(sh.G[q][q].x, 0.0);
          const double2 g = sh.G[p][q];
          const double ag = sqrt(cabs2(g));
          if (a > nu2 && b > nu2 && ag > tol_inner * sqrt(a * b)) {
            const double zeta = (b - a) / (2.0 * ag);
            const double tt = copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
            const double c = 1.0 / sqrt(1.0 + tt * tt);
            const double sa = c * tt / ag;  // s / |gamma|: s e^{i phi} = sa * gamma
            sh.ron[t] = 1; sh.rc[t] = c; sh.rt[t] = tt * ag; sh.ra[t] = a; sh.rb[t] = b;
            sh.rse[t] = make_double2(sa * g.x, sa * g.y);
            sh.inner_rot = 1;
          }
        }
      }
      __syncthreads();
      // columns p, q of G and W:  [x_p, x_q] <- [c x_p - conj(se) x_q,  se x_p + c x_q]
      {
        const int task = t & 127, k = task >> 4, r = task & 15;
        if (sh.ron[k]) {
          const int p = sh.rp[k], q = sh.rq[k];
          const double c = sh.rc[k];
          const double2 se = sh.rse[k];
          if (t < 128) {
            const double2 xp = sh.G[r][p], xq = sh.G[r][q];
            sh.G[r][p] = csub(cscale(xp, c), cmul(cconj(se), xq));
            sh.G[r][q] = cadd(cmul(se, xp), cscale(xq, c));
          } else {
            const CW cw = ccast<CW>(make_double2(c, 0.0));
            const CW sew = ccast<CW>(se);
            const CW xp = sh.W[r][p], xq = sh.W[r][q];
            sh.W[r][p] = csub(cmul(cw, xp), cmul(cconj(sew), xq));
            sh.W[r][q] = cadd(cmul(sew, xp), cmul(cw, xq));
          }
        }
      }
      __syncthreads();
      // rows p, q of G:  [g_p; g_q] <- [c g_p - se g_q;  conj(se) g_p + c g_q]
      if (t < 128) {
        const int k = t >> 4, r = t & 15;
        if (sh.ron[k]) {
          const int p = sh.rp[k], q = sh.rq[k];
          const double c = sh.rc[k];
          const double2 se = sh.rse[k];
          const double2 gp = sh.G[p][r], gq = sh.G[q][r];
          sh.G[p][r] = csub(cscale(gp, c), cmul(se, gq));
          sh.G[q][r] = cadd(cmul(cconj(se), gp), cscale(gq, c));
        }
      }
      __syncthreads();
      if (t < JC / 2 && sh.ron[t]) {
        // The rotated 2x2 block is diag(alpha - t|gamma|, beta + t|gamma|).
        // For nearly parallel columns of very different norms alpha - t|gamma|
        // cancels and can round below zero; it is clamped at zero so no NaN
        // reaches a later comparison (the next outer sweep recomputes the
        // Gram from the rotated vectors themselves).
        const int p = sh.rp[t], q = sh.rq[t];
        sh.G[p][q] = make_double2(0, 0);
        sh.G[q][p] = make_double2(0, 0);
        sh.G[p][p] = make_double2(fmax(sh.ra[t] - sh.rt[t], 0.0), 0);
        sh.G[q][q] = make_double2(sh.rb[t] + sh.rt[t], 0);
      }
      __syncthreads();
    }
    const int again = sh.inner_rot;  // read after the round's closing barrier
    if (!again) break;
  }
  __syncthreads();
  return sweep + (sweep < MAX_INNER ? 1 : 0);
}

// FP32 variant for FP32 storage: the two-sided Jacobi runs on the scaled
// Gram Ghat = D^{-1/2} G D^{-1/2} (unit diagonal, off-diagonals are the
// cosines between columns) with the diagonal D tracked separately.  The
// cosines are O(1) numbers, so FP32 keeps each one accurate to ~u of its
// own pair whatever the spread of the column norms -- the property the
// unscaled FP32 Gram loses.  A rotation J of pair (p, q) acts on Ghat
// through Jt = D^{1/2} J D'^{-1/2}: Jt_pp = c sqrt(a/a'),
// Jt_qp = -s e^{-i phi} sqrt(b/a'), Jt_pq = s e^{i phi} sqrt(a/b'),
// Jt_qq = c sqrt(b/b'), with a' = a - t|gamma|, b' = b + t|gamma|.
// The unitary is accumulated in the same scaled form, Wt = D0^{1/2} W D^{-1/2}
// (D0 the initial diagonal): its entries are O(1), so their FP32 rounding is
// relative to each output column's own norm once W = D0^{-1/2} Wt D^{1/2} is
// formed -- small columns are not contaminated by the rounding of large ones.
struct pair_eig_scaled {
  float d[JC];            // current diagonal of G
  float d0[JC];           // initial diagonal
  float2 G[JC][JC + 1];   // scaled Gram (diagonal implicit 1)
  float2 W[JC][JC + 1];   // scaled unitary Wt, then W
  int rp[JC / 2], rq[JC / 2], ron[JC / 2];
  float na[JC / 2], nb[JC / 2], kpp[JC / 2], kqq[JC / 2];
  float2 kqp[JC / 2], kpq[JC / 2];
  int inner_rot;
};

// The scaled iteration with one update phase per round: the 16 indices form
// 8 disjoint pairs, so every entry of Jt^H Ghat Jt is a 2x2 combination of
// old entries -- G'[x][y] = sum_{a in {x,x'}} sum_{b in {y,y'}} conj(Jt[a][x])
// Ghat[a][b] Jt[b][y] (x' the partner of x, Jt = I on a pair that does not
// rotate) -- and every entry of Wt Jt a combination of two.  Thread t < 256
// owns entry (t / 16, t % 16) of both; the new values go to the other
// buffer, so a round costs two barriers (parameters, update).  Every thread
// of the block calls it (the barriers are block-wide).
struct pair_eig_scaled2 {
  float d[2][JC];
  float d0[JC];
  float2 G[2][JC][JC + 1];
  float2 W[2][JC][JC + 1];
  int partner[JC];          // partner index of each index in this round
  float2 jt[JC][2];         // Jt[x][x] (real in .x) and Jt[x'][x] for column x
  int inner_rot;
};

__device__ int diagonalise_scaled2(pair_eig_scaled2& sh, const int* col, float tol_inner, float nu2, int max_inner,
                                   int* buf_out) {
  const int t = threadIdx.x, x = (t >> 4) & 15, y = t & 15;
  const bool owner = t < NGRAM;
  int cur = 0, sweep = 0;
  // inner_rot holds the number (1-based) of the last sweep that rotated; the
  // caller zeroes it before the first call
  for (; sweep < max_inner; sweep++) {
    for (int ir = 0; ir < JC - 1; ir++) {
      if (t < JC / 2) {
        int p, q;
        tournament(ir, t, JC, p, q);
        sh.partner[p] = q; sh.partner[q] = p;
        const float a = sh.d[cur][p], b = sh.d[cur][q];
        const float2 gs = sh.G[cur][p][q];
        const float ags = sqrtf(gs.x * gs.x + gs.y * gs.y);
        float2 jpp = make_float2(1.f, 0.f), jqp = make_float2(0.f, 0.f), jpq = jqp, jqq = jpp;
        float a2 = a, b2 = b;
        if (col[p] >= 0 && col[q] >= 0 && a > nu2 && b > nu2 && ags > tol_inner) {
          const float ag = ags * sqrtf(a * b);  // |gamma|
          const float zeta = __fdividef(b - a, 2.f * ag);
          const float r1 = sqrtf(fmaf(zeta, zeta, 1.f));
          const float tt = copysignf(__frcp_rn(fabsf(zeta) + r1), zeta);
          const float c = rsqrtf(fmaf(tt, tt, 1.f)), sn = c * tt;
          const float inv = __frcp_rn(ags);
          const float2 e = make_float2(gs.x * inv, gs.y * inv);
          a2 = fmaxf(a - tt * ag, nu2);  // a column driven to the noise level is frozen
          b2 = b + tt * ag;
          const float ia2 = rsqrtf(a2), ib2 = rsqrtf(b2), sqa = sqrtf(a), sqb = sqrtf(b);
          jpp = make_float2(c * sqa * ia2, 0.f);
          jqp = make_float2(-sn * e.x * sqb * ia2, sn * e.y * sqb * ia2);  // -s conj(e) sqrt(b/a')
          jpq = make_float2(sn * e.x * sqa * ib2, sn * e.y * sqa * ib2);   //  s e sqrt(a/b')
          jqq = make_float2(c * sqb * ib2, 0.f);
          sh.inner_rot = sweep + 1;
        }
        // column p of Jt: rows p (jpp) and q (jqp); column q: rows q (jqq) and p (jpq)
        sh.jt[p][0] = jpp; sh.jt[p][1] = jqp;
        sh.jt[q][0] = jqq; sh.jt[q][1] = jpq;
        sh.d[cur ^ 1][p] = a2; sh.d[cur ^ 1][q] = b2;
      }
      __syncthreads();
      if (owner) {
        const int xp = sh.partner[x], yp = sh.partner[y];
        const float2 jxx = sh.jt[x][0], jpx = sh.jt[x][1];  // Jt[x][x], Jt[x'][x]
        const float2 jyy = sh.jt[y][0], jpy = sh.jt[y][1];  // Jt[y][y], Jt[y'][y]
        // Ghat: diagonal implicit 1; the off-diagonal of a rotated pair is
        // zero, that of a pair left alone keeps its (sub-tolerance) value
        float2 gnew = make_float2(0.f, 0.f);
        if (xp == y && x != y) {
          const bool rotated = jxx.x != 1.f || jxx.y != 0.f || jpx.x != 0.f || jpx.y != 0.f;
          if (!rotated) gnew = sh.G[cur][x][y];
        } else if (x != y) {
          const float2 g_xy = sh.G[cur][x][y], g_xq = sh.G[cur][x][yp];
          const float2 g_py = sh.G[cur][xp][y], g_pq = sh.G[cur][xp][yp];
          // column step: h_a = G[a][y] Jt[y][y] + G[a][y'] Jt[y'][y] for a in {x, x'}
          const float2 hx = cadd(cmul(g_xy, jyy), cmul(g_xq, jpy));
          const float2 hp = cadd(cmul(g_py, jyy), cmul(g_pq, jpy));
          // row step: conj(Jt[x][x]) h_x + conj(Jt[x'][x]) h_x'
          gnew = cadd(cmul(cconj(jxx), hx), cmul(cconj(jpx), hp));
        }
        sh.G[cur ^ 1][x][y] = gnew;
        // Wt Jt: column y
        const float2 w_xy = sh.W[cur][x][y], w_xq = sh.W[cur][x][yp];
        sh.W[cur ^ 1][x][y] = cadd(cmul(w_xy, jyy), cmul(w_xq, jpy));
      }
      cur ^= 1;
      __syncthreads();
    }
    const int again = sh.inner_rot == sweep + 1;  // written before the round's closing barrier
    __syncthreads();  // every thread has read it before the next sweep may write it again
    if (!again) break;
  }
  // W = D0^{-1/2} Wt D^{1/2}
  if (owner) {
    const float d0 = sh.d0[x];
    sh.W[cur][x][y] = d0 > 0.f ? cscale(sh.W[cur][x][y], sqrtf(sh.d[cur][y] / d0))
                               : make_float2(x == y ? 1.f : 0.f, 0.f);
  }
  __syncthreads();
  *buf_out = cur;
  return sweep + (sweep < max_inner ? 1 : 0);
}

// The same iteration run by one warp (lanes 0-31 of the calling CTA; the
// other warps skip it and wait at the caller's barrier): the per-round
// barriers become __syncwarp, and the idle warps leave the SM's issue slots
// to the other CTAs resident on it.  Rotation parameters are computed by
// lanes 0-7 (one pair each) and kept in shared memory; the column updates
// (256 row tasks over G and Wt) and row updates (128) are spread over the
// 32 lanes.
__device__ int diagonalise_scaled_warp(pair_eig_scaled& sh, const int* col, float tol_inner, float nu2,
                                       int max_inner) {
  const int lane = threadIdx.x & 31;
  int sweep = 0;
  for (; sweep < max_inner; sweep++) {
    int rotated = 0;
    for (int ir = 0; ir < JC - 1; ir++) {
      int on = 0;
      if (lane < JC / 2) {
        int p, q;
        tournament(ir, lane, JC, p, q);
        sh.rp[lane] = p; sh.rq[lane] = q;
        const float a = sh.d[p], b = sh.d[q];
        const float2 gs = sh.G[p][q];
        const float ags = sqrtf(gs.x * gs.x + gs.y * gs.y);
        if (col[p] >= 0 && col[q] >= 0 && a > nu2 && b > nu2 && ags > tol_inner) {
          const float ag = ags * sqrtf(a * b);  // |gamma|
          const float zeta = __fdividef(b - a, 2.f * ag);
          const float r1 = sqrtf(fmaf(zeta, zeta, 1.f));
          const float tt = copysignf(__frcp_rn(fabsf(zeta) + r1), zeta);
          const float c = rsqrtf(fmaf(tt, tt, 1.f)), sn = c * tt;
          const float inv = __frcp_rn(ags);
          const float2 e = make_float2(gs.x * inv, gs.y * inv);
          const float a2 = fmaxf(a - tt * ag, nu2), b2 = b + tt * ag;
          const float ia2 = rsqrtf(a2), ib2 = rsqrtf(b2), sqa = sqrtf(a), sqb = sqrtf(b);
          sh.na[lane] = a2; sh.nb[lane] = b2;
          sh.kpp[lane] = c * sqa * ia2;
          sh.kqp[lane] = make_float2(-sn * e.x * sqb * ia2, sn * e.y * sqb * ia2);
          sh.kpq[lane] = make_float2(sn * e.x * sqa * ib2, sn * e.y * sqa * ib2);
          sh.kqq[lane] = c * sqb * ib2;
          on = 1;
        }
        sh.ron[lane] = on;
      }
      rotated |= __any_sync(0xffffffffu, on);
      __syncwarp();
      // columns p, q: tasks (matrix, pair k, row r) = lane + 32 i
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int task = lane + 32 * i, mat = task >> 7, k = (task >> 4) & 7, r = task & 15;
        if (!sh.ron[k]) continue;
        const int p = sh.rp[k], q = sh.rq[k];
        if (mat == 0 && (r == p || r == q)) continue;
        float2 (*M)[JC + 1] = mat == 0 ? sh.G : sh.W;
        const float2 xp = M[r][p], xq = M[r][q];
        M[r][p] = cadd(cscale(xp, sh.kpp[k]), cmul(sh.kqp[k], xq));
        M[r][q] = cadd(cmul(sh.kpq[k], xp), cscale(xq, sh.kqq[k]));
      }
      __syncwarp();
      // rows p, q of Ghat; the pair's own 2x2 block and diagonal
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int task = lane + 32 * i, k = task >> 4, r = task & 15;
        if (!sh.ron[k]) continue;
        const int p = sh.rp[k], q = sh.rq[k];
        if (r != p && r != q) {
          const float2 gp = sh.G[p][r], gq = sh.G[q][r];
          sh.G[p][r] = cadd(cscale(gp, sh.kpp[k]), cmul(cconj(sh.kqp[k]), gq));
          sh.G[q][r] = cadd(cmul(cconj(sh.kpq[k]), gp), cscale(gq, sh.kqq[k]));
        } else if (r == p) {
          sh.G[p][q] = make_float2(0.f, 0.f);
          sh.G[q][p] = make_float2(0.f, 0.f);
          sh.d[p] = sh.na[k];
          sh.d[q] = sh.nb[k];
        }
      }
      __syncwarp();
    }
    if (!rotated) break;
  }
  // W = D0^{-1/2} Wt D^{1/2}
  for (int e = lane; e < NGRAM; e += 32) {
    const int i = e >> 4, j = e & 15;
    const float d0 = sh.d0[i];
    sh.W[i][j] = d0 > 0.f ? cscale(sh.W[i][j], sqrtf(sh.d[j] / d0)) : make_float2(i == j ? 1.f : 0.f, 0.f);
  }
  __syncwarp();
  return sweep + (sweep < max_inner ? 1 : 0);
}

// One CTA per block pair: sum the partial Grams, test the pair, and when it
// needs rotating diagonalise its 16x16 Gram; the unitary goes to wout[pair]
// and the decision to rot[pair] (the apply kernel reads both).
__global__ void __launch_bounds__(NT)
eig_kernel(int nn, int nb, int round, int nparts, const double2* __restrict__ parts, double tol, double nu_rel2,
           const double* __restrict__ xnorm2, double2* __restrict__ wout, int* __restrict__ rot,
           int* __restrict__ flags) {
  __shared__ pair_eig_shared<double> sh;
  __shared__ int col[JC];
  __shared__ int any_rot, bad, offmax_blk, offbig_blk;

  const int t = threadIdx.x;
  const int pair = blockIdx.x;
  const double nu2 = nu_rel2 * (*xnorm2);
  pair_columns(round, pair, nb, nn, col);
  if (t == 0) { any_rot = 0; bad = 0; offmax_blk = 0; offbig_blk = 0; }
  __syncthreads();
  // sum the partial Grams of this pair in a fixed order
  for (int e = t; e < NGRAM; e += NT) {
    double2 s = make_double2(0, 0);
    for (int c = 0; c < nparts; c++) s = cadd(s, parts[((size_t)pair * nparts + c) * NGRAM + e]);
    sh.G[e / JC][e % JC] = s;
    sh.W[e / JC][e % JC] = make_double2((e / JC) == (e % JC) ? 1.0 : 0.0, 0.0);
    if (!isfinite(s.x) || !isfinite(s.y)) bad = 1;
  }
  __syncthreads();
  if (bad) {
    if (t == 0) {
      atomicOr(&flags[QT_FLAG_NONFINITE], 1);
      rot[pair] = 0;
    }
    return;
  }
  // is this pair already orthogonal to tol?  (the largest relative
  // off-diagonal above tol is recorded as float bits, one atomic per pair)
  float relmax = 0.f, relbig = 0.f;
  const double big2 = 1e-6 * (*xnorm2);
  for (int e = t; e < NGRAM; e += NT) {
    const int i = e / JC, j = e % JC;
    if (i < j && col[i] >= 0 && col[j] >= 0) {
      const double a = sh.G[i][i].x, b = sh.G[j][j].x;
      const double g = sqrt(cabs2(sh.G[i][j]));
      if (a > nu2 && b > nu2 && g > tol * sqrt(a * b)) {
        any_rot = 1;
        const float rel = (a > 0 && b > 0) ? (float)fmin(g / sqrt(a * b), 1.0) : 1.0f;
        relmax = fmaxf(relmax, rel);
        if (a > big2 && b > big2) relbig = fmaxf(relbig, rel);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    relmax = fmaxf(relmax, __shfl_xor_sync(0xffffffffu, relmax, o));
    relbig = fmaxf(relbig, __shfl_xor_sync(0xffffffffu, relbig, o));
  }
  if ((t & 31) == 0 && relmax > 0.f) atomicMax(&offmax_blk, __float_as_int(relmax));
  if ((t & 31) == 0 && relbig > 0.f) atomicMax(&offbig_blk, __float_as_int(relbig));
  __syncthreads();
  if (t == 0 && offmax_blk > 0) atomicMax(&flags[QT_FLAG_OFFMAX], offmax_blk);
  if (t == 0 && offbig_blk > 0) atomicMax(&flags[QT_FLAG_OFFBIG], offbig_blk);
  __syncthreads();
  if (t == 0) rot[pair] = any_rot;
  if (!any_rot) return;
  if (t == 0) atomicAdd(&flags[QT_FLAG_ROTATED], 1);
  // diagonalised well below the outer threshold so that the rounding of the
  // applied rotation (in the storage precision) cannot leave the pair just
  // above `tol`
  const int inner = diagonalise_pair<double>(sh, col, fmin(tol, 1e-14), nu2);
  if (t == 0) atomicAdd(&flags[QT_FLAG_INNER], inner);
  for (int e = t; e < NGRAM; e += NT) wout[(size_t)pair * NGRAM + e] = sh.W[e / JC][e % JC];
}

// out[r, col[c]] = sum_k Xs[k*lds + r] W[k][c] for r < nrows: each thread a
// 4-row x 4-column tile (rows lane + 32 i, columns 4 cq + j), so one shared
// load of X feeds four complex FMAs and the global stores run along rows.
template <typename TS>
__device__ void rotate_rows(const TS* __restrict__ Xs, int lds, int nrows, TS* __restrict__ out, int64_t ld,
                            const int* col, const TS (*W)[JC + 1]) {
  const int t = threadIdx.x, lane = t & 31, cq = (t >> 5) & 3, rg = t >> 7;
  for (int r0 = rg * 128; r0 < nrows; r0 += 256) {
    TS acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = czero<TS>();
#pragma unroll 4
    for (int k = 0; k < JC; k++) {
      TS w[4], x[4];
#pragma unroll
      for (int j = 0; j < 4; j++) w[j] = W[k][cq * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = r0 + lane + 32 * i;
        x[i] = (r < nrows) ? Xs[k * lds + r] : czero<TS>();
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) cfma(acc[i][j], x[i], w[j]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int r = r0 + lane + 32 * i;
      if (r >= nrows) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int c = col[cq * 4 + j];
        if (c >= 0) out[r + ld * c] = acc[i][j];
      }
    }
  }
}

// rows [0, nrows) of the pair's columns of M -> Xs (column c at Xs + c*lds).
// Thread t copies rows t, t + NT, ...: for each row it issues the 16 column
// loads back to back (independent, coalesced across the warp) before storing.
template <typename TS>
__device__ void stage_rows(const TS* __restrict__ M, int64_t ld, int nrows, int rows_alloc, const int* col,
                           TS* __restrict__ Xs, int lds) {
  for (int rr = threadIdx.x; rr < rows_alloc; rr += NT) {
    TS v[JC];
#pragma unroll
    for (int c = 0; c < JC; c++) v[c] = (rr < nrows && col[c] >= 0) ? M[rr + ld * col[c]] : czero<TS>();
#pragma unroll
    for (int c = 0; c < JC; c++) Xs[c * lds + rr] = v[c];
  }
}

// One round of the sweep in one launch.  A thread-block cluster of `csize`
// CTAs owns one block pair; CTA q of the cluster holds rows
// [q*xrows_c, (q+1)*xrows_c) of the pair's 16 columns of X in shared memory.
// Each CTA forms its partial Gram (accumulated in the storage precision: each
// entry is then accurate relative to its own column norms), the partials are
// summed in FP64 over the cluster through distributed shared memory in rank
// order, CTA 0 of the cluster tests the pair and diagonalises the Gram, the
// other CTAs copy its unitary through distributed shared memory, and every
// CTA rotates its own rows of X and its share of the rows of V.
__global__ void __launch_bounds__(NT)
pair_round_kernel(float2* __restrict__ X, int64_t ldx, int mm, float2* __restrict__ V, int64_t ldv, int nn, int nb, int round,
                  int csize, int xrows_c, int vrows_c, int lds, double tol, double tol_inner, double nu_rel2,
                  const double* __restrict__ xnorm2, int* __restrict__ flags, int max_inner,
                  unsigned long long* __restrict__ phase_ns) {
  typedef float2 TS;
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  TS* Xs = reinterpret_cast<TS*>(dyn_smem);
  __shared__ pair_eig_scaled sh;
  __shared__ TS gpart[NGRAM];
  __shared__ int col[JC];
  __shared__ int any_rot, bad, offmax_blk, offbig_blk;
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const int pair = blockIdx.x / csize;
  const int t = threadIdx.x;
  // optional phase timing (diagnostics): thread 0 of each CTA adds the time
  // spent in each phase to phase_ns[8 * (crank != 0) + phase]
  unsigned long long tp = 0;
  auto phase = [&](int ph) {
    if (phase_ns && t == 0) {
      unsigned long long tn;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tn));
      if (ph > 0) atomicAdd(&phase_ns[8 * (crank != 0) + ph - 1], tn - tp);
      tp = tn;
    }
  };
  phase(0);
  pair_columns(round, pair, nb, nn, col);
  if (t == 0) { any_rot = 0; bad = 0; offmax_blk = 0; offbig_blk = 0; }
  __syncthreads();
  const int xb = crank * xrows_c;
  const int xr = max(0, min(mm, xb + xrows_c) - xb);
  stage_rows<TS>(X + xb, ldx, xr, xrows_c, col, Xs, lds);
  __syncthreads();
  phase(1);  // 0: stage
  // partial Gram over this CTA's rows: the 36 upper 2x2 tiles of the 16x16
  // Gram, four threads per tile on interleaved rows (four independent
  // complex accumulators each), reduced with shuffles in a fixed order
  if (t < 160) {
    const int tile = t >> 2, g = t & 3;
    const bool act = tile < 36;
    int bi = 0, rem = act ? tile : 0;
    while (rem >= 8 - bi) { rem -= 8 - bi; bi++; }
    const int bj = bi + rem;
    const TS* x0 = Xs + (2 * bi) * lds;
    const TS* x1 = x0 + lds;
    const TS* y0 = Xs + (2 * bj) * lds;
    const TS* y1 = y0 + lds;
    TS a00 = czero<TS>(), a01 = czero<TS>(), a10 = czero<TS>(), a11 = czero<TS>();
    if (act) {
      for (int rr = g; rr < xr; rr += 4) {
        const TS p0 = x0[rr], p1 = x1[rr], q0 = y0[rr], q1 = y1[rr];
        cfma_conj(a00, p0, q0);
        cfma_conj(a01, p0, q1);
        cfma_conj(a10, p1, q0);
        cfma_conj(a11, p1, q1);
      }
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      a00.x += __shfl_xor_sync(0xffffffffu, a00.x, o); a00.y += __shfl_xor_sync(0xffffffffu, a00.y, o);
      a01.x += __shfl_xor_sync(0xffffffffu, a01.x, o); a01.y += __shfl_xor_sync(0xffffffffu, a01.y, o);
      a10.x += __shfl_xor_sync(0xffffffffu, a10.x, o); a10.y += __shfl_xor_sync(0xffffffffu, a10.y, o);
      a11.x += __shfl_xor_sync(0xffffffffu, a11.x, o); a11.y += __shfl_xor_sync(0xffffffffu, a11.y, o);
    }
    if (act && g == 0) {
      const int i0 = 2 * bi, j0 = 2 * bj;
      gpart[i0 * JC + j0] = a00;             gpart[j0 * JC + i0] = cconj(a00);
      gpart[(i0 + 1) * JC + j0 + 1] = a11;   gpart[(j0 + 1) * JC + i0 + 1] = cconj(a11);
      gpart[i0 * JC + j0 + 1] = a01;         gpart[(j0 + 1) * JC + i0] = cconj(a01);
      if (bi != bj) { gpart[(i0 + 1) * JC + j0] = a10; gpart[j0 * JC + i0 + 1] = cconj(a10); }
    }
  }
  __syncthreads();
  phase(2);  // 1: Gram
  cluster.sync();
  phase(3);  // 2: first cluster barrier
  const double nu2 = nu_rel2 * (*xnorm2);
  if (crank == 0) {
    // FP64 sums of the partials in rank order; the remote loads are issued
    // together (independent) before the sum
    double2 sum_e;
    {
      const int e = t;  // NT == NGRAM: one Gram entry per thread
      TS v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = q < csize ? cluster.map_shared_rank(gpart, q)[e] : czero<TS>();
      sum_e = make_double2(0, 0);
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (q < csize) sum_e = cadd(sum_e, ccast<double2>(v[q]));
      if (!isfinite(sum_e.x) || !isfinite(sum_e.y)) bad = 1;
    }
    __shared__ double dd[JC];
    const int i = t / JC, j = t % JC;
    if (i == j) {
      dd[i] = sum_e.x;
      sh.d[i] = (float)sum_e.x;
      sh.d0[i] = (float)sum_e.x;
    }
    __syncthreads();
    float2 v = make_float2(0.f, 0.f);
    if (i != j && dd[i] > nu2 && dd[j] > nu2) {
      const double sc = 1.0 / sqrt(dd[i] * dd[j]);
      v = make_float2((float)(sum_e.x * sc), (float)(sum_e.y * sc));
    }
    sh.G[i][j] = v;
    sh.W[i][j] = make_float2(i == j ? 1.f : 0.f, 0.f);
  }
  cluster.sync();  // the partials have been read: CTAs 1.. may leave or move on
  phase(4);  // 3: partial sums + second barrier
  if (crank == 0) {
    // is this pair already orthogonal to tol?  (the largest relative
    // off-diagonal above tol is recorded as float bits)
    if (!bad) {
      // the largest relative off-diagonal above tol: a block maximum first,
      // then one global atomic per pair (thousands of same-address atomics
      // per round would serialise in L2)
      float relmax = 0.f, relbig = 0.f;
      const double big2 = 1e-6 * (*xnorm2);
      for (int e = t; e < NGRAM; e += NT) {
        const int i = e / JC, j = e % JC;
        if (i < j && col[i] >= 0 && col[j] >= 0) {
          double rel = 0, a, b;
          bool live;
          a = sh.d[i]; b = sh.d[j];
          rel = sqrt((double)cabs2(sh.G[i][j]));
          live = a > nu2 && b > nu2;
          if (live && rel > tol) {
            any_rot = 1;
            relmax = fmaxf(relmax, (float)fmin(rel, 1.0));
            if (a > big2 && b > big2) relbig = fmaxf(relbig, (float)fmin(rel, 1.0));
          }
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        relmax = fmaxf(relmax, __shfl_xor_sync(0xffffffffu, relmax, o));
        relbig = fmaxf(relbig, __shfl_xor_sync(0xffffffffu, relbig, o));
      }
      if ((t & 31) == 0 && relmax > 0.f) atomicMax(&offmax_blk, __float_as_int(relmax));
      if ((t & 31) == 0 && relbig > 0.f) atomicMax(&offbig_blk, __float_as_int(relbig));
      __syncthreads();
      if (t == 0 && offmax_blk > 0) atomicMax(&flags[QT_FLAG_OFFMAX], offmax_blk);
      if (t == 0 && offbig_blk > 0) atomicMax(&flags[QT_FLAG_OFFBIG], offbig_blk);
    } else if (t == 0) {
      atomicOr(&flags[QT_FLAG_NONFINITE], 1);
    }
    __syncthreads();
    if (any_rot) {
      if (t == 0) atomicAdd(&flags[QT_FLAG_ROTATED], 1);
      int inner = 0;
      if (t < 32) inner = diagonalise_scaled_warp(sh, col, (float)tol_inner, (float)nu2, max_inner);
      __syncthreads();
      if (t == 0) atomicAdd(&flags[QT_FLAG_INNER], inner);
    }
  }
  __syncthreads();
  phase(5);  // 4: test + pair solver (CTA 0)
  cluster.sync();  // CTA 0's decision and unitary are ready
  if (crank != 0) {
    if (t == 0) any_rot = *cluster.map_shared_rank(&any_rot, 0);
    for (int e = t; e < NGRAM; e += NT) sh.W[e / JC][e % JC] = cluster.map_shared_rank(&sh.W[0][0], 0)[(e / JC) * (JC + 1) + e % JC];
  }
  cluster.sync();  // CTA 0 stays resident until every copy is done
  phase(6);  // 5: third/fourth barrier + unitary copy
  if (!any_rot) return;  // the same decision in every CTA of the cluster
  rotate_rows<TS>(Xs, lds, xr, X + xb, ldx, col, sh.W);
  __syncthreads();
  phase(7);  // 6: rotate X
  __syncthreads();  // Xs is reused for V
  if (V == nullptr) return;  // no accumulated rotations wanted
  const int vb = crank * vrows_c;
  const int vr = max(0, min(nn, vb + vrows_c) - vb);
  stage_rows<TS>(V + vb, ldv, vr, vrows_c, col, Xs, lds);
  __syncthreads();
  rotate_rows<TS>(Xs, lds, vr, V + vb, ldv, col, sh.W);
}

// ---------------------------------------------------------------------------
// FP64 storage: one launch per round, a cluster per pair
// ---------------------------------------------------------------------------
//
// An SM has two FP64 lanes, so a warp instruction in FP64 occupies it for 16
// cycles; what the round costs is FP64 instructions per SM and the latency of
// the pair solver.
//  - The pair's rows are spread over as many CTAs as the chip holds at once
//    (clusters of up to 8, at least 8 rows each): Gram products and rotation
//    are FP64 and shrink with the rows.
//  - The rotation angles come from an FP32 two-sided Jacobi on the scaled Gram
//    (cosines, each accurate relative to its own pair) with the diagonal kept
//    as an FP32 pair (2^-48: the difference of nearly equal norms decides the
//    angle).  Any angle gives a unitary rotation; one that is 1e-7 off leaves
//    1e-7 of the pair's off-diagonal, which the next sweep measures from the
//    FP64 columns again, so the iteration ends as with FP64 angles, at the
//    same tolerance.  Each rotation (c, s e^{i phi}) is brought to unit length
//    in FP64 and accumulated into the FP64 unitary by four further warps, one
//    inner round behind the solver, while the solver's FP32 chain runs.
//  - Every CTA of the cluster sums the partial Grams in rank order and runs the
//    same solver on the same numbers, so the unitary needs no broadcast: one
//    cluster barrier before the sums, one (split) before a CTA may leave.
// Measured at 128 x 128 with V (8 pairs, clusters of 8; us per round): stage
// 1.3, Gram 2.9, barrier 0.5, sums and test 4.6, solver 16, rotation 7.0 --
// against 310 for one CTA per pair with an FP64 solver (Gram 42, solver 183,
// rotation 25, unspread), and 46.5 -> 9.9 ms for the update of a bond of 64.

constexpr int R64_SOLVE = 256;             // solver threads (warps 0-7)
constexpr int R64_ACC = 128;               // unitary accumulation (warps 8-11)
constexpr int NT64 = R64_SOLVE + R64_ACC;

struct pair_solver64 {
  float dh[2][JC], dl[2][JC];  // squared column norms, unevaluated pairs
  float2 G[2][JC][JC + 1];     // scaled Gram (diagonal implicit 1)
  float4 rot[2][JC];           // posted rotations (c, Re s e, Im s e, on) at the pair's lower index
  int round[2];                // inner round of each post; -1: no more
  double2 W[JC][JC + 1];       // the pair's unitary
};

template <int ID>
__device__ inline void bar_sync(int n) { asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(n) : "memory"); }
template <int ID>
__device__ inline void bar_arrive(int n) { asm volatile("bar.arrive %0, %1;" ::"n"(ID), "r"(n) : "memory"); }
// barriers 2, 3: post b is full; 4, 5: post b is free again
__device__ inline void post_full_arrive(int b) { if (b) bar_arrive<3>(NT64); else bar_arrive<2>(NT64); }
__device__ inline void post_full_wait(int b) { if (b) bar_sync<3>(NT64); else bar_sync<2>(NT64); }
__device__ inline void post_free_arrive(int b) { if (b) bar_arrive<5>(NT64); else bar_arrive<4>(NT64); }
__device__ inline void post_free_wait(int b) { if (b) bar_sync<5>(NT64); else bar_sync<4>(NT64); }
__device__ inline void solver64_sync() { bar_sync<1>(R64_SOLVE); }

// Warps 0-7: thread (x, y) computes the rotation of y's pair, takes x's from
// lane x and updates Ghat[x][y] into the other buffer.  Posts every inner
// round that rotates; the last post says so.
__device__ int solve_pair64(pair_solver64& sh, const int* col, float tol_inner, float nu2, int max_inner) {
  const int t = threadIdx.x, x = (t >> 4) & 15, y = t & 15;
  const float tol2 = tol_inner * tol_inner;
  int cur = 0, sweep = 0, posts = 0;
  for (; sweep < max_inner; sweep++) {
    bool rotated_any = false;
    for (int ir = 0; ir < JC - 1; ir++) {
      const int yp = inner_partner(ir, y), xp = inner_partner(ir, x);
      const int p = min(y, yp), q = max(y, yp);
      const float a = sh.dh[cur][p], b = sh.dh[cur][q], al = sh.dl[cur][p], bl = sh.dl[cur][q];
      const float2 gs = sh.G[cur][p][q];
      const float ags2 = gs.x * gs.x + gs.y * gs.y;
      const bool rotp = col[p] >= 0 && col[q] >= 0 && a > nu2 && b > nu2 && ags2 > tol2;
      if (!__any_sync(0xffffffffu, rotp)) continue;  // the same vote in every solver warp
      rotated_any = true;
      float2 jpp = make_float2(1.f, 0.f), jqp = make_float2(0.f, 0.f), jpq = jqp, jqq = jpp;
      float a2 = a, b2 = b, a2l = al, b2l = bl;
      float4 post = make_float4(1.f, 0.f, 0.f, 0.f);
      if (rotp) {
        const float ria = rsqrtf(a), rib = rsqrtf(b), rags = rsqrtf(ags2);
        const float sqa = a * ria, sqb = b * rib;
        const float ag = ags2 * rags * sqa * sqb;  // |gamma|
        // the leading parts subtract exactly where they are close, and the
        // trailing ones matter only there
        const float diff = __fadd_rn(__fsub_rn(b, a), __fsub_rn(bl, al));
        const float zeta = 0.5f * (diff * ria * rib) * rags;
        const float az = fabsf(zeta);
        // (az^2 would overflow where norms 1e14 apart meet cosines of 1e-13)
        const float tt = copysignf(__fdividef(1.f, az > 1e6f ? 2.f * az : az + sqrtf(fmaf(az, az, 1.f))), zeta);
        const float c = rsqrtf(fmaf(tt, tt, 1.f)), sn = c * tt;
        const float2 e = make_float2(gs.x * rags, gs.y * rags);
        const float d = tt * ag;
        // a - d and b + d as pairs
        {
          const float s = __fsub_rn(a, d), bb = __fsub_rn(s, a);
          const float er = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(-d, bb));
          a2 = __fadd_rn(s, __fadd_rn(er, al));
          a2l = __fsub_rn(__fadd_rn(er, al), __fsub_rn(a2, s));
          if (!(a2 > nu2)) { a2 = nu2; a2l = 0.f; }  // a column driven to the noise level is frozen
        }
        {
          const float s = __fadd_rn(b, d), bb = __fsub_rn(s, b);
          const float er = __fadd_rn(__fsub_rn(b, __fsub_rn(s, bb)), __fsub_rn(d, bb));
          b2 = __fadd_rn(s, __fadd_rn(er, bl));
          b2l = __fsub_rn(__fadd_rn(er, bl), __fsub_rn(b2, s));
        }
        const float ia2 = rsqrtf(a2), ib2 = rsqrtf(b2);
        const float fa = sqa * ia2, fb = sqb * ib2, fab = sqb * ia2, fba = sqa * ib2;
        jpp = make_float2(c * fa, 0.f);
        jqp = make_float2(-sn * e.x * fab, sn * e.y * fab);  // -s conj(e) sqrt(b/a')
        jpq = make_float2(sn * e.x * fba, sn * e.y * fba);   //  s e sqrt(a/b')
        jqq = make_float2(c * fb, 0.f);
        post = make_float4(c, sn * e.x, sn * e.y, 1.f);
      }
      const bool low = y == p;
      // post the round's rotations for the accumulation
      const int pb = posts & 1;
      if (posts >= 2) post_free_wait(pb);
      if (x == 0 && low) sh.rot[pb][p] = post;
      if (t == 0) sh.round[pb] = ir;
      post_full_arrive(pb);
      posts++;
      const float2 jyy = low ? jpp : jqq, jpy = low ? jqp : jpq;
      float2 jxx, jpx;
      jxx.x = __shfl_sync(0xffffffffu, jyy.x, x);
      jxx.y = __shfl_sync(0xffffffffu, jyy.y, x);
      jpx.x = __shfl_sync(0xffffffffu, jpy.x, x);
      jpx.y = __shfl_sync(0xffffffffu, jpy.y, x);
      if (x == y) {
        sh.dh[cur ^ 1][y] = low ? a2 : b2;
        sh.dl[cur ^ 1][y] = low ? a2l : b2l;
      }
      float2 gnew = make_float2(0.f, 0.f);
      if (xp == y && x != y) {
        if (!rotp) gnew = sh.G[cur][x][y];
      } else if (x != y) {
        const float2 g_xy = sh.G[cur][x][y], g_xq = sh.G[cur][x][yp];
        const float2 g_py = sh.G[cur][xp][y], g_pq = sh.G[cur][xp][yp];
        const float2 hx = cadd(cmul(g_xy, jyy), cmul(g_xq, jpy));
        const float2 hp = cadd(cmul(g_py, jyy), cmul(g_pq, jpy));
        gnew = cadd(cmul(cconj(jxx), hx), cmul(cconj(jpx), hp));
      }
      sh.G[cur ^ 1][x][y] = gnew;
      cur ^= 1;
      solver64_sync();
    }
    if (!rotated_any) break;  // every solver warp took the same votes
  }
  const int pb = posts & 1;
  if (posts >= 2) post_free_wait(pb);
  if (t == 0) sh.round[pb] = -1;
  post_full_arrive(pb);
  if (posts >= 1) post_free_wait(pb ^ 1);  // every post was taken: the barriers end even
  return sweep + (sweep < max_inner ? 1 : 0);
}

// Warps 8-11: W <- W J for every posted round.  Warp w holds rows 4 w .. 4 w + 3,
// lane (row, pair); a row stays with its warp.
__device__ void accumulate_pair64(pair_solver64& sh) {
  const int t = threadIdx.x - R64_SOLVE, r = t >> 3, k = t & 7;
  for (int i = 0;; i++) {
    const int pb = i & 1;
    post_full_wait(pb);
    const int ir = sh.round[pb];
    if (ir < 0) return;
    int p, q;
    tournament(ir, k, JC, p, q);
    const float4 v = sh.rot[pb][p];
    if (v.w != 0.f) {
      // |(c, sr, si)|^2 = 1 - d with d ~ 1e-7: times 1 + d/2 + 3 d^2/8, to 1e-21
      double c = v.x, sr = v.y, si = v.z;
      const double d = fma(-si, si, fma(-sr, sr, fma(-c, c, 1.0)));
      const double h = d * fma(0.375, d, 0.5);
      c = fma(h, c, c);
      sr = fma(h, sr, sr);
      si = fma(h, si, si);
      // w_p' = c w_p - conj(se) w_q ;  w_q' = se w_p + c w_q
      const double2 u = sh.W[r][p], w = sh.W[r][q];
      sh.W[r][p] = make_double2(fma(c, u.x, -fma(sr, w.x, si * w.y)), fma(c, u.y, -fma(sr, w.y, -(si * w.x))));
      sh.W[r][q] = make_double2(fma(c, w.x, fma(sr, u.x, -(si * u.y))), fma(c, w.y, fma(sr, u.y, si * u.x)));
    }
    __syncwarp();
    post_free_arrive(pb);
  }
}

// rows [0, nrows) of the pair's columns of M -> Xs (column c at Xs + c * lds)
__device__ inline void stage_rows64(const double2* __restrict__ M, int64_t ld, int nrows, const int* col,
                                    double2* __restrict__ Xs, int lds) {
  for (int idx = threadIdx.x; idx < nrows * JC; idx += NT64) {
    const int r = idx % nrows, c = idx / nrows;
    Xs[c * lds + r] = col[c] >= 0 ? M[r + ld * col[c]] : make_double2(0, 0);
  }
}

// M[r, col[c]] = sum_k Xs[k][r] W[k][c]: one output per thread and turn, lanes
// along the rows (FP64-bound: two shared loads per four FMAs of 16 cycles)
__device__ inline void rotate_rows64(const double2* __restrict__ Xs, int lds, int nrows, double2* __restrict__ M,
                                     int64_t ld, const int* col, const double2 (*W)[JC + 1]) {
  for (int idx = threadIdx.x; idx < nrows * JC; idx += NT64) {
    const int r = idx % nrows, c = idx / nrows;
    if (col[c] < 0) continue;
    double2 acc = make_double2(0, 0);
#pragma unroll
    for (int k = 0; k < JC; k++) cfma(acc, Xs[k * lds + r], W[k][c]);
    M[r + ld * col[c]] = acc;
  }
}

// grid: pairs x csize.  CTA q of a cluster holds rows [q xrows, (q + 1) xrows)
// of the pair's columns of X, and (vboth: staged at the start, beside X) rows
// [q vrows, ...) of V.
__global__ void __launch_bounds__(NT64)
pair_round64_kernel(double2* __restrict__ X, int64_t ldx, int mm, double2* __restrict__ V, int64_t ldv, int nn, int nb,
                    int round, int csize, int xrows, int vrows, int lds, int vboth, double tol, double nu_rel2,
                    const double* __restrict__ xnorm2, int* __restrict__ flags, int max_inner,
                    unsigned long long* __restrict__ phase_ns) {
  extern __shared__ __align__(16) unsigned char dyn_smem[];
  double2* Xs = reinterpret_cast<double2*>(dyn_smem);
  double2* Vs = vboth ? Xs + (size_t)JC * lds : Xs;
  __shared__ pair_solver64 sh;
  __shared__ double2 gpart[JC * (JC + 1)];
  __shared__ int col[JC];
  __shared__ int any_rot, bad, offmax_blk, offbig_blk;
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const int pair = blockIdx.x / csize;
  const int t = threadIdx.x;
  unsigned long long tp = 0;
  auto phase = [&](int ph) {  // optional diagnostics: thread 0's time per phase
    if (phase_ns && t == 0) {
      unsigned long long tn;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tn));
      if (ph > 0) atomicAdd(&phase_ns[8 * (crank != 0) + ph - 1], tn - tp);
      tp = tn;
    }
  };
  phase(0);
  pair_columns(round, pair, nb, nn, col);
  if (t == 0) { any_rot = 0; bad = 0; offmax_blk = 0; offbig_blk = 0; }
  // powers-of-two multiples bring ||X||_F^2 into [1, 2) for the solver
  __shared__ double unit_sh;
  __shared__ float nu2_sh, big2_sh;
  if (t == NT64 - 1) {
    const double xn2 = *xnorm2;
    const double unit = xn2 > 0 && isfinite(xn2) ? ldexp(1.0, -ilogb(xn2)) : 1.0;
    unit_sh = unit;
    nu2_sh = (float)(nu_rel2 * xn2 * unit);
    big2_sh = (float)(1e-6 * xn2 * unit);
  }
  for (int e = t; e < NGRAM; e += NT64) sh.W[e / JC][e % JC] = make_double2(e / JC == e % JC ? 1.0 : 0.0, 0.0);
  __syncthreads();
  const int xb = crank * xrows, xr = max(0, min(mm, xb + xrows) - xb);
  const int vb = crank * vrows, vr = V ? max(0, min(nn, vb + vrows) - vb) : 0;
  stage_rows64(X + xb, ldx, xr, col, Xs, lds);
  if (vboth && vr > 0) stage_rows64(V + vb, ldv, vr, col, Vs, lds);
  __syncthreads();
  phase(1);  // 0: stage
  // partial Gram: one upper entry per thread over every row, two row groups
  // from 32 rows on (FP64-bound: sharing operands between entries would save
  // shared loads that cost nothing here, and its reductions would be FP64 adds)
  constexpr int NU = JC * (JC + 1) / 2;
  int gi = 0, gj = 0;
  const int groups = xr >= 32 ? 2 : 1;
  double2 g_e = make_double2(0, 0);
  if (t < NU * groups) {
    int rem = t % NU;
    while (rem >= JC - gi) { rem -= JC - gi; gi++; }
    gj = gi + rem;
    const double2 *xi = Xs + gi * lds, *xj = Xs + gj * lds;
#pragma unroll 4
    for (int rr = t / NU; rr < xr; rr += groups) cfma_conj(g_e, xi[rr], xj[rr]);
    if (t >= NU) gpart[NU + (t - NU)] = g_e;
  }
  if (groups == 2) __syncthreads();
  if (t < NU) {
    if (groups == 2) g_e = cadd(g_e, gpart[NU + t]);
    gpart[t] = g_e;
  }
  phase(2);  // 1: Gram
  cluster.sync();
  phase(3);  // 2: cluster barrier
  // the upper entries, partials added in rank order
  const double unit = unit_sh;
  const float nu2 = nu2_sh, big2 = big2_sh;
  const bool upper = t < NU;
  if (upper) {
    // all remote loads in flight before the first sum
    double2 v[8];
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (q < csize) v[q] = cluster.map_shared_rank(gpart, q)[t];
    g_e = v[0];
#pragma unroll
    for (int q = 1; q < 8; q++)
      if (q < csize) g_e = cadd(g_e, v[q]);
    if (!isfinite(g_e.x) || !isfinite(g_e.y)) bad = 1;
    if (gi == gj) {
      const double d = fmax(g_e.x * unit, 0.0);
      sh.dh[0][gi] = (float)d;
      sh.dl[0][gi] = (float)(d - (double)(float)d);
    }
  }
  // this CTA has read the partials; it may leave once all have
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  __syncthreads();
  if (upper) {
    float2 v = make_float2(0.f, 0.f);
    const float di = sh.dh[0][gi], dj = sh.dh[0][gj];
    if (gi != gj && di > nu2 && dj > nu2) {
      const double ri = rsqrtf(di), rj = rsqrtf(dj) * unit;
      v = make_float2((float)(g_e.x * ri * rj), (float)(g_e.y * ri * rj));
    }
    sh.G[0][gi][gj] = v;
    sh.G[0][gj][gi] = cconj(v);
    // is this pair already orthogonal to tol?
    if (!bad && gi != gj && col[gi] >= 0 && col[gj] >= 0 && di > nu2 && dj > nu2) {
      const float rel = fminf(sqrtf(cabs2(v)), 1.f);
      if (rel > (float)tol) {
        any_rot = 1;
        atomicMax(&offmax_blk, __float_as_int(rel));
        if (di > big2 && dj > big2) atomicMax(&offbig_blk, __float_as_int(rel));
      }
    }
  }
  __syncthreads();
  phase(4);  // 3: sums, cosines, test
  if (t == 0 && crank == 0) {
    if (bad) atomicOr(&flags[QT_FLAG_NONFINITE], 1);
    if (any_rot) atomicAdd(&flags[QT_FLAG_ROTATED], 1);
    if (offmax_blk > 0) atomicMax(&flags[QT_FLAG_OFFMAX], offmax_blk);
    if (offbig_blk > 0) atomicMax(&flags[QT_FLAG_OFFBIG], offbig_blk);
  }
  if (any_rot) {
    // down to 1e-6 of the pair's largest cosine: FP32 angles reach no further
    const float tol_inner = fmaxf(1e-14f, 1e-6f * __int_as_float(offmax_blk));
    if (t < R64_SOLVE) {
      const int inner = solve_pair64(sh, col, fminf(tol_inner, (float)tol), nu2, max_inner);
      if (t == 0 && crank == 0) atomicAdd(&flags[QT_FLAG_INNER], inner);
    } else {
      accumulate_pair64(sh);
    }
    __syncthreads();
    phase(5);  // 4: pair solver
    rotate_rows64(Xs, lds, xr, X + xb, ldx, col, sh.W);
    if (vr > 0) {
      if (!vboth) {
        __syncthreads();  // Xs is reused for V
        stage_rows64(V + vb, ldv, vr, col, Vs, lds);
        __syncthreads();
      }
      rotate_rows64(Vs, lds, vr, V + vb, ldv, col, sh.W);
    }
    phase(6);  // 5: rotation
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// grid (pair, row chunk): apply the pair's unitary to this chunk's rows of X and V.
template <typename TS>
__global__ void __launch_bounds__(NT)
apply_kernel(TS* __restrict__ X, int64_t ldx, int mm, TS* __restrict__ V, int64_t ldv, int nn, int nb, int round,
             int x_rows_per_chunk, int v_rows_per_chunk, const double2* __restrict__ win, const int* __restrict__ rot) {
  typedef typename real_of<TS>::type RS;
  typedef typename cplx_of<RS>::type CS;
  __shared__ CS Wt[JC][JC + 1];
  __shared__ TS Xs[JR][JC + 1];
  __shared__ int col[JC];
  const int pair = blockIdx.x, chunk = blockIdx.y;
  if (!rot[pair]) return;
  pair_columns(round, pair, nb, nn, col);
  for (int e = threadIdx.x; e < NGRAM; e += NT) Wt[e / JC][e % JC] = ccast<CS>(win[(size_t)pair * NGRAM + e]);
  __syncthreads();
  const int xb = chunk * x_rows_per_chunk, vb = chunk * v_rows_per_chunk;
  apply_rows<TS>(X, ldx, xb, min(mm, xb + x_rows_per_chunk), col, Wt, Xs);
  if (V) apply_rows<TS>(V, ldv, vb, min(nn, vb + v_rows_per_chunk), col, Wt, Xs);
}

// ---------------------------------------------------------------------------
// FP32 storage, two launches per round
// ---------------------------------------------------------------------------

constexpr int SLAB = 256;  // rows per shared-memory slab of the Gram kernel
constexpr int NTG = 512;   // threads of the Gram kernel

// grid = pairs: one CTA of 512 threads forms the whole 16x16 Gram of its pair
// (rows streamed through a 256-row shared-memory slab -- each thread loads
// half a row, the next slab prefetched into registers during the current
// one's products; the 36 upper 2x2 tiles, 14 threads each on interleaved
// rows, FP32 accumulation, reduction in a fixed order), tests the pair, and
// runs the scaled pair solver.  The unitary goes to wout[pair], the decision
// to rot[pair].
__global__ void __launch_bounds__(NTG, 1)
pair_eig32_kernel(const float2* __restrict__ X, int64_t ldx, int mm, int nn, int nb, int round, double tol,
                  float tol_inner, double nu_rel2, const double* __restrict__ xnorm2, float2* __restrict__ wout,
                  int* __restrict__ rot, int* __restrict__ flags, int max_inner, unsigned long long* phase_ns) {
  __shared__ float2 slab[SLAB][JC + 1];
  __shared__ float2 gram[NGRAM];
  __shared__ pair_eig_scaled2 sh;
  __shared__ int col[JC];
  __shared__ int any_rot, bad, offmax_blk, offbig_blk;
  const int t = threadIdx.x, pair = blockIdx.x;
  unsigned long long tp = 0;
  auto phase = [&](int ph) {  // optional diagnostics: time per phase into phase_ns[ph - 1]
    if (phase_ns && t == 0) {
      unsigned long long tn;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tn));
      if (ph > 0) atomicAdd(&phase_ns[ph - 1], tn - tp);
      tp = tn;
    }
  };
  phase(0);
  pair_columns(round, pair, nb, nn, col);
  if (t == 0) { any_rot = 0; bad = 0; offmax_blk = 0; offbig_blk = 0; sh.inner_rot = 0; }
  __syncthreads();
  // slab loads: thread t covers row (t & 255) of columns 8 (t >> 8) .. + 7
  const int lr = t & (SLAB - 1), ch = 8 * (t >> 8);
  const float2* cp[8];
#pragma unroll
  for (int c = 0; c < 8; c++) cp[c] = col[ch + c] >= 0 ? X + ldx * col[ch + c] : nullptr;
  float2 pf[8];
#pragma unroll
  for (int c = 0; c < 8; c++) pf[c] = (cp[c] && lr < mm) ? cp[c][lr] : make_float2(0.f, 0.f);
  // 36 upper 2x2 tiles x 14 row groups = 504 threads; group g takes rows
  // g, g + 14, ... of each slab
  constexpr int NGRP = 14;
  const int tile = t / NGRP, g = t - NGRP * (t / NGRP);
  const bool act = t < 36 * NGRP;
  int bi = 0, rem = act ? tile : 0;
  while (rem >= 8 - bi) { rem -= 8 - bi; bi++; }
  const int bj = bi + rem;
  float2 a00 = make_float2(0.f, 0.f), a01 = a00, a10 = a00, a11 = a00;
  for (int r0 = 0; r0 < mm; r0 += SLAB) {
#pragma unroll
    for (int c = 0; c < 8; c++) slab[lr][ch + c] = pf[c];
    __syncthreads();
    const int rn = r0 + SLAB + lr;
#pragma unroll
    for (int c = 0; c < 8; c++) pf[c] = (cp[c] && rn < mm) ? cp[c][rn] : make_float2(0.f, 0.f);
    if (act) {
#pragma unroll 4
      for (int rr = g; rr < SLAB; rr += NGRP) {
        const float2 p0 = slab[rr][2 * bi], p1 = slab[rr][2 * bi + 1], q0 = slab[rr][2 * bj], q1 = slab[rr][2 * bj + 1];
        cfma_conj(a00, p0, q0);
        cfma_conj(a01, p0, q1);
        cfma_conj(a10, p1, q0);
        cfma_conj(a11, p1, q1);
      }
    }
    __syncthreads();
  }
  phase(1);  // 0: Gram products
  // reduce the row groups in a fixed order (partials in the slab buffer)
  float2* red = &slab[0][0];
  if (act) {
    red[(g * 36 + tile) * 4 + 0] = a00;
    red[(g * 36 + tile) * 4 + 1] = a01;
    red[(g * 36 + tile) * 4 + 2] = a10;
    red[(g * 36 + tile) * 4 + 3] = a11;
  }
  __syncthreads();
  if (t < 144) {
    const int tl = t >> 2, q = t & 3;
    float2 v = red[tl * 4 + q];
    for (int gg = 1; gg < NGRP; gg++) v = cadd(v, red[(gg * 36 + tl) * 4 + q]);
    int ti = 0, tr = tl;
    while (tr >= 8 - ti) { tr -= 8 - ti; ti++; }
    const int tj = ti + tr;
    const int r = 2 * ti + (q >> 1), c = 2 * tj + (q & 1);
    if (ti != tj || r <= c) {
      gram[r * JC + c] = v;
      gram[c * JC + r] = cconj(v);
    }
  }
  __syncthreads();
  // scaled Gram, diagonal, test
  const double nu2 = nu_rel2 * (*xnorm2);
  const bool owner = t < NGRAM;
  const int i = (t / JC) & 15, j = t % JC;
  if (owner) {
    const float2 v = gram[t];
    if (!isfinite(v.x) || !isfinite(v.y)) bad = 1;
    if (i == j) { sh.d[0][i] = v.x; sh.d0[i] = v.x; }
  }
  __syncthreads();
  if (owner) {
    const float di = sh.d[0][i], dj = sh.d[0][j];
    float2 v = make_float2(0.f, 0.f);
    if (i != j && di > nu2 && dj > nu2) v = cscale(gram[t], (float)(1.0 / sqrt((double)di * (double)dj)));
    sh.G[0][i][j] = v;
    sh.W[0][i][j] = make_float2(i == j ? 1.f : 0.f, 0.f);
  }
  __syncthreads();
  if (bad) {
    if (t == 0) { atomicOr(&flags[QT_FLAG_NONFINITE], 1); rot[pair] = 0; }
    return;
  }
  {
    float relmax = 0.f, relbig = 0.f;
    const double big2 = 1e-6 * (*xnorm2);
    if (owner && i < j && col[i] >= 0 && col[j] >= 0 && sh.d[0][i] > nu2 && sh.d[0][j] > nu2) {
      const float rel = fminf(sqrtf(cabs2(sh.G[0][i][j])), 1.f);
      if (rel > tol) {
        any_rot = 1;
        relmax = rel;
        if (sh.d[0][i] > big2 && sh.d[0][j] > big2) relbig = rel;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      relmax = fmaxf(relmax, __shfl_xor_sync(0xffffffffu, relmax, o));
      relbig = fmaxf(relbig, __shfl_xor_sync(0xffffffffu, relbig, o));
    }
    if ((t & 31) == 0 && relmax > 0.f) atomicMax(&offmax_blk, __float_as_int(relmax));
    if ((t & 31) == 0 && relbig > 0.f) atomicMax(&offbig_blk, __float_as_int(relbig));
  }
  __syncthreads();
  if (t == 0) {
    rot[pair] = any_rot;
    if (offmax_blk > 0) atomicMax(&flags[QT_FLAG_OFFMAX], offmax_blk);
    if (offbig_blk > 0) atomicMax(&flags[QT_FLAG_OFFBIG], offbig_blk);
    if (any_rot) atomicAdd(&flags[QT_FLAG_ROTATED], 1);
  }
  phase(2);  // 1: reduction, scaled Gram, test
  if (!any_rot) return;
  int buf = 0;
  const int inner = diagonalise_scaled2(sh, col, tol_inner, (float)nu2, max_inner, &buf);
  if (t == 0) atomicAdd(&flags[QT_FLAG_INNER], inner);
  if (owner) wout[(size_t)pair * NGRAM + t] = sh.W[buf][i][j];
  phase(3);  // 2: pair solver
}

// grid (pair, row chunk): rotate this chunk's rows of X (and of V) by the
// pair's unitary.  One row per thread: its 16 values are loaded together
// (independent, coalesced across the warp), multiplied by W from shared
// memory (two entries per 16-byte broadcast load) and stored; no staging,
// no barriers after W is loaded.
__global__ void __launch_bounds__(NT, 3)
pair_apply32_kernel(float2* __restrict__ X, int64_t ldx, int mm, float2* __restrict__ V, int64_t ldv, int nn, int nb,
                    int round, int x_rows_per_chunk, int v_rows_per_chunk, const float2* __restrict__ win,
                    const int* __restrict__ rot) {
  __shared__ __align__(16) float2 Wt[JC][JC];
  __shared__ int col[JC];
  const int pair = blockIdx.x, chunk = blockIdx.y;
  if (!rot[pair]) return;
  pair_columns(round, pair, nb, nn, col);
  Wt[threadIdx.x / JC][threadIdx.x % JC] = win[(size_t)pair * NGRAM + threadIdx.x];
  __syncthreads();
  int cidx[JC];
#pragma unroll
  for (int c = 0; c < JC; c++) cidx[c] = col[c];
  for (int pass = 0; pass < 2; pass++) {
    float2* M = pass == 0 ? X : V;
    if (M == nullptr) break;
    const int64_t ld = pass == 0 ? ldx : ldv;
    const int per = pass == 0 ? x_rows_per_chunk : v_rows_per_chunk;
    const int lim = pass == 0 ? mm : nn;
    const int e = min(lim, chunk * per + per);
    for (int r = chunk * per + threadIdx.x; r < e; r += NT) {
      float2 x[JC];
#pragma unroll
      for (int k = 0; k < JC; k++) x[k] = cidx[k] >= 0 ? M[r + ld * cidx[k]] : make_float2(0.f, 0.f);
      float2 acc[JC];
#pragma unroll
      for (int c = 0; c < JC; c++) acc[c] = make_float2(0.f, 0.f);
      // keep the 256 W entries in shared memory (re-read per row) rather than
      // letting them be hoisted into registers across the row loop
      asm volatile("" ::: "memory");
#pragma unroll
      for (int k = 0; k < JC; k++) {
#pragma unroll
        for (int c = 0; c < JC; c += 2) {
          const float4 w = *reinterpret_cast<const float4*>(&Wt[k][c]);
          cfma(acc[c], x[k], make_float2(w.x, w.y));
          cfma(acc[c + 1], x[k], make_float2(w.z, w.w));
        }
      }
#pragma unroll
      for (int c = 0; c < JC; c++)
        if (cidx[c] >= 0) M[r + ld * cidx[c]] = acc[c];
    }
  }
}

// ---------------------------------------------------------------------------
// FP32 storage: one cooperative launch per sweep
// ---------------------------------------------------------------------------
//
// CTA q owns table q of every round.  Round g (counted over the whole
// iteration) rebuilds its two blocks from the previous round's data and
// unitaries: a block whose round g-1 pair rotated becomes that pair's 16
// columns times the matching 16x8 block of its unitary, otherwise it is
// copied.  The rebuilt columns go to the other buffer of a ping-pong pair
// (round g reads buffer (g-1)&1 and writes buffer g&1), and on their way
// through shared memory they feed the Gram products, so a round reads and
// writes every column once and needs no separate rotation pass.  Rounds are
// chained per CTA through done[q] (the last round CTA q finished): round g
// waits for the round g-1 CTAs whose output it reads (read after write) and
// for those that read what it overwrites -- the previous contents of its
// destination columns and of its unitary slot (write after read).  Every
// wait is bounded; a wait that gives up sets QT_FLAG_ABORT, which ends the
// other CTAs' waits too.  The pending unitaries of the last round are applied
// in place by pair_apply32_kernel after the last sweep.
//
// With halves = 2 each pair is served by two CTAs, CTA 2q + h holding rows
// [row_lo(h), row_hi(h)) of the pair's columns (and the matching rows of V;
// both splits at a multiple of 32 rows, clamped to the matrix, so a V of
// fewer than 32 rows belongs to half 0 alone).
// A row half reads and writes only its own rows, so each half runs the round
// protocol above on its own copies of the round flags, unitaries and rotate
// decisions (done, wbuf, rotbuf offset by h); the two halves of a pair meet
// once per round: each publishes its partial Gram (the 160 upper-tile entries
// of its rows) in gx and its round in xflag, waits (bounded) for the other's,
// and both add the two partials in the same order.  Both then run the same
// pair solver on the same Gram and reach the same unitary, bit for bit.
//
// What bounds a round of up to 512 rows: latency, about 15 us of it at any size,
// half of that the pair solver's chain.  So the rest is kept short: the decision,
// the unitary and the rows of both source blocks are loaded at once, before it
// is known which are needed; V's rows are rebuilt by warps that have no rows of
// X, or loaded ahead of the Gram products; one release publishes the round.
// Measured (us a round, 74 x 102 split / 240 x 160 late in the sweeps): 5.4 / 3.7
// -> 4.1 / 2.5 from the end of the wait to the end of the products.

constexpr int PS_SLAB = 256;                 // rows per slab
constexpr int PS_LDS = JC + 2;               // slab row stride in float2 (16-byte aligned rows)
constexpr int PS_TILES = 10;                 // upper 4x4 tiles of the 16x16 Gram
constexpr int PS_TE = 16;                    // entries per tile
constexpr int PS_NGRP = NTG / PS_TILES;      // 51 row groups per tile
constexpr size_t PS_SMEM = 2 * PS_SLAB * PS_LDS * sizeof(float2);  // double-buffered slab, 73,728 bytes
constexpr int PS_SPIN = 1 << 23;             // polls of a round wait before it gives up
static_assert(PS_TILES * PS_NGRP * PS_TE <= 2 * PS_SLAB * PS_LDS, "Gram partials reuse the slab buffer");

// tile -> (row quad ti, column quad tj), ti <= tj, ordered by ti
__device__ inline void ps_tile(int tile, int& ti, int& tj) {
  ti = 0;
  int rem = tile;
  while (rem >= 4 - ti) { rem -= 4 - ti; ti++; }
  tj = ti + rem;
}

// table q and side (0: first block of the pair, 1: second) of block `blk` in
// round `round` of the circle tournament over n players
__device__ inline void pair_of(int round, int blk, int n, int& q, int& side) {
  if (blk == n - 1) { q = 0; side = 1; return; }
  const int rr = round % (n - 1);
  if (blk == rr) { q = 0; side = 0; return; }
  const int d = (blk - rr + (n - 1)) % (n - 1);
  int partner;
  if (d <= n / 2 - 1) { q = d; partner = (rr - q + (n - 1)) % (n - 1); }
  else { q = n - 1 - d; partner = (rr + q) % (n - 1); }
  side = blk > partner ? 1 : 0;
}

__device__ inline int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline void st_release_gpu(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

struct sweep_solver {
  float d[2][JC];
  float d0[JC];
  float2 G[2][JC][JC + 1];
  float2 W[2][JC][JC + 1];
};

constexpr int SOLVER_THREADS = JC / 2 * JC;  // warps 0-3
__device__ inline void solver_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// The scaled pair solver, run by warps 0-3 alone (the caller's other warps
// skip it and wait at its next block barrier).  Its inner rounds are a serial
// chain (three values from shared memory, the rotation, the update, a
// barrier), so what counts is the chain's length and how many instructions
// share a scheduler with it: thread (k, y) computes the rotation of y's pair
// itself (every half-warp computes the same 16, bit-identically), takes those
// of the k-th pair (x, x') by shuffle, and updates Ghat[x][y], Ghat[x'][y] and
// two rows of Wt into the other buffer from values loaded before the rotation
// is known; one warp per scheduler, one named barrier per inner round.  An
// inner round in which no pair needs a rotation is skipped by every warp alike
// (a warp vote over the same 16 decisions).  Same iteration as
// diagonalise_scaled2; the rotation is evaluated with the special-function
// unit's square roots and reciprocals (a few ulps: the rotation stays unitary
// to FP32 rounding, and the one-sided iteration re-measures every pair from
// the data in the next round anyway).  A round of the 74 x 102 split takes 7.7 us
// here, of a wide one late in the sweeps 3.6; with one thread per entry of the
// Gram (eight warps) and loads behind the rotation 11.0 and 6.2.
// The finished unitary goes to wout (JC x JC).
__device__ int diagonalise_lanes(sweep_solver& sh, const int* col, float tol_inner, float nu2, int max_inner,
                                 float2* __restrict__ wout) {
  const int t = threadIdx.x, k = t >> 4, y = t & 15;
  if (t >= SOLVER_THREADS) return 0;  // warps 4-15
  const float tol2 = tol_inner * tol_inner;
  const unsigned live = __ballot_sync(0xffffffffu, col[y] >= 0);  // bit c of the low half: column c is there
  int cur = 0, sweep = 0;
  for (; sweep < max_inner; sweep++) {
    bool rotated_any = false;
    for (int ir = 0; ir < JC - 1; ir++) {
      int yp = 2 * ir - y;
      yp = yp < 0 ? yp + (JC - 1) : yp >= JC - 1 ? yp - (JC - 1) : yp;
      yp = y == JC - 1 ? ir : y == ir ? JC - 1 : yp;
      int x = ir + k, xp = ir - k;
      x = x >= JC - 1 ? x - (JC - 1) : x;
      xp = k == 0 ? JC - 1 : xp < 0 ? xp + (JC - 1) : xp;
      const int p = min(y, yp), q = max(y, yp);
      const float a = sh.d[cur][p], b = sh.d[cur][q];
      const float2 gs = sh.G[cur][p][q];
      const float2 g_xy = sh.G[cur][x][y], g_xq = sh.G[cur][x][yp];
      const float2 g_py = sh.G[cur][xp][y], g_pq = sh.G[cur][xp][yp];
      const float2 w0_y = sh.W[cur][k][y], w0_q = sh.W[cur][k][yp];
      const float2 w1_y = sh.W[cur][k + JC / 2][y], w1_q = sh.W[cur][k + JC / 2][yp];
      const float ags2 = gs.x * gs.x + gs.y * gs.y;
      const bool rotp = ((live >> p) & (live >> q) & 1) && a > nu2 && b > nu2 && ags2 > tol2;
      if (!__any_sync(0xffffffffu, rotp)) continue;  // the same vote in every solver warp
      rotated_any = true;
      // (evaluated by every lane and dropped where its pair does not rotate: a
      // branch would cost the others its reconvergence)
      const float ria = rsqrtf(a), rib = rsqrtf(b), rags = rsqrtf(ags2);
      const float sqa = a * ria, sqb = b * rib;
      const float ag = ags2 * rags * sqa * sqb;  // |gamma|
      const float zeta = __fdividef(b - a, 2.f * ag);
      const float z2 = fmaf(zeta, zeta, 1.f);
      const float r1 = z2 * rsqrtf(z2);
      const float tt = copysignf(__fdividef(1.f, fabsf(zeta) + r1), zeta);
      const float c = rsqrtf(fmaf(tt, tt, 1.f)), sn = c * tt;
      const float2 e = make_float2(gs.x * rags, gs.y * rags);
      float a2 = fmaxf(fmaf(-tt, ag, a), nu2);  // a column driven to the noise level is frozen
      float b2 = fmaf(tt, ag, b);
      const float ia2 = rsqrtf(a2), ib2 = rsqrtf(b2);
      const float fa = sqa * ia2, fb = sqb * ib2, fab = sqb * ia2, fba = sqa * ib2;
      const float2 jpp = make_float2(rotp ? c * fa : 1.f, 0.f);
      const float2 jqp = make_float2(rotp ? -sn * e.x * fab : 0.f, rotp ? sn * e.y * fab : 0.f);  // -s conj(e) sqrt(b/a')
      const float2 jpq = make_float2(rotp ? sn * e.x * fba : 0.f, rotp ? sn * e.y * fba : 0.f);   //  s e sqrt(a/b')
      const float2 jqq = make_float2(rotp ? c * fb : 1.f, 0.f);
      a2 = rotp ? a2 : a;
      b2 = rotp ? b2 : b;
      // column y of Jt: rows y (real) and y'
      const bool low = y == p;
      const float2 jyy = low ? jpp : jqq, jpy = low ? jqp : jpq;
      // columns x and x' of Jt from lanes x and x' (which hold y == x, x')
      const float2 jxx = make_float2(__shfl_sync(0xffffffffu, jyy.x, x), 0.f);
      const float2 jpx = make_float2(__shfl_sync(0xffffffffu, jpy.x, x), __shfl_sync(0xffffffffu, jpy.y, x));
      const float2 jXX = make_float2(__shfl_sync(0xffffffffu, jyy.x, xp), 0.f);
      const float2 jPX = make_float2(__shfl_sync(0xffffffffu, jpy.x, xp), __shfl_sync(0xffffffffu, jpy.y, xp));
      if (k == 0) sh.d[cur ^ 1][y] = low ? a2 : b2;
      const float2 hx = cadd(cmul(g_xy, jyy), cmul(g_xq, jpy));
      const float2 hp = cadd(cmul(g_py, jyy), cmul(g_pq, jpy));
      float2 gx = cadd(cmul(cconj(jxx), hx), cmul(cconj(jpx), hp));
      float2 gp = cadd(cmul(cconj(jXX), hp), cmul(cconj(jPX), hx));
      const float2 zero = make_float2(0.f, 0.f);
      if (y == x) {
        gx = zero;
        gp = jXX.x != 1.f || jPX.x != 0.f || jPX.y != 0.f ? zero : g_py;
      } else if (y == xp) {
        gx = jxx.x != 1.f || jpx.x != 0.f || jpx.y != 0.f ? zero : g_xy;
        gp = zero;
      }
      sh.G[cur ^ 1][x][y] = gx;
      sh.G[cur ^ 1][xp][y] = gp;
      sh.W[cur ^ 1][k][y] = cadd(cmul(w0_y, jyy), cmul(w0_q, jpy));
      sh.W[cur ^ 1][k + JC / 2][y] = cadd(cmul(w1_y, jyy), cmul(w1_q, jpy));
      cur ^= 1;
      solver_sync();
    }
    if (!rotated_any) break;  // every solver warp took the same votes
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {  // the rows this thread updated itself
    const int x = k + h * (JC / 2);
    const float d0 = sh.d0[x];
    __stcg(wout + x * JC + y, d0 > 0.f ? cscale(sh.W[cur][x][y], sqrtf(sh.d[cur][y]) * rsqrtf(d0))
                                       : make_float2(x == y ? 1.f : 0.f, 0.f));
  }
  return sweep + (sweep < max_inner ? 1 : 0);
}

// Sweeps of nb - 1 rounds from round g0 on: nsweeps of them at most, ending with
// the first that rotates nothing (one sweep only where the caller has a rule
// of its own for the end: MULTI = false, as the code for more costs a round 2 %).
// xb[0] is X itself, xb[1] a scratch copy of its shape (likewise vb for V);
// wbuf holds 2 x pairs unitaries, rotbuf 2 x pairs decisions, done[pairs] the
// completed round of each CTA.
template <bool MULTI>
__global__ void __launch_bounds__(NTG, 1)
jacobi_sweep32_kernel(float2* __restrict__ xb0, float2* __restrict__ xb1, int64_t ldx, int mm,
                      float2* __restrict__ vb0, float2* __restrict__ vb1, int64_t ldv, int nn, int nb, int g0,
                      int has_prev, double tol, float tol_inner, double nu_rel2, const double* __restrict__ xnorm2,
                      float2* __restrict__ wbuf, int* __restrict__ rotbuf, int* __restrict__ done,
                      int* __restrict__ flags, int max_inner, int max_inner0, int nsweeps, float keep2,
                      float* __restrict__ dnorm, unsigned long long* phase_ns, int spin, int stall, int halves, int row_mid, int vrow_mid,
                      float2* __restrict__ gx, int* __restrict__ xflag) {
  extern __shared__ __align__(16) float2 ps_slab[];  // [2][PS_SLAB][PS_LDS]
  __shared__ __align__(16) float2 wsub[2][JC][JW];    // 16x8 unitary blocks that rebuild the two blocks
  __shared__ float2 psum[3][PS_TILES * PS_TE];
  __shared__ float2 gram[NGRAM];
  __shared__ sweep_solver sh;
  __shared__ int col[JC];
  __shared__ int any_rot, bad, offmax_blk, offbig_blk, offkept_blk;
  const int H = halves, t = threadIdx.x, q = blockIdx.x / H, hf = blockIdx.x % H, pairs = gridDim.x / H,
            R = nb - 1;
  // this CTA's rows of X and V, and its half's copies of the round state
  const int row_lo = hf ? row_mid : 0, row_hi = (hf || H == 1) ? mm : row_mid;
  const int vrow_lo = hf ? vrow_mid : 0, vrow_hi = (hf || H == 1) ? nn : vrow_mid;
  done += (size_t)hf * pairs;
  wbuf += (size_t)hf * 2 * pairs * NGRAM;
  rotbuf += (size_t)hf * 2 * pairs;
  if (hf) { phase_ns = nullptr; dnorm = nullptr; }  // half 0 reports for the pair
  __shared__ unsigned long long tp;
  int swept = 0, swept_off = 0, swept_big = 0;  // thread 0: what this CTA has to say about this sweep
  auto phase = [&](int ph) {  // optional diagnostics: time per phase into phase_ns[ph - 1]
    if (phase_ns && t == 0) {
      unsigned long long tn;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tn));
      if (ph > 0) atomicAdd(&phase_ns[ph - 1], tn - tp);
      tp = tn;
    }
  };
  const float nu2 = (float)(nu_rel2 * (*xnorm2));
  const float big2 = (float)(1e-6 * (*xnorm2));
  const float tolf = (float)tol;
  // slab rows: thread t rebuilds row (t & 255) of block (t >> 8)
  const int lr = t & (PS_SLAB - 1), h = t >> 8;
  // Gram products: rows 4 ti .. 4 ti + 3 against columns 4 tj .. 4 tj + 3, row group grp
  const int tile = t / PS_NGRP, grp = t - PS_NGRP * (t / PS_NGRP);
  const bool act = tile < PS_TILES;
  int ti = 0, tj = 0;
  if (act) ps_tile(tile, ti, tj);
  const int nslab = (row_hi - row_lo + PS_SLAB - 1) / PS_SLAB;
  for (int rs = 0; rs < (MULTI ? R * nsweeps : R); rs++) {
    const int r = MULTI ? rs % R : rs, sweep = MULTI ? rs / R : 0;
    const int g = g0 + rs;
    const bool prev = rs > 0 || has_prev;
    const int rp = r > 0 ? r - 1 : R - 1;  // round (within its sweep) of g - 1
    const int rpp = (r + 2 * R - 2) % R;   // ... of g - 2
    phase(0);
    int bi, bj;
    tournament(r, q, nb, bi, bj);
    // ---- what does not depend on other CTAs: this round's columns, and where
    // this half's block was in round g - 1 (pair qq, first or second block, with partner blocks a2 and b2)
    pair_columns(r, q, nb, nn, col);
    if (t == 0) { any_rot = 0; bad = 0; offmax_blk = 0; offbig_blk = 0; offkept_blk = 0; }
    const int blk = h == 0 ? bi : bj;
    int srcq = 0, sside = 0, a2 = blk, b2 = blk;
    if (prev) {
      pair_of(rp, blk, nb, srcq, sside);
      tournament(rp, srcq, nb, a2, b2);
    }
    // ---- wait for the round g - 1 CTAs this round depends on
    int gave_up = 0;
    if (stall && q == 0 && t == 0 && rs == 0) {
      // test hook (QT_JACOBI_STALL_TEST): a bounded wait on a status word that
      // nothing sets, which must end in QT_ETIMEOUT with the context usable
      int it = 0;
      for (; it < spin; it++) {
        if (ld_acquire_gpu(flags + QT_FLAG_STALL) != 0) break;
        if (*(volatile int*)(flags + QT_FLAG_ABORT)) { it = spin; break; }
        __nanosleep(64);
      }
      if (it >= spin) { gave_up = 1; atomicExch(flags + QT_FLAG_ABORT, 1); }
    }
    if (prev && t < 6) {
      int target = -1, qq, s;
      if (t < 2) {  // read after write: the pairs that held our blocks in round g - 1
        pair_of(rp, t == 0 ? bi : bj, nb, qq, s);
        target = qq;
      } else if (g >= 2 && t < 4) {  // write after read: readers of our blocks' round g - 2 columns
        const int blk = t == 2 ? bi : bj;
        int a2, b2;
        pair_of(rpp, blk, nb, qq, s);
        tournament(rpp, qq, nb, a2, b2);
        pair_of(rp, a2 == blk ? b2 : a2, nb, qq, s);
        target = qq;
      } else if (g >= 2) {  // write after read: readers of unitary slot q of round g - 2
        int a2, b2;
        tournament(rpp, q, nb, a2, b2);
        pair_of(rp, t == 4 ? a2 : b2, nb, qq, s);
        target = qq;
      }
      if (target >= 0) {
        int it = 0;
        for (; it < spin; it++) {
          if (ld_acquire_gpu(done + target) >= g - 1) break;
          if ((it & 7) == 7 && *(volatile int*)(flags + QT_FLAG_ABORT)) { it = spin; break; }
          __nanosleep(64);
        }
        if (it >= spin) { gave_up = 1; atomicExch(flags + QT_FLAG_ABORT, 1); }
      }
    }
    if (__syncthreads_or(gave_up)) return;
    phase(1);  // 0: waits
    const float2* __restrict__ src = prev ? (((g - 1) & 1) ? xb1 : xb0) : ((g & 1) ? xb1 : xb0);
    float2* __restrict__ dst = (g & 1) ? xb1 : xb0;
    const float2* __restrict__ vsrc = ((g - 1) & 1) ? vb1 : vb0;
    float2* __restrict__ vdst = (g & 1) ? vb1 : vb0;
    const bool vwork = prev && vb0 != nullptr;
    // V's rows go to the warps in reverse order: those whose X rows lie past
    // the matrix (only one slab then) take them instead, at the same time
    const int vrow = vrow_lo + (PS_SLAB - 32 - (lr & ~31)) + (lr & 31);
    const bool vfirst = vwork && nslab <= 1 && row_lo + (lr & ~31) >= row_hi;
    // column indices stay in shared memory (warp-uniform broadcast reads)
    const int* oc = col + h * JW;
    // ---- the first rows of both source blocks, the unitary and whether there
    // is one, all under one latency
    float2 xr[JC];
    bool hrot = false;
    {
      const int rr = vfirst ? vrow : row_lo + lr, lim = vfirst ? vrow_hi : row_hi;
      const float2* __restrict__ M = (vfirst ? vsrc : src) + rr;
      const int64_t ld = vfirst ? ldv : ldx;
      const size_t slot = (size_t)((g - 1) & 1) * pairs + srcq;
      const int tt = t & (PS_SLAB - 1);
      int rotated = 0;
      float2 wv = make_float2(0.f, 0.f);
      if (prev) {
        rotated = __ldcg(rotbuf + slot);
        // (left over from an earlier round where the pair did not rotate, and not used then)
        if (tt < JC * JW) wv = __ldcg(wbuf + slot * NGRAM + (tt / JW) * JC + sside * JW + tt % JW);
      }
#pragma unroll
      for (int k = 0; k < JC; k++) {
        const int gc = (k < JW ? a2 : b2) * JW + k % JW;
        xr[k] = (gc < nn && rr < lim && (k < JW || prev)) ? __ldcg(M + ld * gc) : make_float2(0.f, 0.f);
      }
      hrot = rotated != 0;
      if (!hrot) {
        if (sside)
#pragma unroll
          for (int k = 0; k < JW; k++) xr[k] = xr[k + JW];
        a2 = blk;
      }
      if (tt < JC * JW) wsub[h][tt / JW][tt % JW] = wv;
    }
    __syncthreads();
    // ---- rebuild the rows slab by slab; Gram products on the previous slab meanwhile
    auto load_row = [&](const float2* __restrict__ M, int64_t ld, int lim, int rr) {
#pragma unroll
      for (int k = 0; k < JW; k++)
        xr[k] = (a2 * JW + k < nn && rr < lim) ? __ldcg(M + rr + ld * (a2 * JW + k)) : make_float2(0.f, 0.f);
      if (hrot) {
#pragma unroll
        for (int k = 0; k < JW; k++)
          xr[JW + k] = (b2 * JW + k < nn && rr < lim) ? __ldcg(M + rr + ld * (b2 * JW + k)) : make_float2(0.f, 0.f);
      }
    };
    auto rebuild = [&](float2* out) {
      if (hrot) {
        // two partial sums per output (the real and the imaginary part of
        // x_k each feed their own): four independent FMAs per complex
        // product instead of two dependent pairs
        float2 ob[JW];
#pragma unroll
        for (int c = 0; c < JW; c++) { out[c] = make_float2(0.f, 0.f); ob[c] = out[c]; }
        asm volatile("" ::: "memory");  // keep wsub in shared memory
#pragma unroll
        for (int k = 0; k < JC; k++) {
#pragma unroll
          for (int c = 0; c < JW; c += 2) {
            const float4 w = *reinterpret_cast<const float4*>(&wsub[h][k][c]);
            out[c].x = fmaf(xr[k].x, w.x, out[c].x);
            out[c].y = fmaf(xr[k].x, w.y, out[c].y);
            ob[c].x = fmaf(-xr[k].y, w.y, ob[c].x);
            ob[c].y = fmaf(xr[k].y, w.x, ob[c].y);
            out[c + 1].x = fmaf(xr[k].x, w.z, out[c + 1].x);
            out[c + 1].y = fmaf(xr[k].x, w.w, out[c + 1].y);
            ob[c + 1].x = fmaf(-xr[k].y, w.w, ob[c + 1].x);
            ob[c + 1].y = fmaf(xr[k].y, w.z, ob[c + 1].y);
          }
        }
#pragma unroll
        for (int c = 0; c < JW; c++) out[c] = cadd(out[c], ob[c]);
      } else {
#pragma unroll
        for (int c = 0; c < JW; c++) out[c] = xr[c];
      }
    };
    auto build_slab = [&](int s) {
      const int rr = row_lo + s * PS_SLAB + lr;
      float2 o[JW];
      rebuild(o);
      if (prev && rr < row_hi) {
#pragma unroll
        for (int c = 0; c < JW; c++)
          if (oc[c] >= 0) __stcg(dst + rr + ldx * oc[c], o[c]);
      }
      float4* sp = reinterpret_cast<float4*>(ps_slab + ((size_t)(s & 1) * PS_SLAB + lr) * PS_LDS + h * JW);
#pragma unroll
      for (int c = 0; c < JW; c += 2) sp[c / 2] = make_float4(o[c].x, o[c].y, o[c + 1].x, o[c + 1].y);
    };
    auto build_vrow = [&](int rr) {
      if (rr - (lr & 31) >= vrow_hi) return;  // the whole warp
      float2 o[JW];
      rebuild(o);
      if (rr < vrow_hi) {
#pragma unroll
        for (int c = 0; c < JW; c++)
          if (oc[c] >= 0) __stcg(vdst + rr + ldv * oc[c], o[c]);
      }
    };
    float2 acc[PS_TE];
#pragma unroll
    for (int e = 0; e < PS_TE; e++) acc[e] = make_float2(0.f, 0.f);
    if (vfirst) build_vrow(vrow);
    else build_slab(0);
    __syncthreads();
    for (int s = 0; s < nslab; s++) {
      if (s + 1 < nslab) load_row(src, ldx, row_hi, row_lo + (s + 1) * PS_SLAB + lr);
      else if (vwork && !vfirst) load_row(vsrc, ldv, vrow_hi, vrow);
      if (act) {
        const float2* base = ps_slab + (size_t)(s & 1) * PS_SLAB * PS_LDS;
        const int rows = min(PS_SLAB, row_hi - row_lo - s * PS_SLAB);
#pragma unroll 1
        for (int rr = grp; rr < rows; rr += PS_NGRP) {
          const float4* rowp = reinterpret_cast<const float4*>(base + (size_t)rr * PS_LDS);
          const float4 p01 = rowp[2 * ti], p23 = rowp[2 * ti + 1], q01 = rowp[2 * tj], q23 = rowp[2 * tj + 1];
          const float2 pv[4] = {make_float2(p01.x, p01.y), make_float2(p01.z, p01.w), make_float2(p23.x, p23.y),
                                make_float2(p23.z, p23.w)};
          const float2 qv[4] = {make_float2(q01.x, q01.y), make_float2(q01.z, q01.w), make_float2(q23.x, q23.y),
                                make_float2(q23.z, q23.w)};
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) cfma_conj(acc[a * 4 + b], pv[a], qv[b]);
        }
      }
      if (s + 1 < nslab) build_slab(s + 1);
      __syncthreads();
    }
    // ---- V rows (rotation only)
    if (vwork) {
      if (!vfirst) build_vrow(vrow);
      for (int rr = vrow + PS_SLAB; rr < vrow_hi; rr += PS_SLAB) {
        load_row(vsrc, ldv, vrow_hi, rr);
        build_vrow(rr);
      }
    }
    phase(2);  // 1: rebuild + Gram products
    // ---- reduce the row groups in a fixed order: three partial sums of 17
    // groups each, then their sum; the diagonal goes to the solver's D
    // (stored group-fastest: neighbouring threads hold neighbouring groups, and
    // the sums start 17 entries apart, so that neither side meets a bank twice;
    // entry-fastest, every lane of a store met the same bank, 3.8 us a round
    // from here to the pair solver instead of 1.5)
    float2* red = ps_slab;
    if (act) {
#pragma unroll
      for (int e = 0; e < PS_TE; e++) red[(tile * PS_TE + e) * PS_NGRP + grp] = acc[e];
    }
    __syncthreads();
    static_assert(PS_NGRP == 3 * 17, "three partial sums of 17 row groups");
    if (t < 3 * PS_TILES * PS_TE) {
      const int ent = t / 3, part = t % 3;
      const float2* rp0 = red + ent * PS_NGRP + part * 17;
      float2 v = rp0[0];
#pragma unroll
      for (int gg = 1; gg < 17; gg++) v = cadd(v, rp0[gg]);
      psum[part][ent] = v;
    }
    __syncthreads();
    float2 xv = make_float2(0.f, 0.f);
    if (t < PS_TILES * PS_TE) {
      xv = cadd(cadd(psum[0][t], psum[1][t]), psum[2][t]);
      if (H > 1) __stcg(gx + (((size_t)(g & 1) * pairs + q) * H + hf) * (PS_TILES * PS_TE) + t, xv);
    }
    if (H > 1) {
      // the two row halves of the pair exchange their partial Grams (bounded wait)
      __threadfence();
      __syncthreads();
      int gave = 0;
      if (t == 0) {
        st_release_gpu(xflag + (size_t)hf * pairs + q, g);
        int it = 0;
        for (; it < spin; it++) {
          if (ld_acquire_gpu(xflag + (size_t)(1 - hf) * pairs + q) >= g) break;
          if ((it & 7) == 7 && *(volatile int*)(flags + QT_FLAG_ABORT)) { it = spin; break; }
          __nanosleep(32);
        }
        if (it >= spin) { gave = 1; atomicExch(flags + QT_FLAG_ABORT, 1); }
      }
      if (__syncthreads_or(gave)) return;
      if (t < PS_TILES * PS_TE) {
        const float2 o = __ldcg(gx + (((size_t)(g & 1) * pairs + q) * H + (1 - hf)) * (PS_TILES * PS_TE) + t);
        xv = hf == 0 ? cadd(xv, o) : cadd(o, xv);  // (half 0) + (half 1) in both CTAs
      }
    }
    if (t < PS_TILES * PS_TE) {
      const float2 v = xv;
      int ai, aj;
      ps_tile(t / PS_TE, ai, aj);
      const int e = t % PS_TE;
      const int rw = 4 * ai + e / 4, cl = 4 * aj + e % 4;
      if (ai != aj || rw <= cl) {
        if (!isfinite(v.x) || !isfinite(v.y)) bad = 1;
        gram[rw * JC + cl] = v;
        gram[cl * JC + rw] = cconj(v);
        if (rw == cl) {
          sh.d[0][rw] = v.x;
          sh.d0[rw] = v.x;
          // the last round of the sweep reports every column's squared norm
          if (dnorm && r == R - 1 && col[rw] >= 0) dnorm[col[rw]] = v.x;
        }
      }
    }
    __syncthreads();
    // ---- scaled Gram, test
    const bool owner = t < NGRAM;
    const int i = (t / JC) & 15, j = t % JC;
    {
      float relmax = 0.f, relbig = 0.f, relkept = 0.f;
      if (owner) {
        const float di = sh.d[0][i], dj = sh.d[0][j];
        const bool live = i != j && di > nu2 && dj > nu2;
        const float2 v = live ? cscale(gram[t], rsqrtf(di) * rsqrtf(dj)) : make_float2(0.f, 0.f);
        sh.G[0][i][j] = v;
        sh.W[0][i][j] = make_float2(i == j ? 1.f : 0.f, 0.f);
        if (!bad && live && i < j && col[i] >= 0 && col[j] >= 0) {
          const float rel = fminf(sqrtf(cabs2(v)), 1.f);
          if (rel > tolf) {
            any_rot = 1;
            relmax = rel;
            if (di > big2 && dj > big2) relbig = rel;
            if (fmaxf(di, dj) > keep2) relkept = rel;
          }
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        relmax = fmaxf(relmax, __shfl_xor_sync(0xffffffffu, relmax, o));
        relbig = fmaxf(relbig, __shfl_xor_sync(0xffffffffu, relbig, o));
        relkept = fmaxf(relkept, __shfl_xor_sync(0xffffffffu, relkept, o));
      }
      if ((t & 31) == 0 && relmax > 0.f) atomicMax(&offmax_blk, __float_as_int(relmax));
      if ((t & 31) == 0 && relbig > 0.f) atomicMax(&offbig_blk, __float_as_int(relbig));
      if ((t & 31) == 0 && relkept > 0.f) atomicMax(&offkept_blk, __float_as_int(relkept));
    }
    __syncthreads();
    if (t == 0) {
      if (bad) atomicOr(&flags[QT_FLAG_NONFINITE], 1);
      __stcg(rotbuf + (size_t)(g & 1) * pairs + q, any_rot);
      if (hf == 0) {  // the pair's statistics, once
        if (MULTI) {
          swept_off = max(r > 0 ? swept_off : 0, offmax_blk);
          swept_big = max(r > 0 ? swept_big : 0, offbig_blk);
        } else {
          if (offmax_blk > 0) atomicMax(&flags[QT_FLAG_OFFMAX], offmax_blk);
          if (offbig_blk > 0) atomicMax(&flags[QT_FLAG_OFFBIG], offbig_blk);
        }
        if (offkept_blk > 0) atomicMax(&flags[QT_FLAG_OFFKEPT], offkept_blk);
        if (any_rot) atomicAdd(&flags[QT_FLAG_ROTATED], 1);
      }
    }
    phase(3);  // 2: reduction, scaled Gram, test
    if (any_rot) {
      const int inner = diagonalise_lanes(sh, col, tol_inner, nu2, sweep < 2 ? max_inner0 : max_inner,
                                          wbuf + (size_t)(g & 1) * pairs * NGRAM + (size_t)q * NGRAM);
      if (t == 0 && hf == 0) atomicAdd(&flags[QT_FLAG_INNER], inner);
    }
    phase(4);  // 3: pair solver
    // ---- publish round g (the barrier orders every thread's stores before
    // thread 0's release, which is cumulative: no fence per thread)
    __syncthreads();
    if (t == 0) st_release_gpu(done + q, g);
    if (!MULTI) continue;
    // ---- several sweeps in this launch: the end of one waits (bounded) until
    // every CTA has said whether it rotated (1) or met a non-finite value
    // (65536), and a sweep without the first or with the second is the last.
    // Sweep s adds up in slot s % 3, its largest off-diagonals beside that (the
    // rule at the sweep limit is about the last sweep alone); CTA 0 clears the
    // next slots before it arrives: whoever read them two sweeps ago has arrived
    // since.
    if (t == 0) swept = (r > 0 ? swept : 0) | (any_rot ? 1 : 0) | (bad ? 65536 : 0);
    if (r < R - 1) continue;
    int stop = 0;
    gave_up = 0;
    if (t == 0) {
      int* count = flags + QT_FLAG_SWEPT;
      int *off = flags + QT_FLAG_SWEPT_OFF + sweep % 3, *big = flags + QT_FLAG_SWEPT_BIG + sweep % 3;
      if (swept) atomicAdd(count + sweep % 3, swept);
      if (swept_off > 0) atomicMax(off, swept_off);
      if (swept_big > 0) atomicMax(big, swept_big);
      if (blockIdx.x == 0) {
        const int next = (sweep + 1) % 3;
        atomicExch(count + next, 0);
        atomicExch(flags + QT_FLAG_SWEPT_OFF + next, 0);
        atomicExch(flags + QT_FLAG_SWEPT_BIG + next, 0);
      }
      __threadfence();
      atomicAdd(flags + QT_FLAG_ARRIVED, 1);
      int it = 0;
      for (; it < spin; it++) {
        if (ld_acquire_gpu(flags + QT_FLAG_ARRIVED) >= (sweep + 1) * (int)gridDim.x) break;
        if ((it & 7) == 7 && *(volatile int*)(flags + QT_FLAG_ABORT)) { it = spin; break; }
        __nanosleep(64);
      }
      if (it >= spin) { gave_up = 1; atomicExch(flags + QT_FLAG_ABORT, 1); }
      const int said = ld_acquire_gpu(count + sweep % 3);
      stop = said == 0 || said >= 65536;
      if (blockIdx.x == 0) {
        flags[QT_FLAG_SWEEPS] = sweep + 1;
        flags[QT_FLAG_CONVERGED] = said == 0;
        flags[QT_FLAG_OFFMAX] = ld_acquire_gpu(off);
        flags[QT_FLAG_OFFBIG] = ld_acquire_gpu(big);
      }
    }
    if (__syncthreads_or(gave_up || stop)) return;
  }
}

// ---------------------------------------------------------------------------
// FP32 storage: columns resident in registers, one cooperative launch per sweep
// ---------------------------------------------------------------------------
//
// CTA c holds two blocks of RB = 4 columns in registers (warp w rows
// 64 RP w ..., lane l rows l, l + 32, ... of them).  A round rotates the 16 cross pairs of its two blocks, four
// disjoint pairs at a time: every warp sums its rows, the sums meet in shared
// memory, every warp adds them in the same order, finds the same four
// rotations and rotates its rows.  A sweep's first round also rotates the pairs
// inside each block.  No Gram, no unitary, no second pass over the rows.
//
// Between rounds one block stays and the other moves on, for most of the sweep
// (ring_blocks): on K CTAs the K moving blocks pass once round the ring of CTAs
// (K rounds), which pairs every staying block with every moving one; then the
// staying blocks pair up among themselves on half of the CTAs and the moving
// ones on the other half, and so on; an odd number of CTAs plays a tournament.
// K + K/2 + ... = 2 K - 1 rounds cover every pair of the 2 K blocks once, and
// half the traffic of a tournament.  A block that leaves is written to its slot
// of the mailbox by the warps that hold it, every number in one 8-byte element of
// a two-element store with the number of the round in its other 4 bytes; the warp of
// the same rows in the next CTA reads the slot until every number carries that
// round.  So the data is its own flag: no fence and no second trip to L2 (a flag
// behind a fence cost 4.5 us a round, twice this), and no CTA-wide barrier.  A
// slot is written only by the CTA that holds its block, i.e. that has read it.
// Every wait is bounded (QT_FLAG_ABORT ends them all and becomes QT_ETIMEOUT);
// leaving blocks are written before any wait and all CTAs are resident, so the
// waits end.
//
// The rotation: FP32 on the scaled sums (cosine and ratio of the norms, O(1)
// numbers at any scale), then brought to unit length from its exactly formed
// defect, as near to unitary as FP32 stores it.
//
// What bounds it: 20 FMAs per row and column pair (2048 x 1152: 0.67 ms a sweep
// over the chip), the four sub-rounds' barrier and rotation chain, and the
// exchange's latency.  Eight columns of 2048 rows are half of an SM's
// registers, and 1152 columns its 144 CTAs.  Measured on the chi = 1024 sketch
// (2048 x 1152): 2.6 ms a sweep, 9.0 us a round (four sub-rounds 4.7, exchange
// 3.5 to 4), against 5.2 ms of the Gram-based sweep kernel, in as many sweeps;
// 512 x 320: 0.35 against 1.03 ms a sweep, 4.4 us a round.  Not taken where the
// caller needs the split of theta' itself: every column is rounded once per
// pair and not once per round of 16 columns, and a 14-qubit circuit came out
// 4.6e-6 off instead of 3.5e-6; a sketch's own error hides that.

constexpr int RB = 4;            // columns per block
constexpr int RING_WARPS = 16;   // warps per CTA at most (128 registers a thread)
constexpr int RING_CTAS = 512;   // CTAs at most (the schedule table in shared memory)

// Rounds of a sweep on K CTAs.
__host__ __device__ inline int ring_rounds(int K) {
  int r = 0;
  while (K % 2 == 0) { r += K; K /= 2; }
  return r + 2 * K - 1;
}

// Blocks (of 2 K) that CTA c holds in round r.
__device__ inline void ring_blocks(int K, int r, int c, int& a, int& b) {
  int size[10], lev = 0, k = K, upper = 0;  // levels above: their group sizes, bit lev of `upper`: second half
  while (k % 2 == 0 && r >= k) {
    r -= k;
    size[lev] = k;
    k /= 2;
    if (c >= k) { upper |= 1 << lev; c -= k; }
    lev++;
  }
  int m[2] = {0, 1}, i[2];  // list (0: staying, 1: moving) and place in it
  if (k % 2 == 0 || k == 1) {
    i[0] = c;
    i[1] = (c + r) % k;
  } else {  // tournament over the 2 k blocks: 0 .. k - 1 the first list
    int x, y;
    tournament(r, c, 2 * k, x, y);
    m[0] = x >= k; i[0] = x - m[0] * k;
    m[1] = y >= k; i[1] = y - m[1] * k;
  }
  for (int h = 0; h < 2; h++) {
    int mm = m[h], ii = i[h];
    for (int l = lev - 1; l >= 0; l--) {
      const int n = size[l], half = n / 2;
      if ((upper >> l) & 1) { ii = mm ? (ii - 1 + n) % n : (ii + half - 1) % n; mm = 1; }
      else { ii = mm ? ii + half : ii; mm = 0; }
    }
    (h ? b : a) = mm * K + ii;
  }
}

struct RingArgs {
  float2* X;
  int64_t ldx;
  int mm, nn;
  int g0;          // rounds before this sweep
  float tol;
  double nu_rel2;
  const double* xnorm2;
  uint4* mail;     // a slot of warps x RB x rows-per-lane x 32 entries for each of the 2 K blocks
  int* flags;
  float keep2;
  float* dnorm;    // the columns' squared norms at the end of the sweep (nullptr: not wanted)
  int spin, stall;
};

// Two FP32 values in a 64-bit register, one instruction for both (sm_100 on).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 x2_pack(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 x2_unpack(f32x2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f32x2 x2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 x2_mul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float x2_sum(f32x2 a) {
  const float2 v = x2_unpack(a);
  return v.x + v.y;
}

// An entry of the mailbox: two elements of 8 bytes, each a number and the round
// that it was sent in.  A vector access is one access per element, in any order,
// so an element arrives whole and a number is there when its round is.
// (Assembled inside the instruction's block: with shifts around it 512 x 320
// sweeps took 0.7 % longer.)
__device__ __forceinline__ void mail_store(uint4* p, float re, float im, unsigned stamp) {
  asm volatile("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
               "st.relaxed.gpu.global.v2.b64 [%0], {a, b};\n\t}" ::"l"(p),
               "r"(__float_as_uint(re)), "r"(__float_as_uint(im)), "r"(stamp)
               : "memory");
}
__device__ __forceinline__ uint4 mail_load(const uint4* p) {  // re, stamp, im, stamp
  uint4 v;
  asm volatile("{\n\t.reg .b64 a, b;\n\t"
               "ld.relaxed.gpu.global.v2.b64 {a, b}, [%4];\n\t"
               "mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// The rows a lane holds of one column: pairs of rows, real and imaginary parts
// apart, so that every product of a rotation is one instruction for two rows.
template <int RP>
struct ring_col { f32x2 re[RP], im[RP]; };

// RP: row pairs per lane (2 RP rows).
template <int RP>
__global__ void __launch_bounds__(32 * RING_WARPS, 1) jacobi_ring32_kernel(RingArgs A) {
  typedef ring_col<RP> Col;
  __shared__ float part[2][RING_WARPS * 4 * RB];
  __shared__ int table[2 * RING_CTAS];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5, nw = blockDim.x >> 5, K = gridDim.x, cta = blockIdx.x;
  const int rounds = ring_rounds(K);
  for (int r = t; r < rounds; r += blockDim.x) {
    int x, y;
    ring_blocks(K, r, cta, x, y);
    table[r] = x << 16 | y;
  }
  if (A.stall && cta == 0 && t == 0) {
    // test hook (QT_JACOBI_STALL_TEST): a bounded wait on a status word that
    // nothing sets, which must end in QT_ETIMEOUT with the context usable
    int it = 0;
    while (it < A.spin && ld_acquire_gpu(A.flags + QT_FLAG_STALL) == 0) { it++; __nanosleep(64); }
    if (it >= A.spin) atomicExch(A.flags + QT_FLAG_ABORT, 1);
  }
  __syncthreads();
  const int row0 = w * 64 * RP + lane;
  const float nu2 = (float)(A.nu_rel2 * (*A.xnorm2)), big2 = (float)(1e-6 * (*A.xnorm2)), tol2 = A.tol * A.tol;

  auto load = [&](Col (&x)[RB], int blk) {
    float2 v[RB][2 * RP];
#pragma unroll
    for (int j = 0; j < RB; j++) {
      const int c = blk * RB + j;
#pragma unroll
      for (int k = 0; k < 2 * RP; k++) {
        const int r = row0 + 32 * k;
        v[j][k] = (c < A.nn && r < A.mm) ? __ldcg(A.X + r + A.ldx * c) : make_float2(0.f, 0.f);
      }
    }
#pragma unroll
    for (int j = 0; j < RB; j++)
#pragma unroll
      for (int k = 0; k < RP; k++) {
        x[j].re[k] = x2_pack(v[j][2 * k].x, v[j][2 * k + 1].x);
        x[j].im[k] = x2_pack(v[j][2 * k].y, v[j][2 * k + 1].y);
      }
  };
  auto store = [&](const Col (&x)[RB], int blk) {
#pragma unroll
    for (int j = 0; j < RB; j++) {
      const int c = blk * RB + j;
#pragma unroll
      for (int k = 0; k < RP; k++) {
        const float2 re = x2_unpack(x[j].re[k]), im = x2_unpack(x[j].im[k]);
        const int r = row0 + 64 * k;
        if (c < A.nn && r < A.mm) __stcg(A.X + r + A.ldx * c, make_float2(re.x, im.x));
        if (c < A.nn && r + 32 < A.mm) __stcg(A.X + r + 32 + A.ldx * c, make_float2(re.y, im.y));
      }
    }
  };
  auto slot = [&](int blk) { return A.mail + ((size_t)blk * nw + w) * (RB * 2 * RP * 32) + lane; };
  auto publish = [&](const Col (&x)[RB], int blk, unsigned stamp) {
    uint4* m = slot(blk);
#pragma unroll
    for (int j = 0; j < RB; j++)
#pragma unroll
      for (int k = 0; k < RP; k++) {
        const float2 re = x2_unpack(x[j].re[k]), im = x2_unpack(x[j].im[k]);
        mail_store(m + (j * 2 * RP + 2 * k) * 32, re.x, im.x, stamp);
        mail_store(m + (j * 2 * RP + 2 * k + 1) * 32, re.y, im.y, stamp);
      }
  };
  auto fetch = [&](Col (&x)[RB], int blk, unsigned stamp) {
    const uint4* m = slot(blk);
    for (int it = 0;; it++) {
      uint4 v[RB][2 * RP];
#pragma unroll
      for (int j = 0; j < RB; j++)
#pragma unroll
        for (int k = 0; k < 2 * RP; k++) v[j][k] = mail_load(m + (j * 2 * RP + k) * 32);
      bool here = true;
#pragma unroll
      for (int j = 0; j < RB; j++)
#pragma unroll
        for (int k = 0; k < 2 * RP; k++) here = here && v[j][k].y == stamp && v[j][k].w == stamp;
#pragma unroll
      for (int j = 0; j < RB; j++)
#pragma unroll
        for (int k = 0; k < RP; k++) {
          x[j].re[k] = x2_pack(__uint_as_float(v[j][2 * k].x), __uint_as_float(v[j][2 * k + 1].x));
          x[j].im[k] = x2_pack(__uint_as_float(v[j][2 * k].z), __uint_as_float(v[j][2 * k + 1].z));
        }
      if (__all_sync(0xffffffffu, here)) break;
      // given up, here or elsewhere: every wait ends, the sweep runs out and the host reports it
      const bool last = it >= A.spin;
      if (last && lane == 0) atomicExch(A.flags + QT_FLAG_ABORT, 1);
      if (last || ((it & 7) == 7 && *(volatile int*)(A.flags + QT_FLAG_ABORT))) break;
    }
  };
  // of the lane's pairs that rotated (warp 0); relmax is infinite once a column's norm was not finite
  float relmax = 0.f, relbig = 0.f, relkept = 0.f;
  float aa = 0.f, bb = 0.f;                         // squared norms of pair lane / 8
  int buf = 0;
  // `n` sums per pair (v, pair by pair) over the CTA's rows of X; lane l ends
  // with sum l n / 32 of every warp, added in the same order in each
  auto total = [&](auto& v, auto count) -> float {
    constexpr int CNT = decltype(count)::value;  // 16 or 8
    constexpr int SH = 32 / CNT;                 // lanes per sum
    int off = 16;
#pragma unroll
    for (int cnt = CNT; cnt > 1; cnt >>= 1, off >>= 1) {
      const bool up = lane & off;
#pragma unroll
      for (int i = 0; i < cnt / 2; i++) {
        const float send = up ? v[i] : v[i + cnt / 2];
        const float keep = up ? v[i + cnt / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
      }
    }
    float s = v[0];
#pragma unroll
    for (int o = SH / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (nw > 1) {
      // each of a sum's lanes adds every SH-th warp's part, then the lanes meet
      if ((lane & (SH - 1)) == 0) part[buf][w * CNT + lane / SH] = s;
      __syncthreads();
      s = 0.f;
      for (int u = lane & (SH - 1); u < nw; u += SH) s += part[buf][u * CNT + lane / SH];
#pragma unroll
      for (int o = 1; o < SH; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      buf ^= 1;
    }
    return s;
  };
  // four disjoint pairs (p[g], q[g]): the same answer in every warp.  `fresh`:
  // the squared norms from the columns; otherwise as the last rotations left
  // them (a round measures them once and rotates each column three times more)
  auto rotate = [&](Col (&p)[RB], Col (&q)[RB], auto fresh) -> bool {
    constexpr bool FRESH = decltype(fresh)::value;
    constexpr int PER = FRESH ? 4 : 2;
    float v[PER * RB];
#pragma unroll
    for (int g = 0; g < RB; g++) {
      f32x2 na = 0, nb = 0, gr = 0, g1 = 0, g2 = 0;
#pragma unroll
      for (int k = 0; k < RP; k++) {
        const f32x2 xr = p[g].re[k], xi = p[g].im[k], yr = q[g].re[k], yi = q[g].im[k];
        if (FRESH) {
          na = x2_fma(xr, xr, x2_fma(xi, xi, na));
          nb = x2_fma(yr, yr, x2_fma(yi, yi, nb));
        }
        gr = x2_fma(xr, yr, x2_fma(xi, yi, gr));
        g1 = x2_fma(xr, yi, g1);
        g2 = x2_fma(xi, yr, g2);
      }
      v[PER * g] = x2_sum(gr);
      v[PER * g + 1] = x2_sum(g1) - x2_sum(g2);
      if (FRESH) {
        v[PER * g + 2] = x2_sum(na);
        v[PER * g + 3] = x2_sum(nb);
      }
    }
    const float s = total(v, std::integral_constant<int, PER * RB>());
    const int base = lane & ~7;
    const float gr = __shfl_sync(0xffffffffu, s, base), gi = __shfl_sync(0xffffffffu, s, base + 8 / PER);
    if (FRESH) {
      aa = __shfl_sync(0xffffffffu, s, base + 4);
      bb = __shfl_sync(0xffffffffu, s, base + 6);
      // (every comparison below is false for a NaN: its column would count as converged)
      if (!(aa <= FLT_MAX && bb <= FLT_MAX)) relmax = INFINITY;
    }
    const float ra = rsqrtf(aa), rb = rsqrtf(bb);
    const float er = gr * ra * rb, ei = gi * ra * rb;  // e^{i phi} times the cosine
    const float c2 = fmaf(er, er, ei * ei);
    const bool rot = aa > nu2 && bb > nu2 && c2 > tol2;
    const unsigned on = __ballot_sync(0xffffffffu, rot);
    if (!on) return false;
    float c = 1.f, sr = 0.f, si = 0.f;
    if (rot) {
      const float rc = rsqrtf(c2);
      const float zeta = 0.5f * ((bb - aa) * ra * rb) * rc;
      const float az = fabsf(zeta);
      const float tt = copysignf(__fdividef(1.f, az > 1e6f ? 2.f * az : az + sqrtf(fmaf(az, az, 1.f))), zeta);
      const float c0 = rsqrtf(fmaf(tt, tt, 1.f));
      const float s0 = c0 * tt * rc;
      const float sr0 = s0 * er, si0 = s0 * ei;
      // the defect 1 - |(c0, sr0, si0)|^2, each step one rounding of a number <= 1
      const float h = 0.5f * fmaf(-si0, si0, fmaf(-sr0, sr0, fmaf(-c0, c0, 1.f)));
      c = fmaf(h, c0, c0);
      sr = fmaf(h, sr0, sr0);
      si = fmaf(h, si0, si0);
      const float rel = fminf(c2 * rc, 1.f);
      if (w == 0) {
        relmax = fmaxf(relmax, rel);
        if (aa > big2 && bb > big2) relbig = fmaxf(relbig, rel);
        if (fmaxf(aa, bb) > A.keep2) relkept = fmaxf(relkept, rel);
      }
      const float d = tt * rel * (aa * ra) * (bb * rb);  // t |gamma|
      aa = fmaxf(aa - d, 0.f);
      bb = bb + d;
    }
#pragma unroll
    for (int g = 0; g < RB; g++) {
      const float cg = __shfl_sync(0xffffffffu, c, 8 * g);
      const float srg = __shfl_sync(0xffffffffu, sr, 8 * g), sig = __shfl_sync(0xffffffffu, si, 8 * g);
      if (!((on >> (8 * g)) & 1)) continue;
      const f32x2 cc = x2_pack(cg, cg), ss = x2_pack(srg, srg), ns = x2_pack(-srg, -srg), ii = x2_pack(sig, sig),
                  ni = x2_pack(-sig, -sig);
#pragma unroll
      for (int k = 0; k < RP; k++) {
        // x_p' = c x_p - conj(se) x_q ;  x_q' = se x_p + c x_q
        const f32x2 xr = p[g].re[k], xi = p[g].im[k], yr = q[g].re[k], yi = q[g].im[k];
        p[g].re[k] = x2_fma(cc, xr, x2_fma(ns, yr, x2_mul(ni, yi)));
        p[g].im[k] = x2_fma(cc, xi, x2_fma(ns, yi, x2_mul(ii, yr)));
        q[g].re[k] = x2_fma(cc, yr, x2_fma(ss, xr, x2_mul(ni, xi)));
        q[g].im[k] = x2_fma(cc, yi, x2_fma(ss, xi, x2_mul(ii, xr)));
      }
    }
    return true;
  };

  const std::true_type fresh;
  const std::false_type tracked;
  Col xa[RB], xb[RB];
  int ka = table[0] >> 16, kb = table[0] & 0xffff;
  load(xa, ka);
  load(xb, kb);
  int rotated = 0;
  for (int r = 0; r < rounds; r++) {
    bool ch = false;
    if (r == 0) {
      // the pairs inside each block, once a sweep: columns 1, 2, 3 of each move
      // round one place per step
#pragma unroll 1
      for (int st = 0; st < 3; st++) {
        Col p[RB] = {xa[0], xa[2], xb[0], xb[2]}, q[RB] = {xa[1], xa[3], xb[1], xb[3]};
        ch |= rotate(p, q, fresh);
        xa[0] = p[0]; xa[1] = p[1]; xa[2] = q[1]; xa[3] = q[0];
        xb[0] = p[2]; xb[1] = p[3]; xb[2] = q[3]; xb[3] = q[2];
      }
    }
    // the cross pairs; b's columns move one place per step
    ch |= rotate(xa, xb, fresh);
#pragma unroll 1
    for (int st = 1; st < RB; st++) {
      const Col f = xb[0];
      xb[0] = xb[1]; xb[1] = xb[2]; xb[2] = xb[3]; xb[3] = f;
      bb = __shfl_sync(0xffffffffu, bb, (lane + 8) & 31);
      ch |= rotate(xa, xb, tracked);
    }
    {
      const Col f = xb[0];
      xb[0] = xb[1]; xb[1] = xb[2]; xb[2] = xb[3]; xb[3] = f;
    }
    rotated += ch;
    if (r + 1 == rounds) break;
    // ---- exchange: publish what leaves, then wait for what comes
    const int na = table[r + 1] >> 16, nb = table[r + 1] & 0xffff;
    const unsigned stamp = A.g0 + r + 1;
    if (kb == na || ka == nb) {
#pragma unroll
      for (int j = 0; j < RB; j++) { const Col f = xa[j]; xa[j] = xb[j]; xb[j] = f; }
      const int f = ka; ka = kb; kb = f;
    }
    const bool fa = na != ka, fb = nb != kb;
    if (fa) publish(xa, ka, stamp);
    if (fb) publish(xb, kb, stamp);
    ka = na;
    kb = nb;
    if (fa) fetch(xa, ka, stamp);
    if (fb) fetch(xb, kb, stamp);
  }
  store(xa, ka);
  store(xb, kb);
  if (A.dnorm) {
    float v[2 * RB];
#pragma unroll
    for (int j = 0; j < RB; j++) {
      f32x2 f = 0, g = 0;
#pragma unroll
      for (int k = 0; k < RP; k++) {
        f = x2_fma(xa[j].re[k], xa[j].re[k], x2_fma(xa[j].im[k], xa[j].im[k], f));
        g = x2_fma(xb[j].re[k], xb[j].re[k], x2_fma(xb[j].im[k], xb[j].im[k], g));
      }
      v[j] = x2_sum(f);
      v[RB + j] = x2_sum(g);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2 * RB; j++) {
      for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
      if (lane == 0) part[0][w * 2 * RB + j] = v[j];
    }
    __syncthreads();
    if (t < 2 * RB) {
      float f = 0.f;
      for (int u = 0; u < nw; u++) f += part[0][u * 2 * RB + t];
      const int c = (t < RB ? ka : kb) * RB + t % RB;
      if (c < A.nn) A.dnorm[c] = f;
    }
  }
  if (w == 0) {
    for (int o = 16; o > 0; o >>= 1) {
      relmax = fmaxf(relmax, __shfl_xor_sync(0xffffffffu, relmax, o));
      relbig = fmaxf(relbig, __shfl_xor_sync(0xffffffffu, relbig, o));
      relkept = fmaxf(relkept, __shfl_xor_sync(0xffffffffu, relkept, o));
    }
    if (lane == 0) {
      if (relmax > 1.f) atomicOr(&A.flags[QT_FLAG_NONFINITE], 1);
      if (rotated) atomicAdd(&A.flags[QT_FLAG_ROTATED], rotated);
      if (relmax > 0.f) atomicMax(&A.flags[QT_FLAG_OFFMAX], __float_as_int(relmax));
      if (relbig > 0.f) atomicMax(&A.flags[QT_FLAG_OFFBIG], __float_as_int(relbig));
      if (relkept > 0.f) atomicMax(&A.flags[QT_FLAG_OFFKEPT], __float_as_int(relkept));
    }
  }
}

// ||X||_F^2 in FP64, one CTA per column, added into *out.
template <typename TS>
__global__ void frob_kernel(const TS* __restrict__ X, int64_t ldx, int mm, double* out) {
  double s = 0;
  for (int i = threadIdx.x; i < mm; i += blockDim.x) {
    const double re = X[i + ldx * blockIdx.x].x, im = X[i + ldx * blockIdx.x].y;
    s = fma(re, re, s);
    s = fma(im, im, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

template <typename TS> struct gram_of;
template <> struct gram_of<double2> { typedef double type; };
template <> struct gram_of<float2> { typedef float type; };

}  // namespace

int qt_jacobi_layout(int64_t mm, int64_t nn, int* nb_out, int* chunks_out) {
  int nb = (int)((nn + JW - 1) / JW);
  if (nb % 2) nb++;
  if (nb < 2) nb = 2;
  const int pairs = nb / 2;
  // enough CTAs to cover the 152 SMs about twice, each chunk at least 128 rows
  int chunks = (int)((2 * 152 + pairs - 1) / pairs);
  chunks = std::max(1, std::min<int>(chunks, (int)((mm + 127) / 128)));
  *nb_out = nb;
  *chunks_out = chunks;
  // double2 entries: partial Grams, ||X||_F^2, two round slots of one 16x16
  // unitary per pair, two round slots of the pairs' rotate flags
  return pairs * chunks * NGRAM + 1 + pairs * NGRAM + pairs;
}

// Cluster shape of the one-launch FP32 round: the smallest cluster (<= 8 CTAs)
// whose row slice of the 16 pair columns fits in FUSED_SMEM bytes of shared
// memory, widened while the grid would leave SMs idle.  0 = does not fit.
constexpr size_t FUSED_SMEM = 100 * 1024;
static int fused_shape(int64_t mm, int pairs, int* rows_c, int* lds, size_t* smem) {
  const size_t elem = sizeof(float2);
  int csize = 0;
  for (int c = 1; c <= 8; c *= 2) {
    const int64_t rc = (mm + c - 1) / c;
    if ((size_t)(((rc + 15) / 16) * 16 + 1) * JC * elem <= FUSED_SMEM) { csize = c; break; }
  }
  if (csize == 0) return 0;
  while (csize < 8 && (int64_t)pairs * csize < 152 && (mm + 2 * csize - 1) / (2 * csize) >= 64) csize *= 2;
  // QT_JACOBI_CLUSTER=c (1, 2, 4 or 8) overrides the cluster size when the slice still fits
  if (const char* env = std::getenv("QT_JACOBI_CLUSTER")) {
    const int c = std::atoi(env);
    const int64_t rc = (mm + c - 1) / c;
    if ((c == 1 || c == 2 || c == 4 || c == 8) && (size_t)(((rc + 15) / 16) * 16 + 1) * JC * elem <= 200 * 1024)
      csize = c;
  }
  const int64_t rc = (mm + csize - 1) / csize;
  *rows_c = (int)rc;
  *lds = (int)(((rc + 15) / 16) * 16 + 1);  // odd multiple-of-16-plus-one stride: conflict-free Gram reads
  *smem = (size_t)(*lds) * JC * elem;
  return csize;
}

static int launch_pair_round(qt_handle* h, int csize, int pairs, size_t smem, float2* X, int64_t ldx, int mm, float2* V,
                             int64_t ldv, int nn, int nb, int round, int xrows_c, int vrows_c, int lds, double tol,
                             double tol_inner, double nu_rel2, const double* xnorm2, int max_inner,
                             unsigned long long* phase_ns) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)(pairs * csize));
  lc.blockDim = dim3(NT);
  lc.dynamicSmemBytes = smem;
  lc.stream = h->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  if (h->prof) qt_prof_before(h, "pair_round_kernel");
  const cudaError_t e = cudaLaunchKernelEx(&lc, pair_round_kernel, X, ldx, mm, V, ldv, nn, nb, round, csize,
                                           xrows_c, vrows_c, lds, tol, tol_inner, nu_rel2, xnorm2, h->d_flags, max_inner,
                                           phase_ns);
  if (h->prof) qt_prof_after(h);
  h->launches++;
  if (e != cudaSuccess) return qt_fail(h, QT_ECUDA, std::string("launch pair_round_kernel: ") + cudaGetErrorString(e));
  return QT_OK;
}

// Shape of the FP64 round: the widest cluster (<= 8 CTAs) that keeps the grid
// on the chip at once (152 SMs) with at least 8 rows of X per CTA, wider still
// while the row slices do not fit.  Rows and not columns are spread because
// the FP64 work of a CTA is its rows times the pair's 16 x 16 entries.
// 128 x 128 with V (8 pairs), 10 sweeps: clusters of 8 9.9 ms an update, of 16
// (8 rows each) 11.3 ms -- what the rotation gains, the launch of the wider
// clusters loses.
struct round64_shape {
  int csize = 0, xrows = 0, vrows = 0, lds = 0, vboth = 0;
  size_t smem = 0;
};
constexpr size_t R64_SMEM = 200 * 1024;
static bool round64_fill(int64_t mm, int64_t vn, int c, round64_shape* s) {
  s->csize = c;
  s->xrows = (int)((mm + c - 1) / c);
  s->vrows = (int)((vn + c - 1) / c);
  s->lds = std::max(s->xrows, s->vrows) | 1;  // odd: columns start in different banks
  const size_t slice = (size_t)s->lds * JC * sizeof(double2);
  s->vboth = vn > 0 && 2 * slice <= R64_SMEM;
  s->smem = slice * (s->vboth ? 2 : 1);
  return s->smem <= R64_SMEM;
}
static round64_shape shape_round64(int64_t mm, int64_t vn, int pairs) {
  round64_shape s, best;
  for (int c = 1; c <= 8; c *= 2) {
    if (!round64_fill(mm, vn, c, &s)) continue;
    const bool wider = c > 1 && pairs * c <= 152 && s.xrows >= 8;
    if (best.csize && !wider) break;
    best = s;
  }
  // QT_JACOBI_CLUSTER=c (1, 2, 4 or 8) overrides the cluster size where the slice fits
  if (const char* env = std::getenv("QT_JACOBI_CLUSTER")) {
    const int c = std::atoi(env);
    if ((c == 1 || c == 2 || c == 4 || c == 8) && round64_fill(mm, vn, c, &s)) best = s;
  }
  return best;
}

static int launch_pair_round64(qt_handle* h, const round64_shape& sh, int pairs, double2* X, int64_t ldx, int mm,
                               double2* V, int64_t ldv, int nn, int nb, int round, double tol, double nu_rel2,
                               const double* xnorm2, int max_inner, unsigned long long* phase_ns) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)(pairs * sh.csize));
  lc.blockDim = dim3(NT64);
  lc.dynamicSmemBytes = sh.smem;
  lc.stream = h->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)sh.csize;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  if (h->prof) qt_prof_before(h, "pair_round64_kernel");
  const cudaError_t e = cudaLaunchKernelEx(&lc, pair_round64_kernel, X, ldx, mm, V, ldv, nn, nb, round, sh.csize,
                                           sh.xrows, sh.vrows, sh.lds, sh.vboth, tol, nu_rel2, xnorm2, h->d_flags,
                                           max_inner, phase_ns);
  if (h->prof) qt_prof_after(h);
  h->launches++;
  if (e != cudaSuccess)
    return qt_fail(h, QT_ECUDA, std::string("launch pair_round64_kernel: ") + cudaGetErrorString(e));
  return QT_OK;
}

// Whether one CTA per pair of jacobi_sweep32_kernel can be resident at once
// (the cooperative launch needs it).
static bool sweep32_fits(qt_handle* h, int pairs) {
  static int max_ctas = -1;
  if (max_ctas < 0) {
    int dev = 0, coop = 0, sms = 0, per_sm[2] = {0, 0};
    auto resident = [](auto kernel, int* ctas) {
      return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PS_SMEM) == cudaSuccess &&
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, kernel, NTG, PS_SMEM) == cudaSuccess;
    };
    max_ctas = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        resident(jacobi_sweep32_kernel<false>, &per_sm[0]) && resident(jacobi_sweep32_kernel<true>, &per_sm[1]))
      max_ctas = std::min(per_sm[0], per_sm[1]) * sms;
    cudaGetLastError();
  }
  (void)h;
  return pairs <= max_ctas;
}

static int launch_sweep32(qt_handle* h, int pairs, float2* x0, float2* x1, int64_t ldx, int mm, float2* v0,
                          float2* v1, int64_t ldv, int nn, int nb, int g0, int has_prev, double tol, float tol_inner,
                          double nu_rel2, const double* xnorm2, float2* wbuf, int* rotbuf, int* done, int max_inner,
                          int max_inner0, int nsweeps, float keep2, float* dnorm, unsigned long long* phase_ns,
                          int halves, float2* gx, int* xflag) {
  // row split of the two halves of a pair: at a multiple of 32 rows, never
  // past the last row (a V of fewer than 32 rows belongs to half 0 alone)
  const int row_mid = std::min(((mm / 2 + 31) / 32) * 32, mm);
  const int vrow_mid = std::min(((nn / 2 + 31) / 32) * 32, nn);
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)(pairs * halves));
  lc.blockDim = dim3(NTG);
  lc.dynamicSmemBytes = PS_SMEM;
  lc.stream = h->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  // QT_JACOBI_STALL_TEST=N (tests only): CTA 0 waits at most N polls on a
  // status word nothing sets, and every round wait is limited to N polls
  const char* stall_env = std::getenv("QT_JACOBI_STALL_TEST");
  const int stall_polls = stall_env ? std::atoi(stall_env) : 0;
  const int spin = stall_polls > 0 ? stall_polls : PS_SPIN;
  const int stall = stall_polls > 0 ? 1 : 0;
  if (h->prof) qt_prof_before(h, "jacobi_sweep32_kernel");
  const auto kernel = nsweeps > 1 ? jacobi_sweep32_kernel<true> : jacobi_sweep32_kernel<false>;
  const cudaError_t e =
      cudaLaunchKernelEx(&lc, kernel, x0, x1, ldx, mm, v0, v1, ldv, nn, nb, g0, has_prev, tol, tol_inner, nu_rel2,
                         xnorm2, wbuf, rotbuf, done, h->d_flags, max_inner, max_inner0, nsweeps, keep2, dnorm, phase_ns,
                         spin, stall, halves, row_mid, vrow_mid, gx, xflag);
  if (h->prof) qt_prof_after(h);
  h->launches++;
  if (e != cudaSuccess)
    return qt_fail(h, QT_ECUDA, std::string("launch jacobi_sweep32_kernel: ") + cudaGetErrorString(e));
  return QT_OK;
}

// Launch shape of jacobi_ring32_kernel: two rows per lane up to 512 rows, then
// four, so that a CTA has up to 8 warps, 16 only from 1024 rows on (a warp's
// share of a round beside its products -- shuffles, rotation, barrier -- is the
// same however few rows it holds).
struct ring_shape {
  int rows = 0, warps = 0, ctas = 0;  // rows per lane
};
static const void* ring_kernel(int rows) {
  return rows == 2 ? (const void*)jacobi_ring32_kernel<1> : (const void*)jacobi_ring32_kernel<2>;
}
// ctas = 0 where it does not apply: more rows than 16 warps hold, or more
// blocks than the resident CTAs.  QT_JACOBI_RING=0 turns it off.
static ring_shape shape_ring32(int64_t mm, int64_t nn) {
  ring_shape s;
  const char* env = std::getenv("QT_JACOBI_RING");
  if (env && env[0] == '0') return s;
  s.rows = mm <= 512 ? 2 : 4;
  const int64_t warps = (mm + 32 * s.rows - 1) / (32 * s.rows), ctas = ((nn + RB - 1) / RB + 1) / 2;
  if (warps > RING_WARPS || ctas > RING_CTAS) return s;
  s.warps = (int)warps;
  int dev = 0, coop = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ring_kernel(s.rows), 32 * s.warps, 0) != cudaSuccess) {
    cudaGetLastError();
    return s;
  }
  if (ctas <= (int64_t)per_sm * sms) s.ctas = (int)ctas;
  return s;
}

static int launch_ring32(qt_handle* h, const ring_shape& s, RingArgs a) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)s.ctas);
  lc.blockDim = dim3(32 * s.warps);
  lc.stream = h->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  // QT_JACOBI_STALL_TEST=N (tests only): CTA 0 waits at most N polls on a
  // status word nothing sets, and every block wait is limited to N polls
  const char* stall_env = std::getenv("QT_JACOBI_STALL_TEST");
  const int stall_polls = stall_env ? std::atoi(stall_env) : 0;
  a.spin = stall_polls > 0 ? stall_polls : PS_SPIN;
  a.stall = stall_polls > 0 ? 1 : 0;
  void* args[] = {&a};
  if (h->prof) qt_prof_before(h, "jacobi_ring32_kernel");
  const cudaError_t e = cudaLaunchKernelExC(&lc, ring_kernel(s.rows), args);
  if (h->prof) qt_prof_after(h);
  h->launches++;
  if (e != cudaSuccess)
    return qt_fail(h, QT_ECUDA, std::string("launch jacobi_ring32_kernel: ") + cudaGetErrorString(e));
  return QT_OK;
}

template <typename TS>
int qt_jacobi_svd_ws(qt_handle* h, TS* X, int64_t mm, int64_t nn, int64_t ldx, TS* V, int64_t ldv, double tol,
                     int max_sweeps, int* sweeps_out, double2* parts, double nu_rel_in, int keep_count,
                     bool pairwise) {
  typedef typename gram_of<TS>::type TG;
  if (mm < nn) return qt_fail(h, QT_EINVAL, "jacobi: needs rows >= columns");
  if (V) QT_TRY(qt_set_identity<TS>(h, V, nn, ldv));
  *sweeps_out = 0;
  if (nn <= 1) return QT_OK;
  int nb = 0, chunks = 1;
  qt_jacobi_layout(mm, nn, &nb, &chunks);
  const int pairs = nb / 2, rounds = nb - 1;
  const int xrows = (int)(((mm + chunks - 1) / chunks + JR - 1) / JR * JR);
  const int vrows = (int)(((nn + chunks - 1) / chunks + JR - 1) / JR * JR);
  const dim3 grid(pairs, chunks);
  // the last workspace entry holds ||X||_F^2 (rotation-invariant); the noise
  // floor nu (below) is relative to ||X||_F
  double* xnorm2 = reinterpret_cast<double*>(parts + (size_t)pairs * chunks * NGRAM);
  double2* wbuf = parts + (size_t)pairs * chunks * NGRAM + 1;
  int* rotf = reinterpret_cast<int*>(wbuf + (size_t)pairs * NGRAM);
  {
    // ||X||_F^2 over the nn columns (ldx may exceed mm)
    QT_CHECK_CUDA(h, cudaMemsetAsync(xnorm2, 0, sizeof(double), h->stream));
    QT_LAUNCH(h, frob_kernel<TS>, (unsigned)nn, 256, 0, X, ldx, (int)mm, xnorm2);
  }
  const bool fp32 = sizeof(typename real_of<TS>::type) == 4;
  const double u = fp32 ? 5.96e-8 : 1.11e-16;
  // Frozen-column threshold nu (relative to ||X||_F).  FP64: 4 sqrt(rows) u.
  // FP32 default: 4 u, so that the weight of the frozen columns stays below
  // the chosen mode's noise floor and the tail rule can resolve values near
  // it.  Columns between 4 u and sqrt(rows) u are rounding noise of FP32
  // products that keep rotating with O(1) cosines for tens of sweeps; callers
  // whose rank is decided far above them (a chi_max cap, a cutoff well above
  // the floor) pass nu_rel = sqrt(rows) u and save those sweeps.
  const double nu_rel = nu_rel_in > 0 ? nu_rel_in
                        : (fp32 ? 4.0 * u : 4.0 * std::sqrt((double)std::max<int64_t>(mm, 16)) * u);
  const double nu_rel2 = nu_rel * nu_rel;
  // Round implementation (cfg.jacobi_kernel): FP32 storage by default rotates
  // register-resident columns in one launch per sweep where the caller takes
  // pairwise rotations, else (and with more columns than that holds) runs the
  // Gram-based sweep kernel, beyond its size two launches per round (Gram + pair
  // solver, then the rotation; also 3); 2 asks for the one-launch cluster
  // round, 1 for the three-kernel round.  FP64 storage uses the one-launch
  // round where a pair's rows fit a cluster's shared memory.
  // A caller that allows few sweeps gets the rounds that need the fewest, at the
  // price of their time: the Gram-based sweep kernel instead of pairwise
  // rotations (4 or 5 sweeps of a capped sketch where those take 5 to 7); FP64
  // pair solves of up to 12 and 3 inner sweeps instead of one (up to 24 columns 4
  // to 6 sweeps instead of 6 or 7), and below three sweeps the three-kernel
  // round, whose FP64 angles finish a single pair of blocks at once.  (The
  // default limit is 80.)
  const bool few = max_sweeps < 12;
  const int jk = !fp32 && max_sweeps < 3 ? 1 : h->cfg.jacobi_kernel;
  const ring_shape ring = fp32 && jk == 0 && pairwise && !V && !few ? shape_ring32(mm, nn) : ring_shape();
  const bool sweep_kernel = fp32 && jk == 0 && !ring.ctas && sweep32_fits(h, pairs);
  const bool two_launch = fp32 && (jk == 3 || (jk == 0 && !sweep_kernel && !ring.ctas));
  int xrows_c = 0, lds = 0;
  size_t smem = 0;
  const bool one_launch = jk != 1 && !two_launch && !sweep_kernel && !ring.ctas;
  const round64_shape r64 = one_launch && !fp32 ? shape_round64(mm, V ? nn : 0, pairs) : round64_shape();
  const int csize = !one_launch ? 0 : fp32 ? fused_shape(mm, pairs, &xrows_c, &lds, &smem) : r64.csize;
  // two-launch shape: one row per rotation thread, about eight CTAs per SM
  int achunks = std::max(1, std::min<int>((8 * 152 + pairs - 1) / pairs, (int)((mm + NT - 1) / NT)));
  const int axrows = (int)(((mm + achunks - 1) / achunks + 31) / 32 * 32);
  const int avrows = (int)(((nn + achunks - 1) / achunks + 31) / 32 * 32);
  const int vrows_c = csize ? (int)((nn + csize - 1) / csize) : 0;
  // the inner eigen-solve is driven well below the outer threshold so that the
  // rounding of the applied rotation cannot leave the pair just above `tol`
  const double tol_inner = fp32 ? tol / 16.0 : std::min(tol, 1e-14);
  if (csize && fp32)
    QT_CHECK_CUDA(h, cudaFuncSetAttribute(pair_round_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (csize && !fp32)
    QT_CHECK_CUDA(h, cudaFuncSetAttribute(pair_round64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)r64.smem));
  // QT_JACOBI_TRACE=1 in the environment prints one line per sweep to stderr;
  // QT_JACOBI_PHASES=1 adds the average time per phase of the one-launch
  // rounds at the end (CTA 0 of each cluster / the others); a handle without
  // a pool (the allocation-free entry point's) allocates nothing and skips them
  static const bool trace = std::getenv("QT_JACOBI_TRACE") != nullptr;
  static const bool phases = std::getenv("QT_JACOBI_PHASES") != nullptr;
  unsigned long long* phase_ns = nullptr;
  qt_scratch pscratch(h);
  if (phases && h->pool && (csize || two_launch || sweep_kernel)) {
    QT_TRY(pscratch.get(&phase_ns, 16));
    QT_CHECK_CUDA(h, cudaMemsetAsync(phase_ns, 0, 16 * sizeof(unsigned long long), h->stream));
  }
  // sweep kernel: ping-pong copies of X and V, the round counter, and
  // whether the last round's unitaries are still to be applied
  TS* X1 = nullptr;
  TS* V1 = nullptr;
  int* done = reinterpret_cast<int*>(parts);
  int gcount = 0;
  bool pending = false;
  // kept-set convergence (keep_count > 0, sweep kernel): the last round of
  // each sweep reports the squared column norms; a column within a factor
  // keep_margin of the keep_count-th largest norm counts as kept
  static const double keep_margin =
      std::getenv("QT_JACOBI_KEEP_MARGIN") ? std::atof(std::getenv("QT_JACOBI_KEEP_MARGIN")) : 0.25;
  static const bool keep_stop = !std::getenv("QT_JACOBI_KEEP_STOP") || std::atoi(std::getenv("QT_JACOBI_KEEP_STOP"));
  const bool keep_track = (sweep_kernel || ring.ctas) && keep_count > 0 && keep_count < nn;
  float* dnorm = nullptr;
  std::vector<float> hnorm;
  float keep2 = 0.f;
  double prev_tail2 = -1.0, prev_change = -1.0;
  static const double keep_tol =
      std::getenv("QT_JACOBI_KEEP_TOL") ? std::atof(std::getenv("QT_JACOBI_KEEP_TOL")) : 1e-3;
  // Two CTAs per pair (each holding half of the rows) when the doubled grid
  // is still resident and each half has rows to work on; QT_JACOBI_HALVES=1
  // keeps one CTA per pair.  The halves run on their own copies of the round
  // flags, unitaries and rotate decisions, and exchange partial Grams.
  const int halves_env = std::getenv("QT_JACOBI_HALVES") ? std::atoi(std::getenv("QT_JACOBI_HALVES")) : 2;
  const int halves = (sweep_kernel && halves_env == 2 && mm >= 512 && sweep32_fits(h, 2 * pairs)) ? 2 : 1;
  float2* gx = nullptr;
  int* xflag = nullptr;
  if (sweep_kernel && halves == 2) {
    double2* wb2;
    int *rf2, *dn2;
    QT_TRY(pscratch.get(&wb2, (size_t)2 * pairs * NGRAM));  // 2 halves x 2 round slots x pairs x NGRAM float2
    QT_TRY(pscratch.get(&rf2, (size_t)4 * pairs));
    QT_TRY(pscratch.get(&dn2, (size_t)2 * pairs));
    QT_TRY(pscratch.get(&xflag, (size_t)2 * pairs));
    QT_TRY(pscratch.get(&gx, (size_t)2 * pairs * 2 * 160));
    wbuf = wb2;
    rotf = rf2;
    done = dn2;
    QT_CHECK_CUDA(h, cudaMemsetAsync(xflag, 0xff, sizeof(int) * 2 * pairs, h->stream));
  }
  if (sweep_kernel) {
    QT_TRY(pscratch.get(&X1, (size_t)ldx * nn));
    if (V) QT_TRY(pscratch.get(&V1, (size_t)ldv * nn));
    QT_CHECK_CUDA(h, cudaMemsetAsync(done, 0xff, sizeof(int) * pairs * halves, h->stream));
  }
  uint4* ring_mail = nullptr;
  if (ring.ctas) {
    const size_t n = (size_t)2 * ring.ctas * ring.warps * RB * ring.rows * 32;
    QT_TRY(pscratch.get(&ring_mail, n));
    QT_CHECK_CUDA(h, cudaMemsetAsync(ring_mail, 0, sizeof(uint4) * n, h->stream));  // round 0: nothing sent
  }
  if (keep_track) {
    QT_TRY(pscratch.get(&dnorm, (size_t)nn));
    hnorm.resize(nn);
  }
  const int sweep_rounds = ring.ctas ? ring_rounds(ring.ctas) : rounds;
  const int pair_cols = ring.ctas ? 2 * RB : JC;  // columns of a CTA's pair of blocks
  int sweep = 0;
  for (; sweep < max_sweeps; sweep++) {
    // FP32 storage: up to 2 inner sweeps of the pair solver in the first two
    // outer sweeps (measured fastest); once the pairs are close to orthogonal
    // one inner sweep of rotations reduces them quadratically and the outer
    // test decides convergence.  FP64 storage: one throughout (1, 2, 4 and 12
    // in the first two took 10.9, 11.3, 13.6 and 14.0 ms at 128 x 128).
    // QT_JACOBI_INNER0 / QT_JACOBI_INNER override the two caps.
    static const char *inner_env = std::getenv("QT_JACOBI_INNER"), *inner_env0 = std::getenv("QT_JACOBI_INNER0");
    const int inner_cap = inner_env ? std::atoi(inner_env) : !fp32 && few ? 3 : 1;
    const int inner_cap0 = inner_env0 ? std::atoi(inner_env0) : fp32 ? 2 : few ? MAX_INNER : 1;
    const int max_inner = std::max(1, std::min(sweep < 2 ? inner_cap0 : inner_cap, MAX_INNER));
    // The sweep kernel goes on to the next sweep by itself where "no pair
    // rotated" is the only rule that ends the sweeps: a launch, its status
    // copy and synchronisation per sweep cost 25 us each, a sweep of 64 x 64
    // 100 us.  (The trace wants every sweep's figures.)
    const bool multi = sweep_kernel && !keep_track && !trace && max_sweeps > 1;
    const int inner_rest = std::max(1, std::min(inner_cap, MAX_INNER));
    QT_CHECK_CUDA(h, cudaMemsetAsync(h->d_flags, 0, sizeof(int) * QT_FLAG_COUNT, h->stream));
    if (sweep_kernel) {
      if constexpr (sizeof(typename real_of<TS>::type) == 4) {
        QT_TRY(launch_sweep32(h, pairs, (float2*)X, (float2*)X1, ldx, (int)mm, (float2*)V, (float2*)V1, ldv, (int)nn,
                              nb, gcount, pending ? 1 : 0, tol, (float)tol_inner, nu_rel2, (const double*)xnorm2,
                              (float2*)wbuf, rotf, done, multi ? inner_rest : max_inner, max_inner, multi ? max_sweeps : 1,
                              keep2, dnorm, phase_ns, halves, gx, xflag));
      }
      pending = true;
    }
    if (ring.ctas) {
      if constexpr (sizeof(typename real_of<TS>::type) == 4) {
        RingArgs a = {};
        a.X = (float2*)X; a.ldx = ldx; a.mm = (int)mm; a.nn = (int)nn; a.g0 = gcount; a.tol = (float)tol; a.nu_rel2 = nu_rel2; a.xnorm2 = xnorm2;
        a.mail = ring_mail; a.flags = h->d_flags; a.keep2 = keep2; a.dnorm = dnorm;
        QT_TRY(launch_ring32(h, ring, a));
      }
      gcount += sweep_rounds;
    }
    for (int r = 0; r < rounds && !sweep_kernel && !ring.ctas; r++) {
      if (two_launch) {
        if constexpr (sizeof(typename real_of<TS>::type) == 4) {
          QT_LAUNCH(h, pair_eig32_kernel, pairs, NTG, 0, (const float2*)X, ldx, (int)mm, (int)nn, nb, r, tol,
                    (float)tol_inner, nu_rel2, (const double*)xnorm2, (float2*)wbuf, rotf, h->d_flags, max_inner,
                    phase_ns);
          QT_LAUNCH(h, pair_apply32_kernel, dim3(pairs, achunks), NT, 0, (float2*)X, ldx, (int)mm, (float2*)V, ldv,
                    (int)nn, nb, r, axrows, avrows, (const float2*)wbuf, (const int*)rotf);
        }
        continue;
      }
      if (csize) {
        if constexpr (sizeof(typename real_of<TS>::type) == 4)
          QT_TRY(launch_pair_round(h, csize, pairs, smem, X, ldx, (int)mm, V, ldv, (int)nn, nb, r, xrows_c, vrows_c,
                                   lds, tol, tol_inner, nu_rel2, xnorm2, max_inner, phase_ns));
        else
          QT_TRY(launch_pair_round64(h, r64, pairs, X, ldx, (int)mm, V, ldv, (int)nn, nb, r, tol, nu_rel2, xnorm2,
                                     max_inner, phase_ns));
        continue;
      }
      QT_LAUNCH(h, (gram_kernel<TS, TG>), grid, NT, 0, X, ldx, (int)mm, (int)nn, nb, r, xrows, parts);
      QT_LAUNCH(h, eig_kernel, pairs, NT, 0, (int)nn, nb, r, chunks, (const double2*)parts, tol, nu_rel2,
                (const double*)xnorm2, wbuf, rotf, h->d_flags);
      QT_LAUNCH(h, apply_kernel<TS>, grid, NT, 0, X, ldx, (int)mm, V, ldv, (int)nn, nb, r, xrows, vrows,
                (const double2*)wbuf, (const int*)rotf);
    }
    QT_CHECK_CUDA(h, cudaMemcpyAsync(h->h_flags, h->d_flags, sizeof(int) * QT_FLAG_COUNT, cudaMemcpyDeviceToHost,
                                     h->stream));
    if (keep_track)
      QT_CHECK_CUDA(h, cudaMemcpyAsync(hnorm.data(), dnorm, sizeof(float) * nn, cudaMemcpyDeviceToHost, h->stream));
    QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
    const int ran = multi ? std::max(1, h->h_flags[QT_FLAG_SWEEPS]) : 1;  // sweeps of this launch
    if (sweep_kernel) gcount += ran * rounds;
    sweep += ran - 1;
    {
      const double es = (double)sizeof(TS);
      h->work_jacobi_rounds += ran * sweep_rounds;
      h->work_jacobi_pairs += h->h_flags[QT_FLAG_ROTATED];
      h->work_jacobi_inner += h->h_flags[QT_FLAG_INNER];
      const double read = (double)ran * sweep_rounds * (double)mm * (double)nn * es;
      const double pair = (double)h->h_flags[QT_FLAG_ROTATED] * pair_cols * es;
      h->work_jacobi_bytes += read + pair * ((double)mm + (V ? 2.0 * (double)nn : 0.0));
      h->work_jacobi_gram_bytes += read;
      h->work_jacobi_rot_bytes += pair * ((double)mm + (V ? (double)nn : 0.0));
    }
    float offkept = 0.f;
    std::memcpy(&offkept, &h->h_flags[QT_FLAG_OFFKEPT], sizeof(float));
    const float keep2_used = keep2;
    double tail2 = -1.0, tail2_change = -1.0, all2 = 0.0;
    if (keep_track) {
      // the weight left outside the keep_count largest columns bounds the
      // truncation error of the final split from above (those columns span
      // at least their own weight); its change over the sweep measures how
      // much the kept set still moves
      std::vector<float> srt(hnorm);
      std::nth_element(srt.begin(), srt.begin() + (keep_count - 1), srt.end(), std::greater<float>());
      keep2 = (float)(keep_margin * keep_margin) * srt[keep_count - 1];
      tail2 = 0.0;
      for (int64_t c = keep_count; c < nn; c++) tail2 += (double)srt[c];
      for (float v : srt) all2 += (double)v;
      if (prev_tail2 >= 0.0) tail2_change = prev_tail2 - tail2;
      prev_tail2 = tail2;
    }
    if (trace) {
      float off;
      std::memcpy(&off, &h->h_flags[QT_FLAG_OFFMAX], sizeof(float));
      float offbig;
      std::memcpy(&offbig, &h->h_flags[QT_FLAG_OFFBIG], sizeof(float));
      std::fprintf(stderr,
                   "jacobi %lldx%lld sweep %d: rotated pairs %d, inner sweeps %d, max rel off-diagonal %.3e "
                   "(columns above 1e-3 ||X||: %.3e; above the keep threshold %.3e: %.3e); tail weight %.6e, "
                   "change %.3e\n",
                   (long long)mm, (long long)nn, sweep, h->h_flags[QT_FLAG_ROTATED], h->h_flags[QT_FLAG_INNER], off,
                   offbig, std::sqrt((double)keep2_used), offkept, tail2, tail2_change);
    }
    if (h->h_flags[QT_FLAG_ABORT]) return qt_fail(h, QT_ETIMEOUT, "jacobi: a round of the sweep kernel gave up waiting");
    if (h->h_flags[QT_FLAG_NONFINITE]) return qt_fail(h, QT_ENUMERIC, "jacobi: non-finite value in the matrix");
    if (multi ? h->h_flags[QT_FLAG_CONVERGED] : h->h_flags[QT_FLAG_ROTATED] == 0) break;
    // kept set converged: no pair with a column above the threshold rotated,
    // or the tail weight moved by at most keep_tol of itself over this sweep
    // after at most 10 keep_tol over the previous one (the iteration is in
    // its fast-converging phase, where the remaining sweeps would change the
    // tail by about as much again: the truncation error is then final to
    // ~keep_tol / 2 relative)
    if (keep_track && keep_stop && keep2_used > 0.f && offkept == 0.f) break;
    // The kept space itself is off by about the root of what the tail has yet
    // to lose.  The ring's sweeps rotate each pair once, and their tail can
    // settle to 1e-3 with the kept space still 4e-5 off (a bond of 45 whose
    // truncation error is large), so what the next sweep would take, by the
    // ratio of the last two, has to be below 1e-12 ||X||_F^2 too.
    const bool settled = !ring.ctas || tail2_change * tail2_change <= 1e-12 * all2 * prev_change;
    if (keep_track && keep_stop && tail2_change >= 0.0 && prev_change >= 0.0 && tail2_change <= keep_tol * tail2 &&
        prev_change <= 10.0 * keep_tol * tail2 && settled)
      break;
    prev_change = tail2_change;
  }
  *sweeps_out = sweep + (sweep < max_sweeps ? 1 : 0);
  if (sweep_kernel && pending) {
    // the last round's unitaries, in place, then the data back into X and V
    if constexpr (sizeof(typename real_of<TS>::type) == 4) {
      const int b = (gcount - 1) & 1;
      float2* xf = (float2*)(b ? X1 : X);
      float2* vf = V ? (float2*)(b ? V1 : V) : nullptr;
      QT_LAUNCH(h, pair_apply32_kernel, dim3(pairs, achunks), NT, 0, xf, ldx, (int)mm, vf, ldv, (int)nn, nb,
                rounds - 1, axrows, avrows, (const float2*)wbuf + (size_t)b * pairs * NGRAM, (const int*)rotf + b * pairs);
      if (b) {
        QT_CHECK_CUDA(h, cudaMemcpy2DAsync(X, ldx * sizeof(TS), X1, ldx * sizeof(TS), mm * sizeof(TS), nn,
                                           cudaMemcpyDeviceToDevice, h->stream));
        if (V)
          QT_CHECK_CUDA(h, cudaMemcpy2DAsync(V, ldv * sizeof(TS), V1, ldv * sizeof(TS), nn * sizeof(TS), nn,
                                             cudaMemcpyDeviceToDevice, h->stream));
      }
    }
  }
  if (phase_ns) QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));  // the counters are written on h->stream
  if (phase_ns && sweep_kernel) {
    unsigned long long hp[4];
    QT_CHECK_CUDA(h, cudaMemcpy(hp, phase_ns, sizeof(hp), cudaMemcpyDeviceToHost));
    const double ctas = (double)gcount * pairs;
    std::fprintf(stderr, "jacobi sweep kernel, us per CTA per round: waits %.2f, rebuild+products %.2f, "
                 "reduction+test %.2f, solver %.2f\n", hp[0] / ctas * 1e-3, hp[1] / ctas * 1e-3, hp[2] / ctas * 1e-3,
                 hp[3] / ctas * 1e-3);
  } else if (phase_ns && two_launch) {
    unsigned long long hp[3];
    QT_CHECK_CUDA(h, cudaMemcpy(hp, phase_ns, sizeof(hp), cudaMemcpyDeviceToHost));
    const double launches = (double)(*sweeps_out) * rounds * pairs;
    std::fprintf(stderr, "jacobi Gram kernel, us per CTA: products %.2f, reduction+test %.2f, solver (rotating pairs "
                 "only, averaged over all) %.2f\n", hp[0] / launches * 1e-3, hp[1] / launches * 1e-3,
                 hp[2] / launches * 1e-3);
  } else if (phase_ns) {
    unsigned long long hp[16];
    QT_CHECK_CUDA(h, cudaMemcpy(hp, phase_ns, sizeof(hp), cudaMemcpyDeviceToHost));
    const double launches = (double)(*sweeps_out) * rounds;
    const char* nm32[7] = {"stage", "gram", "barrier1", "sums+barrier2", "test+solver", "barriers+copy", "rotate"};
    const char* nm64[7] = {"stage", "gram", "barrier", "sums+test", "solver", "rotate", "-"};
    const char** nm = fp32 ? nm32 : nm64;
    for (int g = 0; g < 2; g++) {
      const double ctas = launches * pairs * (g == 0 ? 1 : csize - 1);
      std::fprintf(stderr, "jacobi phases (%s), us per CTA per round:", g == 0 ? "CTA 0" : "other CTAs");
      for (int i = 0; i < 7; i++) std::fprintf(stderr, " %s %.2f", nm[i], ctas > 0 ? hp[8 * g + i] / ctas * 1e-3 : 0.0);
      std::fprintf(stderr, "\n");
    }
  }
  if (sweep >= max_sweeps) {
    // Out of sweeps: accept when the worst remaining pair is orthogonal to
    // 1e-6 relative (its effect on the singular values is below 1e-12), or --
    // FP32 storage -- when every column above 1e-3 ||X||_F has converged and
    // only columns near the rounding level still rotate (their total weight,
    // all the tail rule needs of them, is rotation-invariant).
    float off, offbig;
    std::memcpy(&off, &h->h_flags[QT_FLAG_OFFMAX], sizeof(float));
    std::memcpy(&offbig, &h->h_flags[QT_FLAG_OFFBIG], sizeof(float));
    if (off < 1e-6f) return QT_OK;
    if (fp32 && offbig <= tol) return QT_OK;
    return qt_fail(h, QT_ENUMERIC, "jacobi: no convergence within the sweep limit (off " + std::to_string(off) + ")");
  }
  return QT_OK;
}
template int qt_jacobi_svd_ws<double2>(qt_handle*, double2*, int64_t, int64_t, int64_t, double2*, int64_t, double,
                                       int, int*, double2*, double, int, bool);
template int qt_jacobi_svd_ws<float2>(qt_handle*, float2*, int64_t, int64_t, int64_t, float2*, int64_t, double, int,
                                      int*, double2*, double, int, bool);

template <typename TS>
int qt_jacobi_svd(qt_handle* h, TS* X, int64_t mm, int64_t nn, int64_t ldx, TS* V, int64_t ldv, double tol,
                  int max_sweeps, int* sweeps_out, double nu_rel, int keep_count, bool pairwise) {
  int nb = 0, chunks = 0;
  const int nparts = qt_jacobi_layout(mm, nn, &nb, &chunks);
  qt_scratch s(h);
  double2* parts;
  QT_TRY(s.get(&parts, (size_t)nparts));
  return qt_jacobi_svd_ws<TS>(h, X, mm, nn, ldx, V, ldv, tol, max_sweeps, sweeps_out, parts, nu_rel, keep_count,
                              pairwise);
}
template int qt_jacobi_svd<double2>(qt_handle*, double2*, int64_t, int64_t, int64_t, double2*, int64_t, double, int,
                                    int*, double, int, bool);
template int qt_jacobi_svd<float2>(qt_handle*, float2*, int64_t, int64_t, int64_t, float2*, int64_t, double, int,
                                   int*, double, int, bool);
