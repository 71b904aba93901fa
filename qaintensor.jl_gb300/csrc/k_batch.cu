// Batched two-qubit gate + truncated-SVD updates over many independent
// circuits (uneven qubit counts, bond caps and depths).
//
// Storage: every circuit c owns nsites(c) site slots of cap(c) x 2 x cap(c)
// complex64 (cap = its chi_max) in one device buffer, and a bond-dimension
// array bonds[c][0..n] on the device (site i is (bonds[i], 2, bonds[i+1])).
//
// One launch per circuit layer: a persistent kernel whose CTAs take
// (circuit, site) tasks from an atomic counter and run a whole update each:
//   theta' = G (A B)            FP32, tiled product, gate folded per (a, b), kept in a
//                               per-CTA slab
//   one-sided Jacobi on theta'  FP32 columns in shared memory (in the slab, i.e. in L2,
//                               where theta' does not fit), rotation angles as
//                               FP64 gives them (qt_cta.cuh)
//   sigma_j = ||x_j||           FP64, bitonic sort, tail rule (FP64, sequential) at
//                               the caller's cutoff, cap; a decision below the FP32
//                               resolution without a certificate (cap or exact rank
//                               bound) is left to an FP64 split
//   A' = x_perm(j) / sigma_j    written into site slot w
//   B' = A'^H theta'            written into site slot w+1 (no V accumulation)
//   bonds[w+1] = k
// The tasks left to the FP64 split are listed, and a second kernel of the layer
// takes them, a cluster of eight CTAs each or, where many are left, one CTA
// each (batch_split64_kernel).  Tasks of one brickwork layer touch disjoint
// sites, so CTAs never race.  A whole program (every layer) is a fixed sequence
// of a counter reset and kernels that the host captures once in a CUDA graph.
// The layer kernel has no waits on other CTAs: a CTA stops when the counter
// passes the task count.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "qt_cta.cuh"
#include "qt_internal.cuh"
#include "qt_rank_model.h"

namespace {

constexpr int BT = 256;            // threads per CTA
constexpr int BWARPS = BT / 32;
constexpr int MAXN = 256;          // largest 2 * cap handled (cap <= 128)

struct BatchArgs {
  float2* sites;
  const int64_t* site_off;   // per circuit: float2 offset of site 0
  const int* cap;            // per circuit: chi_max
  const int* nsites;         // per circuit: qubits
  int* bonds;                // bond dims, bond_off[c] + i, i = 0..n
  const int* bond_off;
  const int* task_circ;
  const int* task_site;
  const double2* task_gate;  // 16 per task, column-major
  const int* task_grank;     // per task: the gate's operator-Schmidt rank
  int task_begin, task_end;
  int* counter;
  float2* slab;              // per CTA: 4 * slab_elems float2 (FP32 X, T; per cluster or CTA the FP64 T, X)
  int slab_elems;
  int* left;                 // tasks of this layer left to the FP64 split, and how many
  int* nleft;
  int alone_above;           // more tasks left than this: one CTA each, not a cluster
  int smem_elems;            // float2 entries of the CTA's dynamic shared memory
  double cutoff;
  double floor_rel;          // FP32 resolution relative to ||theta'||_F (<= 0: 4 sqrt(max(m, n)) u)
  float tol;                 // FP32 Jacobi tolerance (relative off-diagonal)
  int max_sweeps;
  int* task_rank;
  int* task_sweeps;
  float* task_discarded;
  int* task_cert;            // QT_CERT_* of the rank decision (QT_CERT_NONE: the FP64 split decided)
};

// theta' = G (A B) into T (m x n, ld m) and X (ld ldx): the product into T, then the
// gate on the four physical values of each (a, b).  C = float2 (FP32 products)
// or double2 (FP64).
template <int NT, int TMAX, typename C>
__device__ void form_theta(const float2* A, const float2* B, int chil, int chim, int chir, const C* g, C* X, int ldx, C* T,
                           void* sm) {
  const int m = 2 * chil, n = 2 * chir;
  cta_gemm<NT, TMAX, C>(false, false, m, n, chim, A, m, nullptr, B, chim, sm,
                        [&](int r, int col, C v) { T[r + (size_t)m * col] = v; });
  for (int idx = threadIdx.x; idx < chil * chir; idx += NT) {
    const int a = idx % chil, b = idx / chil;
    C th[4];
#pragma unroll
    for (int q = 0; q < 4; q++) th[q] = T[a + chil * (q & 1) + (size_t)m * ((q >> 1) + 2 * b)];
#pragma unroll
    for (int o = 0; o < 4; o++) {
      C v = czero<C>();
#pragma unroll
      for (int q = 0; q < 4; q++) cfma(v, g[o + 4 * q], th[q]);
      const int row = a + chil * (o & 1), col = (o >> 1) + 2 * b;
      T[row + (size_t)m * col] = v;
      X[row + (size_t)ldx * col] = v;
    }
  }
  __syncthreads();
}

// ||X||_F^2 in FP64 over the CTA.
template <int NT, typename C>
__device__ double fro2_of(const C* X, int cnt, double* s_red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double part = 0;
  for (int i = threadIdx.x; i < cnt; i += NT) part += (double)X[i].x * X[i].x + (double)X[i].y * X[i].y;
  part = cta_warp_sum(part);
  __syncthreads();
  if (lane == 0) s_red[warp] = part;
  __syncthreads();
  double fro2 = 0;
  for (int i = 0; i < NT / 32; i++) fro2 += s_red[i];
  return fro2;
}

// Bitonic sort, descending by value, ties by index; np2 entries, a power of two.
template <int NT>
__device__ void sort_values(int np2, double* s_sig, int* s_perm) {
  for (int k2 = 2; k2 <= np2; k2 <<= 1)
    for (int j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
      for (int i = threadIdx.x; i < np2; i += NT) {
        const int l = i ^ j2;
        if (l > i) {
          const bool desc = ((i & k2) == 0);
          const double x = s_sig[i], y = s_sig[l];
          const bool sw = desc ? (x < y || (x == y && s_perm[i] > s_perm[l]))
                               : (x > y || (x == y && s_perm[i] < s_perm[l]));
          if (sw) {
            s_sig[i] = y; s_sig[l] = x;
            const int tp = s_perm[i]; s_perm[i] = s_perm[l]; s_perm[l] = tp;
          }
        }
      }
      __syncthreads();
    }
}

// Column norms of X in FP64, sorted descending into s_sig / s_perm (bitonic).
template <int NT, typename C>
__device__ void sorted_norms(const C* X, int ld, int m, int n, double* s_sig, int* s_perm) {
  int np2 = 1;
  while (np2 < n) np2 <<= 1;
  for (int j = threadIdx.x; j < np2; j += NT) {
    double s = -1.0;
    if (j < n) {
      s = 0;
#pragma unroll 8
      for (int i = 0; i < m; i++) {
        const C v = X[i + (size_t)ld * j];
        s += (double)v.x * v.x + (double)v.y * v.y;
      }
      s = sqrt(s);
    }
    s_sig[j] = s;
    s_perm[j] = j;
  }
  __syncthreads();
  sort_values<NT>(np2, s_sig, s_perm);
}

// The tail rule of src/svd.jl:29-33 (sequential from the smallest value,
// strict >, k >= 1) on the n sorted values.  The square root, a dependent
// FP64 chain per value, is taken only where the sum lies within rounding of
// cutoff^2; elsewhere the comparison of the squares gives the same answer.
__device__ int tail_rule(const double* s, int n, double cutoff) {
  const double c2 = cutoff * cutoff;
  const bool squares = c2 > 1e-290;
  const double lo = squares ? c2 * (1.0 - 1e-14) : 0.0, hi = squares ? c2 * (1.0 + 1e-14) : INFINITY;
  double acc = 0;
  for (int i = n - 1; i >= 0; i--) {
    acc += s[i] * s[i];
    if (acc < lo) continue;
    if (acc > hi || sqrt(acc) > cutoff) return i + 1;
  }
  return 1;
}

// RMAX: rows of theta' per lane at most (m <= 32 RMAX), by the bucket's cap.
//
// What bounds it: the Jacobi's FMAs and, where theta' exceeds the shared
// memory, its column traffic to L2; one CTA works alone on a task, so the
// tasks in flight are what fills the chip.
template <int NT, int RMAX>
__global__ void __launch_bounds__(NT) batch_layer_kernel(BatchArgs p) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ int s_task, s_k, s_fb;
  __shared__ float2 g[16];
  __shared__ double s_sig[MAXN];
  __shared__ int s_perm[MAXN];
  __shared__ double s_red[NT / 32];
  constexpr int TMAX = RMAX >= 2 ? 64 : 32;
  const int tid = threadIdx.x;
  float2* slab = p.slab + (size_t)blockIdx.x * 4 * p.slab_elems;
  float2* T = slab + p.slab_elems;

  for (;;) {
    if (tid == 0) s_task = p.task_begin + atomicAdd(p.counter, 1);
    __syncthreads();
    const int task = s_task;
    if (task >= p.task_end) break;
    const int c = p.task_circ[task], w = p.task_site[task];
    int* bond = p.bonds + p.bond_off[c];
    const int chil = bond[w], chim = bond[w + 1], chir = bond[w + 2];
    const int cap = p.cap[c], nq = p.nsites[c];
    const size_t slot = (size_t)cap * 2 * cap;
    float2* A = p.sites + p.site_off[c] + (size_t)w * slot;
    float2* B = A + slot;
    const int m = 2 * chil, n = 2 * chir;
    if (tid < 16) {
      const double2 v = p.task_gate[(size_t)task * 16 + tid];
      g[tid] = make_float2((float)v.x, (float)v.y);
    }
    __syncthreads();

    // 1. theta' = G (A B) in FP32.  In shared memory the columns are an odd
    // number of entries apart, so that threads on different columns meet
    // different banks.
    const bool in_smem = (m + 1) * n <= p.smem_elems;
    float2* X = in_smem ? reinterpret_cast<float2*>(dyn) : slab;
    const int ldx = in_smem ? m + 1 : m;
    form_theta<NT, TMAX, float2>(A, B, chil, chim, chir, g, X, ldx, T, dyn);
    const double fro2 = fro2_of<NT>(T, m * n, s_red);
    const double nu = 4.0 * sqrt((double)max(m, 16)) * 5.96e-8;

    // 2. one-sided Jacobi on the columns of X, 3. sorted FP64 norms
    int sweeps = cta_jacobi_any<NT, RMAX>(X, ldx, m, n, (double)p.tol, nu * nu * fro2, p.max_sweeps);
    sorted_norms<NT, float2>(X, ldx, m, n, s_sig, s_perm);

    // 4. the tail rule at the caller's cutoff, then the cap.  Below the FP32
    // resolution eta the decision needs a certificate: the cap binding with
    // margin, or exactly as many values above eta as the exact rank bound
    // allows (the gate's operator-Schmidt rank times the inner bond, the
    // Hilbert-space dimensions of the two sides).  Otherwise the FP64 split
    // below decides.
    const int kcap = min(cap, min(m, n));
    if (tid == 0) {
      const double eta = (p.floor_rel > 0 ? p.floor_rel : 4.0 * sqrt((double)max(m, n)) * 5.96e-8) * sqrt(fro2);
      int kc = tail_rule(s_sig, n, p.cutoff);
      int cert = QT_CERT_NONE;
      if (p.cutoff >= eta) {
        // (Not so where frozen columns are kept: eta is about nu, and the rule
        // drops by accumulated weight.  Their unit vectors are not orthogonal
        // to the larger ones, and A' A'^H theta' is no projection then.)
        cert = QT_CERT_RESOLVED;
      } else if (cap < min(m, n) && kc > cap) {
        double t2 = 0;
        for (int i = n - 1; i >= cap; i--) t2 += s_sig[i] * s_sig[i];
        if (sqrt(t2) > p.cutoff + eta) cert = QT_CERT_CAP;
      }
      if (cert == QT_CERT_NONE) {
        int srank = min(min(m, n), p.task_grank[task] * chim);
        if (w + 1 < 30) srank = min(srank, 1 << (w + 1));
        if (nq - w - 1 < 30) srank = min(srank, 1 << (nq - w - 1));
        int kr = 0;
        while (kr < n && s_sig[kr] > eta) kr++;
        if (kr == srank) {
          kc = srank;
          cert = QT_CERT_STRUCT;
        }
      }
      const int k = min(kc, kcap);
      double disc = 0;
      for (int i = k; i < n; i++) disc += s_sig[i] * s_sig[i];
      s_k = k;
      s_fb = cert == QT_CERT_NONE;
      p.task_rank[task] = k;
      p.task_sweeps[task] = sweeps;
      p.task_discarded[task] = (float)disc;
      p.task_cert[task] = cert;
    }
    __syncthreads();

    if (!s_fb) {
      const int k = s_k;
      // 5. A' (chil, 2, k) = unit columns, into site slot w
      for (int j = tid >> 5; j < k; j += NT / 32) {
        const double s = s_sig[j];
        const float inv = s > 0 ? (float)(1.0 / s) : 0.f;
        const float2* x = X + (size_t)ldx * s_perm[j];
        for (int r = tid & 31; r < m; r += 32) A[r + (size_t)m * j] = make_float2(x[r].x * inv, x[r].y * inv);
      }
      __syncthreads();
      // 6. B' (k, 2, chir) = A'^H theta', into site slot w+1
      cta_gemm<NT, TMAX, float2>(true, false, k, n, m, A, m, nullptr, T, m, dyn,
                                 [&](int r, int col, float2 v) { B[r + (size_t)k * col] = v; });
      if (tid == 0) bond[w + 1] = k;
    } else if (tid == 0) {
      p.left[atomicAdd(p.nleft, 1)] = task;
    }
    __syncthreads();
  }
}

// The exact FP64 split of the tasks a layer left: theta' from the complex64
// sites in FP64, one-sided FP64 Jacobi (tolerance and freeze at FP64 rounding),
// the tail rule at the caller's cutoff.
//
// What bounds it: FP64 products (24 instructions per row of a column pair on
// the two FP64 lanes of an SM), of few tasks a layer.  So a cluster of eight
// CTAs takes one task: CTA q holds the rows congruent to q modulo 8 of every
// column in shared memory (at most 32 x 256); a round's sums meet through
// distributed shared memory, and every CTA finds the same rotations and
// rotates its rows.  Four lanes share a pair, a warp eight pairs: an FP64
// instruction costs the same however many lanes take part.  The sums keep the
// order of one warp on whole columns (row r on lane r % 32, lanes 16, 8, 4, 2
// and 1 apart added in turn: the first two inside a CTA, the others between
// CTAs), because nearly equal columns leave the sign of a rotation to the
// last bit, and later FP32 splits of the same circuit see which one was taken.
// A 128 x 128 task (about 27 sweeps): 31 ms, 9 us a round, 8 us of them FP64
// issue; by one CTA, as the layer kernel's last step, 95 ms.
// That pays while few tasks are left.  From some number on (see
// split64_alone_above) every CTA takes a task by itself, a warp to a pair and
// the columns in the slab where shared memory does not hold them: the same sums
// in the same order, so that a circuit's results do not depend on how many
// others run beside it.
constexpr int S64_NT = 256, S64_C = 8, S64_W = S64_NT / 32;
constexpr int S64_LD = 36;                    // rows of a slice, at most; 4 (mod 8) for the banks
constexpr size_t S64_ROTS = MAXN / 2 * 5;     // rotations of a round's pairs: c, s, er, ei, on
constexpr size_t S64_SUMS = MAXN / 2 * 4;     // sums of a round's pairs
constexpr size_t S64_SMEM = (2 * S64_SUMS + S64_ROTS + 2 * S64_LD * MAXN) * sizeof(double);

// Sums of this CTA's rows of each pair, aa bb gr gi, LP lanes on a pair.
template <int LP>
__device__ __forceinline__ void split64_sums(const double2* X, int ld, int rows, int n, int round, double* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane % LP, pairs = n / 2;
  constexpr int PW = 32 / LP;
  for (int first = PW * warp; first < pairs; first += PW * S64_W) {
    const int q = first + lane / LP;
    int a, b;
    cta_tourney(round, min(q, pairs - 1), n, a, b);
    const double2 *xp = X + (size_t)ld * a, *xq = X + (size_t)ld * b;
    double v0 = 0, v1 = 0, v2 = 0, v3 = 0;
    for (int j = lr; j < rows; j += LP) {
      const double2 u = xp[j], w = xq[j];
      v0 = fma(u.x, u.x, fma(u.y, u.y, v0));
      v1 = fma(w.x, w.x, fma(w.y, w.y, v1));
      v2 = fma(u.x, w.x, fma(u.y, w.y, v2));
      v3 = fma(u.x, w.y, fma(-u.y, w.x, v3));
    }
    const bool up2 = lr & (LP / 2), up1 = lr & (LP / 4);
    const double x0 = (up2 ? v2 : v0) + __shfl_xor_sync(0xffffffffu, up2 ? v0 : v2, LP / 2);
    const double x1 = (up2 ? v3 : v1) + __shfl_xor_sync(0xffffffffu, up2 ? v1 : v3, LP / 2);
    double s = (up1 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, up1 ? x0 : x1, LP / 4);
#pragma unroll
    for (int o = LP / 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (q < pairs && lr % (LP / 4) == 0) part[4 * q + lr / (LP / 4)] = s;
  }
}

// (every rounding written out, as in cta_store_rotated: the same bits with every LP)
template <int LP>
__device__ __forceinline__ void split64_rotate(double2* X, int ld, int rows, int n, int round, const double* rot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane % LP, pairs = n / 2;
  constexpr int PW = 32 / LP;
  for (int q = PW * warp + lane / LP; q < pairs; q += PW * S64_W) {
    if (rot[5 * q + 4] == 0) continue;
    const double c = rot[5 * q], s = rot[5 * q + 1], er = rot[5 * q + 2], ei = rot[5 * q + 3];
    int a, b;
    cta_tourney(round, q, n, a, b);
    double2 *xp = X + (size_t)ld * a, *xq = X + (size_t)ld * b;
    for (int j = lr; j < rows; j += LP) {
      const double2 u = xp[j], v = xq[j];
      xp[j] = make_double2(fma(c, u.x, -__dmul_rn(s, fma(er, v.x, __dmul_rn(ei, v.y)))),
                           fma(c, u.y, -__dmul_rn(s, fma(er, v.y, -__dmul_rn(ei, v.x)))));
      xq[j] = make_double2(fma(c, v.x, __dmul_rn(s, fma(er, u.x, -__dmul_rn(ei, u.y)))),
                           fma(s, fma(ei, u.x, __dmul_rn(er, u.y)), __dmul_rn(c, v.y)));
    }
  }
}

struct split64_shared {
  double2 g64[16];
  double sig[MAXN], red[S64_NT / 32];
  int perm[MAXN], k, next;
};

// One task by CW CTAs (CW = 1: this one alone), `rank` of them.
template <int CW>
__device__ void split64_task(const BatchArgs& p, int task, int rank, double2* T, double2* Xg, unsigned char* dyn,
                             split64_shared& sh) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  auto meet = [&]() {
    if constexpr (CW > 1) cl.sync();
    else __syncthreads();
  };
  constexpr int LP = 32 / CW;  // lanes per pair
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* part = reinterpret_cast<double*>(dyn);  // two rounds' sums
  double* rot = part + 2 * S64_SUMS;
  double2* Xs = reinterpret_cast<double2*>(rot + S64_ROTS);
  const int c = p.task_circ[task], w = p.task_site[task];
  int* bond = p.bonds + p.bond_off[c];
  const int chil = bond[w], chim = bond[w + 1], chir = bond[w + 2], cap = p.cap[c];
  const size_t slot = (size_t)cap * 2 * cap;
  float2* A = p.sites + p.site_off[c] + (size_t)w * slot;
  float2* B = A + slot;
  const int m = 2 * chil, n = 2 * chir, pairs = n / 2;
  // a cluster: rows CW j + rank of every column in shared memory, j < 4 K with
  // the zeros, of which the last CTAs have one more; one CTA: every row, in the slab
  // where shared memory does not hold them (ld odd: columns start in different banks)
  const int K = ((m + CW - 1) / CW + 3) / 4;
  const bool in_smem = CW > 1 || (m | 1) * n <= S64_LD * MAXN;
  double2* X = in_smem ? Xs : Xg;
  const int ld = CW > 1 ? 4 * (K | 1) : in_smem ? m | 1 : m, rows = CW > 1 ? 4 * K : m;
  if (tid < 16) sh.g64[tid] = p.task_gate[(size_t)task * 16 + tid];
  __syncthreads();
  // theta': this CTA's columns (the two values of s2 together), then its rows
  const int b0 = rank * chir / CW, b1 = (rank + 1) * chir / CW;
  double2* Tb = T + (size_t)m * 2 * b0;
  const float2* Bb = B + (size_t)chim * 2 * b0;
  if (b1 > b0) form_theta<S64_NT, 32, double2>(A, Bb, chil, chim, b1 - b0, sh.g64, Tb, m, Tb, dyn);
  meet();
  for (int j = warp; j < n; j += S64_W)
    for (int r = lane; r < rows; r += 32)
      X[r + (size_t)ld * j] = CW * r + rank < m ? T[CW * r + rank + (size_t)m * j] : make_double2(0, 0);
  const double f64 = fro2_of<S64_NT>(T, m * n, sh.red);  // the same in every CTA
  const double tol = 16.0 * sqrt((double)max(m, 16)) * 1.11e-16, nu = 4.0 * sqrt((double)max(m, 16)) * 1.11e-16;
  const double nu2 = nu * nu * f64;
  int sweeps = 0, buf = 0;
  for (int sweep = 0; sweep < p.max_sweeps; sweep++) {
    bool rotated = false;
    for (int r = 0; r < n - 1; r++) {
      double* pb = part + buf * S64_SUMS;
      split64_sums<LP>(X, ld, rows, n, r, pb);
      meet();  // (two buffers: whoever reads this round's sums has left the last round's)
      if (tid < pairs) {
        double2 v[CW], u[CW];
#pragma unroll
        for (int q = 0; q < CW; q++) {
          const double2* o = reinterpret_cast<const double2*>((CW > 1 ? cl.map_shared_rank(pb, q) : pb) + 4 * tid);
          v[q] = o[0];
          u[q] = o[1];
        }
#pragma unroll
        for (int off = CW / 2; off > 0; off >>= 1)
#pragma unroll
          for (int q = 0; q < off; q++) {
            v[q].x += v[q + off].x; v[q].y += v[q + off].y;
            u[q].x += u[q + off].x; u[q].y += u[q + off].y;
          }
        const cta_rotation<double> o = cta_angle64<double>(v[0].x, v[0].y, u[0].x, u[0].y, tol, nu2);
        double* d = rot + 5 * tid;
        d[0] = o.c; d[1] = o.s; d[2] = o.er; d[3] = o.ei;
        d[4] = o.on ? 1.0 : 0.0;
        rotated |= o.on;
      }
      __syncthreads();
      split64_rotate<LP>(X, ld, rows, n, r, rot);
      __syncthreads();
      buf ^= 1;
    }
    sweeps = sweep + 1;
    if (!__syncthreads_or(rotated)) break;  // the same answer in every CTA
  }
  if (in_smem)
    for (int j = warp; j < n; j += S64_W)
      for (int r = lane; CW * r + rank < m; r += 32) Xg[CW * r + rank + (size_t)m * j] = X[r + (size_t)ld * j];
  meet();
  sorted_norms<S64_NT, double2>(Xg, m, m, n, sh.sig, sh.perm);  // the same in every CTA
  if (tid == 0) {
    const int k = min(tail_rule(sh.sig, n, p.cutoff), min(cap, min(m, n)));
    double disc = 0;
    for (int j = k; j < n; j++) disc += sh.sig[j] * sh.sig[j];
    sh.k = k;
    if (rank == 0) {
      p.task_rank[task] = k;
      p.task_sweeps[task] += sweeps;
      p.task_discarded[task] = (float)disc;
    }
  }
  __syncthreads();
  const int k = sh.k;
  // A' = unit columns (this CTA's rows), B' = A'^H theta' (its columns), both from the FP64 columns
  for (int j = warp; j < k; j += S64_W) {
    const double s = sh.sig[j], inv = s > 0 ? 1.0 / s : 0.0;
    const double2* x = X + (size_t)ld * sh.perm[j];
    for (int r = lane; CW * r + rank < m; r += 32)
      A[CW * r + rank + (size_t)m * j] = make_float2((float)(x[r].x * inv), (float)(x[r].y * inv));
  }
  __syncthreads();  // the product's tiles take the start of the shared memory
  if (b1 > b0)
    cta_gemm<S64_NT, 32, double2>(true, false, k, 2 * (b1 - b0), m, Xg, m, sh.perm, Tb, m, dyn,
                                  [&](int r, int col, double2 v) {
                                    const double s = sh.sig[r], inv = s > 0 ? 1.0 / s : 0.0;
                                    B[r + (size_t)k * (2 * b0 + col)] = make_float2((float)(v.x * inv), (float)(v.y * inv));
                                  });
  if (rank == 0 && tid == 0) bond[w + 1] = k;
  meet();
}

__global__ void __cluster_dims__(S64_C, 1, 1) __launch_bounds__(S64_NT) batch_split64_kernel(BatchArgs p) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ split64_shared sh;
  const int left = *p.nleft, tid = threadIdx.x;
  if (left == 0) return;
  if (left > p.alone_above) {
    double2* T = reinterpret_cast<double2*>(p.slab + (size_t)blockIdx.x * 4 * p.slab_elems);
    for (;;) {
      if (tid == 0) sh.next = atomicAdd(p.counter, 1);
      __syncthreads();
      const int i = sh.next;
      if (i >= left) return;
      split64_task<1>(p, p.left[i], 0, T, T + p.slab_elems, dyn, sh);
    }
  }
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  const int rank = (int)cl.block_rank();
  double2* T = reinterpret_cast<double2*>(p.slab + (size_t)(blockIdx.x - rank) * 4 * p.slab_elems);
  for (;;) {
    if (rank == 0 && tid == 0) sh.next = atomicAdd(p.counter, 1);
    cl.sync();
    const int i = *cl.map_shared_rank(&sh.next, 0);
    if (i >= left) break;
    split64_task<S64_C>(p, p.left[i], rank, T, T + p.slab_elems, dyn, sh);
  }
  cl.sync();  // no CTA leaves while another may still read its shared memory
}

// <Z_site> per circuit in FP32, one CTA per circuit (grid-stride): the
// environment L of the sites left of the measured one (L <- sum_s A_s^H L
// A_s), R of those right of it (R <- sum_s A_s R A_s^H), and
// d_s = tr(A_s^H L A_s R) at the measured site, so <Z> = (d_0 - d_1) /
// (d_0 + d_1).  Each site is passed once, by two tiled products over both
// physical values at a time.
constexpr int EXPECT_TILE = 64;
__global__ void __launch_bounds__(BT)
batch_expect_kernel(const float2* sites, const int64_t* site_off, const int* cap, const int* nsites, const int* bonds,
                    const int* bond_off, int ncirc, int site, float2* slab, int slab_elems, double* out) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double s_red[2][BWARPS];
  const int tid = threadIdx.x;
  for (int c = blockIdx.x; c < ncirc; c += gridDim.x) {
    const int n = nsites[c];
    const int* bd = bonds + bond_off[c];
    const size_t e2 = (size_t)cap[c] * cap[c], slot = 2 * e2;
    float2* L = slab + (size_t)blockIdx.x * 4 * slab_elems;
    float2 *R = L + e2, *T = R + e2, *U = T + slot;
    const float2* base = sites + site_off[c];
    auto eye = [&](float2* E, int d) {
      for (int i = tid; i < d * d; i += BT) E[i] = make_float2((i % d) == (i / d) ? 1.f : 0.f, 0.f);
    };
    eye(L, bd[0]);
    eye(R, bd[n]);
    __syncthreads();
    // a site (cl, 2, cr) is its (cl x 2 cr) matrix with ld cl and its (2 cl x
    // cr) matrix with ld 2 cl in the same memory
    auto times_left = [&](const float2* A, int cl, int cr) {  // T = L A
      cta_gemm<BT, EXPECT_TILE, float2>(false, false, cl, 2 * cr, cl, L, cl, nullptr, A, cl, dyn,
                                [&](int r, int col, float2 v) { T[r + (size_t)cl * col] = v; });
    };
    auto times_right = [&](const float2* A, int cl, int cr) {  // U = A R
      cta_gemm<BT, EXPECT_TILE, float2>(false, false, 2 * cl, cr, cr, A, 2 * cl, nullptr, R, cr, dyn,
                                [&](int r, int col, float2 v) { U[r + (size_t)2 * cl * col] = v; });
    };
    for (int st = 0; st < site; st++) {
      const float2* A = base + (size_t)st * slot;
      const int cl = bd[st], cr = bd[st + 1];
      times_left(A, cl, cr);
      cta_gemm<BT, EXPECT_TILE, float2>(true, false, cr, cr, 2 * cl, A, 2 * cl, nullptr, T, 2 * cl, dyn,
                                [&](int r, int col, float2 v) { L[r + (size_t)cr * col] = v; });
    }
    for (int st = n - 1; st > site; st--) {
      const float2* A = base + (size_t)st * slot;
      const int cl = bd[st], cr = bd[st + 1];
      times_right(A, cl, cr);
      cta_gemm<BT, EXPECT_TILE, float2>(false, true, cl, cl, 2 * cr, U, cl, nullptr, A, cl, dyn,
                                [&](int r, int col, float2 v) { R[r + (size_t)cl * col] = v; });
    }
    const float2* A = base + (size_t)site * slot;
    const int cl = bd[site], cr = bd[site + 1];
    times_left(A, cl, cr);
    times_right(A, cl, cr);
    // R is Hermitian: tr(A_s^H L A_s R) = sum T_s conj(U_s)
    double d[2] = {0, 0};
    for (int j = tid >> 5; j < cr; j += BWARPS) {
      float f[2] = {0.f, 0.f};
      for (int i = tid & 31; i < 2 * cl; i += 32) {
        const float2 t = T[i + (size_t)2 * cl * j], u = U[i + (size_t)2 * cl * j];
        f[i >= cl] = fmaf(t.x, u.x, fmaf(t.y, u.y, f[i >= cl]));
      }
      d[0] += f[0];
      d[1] += f[1];
    }
    for (int s = 0; s < 2; s++) {
      d[s] = cta_warp_sum(d[s]);
      if ((tid & 31) == 0) s_red[s][tid >> 5] = d[s];
    }
    __syncthreads();
    if (tid == 0) {
      double t0 = 0, t1 = 0;
      for (int i = 0; i < BWARPS; i++) { t0 += s_red[0][i]; t1 += s_red[1][i]; }
      out[c] = (t0 - t1) / (t0 + t1);
    }
    __syncthreads();
  }
}

__global__ void batch_init_kernel(float2* sites, const int64_t* site_off, const int* cap, const int* nsites, int ncirc) {
  for (int c = blockIdx.x; c < ncirc; c += gridDim.x) {
    const size_t slot = (size_t)cap[c] * 2 * cap[c];
    for (int i = threadIdx.x; i < nsites[c]; i += blockDim.x) {
      float2* s = sites + site_off[c] + (size_t)i * slot;
      s[0] = make_float2(1.f, 0.f);  // (1,2,1): |0>
      s[1] = make_float2(0.f, 0.f);
    }
  }
}

}  // namespace

struct qt_batch {
  int ncirc = 0, capmax = 0;
  std::vector<int> nsites, cap;
  std::vector<int64_t> site_off;
  std::vector<int> bond_off;
  float2* d_sites = nullptr;
  int64_t* d_site_off = nullptr;
  int *d_cap = nullptr, *d_nsites = nullptr, *d_bonds = nullptr, *d_bond_off = nullptr;
  float2* d_slab = nullptr;
  int ctas = 0;
  int bucket_elems[4] = {0, 0, 0, 0};  // entries of the largest theta' per bond-cap bucket (0: no circuit in it)
  int* d_counter = nullptr;  // three counters per launch: tasks taken, tasks left to FP64, of those taken
  int* d_left = nullptr;     // the tasks left to FP64, in the range of their launch
  int counter_cap = 0;
  // the last program (device copies) and its captured graph
  int* d_tc = nullptr;
  int* d_ts = nullptr;
  double2* d_tg = nullptr;
  int* d_rank = nullptr;
  int* d_sweeps = nullptr;
  int* d_grank = nullptr;
  int* d_cert = nullptr;
  float* d_disc = nullptr;
  int ntask_cap = 0;
  std::vector<int> order;    // device task index -> the caller's task index
  cudaGraphExec_t graph = nullptr;
  // launch shape per bond-cap bucket (caps <= 16, 32, 64, 128): threads per
  // CTA and CTAs per SM of the persistent layer kernel (qt_batch_set_launch)
  int threads[4] = {128, 256, 256, 256};
  int cps[4] = {4, 2, 1, 1};
  size_t slab_count = 0;     // float2 entries of the slab
  // float2 entries that the launches of every bucket need (4 theta' per CTA),
  // and the observable kernel's one CTA per SM
  size_t slab_need() const {
    size_t need = 0;
    for (int bk = 0; bk < 4; bk++) need = std::max(need, (size_t)ctas * cps[bk] * 4 * bucket_elems[bk]);
    return need;
  }
  // clusters of the FP64 split of `tasks` tasks: one per eight CTAs of the
  // slab, an eighth of the chip's SMs at most
  int split_clusters(int tasks) const { return std::max(1, std::min(tasks, ctas / S64_C)); }
};

namespace {

int bucket_of(int cap) { return cap <= 16 ? 0 : cap <= 32 ? 1 : cap <= 64 ? 2 : 3; }

// Dynamic shared memory of the layer kernel: the whole theta' of a bucket
// (caps 16, 32 and 64: 8, 33 and 132 KB) and the product tiles; 200 KB for
// caps up to 128, whose theta' (512 KB) fits up to bonds of 80 and is kept in
// the slab above.
size_t batch_smem(int bk) {
  static const size_t theta[4] = {33 * 32, 65 * 64, 129 * 128, 25600};
  return std::max(theta[bk] * sizeof(float2),
                  cta_gemm_smem<float2>(bk == 0 ? 32 : 64));
}

// From how many tasks left in a launch on its FP64 splits take one CTA each
// instead of a cluster of eight: a cluster ends a task sooner, alone more of
// them run at once (152 against 19).  The line lies where the two take the
// same time for whole programs (ms at tasks per layer, alone / cluster):
// caps 16: 9.5 / 9.1 at 28, 9.8 / 10.9 at 32; 32: 49.6 / 45.1 at 75, 48.7 /
// 59.3 at 80 (a wave of clusters more); 64: 85.2 / 66.7 at 90, 85.2 / 90.6 at
// 108; 128: 854 / 810 at 280, 905 / 982 at 336.  Far from it: 1536 tasks of
// caps 8 12 / 95, 7 tasks of caps 128 732 / 204.
int split64_alone_above(int bk) {
  static const int line[4] = {28, 76, 100, 300};
  return line[bk];
}

typedef void (*layer_fn)(BatchArgs);

template <int NT>
layer_fn layer_kernel_rows(int bk) {
  static const layer_fn fn[4] = {batch_layer_kernel<NT, 1>, batch_layer_kernel<NT, 2>, batch_layer_kernel<NT, 4>,
                                 batch_layer_kernel<NT, 8>};
  return fn[bk];
}

layer_fn layer_kernel(int threads, int bk) {
  switch (threads) {
    case 128: return layer_kernel_rows<128>(bk);
    case 512: return layer_kernel_rows<512>(bk);
    case 1024: return layer_kernel_rows<1024>(bk);
    default: return layer_kernel_rows<256>(bk);
  }
}

}  // namespace

static void batch_free_program(qt_batch* b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  b->graph = nullptr;
  cudaFree(b->d_tc); cudaFree(b->d_ts); cudaFree(b->d_tg);
  cudaFree(b->d_rank); cudaFree(b->d_sweeps); cudaFree(b->d_disc); cudaFree(b->d_grank); cudaFree(b->d_cert);
  cudaFree(b->d_left);
  b->d_tc = b->d_ts = nullptr; b->d_tg = nullptr; b->d_rank = b->d_sweeps = nullptr; b->d_disc = nullptr;
  b->d_grank = b->d_cert = b->d_left = nullptr;
  b->ntask_cap = 0;
}

extern "C" int qt_batch_create(qt_handle* h, int ncirc, const int* nqubits, const int* chi_max, qt_batch** out) {
  if (!h || !nqubits || !chi_max || !out || ncirc < 1) return qt_fail(h, QT_EINVAL, "batch_create: bad argument");
  *out = nullptr;
  cudaSetDevice(h->device);
  qt_batch* b = new qt_batch();
  b->ncirc = ncirc;
  int64_t off = 0;
  int boff = 0;
  for (int c = 0; c < ncirc; c++) {
    if (nqubits[c] < 2 || chi_max[c] < 1 || chi_max[c] > MAXN / 2) {
      delete b;
      return qt_fail(h, QT_ENOTSUP, "batch_create: needs >= 2 qubits and 1 <= chi_max <= 128");
    }
    b->nsites.push_back(nqubits[c]);
    b->cap.push_back(chi_max[c]);
    b->site_off.push_back(off);
    b->bond_off.push_back(boff);
    off += (int64_t)nqubits[c] * chi_max[c] * 2 * chi_max[c];
    boff += nqubits[c] + 1;
    b->capmax = std::max(b->capmax, chi_max[c]);
    int& be = b->bucket_elems[bucket_of(chi_max[c])];
    be = std::max(be, 4 * chi_max[c] * chi_max[c]);
  }
  int dev_sms = 152;
  cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, h->device);
  b->ctas = dev_sms;
  b->slab_count = b->slab_need();
  std::vector<int> bonds(boff, 1);
  bool ok = cudaMalloc(&b->d_sites, sizeof(float2) * off) == cudaSuccess &&
            cudaMalloc(&b->d_site_off, sizeof(int64_t) * ncirc) == cudaSuccess &&
            cudaMalloc(&b->d_cap, sizeof(int) * ncirc) == cudaSuccess &&
            cudaMalloc(&b->d_nsites, sizeof(int) * ncirc) == cudaSuccess &&
            cudaMalloc(&b->d_bonds, sizeof(int) * boff) == cudaSuccess &&
            cudaMalloc(&b->d_bond_off, sizeof(int) * ncirc) == cudaSuccess &&
            cudaMalloc(&b->d_slab, sizeof(float2) * b->slab_count) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    qt_batch_free(h, b);
    return qt_fail(h, QT_ENOMEM, "batch_create: device allocation failed");
  }
  cudaMemcpy(b->d_site_off, b->site_off.data(), sizeof(int64_t) * ncirc, cudaMemcpyHostToDevice);
  cudaMemcpy(b->d_cap, b->cap.data(), sizeof(int) * ncirc, cudaMemcpyHostToDevice);
  cudaMemcpy(b->d_nsites, b->nsites.data(), sizeof(int) * ncirc, cudaMemcpyHostToDevice);
  cudaMemcpy(b->d_bonds, bonds.data(), sizeof(int) * boff, cudaMemcpyHostToDevice);
  cudaMemcpy(b->d_bond_off, b->bond_off.data(), sizeof(int) * ncirc, cudaMemcpyHostToDevice);
  batch_init_kernel<<<std::min(ncirc, 1024), 128, 0, h->stream>>>(b->d_sites, b->d_site_off, b->d_cap, b->d_nsites,
                                                                    ncirc);
  h->launches++;
  QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  *out = b;
  return QT_OK;
}

extern "C" int qt_batch_free(qt_handle* h, qt_batch* b) {
  if (!b) return QT_OK;
  if (h) {
    cudaSetDevice(h->device);
    cudaStreamSynchronize(h->stream);
  }
  batch_free_program(b);
  cudaFree(b->d_sites); cudaFree(b->d_site_off); cudaFree(b->d_cap); cudaFree(b->d_nsites);
  cudaFree(b->d_bonds); cudaFree(b->d_bond_off); cudaFree(b->d_slab); cudaFree(b->d_counter);
  delete b;
  return QT_OK;
}

// Run a whole program: layers [layer_start[l], layer_start[l+1]) of tasks
// (circuit, site 0-based, gate); tasks of one layer must touch disjoint
// sites.  With use_graph the launch sequence is captured once and replayed.
extern "C" int qt_batch_run(qt_handle* h, qt_batch* b, int nlayers, const int* layer_start, const int* circ,
                            const int* site, const double* gates, double cutoff, int use_graph) {
  if (!h || !b || nlayers < 0 || !layer_start) return qt_fail(h, QT_EINVAL, "batch_run: bad argument");
  if (!(cutoff >= 0)) return qt_fail(h, QT_EINVAL_ERR_NEG, "Error must be positive");
  cudaSetDevice(h->device);
  const int ntask = layer_start[nlayers];
  for (int t = 0; t < ntask; t++) {
    if (circ[t] < 0 || circ[t] >= b->ncirc || site[t] < 0 || site[t] + 1 >= b->nsites[circ[t]])
      return qt_fail(h, QT_EBOUNDS, "batch_run: task site out of range");
  }
  batch_free_program(b);
  // tasks of each layer grouped by the bucket of their circuit's cap (stable):
  // one launch per (layer, bucket) with that bucket's launch shape
  std::vector<int> order;
  std::vector<int> seg_begin, seg_end, seg_bucket;
  order.reserve(ntask);
  for (int l = 0; l < nlayers; l++) {
    for (int bk = 0; bk < 4; bk++) {
      const int start = (int)order.size();
      for (int t = layer_start[l]; t < layer_start[l + 1]; t++)
        if (bucket_of(b->cap[circ[t]]) == bk) order.push_back(t);
      if ((int)order.size() > start) {
        seg_begin.push_back(start);
        seg_end.push_back((int)order.size());
        seg_bucket.push_back(bk);
      }
    }
  }
  const int nseg = (int)seg_begin.size();
  std::vector<int> oc(ntask), os(ntask);
  std::vector<double> og((size_t)32 * ntask);
  for (int i = 0; i < ntask; i++) {
    oc[i] = circ[order[i]];
    os[i] = site[order[i]];
    std::memcpy(&og[(size_t)32 * i], gates + (size_t)32 * order[i], sizeof(double) * 32);
  }
  b->order = order;
  const int dev_sms = b->ctas;
  if (b->slab_need() > b->slab_count) {  // launch shapes set since
    cudaFree(b->d_slab);
    b->d_slab = nullptr;
    b->slab_count = 0;
    const size_t need = b->slab_need();
    if (cudaMalloc(&b->d_slab, sizeof(float2) * need) != cudaSuccess) {
      cudaGetLastError();
      return qt_fail(h, QT_ENOMEM, "batch_run: slab allocation failed");
    }
    b->slab_count = need;
  }
  if (ntask > 0) {
    bool ok = cudaMalloc(&b->d_tc, sizeof(int) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_ts, sizeof(int) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_tg, sizeof(double2) * 16 * (size_t)ntask) == cudaSuccess &&
              cudaMalloc(&b->d_rank, sizeof(int) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_sweeps, sizeof(int) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_disc, sizeof(float) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_grank, sizeof(int) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_cert, sizeof(int) * ntask) == cudaSuccess &&
              cudaMalloc(&b->d_left, sizeof(int) * ntask) == cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      return qt_fail(h, QT_ENOMEM, "batch_run: device allocation failed");
    }
    b->ntask_cap = ntask;
    QT_CHECK_CUDA(h, cudaMemcpyAsync(b->d_tc, oc.data(), sizeof(int) * ntask, cudaMemcpyHostToDevice, h->stream));
    QT_CHECK_CUDA(h, cudaMemcpyAsync(b->d_ts, os.data(), sizeof(int) * ntask, cudaMemcpyHostToDevice, h->stream));
    QT_CHECK_CUDA(h, cudaMemcpyAsync(b->d_tg, og.data(), sizeof(double2) * 16 * ntask, cudaMemcpyHostToDevice,
                                     h->stream));
    std::vector<int> grank(ntask);
    for (int t = 0; t < ntask; t++) grank[t] = qt_gate_schmidt_rank(og.data() + 32 * (size_t)t);
    QT_CHECK_CUDA(h, cudaMemcpyAsync(b->d_grank, grank.data(), sizeof(int) * ntask, cudaMemcpyHostToDevice,
                                     h->stream));
    QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  }
  if (b->counter_cap < nseg) {
    cudaFree(b->d_counter);
    b->d_counter = nullptr;
    b->counter_cap = 0;
    if (cudaMalloc(&b->d_counter, sizeof(int) * 3 * std::max(nseg, 1)) != cudaSuccess)
      return qt_fail(h, QT_ENOMEM, "batch_run: counter allocation failed");
    b->counter_cap = nseg;
  }
  BatchArgs a;
  a.sites = b->d_sites; a.site_off = b->d_site_off; a.cap = b->d_cap; a.nsites = b->d_nsites; a.bonds = b->d_bonds;
  a.task_grank = b->d_grank; a.task_cert = b->d_cert;
  a.bond_off = b->d_bond_off; a.task_circ = b->d_tc; a.task_site = b->d_ts; a.task_gate = b->d_tg;
  a.slab = b->d_slab; a.slab_elems = 0; a.smem_elems = 0; a.cutoff = cutoff;
  a.floor_rel = h->cfg.noise_floor;  // <= 0: the default resolution of each task's shape
  // FP32 Jacobi tolerance: a pair is rotated while its relative
  // off-diagonal exceeds 16 u (u = 2^-24).  The FP32 Gram of a converged pair
  // is accurate to a few u at these sizes (m <= 256), so the sweeps still end,
  // one or two after a tolerance of 16 sqrt(m) u would; the truncated state,
  // whose error at a cap inside a dense spectrum grows with the tolerance over
  // the gap at the cut, comes out about 10x closer to the exact split's
  // (a simulated FP32 Jacobi on 256 x 256 Haar-circuit bonds: 6.6e-5 -> 6e-6)
  a.tol = (float)(h->cfg.jacobi_tol > 0 ? h->cfg.jacobi_tol : 16.0 * 5.96e-8);
  a.max_sweeps = std::max(4, h->cfg.max_sweeps);
  a.task_rank = b->d_rank; a.task_sweeps = b->d_sweeps; a.task_discarded = b->d_disc;
  for (int bk = 0; bk < 4; bk++)  // before a capture begins
    if (b->bucket_elems[bk])
      QT_CHECK_CUDA(h, cudaFuncSetAttribute((const void*)layer_kernel(b->threads[bk], bk),
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_smem(bk)));
  QT_CHECK_CUDA(h, cudaFuncSetAttribute((const void*)batch_split64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)S64_SMEM));
  auto launch_all = [&]() -> int {
    QT_CHECK_CUDA(h, cudaMemsetAsync(b->d_counter, 0, sizeof(int) * 3 * std::max(nseg, 1), h->stream));
    for (int sg = 0; sg < nseg; sg++) {
      const int bk = seg_bucket[sg];
      BatchArgs al = a;
      al.task_begin = seg_begin[sg];
      al.task_end = seg_end[sg];
      al.counter = b->d_counter + 3 * sg;
      al.nleft = al.counter + 1;
      al.left = b->d_left + seg_begin[sg];
      const int grid = std::min(dev_sms * b->cps[bk], seg_end[sg] - seg_begin[sg]);
      al.slab_elems = b->bucket_elems[bk];
      al.smem_elems = (int)(batch_smem(bk) / sizeof(float2));
      const layer_fn batch_layer_kernel_fn = layer_kernel(b->threads[bk], bk);
      QT_LAUNCH(h, batch_layer_kernel_fn, grid, b->threads[bk], batch_smem(bk), al);
      al.counter += 2;
      al.alone_above = split64_alone_above(bk);
      QT_LAUNCH(h, batch_split64_kernel, S64_C * b->split_clusters(seg_end[sg] - seg_begin[sg]), S64_NT, S64_SMEM, al);
    }
    return QT_OK;
  };
  if (use_graph) {
    cudaGraph_t g;
    QT_CHECK_CUDA(h, cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    int rc = launch_all();
    cudaError_t e = cudaStreamEndCapture(h->stream, &g);
    if (rc != QT_OK) return rc;
    if (e != cudaSuccess) return qt_fail(h, QT_ECUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return qt_fail(h, QT_ECUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
    QT_CHECK_CUDA(h, cudaGraphLaunch(b->graph, h->stream));
  } else {
    QT_TRY(launch_all());
  }
  QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  return QT_OK;
}

// Replay the last captured program (fresh state needs qt_batch_reset first).
extern "C" int qt_batch_replay(qt_handle* h, qt_batch* b) {
  if (!h || !b || !b->graph) return qt_fail(h, QT_EINVAL, "batch_replay: no captured program");
  cudaSetDevice(h->device);
  QT_CHECK_CUDA(h, cudaGraphLaunch(b->graph, h->stream));
  QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  return QT_OK;
}

// Back to |0...0> on every circuit.
extern "C" int qt_batch_reset(qt_handle* h, qt_batch* b) {
  if (!h || !b) return qt_fail(h, QT_EINVAL, "batch_reset: bad argument");
  cudaSetDevice(h->device);
  std::vector<int> bonds(b->bond_off.back() + b->nsites.back() + 1, 1);
  QT_CHECK_CUDA(h, cudaMemcpyAsync(b->d_bonds, bonds.data(), sizeof(int) * bonds.size(), cudaMemcpyHostToDevice,
                                   h->stream));
  QT_LAUNCH(h, batch_init_kernel, std::min(b->ncirc, 1024), 128, 0, b->d_sites, b->d_site_off, b->d_cap, b->d_nsites,
            b->ncirc);
  QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  return QT_OK;
}

extern "C" int qt_batch_task_stats(qt_handle* h, const qt_batch* b, int* rank, int* sweeps, float* discarded) {
  if (!h || !b) return qt_fail(h, QT_EINVAL, "batch_task_stats: bad argument");
  const int n = b->ntask_cap;
  if (n == 0) return QT_OK;
  // device order -> the caller's task order
  std::vector<int> ri(n), si(n);
  std::vector<float> di(n);
  QT_CHECK_CUDA(h, cudaMemcpy(ri.data(), b->d_rank, sizeof(int) * n, cudaMemcpyDeviceToHost));
  QT_CHECK_CUDA(h, cudaMemcpy(si.data(), b->d_sweeps, sizeof(int) * n, cudaMemcpyDeviceToHost));
  QT_CHECK_CUDA(h, cudaMemcpy(di.data(), b->d_disc, sizeof(float) * n, cudaMemcpyDeviceToHost));
  for (int i = 0; i < n; i++) {
    const int t = b->order[i];
    if (rank) rank[t] = ri[i];
    if (sweeps) sweeps[t] = si[i];
    if (discarded) discarded[t] = di[i];
  }
  return QT_OK;
}

extern "C" int qt_batch_set_launch(qt_handle* h, qt_batch* b, int bucket_cap, int threads, int ctas_per_sm) {
  if (!h || !b) return qt_fail(h, QT_EINVAL, "batch_set_launch: bad argument");
  if (bucket_cap != 16 && bucket_cap != 32 && bucket_cap != 64 && bucket_cap != 128)
    return qt_fail(h, QT_EINVAL, "batch_set_launch: bucket_cap must be 16, 32, 64 or 128");
  if (threads != 128 && threads != 256 && threads != 512 && threads != 1024)
    return qt_fail(h, QT_EINVAL, "batch_set_launch: threads must be 128, 256, 512 or 1024");
  if (ctas_per_sm < 1 || ctas_per_sm > 4) return qt_fail(h, QT_EINVAL, "batch_set_launch: ctas_per_sm must be 1..4");
  const int bk = bucket_of(bucket_cap);
  b->threads[bk] = threads;
  b->cps[bk] = ctas_per_sm;
  return QT_OK;
}

extern "C" int qt_batch_get_launch(const qt_batch* b, int bucket_cap, int* threads, int* ctas_per_sm) {
  if (!b || !threads || !ctas_per_sm) return QT_EINVAL;
  const int bk = bucket_of(bucket_cap);
  *threads = b->threads[bk];
  *ctas_per_sm = b->cps[bk];
  return QT_OK;
}

extern "C" int qt_batch_cert_counts(qt_handle* h, const qt_batch* b, int64_t* out) {
  if (!h || !b || !out) return qt_fail(h, QT_EINVAL, "batch_cert_counts: bad argument");
  for (int i = 0; i < QT_CERT_SLOTS; i++) out[i] = 0;
  const int n = b->ntask_cap;
  if (n == 0) return QT_OK;
  std::vector<int> cert(n);
  QT_CHECK_CUDA(h, cudaMemcpy(cert.data(), b->d_cert, sizeof(int) * n, cudaMemcpyDeviceToHost));
  for (int c : cert) out[(c >= 0 && c < QT_CERT_SLOTS) ? c : QT_CERT_NONE]++;
  return QT_OK;
}

extern "C" int qt_batch_bond_dims(qt_handle* h, const qt_batch* b, int c, int* dims) {
  if (!h || !b || !dims || c < 0 || c >= b->ncirc) return qt_fail(h, QT_EINVAL, "batch_bond_dims: bad argument");
  QT_CHECK_CUDA(h, cudaMemcpy(dims, b->d_bonds + b->bond_off[c], sizeof(int) * (b->nsites[c] + 1),
                              cudaMemcpyDeviceToHost));
  return QT_OK;
}

// Site (0-based) of circuit c as a compact (chiL, 2, chiR) complex64 array.
extern "C" int qt_batch_download_site(qt_handle* h, const qt_batch* b, int c, int s, void* host) {
  if (!h || !b || !host || c < 0 || c >= b->ncirc || s < 0 || s >= b->nsites[c])
    return qt_fail(h, QT_EINVAL, "batch_download_site: bad argument");
  int d[2];
  QT_CHECK_CUDA(h, cudaMemcpy(d, b->d_bonds + b->bond_off[c] + s, sizeof(int) * 2, cudaMemcpyDeviceToHost));
  const size_t slot = (size_t)b->cap[c] * 2 * b->cap[c];
  QT_CHECK_CUDA(h, cudaMemcpy(host, b->d_sites + b->site_off[c] + (size_t)s * slot, sizeof(float2) * d[0] * 2 * d[1],
                              cudaMemcpyDeviceToHost));
  return QT_OK;
}

extern "C" int qt_batch_expect_z(qt_handle* h, qt_batch* b, int site, double* out) {
  if (!h || !b || !out) return qt_fail(h, QT_EINVAL, "batch_expect_z: bad argument");
  for (int c = 0; c < b->ncirc; c++)
    if (site < 0 || site >= b->nsites[c]) return qt_fail(h, QT_EBOUNDS, "batch_expect_z: site out of range");
  cudaSetDevice(h->device);
  double* d_out;
  QT_CHECK_CUDA(h, cudaMalloc(&d_out, sizeof(double) * b->ncirc));
  const int grid = std::min(b->ncirc, b->ctas);
  // the slab holds 16 cap^2 entries per CTA of the widest bucket; the sweep needs 6 cap^2
  batch_expect_kernel<<<grid, BT, cta_gemm_smem<float2>(EXPECT_TILE), h->stream>>>(
      b->d_sites, b->d_site_off, b->d_cap, b->d_nsites, b->d_bonds, b->d_bond_off, b->ncirc, site, b->d_slab,
      b->bucket_elems[bucket_of(b->capmax)], d_out);
  h->launches++;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, d_out, sizeof(double) * b->ncirc, cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(d_out);
  if (e != cudaSuccess) return qt_fail(h, QT_ECUDA, std::string("batch_expect_z: ") + cudaGetErrorString(e));
  return QT_OK;
}
