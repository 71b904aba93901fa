// Expectation values by transfer sweeps in FP64, w_s = 1 or the eigenvalue of
// Z (+1, -1) on the measured sites:
//   from the left   L <- sum_s A_s^H L A_s   up to the measured sites,
//   from the right  R <- sum_s A_s R A_s^H   down to them,
//   across them     L_num <- sum_s w_s A_s^H L_num A_s beside L_den,
// and <psi|O|psi> = tr(L_num R), <psi|psi> = tr(L_den R).  The reference has no
// observable routine; its closure-network pattern is the expectation_value
// cell of examples/expectation_value_optimization_example.ipynb.
//
// What bounds it: FP64 products, 8 chi^3 FMAs a site and direction on two FP64
// lanes per SM.  So every site is passed once for numerator and denominator
// together, L and R (Hermitian) are computed on and above the diagonal tiles
// only, and the two directions' steps share a launch, whose tiles of 16 x 16
// then cover the chip (128 states: 2 x 128 CTAs).  A site (cl, 2, cr) is its
// (cl x 2 cr) matrix with ld cl and its (2 cl x cr) matrix with ld 2 cl in the
// same memory, so both values of s go through one product; complex64 sites are
// widened as they are read.
// <ZZ> on the 15 bonds of 16 sites at 128: 36.1 -> 10.7 ms (one sweep per
// norm and per value, four products and a conversion per site before).
#include <cuda_runtime.h>

#include <algorithm>

#include "qt_internal.cuh"

namespace {

// C (M x N, ld M) = op(A) op(B); rows k >= ksplit of op(B) weighted by w.
struct EnvProduct {
  const void *A, *B;
  double2* C;
  int M, N, K, lda, ldb;
  int a64, b64;            // element: complex128 (else complex64)
  int conj_a, conj_b;      // op = conjugate transpose
  int hermitian;           // C is: tiles below the diagonal are mirrored
  int ksplit;
  double w;
};
struct EnvLaunch { EnvProduct p[2]; };

__device__ inline double2 env_load(const void* p, int wide, size_t i) {
  return wide ? ((const double2*)p)[i] : ccast<double2>(((const float2*)p)[i]);
}

constexpr int ET = 16;  // output tile, depth of a slice
__global__ void __launch_bounds__(ET * ET) env_product_kernel(EnvLaunch l) {
  const EnvProduct& p = l.p[blockIdx.z];
  const int m0 = blockIdx.x * ET, n0 = blockIdx.y * ET;
  if (m0 >= p.M || n0 >= p.N || (p.hermitian && m0 > n0)) return;
  __shared__ double2 As[ET][ET + 1], Bs[ET][ET + 1];  // [k][row], [k][column]
  const int t = threadIdx.x, lo = t % ET, hi = t / ET;
  double2 acc = make_double2(0, 0);
  for (int k0 = 0; k0 < p.K; k0 += ET) {
    {
      const int m = p.conj_a ? hi : lo, k = p.conj_a ? lo : hi;
      double2 v = make_double2(0, 0);
      if (m0 + m < p.M && k0 + k < p.K)
        v = p.conj_a ? cconj(env_load(p.A, p.a64, (k0 + k) + (size_t)p.lda * (m0 + m)))
                     : env_load(p.A, p.a64, (m0 + m) + (size_t)p.lda * (k0 + k));
      As[k][m] = v;
    }
    {
      const int n = p.conj_b ? lo : hi, k = p.conj_b ? hi : lo;
      double2 v = make_double2(0, 0);
      if (n0 + n < p.N && k0 + k < p.K)
        v = p.conj_b ? cconj(env_load(p.B, p.b64, (n0 + n) + (size_t)p.ldb * (k0 + k)))
                     : env_load(p.B, p.b64, (k0 + k) + (size_t)p.ldb * (n0 + n));
      if (k0 + k >= p.ksplit) v = cscale(v, p.w);
      Bs[k][n] = v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < ET; k++) cfma(acc, As[k][lo], Bs[k][hi]);
    __syncthreads();
  }
  const int m = m0 + lo, n = n0 + hi;
  if (m < p.M && n < p.N) {
    p.C[m + (size_t)p.M * n] = acc;
    if (p.hermitian && m0 != n0) p.C[n + (size_t)p.M * m] = cconj(acc);
  }
}

// out[b] = Re tr(L_b R) for Hermitian R (n entries each), one CTA per b
__global__ void __launch_bounds__(512) env_trace_kernel(const double2* L0, const double2* L1, const double2* R,
                                                        int64_t n, double* out) {
  const double2* L = blockIdx.x ? L1 : L0;
  double s = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s = fma(L[i].x, R[i].x, fma(L[i].y, R[i].y, s));
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double red[16];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) tot += red[w];
    out[blockIdx.x] = tot;
  }
}

int env_launch(qt_handle* h, const EnvProduct* p, int count) {
  EnvLaunch l;
  int mt = 0, nt = 0;
  for (int i = 0; i < count; i++) {
    l.p[i] = p[i];
    mt = std::max(mt, (p[i].M + ET - 1) / ET);
    nt = std::max(nt, (p[i].N + ET - 1) / ET);
  }
  for (int i = count; i < 2; i++) l.p[i] = p[0];
  QT_LAUNCH(h, env_product_kernel, dim3((unsigned)mt, (unsigned)nt, (unsigned)count), ET * ET, 0, l);
  return QT_OK;
}

}  // namespace

// *num = <psi|O|psi> (O: Z on `nops` sites from `site`; nops = 0: the identity),
// *den = <psi|psi>; either may be null.
int qt_mps_expect2(qt_handle* h, const qt_mps* mps, int site, int nops, double* num, double* den) {
  const int n = mps->nsites;
  if (nops > 0 && (site < 0 || site + nops > n)) return qt_fail(h, QT_EBOUNDS, "expectation: site out of range");
  const int w64 = mps->dtype == QT_C128;
  int64_t maxchi = 1, maxsite = 1;
  for (int i = 0; i < n; i++) {
    maxchi = std::max(maxchi, std::max(mps->chil[i], mps->chir[i]));
    maxsite = std::max(maxsite, mps->chil[i] * 2 * mps->chir[i]);
  }
  const int lo = nops > 0 ? site : n / 2, hi = nops > 0 ? site + nops : n / 2;  // left chain [0, lo), right chain [hi, n)
  qt_scratch s(h);
  double2 *L, *R, *Lnum, *T, *U;
  double* out;
  QT_TRY(s.get(&L, (size_t)maxchi * maxchi));
  QT_TRY(s.get(&R, (size_t)maxchi * maxchi));
  QT_TRY(s.get(&Lnum, (size_t)maxchi * maxchi));
  QT_TRY(s.get(&T, (size_t)maxsite));
  QT_TRY(s.get(&U, (size_t)maxsite));
  QT_TRY(s.get(&out, 2));
  // the open boundary legs are traced, as <psi|psi> does
  QT_TRY(qt_set_identity<double2>(h, L, mps->chil[0], mps->chil[0]));
  QT_TRY(qt_set_identity<double2>(h, R, mps->chir[n - 1], mps->chir[n - 1]));
  auto left1 = [&](int i, const double2* E, double2* t) {  // t (cl x 2 cr) = E A
    const int cl = (int)mps->chil[i], cr = (int)mps->chir[i];
    return EnvProduct{E, mps->site[i], t, cl, 2 * cr, cl, cl, cl, 1, w64, 0, 0, 0, cl, 1.0};
  };
  auto left2 = [&](int i, const double2* t, double2* E, double w) {  // E (cr x cr) = A^H (w t)
    const int cl = (int)mps->chil[i], cr = (int)mps->chir[i];
    return EnvProduct{mps->site[i], t, E, cr, cr, 2 * cl, 2 * cl, 2 * cl, w64, 1, 1, 0, 1, cl, w};
  };
  auto right1 = [&](int i) {  // U (2 cl x cr) = A R
    const int cl = (int)mps->chil[i], cr = (int)mps->chir[i];
    return EnvProduct{mps->site[i], R, U, 2 * cl, cr, cr, 2 * cl, cr, w64, 1, 0, 0, 0, cr, 1.0};
  };
  auto right2 = [&](int i) {  // R (cl x cl) = U A^H
    const int cl = (int)mps->chil[i], cr = (int)mps->chir[i];
    return EnvProduct{U, mps->site[i], R, cl, cl, 2 * cr, cl, cl, 1, w64, 0, 1, 1, 2 * cr, 1.0};
  };
  for (int a = 0, b = n - 1; a < lo || b >= hi; a++, b--) {
    EnvProduct one[2], two[2];
    int c = 0;
    if (a < lo) { one[c] = left1(a, L, T); two[c++] = left2(a, T, L, 1.0); }
    if (b >= hi) { one[c] = right1(b); two[c++] = right2(b); }
    QT_TRY(env_launch(h, one, c));
    QT_TRY(env_launch(h, two, c));
  }
  const double2* Ln = L;
  for (int i = lo; i < hi; i++) {
    // numerator and denominator part at the first measured site
    EnvProduct one[2] = {left1(i, L, T), left1(i, Lnum, U)};
    QT_TRY(env_launch(h, one, i == lo ? 1 : 2));
    EnvProduct two[2] = {left2(i, T, L, 1.0), left2(i, i == lo ? T : U, Lnum, -1.0)};
    QT_TRY(env_launch(h, two, 2));
    Ln = Lnum;
  }
  const int64_t c = hi < n ? mps->chil[hi] : mps->chir[n - 1];
  QT_LAUNCH(h, env_trace_kernel, 2, 512, 0, L, Ln, R, c * c, out);
  double v[2];
  QT_CHECK_CUDA(h, cudaMemcpyAsync(v, out, sizeof(v), cudaMemcpyDeviceToHost, h->stream));
  QT_CHECK_CUDA(h, cudaStreamSynchronize(h->stream));
  if (den) *den = v[0];
  if (num) *num = v[1];
  return QT_OK;
}

int qt_mps_expect(qt_handle* h, const qt_mps* mps, int site, int nops, double* out) {
  return qt_mps_expect2(h, mps, site, nops, out, nullptr);
}
