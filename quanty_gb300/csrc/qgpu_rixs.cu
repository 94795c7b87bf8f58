// Resonant (RIXS) spectra and the Krylov-basis Lanczos they need.
//
// The reference (ResonantSpectra, Core/ResonantSpectra.cpp:6-283) computes
// <psi|T1^dag G1^dag T2^dag G2 T2 G1 T1|psi> as follows: T1|psi>; a Lanczos of H1 that keeps
// its Krylov vectors (LanczosTriDiagonalizeKrylovCC, Core/Lanczos.cpp:3705); the eigensystem
// of that tridiagonal matrix; for every incident energy w_p the Krylov-projected resolvent
// G1(w_p) T1|psi> = b0 sum_i c_i(p) K_i with c_i(p) = sum_k e_k(i) e_k(0) / (w_p - E_k + i G1/2);
// then for every T2 a Lanczos of H2 on T2 G1 T1 |psi> and the continued fraction.
//
// Here every incident energy and every T2 runs at once: the G1 T1|psi> vectors of all w_p form
// one n1 x (NE1+1) block (one combination kernel over the stored Krylov vectors), T2 is applied
// to the whole block with the multi-vector pull kernel into the common closure basis of all
// T2 targets under H2, and the NT2 (NE1+1) second-stage Lanczos recursions run as one batched
// qg_lanczos_tridiag; all spectra come from one continued-fraction kernel.
#include <cfloat>
#include <cmath>
#include <complex>
#include <vector>

#include "qgpu_internal.cuh"
#include "qgpu_onevec.cuh"

typedef std::complex<double> cd;

static inline unsigned gridn(int64_t n) { return (unsigned)((n + 255) / 256); }

// ------------------------------------------------------------------ small device kernels

// ------------------------------------------------------------------ Krylov-basis Lanczos

#define KRY_PART 2048  // stored vectors per pass: their coefficients fit a block's default shared memory

// scalars of the recursion, in device memory
template <typename T>
struct KryScal {
  T d;            // the last single projection
  double scale;   // 1 / b of the last vector, 0 below 100 DBL_MIN
  double overlap; // sum of the orthogonality test so far
  double keep;    // 0 when the orthogonality test failed
  double err;     // accumulated error of the truncation schedule
  double thr2;    // (eps / err)^2
  unsigned int shares;  // of the test that are done
  unsigned int tickets[2 + 2 * ONE_SHARES];  // single sums, then project and test by share
};

// wo = w - d v_d (d of the pass before; none for the first), then <v|wo> into d, and its real
// part into a_out
template <bool REAL>
__global__ void __launch_bounds__(256)
    k_kry_dot(int64_t n, typename OneT<REAL>::T *__restrict__ w, const typename OneT<REAL>::T *__restrict__ vd,
              const typename OneT<REAL>::T *__restrict__ v, typename OneT<REAL>::T *__restrict__ part,
              KryScal<typename OneT<REAL>::T> *sc, double *a_out) {
  typedef typename OneT<REAL>::T T;
  const T d = sc->d;
  one_multidot<T>(
      v, n, 1,
      [&](int64_t r) {
        if (!vd) return w[r];
        const T x = one_sub(w[r], d, vd[r]);
        w[r] = x;
        return x;
      },
      part, &sc->tickets[0],
      [&](int, T t) {
        sc->d = t;
        if (a_out) *a_out = one_complex(t).x;
      });
}

// wo = w - d v_d (or wo = w without v_d), then c_i = <v_i|wo> for i < k
template <bool REAL>
__global__ void __launch_bounds__(256)
    k_kry_project(const typename OneT<REAL>::T *__restrict__ V, int64_t n, int k, const typename OneT<REAL>::T *w,
                  const typename OneT<REAL>::T *__restrict__ vd, typename OneT<REAL>::T *wo,
                  typename OneT<REAL>::T *__restrict__ part, typename OneT<REAL>::T *__restrict__ c,
                  KryScal<typename OneT<REAL>::T> *sc) {
  typedef typename OneT<REAL>::T T;
  const T d = sc->d;
  one_multidot<T>(
      V, n, k,
      [&](int64_t r) {
        if (!vd) return w[r];
        const T x = one_sub(w[r], d, vd[r]);
        if (blockIdx.y == 0) wo[r] = x;
        return x;
      },
      part, &sc->tickets[2], [&](int i, T t) { c[i] = t; });
}

// w -= sum_i c_i v_i (i < k); done: its norm into b and the scale
template <bool REAL>
__global__ void __launch_bounds__(128)
    k_kry_update(const typename OneT<REAL>::T *__restrict__ V, int64_t n, int k, const typename OneT<REAL>::T *__restrict__ c,
                 typename OneT<REAL>::T *__restrict__ w, double *__restrict__ part,
                 KryScal<typename OneT<REAL>::T> *sc, double *b_out, int done) {
  typedef typename OneT<REAL>::T T;
  extern __shared__ __align__(16) char kry_smem[];
  T *cs = reinterpret_cast<T *>(kry_smem);
  __shared__ double sh[4];
  __shared__ int s_last;
  const int tid = threadIdx.x;
  for (int i = tid; i < k; i += 128) cs[i] = c[i];
  __syncthreads();
  double s = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * 128 + tid; r < n; r += (int64_t)gridDim.x * 128) {
    const T x = one_minus_sum(w[r], V, n, k, cs, r);
    if (k) w[r] = x;
    s += one_norm2(x);
  }
  if (!done) return;
  s = one_total128(s, part, sh, &s_last, &sc->tickets[1]);
  if (s_last && tid == 0) {
    const double b = sqrt(s);
    *b_out = b;
    sc->scale = (b < 100 * DBL_MIN) ? 0.0 : 1.0 / b;
  }
}

// v = scale w (the first part), and the reference's orthogonality test of it against the k vectors
// of this part: sum_i |<v_i|v>|^2 over the parts > eps loses it (keep = 0); after the last part
// the truncation schedule err *= b^2/(b^2 + DBL_MIN + DBL_EPSILON a^2), thr2 = (eps / err)^2
template <bool REAL>
__global__ void __launch_bounds__(256)
    k_kry_test(const typename OneT<REAL>::T *__restrict__ V, int64_t n, int k, const typename OneT<REAL>::T *__restrict__ w,
               typename OneT<REAL>::T *__restrict__ v, typename OneT<REAL>::T *__restrict__ part,
               typename OneT<REAL>::T *__restrict__ c, KryScal<typename OneT<REAL>::T> *sc, double eps, const double *a_i, const double *b_i, int first,
               int done) {
  typedef typename OneT<REAL>::T T;
  const double scale = sc->scale;
  __shared__ int s_all;
  const bool last = one_multidot<T>(
      V, n, k,
      [&](int64_t r) {
        if (!first) return v[r];
        const T x = one_scaled(w[r], scale);
        if (blockIdx.y == 0) v[r] = x;
        return x;
      },
      part, &sc->tickets[2 + ONE_SHARES], [&](int i, T t) { c[i] = t; });
  if (!last) return;
  __syncthreads();
  if (threadIdx.x == 0) {  // the last share's block adds the squares of all sums
    __threadfence();
    s_all = atomicAdd(&sc->shares, 1u) == gridDim.y - 1;
    if (s_all) sc->shares = 0u;
  }
  __syncthreads();
  if (!s_all || threadIdx.x >= 32) return;
  __threadfence();
  double t2 = 0.0;
  for (int i = threadIdx.x; i < k; i += 32) t2 += one_abs2(one_ldcg(c + i));
  for (int o = 16; o; o >>= 1) t2 += __shfl_xor_sync(0xffffffffu, t2, o);
  if (threadIdx.x == 0) {
    if (!first) t2 += sc->overlap;
    sc->overlap = t2;
    if (!done) return;
    sc->keep = t2 > eps ? 0.0 : 1.0;
    const double b = *b_i, a = *a_i;
    const double e = sc->err * (b * b / (b * b + DBL_MIN + DBL_EPSILON * a * a));
    sc->err = e;
    const double th = eps / e;
    sc->thr2 = th * th;
  }
}

// the test's verdict and the truncation: |v_r|^2 <= thr2 drops; `in` times the scale when given
template <bool REAL>
__global__ void k_kry_trunc(int64_t n, typename OneT<REAL>::T *__restrict__ v, const typename OneT<REAL>::T *__restrict__ in,
                            const KryScal<typename OneT<REAL>::T> *__restrict__ sc) {
  typedef typename OneT<REAL>::T T;
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  T x = in ? one_scaled(in[r], sc->scale) : one_scaled(v[r], sc->keep);
  if (!(one_abs2(x) > sc->thr2)) x = one_zero(T());
  v[r] = x;
}

// Lanczos keeping the Krylov vectors, the reference's LanczosTriDiagonalizeKrylovCC: modified
// Gram-Schmidt of H K_{i-1} against all earlier vectors in reverse order, normalisation, the
// orthogonality test, truncation at eps/err.  The first two projections (K_{i-1}, K_{i-2}) are
// taken one after the other; what is left along the others is rounding and truncation, so
// their order does not matter and one pass over the stored vectors takes them together.  Each
// vector is projected out once, as in the reference: past an invariant space the remainder
// then fails the orthogonality test, which ends the list of vectors.  Seven launches per step
// instead of four per stored vector, and no single-thread sum: with 24 vectors of 290,280
// determinants the RIXS of a 46-orbital impurity takes 60 ms instead of 83.
template <bool REAL>
static qg_status lanczos_krylov_t(qg_context ctx, qg_operator op, qg_basis b, const double2 *v0, int ntri, double eps,
                                  double *a_host, double *b_host, double2 *Kout) {
  typedef typename OneT<REAL>::T T;
  cudaStream_t s = ctx->stream;
  const int64_t n = b->n;
  const unsigned gp = one_multidot_grid(ctx, n, 1).x;
  const unsigned gu = (unsigned)std::min<int64_t>((n + 127) / 128, 8LL * ctx->num_sms);
  const int Pa = qg_apply_grid(b);
  T *K = nullptr, *w = nullptr, *wo = nullptr, *part = nullptr, *c = nullptr;
  double *ab = nullptr, *npart = nullptr, *zero = nullptr;
  double2 *dpart = nullptr;
  KryScal<T> *sc = nullptr;
  cudaError_t e = qg_malloc(ctx, &w, n * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &wo, n * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &part, (size_t)gp * std::min(ntri, KRY_PART) * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &c, (size_t)std::min(ntri, KRY_PART) * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &ab, (2 * (size_t)ntri + 1) * sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &npart, (size_t)gu * sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &sc, sizeof(KryScal<T>));
  if (REAL) {  // real vectors of their own, handed out as complex ones at the end
    if (e == cudaSuccess) e = qg_malloc(ctx, &K, (size_t)n * ntri * sizeof(T));
    if (e == cudaSuccess) e = qg_malloc(ctx, &dpart, (size_t)Pa * 16);
    if (e == cudaSuccess) e = qg_malloc(ctx, &zero, sizeof(double));
    if (e == cudaSuccess) e = cudaMemsetAsync(zero, 0, sizeof(double), s);
  } else {
    K = reinterpret_cast<T *>(Kout);
  }
  KryScal<T> init = {};
  init.err = 1.0;
  init.keep = 1.0;
  init.thr2 = eps * eps;
  if (e == cudaSuccess) e = cudaMemcpyAsync(sc, &init, sizeof(init), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(ab, 0, (2 * (size_t)ntri + 1) * sizeof(double), s);
  qg_status st = e == cudaSuccess ? QG_OK : qg_cuda_fail(ctx, e, "lanczos_krylov");
  if (st == QG_OK) st = qg_apply_prepare(ctx, op, b, ntri);
  double *ah = ab, *bh = ab + ntri + 1;
  const unsigned g1 = gridn(n);
  auto apply = [&](const T *x, T *y) -> qg_status {
    if (!REAL) return qg_apply_launch(ctx, op, b, b, (const double *)x, (double *)y, 1, nullptr);
    ApplyFuse fz;  // the real-vector form of the list apply is its fused one: y = H x - 0 x
    fz.prev = (const double2 *)x;
    fz.beta = zero;
    fz.dot_part = dpart;
    fz.real_vector = 1;
    return qg_apply_strided(ctx, op, b, b, (const double *)x, 1, (double *)y, 1, 1, &fz);
  };
  if (st == QG_OK) {  // K_0
    k_one_in<REAL><<<g1, 256, 0, s>>>(n, v0, w);
    k_kry_update<REAL><<<gu, 128, 0, s>>>(K, n, 0, c, w, npart, sc, bh, 1);
    k_kry_trunc<REAL><<<g1, 256, 0, s>>>(n, K, w, sc);
    ctx->launches += 3;
    st = qg_check_launch(ctx, "lanczos_krylov");
  }
  for (int i = 1; i < ntri && st == QG_OK; i++) {
    T *Ki = K + (int64_t)i * n, *p1 = Ki - n, *p2 = p1 - n;
    st = apply(p1, w);
    if (st != QG_OK) break;
    k_kry_dot<REAL><<<gp, 256, one_multidot_smem<T>(1), s>>>(n, w, nullptr, p1, part, sc, ah + i);
    if (i >= 2) {
      k_kry_dot<REAL><<<gp, 256, one_multidot_smem<T>(1), s>>>(n, w, p1, p2, part, sc, nullptr);
      ctx->launches++;
    }
    // the stored vectors in parts that a block's shared memory holds the coefficients of
    const int k = std::max(0, i - 2), np = std::max(1, (k + KRY_PART - 1) / KRY_PART);
    for (int p = 0; p < np; p++) {
      const int k0 = p * KRY_PART, kp = std::min(KRY_PART, k - k0);
      k_kry_project<REAL><<<one_multidot_grid(ctx, n, kp), 256, one_multidot_smem<T>(kp), s>>>(
          K + (int64_t)k0 * n, n, kp, p ? wo : w, p ? nullptr : i >= 2 ? p2 : p1, wo, part, c, sc);
      k_kry_update<REAL><<<gu, 128, (size_t)kp * sizeof(T), s>>>(K + (int64_t)k0 * n, n, kp, c, wo, npart, sc, bh + i,
                                                                 p == np - 1);
    }
    const int nt = (i + KRY_PART - 1) / KRY_PART;
    for (int p = 0; p < nt; p++) {
      const int k0 = p * KRY_PART, kp = std::min(KRY_PART, i - k0);
      k_kry_test<REAL><<<one_multidot_grid(ctx, n, kp), 256, one_multidot_smem<T>(kp), s>>>(
          K + (int64_t)k0 * n, n, kp, wo, Ki, part, c, sc, eps, ah + i, bh + i, p == 0, p == nt - 1);
    }
    k_kry_trunc<REAL><<<g1, 256, 0, s>>>(n, Ki, nullptr, sc);
    ctx->launches += 2 + 2 * np + nt;
    st = qg_check_launch(ctx, "lanczos_krylov");
  }
  if (st == QG_OK) {  // a[ntri] = <K_last|H|K_last>
    T *last = K + (int64_t)(ntri - 1) * n;
    st = apply(last, w);
    if (st == QG_OK) {
      k_kry_dot<REAL><<<gp, 256, one_multidot_smem<T>(1), s>>>(n, w, nullptr, last, part, sc, ah + ntri);
      ctx->launches++;
    }
  }
  if (st == QG_OK && REAL) {
    k_one_out<REAL><<<gridn(n * ntri), 256, 0, s>>>(n * ntri, K, Kout);
    ctx->launches++;
    st = qg_check_launch(ctx, "lanczos_krylov");
  }
  if (st == QG_OK) {
    e = cudaMemcpyAsync(a_host, ah, (ntri + 1) * 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(b_host, bh, ntri * 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) st = qg_cuda_fail(ctx, e, "lanczos_krylov");
    a_host[0] = 0.0;
  }
  cudaStreamSynchronize(s);
  qg_free(w);
  qg_free(wo);
  qg_free(part);
  qg_free(c);
  qg_free(ab);
  qg_free(npart);
  qg_free(sc);
  if (REAL) qg_free(K);
  qg_free(dpart);
  qg_free(zero);
  return st;
}

// K_dev: ntri * n complex (vector-major).  A real operator (with connection lists) on a real
// vector keeps every vector real; without room for the real vectors beside K_dev the complex
// form runs.
static qg_status lanczos_krylov(qg_context ctx, qg_operator op, qg_basis b, const double *v0, int ntri, double eps,
                                double *a_host, double *b_host, double2 *K) {
  bool real = qg_operator_values_real(op) && qg_apply_uses_lists(op, b);
  if (real) QG_TRY(qg_all_real(ctx, (const double2 *)v0, b->n, &real));
  if (real) {
    const qg_status st = lanczos_krylov_t<true>(ctx, op, b, (const double2 *)v0, ntri, eps, a_host, b_host, K);
    if (st != QG_ERR_OOM) return st;
  }
  return lanczos_krylov_t<false>(ctx, op, b, (const double2 *)v0, ntri, eps, a_host, b_host, K);
}

extern "C" qg_status qg_lanczos_krylov(qg_context ctx, qg_operator op, qg_basis b, const double *v0_dev, int32_t ntri,
                                       double eps, double *a_host, double *b_host, double *krylov_dev) {
  if (!ctx || !op || !b || !v0_dev || ntri <= 0 || !a_host || !b_host || !krylov_dev || op->nf != b->nf)
    return QG_ERR_ARG;
  if (!b->n) return QG_ERR_ARG;
  qg_status st = lanczos_krylov(ctx, op, b, v0_dev, ntri, eps, a_host, b_host, (double2 *)krylov_dev);
  if (st == QG_OK) st = qg_check_device_error(ctx, "qg_lanczos_krylov");
  return st;
}

// ------------------------------------------------------------------ RIXS

extern "C" qg_status qg_resonant_spectra(qg_context ctx, qg_operator H1, qg_operator H2, qg_operator T1,
                                         const qg_operator *T2, int32_t nt2, qg_basis psi_basis, const double *psi_dev,
                                         qg_rixs_settings *o, double *g_host) {
  if (!ctx || !H1 || !H2 || !T1 || !T2 || nt2 <= 0 || !psi_basis || !psi_dev || !o || !g_host) return QG_ERR_ARG;
  if (o->ntri1 <= 0 || o->ntri2 <= 0 || o->ne1 <= 0 || o->ne2 <= 0) return QG_ERR_ARG;
  cudaStream_t s = ctx->stream;
  qg_status st = QG_OK;
  // energies <psi|H|psi>/<psi|psi>
  double nrm2 = 0;
  {
    double t[2];
    QG_TRY(qg_dot(ctx, psi_basis->n, 1, psi_dev, psi_dev, t));
    nrm2 = t[0];
  }
  double div = nrm2 > DBL_EPSILON ? nrm2 : 1.0;
  if (o->energy1 == DBL_MAX) {
    double v[2];
    QG_TRY(qg_expectation(ctx, H1, psi_basis, psi_dev, 1, v));
    o->energy1 = v[0] / div;
  }
  if (o->energy2 == DBL_MAX) {
    double v[2];
    QG_TRY(qg_expectation(ctx, H2, psi_basis, psi_dev, 1, v));
    o->energy2 = v[0] / div;
  }
  // T1 |psi> on its target basis, then on the closure under H1
  qg_basis bt = nullptr, b1 = nullptr, bt2 = nullptr, b2 = nullptr;
  double *tpsi = nullptr, *x1 = nullptr, *K = nullptr, *gt = nullptr, *x2 = nullptr;
  double2 *Cd = nullptr;
  int np = o->ne1 + 1, ncol = nt2 * np;
  std::vector<double> a1(o->ntri1 + 1), b1v(o->ntri1);
  cudaError_t e = cudaSuccess;
  do {
    if ((st = qg_operator_psi_basis(ctx, T1, psi_basis, o->res1, &bt)) != QG_OK) break;
    if ((e = qg_malloc(ctx, &tpsi, std::max<int64_t>(bt->n, 1) * 16)) != cudaSuccess) break;
    if ((st = qg_apply(ctx, T1, bt, psi_basis, psi_dev, tpsi, 1)) != QG_OK) break;
    int rounds = 0;
    if ((st = qg_basis_closure(ctx, H1, bt, o->res1, -1, &b1, &rounds)) != QG_OK) break;
    int64_t n1 = b1->n;
    if ((e = qg_malloc(ctx, &x1, std::max<int64_t>(n1, 1) * 16)) != cudaSuccess) break;
    if ((st = qg_basis_map(ctx, bt, tpsi, b1, x1, 1)) != QG_OK) break;
    if ((e = qg_malloc(ctx, &K, (size_t)o->ntri1 * std::max<int64_t>(n1, 1) * 16)) != cudaSuccess) break;
    if ((st = lanczos_krylov(ctx, H1, b1, x1, o->ntri1, o->epsilon, a1.data(), b1v.data(), (double2 *)K)) != QG_OK)
      break;
    // diagonal a[1..nt], off-diagonal b[1..nt-1] (TriDiagonalMatrixToEigensystem's matrix)
    std::vector<double> ev(o->ntri1), Z((size_t)o->ntri1 * o->ntri1);
    if ((st = qg_tri_eigh(ctx, o->ntri1, a1.data() + 1, b1v.data() + 1, o->ntri1, ev.data(), Z.data())) != QG_OK) break;
    int nt = o->ntri1;
    // intermediate-state energy range defaults (Core/ResonantSpectra.cpp:80-112)
    if (o->emin1 > 0.001 * DBL_MAX && o->emax1 < -0.001 * DBL_MAX) {
      o->emin1 = 1.1 * ev[0] - 0.1 * ev[nt - 1];
      o->emax1 = 1.1 * ev[nt - 1] - 0.1 * ev[0];
    }
    if (o->emin1 > 0.001 * DBL_MAX) o->emin1 = 1.1 * ev[0] - 0.1 * o->emax1;
    if (o->emax1 < -0.001 * DBL_MAX) o->emax1 = 1.1 * ev[nt - 1] - 0.1 * o->emin1;
    if (o->gamma1 == 0 && o->ne1 == 0) {
      o->ne1 = 1000;
      o->gamma1 = 5 * (o->emax1 - o->emin1) / o->ne1;
    }
    if (o->ne1 == 0) o->ne1 = (int32_t)(5 * (o->emax1 - o->emin1) / o->gamma1);
    if (o->gamma1 == 0) o->gamma1 = 5 * (o->emax1 - o->emin1) / o->ne1;
    np = o->ne1 + 1;
    ncol = nt2 * np;
    // Krylov-projected resolvent coefficients, all incident energies
    std::vector<cd> C((size_t)nt * np);
    for (int p = 0; p < np; p++) {
      double w = o->emin1 + (o->emax1 - o->emin1) * p / (double)o->ne1 + o->energy1;
      for (int i = 0; i < nt; i++) {
        cd acc(0, 0);
        for (int k = 0; k < nt; k++) {
          cd inv = 1.0 / cd(w - ev[k], 0.5 * o->gamma1);
          acc += inv * Z[(size_t)i * nt + k] * Z[(size_t)k] * 1.0;  // e_k(i) e_k(0)
        }
        C[(size_t)i * np + p] = b1v[0] * acc;
      }
    }
    if ((e = qg_malloc(ctx, &Cd, C.size() * 16)) != cudaSuccess) break;
    if ((e = cudaMemcpyAsync(Cd, C.data(), C.size() * 16, cudaMemcpyHostToDevice, s)) != cudaSuccess) break;
    if ((e = qg_malloc(ctx, &gt, (size_t)std::max<int64_t>(n1, 1) * np * 16)) != cudaSuccess) break;
    if ((st = qg_block_combine(ctx, (const double2 *)K, n1, nt, Cd, np, (double2 *)gt)) != QG_OK) break;
    // T2 targets of all operators, their closure under H2: the common final-state basis
    for (int j = 0; j < nt2 && st == QG_OK; j++) {
      qg_basis tj = nullptr;
      st = qg_operator_psi_basis(ctx, T2[j], b1, o->res2, &tj);
      if (st != QG_OK) break;
      if (!bt2) {
        bt2 = tj;
      } else {
        qg_basis u = nullptr;
        st = qg_basis_union(ctx, bt2, tj, &u);
        qg_basis_destroy(bt2);
        qg_basis_destroy(tj);
        bt2 = u;
      }
    }
    if (st != QG_OK) break;
    if ((st = qg_basis_closure(ctx, H2, bt2, o->res2, -1, &b2, &rounds)) != QG_OK) break;
    int64_t n2 = b2->n;
    if ((e = qg_malloc(ctx, &x2, (size_t)std::max<int64_t>(n2, 1) * ncol * 16)) != cudaSuccess) break;
    for (int j = 0; j < nt2 && st == QG_OK; j++)
      st = qg_apply_strided(ctx, T2[j], b2, b1, gt, np, x2 + 2 * (size_t)j * np, ncol, np, nullptr, false);
    if (st != QG_OK) break;
    // all second-stage recursions at once
    std::vector<double> a2((size_t)ncol * (o->ntri2 + 1)), b2v((size_t)ncol * o->ntri2);
    st = qg_lanczos_tridiag(ctx, H2, b2, x2, ncol, o->ntri2, o->epsilon, std::sqrt(DBL_EPSILON) + o->gamma2, a2.data(),
                            b2v.data(), nullptr);
    if (st != QG_OK) break;
    // final-state energy range from the poles (Core/ResonantSpectra.cpp:221-262)
    double lo = DBL_MAX, hi = -DBL_MAX;
    std::vector<double> ends(2 * (size_t)ncol);
    if ((st = qg_tri_extremes(ctx, ncol, o->ntri2, a2.data(), b2v.data(), 0, ends.data())) != QG_OK) break;
    for (int c = 0; c < ncol; c++) {
      lo = std::min(lo, ends[2 * c] - o->energy2);
      hi = std::max(hi, ends[2 * c + 1] - o->energy2);
    }
    if (o->emin2 > 0.001 * DBL_MAX || o->emax2 < -0.001 * DBL_MAX) {
      if (o->emin2 > 0.001 * DBL_MAX && o->emax2 < -0.001 * DBL_MAX) {
        o->emin2 = 1.1 * lo - 0.1 * hi;
        o->emax2 = 1.1 * hi - 0.1 * lo;
      } else if (o->emin2 > 0.001 * DBL_MAX) {
        o->emin2 = 1.1 * lo - 0.1 * o->emax2;
      } else {
        o->emax2 = 1.1 * hi - 0.1 * o->emin2;
      }
    }
    if (o->gamma2 == 0 && o->ne2 == 0) {
      o->ne2 = 1000;
      o->gamma2 = 5 * (o->emax2 - o->emin2) / o->ne2;
    }
    if (o->ne2 == 0) o->ne2 = (int32_t)(5 * (o->emax2 - o->emin2) / o->gamma2);
    if (o->gamma2 == 0) o->gamma2 = 5 * (o->emax2 - o->emin2) / o->ne2;
    std::vector<double> e0(ncol, o->energy2);
    st = qg_cf_spectra(ctx, ncol, o->ntri2, a2.data(), b2v.data(), e0.data(), o->emin2,
                       (o->emax2 - o->emin2) / o->ne2, o->ne2, o->gamma2, g_host);
  } while (0);
  if (e != cudaSuccess && st == QG_OK) st = qg_cuda_fail(ctx, e, "qg_resonant_spectra");
  cudaStreamSynchronize(s);
  qg_free(tpsi);
  qg_free(x1);
  qg_free(K);
  qg_free(Cd);
  qg_free(gt);
  qg_free(x2);
  qg_basis_destroy(bt);
  qg_basis_destroy(b1);
  qg_basis_destroy(bt2);
  qg_basis_destroy(b2);
  if (st == QG_OK) st = qg_check_device_error(ctx, "qg_resonant_spectra");
  return st;
}
