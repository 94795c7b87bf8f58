// Lowest eigenpairs of a Hermitian operator on a fixed basis: restarted block Lanczos with
// full (twice repeated) reorthogonalisation and Rayleigh-Ritz restarts.
//
// The reference's solver (BlockLanczosGroundStateConserveBasisKrylovComplex,
// Core/BlockLanczos.cpp:5350-5606) grows a block Krylov space with fixed-basis H*psi
// (:5489-5496), reorthogonalises twice against all Krylov vectors (:5498-5527), diagonalises
// the projected matrix with zheevd (:5530) and restarts from the Ritz vectors (:5554-5573)
// until the variance <H^2> - <H>^2 of every vector is below "Zero".  The same structure here:
// H*psi is the pull kernel, the Gram products and updates of whole blocks are plain complex
// products over the n x K Krylov block (row-major, K columns; qgpu_blocks.cu), single
// columns use the partial-sum kernels below, and the projected matrix (K <= a few hundred)
// is diagonalised on the device (cyclic Jacobi, qgpu_jacobi.cu), its lowest eigenvectors left
// in device memory for the Ritz combination.
//
// Block size: when more than three states are wanted, a few guard vectors join the block
// (up to half the wanted count, at most 8) and only the wanted states are tested for
// convergence, so a cluster of nearly degenerate states straddling the last wanted one does
// not stall the restarts.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "qgpu_internal.cuh"
#include "qgpu_onevec.cuh"

typedef std::complex<double> cd;

// C[i][j] partial = sum_rows conj(A[r][a0+i]) * B[r][b0+j]; thread per (i, j), gridDim.y row chunks
__global__ void k_gram_partial(const double2 *__restrict__ A, int lda, int a0, int ka, const double2 *__restrict__ B,
                               int ldb, int b0, int kb, int64_t n, int64_t chunk, double2 *part) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ka * kb) return;
  int i = q / kb, j = q % kb;  // row-major C[i * kb + j], the layout every consumer reads
  int64_t r0 = blockIdx.y * chunk, r1 = r0 + chunk;
  if (r1 > n) r1 = n;
  double sr = 0, si = 0;
  for (int64_t r = r0; r < r1; r++) {
    double2 a = A[r * lda + a0 + i], b = B[r * ldb + b0 + j];
    sr += a.x * b.x + a.y * b.y;
    si += a.x * b.y - a.y * b.x;
  }
  part[(int64_t)blockIdx.y * ka * kb + q] = make_double2(sr, si);
}

// Gram products against ONE column b (kb = 1): part[blk][i] = sum over the block's rows of
// conj(A[r][a0+i]) b[r].  With ka <= 8 a thread takes whole rows and keeps the ka sums in
// registers; with more columns a warp takes a row and its lanes take the columns (coalesced
// reads of the row).  Grid-stride over rows with many blocks, so the reduction is wide rather
// than a long serial walk per thread; sums are combined in a fixed order.
// REAL (also below): both sides are real, one multiply-add per term.
template <int KMAX, bool REAL>
__global__ void k_gram_col_rows(const double2 *__restrict__ A, int lda, int a0, int ka, const double2 *__restrict__ B,
                                int ldb, int b0, int64_t n, double2 *part) {
  __shared__ double2 sh[8][KMAX];
  double2 acc[KMAX];
#pragma unroll
  for (int i = 0; i < KMAX; i++) acc[i] = make_double2(0.0, 0.0);
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    double2 b = B[r * ldb + b0];
#pragma unroll
    for (int i = 0; i < KMAX; i++) {
      if (i < ka) {
        double2 a = A[r * lda + a0 + i];
        if (REAL) {
          acc[i].x += a.x * b.x;
        } else {
          acc[i].x += a.x * b.x + a.y * b.y;
          acc[i].y += a.x * b.y - a.y * b.x;
        }
      }
    }
  }
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < KMAX; i++) {
    double2 v = acc[i];
    for (int o = 16; o; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if (lane == 0) sh[wid][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < ka) {
    double2 t = make_double2(0.0, 0.0);
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      t.x += sh[w][threadIdx.x].x;
      t.y += sh[w][threadIdx.x].y;
    }
    part[(int64_t)blockIdx.x * ka + threadIdx.x] = t;
  }
}

#define QG_GRAM_LANE_COLS 8  // columns per lane at most: ka <= 256
template <int M, bool REAL>
__global__ void k_gram_col_lanes(const double2 *__restrict__ A, int lda, int a0, int ka,
                                 const double2 *__restrict__ B, int ldb, int b0, int64_t n, double2 *part) {
  __shared__ double2 sh[8][32 * M];
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double2 acc[M];
#pragma unroll
  for (int m = 0; m < M; m++) acc[m] = make_double2(0.0, 0.0);
  for (int64_t r = (int64_t)blockIdx.x * nw + wid; r < n; r += (int64_t)gridDim.x * nw) {
    double2 b = B[r * ldb + b0];
#pragma unroll
    for (int m = 0; m < M; m++) {
      int i = lane + 32 * m;
      if (i < ka) {
        double2 a = A[r * lda + a0 + i];
        if (REAL) {
          acc[m].x += a.x * b.x;
        } else {
          acc[m].x += a.x * b.x + a.y * b.y;
          acc[m].y += a.x * b.y - a.y * b.x;
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < M; m++) sh[wid][lane + 32 * m] = acc[m];
  __syncthreads();
  for (int i = threadIdx.x; i < ka; i += blockDim.x) {
    double2 t = make_double2(0.0, 0.0);
    for (int w = 0; w < nw; w++) {
      t.x += sh[w][i].x;
      t.y += sh[w][i].y;
    }
    part[(int64_t)blockIdx.x * ka + i] = t;
  }
}

__global__ void k_gram_reduce(const double2 *part, int nchunk, int m, double2 *out) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m) return;
  double sr = 0, si = 0;
  for (int c = 0; c < nchunk; c++) {
    sr += part[(int64_t)c * m + q].x;
    si += part[(int64_t)c * m + q].y;
  }
  out[q] = make_double2(sr, si);
}

// the same with a warp per output: lanes stride over the partials, then a shuffle tree
__global__ void k_gram_reduce_warp(const double2 *part, int nchunk, int m, double2 *out) {
  int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (q >= m) return;
  double sr = 0, si = 0;
  for (int c = lane; c < nchunk; c += 32) {
    sr += part[(int64_t)c * m + q].x;
    si += part[(int64_t)c * m + q].y;
  }
  for (int o = 16; o; o >>= 1) {
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    si += __shfl_xor_sync(0xffffffffu, si, o);
  }
  if (lane == 0) out[q] = make_double2(sr, si);
}


// deterministic pseudo-random fill of columns c0 .. c0+k-1 (guard vectors); real entries for
// a real operator, so real start vectors keep the whole block, and the eigenvectors, real
__global__ void k_fill_cols(double2 *B, int ldb, int c0, int k, int64_t n, uint64_t salt, int real) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n * k) return;
  int64_t r = i / k;
  int c = (int)(i % k);
  uint64_t h = qg_mix64((uint64_t)i * 0x9e3779b97f4a7c15ull + salt);
  double a = (double)(h >> 11) * (1.0 / 9007199254740992.0) - 0.5;
  double b = (double)(qg_mix64(h) >> 11) * (1.0 / 9007199254740992.0) - 0.5;
  B[r * ldb + c0 + c] = make_double2(a, real ? 0.0 : b);
}

// flag = 1 when any of the n values has a non-zero imaginary part (one global OR per block)
__global__ void k_any_imag(const double2 *__restrict__ v, int64_t n, unsigned int *flag) {
  int found = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n && !found;
       i += (int64_t)gridDim.x * blockDim.x)
    found = v[i].y != 0.0;
  if (__syncthreads_or(found) && threadIdx.x == 0) atomicOr(flag, 1u);
}

__global__ void k_copy_cols(const double2 *src, int lds, int s0, double2 *dst, int ldd, int d0, int k, int64_t n) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * k) return;
  int64_t r = t / k;
  int j = (int)(t % k);
  dst[r * ldd + d0 + j] = src[r * lds + s0 + j];
}

namespace {

struct Gram {
  qg_context ctx;
  int64_t n;
  double2 *part = nullptr, *out = nullptr;
  int64_t cap = 0, part_elems = 0;
  int nchunk = 1;
  int64_t chunk = 1;
  int nblk = 1;  // blocks of the one-column Gram kernels
  bool real = false;  // every vector real
  qg_status init(qg_context c, int64_t nn, int maxm, int kcol) {
    ctx = c;
    n = nn;
    chunk = std::max<int64_t>(4096, (nn + 1023) / 1024);
    nchunk = (int)((nn + chunk - 1) / chunk);
    if (nchunk < 1) nchunk = 1;
    nblk = (int)std::max<int64_t>(1, std::min<int64_t>(4LL * c->num_sms, (nn + 255) / 256));
    cap = maxm;
    // partial sums: one column against up to kcol columns (nchunk chunks, or nblk blocks of the
    // one-column kernels), or the row-chunk tiles of a block product (qg_block_gram uses as many
    // chunks as fit, at most the few dozen that fill the SMs)
    part_elems = std::max<int64_t>(std::max<int64_t>(nchunk * (int64_t)kcol, (int64_t)nblk * 32 * QG_GRAM_LANE_COLS), 16 * (int64_t)maxm);
    QG_CUDA(ctx, qg_malloc(ctx, &part, (size_t)part_elems * 16));
    QG_CUDA(ctx, qg_malloc(ctx, &out, (size_t)maxm * 16));
    return QG_OK;
  }
  void release() {
    qg_free(part);
    qg_free(out);
  }
  template <bool REAL>
  void col_gram(cudaStream_t s, const double2 *A, int lda, int a0, int ka, const double2 *B, int ldb, int b0) {
    if (ka == 1)
      k_gram_col_rows<1, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
    else if (ka <= 4)
      k_gram_col_rows<4, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
    else if (ka <= 8)
      k_gram_col_rows<8, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
    else if (ka <= 32)
      k_gram_col_lanes<1, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
    else if (ka <= 64)
      k_gram_col_lanes<2, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
    else if (ka <= 128)
      k_gram_col_lanes<4, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
    else
      k_gram_col_lanes<8, REAL><<<nblk, 256, 0, s>>>(A, lda, a0, ka, B, ldb, b0, n, part);
  }
  // out (device) and host = A[:, a0:a0+ka]^dag B[:, b0:b0+kb]
  qg_status run(const double2 *A, int lda, int a0, int ka, const double2 *B, int ldb, int b0, int kb,
                std::vector<cd> *host) {
    int m = ka * kb;
    if (m > cap || m <= 0) return QG_ERR_ARG;
    if (kb > 1) {  // a block against a block: tiled products, partial sums per row chunk
      QG_TRY(qg_block_gram(ctx, A + a0, lda, ka, B + b0, ldb, kb, n, out, part, part_elems, real));
    } else if (ka <= 32 * QG_GRAM_LANE_COLS) {  // one column: wide partial sums, fixed-order reduction
      cudaStream_t s = ctx->stream;
      if (real)
        col_gram<true>(s, A, lda, a0, ka, B, ldb, b0);
      else
        col_gram<false>(s, A, lda, a0, ka, B, ldb, b0);
      k_gram_reduce_warp<<<(m + 7) / 8, 256, 0, s>>>(part, nblk, m, out);
      ctx->launches += 2;
    } else {
      dim3 g((m + 127) / 128, nchunk);
      k_gram_partial<<<g, 128, 0, ctx->stream>>>(A, lda, a0, ka, B, ldb, b0, kb, n, chunk, part);
      k_gram_reduce<<<(m + 127) / 128, 128, 0, ctx->stream>>>(part, nchunk, m, out);
      ctx->launches += 2;
    }
    if (host) {
      host->resize(m);
      QG_CUDA(ctx, cudaMemcpyAsync(host->data(), out, m * 16, cudaMemcpyDeviceToHost, ctx->stream));
      QG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return qg_check_launch(ctx, "gram");
  }
};

}  // namespace

// *real = none of the n values of v has an imaginary part
qg_status qg_all_real(qg_context ctx, const double2 *v, int64_t n, bool *real) {
  unsigned int *d_im = nullptr, h_im = 1;
  cudaStream_t s = ctx->stream;
  cudaError_t e = qg_malloc(ctx, &d_im, sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaMemsetAsync(d_im, 0, sizeof(unsigned int), s);
  if (e == cudaSuccess) {
    k_any_imag<<<(unsigned)std::min<int64_t>((n + 255) / 256, 4LL * ctx->num_sms), 256, 0, s>>>(v, n, d_im);
    ctx->launches++;
    e = cudaMemcpyAsync(&h_im, d_im, sizeof(unsigned int), cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  qg_free(d_im);
  if (e != cudaSuccess) return qg_cuda_fail(ctx, e, "qg_block_groundstate");
  *real = h_im == 0;
  return QG_OK;
}

// ------------------------------------------------------------------ one state: every step on the device

// A block of one vector has no block products, only passes over the Krylov vectors, so its
// steps are kept free of the host: the vectors are stored one after another (contiguous for the
// gathers of H*psi; one real number per entry for a real problem) and the projected matrix, the
// norms and the deflation flag stay in device memory until the restart.  Per step:
//   w = H v_j - b_j v_(j-1), with the partials of a_j = <v_j|H v_j>     (the Lanczos apply)
//   w -= a_j v_j;  c = V^H w                                            (k_one_project)
//   w -= V c;  b_(j+1) = |w|                                            (k_one_update)
//   v_(j+1) = w / b_(j+1)                                               (k_one_scale)
// The three-term part removes what is not small, so the one full projection after it leaves
// w orthogonal to eps, as the second of two full ones does, as long as it does not take more than
// it leaves (|c| <= |w|): V is read twice per step, not four times.  Where it does take more, w was
// rounding along the stored vectors (the space is invariant to rounding), what is left is not
// orthogonal to them, and each further such step would multiply the loss: the space ends there.
// The steps after it are zero, and the Ritz vector, normalised before its residual is taken, is formed of
// the vectors before it.  Bound by those two reads from L2 (FP64 above a few hundred thousand rows) and by the
// latency of four dependent kernels of 5 to 15 us, so each is launched while the one before it drains.
// Ground state of a 29,635-determinant impurity to a variance of 1e-12, 1305 steps in 9 restarts, with
// closure and spectrum: 58 ms (75 with plain launches and every projected matrix reduced in full);
// with block products of one column (complex storage, 16 bytes per entry strided by the Krylov
// dimension), host round trips and allocations in every step 578 ms.  Not faster: a block's warps sharing out the vectors of the update, over 32 or
// 64 rows (to a variance of 1e-10 43.2 to 53 ms, a row per thread 42.5 and 50.8), and letting the next
// kernel's blocks up before the last block of the one before has ended (52).

// scalars of the chain, in device memory
struct OneScal {
  double alpha;  // a_j of the current step
  double beta;   // |w| of the last update, and with it the b of the next apply
  double scale;  // 1 / beta, 0 for a vanished vector
  double norm2;  // the squared norm of the last update
  unsigned long long stray;  // bits of the largest part of the projected matrix beside its tridiagonal one
  int dead;      // first step whose next vector is lost (the space is invariant), else a large number
  unsigned int tickets[1 + ONE_SHARES];
};

#define ONE_ALPHA 1024  // up to so many partials of the apply every block sums for itself

// alpha = sum of the apply's partials (one block of 256, fixed order)
__device__ __forceinline__ double one_alpha(const double2 *__restrict__ part, int np) {
  __shared__ double sh[8];
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += 256) s += part[i].x;
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  s = sh[lane & 7];
  for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__global__ void __launch_bounds__(256) k_one_alpha(const double2 *__restrict__ part, int np, OneScal *sc) {
  const double s = one_alpha(part, np);
  if (threadIdx.x == 0) sc->alpha = s;
}

// wo = w - alpha v_j, then c_i = <v_i|wo> for i <= j and column j of the projected matrix
// (ct[i] = c_i + a_j [i == j] + b_j [i == j - 1]).  np: alpha from the apply's np partials here (a
// launch less; every block sums them alike), 0: from k_one_alpha
template <bool REAL>
__global__ void __launch_bounds__(256)
    k_one_project(const typename OneT<REAL>::T *V, int64_t n, int j, const typename OneT<REAL>::T *w,
                  typename OneT<REAL>::T *wo, typename OneT<REAL>::T *part, typename OneT<REAL>::T *c,
                  typename OneT<REAL>::T *ct, OneScal *sc, const double2 *dpart, int np) {
  typedef typename OneT<REAL>::T T;
  qg_chain_wait();
  const double alpha = np ? one_alpha(dpart, np) : sc->alpha, beta = sc->beta;
  const T *vj = V + (int64_t)j * n;
  one_multidot<T>(
      V, n, j + 1,
      [&](int64_t r) {
        const T v = one_axpy(w[r], alpha, vj[r]);
        if (blockIdx.y == 0) wo[r] = v;
        return v;
      },
      part, &sc->tickets[1],
      [&](int i, T t) {
        c[i] = t;
        ct[i] = one_plus_real(t, i == j ? alpha : i == j - 1 ? beta : 0.0);
        const double2 z = one_complex(t);
        const double m = i < j - 1 ? fmax(fabs(z.x), fabs(z.y)) : i == j - 1 ? fabs(z.y) : 0.0;
        if (m != 0.0) atomicMax(&sc->stray, (unsigned long long)__double_as_longlong(m));
      });
}

#define ONE_TINY 0x05d00000  // upper word of 2^-930: a squared norm below has lost digits

// w -= sum_i c_i v_i over i < k (out = w), and the squared norm of the result: the last block
// leaves beta = |w|, its reciprocal and, when the vector vanished or the projection took more than it
// left, zero for both and the step in `dead`.
template <bool REAL>
__global__ void __launch_bounds__(128)
    k_one_update(const typename OneT<REAL>::T *V, int64_t n, int k, const typename OneT<REAL>::T *c,
                 typename OneT<REAL>::T *w, double *part, int step, OneScal *sc) {
  typedef typename OneT<REAL>::T T;
  extern __shared__ __align__(16) char smem_raw[];
  T *cs = reinterpret_cast<T *>(smem_raw);
  __shared__ double sh[4];
  __shared__ int s_last;
  __shared__ int s_top[4];
  const int tid = threadIdx.x;
  qg_chain_wait();
  int top = 0;  // the largest upper word of c's parts
  for (int i = tid; i < k; i += 128) {
    const T ci = c[i];
    const double2 z = one_complex(ci);
    cs[i] = ci;
    top = max(top, max(__double2hiint(z.x) & 0x7fffffff, __double2hiint(z.y) & 0x7fffffff));
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if ((tid & 31) == 0) s_top[tid >> 5] = top;
  __syncthreads();
  double s = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * 128 + tid; r < n; r += (int64_t)gridDim.x * 128) {
    const T x = one_minus_sum(w[r], V, n, k, cs, r);
    if (k) w[r] = x;
    s += one_norm2(x);
  }
  const double t = one_total128(s, part, sh, &s_last, &sc->tickets[0]);
  if (s_last && tid == 0) {
    const double b = sqrt(t), inv = 1.0 / b;
    // |c|^2 <= t by the exponents (integers, beside the FP64 chain of the root), summed only where they do not
    // settle it: no part of c reaches 2^(et + 1), so the sum of the 2 k squares stays below 2^(2 et + 2 + bits)
    const int th = __double2hiint(t);
    bool lost = !(t > 0.0);
    if (k) {
      const int et = (max(max(s_top[0], s_top[1]), max(s_top[2], s_top[3])) >> 20) - 1023;
      lost = th < ONE_TINY || th >= 0x7ff00000;
      if (!lost && 2 * et + 2 + (32 - __clz(2 * k - 1)) > (th >> 20) - 1023) {
        double c2 = 0.0;
        for (int i = 0; i < k; i++) c2 += one_abs2(cs[i]);
        lost = !(c2 <= t);
      }
    }
    sc->norm2 = t;
    sc->beta = lost ? 0.0 : b;
    sc->scale = lost ? 0.0 : inv;
    if (lost && step < sc->dead) sc->dead = step;
  }
}

template <bool REAL>
__global__ void k_one_scale(int64_t n, const typename OneT<REAL>::T *w, const OneScal *sc, typename OneT<REAL>::T *v,
                            double *tsub) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  qg_chain_wait();
  if (r == 0 && tsub) *tsub = sc->beta;
  if (r < n) v[r] = one_scaled(w[r], sc->scale);
}

// d[i], e[i] = M[i][i], M[i][i + 1] of k_one_matrix, the real parts
template <bool REAL>
__global__ void k_one_tri(int k, int ldt, const typename OneT<REAL>::T *__restrict__ ct, const double *__restrict__ sub,
                          double *__restrict__ de) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  de[i] = one_complex(ct[(int64_t)i * ldt + i]).x;
  double a = i + 1 < k ? one_complex(ct[(int64_t)(i + 1) * ldt + i]).x : 0.0;
  const double b = i + 1 < k ? sub[i] : 0.0;
  de[k + i] = a == 0.0 ? b : b == 0.0 ? a : 0.5 * (a + b);
}

// M (k x k row-major): the Hermitian part of the projected matrix, column j of it in ct[j * ldt +
// 0..j], its subdiagonal in sub[j]; entries known on one side only come from that side
template <bool REAL>
__global__ void k_one_matrix(int k, int ldt, const typename OneT<REAL>::T *__restrict__ ct, const double *__restrict__ sub,
                             double2 *__restrict__ M) {
  typedef typename OneT<REAL>::T T;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= k * k) return;
  const int i = t / k, j = t % k, lo = i < j ? i : j, hi = i < j ? j : i;
  T a = ct[(int64_t)hi * ldt + lo];  // row lo, column hi
  if (lo == hi) {
    M[t] = make_double2(one_complex(a).x, 0.0);
    return;
  }
  if (hi == lo + 1) {
    const T b = one_plus_real(one_zero(T()), sub[lo]);
    a = one_is0(a) ? b : one_is0(b) ? a : one_scaled(one_sum(a, b), 0.5);
  }
  M[t] = one_complex(i < j ? a : one_conj(a));
}

// x = sum_i y_i v_i (y: the lowest eigenvector of the projected matrix, k entries)
template <bool REAL>
__global__ void __launch_bounds__(128)
    k_one_combine(const typename OneT<REAL>::T *__restrict__ V, int64_t n, int k, const double2 *__restrict__ y,
                  typename OneT<REAL>::T *__restrict__ x) {
  typedef typename OneT<REAL>::T T;
  extern __shared__ __align__(16) char smem_raw[];
  T *cs = reinterpret_cast<T *>(smem_raw);
  for (int i = threadIdx.x; i < k; i += 128) {
    T t;
    one_take(y[i], t);
    cs[i] = one_scaled(t, -1.0);
  }
  __syncthreads();
  const int64_t r = blockIdx.x * (int64_t)128 + threadIdx.x;
  if (r >= n) return;
  x[r] = one_minus_sum(one_zero(T()), V, n, k, cs, r);
}

#define ONE_STRAY 4.0  // measured 0.25 to 1.1 where the space has not run out (1,245 and 29,635
                       // determinants, 101 to 167 vectors)
#define ONE_MAX_K 2500  // the coefficients of a step fit one block's default shared memory

// One wanted state on a basis with connection lists: the restarts of qg_block_groundstate with
// the same Krylov dimensions, start and convergence test.  x_dev: start vector in, state out.
template <bool REAL>
static qg_status groundstate_one(qg_context ctx, qg_operator op, qg_basis b, double2 *x_dev, double *energy, double tol,
                                 int K, int max_restarts, int *applies, bool *converged) {
  typedef typename OneT<REAL>::T T;
  cudaStream_t s = ctx->stream;
  const int64_t n = b->n;
  const int Pa = qg_apply_grid(b);
  const unsigned gp = one_multidot_grid(ctx, n, 1).x;
  const unsigned gu = (unsigned)std::min<int64_t>((n + 127) / 128, 8LL * ctx->num_sms);
  const unsigned g1 = (unsigned)((n + 255) / 256), gc = (unsigned)((n + 127) / 128);
  T *V = nullptr, *w = nullptr, *wo = nullptr, *x = nullptr, *part = nullptr, *c = nullptr, *ct = nullptr;
  double *npart = nullptr, *sub = nullptr, *wd = nullptr, *zero = nullptr;
  double2 *dpart = nullptr, *Md = nullptr, *Y = nullptr;
  OneScal *sc = nullptr;
  cudaError_t e = qg_malloc(ctx, &V, (size_t)n * K * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &w, (size_t)n * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &wo, (size_t)n * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &x, (size_t)n * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &part, (size_t)gp * K * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &c, (size_t)K * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &ct, (size_t)K * K * sizeof(T));
  if (e == cudaSuccess) e = qg_malloc(ctx, &npart, (size_t)gu * sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &sub, (size_t)K * sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &wd, (size_t)K * sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &zero, sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &dpart, (size_t)Pa * 16);
  if (e == cudaSuccess) e = qg_malloc(ctx, &Md, (size_t)K * K * 16);
  if (e == cudaSuccess) e = qg_malloc(ctx, &Y, (size_t)K * 16);
  if (e == cudaSuccess) e = qg_malloc(ctx, &sc, sizeof(OneScal));
  if (e == cudaSuccess) e = cudaMemsetAsync(zero, 0, sizeof(double), s);
  qg_status st = QG_OK;
  if (e != cudaSuccess) {
    cudaGetLastError();
    ctx->last_error = "qg_block_groundstate: out of device memory";
    st = QG_ERR_OOM;
  }
  if (st == QG_OK) {
    k_one_in<REAL><<<g1, 256, 0, s>>>(n, x_dev, x);
    ctx->launches++;
  }
  if (st == QG_OK) st = qg_apply_prepare(ctx, op, b, K);
  // the lowest eigenpair of the projected matrix into wd, Y.  What the projections found beside the
  // tridiagonal part is rounding (about eps |H|) unless a vector all but vanished, and then the matrix is
  // reduced in full.  Within ONE_STRAY eps of the norm, the size of a reduction's own backward error, the
  // tridiagonal part is solved alone: 42.5 -> 35.5 ms for 29,635 determinants to a variance of 1e-10, as
  // the reduction is a chain of meetings of the grid, 5 us for each of up to 200 columns per restart.
  std::vector<double> de(2 * (size_t)K), tw(K), tz(K);
  std::vector<double2> ty(K);
  auto lowest = [&](int k, unsigned long long stray) -> qg_status {
    if (k > 1) {
      k_one_tri<REAL><<<(unsigned)((k + 127) / 128), 128, 0, s>>>(k, K, ct, sub, (double *)Md);
      ctx->launches++;
      cudaError_t ce = cudaMemcpyAsync(de.data(), Md, (size_t)2 * k * sizeof(double), cudaMemcpyDeviceToHost, s);
      if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
      if (ce != cudaSuccess) return qg_cuda_fail(ctx, ce, "qg_block_groundstate");
      double top = 0.0, off;
      for (int i = 0; i < 2 * k - 1; i++) top = std::max(top, fabs(de[i]));
      memcpy(&off, &stray, sizeof(off));
      if (off <= ONE_STRAY * 2.220446049250313e-16 * top) {  // false for NaN
        const qg_status ts = qg_tri_eigh(ctx, k, de.data(), de.data() + k, 1, tw.data(), tz.data());
        if (ts != QG_OK) return ts;
        for (int i = 0; i < k; i++) ty[i] = make_double2(tz[i], 0.0);
        ce = cudaMemcpyAsync(Y, ty.data(), (size_t)k * sizeof(double2), cudaMemcpyHostToDevice, s);
        if (ce == cudaSuccess) ce = cudaMemcpyAsync(wd, tw.data(), sizeof(double), cudaMemcpyHostToDevice, s);
        return ce == cudaSuccess ? QG_OK : qg_cuda_fail(ctx, ce, "qg_block_groundstate");
      }
    }
    k_one_matrix<REAL><<<(unsigned)((k * k + 255) / 256), 256, 0, s>>>(k, K, ct, sub, Md);
    ctx->launches++;
    return qg_eigh_device(ctx, k, Md, wd, Y, 1);
  };
  int Kcur = std::min(K, std::max(2, 101));
  OneScal h;
  for (int restart = 0; restart <= max_restarts && st == QG_OK && !*converged; restart++) {
    if (restart > 0) Kcur = std::min(K, Kcur + 11);
    OneScal init = {};
    init.dead = 1 << 30;
    e = cudaMemcpyAsync(sc, &init, sizeof(init), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) {
      st = qg_cuda_fail(ctx, e, "qg_block_groundstate");
      break;
    }
    // v_0 = x / |x|
    k_one_update<REAL><<<gu, 128, 0, s>>>(V, n, 0, c, x, npart, -1, sc);
    k_one_scale<REAL><<<g1, 256, 0, s>>>(n, x, sc, V, nullptr);
    ctx->launches += 2;
    ApplyFuse fz;
    fz.dot_part = dpart;
    fz.real_vector = REAL;
    for (int j = 0; j < Kcur && st == QG_OK; j++) {
      const T *vj = V + (size_t)j * n;
      fz.prev = (const double2 *)(j ? vj - n : vj);
      fz.beta = j ? &sc->beta : zero;
      st = qg_apply_strided(ctx, op, b, b, (const double *)vj, 1, (double *)w, 1, 1, &fz);
      (*applies)++;
      if (st != QG_OK) break;
      if (Pa > ONE_ALPHA) {
        k_one_alpha<<<1, 256, 0, s>>>(dpart, Pa, sc);
        ctx->launches++;
      }
      qg_chain_launch(ctx, k_one_project<REAL>, one_multidot_grid(ctx, n, j + 1), 256, one_multidot_smem<T>(j + 1), V, n,
                      j, w, wo, part, c, ct + (size_t)j * K, sc, dpart, Pa > ONE_ALPHA ? 0 : Pa);
      if (j + 1 < Kcur) {
        qg_chain_launch(ctx, k_one_update<REAL>, gu, 128, (size_t)(j + 1) * sizeof(T), V, n, j + 1, c, wo, npart, j, sc);
        qg_chain_launch(ctx, k_one_scale<REAL>, g1, 256, 0, n, wo, sc, V + (size_t)(j + 1) * n, sub + j);
      }
    }
    if (st == QG_OK) st = qg_check_launch(ctx, "qg_block_groundstate");
    if (st != QG_OK) break;
    e = cudaMemcpyAsync(&h, sc, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      st = qg_cuda_fail(ctx, e, "qg_block_groundstate");
      break;
    }
    const int k = std::min(Kcur, h.dead + 1);  // the vectors before the one that was lost
    if (k <= 0) {
      ctx->last_error = "qg_block_groundstate: start vectors are zero";
      st = QG_ERR_ARG;
      break;
    }
    if ((st = lowest(k, h.stray)) != QG_OK) break;
    k_one_combine<REAL><<<gc, 128, (size_t)k * sizeof(T), s>>>(V, n, k, Y, x);
    k_one_update<REAL><<<gu, 128, 0, s>>>(V, n, 0, c, x, npart, 1 << 30, sc);
    k_one_scale<REAL><<<g1, 256, 0, s>>>(n, x, sc, x, nullptr);
    ctx->launches += 3;
    // the variance |H x - theta x|^2, from the residual itself
    fz.prev = (const double2 *)x;
    fz.beta = wd;
    st = qg_apply_strided(ctx, op, b, b, (const double *)x, 1, (double *)w, 1, 1, &fz);
    (*applies)++;
    if (st != QG_OK) break;
    k_one_update<REAL><<<gu, 128, 0, s>>>(V, n, 0, c, w, npart, 1 << 30, sc);
    ctx->launches++;
    e = cudaMemcpyAsync(&h, sc, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(energy, wd, sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      st = qg_cuda_fail(ctx, e, "qg_block_groundstate");
      break;
    }
    *converged = h.norm2 < tol;
  }
  if (st == QG_OK) {
    k_one_out<REAL><<<g1, 256, 0, s>>>(n, x, x_dev);
    ctx->launches++;
    st = qg_check_launch(ctx, "qg_block_groundstate");
  }
  cudaStreamSynchronize(s);
  qg_free(V);
  qg_free(w);
  qg_free(wo);
  qg_free(x);
  qg_free(part);
  qg_free(c);
  qg_free(ct);
  qg_free(npart);
  qg_free(sub);
  qg_free(wd);
  qg_free(zero);
  qg_free(dpart);
  qg_free(Md);
  qg_free(Y);
  qg_free(sc);
  return st;
}

extern "C" qg_status qg_block_groundstate(qg_context ctx, qg_operator op, qg_basis b, int32_t nwant, double *x_dev,
                                          double *energies_host, double tol, int32_t max_krylov,
                                          int32_t max_restarts, int32_t *iterations) {
  if (!ctx || !op || !b || !x_dev || !energies_host || nwant <= 0 || op->nf != b->nf) return QG_ERR_ARG;
  int64_t n = b->n;
  if (n < nwant) {
    ctx->last_error = "qg_block_groundstate: basis smaller than the number of states";
    return QG_ERR_ARG;
  }
  int guard = nwant > 3 ? std::min(nwant / 2, 8) : 0;
  int p = (int)std::min<int64_t>(nwant + guard, n);
  int K = max_krylov > 0 ? max_krylov : 128;
  if (K < 2 * p) K = 2 * p;
  if (K > n) K = (int)n;
  K = (K / p) * p;
  if (K < p) K = p;
  cudaStream_t s = ctx->stream;
  if (p == 1 && K <= ONE_MAX_K && qg_apply_uses_lists(op, b)) {
    bool real = qg_operator_values_real(op), conv = false;
    int applies = 0;
    double energy = 0.0;
    if (real) QG_TRY(qg_all_real(ctx, (const double2 *)x_dev, n, &real));
    qg_status st = real ? groundstate_one<true>(ctx, op, b, (double2 *)x_dev, &energy, tol, K, max_restarts, &applies, &conv)
                        : groundstate_one<false>(ctx, op, b, (double2 *)x_dev, &energy, tol, K, max_restarts, &applies, &conv);
    energies_host[0] = energy;
    if (iterations) *iterations = applies;
    if (st == QG_OK) st = qg_check_device_error(ctx, "qg_block_groundstate");
    if (st == QG_OK && !conv) {
      ctx->last_error = "qg_block_groundstate: not converged within the restart limit";
      return QG_ERR_TIMEOUT;
    }
    return st;
  }
  double2 *V = nullptr, *W = nullptr, *Cd = nullptr, *X = nullptr, *Md = nullptr, *Sd = nullptr;
  double *wd = nullptr;
  size_t vb = (size_t)n * K * 16, wb = (size_t)n * p * 16;
  cudaError_t e = qg_malloc(ctx, &V, vb);
  if (e == cudaSuccess) e = qg_malloc(ctx, &W, wb);
  if (e == cudaSuccess) e = qg_malloc(ctx, &X, wb);
  if (e == cudaSuccess) e = qg_malloc(ctx, &Cd, (size_t)K * std::max(K, p) * 16);
  if (e == cudaSuccess) e = qg_malloc(ctx, &Md, (size_t)K * K * 16);
  if (e == cudaSuccess) e = qg_malloc(ctx, &wd, (size_t)K * sizeof(double));
  if (e == cudaSuccess) e = qg_malloc(ctx, &Sd, (size_t)p * p * 16);
  if (e != cudaSuccess) {
    qg_free(V);
    qg_free(W);
    qg_free(X);
    qg_free(Cd);
    qg_free(Md);
    qg_free(wd);
    qg_free(Sd);
    ctx->last_error = "qg_block_groundstate: out of device memory";
    return QG_ERR_OOM;
  }
  auto grid = [](int64_t t) { return (unsigned)((t + 255) / 256); };
  // the block: the caller's start vectors, then the guard vectors
  k_copy_cols<<<grid(n * nwant), 256, 0, s>>>((const double2 *)x_dev, nwant, 0, X, p, 0, nwant, n);
  ctx->launches++;
  if (p > nwant) {
    k_fill_cols<<<grid(n * (p - nwant)), 256, 0, s>>>(X, p, nwant, p - nwant, n, 0x5eedull,
                                                      qg_operator_values_real(op) ? 1 : 0);
    ctx->launches++;
  }
  Gram G;
  qg_status st = G.init(ctx, n, K * std::max(K, p), K);
  // a real operator with real start vectors keeps every vector, every projection and the Ritz
  // vectors real (the reference's real-vector solver): the block products then run in real
  // arithmetic, one FMA per term instead of four
  if (st == QG_OK && qg_operator_values_real(op)) st = qg_all_real(ctx, X, n * p, &G.real);
  std::vector<double> theta(p, 0.0);
  int it = 0;
  bool converged = false;
  std::vector<cd> c, T;
  // Krylov dimension per restart: starts at p + 100 and grows by p + 10 per restart up to K
  // (the reference's NKrylovStart / NKrylovStep schedule, Core/BlockLanczos.cpp:5130, :5311)
  int Kcur = std::min(K, std::max(2 * p, ((p + 100) / p) * p));
  for (int restart = 0; restart <= max_restarts && st == QG_OK && !converged; restart++) {
    if (restart > 0) Kcur = std::min(K, ((Kcur + p + 10) / p) * p);
    // V[:, 0:p] = X, orthonormalised (modified Gram-Schmidt, twice)
    k_copy_cols<<<grid(n * p), 256, 0, s>>>(X, p, 0, V, K, 0, p, n);
    ctx->launches++;
    int k = 0;  // orthonormal columns in V
    T.assign((size_t)K * K, cd(0, 0));
    // Loewdin orthonormalisation of the ka columns of A (ld lda): the eigenvectors U and values
    // s^2 of the Gram matrix A^H A; directions with s at most 1e-10 of the largest are dropped.
    // Sm (ka x kk row-major) makes Q = A Sm orthonormal and Rm (kk x ka) gives A = Q Rm on the
    // kept span; *cond gets the smallest kept s over the largest.  Returns kk.
    auto lowdin_pass = [&](const double2 *A, int lda, int ka, std::vector<cd> &Sm, std::vector<cd> &Rm,
                           double *cond) -> int {
      std::vector<cd> Gh;
      st = G.run(A, lda, 0, ka, A, lda, 0, ka, &Gh);
      if (st != QG_OK) return 0;
      for (int r = 0; r < ka; r++)
        for (int c = r; c < ka; c++) {
          const cd h = 0.5 * (Gh[(size_t)r * ka + c] + std::conj(Gh[(size_t)c * ka + r]));
          Gh[(size_t)r * ka + c] = h;
          Gh[(size_t)c * ka + r] = std::conj(h);
        }
      std::vector<double> w(ka);
      std::vector<cd> U((size_t)ka * ka);
      st = qg_eigh_host_io(ctx, ka, (const double *)Gh.data(), w.data(), (double *)U.data(), ka);
      if (st != QG_OK) return 0;
      const double smax = std::sqrt(std::max(w[ka - 1], 0.0));
      std::vector<int> keep;
      for (int q = ka - 1; q >= 0; q--)
        if (smax > 0.0 && std::sqrt(std::max(w[q], 0.0)) > 1e-10 * smax) keep.push_back(q);
      const int kk = (int)keep.size();
      *cond = kk ? std::sqrt(std::max(w[keep[kk - 1]], 0.0)) / smax : 0.0;
      Sm.assign((size_t)ka * std::max(kk, 1), cd(0, 0));
      Rm.assign((size_t)std::max(kk, 1) * ka, cd(0, 0));
      for (int c = 0; c < kk; c++) {
        const double sv = std::sqrt(w[keep[c]]);
        for (int r = 0; r < ka; r++) {
          const cd u = U[(size_t)r * ka + keep[c]];
          Sm[(size_t)r * kk + c] = u / sv;
          Rm[(size_t)c * ka + r] = sv * std::conj(u);
        }
      }
      return kk;
    };
    // orthonormalise V[:, c0:c0+cnt] with Loewdin inside the block, twice.  The block has already
    // been projected twice against V[:, 0:c0] as a whole, which stays enough unless the block
    // is nearly dependent: when the first pass's smallest kept s is below a tenth of the largest
    // (its 1/s scaling amplifies what the projections left), the result is projected against
    // V[:, 0:c0] once more before the second pass.  The result lands in V[:, c0:c0+kept].
    // coef (c0 + cnt rows x cnt) gets R with W_j = sum_i V_i R[i][j] over old and new columns.
    auto orth_block = [&](int c0, int cnt, std::vector<cd> *coef) -> int {
      std::vector<cd> S1, R1, S2, R2, Ch;
      double cond1 = 0.0, cond2 = 0.0;
      const int k1 = lowdin_pass(V + c0, K, cnt, S1, R1, &cond1);
      if (st != QG_OK || k1 == 0) return 0;
      cudaError_t ce = cudaMemcpyAsync(Sd, S1.data(), S1.size() * 16, cudaMemcpyHostToDevice, s);
      if (ce != cudaSuccess) {
        st = qg_cuda_fail(ctx, ce, "block orthonormalisation");
        return 0;
      }
      st = qg_block_update(ctx, V + c0, K, cnt, Sd, W, p, k1, n, 1.0, 0.0, G.real);  // Q1 = V_b S1
      if (st != QG_OK) return 0;
      if (c0 > 0 && cond1 < 0.1) {  // Q1 -= V_old (V_old^H Q1)
        st = G.run(V, K, 0, c0, W, p, 0, k1, &Ch);
        if (st == QG_OK) st = qg_block_update(ctx, V, K, c0, G.out, W, p, k1, n, -1.0, 1.0, G.real);
        if (st != QG_OK) return 0;
      }
      const int k2 = lowdin_pass(W, p, k1, S2, R2, &cond2);
      if (st != QG_OK || k2 == 0) return 0;
      ce = cudaMemcpyAsync(Sd, S2.data(), S2.size() * 16, cudaMemcpyHostToDevice, s);
      if (ce != cudaSuccess) {
        st = qg_cuda_fail(ctx, ce, "block orthonormalisation");
        return 0;
      }
      st = qg_block_update(ctx, W, p, k1, Sd, V + c0, K, k2, n, 1.0, 0.0, G.real);  // Q2 = Q1 S2
      if (st != QG_OK) return 0;
      if (coef) {
        for (int i = 0; i < k2; i++)  // new columns: R2 R1
          for (int j = 0; j < cnt; j++) {
            cd a(0, 0);
            for (int t = 0; t < k1; t++) a += R2[(size_t)i * k1 + t] * R1[(size_t)t * cnt + j];
            (*coef)[(size_t)(c0 + i) * cnt + j] = a;
          }
        for (int i = 0; i < c0 && !Ch.empty(); i++)  // old columns: C R1
          for (int j = 0; j < cnt; j++) {
            cd a(0, 0);
            for (int t = 0; t < k1; t++) a += Ch[(size_t)i * k1 + t] * R1[(size_t)t * cnt + j];
            (*coef)[(size_t)i * cnt + j] += a;
          }
      }
      return k2;
    };
    k = orth_block(0, p, nullptr);
    if (st != QG_OK) break;
    if (k == 0) {
      ctx->last_error = "qg_block_groundstate: start vectors are zero";
      st = QG_ERR_ARG;
      break;
    }
    int j0 = 0, bs = k;
    while (st == QG_OK) {
      // W = H V[:, j0:j0+bs]
      st = qg_apply_strided(ctx, op, b, b, (const double *)(V + j0), K, (double *)W, p, bs, nullptr);
      it++;
      if (st != QG_OK) break;
      // T[0:k, j0:j0+bs] = V^dag W (twice, the second pass corrects), W -= V C
      for (int pass = 0; pass < 2 && st == QG_OK; pass++) {
        st = G.run(V, K, 0, k, W, p, 0, bs, &c);
        if (st != QG_OK) break;
        for (int i = 0; i < k; i++)
          for (int j = 0; j < bs; j++) T[(size_t)i * K + j0 + j] += c[(size_t)i * bs + j];
        st = qg_block_update(ctx, V, K, k, G.out, W, p, bs, n, -1.0, 1.0, G.real);
      }
      if (st != QG_OK || k + bs > Kcur) break;
      // append W as new columns and orthonormalise them
      k_copy_cols<<<grid(n * bs), 256, 0, s>>>(W, p, 0, V, K, k, bs, n);
      ctx->launches++;
      std::vector<cd> R((size_t)(k + bs) * bs, cd(0, 0));
      int kept = orth_block(k, bs, &R);
      if (st != QG_OK) break;
      // H V_j has components R on the new columns (and small corrections on old ones)
      for (int i = 0; i < kept; i++)
        for (int j = 0; j < bs; j++) T[(size_t)(k + i) * K + j0 + j] += R[(size_t)(k + i) * bs + j];
      for (int i = 0; i < k; i++)
        for (int j = 0; j < bs; j++) T[(size_t)i * K + j0 + j] += R[(size_t)i * bs + j];
      if (kept == 0) break;  // the block Krylov space is invariant: the projection is exact
      j0 = k;
      k += kept;
      bs = kept;
      if (k + bs > Kcur) {
        // last block: its projections are needed for the Rayleigh quotient
        st = qg_apply_strided(ctx, op, b, b, (const double *)(V + j0), K, (double *)W, p, bs, nullptr);
        it++;
        if (st == QG_OK) st = G.run(V, K, 0, k, W, p, 0, bs, &c);
        if (st == QG_OK)
          for (int i = 0; i < k; i++)
            for (int j = 0; j < bs; j++) T[(size_t)i * K + j0 + j] = c[(size_t)i * bs + j];
        break;
      }
    }
    if (st != QG_OK) break;
    // projected matrix: Hermitian part of the k x k leading block
    std::vector<cd> M((size_t)k * k);
    for (int i = 0; i < k; i++)
      for (int j = 0; j < k; j++) {
        cd a = T[(size_t)i * K + j], bb = std::conj(T[(size_t)j * K + i]);
        // entries above the computed block columns are only known through symmetry
        M[(size_t)i * k + j] = (a == cd(0, 0)) ? bb : ((bb == cd(0, 0)) ? a : 0.5 * (a + bb));
      }
    // Ritz pairs on the device: the lowest p eigenvectors of M straight into Cd (k x p)
    const int nv = std::min(p, k);
    e = cudaMemcpyAsync(Md, M.data(), M.size() * 16, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && nv < p) e = cudaMemsetAsync(Cd, 0, (size_t)k * p * 16, s);
    if (e != cudaSuccess) {
      st = qg_cuda_fail(ctx, e, "projected matrix upload");
      break;
    }
    st = qg_eigh_device(ctx, k, Md, wd, Cd, nv);
    if (st != QG_OK) break;
    if (nv < p) {  // eigenvectors packed k x nv; spread them to k x p (the remaining columns stay zero)
      std::vector<cd> Yp((size_t)k * nv), Yw((size_t)k * p, cd(0, 0));
      e = cudaMemcpyAsync(Yp.data(), Cd, Yp.size() * 16, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      for (int i = 0; i < k && e == cudaSuccess; i++)
        for (int j = 0; j < nv; j++) Yw[(size_t)i * p + j] = Yp[(size_t)i * nv + j];
      if (e == cudaSuccess) e = cudaMemcpyAsync(Cd, Yw.data(), Yw.size() * 16, cudaMemcpyHostToDevice, s);
      if (e != cudaSuccess) {
        st = qg_cuda_fail(ctx, e, "ritz vectors");
        break;
      }
    }
    st = qg_block_update(ctx, V, K, k, Cd, X, p, p, n, 1.0, 0.0, G.real);
    if (st != QG_OK) break;
    std::vector<double> w(nv);
    e = cudaMemcpyAsync(w.data(), wd, (size_t)nv * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      st = qg_cuda_fail(ctx, e, "ritz values");
      break;
    }
    for (int j = 0; j < p; j++) theta[j] = j < nv ? w[j] : 0.0;
    // convergence: variance <(H - theta)^2> = |H x - theta x|^2 per vector, formed from the
    // residual itself (no cancellation between <H^2> and <H>^2)
    st = qg_apply_strided(ctx, op, b, b, (const double *)X, p, (double *)W, p, p, nullptr);
    it++;
    if (st != QG_OK) break;
    {
      std::vector<cd> th((size_t)p * p, cd(0, 0));
      for (int j = 0; j < p; j++) th[(size_t)j * p + j] = theta[j];
      e = cudaMemcpyAsync(Cd, th.data(), th.size() * 16, cudaMemcpyHostToDevice, s);
      if (e != cudaSuccess) {
        st = qg_cuda_fail(ctx, e, "residual");
        break;
      }
      st = qg_block_update(ctx, X, p, p, Cd, W, p, p, n, -1.0, 1.0, G.real);
      if (st != QG_OK) break;
    }
    std::vector<cd> hh;
    double worst = 0;
    for (int j = 0; j < nwant && st == QG_OK; j++) {
      st = G.run(W, p, j, 1, W, p, j, 1, &hh);
      if (st != QG_OK) break;
      worst = std::max(worst, std::fabs(hh[0].real()));
    }
    if (worst < tol) converged = true;
  }
  G.release();
  if (st == QG_OK) {
    k_copy_cols<<<grid(n * nwant), 256, 0, s>>>(X, p, 0, (double2 *)x_dev, nwant, 0, nwant, n);
    ctx->launches++;
  }
  cudaStreamSynchronize(s);
  qg_free(V);
  qg_free(W);
  qg_free(X);
  qg_free(Cd);
  qg_free(Md);
  qg_free(wd);
  qg_free(Sd);
  for (int j = 0; j < nwant; j++) energies_host[j] = theta[j];
  if (iterations) *iterations = it;
  if (st == QG_OK) st = qg_check_device_error(ctx, "qg_block_groundstate");
  if (st == QG_OK && !converged) {
    ctx->last_error = "qg_block_groundstate: not converged within the restart limit";
    return QG_ERR_TIMEOUT;
  }
  return st;
}
