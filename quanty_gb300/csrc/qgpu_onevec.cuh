// Passes of one vector over stored vectors (one after another, entry r of vector i at V[i * n + r]):
// the projections of the one-state eigensolver (qgpu_eigen.cu) and of the Krylov-basis Lanczos
// (qgpu_rixs.cu), for complex vectors and, where every entry is real, for one real number per
// entry (half the bytes and a quarter of the multiply-adds).
#pragma once
#include <algorithm>

#include "qgpu_internal.cuh"

template <bool REAL>
struct OneT;
template <>
struct OneT<true> {
  typedef double T;
};
template <>
struct OneT<false> {
  typedef double2 T;
};

__device__ __forceinline__ double one_zero(double) { return 0.0; }
__device__ __forceinline__ double2 one_zero(double2) { return make_double2(0.0, 0.0); }
// acc + conj(a) b
__device__ __forceinline__ double one_dot(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ double2 one_dot(double2 acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
  return acc;
}
// acc - a b
__device__ __forceinline__ double one_sub(double acc, double a, double b) { return fma(-a, b, acc); }
__device__ __forceinline__ double2 one_sub(double2 acc, double2 a, double2 b) {
  acc.x = fma(-a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(-a.x, b.y, fma(-a.y, b.x, acc.y));
  return acc;
}
__device__ __forceinline__ double one_axpy(double w, double a, double v) { return fma(-a, v, w); }
__device__ __forceinline__ double2 one_axpy(double2 w, double a, double2 v) { return qg_axpy2(w, a, v); }
__device__ __forceinline__ double one_scaled(double v, double s) { return v * s; }
__device__ __forceinline__ double2 one_scaled(double2 v, double s) { return make_double2(v.x * s, v.y * s); }
__device__ __forceinline__ double one_sum(double a, double b) { return a + b; }
__device__ __forceinline__ double2 one_sum(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double one_norm2(double v) { return v * v; }
__device__ __forceinline__ double one_norm2(double2 v) { return qg_norm2(v); }
__device__ __forceinline__ double one_plus_real(double a, double r) { return a + r; }
__device__ __forceinline__ double2 one_plus_real(double2 a, double r) { return make_double2(a.x + r, a.y); }
__device__ __forceinline__ double one_shfl(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double2 one_shfl(double2 v, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ double one_ldcg(const double *p) { return __ldcg(p); }
__device__ __forceinline__ double2 one_ldcg(const double2 *p) { return __ldcg(p); }
__device__ __forceinline__ double2 one_complex(double v) { return make_double2(v, 0.0); }
__device__ __forceinline__ double2 one_complex(double2 v) { return v; }
__device__ __forceinline__ double one_conj(double v) { return v; }
__device__ __forceinline__ double2 one_conj(double2 v) { return make_double2(v.x, -v.y); }
__device__ __forceinline__ bool one_is0(double v) { return v == 0.0; }
__device__ __forceinline__ bool one_is0(double2 v) { return v.x == 0.0 && v.y == 0.0; }
__device__ __forceinline__ void one_take(double2 v, double &o) { o = v.x; }
__device__ __forceinline__ void one_take(double2 v, double2 &o) { o = v; }

__device__ __forceinline__ double one_abs2(double v) { return v * v; }
__device__ __forceinline__ double one_abs2(double2 v) { return v.x * v.x + v.y * v.y; }

// complex entries in / out
template <bool REAL>
static __global__ void k_one_in(int64_t n, const double2 *__restrict__ x, typename OneT<REAL>::T *__restrict__ v) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r < n) one_take(x[r], v[r]);
}
template <bool REAL>
static __global__ void k_one_out(int64_t n, const typename OneT<REAL>::T *__restrict__ v, double2 *__restrict__ x) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r < n) x[r] = one_complex(v[r]);
}

#define ONE_SHARES 8  // at most so many blocks share out the vectors of one row chunk

// sink(i, <v_i|x>) for i < k with x_r = load(r), r < n (every r is loaded once per blockIdx.y).
// A block of 256 threads walks chunks of 256 rows, their x in shared memory; its warps take the
// vectors of the block's share (blockIdx.y) four at a time, so that the four lane sums fold into
// one another (6 additions instead of 20).  The last block of a share to arrive sums the
// blocks' partials in order, 32 sums at a time, and calls sink from one thread per sum; true on its
// threads (of each share's last block).  part: k * gridDim.x; ticket: one per share (ONE_SHARES).
template <typename T, typename Load, typename Sink>
__device__ __forceinline__ bool one_multidot(const T *__restrict__ V, int64_t n, int k, Load load, T *__restrict__ part,
                                             unsigned int *ticket, Sink sink) {
  extern __shared__ __align__(16) char one_smem[];
  T *acc = reinterpret_cast<T *>(one_smem);  // the block's share of k sums
  __shared__ T sw[256];
  __shared__ int s_last;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int share = ((k + (int)gridDim.y - 1) / (int)gridDim.y + 3) & ~3;
  const int b0 = min(k, (int)blockIdx.y * share), b1 = min(k, b0 + share);
  for (int i = tid; i < b1 - b0; i += 256) acc[i] = one_zero(T());
  for (int64_t r0 = (int64_t)blockIdx.x * 256; r0 < n; r0 += (int64_t)gridDim.x * 256) {
    const int64_t r = r0 + tid;
    __syncthreads();  // the previous chunk is done with sw
    sw[tid] = r < n ? load(r) : one_zero(T());
    __syncthreads();
    const int rows = (int)(n - r0 < 256 ? n - r0 : 256);
    for (int i0 = b0 + wid * 4; i0 < b1; i0 += 32) {
      T a[4];
#pragma unroll
      for (int q = 0; q < 4; q++) a[q] = one_zero(T());
#pragma unroll
      for (int t = 0; t < 8; t++) {
        const int rr = lane + 32 * t;
        if (rr < rows) {
          const T x = sw[rr];
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (i0 + q < b1) a[q] = one_dot(a[q], V[(int64_t)(i0 + q) * n + r0 + rr], x);
        }
      }
      // fold: lanes of bit 4 keep sums 2, 3, the others 0, 1; then bit 3 the odd one
      const bool h1 = lane & 16, h2 = lane & 8;
      T k0 = h1 ? a[2] : a[0], k1 = h1 ? a[3] : a[1], g0 = h1 ? a[0] : a[2], g1 = h1 ? a[1] : a[3];
      k0 = one_sum(k0, one_shfl(g0, 16));
      k1 = one_sum(k1, one_shfl(g1, 16));
      T f = h2 ? k1 : k0, g = h2 ? k0 : k1;
      f = one_sum(f, one_shfl(g, 8));
      for (int o = 4; o; o >>= 1) f = one_sum(f, one_shfl(f, o));
      const int q = (h1 ? 2 : 0) + (h2 ? 1 : 0);
      if ((lane & 7) == 0 && i0 + q < b1) acc[i0 - b0 + q] = one_sum(acc[i0 - b0 + q], f);
    }
  }
  __syncthreads();
  for (int i = tid; i < b1 - b0; i += 256) part[(int64_t)blockIdx.x * k + b0 + i] = acc[i];
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(ticket + blockIdx.y, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  for (int i0 = b0; i0 < b1; i0 += 32) {  // a lane per sum, the warps sharing the blocks (sw: their eight parts)
    T s = one_zero(T());
    if (i0 + lane < b1) {
#pragma unroll 8
      for (int b = wid; b < (int)gridDim.x; b += 8) s = one_sum(s, one_ldcg(part + (int64_t)b * k + i0 + lane));
    }
    sw[tid] = s;
    __syncthreads();
    if (wid == 0 && i0 + lane < b1) {
      for (int g = 1; g < 8; g++) s = one_sum(s, sw[32 * g + lane]);
      sink(i0 + lane, s);
    }
    __syncthreads();
  }
  if (tid == 0) ticket[blockIdx.y] = 0u;
  return true;
}

// w - sum_i c_i v_i at row r over i < k (c in shared memory), eight loads in flight
template <typename T>
__device__ __forceinline__ T one_minus_sum(T x, const T *__restrict__ V, int64_t n, int k, const T *c, int64_t r) {
  T y = one_zero(T());
  int i = 0;
  for (; i + 8 <= k; i += 8) {
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = V[(int64_t)(i + q) * n + r];
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
      x = one_sub(x, v[q], c[i + q]);
      y = one_sub(y, v[q + 1], c[i + q + 1]);
    }
  }
  for (; i < k; i++) x = one_sub(x, V[(int64_t)i * n + r], c[i]);
  return one_sum(x, y);
}

// the grid's sum of s over blocks of 128 threads, in thread 0 of the last block (*last set there);
// sh: 4 doubles, part: gridDim.x
__device__ __forceinline__ double one_total128(double s, double *__restrict__ part, double *sh, int *last,
                                               unsigned int *ticket) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sh[wid] = s;
  __syncthreads();
  if (tid == 0) {
    part[blockIdx.x] = (sh[0] + sh[1]) + (sh[2] + sh[3]);
    __threadfence();
    *last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!*last) return 0.0;
  __threadfence();
  s = 0.0;
#pragma unroll 8
  for (int b = tid; b < (int)gridDim.x; b += 128) s += __ldcg(part + b);
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sh[wid] = s;
  __syncthreads();
  if (tid == 0) *ticket = 0u;
  return (sh[0] + sh[1]) + (sh[2] + sh[3]);
}

// the launch of one_multidot: where the rows are few the vectors are shared out over enough blocks for four on
// every SM (a basis of 29,635 rows, 1305 steps over 75 vectors on average: 38.9 -> 27.6 ms)
static inline dim3 one_multidot_grid(qg_context ctx, int64_t n, int k) {
  const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4LL * ctx->num_sms));
  const int gy = std::max(1, std::min(std::min((k + 31) / 32, ONE_SHARES), (4 * ctx->num_sms + gx - 1) / gx));
  return dim3((unsigned)gx, (unsigned)gy);
}
template <typename T>
static inline size_t one_multidot_smem(int k) {
  return (size_t)(k + 3) * sizeof(T);
}
