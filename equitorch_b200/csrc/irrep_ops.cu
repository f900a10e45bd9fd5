// Streaming kernels for the per-irrep layers that follow a tensor product (gate, norms, RMS normalisation).
//
//   irrep_scale:  out[n, i, c] = x[n, i, c] * s(n, irrep(i), c)        s given per sample and channel (N, K, C),
//                                                                       shared (K, C) or per sample (N, K)
//   irrep_dot:    out[n, k, c] = sum_{i in irrep k} a[n, i, c] * b[n, i, c]
//
// Both are pure HBM streams over (N, D, C) features: one 128-bit load per operand and element group, the
// irrep of a component comes from a table in shared memory, no index loads from global memory.  The gate,
// the application of a normalisation and every gradient of these layers are instances of the two.
#include <algorithm>

#include "common.cuh"

namespace eqt {
namespace {

constexpr int MAX_COMPONENTS = 1024;   // irreps.dim handled by the shared-memory irrep table

template <typename T, int V> struct Vec;
template <> struct Vec<float, 4> { using type = float4; };
template <> struct Vec<double, 2> { using type = double2; };
template <> struct Vec<float, 1> { using type = float; };
template <> struct Vec<double, 1> { using type = double; };
template <> struct Vec<__nv_bfloat16, 8> { using type = uint4; };
template <> struct Vec<__nv_bfloat16, 1> { using type = __nv_bfloat16; };

// V storage elements of type T <-> V values of the arithmetic type (float for bfloat16 storage)
template <typename T, int V>
__device__ __forceinline__ void load(const T* p, typename Acc<T>::type (&v)[V]) {
  const typename Vec<T, V>::type t = __ldg(reinterpret_cast<const typename Vec<T, V>::type*>(p));
  const T* q = reinterpret_cast<const T*>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = static_cast<typename Acc<T>::type>(q[i]);
}
template <typename T, int V>
__device__ __forceinline__ void store(T* p, const typename Acc<T>::type (&v)[V]) {
  typename Vec<T, V>::type t;
  T* q = reinterpret_cast<T*>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) q[i] = static_cast<T>(v[i]);
  *reinterpret_cast<typename Vec<T, V>::type*>(p) = t;
}

// s_mode: 0 = s (N, K, C), 1 = s (K, C), 2 = s (N, K)
template <typename T, int V>
__global__ void __launch_bounds__(256) irrep_scale_kernel(const T* __restrict__ x, const T* __restrict__ s, T* __restrict__ out,
                                                          const int64_t* __restrict__ irrep_index, int64_t n, int d, int k,
                                                          int c, int s_mode) {
  __shared__ uint16_t kidx[MAX_COMPONENTS];
  for (int i = threadIdx.x; i < d; i += blockDim.x) kidx[i] = (uint16_t)__ldg(irrep_index + i);
  __syncthreads();
  const int cv = c / V;
  const int64_t per_sample = (int64_t)d * cv, total = n * per_sample;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = idx / per_sample;
    const int rem = (int)(idx - row * per_sample);
    const int i = rem / cv, c0 = (rem - i * cv) * V;
    const int kk = kidx[i];
    typename Acc<T>::type xv[V], sv[V], ov[V];
    load<T, V>(x + (row * d + i) * c + c0, xv);
    if (s_mode == 2) {
      const typename Acc<T>::type t = ld(s + row * k + kk);
#pragma unroll
      for (int q = 0; q < V; ++q) sv[q] = t;
    } else {
      load<T, V>(s + ((s_mode == 0 ? row * k : 0) + kk) * c + c0, sv);
    }
#pragma unroll
    for (int q = 0; q < V; ++q) ov[q] = xv[q] * sv[q];
    store<T, V>(out + (row * d + i) * c + c0, ov);
  }
}

template <typename T, int V>
__global__ void __launch_bounds__(256) irrep_dot_kernel(const T* a, const T* b, T* __restrict__ out,
                                                        const int64_t* __restrict__ irrep_seg, int64_t n, int d, int k, int c) {
  __shared__ int seg[MAX_COMPONENTS + 1];
  for (int i = threadIdx.x; i <= k; i += blockDim.x) seg[i] = (int)__ldg(irrep_seg + i);
  __syncthreads();
  const int cv = c / V;
  const int64_t per_sample = (int64_t)k * cv, total = n * per_sample;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = idx / per_sample;
    const int rem = (int)(idx - row * per_sample);
    const int kk = rem / cv, c0 = (rem - kk * cv) * V;
    using A = typename Acc<T>::type;
    A acc[V];
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = A(0);
    for (int i = seg[kk]; i < seg[kk + 1]; ++i) {
      A av[V], bv[V];
      load<T, V>(a + (row * d + i) * c + c0, av);
      if (a == b) {
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] = fma(av[q], av[q], acc[q]);
      } else {
        load<T, V>(b + (row * d + i) * c + c0, bv);
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] = fma(av[q], bv[q], acc[q]);
      }
    }
    store<T, V>(out + (row * k + kk) * c + c0, acc);
  }
}

// Both gradients of out = x * s with s per sample and channel, in one pass over the gradient of the output:
//   gx[n, i, c] = g[n, i, c] * s[n, irrep(i), c],   gs[n, k, c] = sum_{i in irrep k} g[n, i, c] * x[n, i, c]
// Bound by HBM: x, g, s read once, gx, gs written once.  As two kernels g was read twice (100k x 16 x 64 float32:
// 146 + 156 us, 221 us in one, 0.99 of the measured copy rate).  A thread owns (sample, irrep, channel group), as in irrep_dot_kernel.
template <typename T, int V>
__global__ void __launch_bounds__(256) irrep_scale_backward_kernel(const T* __restrict__ x, const T* __restrict__ s,
                                                                   const T* __restrict__ g, T* __restrict__ gx, T* __restrict__ gs,
                                                                   const int64_t* __restrict__ irrep_seg, int64_t n, int d, int k,
                                                                   int c) {
  __shared__ int seg[MAX_COMPONENTS + 1];
  for (int i = threadIdx.x; i <= k; i += blockDim.x) seg[i] = (int)__ldg(irrep_seg + i);
  __syncthreads();
  const int cv = c / V;
  const int64_t per_sample = (int64_t)k * cv, total = n * per_sample;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = idx / per_sample;
    const int rem = (int)(idx - row * per_sample);
    const int kk = rem / cv, c0 = (rem - kk * cv) * V;
    using A = typename Acc<T>::type;
    A acc[V], sv[V];
    load<T, V>(s + (row * k + kk) * c + c0, sv);
#pragma unroll
    for (int q = 0; q < V; ++q) acc[q] = A(0);
    const int64_t base = row * d * c + c0;
    const int last = seg[kk + 1];
    for (int i0 = seg[kk]; i0 < last; i0 += 4) {          // the loads of four components before the first is used
      A xv[4][V], gv[4][V];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < last) {
          load<T, V>(x + base + (int64_t)(i0 + u) * c, xv[u]);
          load<T, V>(g + base + (int64_t)(i0 + u) * c, gv[u]);
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < last) {
#pragma unroll
          for (int q = 0; q < V; ++q) {
            acc[q] = fma(gv[u][q], xv[u][q], acc[q]);
            gv[u][q] *= sv[q];
          }
          store<T, V>(gx + base + (int64_t)(i0 + u) * c, gv[u]);
        }
    }
    store<T, V>(gs + (row * k + kk) * c + c0, acc);
  }
}

template <typename T, int V>
int run_scale(const void* x, const void* s, void* out, const int64_t* index, int64_t n, int d, int k, int c, int mode,
              cudaStream_t st) {
  const int64_t work = n * d * (c / V);
  irrep_scale_kernel<T, V><<<flat_grid(work, 256, 16), 256, 0, st>>>(static_cast<const T*>(x), static_cast<const T*>(s),
                                                                            static_cast<T*>(out), index, n, d, k, c, mode);
  return check_launch("irrep_scale_kernel");
}
template <typename T, int V>
int run_dot(const void* a, const void* b, void* out, const int64_t* seg, int64_t n, int d, int k, int c, cudaStream_t st) {
  const int64_t work = n * k * (c / V);
  irrep_dot_kernel<T, V><<<flat_grid(work, 256, 16), 256, 0, st>>>(static_cast<const T*>(a), static_cast<const T*>(b),
                                                                          static_cast<T*>(out), seg, n, d, k, c);
  return check_launch("irrep_dot_kernel");
}

int check_sizes(int64_t n, int d, int k, int c, int dtype) {
  if (n < 0 || d <= 0 || k <= 0 || c <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (d > MAX_COMPONENTS || k > d) return fail(EQT_ERR_UNSUPPORTED, "at most %d components, num_irreps <= components", MAX_COMPONENTS);
  if (dtype != EQT_F32 && dtype != EQT_F64 && dtype != EQT_BF16) return fail(EQT_ERR_UNSUPPORTED, "float32, float64 or bfloat16 only");
  return EQT_OK;
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace eqt

extern "C" int eqt_irrep_scale(const void* x, const void* s, void* out, const int64_t* irrep_index, int64_t n, int32_t d,
                               int32_t k, int32_t c, int32_t s_mode, int32_t dtype, void* stream) {
  using namespace eqt;
  if (int rc = check_sizes(n, d, k, c, dtype)) return rc;
  if (s_mode < 0 || s_mode > 2) return fail(EQT_ERR_BAD_ARGUMENT, "s_mode must be 0, 1 or 2");
  if (n == 0) return EQT_OK;
  if (!x || !s || !out || !irrep_index) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec_ok = aligned16(x) && aligned16(out) && (s_mode == 2 || aligned16(s));
  if (dtype == EQT_F32) {
    if (c % 4 == 0 && vec_ok) return run_scale<float, 4>(x, s, out, irrep_index, n, d, k, c, s_mode, st);
    return run_scale<float, 1>(x, s, out, irrep_index, n, d, k, c, s_mode, st);
  }
  if (dtype == EQT_BF16) {   // bfloat16 storage, float32 arithmetic
    if (c % 8 == 0 && vec_ok) return run_scale<__nv_bfloat16, 8>(x, s, out, irrep_index, n, d, k, c, s_mode, st);
    return run_scale<__nv_bfloat16, 1>(x, s, out, irrep_index, n, d, k, c, s_mode, st);
  }
  if (c % 2 == 0 && vec_ok) return run_scale<double, 2>(x, s, out, irrep_index, n, d, k, c, s_mode, st);
  return run_scale<double, 1>(x, s, out, irrep_index, n, d, k, c, s_mode, st);
}

extern "C" int eqt_irrep_dot(const void* a, const void* b, void* out, const int64_t* irrep_seg, int64_t n, int32_t d,
                             int32_t k, int32_t c, int32_t dtype, void* stream) {
  using namespace eqt;
  if (int rc = check_sizes(n, d, k, c, dtype)) return rc;
  if (n == 0) return EQT_OK;
  if (!a || !b || !out || !irrep_seg) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec_ok = aligned16(a) && aligned16(b) && aligned16(out);
  if (dtype == EQT_F32) {
    if (c % 4 == 0 && vec_ok) return run_dot<float, 4>(a, b, out, irrep_seg, n, d, k, c, st);
    return run_dot<float, 1>(a, b, out, irrep_seg, n, d, k, c, st);
  }
  if (dtype == EQT_BF16) {
    if (c % 8 == 0 && vec_ok) return run_dot<__nv_bfloat16, 8>(a, b, out, irrep_seg, n, d, k, c, st);
    return run_dot<__nv_bfloat16, 1>(a, b, out, irrep_seg, n, d, k, c, st);
  }
  if (c % 2 == 0 && vec_ok) return run_dot<double, 2>(a, b, out, irrep_seg, n, d, k, c, st);
  return run_dot<double, 1>(a, b, out, irrep_seg, n, d, k, c, st);
}

namespace eqt {
namespace {
template <typename T, int V>
int run_scale_backward(const void* x, const void* s, const void* g, void* gx, void* gs, const int64_t* seg, int64_t n, int d, int k,
                       int c, cudaStream_t st) {
  irrep_scale_backward_kernel<T, V><<<flat_grid(n * k * (c / V), 256, 16), 256, 0, st>>>(
      static_cast<const T*>(x), static_cast<const T*>(s), static_cast<const T*>(g), static_cast<T*>(gx), static_cast<T*>(gs), seg, n,
      d, k, c);
  return check_launch("irrep_scale_backward_kernel");
}
}  // namespace
}  // namespace eqt

extern "C" int eqt_irrep_scale_backward(const void* x, const void* s, const void* g, void* gx, void* gs, const int64_t* irrep_seg,
                                        int64_t n, int32_t d, int32_t k, int32_t c, int32_t dtype, void* stream) {
  using namespace eqt;
  if (int rc = check_sizes(n, d, k, c, dtype)) return rc;
  if (n == 0) return EQT_OK;
  if (!x || !s || !g || !gx || !gs || !irrep_seg) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec_ok = aligned16(x) && aligned16(s) && aligned16(g) && aligned16(gx) && aligned16(gs);
  if (dtype == EQT_F32) {
    if (c % 4 == 0 && vec_ok) return run_scale_backward<float, 4>(x, s, g, gx, gs, irrep_seg, n, d, k, c, st);
    return run_scale_backward<float, 1>(x, s, g, gx, gs, irrep_seg, n, d, k, c, st);
  }
  if (dtype == EQT_BF16) {
    if (c % 8 == 0 && vec_ok) return run_scale_backward<__nv_bfloat16, 8>(x, s, g, gx, gs, irrep_seg, n, d, k, c, st);
    return run_scale_backward<__nv_bfloat16, 1>(x, s, g, gx, gs, irrep_seg, n, d, k, c, st);
  }
  if (c % 2 == 0 && vec_ok) return run_scale_backward<double, 2>(x, s, g, gx, gs, irrep_seg, n, d, k, c, st);
  return run_scale_backward<double, 1>(x, s, g, gx, gs, irrep_seg, n, d, k, c, st);
}

// ------------------------------------------------------------------------------------------------------
// Fused BatchRMSNorm in training mode (statistics of the batch), float32 / float64.
//   forward:  stat[k, c] = sum_{n, i in k} x^2 * factor_k,  factor_k = 1 / N (/ dim_k);   out = x * w / sqrt(stat + eps)
//   backward: q[k, c] = sum_{n, i in k} x g;   gw = q r;   gx = g w r - x (q w r^3 factor_k),   r = 1 / sqrt(stat + eps)
// Each direction is a column sum over the samples, a small fold and one streaming pass.  Bound by HBM: forward reads x
// twice and writes out, backward reads x and g twice and writes gx.  As a composition of per-irrep operators the
// statistics went through a (N, K, C) tensor and x received its gradient in two parts that were added afterwards
// (100k x 16 x 64 float32: 430 us forward, 1030 us backward; 215 and 315 us so).
// ------------------------------------------------------------------------------------------------------
namespace eqt {
namespace {

constexpr int COLUMN_THREADS = 512;   // a row of up to 512 vectors per block and pass, several rows where it is shorter
constexpr int COLUMN_UNROLL = 4;      // rows in flight per thread: 4 x 16 bytes per operand

// partial[block, i, c] = sum over the block's samples of a[n, i, c] * b[n, i, c]
template <typename T, int V>
__global__ void __launch_bounds__(COLUMN_THREADS) column_sum_kernel(const T* a, const T* b, T* __restrict__ partial, int64_t n,
                                                                    int cols) {
  __shared__ T fold[COLUMN_THREADS * V];
  const int first = blockIdx.y * COLUMN_THREADS, width = min(cols - first, COLUMN_THREADS), rows = COLUMN_THREADS / width;
  const int sub = threadIdx.x / width, col = first + threadIdx.x - sub * width;
  T acc[V];
#pragma unroll
  for (int q = 0; q < V; ++q) acc[q] = T(0);
  if (sub < rows) {
    const int64_t step = (int64_t)gridDim.x * rows;
    for (int64_t row = (int64_t)blockIdx.x * rows + sub; row < n; row += step * COLUMN_UNROLL) {
      T av[COLUMN_UNROLL][V], bv[COLUMN_UNROLL][V];
#pragma unroll
      for (int u = 0; u < COLUMN_UNROLL; ++u) {
        const int64_t r = row + u * step;
        if (r < n) {
          load<T, V>(a + (r * cols + col) * V, av[u]);
          if (a != b) load<T, V>(b + (r * cols + col) * V, bv[u]);
        } else {
#pragma unroll
          for (int q = 0; q < V; ++q) av[u][q] = bv[u][q] = T(0);
        }
      }
#pragma unroll
      for (int u = 0; u < COLUMN_UNROLL; ++u)
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] = fma(av[u][q], a != b ? bv[u][q] : av[u][q], acc[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < V; ++q) fold[threadIdx.x * V + q] = acc[q];
  __syncthreads();
  if (sub == 0) {
    for (int r = 1; r < rows; ++r)
#pragma unroll
      for (int q = 0; q < V; ++q) acc[q] += fold[(threadIdx.x + r * width) * V + q];
    store<T, V>(partial + ((int64_t)blockIdx.x * cols + col) * V, acc);
  }
}

template <typename T> struct BatchFold {
  const T* partial;      // (blocks, d, c)
  const T* weight;       // (k, c) or NULL
  T* stat;               // (k, c): written forward, read backward
  T* scale;              // (k, c): w r
  T* coef;               // (k, c): -q w r^3 factor (backward)
  T* grad_weight;        // (k, c) or NULL (backward)
  const int64_t* irrep_seg;
  int64_t n;
  int blocks, d, k, c, scaled;
  T eps;
};

// One block folds eight channels of one irrep: 128 threads deep over (partial block, component).  A few hundred values per
// result, so they are added and the factors formed in 64 bits and rounded once: with 32 bits the roundings of 1 / sqrt and of
// its product with the weight were in every value of the output (5,000 samples: 7.1e-8 of the norm, 3.5e-8 so).
template <typename T, bool BACKWARD>
__global__ void __launch_bounds__(1024) batch_fold_kernel(BatchFold<T> f) {
  __shared__ double part[32][8];
  const int lane8 = threadIdx.x & 7, deep = threadIdx.x >> 3, kk = blockIdx.y, cc = blockIdx.x * 8 + lane8;
  const int first = (int)__ldg(f.irrep_seg + kk), dim = (int)__ldg(f.irrep_seg + kk + 1) - first;
  double sum = 0.;
  if (cc < f.c) {
    double lanes[4] = {0., 0., 0., 0.};          // four chains: the loads of a step do not wait for its additions
    for (int b = deep; b < f.blocks; b += 128) {
      const T* p = f.partial + ((int64_t)b * f.d + first) * f.c + cc;
      int m = 0;
      for (; m + 4 <= dim; m += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) lanes[u] += __ldg(p + (int64_t)(m + u) * f.c);
      for (; m < dim; ++m) lanes[0] += __ldg(p + (int64_t)m * f.c);
    }
    sum = (lanes[0] + lanes[1]) + (lanes[2] + lanes[3]);
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 8);
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
  if ((threadIdx.x & 31) < 8) part[threadIdx.x >> 5][lane8] = sum;
  __syncthreads();
  if (threadIdx.x >= 8 || cc >= f.c) return;
  sum = 0.;
  for (int w = 0; w < 32; ++w) sum += part[w][lane8];
  const int at = kk * f.c + cc;
  const double factor = 1. / (double(f.n) * (f.scaled ? dim : 1));
  const double stat = BACKWARD ? double(f.stat[at]) : sum * factor;
  const double r = 1. / sqrt(stat + double(f.eps)), w = f.weight ? double(f.weight[at]) : 1.;
  f.scale[at] = T(w * r);
  if (BACKWARD) {
    f.coef[at] = T(-(sum * w) * (r * r * r) * factor);
    if (f.grad_weight) f.grad_weight[at] = T(sum * r);
  } else {
    f.stat[at] = T(stat);
  }
}

// out = a * scale (+ b * coef), scale and coef per (irrep, channel).  Walks the samples from the last to the first: the
// column sums before it read them from the first to the last, so their tail is still in L2.
template <typename T, int V, bool TWO>
__global__ void __launch_bounds__(256) batch_apply_kernel(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ scale,
                                                          const T* __restrict__ coef, T* __restrict__ out,
                                                          const int64_t* __restrict__ irrep_index, int64_t n, int d, int c) {
  __shared__ uint16_t kidx[MAX_COMPONENTS];
  for (int i = threadIdx.x; i < d; i += blockDim.x) kidx[i] = (uint16_t)__ldg(irrep_index + i);
  __syncthreads();
  const int cv = c / V;
  const int64_t per_sample = (int64_t)d * cv, total = n * per_sample;
  for (int64_t rev = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; rev < total; rev += (int64_t)gridDim.x * blockDim.x) {
    const int64_t idx = total - 1 - rev, row = idx / per_sample;
    const int rem = (int)(idx - row * per_sample), i = rem / cv, at = kidx[i] * c + (rem - i * cv) * V;
    T av[V], bv[V], sv[V], cvv[V];
    load<T, V>(a + idx * V, av);
    if (TWO) load<T, V>(b + idx * V, bv);
    load<T, V>(scale + at, sv);
    if (TWO) load<T, V>(coef + at, cvv);
#pragma unroll
    for (int q = 0; q < V; ++q) av[q] = TWO ? fma(av[q], sv[q], bv[q] * cvv[q]) : av[q] * sv[q];
    store<T, V>(out + idx * V, av);
  }
}

// Blocks over the samples: the two per SM that are resident at once (64 registers, 512 threads), fewer where that would leave a thread less than one unrolled pass.
int column_blocks(int64_t n, int cols) {
  const int tiles = (int)ceil_div(cols, COLUMN_THREADS), rows = cols < COLUMN_THREADS ? COLUMN_THREADS / cols : 1;
  const int64_t want = std::max<int64_t>(1, (int64_t)sm_count() * 2 / tiles), most = ceil_div(n, (int64_t)rows * COLUMN_UNROLL);
  return (int)std::max<int64_t>(1, std::min(want, most));
}

template <typename T, int V>
int run_batch(const T* x, const T* g, const T* w, T* stat, T* out, T* gw, T* scratch, const int64_t* seg, const int64_t* index,
              int64_t n, int d, int k, int c, int scaled, T eps, cudaStream_t st) {
  const int cols = d * (c / V), blocks = column_blocks(n, cols);
  T* partial = scratch + 2 * (int64_t)k * c;
  BatchFold<T> f{partial, w, stat, scratch, scratch + (int64_t)k * c, gw, seg, n, blocks, d, k, c, scaled, eps};
  const dim3 sum_grid(blocks, (unsigned)ceil_div(cols, COLUMN_THREADS)), fold_grid((unsigned)ceil_div(c, 8), k);
  column_sum_kernel<T, V><<<sum_grid, COLUMN_THREADS, 0, st>>>(x, g ? g : x, partial, n, cols);
  if (int rc = check_launch("column_sum_kernel")) return rc;
  if (g) batch_fold_kernel<T, true><<<fold_grid, 1024, 0, st>>>(f);
  else batch_fold_kernel<T, false><<<fold_grid, 1024, 0, st>>>(f);
  if (int rc = check_launch("batch_fold_kernel")) return rc;
  if (!out) return EQT_OK;
  const unsigned grid = flat_grid(n * cols, 256, 16);
  if (g) batch_apply_kernel<T, V, true><<<grid, 256, 0, st>>>(g, x, f.scale, f.coef, out, index, n, d, c);
  else batch_apply_kernel<T, V, false><<<grid, 256, 0, st>>>(x, nullptr, f.scale, nullptr, out, index, n, d, c);
  return check_launch("batch_apply_kernel");
}

int batch_rms(const void* x, const void* g, const void* w, void* stat, void* out, void* gw, void* scratch, int64_t scratch_size,
              const int64_t* seg, const int64_t* index, int64_t n, int d, int k, int c, int scaled, double eps, int dtype, void* stream) {
  if (int rc = check_sizes(n, d, k, c, dtype)) return rc;
  if (n == 0) return fail(EQT_ERR_BAD_ARGUMENT, "batch statistics need at least one sample");
  if (dtype == EQT_BF16 || (int64_t)d * c > INT32_MAX / 2 || k > 65535) return fail(EQT_ERR_UNSUPPORTED, "float32 or float64 only");
  if (scratch_size < eqt_batch_rms_scratch(n, d, k, c, dtype)) return fail(EQT_ERR_BAD_ARGUMENT, "scratch too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // every tensor of (k, c) or (.., d, c) shape is read in the same units; scratch holds three of them back to back
  const bool vec_ok = aligned16(x) && aligned16(g) && aligned16(out) && aligned16(scratch);
  if (dtype == EQT_F32) {
    using T = float;
    auto* run = c % 4 == 0 && vec_ok ? run_batch<T, 4> : run_batch<T, 1>;
    return run(static_cast<const T*>(x), static_cast<const T*>(g), static_cast<const T*>(w), static_cast<T*>(stat), static_cast<T*>(out),
               static_cast<T*>(gw), static_cast<T*>(scratch), seg, index, n, d, k, c, scaled, (T)eps, st);
  }
  using T = double;
  auto* run = c % 2 == 0 && vec_ok ? run_batch<T, 2> : run_batch<T, 1>;
  return run(static_cast<const T*>(x), static_cast<const T*>(g), static_cast<const T*>(w), static_cast<T*>(stat), static_cast<T*>(out),
             static_cast<T*>(gw), static_cast<T*>(scratch), seg, index, n, d, k, c, scaled, eps, st);
}

}  // namespace
}  // namespace eqt

extern "C" int64_t eqt_batch_rms_scratch(int64_t n, int32_t d, int32_t k, int32_t c, int32_t dtype) {
  using namespace eqt;
  if (n <= 0 || d <= 0 || k <= 0 || c <= 0) return 0;
  // enough for either unit: one element per column needs the larger number of tiles, a vector per column more blocks
  const int v = dtype == EQT_F32 ? 4 : 2;
  const int vec = c % v == 0 ? column_blocks(n, d * (c / v)) : 0;
  return 2 * (int64_t)k * c + std::max<int64_t>(column_blocks(n, d * c), vec) * d * c;
}

extern "C" int eqt_batch_rms_forward(const void* x, const void* weight, void* out, void* stat, void* scratch, int64_t scratch_size,
                                     const int64_t* irrep_seg, const int64_t* irrep_index, int64_t n, int32_t d, int32_t k, int32_t c,
                                     int32_t scaled, double eps, int32_t dtype, void* stream) {
  using namespace eqt;
  if (!x || !out || !stat || !scratch || !irrep_seg || !irrep_index) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  return batch_rms(x, nullptr, weight, stat, out, nullptr, scratch, scratch_size, irrep_seg, irrep_index, n, d, k, c, scaled, eps,
                   dtype, stream);
}

extern "C" int eqt_batch_rms_backward(const void* x, const void* grad_out, const void* weight, const void* stat, void* grad_x,
                                      void* grad_weight, void* scratch, int64_t scratch_size, const int64_t* irrep_seg,
                                      const int64_t* irrep_index, int64_t n, int32_t d, int32_t k, int32_t c, int32_t scaled,
                                      double eps, int32_t dtype, void* stream) {
  using namespace eqt;
  if (!x || !grad_out || !stat || !scratch || !irrep_seg || !irrep_index) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  return batch_rms(x, grad_out, weight, const_cast<void*>(stat), grad_x, grad_weight, scratch, scratch_size, irrep_seg, irrep_index, n,
                   d, k, c, scaled, eps, dtype, stream);
}

// ------------------------------------------------------------------------------------------------------
// Fused LayerRMSNorm: one warp per sample.  The components of an irrep are a contiguous run of dim_k * C
// floats, so the warp sums the squares of the run, turns the sum into 1/sigma and rescales the run (second
// read from L1): one HBM read and one write per element instead of four passes.  The backward pass is fused
// the same way; the gradient of the weight is accumulated per lane over the warp's samples (a lane always
// meets the same channels because C / V divides 32) and written as one partial per warp, summed by the caller
// in a fixed order.
// ------------------------------------------------------------------------------------------------------
namespace eqt {
namespace {

constexpr int LRN_MAX_IRREPS = 16;

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename T> __device__ __forceinline__ T rsqrt_t(T v);
template <> __device__ __forceinline__ float rsqrt_t<float>(float v) { return 1.0f / sqrtf(v); }
template <> __device__ __forceinline__ double rsqrt_t<double>(double v) { return 1.0 / sqrt(v); }

template <typename T, int V>
__global__ void __launch_bounds__(256) layer_rms_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w, T* __restrict__ out,
                                                            T* __restrict__ rsigma, const int64_t* __restrict__ irrep_seg,
                                                            int64_t n, int d, int k, int c, int scaled, T eps) {
  __shared__ int seg[LRN_MAX_IRREPS + 1];
  for (int i = threadIdx.x; i <= k; i += blockDim.x) seg[i] = (int)__ldg(irrep_seg + i);
  __syncthreads();
  const int lane = threadIdx.x & 31, cv = c / V;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = warp; row < n; row += warps) {
    for (int kk = 0; kk < k; ++kk) {
      const int dim = seg[kk + 1] - seg[kk], vecs = dim * cv;
      const T* xr = x + (row * d + seg[kk]) * c;
      T* orow = out + (row * d + seg[kk]) * c;
      T sum = T(0);
      for (int j = lane; j < vecs; j += 32) {
        T v[V];
        load<T, V>(xr + j * V, v);
#pragma unroll
        for (int q = 0; q < V; ++q) sum = fma(v[q], v[q], sum);
      }
      sum = warp_sum(sum);
      const T stat = sum / T(c) * (scaled ? T(1) / T(dim) : T(1));
      const T r = rsqrt_t<T>(stat + eps);
      if (lane == 0) rsigma[row * k + kk] = r;
      for (int j = lane; j < vecs; j += 32) {
        T v[V], wv[V];
        load<T, V>(xr + j * V, v);
        if (w) {
          load<T, V>(w + kk * c + (j % cv) * V, wv);
#pragma unroll
          for (int q = 0; q < V; ++q) v[q] = v[q] * r * wv[q];
        } else {
#pragma unroll
          for (int q = 0; q < V; ++q) v[q] = v[q] * r;
        }
        store<T, V>(orow + j * V, v);
      }
    }
  }
}

// gx = r w go - x r^3 t / (C [dim]),  t = sum over the irrep block of go w x;  gw partial per warp
template <typename T, int V>
__global__ void __launch_bounds__(256) layer_rms_bwd_kernel(const T* __restrict__ x, const T* __restrict__ go, const T* __restrict__ w,
                                                            const T* __restrict__ rsigma, T* __restrict__ gx, T* __restrict__ gw_partial,
                                                            const int64_t* __restrict__ irrep_seg, int64_t n, int d, int k, int c,
                                                            int scaled) {
  __shared__ T fold[LRN_MAX_IRREPS * 32 * V];
  __shared__ int seg[LRN_MAX_IRREPS + 1];
  for (int i = threadIdx.x; i <= k; i += blockDim.x) seg[i] = (int)__ldg(irrep_seg + i);
  __syncthreads();
  const int lane = threadIdx.x & 31, cv = c / V;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  T gwa[LRN_MAX_IRREPS][V];
#pragma unroll
  for (int kk = 0; kk < LRN_MAX_IRREPS; ++kk)
#pragma unroll
    for (int q = 0; q < V; ++q) gwa[kk][q] = T(0);
  const int cslot = lane % cv;   // the channel group this lane meets in every run (cv divides 32)
  for (int64_t row = warp; row < n; row += warps) {
#pragma unroll
    for (int kk = 0; kk < LRN_MAX_IRREPS; ++kk) {
      if (kk >= k) break;
      const int dim = seg[kk + 1] - seg[kk], vecs = dim * cv;
      const int64_t off = (row * d + seg[kk]) * c;
      const T r = __ldg(rsigma + row * k + kk);
      T wv[V];
      if (w) load<T, V>(w + kk * c + cslot * V, wv);
      else {
#pragma unroll
        for (int q = 0; q < V; ++q) wv[q] = T(1);
      }
      T t = T(0);
      for (int j = lane; j < vecs; j += 32) {
        T xv[V], gv[V];
        load<T, V>(x + off + j * V, xv);
        load<T, V>(go + off + j * V, gv);
#pragma unroll
        for (int q = 0; q < V; ++q) {
          const T gxv = gv[q] * xv[q];
          t = fma(gxv, wv[q], t);
          gwa[kk][q] = fma(gxv, r, gwa[kk][q]);
        }
      }
      t = warp_sum(t);
      const T coef = t * r * r * r / (T(c) * (scaled ? T(dim) : T(1)));
      for (int j = lane; j < vecs; j += 32) {
        T xv[V], gv[V];
        load<T, V>(x + off + j * V, xv);
        load<T, V>(go + off + j * V, gv);
#pragma unroll
        for (int q = 0; q < V; ++q) gv[q] = r * wv[q] * gv[q] - xv[q] * coef;
        store<T, V>(gx + off + j * V, gv);
      }
    }
  }
  if (gw_partial) {
    // lanes with the same channel group (lane, lane + cv, ...) hold partial sums of the same weights: fold them, then
    // the block's warps in order
    for (int i = threadIdx.x; i < k * c; i += blockDim.x) fold[i] = T(0);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < LRN_MAX_IRREPS; ++kk) {          // all warps at once: only the additions below take turns
      if (kk >= k) break;
#pragma unroll
      for (int q = 0; q < V; ++q)
        for (int o = 16; o >= cv; o >>= 1) gwa[kk][q] += __shfl_xor_sync(0xffffffffu, gwa[kk][q], o);
    }
    for (int turn = 0; turn < 8; ++turn) {
#pragma unroll
      for (int kk = 0; kk < LRN_MAX_IRREPS; ++kk) {
        if (kk >= k || (threadIdx.x >> 5) != turn || lane >= cv) break;
#pragma unroll
        for (int q = 0; q < V; ++q) fold[kk * c + lane * V + q] += gwa[kk][q];
      }
      __syncthreads();
    }
    for (int i = threadIdx.x; i < k * c; i += blockDim.x) gw_partial[(int64_t)blockIdx.x * k * c + i] = fold[i];
  }
}

// Float32 rows of at most 32 * NV vectors: the warp holds its sample in registers, so all of a sample's loads are in flight
// at once and nothing is read twice; an element's irrep and channels depend on its position alone and are found before
// the loop.  The kernels above walk the irreps one after the other (a load, a butterfly and a second read per irrep) and
// stay for longer rows, rows of fewer than four vectors and float64.  100k x 16 x 64: forward 222 -> 170 us, backward 380 + 58
// -> 235 + 4 us.  (16 vectors a lane leave one block of eight warps per SM: 50k x 9 x 128 forward 178 us, 96 us above; 500k rows
// of one vector 136 and 114 us.)
//
// sum[u] over the warp of the values that belong to irrep k0 + u: four butterflies side by side, so that their latencies
// overlap.
template <int NV>
__device__ __forceinline__ void irrep_sums(const float (&v)[NV], const int (&kj)[NV], int k0, float (&sum)[4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    sum[u] = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) sum[u] += kj[j] == k0 + u ? v[j] : 0.f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int u = 0; u < 4; ++u) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o);
}

template <int NV>
__global__ void __launch_bounds__(256, NV <= 5 ? 3 : 2) layer_rms_fwd_rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                 float* __restrict__ out, float* __restrict__ rsigma,
                                                                 const int64_t* __restrict__ irrep_seg, int64_t n, int d, int k, int c,
                                                                 int scaled, float eps) {
  __shared__ int seg[LRN_MAX_IRREPS + 1];
  for (int i = threadIdx.x; i <= k; i += blockDim.x) seg[i] = (int)__ldg(irrep_seg + i);
  __syncthreads();
  const int lane = threadIdx.x & 31, cv = c / 4, vecs = d * cv;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int kj[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int f = lane + 32 * j, comp = f / cv;
    kj[j] = -1;
    if (f < vecs)
      for (int kk = 0; kk < k; ++kk)
        if (comp >= seg[kk] && comp < seg[kk + 1]) kj[j] = kk;
  }
  for (int64_t row = warp; row < n; row += warps) {
    float v[NV][4], sq[NV], r[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      if (lane + 32 * j < vecs) load<float, 4>(x + row * vecs * 4 + (lane + 32 * j) * 4, v[j]);
      else v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      sq[j] = fmaf(v[j][0], v[j][0], fmaf(v[j][1], v[j][1], fmaf(v[j][2], v[j][2], v[j][3] * v[j][3])));
      r[j] = 0.f;
    }
    for (int k0 = 0; k0 < k; k0 += 4) {
      float sum[4];
      irrep_sums<NV>(sq, kj, k0, sum);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k0 + u >= k) break;
        const int dim = seg[k0 + u + 1] - seg[k0 + u];
        const float rs = rsqrt_t<float>(sum[u] / float(c) * (scaled ? 1.f / float(dim) : 1.f) + eps);
        if (lane == 0) rsigma[row * k + k0 + u] = rs;
#pragma unroll
        for (int j = 0; j < NV; ++j)
          if (kj[j] == k0 + u) r[j] = rs;
      }
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int f = lane + 32 * j;
      if (f >= vecs) continue;
      float wv[4] = {1.f, 1.f, 1.f, 1.f};
      if (w && kj[j] >= 0) load<float, 4>(w + kj[j] * c + (f % cv) * 4, wv);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[j][q] = v[j][q] * r[j] * wv[q];
      store<float, 4>(out + row * vecs * 4 + f * 4, v[j]);
    }
  }
}

constexpr int lrn_bwd_threads(int nv) { return nv <= 5 ? 256 : 128; }   // 160 registers at NV = 8: three blocks of four warps
template <int NV>
__global__ void __launch_bounds__(lrn_bwd_threads(NV), NV <= 3 || NV > 5 ? 3 : 2) layer_rms_bwd_rows_kernel(const float* __restrict__ x, const float* __restrict__ go,
                                                                 const float* __restrict__ w, const float* __restrict__ rsigma,
                                                                 float* __restrict__ gx, float* __restrict__ gw_partial,
                                                                 const int64_t* __restrict__ irrep_seg, int64_t n, int d, int k, int c,
                                                                 int scaled) {
  __shared__ int seg[LRN_MAX_IRREPS + 1];
  __shared__ float fold[NV * 128];
  for (int i = threadIdx.x; i <= k; i += blockDim.x) seg[i] = (int)__ldg(irrep_seg + i);
  for (int i = threadIdx.x; i < NV * 128; i += blockDim.x) fold[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, cv = c / 4, vecs = d * cv;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5, warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int kj[NV];
  float gwa[NV][4];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int f = lane + 32 * j, comp = f / cv;
    kj[j] = -1;
    if (f < vecs)
      for (int kk = 0; kk < k; ++kk)
        if (comp >= seg[kk] && comp < seg[kk + 1]) kj[j] = kk;
#pragma unroll
    for (int q = 0; q < 4; ++q) gwa[j][q] = 0.f;
  }
  for (int64_t row = warp; row < n; row += warps) {
    float xv[NV][4], gv[NV][4], t[NV], coef[NV], r[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int f = lane + 32 * j;
      if (f < vecs) {
        load<float, 4>(x + row * vecs * 4 + f * 4, xv[j]);
        load<float, 4>(go + row * vecs * 4 + f * 4, gv[j]);
        r[j] = kj[j] >= 0 ? __ldg(rsigma + row * k + kj[j]) : 0.f;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[j][q] = gv[j][q] = 0.f;
        r[j] = 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      float wv[4] = {1.f, 1.f, 1.f, 1.f};
      if (w && kj[j] >= 0) load<float, 4>(w + kj[j] * c + ((lane + 32 * j) % cv) * 4, wv);
      t[j] = coef[j] = 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        gwa[j][q] = fmaf(gv[j][q] * xv[j][q], r[j], gwa[j][q]);
        gv[j][q] *= wv[q];
        t[j] = fmaf(gv[j][q], xv[j][q], t[j]);
      }
    }
    for (int k0 = 0; k0 < k; k0 += 4) {
      float sum[4];
      irrep_sums<NV>(t, kj, k0, sum);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k0 + u >= k) break;
        sum[u] /= float(c) * (scaled ? float(seg[k0 + u + 1] - seg[k0 + u]) : 1.f);
#pragma unroll
        for (int j = 0; j < NV; ++j)
          if (kj[j] == k0 + u) coef[j] = sum[u] * r[j] * r[j] * r[j];
      }
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int f = lane + 32 * j;
      if (f >= vecs) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q) gv[j][q] = r[j] * gv[j][q] - xv[j][q] * coef[j];
      store<float, 4>(gx + row * vecs * 4 + f * 4, gv[j]);
    }
  }
  if (!gw_partial) return;
  // the block's warps in order, then the components of each irrep: the same sum on every run
  for (int t = 0; t < lrn_bwd_threads(NV) / 32; ++t) {
    if ((threadIdx.x >> 5) == t) {
#pragma unroll
      for (int j = 0; j < NV; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) fold[(lane + 32 * j) * 4 + q] += gwa[j][q];
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < k * c; i += blockDim.x) {
    const int kk = i / c, ch = i - kk * c;
    float sum = 0.f;
    for (int m = seg[kk]; m < seg[kk + 1]; ++m) sum += fold[m * c + ch];
    gw_partial[(int64_t)blockIdx.x * k * c + i] = sum;
  }
}

// The smallest instance that holds a row of `vecs` vectors, 0 where the kernels that walk the irreps are the better ones.
int layer_rms_row_vectors(int vecs, int fewest) {
  for (int nv : {2, 3, 5, 8})
    if (vecs >= fewest && vecs <= 32 * nv) return nv;
  return 0;
}

// out[j] = sum of the rows of in (rows, cols), in 64 bits: a block takes eight columns, 128 threads deep.
template <typename T>
__global__ void __launch_bounds__(1024) row_sum_kernel(const T* __restrict__ in, T* __restrict__ out, int rows, int cols) {
  __shared__ double part[32][8];
  const int lane8 = threadIdx.x & 7, col = blockIdx.x * 8 + lane8;
  double sum = 0.;
  if (col < cols)
    for (int r = threadIdx.x >> 3; r < rows; r += 128) sum += __ldg(in + (int64_t)r * cols + col);
  sum += __shfl_xor_sync(0xffffffffu, sum, 8);
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
  if ((threadIdx.x & 31) < 8) part[threadIdx.x >> 5][lane8] = sum;
  __syncthreads();
  if (threadIdx.x >= 8 || col >= cols) return;
  sum = 0.;
  for (int w = 0; w < 32; ++w) sum += part[w][lane8];
  out[col] = T(sum);
}

int layer_rms_grid(int64_t n) {
  // each warp walks samples with stride `warps`; six CTAs per SM are whole waves for one, two and three resident ones
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 7) / 8, (int64_t)sm_count() * 6));
}

bool layer_rms_ok(int d, int k, int c, int v) {
  return k <= LRN_MAX_IRREPS && d <= MAX_COMPONENTS && c % v == 0 && 32 % (c / v) == 0;
}

}  // namespace
}  // namespace eqt

extern "C" int eqt_row_sum(const void* in, void* out, int64_t rows, int64_t cols, int32_t dtype, void* stream) {
  using namespace eqt;
  if (rows < 0 || cols <= 0 || rows > INT32_MAX || cols > INT32_MAX) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (dtype != EQT_F32 && dtype != EQT_F64) return fail(EQT_ERR_UNSUPPORTED, "float32 or float64 only");
  if (!in || !out) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  const unsigned grid = (unsigned)ceil_div(cols, 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == EQT_F32) row_sum_kernel<float><<<grid, 1024, 0, st>>>(static_cast<const float*>(in), static_cast<float*>(out), (int)rows, (int)cols);
  else row_sum_kernel<double><<<grid, 1024, 0, st>>>(static_cast<const double*>(in), static_cast<double*>(out), (int)rows, (int)cols);
  return check_launch("row_sum_kernel");
}

extern "C" int eqt_layer_rms_num_partials(int64_t n) { return eqt::layer_rms_grid(n); }

extern "C" int eqt_layer_rms_forward(const void* x, const void* weight, void* out, void* rsigma, const int64_t* irrep_seg,
                                     int64_t n, int32_t d, int32_t k, int32_t c, int32_t scaled, double eps, int32_t dtype,
                                     void* stream) {
  using namespace eqt;
  if (int rc = check_sizes(n, d, k, c, dtype)) return rc;
  if (n == 0) return EQT_OK;
  if (!x || !out || !rsigma || !irrep_seg) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  const int v = dtype == EQT_F32 ? 4 : 2;
  if (!layer_rms_ok(d, k, c, v) || !aligned16(x) || !aligned16(out) || (weight && !aligned16(weight)))
    return fail(EQT_ERR_UNSUPPORTED, "fused LayerRMSNorm needs <= %d irreps, C / %d dividing 32 and 16-byte aligned tensors",
                LRN_MAX_IRREPS, v);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int nv = dtype == EQT_F32 ? layer_rms_row_vectors(d * (c / 4), 4) : 0;
  const int grid = nv ? layer_rms_grid(n) : (int)std::max<int64_t>(1, std::min<int64_t>((n + 7) / 8, (int64_t)sm_count() * 8));
  if (nv) {
    auto* kernel = nv == 2 ? layer_rms_fwd_rows_kernel<2> : nv == 3 ? layer_rms_fwd_rows_kernel<3> : nv == 5 ? layer_rms_fwd_rows_kernel<5>
                 : layer_rms_fwd_rows_kernel<8>;
    kernel<<<grid, 256, 0, st>>>(static_cast<const float*>(x), static_cast<const float*>(weight), static_cast<float*>(out),
                                 static_cast<float*>(rsigma), irrep_seg, n, d, k, c, scaled, (float)eps);
  } else if (dtype == EQT_F32)
    layer_rms_fwd_kernel<float, 4><<<grid, 256, 0, st>>>(static_cast<const float*>(x), static_cast<const float*>(weight),
                                                         static_cast<float*>(out), static_cast<float*>(rsigma), irrep_seg, n, d, k,
                                                         c, scaled, (float)eps);
  else
    layer_rms_fwd_kernel<double, 2><<<grid, 256, 0, st>>>(static_cast<const double*>(x), static_cast<const double*>(weight),
                                                          static_cast<double*>(out), static_cast<double*>(rsigma), irrep_seg, n, d,
                                                          k, c, scaled, eps);
  return check_launch("layer_rms_fwd_kernel");
}

extern "C" int eqt_layer_rms_backward(const void* x, const void* grad_out, const void* weight, const void* rsigma, void* grad_x,
                                      void* grad_weight_partial, const int64_t* irrep_seg, int64_t n, int32_t d, int32_t k,
                                      int32_t c, int32_t scaled, int32_t dtype, void* stream) {
  using namespace eqt;
  if (int rc = check_sizes(n, d, k, c, dtype)) return rc;
  if (n == 0) return EQT_OK;
  if (!x || !grad_out || !rsigma || !grad_x || !irrep_seg) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  const int v = dtype == EQT_F32 ? 4 : 2;
  if (!layer_rms_ok(d, k, c, v) || !aligned16(x) || !aligned16(grad_out) || !aligned16(grad_x) || (weight && !aligned16(weight)) ||
      (grad_weight_partial && !aligned16(grad_weight_partial)))
    return fail(EQT_ERR_UNSUPPORTED, "fused LayerRMSNorm needs <= %d irreps, C / %d dividing 32 and 16-byte aligned tensors",
                LRN_MAX_IRREPS, v);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = layer_rms_grid(n);
  const int nv = dtype == EQT_F32 ? layer_rms_row_vectors(d * (c / 4), 1) : 0;
  if (nv) {
    auto* kernel = nv == 2 ? layer_rms_bwd_rows_kernel<2> : nv == 3 ? layer_rms_bwd_rows_kernel<3> : nv == 5 ? layer_rms_bwd_rows_kernel<5>
                                                       : layer_rms_bwd_rows_kernel<8>;
    kernel<<<grid, lrn_bwd_threads(nv), 0, st>>>(static_cast<const float*>(x), static_cast<const float*>(grad_out), static_cast<const float*>(weight),
                                 static_cast<const float*>(rsigma), static_cast<float*>(grad_x),
                                 static_cast<float*>(grad_weight_partial), irrep_seg, n, d, k, c, scaled);
  } else if (dtype == EQT_F32)
    layer_rms_bwd_kernel<float, 4><<<grid, 256, 0, st>>>(static_cast<const float*>(x), static_cast<const float*>(grad_out),
                                                         static_cast<const float*>(weight), static_cast<const float*>(rsigma),
                                                         static_cast<float*>(grad_x), static_cast<float*>(grad_weight_partial),
                                                         irrep_seg, n, d, k, c, scaled);
  else
    layer_rms_bwd_kernel<double, 2><<<grid, 256, 0, st>>>(static_cast<const double*>(x), static_cast<const double*>(grad_out),
                                                          static_cast<const double*>(weight), static_cast<const double*>(rsigma),
                                                          static_cast<double*>(grad_x), static_cast<double*>(grad_weight_partial),
                                                          irrep_seg, n, d, k, c, scaled);
  return check_launch("layer_rms_bwd_kernel");
}
