// Spherical harmonics (table-driven degree recurrence, forward and reverse mode) and the
// row gather / CSR segment-sum that surround a tensor-product layer in a graph network.
#include <algorithm>

#include "common.cuh"

namespace eqt {
namespace {

#include "generated/sh_specs.inc"

struct ShTab {
  const int32_t* ptr;
  const int32_t* m_out;
  const int32_t* m_in;
  const int32_t* axis;
  const double* coef;
  int l_max;
};

// One thread per point.  All (l_max+1)^2 values of a point live in one shared-memory column
// (component-major, thread-minor => conflict free); the block then writes its contiguous
// slab of the output with coalesced stores.
template <typename T>
__global__ void sh_forward_kernel(const T* __restrict__ xyz, T* __restrict__ out, int64_t n, ShTab tab,
                                  int normalize, typename Acc<T>::type out_scale) {
  using A = typename Acc<T>::type;
  extern __shared__ unsigned char smem_raw[];
  A* col = reinterpret_cast<A*>(smem_raw);
  const int K = (tab.l_max + 1) * (tab.l_max + 1);
  const int B = blockDim.x, tid = threadIdx.x;
  for (int64_t base = (int64_t)blockIdx.x * B; base < n; base += (int64_t)gridDim.x * B) {
    const int64_t pt = base + tid;
    if (pt < n) {
      A r[3] = {ld(xyz + pt * 3), ld(xyz + pt * 3 + 1), ld(xyz + pt * 3 + 2)};
      if (normalize) {
        const A inv = A(1) / max(sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), A(1e-12));
        r[0] *= inv; r[1] *= inv; r[2] *= inv;
      }
      col[tid] = A(1);
      for (int l = 1; l <= tab.l_max; ++l) {
        A* cur = col + (l * l) * B + tid;
        const A* prev = col + ((l - 1) * (l - 1)) * B + tid;
        for (int m = 0; m < 2 * l + 1; ++m) cur[m * B] = A(0);
        for (int e = tab.ptr[l]; e < tab.ptr[l + 1]; ++e)
          cur[tab.m_out[e] * B] += static_cast<A>(tab.coef[e]) * r[tab.axis[e]] * prev[tab.m_in[e] * B];
      }
    }
    __syncthreads();
    const int64_t rows = min((int64_t)B, n - base);
    for (int64_t q = tid; q < rows * K; q += B) {
      const int th = q / K, comp = q % K;
      st(out + base * K + q, col[comp * B + th] * out_scale);
    }
    __syncthreads();
  }
}

// Reverse mode through forward-mode columns: alongside Y the three partial derivatives
// dY/dx, dY/dy, dY/dz of the previous and the current degree are kept in shared memory
// (8 columns of 2 l_max + 1 entries per thread), and the cotangent is contracted degree by
// degree, so nothing of size (l_max+1)^2 is stored.
template <typename T>
__global__ void sh_backward_kernel(const T* __restrict__ xyz, const T* __restrict__ gout, T* __restrict__ gxyz,
                                   int64_t n, ShTab tab, int normalize, typename Acc<T>::type out_scale) {
  using A = typename Acc<T>::type;
  extern __shared__ unsigned char smem_raw[];
  A* sm = reinterpret_cast<A*>(smem_raw);
  const int W = 2 * tab.l_max + 1, K = (tab.l_max + 1) * (tab.l_max + 1);
  const int B = blockDim.x, tid = threadIdx.x;
  // layout: [buffer 0/1][quantity 0..3 = Y, dx, dy, dz][component][thread]
  auto at = [&](int buf, int q, int m) -> A& { return sm[((buf * 4 + q) * W + m) * B + tid]; };
  for (int64_t pt = (int64_t)blockIdx.x * B + tid; pt < n; pt += (int64_t)gridDim.x * B) {
    A u[3] = {ld(xyz + pt * 3), ld(xyz + pt * 3 + 1), ld(xyz + pt * 3 + 2)};
    A r[3] = {u[0], u[1], u[2]};
    A norm = A(1);
    if (normalize) {
      norm = max(sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]), A(1e-12));
      r[0] /= norm; r[1] /= norm; r[2] /= norm;
    }
    A g[3] = {0, 0, 0};
    at(0, 0, 0) = A(1);
    at(0, 1, 0) = at(0, 2, 0) = at(0, 3, 0) = A(0);
    const T* go = gout + pt * K;
    for (int l = 1; l <= tab.l_max; ++l) {
      const int cb = l & 1, pb = cb ^ 1;
      for (int m = 0; m < 2 * l + 1; ++m)
        for (int q = 0; q < 4; ++q) at(cb, q, m) = A(0);
      for (int e = tab.ptr[l]; e < tab.ptr[l + 1]; ++e) {
        const int mo = tab.m_out[e], mi = tab.m_in[e], ax = tab.axis[e];
        const A c = static_cast<A>(tab.coef[e]);
        const A yp = at(pb, 0, mi);
        at(cb, 0, mo) += c * r[ax] * yp;
        at(cb, 1, mo) += c * (r[ax] * at(pb, 1, mi) + (ax == 0 ? yp : A(0)));
        at(cb, 2, mo) += c * (r[ax] * at(pb, 2, mi) + (ax == 1 ? yp : A(0)));
        at(cb, 3, mo) += c * (r[ax] * at(pb, 3, mi) + (ax == 2 ? yp : A(0)));
      }
      for (int m = 0; m < 2 * l + 1; ++m) {
        const A w = ld(go + l * l + m);
        g[0] += w * at(cb, 1, m);
        g[1] += w * at(cb, 2, m);
        g[2] += w * at(cb, 3, m);
      }
    }
    g[0] *= out_scale; g[1] *= out_scale; g[2] *= out_scale;
    if (normalize) {
      // v = u / max(|u|, eps):  dv = (I - v v^T) / |u| above eps, I / eps below
      const A un = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
      if (un > A(1e-12)) {
        const A dot = g[0] * r[0] + g[1] * r[1] + g[2] * r[2];
        g[0] = (g[0] - r[0] * dot) / norm; g[1] = (g[1] - r[1] * dot) / norm; g[2] = (g[2] - r[2] * dot) / norm;
      } else {
        g[0] /= norm; g[1] /= norm; g[2] /= norm;
      }
    }
    st(gxyz + pt * 3, g[0]); st(gxyz + pt * 3 + 1, g[1]); st(gxyz + pt * 3 + 2, g[2]);
  }
}

template <typename Kern>
int configure_smem(Kern kern, size_t bytes) {
  if (bytes > 48 * 1024) {
    if (bytes > 227 * 1024) return fail(EQT_ERR_UNSUPPORTED, "l_max needs %zu bytes of shared memory", bytes);
    return allow_shared(kern, 227 * 1024);
  }
  return EQT_OK;
}

// Small l_max: the recurrence as straight-line code on registers (generated/sh_specs.inc).  The forward kernel
// still goes through a shared-memory transpose so that a block writes its slab of the output contiguously.
template <typename T, int LMAX>
__global__ void __launch_bounds__(256) sh_forward_unrolled_kernel(const T* __restrict__ xyz, T* __restrict__ out, int64_t n,
                                                                  int normalize, typename Acc<T>::type out_scale) {
  using A = typename Acc<T>::type;
  using U = ShUnrolled<A, LMAX>;
  constexpr int K = U::K;
  extern __shared__ unsigned char smem_raw[];
  A* col = reinterpret_cast<A*>(smem_raw);
  const int B = blockDim.x, tid = threadIdx.x;
  for (int64_t base = (int64_t)blockIdx.x * B; base < n; base += (int64_t)gridDim.x * B) {
    const int64_t pt = base + tid;
    if (pt < n) {
      A r[3] = {ld(xyz + pt * 3), ld(xyz + pt * 3 + 1), ld(xyz + pt * 3 + 2)};
      if (normalize) {
        const A inv = A(1) / max(sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), A(1e-12));
        r[0] *= inv; r[1] *= inv; r[2] *= inv;
      }
      A y[K];
      U::forward(r, y);
#pragma unroll
      for (int k = 0; k < K; ++k) col[k * B + tid] = y[k] * out_scale;
    }
    __syncthreads();
    const int64_t rows = min((int64_t)B, n - base);
    for (int64_t q = tid; q < rows * K; q += B) {
      const int th = q / K, comp = q % K;
      st(out + base * K + q, col[comp * B + th]);
    }
    __syncthreads();
  }
}

template <typename T, int LMAX>
__global__ void __launch_bounds__(256) sh_backward_unrolled_kernel(const T* __restrict__ xyz, const T* __restrict__ gout,
                                                                   T* __restrict__ gxyz, int64_t n, int normalize,
                                                                   typename Acc<T>::type out_scale) {
  using A = typename Acc<T>::type;
  using U = ShUnrolled<A, LMAX>;
  constexpr int K = U::K;
  for (int64_t pt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; pt < n; pt += (int64_t)gridDim.x * blockDim.x) {
    A u[3] = {ld(xyz + pt * 3), ld(xyz + pt * 3 + 1), ld(xyz + pt * 3 + 2)};
    A r[3] = {u[0], u[1], u[2]};
    A norm = A(1);
    if (normalize) {
      norm = max(sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]), A(1e-12));
      r[0] /= norm; r[1] /= norm; r[2] /= norm;
    }
    A go[K], g[3];
#pragma unroll
    for (int k = 0; k < K; ++k) go[k] = ld(gout + pt * K + k);
    U::backward(r, go, g);
    g[0] *= out_scale; g[1] *= out_scale; g[2] *= out_scale;
    if (normalize) {
      // v = u / max(|u|, eps):  dv = (I - v v^T) / |u| above eps, I / eps below
      const A un = sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
      if (un > A(1e-12)) {
        const A dot = g[0] * r[0] + g[1] * r[1] + g[2] * r[2];
        g[0] = (g[0] - r[0] * dot) / norm; g[1] = (g[1] - r[1] * dot) / norm; g[2] = (g[2] - r[2] * dot) / norm;
      } else {
        g[0] /= norm; g[1] /= norm; g[2] /= norm;
      }
    }
    st(gxyz + pt * 3, g[0]); st(gxyz + pt * 3 + 1, g[1]); st(gxyz + pt * 3 + 2, g[2]);
  }
}

template <typename T, int LMAX>
int sh_launch_unrolled(bool backward, const void* xyz, const void* gout, void* out, int64_t n, int normalize, double out_scale,
                       cudaStream_t s) {
  using A = typename Acc<T>::type;
  constexpr int K = (LMAX + 1) * (LMAX + 1);
  const unsigned grid = flat_grid(n, 256, 8);
  if (backward) {
    sh_backward_unrolled_kernel<T, LMAX><<<grid, 256, 0, s>>>(static_cast<const T*>(xyz), static_cast<const T*>(gout),
                                                              static_cast<T*>(out), n, normalize, (A)out_scale);
    return check_launch("sh_backward_unrolled_kernel");
  }
  if (int rc = configure_smem(sh_forward_unrolled_kernel<T, LMAX>, sizeof(A) * K * 256)) return rc;
  sh_forward_unrolled_kernel<T, LMAX><<<grid, 256, sizeof(A) * K * 256, s>>>(static_cast<const T*>(xyz), static_cast<T*>(out), n,
                                                                             normalize, (A)out_scale);
  return check_launch("sh_forward_unrolled_kernel");
}

// ---- rows of nodes and edges ----------------------------------------------------------------------------------------
// All of these move whole rows, so they work on 16-byte units where rows and pointers allow it (U = units' element
// count) and on elements otherwise, with a 32-bit flat index (the launchers check that it fits).  Bound: HBM / L2.
// 20,480 rows of 480: gather of bfloat16 24 -> 6 us, sum of float32 into 960 segments 18 -> 8.5 us.
template <typename T, int U> struct alignas(sizeof(T) * U) Unit { T v[U]; };

template <typename T, int U>
__global__ void __launch_bounds__(256) segment_sum_kernel(const T* __restrict__ in, const int64_t* __restrict__ ptr,
                                                          const int64_t* __restrict__ perm, T* __restrict__ out,
                                                          uint32_t segments, uint32_t units) {
  using A = typename Acc<T>::type;
  using Q = Unit<T, U>;
  const Q* src = reinterpret_cast<const Q*>(in);
  Q* dst = reinterpret_cast<Q*>(out);
  const uint32_t total = segments * units;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const uint32_t d = idx / units, c = idx - d * units;
    A acc[U];
#pragma unroll
    for (int i = 0; i < U; ++i) acc[i] = A(0);
    const int64_t e1 = __ldg(ptr + d + 1);
    int64_t e = __ldg(ptr + d);
    for (; e + 4 <= e1; e += 4) {                      // four rows in flight, added in ascending order
      Q q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k] = src[(perm ? __ldg(perm + e + k) : e + k) * units + c];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < U; ++i) acc[i] += static_cast<A>(q[k].v[i]);
    }
    for (; e < e1; ++e) {
      const Q q = src[(perm ? __ldg(perm + e) : e) * units + c];
#pragma unroll
      for (int i = 0; i < U; ++i) acc[i] += static_cast<A>(q.v[i]);
    }
    Q o;
#pragma unroll
    for (int i = 0; i < U; ++i) o.v[i] = static_cast<T>(acc[i]);
    dst[idx] = o;
  }
}

template <typename T, int U>
__global__ void __launch_bounds__(256) gather_rows_kernel(const T* __restrict__ in, const int64_t* __restrict__ index,
                                                          T* __restrict__ out, uint32_t rows, uint32_t units) {
  using Q = Unit<T, U>;
  const Q* src = reinterpret_cast<const Q*>(in);
  Q* dst = reinterpret_cast<Q*>(out);
  const uint32_t total = rows * units;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const uint32_t r = idx / units, c = idx - r * units;
    dst[idx] = src[__ldg(index + r) * units + c];
  }
}

// Adjoint of the segment sum: every row of segment d becomes row d of `in`; rows outside all segments become zero.
// A warp holds 32 units of one segment's row and writes them to its edges (short segments; long ones below).
template <typename T, int U>
__global__ void __launch_bounds__(256) expand_segments_kernel(const T* __restrict__ in, const int64_t* __restrict__ ptr,
                                                              T* __restrict__ out, int64_t segments, int64_t rows, uint32_t units) {
  using Q = Unit<T, U>;
  const Q* src = reinterpret_cast<const Q*>(in);
  Q* dst = reinterpret_cast<Q*>(out);
  const int lane = threadIdx.x & 31;
  const int64_t warp = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5), warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  Q zero;
#pragma unroll
  for (int i = 0; i < U; ++i) zero.v[i] = static_cast<T>(0.f);
  for (uint32_t c = blockIdx.y * 32 + lane; c < units; c += gridDim.y * 32) {
    for (int64_t d = warp; d < segments; d += warps) {
      const int64_t e0 = max(__ldg(ptr + d), (int64_t)0), e1 = min(__ldg(ptr + d + 1), rows);
      if (e0 >= e1) continue;
      const Q q = src[d * units + c];
      for (int64_t e = e0; e < e1; ++e) dst[e * units + c] = q;
    }
    const int64_t first = min(segments ? __ldg(ptr) : rows, rows), last = segments ? __ldg(ptr + segments) : rows;
    for (int64_t e = warp; e < first; e += warps) dst[e * units + c] = zero;
    for (int64_t e = max(last, (int64_t)0) + warp; e < rows; e += warps) dst[e * units + c] = zero;
  }
}

// The same with the work spread over the rows, for long segments: a warp takes `EXPAND_RUN` consecutive rows per row it holds at
// a time (32 / lanes of them: `lanes` is the power of two that holds a row's units, at most a warp), finds the segment of the
// first by a 32-way search and walks on from there.  1M rows of 64 float32 in one segment 39 us (above, 11.7 ms), 100k in 32
// segments 6.4 us (104 us); short segments are better off above: 20,480 rows of 480 float32 in 960 segments 8.2 us against 9.0,
// 100k rows of 16 in 100k segments 11 against 18.
constexpr int EXPAND_RUN = 16;
template <typename T, int U>
__global__ void __launch_bounds__(256) expand_rows_kernel(const T* __restrict__ in, const int64_t* __restrict__ ptr,
                                                          T* __restrict__ out, int64_t segments, int64_t rows, uint32_t units,
                                                          int lanes) {
  using Q = Unit<T, U>;
  const Q* src = reinterpret_cast<const Q*>(in);
  Q* dst = reinterpret_cast<Q*>(out);
  Q zero;
#pragma unroll
  for (int i = 0; i < U; ++i) zero.v[i] = static_cast<T>(0.f);
  const int lane = threadIdx.x & 31, side = 32 / lanes, sub = lane / lanes;
  const int64_t span = (int64_t)EXPAND_RUN * side, warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r0 = (blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * span; r0 < rows; r0 += warps * span) {
    const int64_t r1 = min(r0 + span, rows);
    int64_t first = -1, above = segments + 1;              // ptr[first] <= r0 < ptr[above], ptr[-1] = -inf
    while (above - first > 1) {
      const int64_t step = (above - first + 32) / 33, at = first + (lane + 1) * step;
      const bool below = at < above && __ldg(ptr + at) <= r0;
      const int hits = __popc(__ballot_sync(0xffffffffu, below));
      above = min(above, first + (hits + 1) * step);
      first += hits * step;
    }
    for (uint32_t c = blockIdx.y * 32 + lane % lanes; c < units; c += gridDim.y * 32) {
      int64_t d = first, end = d < segments ? __ldg(ptr + d + 1) : rows;
      Q q = d >= 0 && d < segments ? src[d * units + c] : zero;
      for (int64_t e = r0 + sub; e < r1; e += side) {
        if (e >= end && d < segments) {
          do end = ++d < segments ? __ldg(ptr + d + 1) : rows; while (d < segments && e >= end);
          q = d < segments ? src[d * units + c] : zero;
        }
        dst[e * units + c] = q;
      }
    }
  }
}

// Adjoint of the gather: out[index[e]] += in[e] in float32 whatever the storage type, with 16-byte reductions at L2
// where the row width allows.  Replaces element-wise atomics in the storage type (73 us for 20,480 rows of 480
// bfloat16, 12 us here) and their bfloat16 sums.
template <typename T, int U>
__global__ void __launch_bounds__(256) scatter_add_rows_kernel(const T* __restrict__ in, const int64_t* __restrict__ index,
                                                               float* __restrict__ out, uint32_t rows, uint32_t units, int64_t out_rows) {
  using Q = Unit<T, U>;
  const Q* src = reinterpret_cast<const Q*>(in);
  const uint32_t total = rows * units;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const uint32_t r = idx / units, c = idx - r * units;
    const int64_t to = __ldg(index + r);
    if (to < 0 || to >= out_rows) continue;
    const Q q = src[idx];
    float* o = out + (to * units + c) * U;
    if constexpr (U == 4)
      atomicAdd(reinterpret_cast<float4*>(o), make_float4(static_cast<float>(q.v[0]), static_cast<float>(q.v[1]),
                                                          static_cast<float>(q.v[2]), static_cast<float>(q.v[3])));
    else
      atomicAdd(o, static_cast<float>(q.v[0]));
  }
}

inline bool unit_ok(int64_t width, size_t elem, size_t bytes, const void* a, const void* b) {
  return (width * elem) % bytes == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & (bytes - 1)) == 0;
}

// rows are processed in pieces whose flat unit index (grid stride included) fits 32 bits
template <typename F> int row_pieces(int64_t rows, int64_t units, F launch) {
  const int64_t cap = std::max<int64_t>(1, (int64_t(1) << 31) / std::max<int64_t>(1, units));
  if (units >= (int64_t(1) << 31)) return fail(EQT_ERR_UNSUPPORTED, "rows of more than 2^31 elements");
  for (int64_t r = 0; r < rows; r += cap)
    if (int rc = launch(r, std::min(cap, rows - r))) return rc;
  return EQT_OK;
}

template <typename T>
int run_segment_sum(const T* in, const int64_t* ptr, const int64_t* perm, T* out, int64_t segments, int64_t width, cudaStream_t s) {
  constexpr int U = 16 / sizeof(T);
  const bool wide = unit_ok(width, sizeof(T), 16, in, out);
  const int64_t units = wide ? width / U : width;
  return row_pieces(segments, units, [&](int64_t r, int64_t n) {
    const unsigned grid = flat_grid(n * units, 256);
    if (wide) segment_sum_kernel<T, U><<<grid, 256, 0, s>>>(in, ptr + r, perm, out + r * width, (uint32_t)n, (uint32_t)units);
    else segment_sum_kernel<T, 1><<<grid, 256, 0, s>>>(in, ptr + r, perm, out + r * width, (uint32_t)n, (uint32_t)units);
    return check_launch("segment_sum_kernel");
  });
}

template <typename T>
int run_gather_rows(const T* in, const int64_t* index, T* out, int64_t rows, int64_t width, cudaStream_t s) {
  constexpr int U = 16 / sizeof(T);
  const bool wide = unit_ok(width, sizeof(T), 16, in, out);
  const int64_t units = wide ? width / U : width;
  return row_pieces(rows, units, [&](int64_t r, int64_t n) {
    const unsigned grid = flat_grid(n * units, 256);
    if (wide) gather_rows_kernel<T, U><<<grid, 256, 0, s>>>(in, index + r, out + r * width, (uint32_t)n, (uint32_t)units);
    else gather_rows_kernel<T, 1><<<grid, 256, 0, s>>>(in, index + r, out + r * width, (uint32_t)n, (uint32_t)units);
    return check_launch("gather_rows_kernel");
  });
}

template <typename T>
int run_expand_segments(const T* in, const int64_t* ptr, T* out, int64_t segments, int64_t rows, int64_t width, cudaStream_t s) {
  constexpr int U = 16 / sizeof(T);
  const bool wide = unit_ok(width, sizeof(T), 16, in, out);
  const int64_t units = wide ? width / U : width;
  const unsigned columns = (unsigned)std::min<int64_t>(ceil_div(units, 32), 65535);
  if (rows >= 32 * segments) {                          // long segments on average: see the kernels
    int lanes = 1;
    while (lanes < 32 && lanes < units) lanes *= 2;
    const dim3 grid(flat_grid(ceil_div(rows, (int64_t)EXPAND_RUN * (32 / lanes)) * 32, 256, 16), columns);
    if (wide) expand_rows_kernel<T, U><<<grid, 256, 0, s>>>(in, ptr, out, segments, rows, (uint32_t)units, lanes);
    else expand_rows_kernel<T, 1><<<grid, 256, 0, s>>>(in, ptr, out, segments, rows, (uint32_t)units, lanes);
    return check_launch("expand_rows_kernel");
  }
  const dim3 grid(flat_grid(segments * 32, 256, 16), columns);
  if (wide) expand_segments_kernel<T, U><<<grid, 256, 0, s>>>(in, ptr, out, segments, rows, (uint32_t)units);
  else expand_segments_kernel<T, 1><<<grid, 256, 0, s>>>(in, ptr, out, segments, rows, (uint32_t)units);
  return check_launch("expand_segments_kernel");
}

template <typename T>
int run_scatter_add(const T* in, const int64_t* index, float* out, int64_t rows, int64_t width, int64_t out_rows, cudaStream_t s) {
  const bool wide = width % 4 == 0 && unit_ok(width, sizeof(T), 4 * sizeof(T), in, in) && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const int64_t units = wide ? width / 4 : width;
  return row_pieces(rows, units, [&](int64_t r, int64_t n) {
    const unsigned grid = flat_grid(n * units, 256);
    if (wide) scatter_add_rows_kernel<T, 4><<<grid, 256, 0, s>>>(in + r * width, index + r, out, (uint32_t)n, (uint32_t)units, out_rows);
    else scatter_add_rows_kernel<T, 1><<<grid, 256, 0, s>>>(in + r * width, index + r, out, (uint32_t)n, (uint32_t)units, out_rows);
    return check_launch("scatter_add_rows_kernel");
  });
}

int check_table(const eqt_sh_table* t) {
  if (!t) return fail(EQT_ERR_BAD_ARGUMENT, "sh table is NULL");
  if (t->l_max < 0 || t->l_max > 64) return fail(EQT_ERR_UNSUPPORTED, "l_max %d outside [0, 64]", t->l_max);
  if (t->l_max > 0 && (!t->ptr || !t->m_out || !t->m_in || !t->axis || !t->coef))
    return fail(EQT_ERR_BAD_ARGUMENT, "sh table has NULL arrays");
  return EQT_OK;
}

template <typename T>
int sh_launch(bool backward, const void* xyz, const void* gout, void* out, int64_t n, const eqt_sh_table* t,
              int normalize, double out_scale, cudaStream_t s) {
  using A = typename Acc<T>::type;
  if (n == 0) return EQT_OK;
  switch (t->l_max) {   // straight-line kernels for the degrees generated at build time
    case 1: return sh_launch_unrolled<T, 1>(backward, xyz, gout, out, n, normalize, out_scale, s);
    case 2: return sh_launch_unrolled<T, 2>(backward, xyz, gout, out, n, normalize, out_scale, s);
    case 3: return sh_launch_unrolled<T, 3>(backward, xyz, gout, out, n, normalize, out_scale, s);
    case 4: return sh_launch_unrolled<T, 4>(backward, xyz, gout, out, n, normalize, out_scale, s);
    default: break;
  }
  ShTab tab{t->ptr, t->m_out, t->m_in, t->axis, t->coef, t->l_max};
  const int K = (t->l_max + 1) * (t->l_max + 1), W = 2 * t->l_max + 1;
  const size_t per_thread = sizeof(A) * (backward ? 8 * W : K);
  int threads = 256;
  while (threads > 32 && per_thread * threads > 64 * 1024) threads >>= 1;
  const size_t bytes = per_thread * threads;
  const unsigned grid = flat_grid(n, threads, 8);
  if (backward) {
    if (int rc = configure_smem(sh_backward_kernel<T>, bytes)) return rc;
    sh_backward_kernel<T><<<grid, threads, bytes, s>>>(static_cast<const T*>(xyz), static_cast<const T*>(gout),
                                                        static_cast<T*>(out), n, tab, normalize, (A)out_scale);
    return check_launch("sh_backward_kernel");
  }
  if (int rc = configure_smem(sh_forward_kernel<T>, bytes)) return rc;
  sh_forward_kernel<T><<<grid, threads, bytes, s>>>(static_cast<const T*>(xyz), static_cast<T*>(out), n, tab,
                                                     normalize, (A)out_scale);
  return check_launch("sh_forward_kernel");
}

}  // namespace
}  // namespace eqt

extern "C" int eqt_sh_forward(int32_t dtype, const void* xyz, void* out, int64_t n, const eqt_sh_table* table,
                              int32_t normalize, double out_scale, void* stream) {
  using namespace eqt;
  if (int rc = check_table(table)) return rc;
  if (n < 0 || (n > 0 && (!xyz || !out))) return fail(EQT_ERR_BAD_ARGUMENT, "bad xyz/out/n");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == EQT_F32) return sh_launch<float>(false, xyz, nullptr, out, n, table, normalize, out_scale, s);
  if (dtype == EQT_F64) return sh_launch<double>(false, xyz, nullptr, out, n, table, normalize, out_scale, s);
  return fail(EQT_ERR_UNSUPPORTED, "spherical harmonics support float32 and float64");
}

extern "C" int eqt_sh_backward(int32_t dtype, const void* xyz, const void* grad_out, void* grad_xyz, int64_t n,
                               const eqt_sh_table* table, int32_t normalize, double out_scale, void* stream) {
  using namespace eqt;
  if (int rc = check_table(table)) return rc;
  if (n < 0 || (n > 0 && (!xyz || !grad_out || !grad_xyz))) return fail(EQT_ERR_BAD_ARGUMENT, "bad pointers/n");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype == EQT_F32) return sh_launch<float>(true, xyz, grad_out, grad_xyz, n, table, normalize, out_scale, s);
  if (dtype == EQT_F64) return sh_launch<double>(true, xyz, grad_out, grad_xyz, n, table, normalize, out_scale, s);
  return fail(EQT_ERR_UNSUPPORTED, "spherical harmonics support float32 and float64");
}

extern "C" int eqt_segment_sum(int32_t dtype, const void* in, const int64_t* ptr, const int64_t* perm, void* out,
                               int64_t num_segments, int64_t width, void* stream) {
  using namespace eqt;
  if (num_segments < 0 || width < 0) return fail(EQT_ERR_BAD_ARGUMENT, "negative size");
  if (num_segments == 0 || width == 0) return EQT_OK;
  if (!in || !ptr || !out) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case EQT_F32: return run_segment_sum((const float*)in, ptr, perm, (float*)out, num_segments, width, s);
    case EQT_F64: return run_segment_sum((const double*)in, ptr, perm, (double*)out, num_segments, width, s);
    case EQT_BF16: return run_segment_sum((const __nv_bfloat16*)in, ptr, perm, (__nv_bfloat16*)out, num_segments, width, s);
    default: return fail(EQT_ERR_BAD_ARGUMENT, "unknown dtype %d", dtype);
  }
}

extern "C" int eqt_gather_rows(int32_t dtype, const void* in, const int64_t* index, void* out, int64_t num_rows,
                               int64_t width, void* stream) {
  using namespace eqt;
  if (num_rows < 0 || width < 0) return fail(EQT_ERR_BAD_ARGUMENT, "negative size");
  if (num_rows == 0 || width == 0) return EQT_OK;
  if (!in || !index || !out) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case EQT_F32: return run_gather_rows((const float*)in, index, (float*)out, num_rows, width, s);
    case EQT_F64: return run_gather_rows((const double*)in, index, (double*)out, num_rows, width, s);
    case EQT_BF16: return run_gather_rows((const __nv_bfloat16*)in, index, (__nv_bfloat16*)out, num_rows, width, s);
    default: return fail(EQT_ERR_BAD_ARGUMENT, "unknown dtype %d", dtype);
  }
}

extern "C" int eqt_expand_segments(int32_t dtype, const void* in, const int64_t* ptr, void* out, int64_t num_segments,
                                   int64_t num_rows, int64_t width, void* stream) {
  using namespace eqt;
  if (num_segments < 0 || num_rows < 0 || width < 0) return fail(EQT_ERR_BAD_ARGUMENT, "negative size");
  if (num_rows == 0 || width == 0) return EQT_OK;
  if ((num_segments > 0 && (!in || !ptr)) || !out) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (num_segments == 0 && (dtype == EQT_F32 || dtype == EQT_F64 || dtype == EQT_BF16)) {
    cudaError_t e = cudaMemsetAsync(out, 0, (dtype == EQT_F64 ? 8 : dtype == EQT_F32 ? 4 : 2) * (size_t)(num_rows * width), s);
    return e == cudaSuccess ? EQT_OK : fail(EQT_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
  }
  switch (dtype) {
    case EQT_F32: return run_expand_segments((const float*)in, ptr, (float*)out, num_segments, num_rows, width, s);
    case EQT_F64: return run_expand_segments((const double*)in, ptr, (double*)out, num_segments, num_rows, width, s);
    case EQT_BF16: return run_expand_segments((const __nv_bfloat16*)in, ptr, (__nv_bfloat16*)out, num_segments, num_rows, width, s);
    default: return fail(EQT_ERR_BAD_ARGUMENT, "unknown dtype %d", dtype);
  }
}

extern "C" int eqt_scatter_add_rows(int32_t dtype, const void* in, const int64_t* index, float* out, int64_t num_rows, int64_t width,
                                    int64_t out_rows, void* stream) {
  using namespace eqt;
  if (num_rows < 0 || width < 0 || out_rows < 0) return fail(EQT_ERR_BAD_ARGUMENT, "negative size");
  if (out_rows == 0 || width == 0) return EQT_OK;
  if (!out || (num_rows > 0 && (!in || !index))) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (dtype != EQT_F32 && dtype != EQT_BF16) return fail(EQT_ERR_UNSUPPORTED, "row scatter sums float32 or bfloat16 rows");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(float) * (size_t)(out_rows * width), s);
  if (e != cudaSuccess) return fail(EQT_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
  if (num_rows == 0) return EQT_OK;
  switch (dtype) {
    case EQT_F32: return run_scatter_add((const float*)in, index, out, num_rows, width, out_rows, s);
    case EQT_BF16: return run_scatter_add((const __nv_bfloat16*)in, index, out, num_rows, width, out_rows, s);
    default: return EQT_ERR_UNSUPPORTED;
  }
}
