// Generic batched sparse-dense products (table driven).
//
// One kernel family per product shape.  All of them read the sorted table
// (scale, index1, index2, seg, gather_index, index_out) straight from global memory: the
// loads are warp-uniform, so they are broadcast from L1.  The hot configurations of the
// tensor-product layers do not go through these kernels but through the fused ones in
// so3_fused.cu; these cover every flag combination of the operator API.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <type_traits>

#include "common.cuh"

namespace eqt {

thread_local char t_error[512] = "";
std::atomic<int64_t> g_launches{0};
char* error_buffer() { return t_error; }
int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(t_error, sizeof(t_error), fmt, ap);
  va_end(ap);
  return code;
}
int sm_count() {
  constexpr int kMaxDevices = 64;
  static std::atomic<int> cached[kMaxDevices];   // zero-initialised; a race only repeats the query
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev >= 0 && dev < kMaxDevices) {
    const int n = cached[dev].load(std::memory_order_relaxed);
    if (n > 0) return n;
  }
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  if (dev >= 0 && dev < kMaxDevices) cached[dev].store(n, std::memory_order_relaxed);
  return n;
}

namespace {

struct P {  // kernel-side copy of eqt_product_args with strides resolved
  const void* in1;
  const void* in2;
  void* out;
  const void* scale;
  const int64_t* i1;
  const int64_t* i2;
  const int64_t* seg;
  const int64_t* gather;
  const int64_t* iout;
  int64_t n, rows1, rows2, num_out, out_size, c1, c2;
  int64_t bs1, bs2;  // batch strides in elements (0 when shared)
};

struct Entry {
  int64_t r1, r2, tt;
};

__device__ __forceinline__ void seg_range(const P& p, int64_t o, int64_t& t0, int64_t& t1) {
  if (p.seg) {
    t0 = __ldg(p.seg + o);
    t1 = __ldg(p.seg + o + 1);
  } else {
    t0 = o;
    t1 = o + 1;
  }
}
__device__ __forceinline__ Entry entry(const P& p, int64_t t) {
  Entry e;
  e.tt = p.gather ? __ldg(p.gather + t) : t;
  e.r1 = p.i1 ? __ldg(p.i1 + e.tt) : e.tt;
  e.r2 = p.i2 ? __ldg(p.i2 + e.tt) : e.tt;
  return e;
}
template <typename T>
__device__ __forceinline__ typename Acc<T>::type scale_of(const P& p, int64_t tt) {
  using A = typename Acc<T>::type;
  return p.scale ? __ldg(static_cast<const A*>(p.scale) + tt) : A(1);
}
__device__ __forceinline__ int64_t out_row(const P& p, int64_t o) { return p.iout ? __ldg(p.iout + o) : o; }

// ------------------------------------------------------------------------------------------
// channel-wise family: MUL, VECSCA, SCALE
// ------------------------------------------------------------------------------------------
template <typename T, int OP>
__global__ void __launch_bounds__(256) ew_kernel(P p) {
  using A = typename Acc<T>::type;
  const T* x = static_cast<const T*>(p.in1);
  const T* y = static_cast<const T*>(p.in2);
  T* out = static_cast<T*>(p.out);
  const int64_t C = p.c1;
  const int64_t total = p.n * p.num_out * C;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = idx % C;
    const int64_t o = (idx / C) % p.num_out;
    const int64_t n = idx / (C * p.num_out);
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    A acc = 0;
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = entry(p, t);
      A v = ld(x + n * p.bs1 + e.r1 * C + c);
      if (OP == EQT_OP_MUL) v *= ld(y + n * p.bs2 + e.r2 * C + c);
      if (OP == EQT_OP_VECSCA) v *= ld(y + n * p.bs2 + e.r2);
      acc += v * scale_of<T>(p, e.tt);
    }
    st(out + (n * p.out_size + out_row(p, o)) * C + c, acc);
  }
}

// float, C % 4 == 0, 16-byte aligned operands: a thread owns four channels of one output row and walks a range of samples, four
// at a time, so that its place, the row's segment and the first entry are found once and four 128-bit loads per operand are in
// flight.  With one flattened index over samples, rows and channels every element paid three divisions and the chain of table
// loads in front of its operands (7k nodes, 35 rows x 128 channels: 44 us a pass, 40 us so; the tables in shared memory
// instead: 42).  Where all rows of a sample have fewer items than the block threads, `sets` = threads / items of them take every
// sets-th sample of the block's range (1M samples of one row of 4 channels: 130 us with the other threads idle, 6.5 us so, 9.5 us
// with the flattened index; 100k samples of 9 rows x 16 channels: 38.6, 28.9 and 34.7 us).
constexpr int EW_THREADS = 128;
template <int OP, bool SETS>
__global__ void __launch_bounds__(EW_THREADS) ew_kernel_f4(P p, int64_t chunk, int several) {
  const int sets = SETS ? several : 1;
  const float* x = static_cast<const float*>(p.in1);
  const float* y = static_cast<const float*>(p.in2);
  const int64_t C = p.c1, c4 = C / 4, items = p.num_out * c4;
  const int64_t set = SETS ? threadIdx.x / items : 0;
  const int64_t item = SETS ? threadIdx.x - set * items : blockIdx.x * (int64_t)EW_THREADS + threadIdx.x;
  if (item >= items || set >= sets) return;
  const int64_t o = item / c4, c = (item - o * c4) * 4;
  const int64_t n0 = blockIdx.y * chunk, n1 = min(n0 + chunk, p.n);
  int64_t t0, t1;
  seg_range(p, o, t0, t1);
  const Entry first = t0 < t1 ? entry(p, t0) : Entry{0, 0, 0};
  const float first_scale = t0 < t1 ? scale_of<float>(p, first.tt) : 0.f;
  float* out = static_cast<float*>(p.out) + out_row(p, o) * C + c;
  const int64_t out_stride = p.out_size * C;
  for (int64_t n = n0 + set; n < n1; n += 4 * sets) {                 // its samples: n, n + sets, n + 2 sets, n + 3 sets
    float4 acc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = t == t0 ? first : entry(p, t);
      const float scale = t == t0 ? first_scale : scale_of<float>(p, e.tt);
      float4 v[4], w[4];
      float s[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s[u] = scale;
        if (n + u * sets >= n1) continue;
        v[u] = __ldg(reinterpret_cast<const float4*>(x + (n + u * sets) * p.bs1 + e.r1 * C + c));
        if (OP == EQT_OP_MUL) w[u] = __ldg(reinterpret_cast<const float4*>(y + (n + u * sets) * p.bs2 + e.r2 * C + c));
        if (OP == EQT_OP_VECSCA) s[u] *= __ldg(y + (n + u * sets) * p.bs2 + e.r2);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (n + u * sets >= n1) continue;
        if (OP == EQT_OP_MUL) { v[u].x *= w[u].x; v[u].y *= w[u].y; v[u].z *= w[u].z; v[u].w *= w[u].w; }
        acc[u].x += v[u].x * s[u]; acc[u].y += v[u].y * s[u]; acc[u].z += v[u].z * s[u]; acc[u].w += v[u].w * s[u];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (n + u * sets < n1) *reinterpret_cast<float4*>(out + (n + u * sets) * out_stride) = acc[u];
  }
}

// bfloat16 storage, C % 8 == 0, 16-byte aligned operands: eight channels per thread, 128-bit accesses, float sums,
// 32-bit index arithmetic (the launcher checks that the element count fits).
template <int OP>
__global__ void __launch_bounds__(256) ew_kernel_b8(P p) {
  const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(p.in1);
  const __nv_bfloat16* y = static_cast<const __nv_bfloat16*>(p.in2);
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out);
  const uint32_t C = (uint32_t)p.c1, C8 = C / 8, num_out = (uint32_t)p.num_out;
  const uint32_t total = (uint32_t)p.n * num_out * C8;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    const uint32_t c = (idx % C8) * 8;
    const uint32_t o = (idx / C8) % num_out;
    const int64_t n = idx / (C8 * num_out);
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = entry(p, t);
      const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + n * p.bs1 + e.r1 * C + c));
      const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&xv);
      float s = p.scale ? __ldg(static_cast<const float*>(p.scale) + e.tt) : 1.f;
      float v[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(xp[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
      }
      if (OP == EQT_OP_MUL) {
        const uint4 yv = __ldg(reinterpret_cast<const uint4*>(y + n * p.bs2 + e.r2 * C + c));
        const __nv_bfloat162* yp = reinterpret_cast<const __nv_bfloat162*>(&yv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __bfloat1622float2(yp[i]);
          v[2 * i] *= f.x;
          v[2 * i + 1] *= f.y;
        }
      }
      if (OP == EQT_OP_VECSCA) s *= __bfloat162float(__ldg(y + n * p.bs2 + e.r2));
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += v[i] * s;
    }
    uint4 ov;
    __nv_bfloat162* op2 = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
    for (int i = 0; i < 4; ++i) op2[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
    *reinterpret_cast<uint4*>(out + (n * p.out_size + out_row(p, o)) * C + c) = ov;
  }
}

// Batch-summed form: out[o, c] = sum_n sum_t ...   block = 32 channels x 8 batch lanes,
// grid = (num_out * channel tiles, batch chunks); one atomicAdd per block and output element.
template <typename T, int OP>
__global__ void __launch_bounds__(256) ew_acc_kernel(P p, int64_t chunk) {
  using A = typename Acc<T>::type;
  __shared__ A red[8][33];
  const T* x = static_cast<const T*>(p.in1);
  const T* y = static_cast<const T*>(p.in2);
  A* out = static_cast<A*>(p.out);
  const int64_t C = p.c1;
  const int64_t ctiles = ceil_div(C, 32);
  const int64_t o = blockIdx.x / ctiles;
  const int64_t c = (blockIdx.x % ctiles) * 32 + threadIdx.x;
  const int64_t n0 = blockIdx.y * chunk;
  const int64_t n1 = min(n0 + chunk, p.n);
  int64_t t0, t1;
  seg_range(p, o, t0, t1);
  A acc = 0;
  // The entries of the output row are the same for every sample: they are staged in shared memory once (up to
  // ACC_STAGE of them), and four samples are in flight per thread - with one, a thread waited for the latency of
  // memory at every sample and the kernel ran at a seventh of the bandwidth.
  constexpr int ACC_STAGE = 64;
  __shared__ int32_t e_r1[ACC_STAGE], e_r2[ACC_STAGE];
  __shared__ A e_sc[ACC_STAGE];
  const bool staged = t1 - t0 <= ACC_STAGE;
  if (staged) {
    const int tid = threadIdx.y * 32 + threadIdx.x;
    if (tid < t1 - t0) {
      const Entry e = entry(p, t0 + tid);
      e_r1[tid] = (int32_t)e.r1;
      e_r2[tid] = (int32_t)e.r2;
      e_sc[tid] = scale_of<T>(p, e.tt);
    }
    __syncthreads();
  }
  if (c < C && staged) {
    const int ne = (int)(t1 - t0);
    for (int64_t n = n0 + threadIdx.y; n < n1; n += 32) {
      A part[4] = {0, 0, 0, 0};
      for (int t = 0; t < ne; ++t) {
        const int64_t o1 = (int64_t)e_r1[t] * C + c, o2 = OP == EQT_OP_MUL ? (int64_t)e_r2[t] * C + c : (int64_t)e_r2[t];
        const A sc = e_sc[t];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t nn = n + 8 * u;
          if (nn < n1) {
            A v = ld(x + nn * p.bs1 + o1);
            if (OP == EQT_OP_MUL || OP == EQT_OP_VECSCA) v *= ld(y + nn * p.bs2 + o2);
            part[u] += v * sc;
          }
        }
      }
      acc += (part[0] + part[1]) + (part[2] + part[3]);
    }
  } else if (c < C) {
    for (int64_t n = n0 + threadIdx.y; n < n1; n += 8) {
      for (int64_t t = t0; t < t1; ++t) {
        const Entry e = entry(p, t);
        A v = ld(x + n * p.bs1 + e.r1 * C + c);
        if (OP == EQT_OP_MUL) v *= ld(y + n * p.bs2 + e.r2 * C + c);
        if (OP == EQT_OP_VECSCA) v *= ld(y + n * p.bs2 + e.r2);
        acc += v * scale_of<T>(p, e.tt);
      }
    }
  }
  red[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && c < C) {
    A s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[k][threadIdx.x];
    atomicAdd(out + out_row(p, o) * C + c, s);
  }
}

// The same for float32 with C % 4 == 0 and 16-byte aligned operands: a thread owns four channels, so that a load is 16 bytes and
// eight of them are in flight per thread (7k nodes, 35 rows x 128 channels into 11 weight rows: 121 us with 4-byte loads,
// 47 us so).  blockDim = (lanes, 256 / lanes), lanes = the power of two that holds C / 4, at most 32.
template <int OP>
__global__ void __launch_bounds__(256) ew_acc_f4_kernel(P p, int64_t chunk) {
  constexpr int STAGE = 64;
  __shared__ int32_t e_r1[STAGE], e_r2[STAGE];
  __shared__ float e_sc[STAGE];
  __shared__ float4 red[256];
  const float* x = static_cast<const float*>(p.in1);
  const float* y = static_cast<const float*>(p.in2);
  float* out = static_cast<float*>(p.out);
  const int64_t C = p.c1, tiles = ceil_div(C / 4, (int64_t)blockDim.x);
  const int64_t o = blockIdx.x / tiles, c = ((blockIdx.x % tiles) * blockDim.x + threadIdx.x) * 4;
  const int64_t n0 = blockIdx.y * chunk, n1 = min(n0 + chunk, p.n);
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  int64_t t0, t1;
  seg_range(p, o, t0, t1);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int64_t tb = t0; tb < t1; tb += STAGE) {
    const int ne = (int)min((int64_t)STAGE, t1 - tb);
    __syncthreads();
    if (tid < ne) {
      const Entry e = entry(p, tb + tid);
      e_r1[tid] = (int32_t)e.r1;
      e_r2[tid] = (int32_t)e.r2;
      e_sc[tid] = scale_of<float>(p, e.tt);
    }
    __syncthreads();
    if (c >= C) continue;
    for (int64_t n = n0 + threadIdx.y; n < n1; n += 4 * blockDim.y) {
      float4 part[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) part[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int t = 0; t < ne; ++t) {
        const int64_t o1 = (int64_t)e_r1[t] * C + c, o2 = OP == EQT_OP_MUL ? (int64_t)e_r2[t] * C + c : (int64_t)e_r2[t];
        float4 v[4], w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t nn = n + u * (int)blockDim.y;
          v[u] = w[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (nn >= n1) continue;
          v[u] = __ldg(reinterpret_cast<const float4*>(x + nn * p.bs1 + o1));
          if (OP == EQT_OP_MUL) w[u] = __ldg(reinterpret_cast<const float4*>(y + nn * p.bs2 + o2));
          if (OP == EQT_OP_VECSCA) w[u].x = __ldg(y + nn * p.bs2 + o2);
        }
        const float sc = e_sc[t];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (OP == EQT_OP_MUL) { v[u].x *= w[u].x; v[u].y *= w[u].y; v[u].z *= w[u].z; v[u].w *= w[u].w; }
          if (OP == EQT_OP_VECSCA) { v[u].x *= w[u].x; v[u].y *= w[u].x; v[u].z *= w[u].x; v[u].w *= w[u].x; }
          part[u].x = fmaf(v[u].x, sc, part[u].x); part[u].y = fmaf(v[u].y, sc, part[u].y);
          part[u].z = fmaf(v[u].z, sc, part[u].z); part[u].w = fmaf(v[u].w, sc, part[u].w);
        }
      }
      acc.x += (part[0].x + part[1].x) + (part[2].x + part[3].x);
      acc.y += (part[0].y + part[1].y) + (part[2].y + part[3].y);
      acc.z += (part[0].z + part[1].z) + (part[2].z + part[3].z);
      acc.w += (part[0].w + part[1].w) + (part[2].w + part[3].w);
    }
  }
  red[tid] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && c < C) {
    for (int k = 1; k < (int)blockDim.y; ++k) {
      const float4 v = red[k * blockDim.x + threadIdx.x];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    float* to = out + out_row(p, o) * C + c;
    atomicAdd(to, acc.x);
    atomicAdd(to + 1, acc.y);
    atomicAdd(to + 2, acc.z);
    atomicAdd(to + 3, acc.w);
  }
}

// ------------------------------------------------------------------------------------------
// OUTER
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) outer_kernel(P p) {
  using A = typename Acc<T>::type;
  const T* x = static_cast<const T*>(p.in1);
  const T* y = static_cast<const T*>(p.in2);
  T* out = static_cast<T*>(p.out);
  const int64_t C1 = p.c1, C2 = p.c2, CC = C1 * C2;
  const int64_t total = p.n * p.num_out * CC;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = idx % C2;
    const int64_t a = (idx / C2) % C1;
    const int64_t o = (idx / CC) % p.num_out;
    const int64_t n = idx / (CC * p.num_out);
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    A acc = 0;
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = entry(p, t);
      acc += ld(x + n * p.bs1 + e.r1 * C1 + a) * ld(y + n * p.bs2 + e.r2 * C2 + b) * scale_of<T>(p, e.tt);
    }
    st(out + (n * p.out_size + out_row(p, o)) * CC + idx % CC, acc);
  }
}

// One warp per (sample, output row), C2 / 4 a power of two up to 32: a lane keeps its four columns of y for all rows a
// it serves, so an entry costs one 4-wide load of y, one broadcast load of x and four FMAs per four outputs, and the
// row leaves as 128-bit stores of consecutive lanes.  Bound: the C1 * C2 values written per row.  The form above spends
// several 64-bit divisions per output element; 2000 samples x 35 rows x 32 x 32 float32: 929 -> 78 us (3.7 TB/s).
template <typename T> struct alignas(4 * sizeof(T)) Quad { T v[4]; };
template <typename T>
__global__ void __launch_bounds__(256) outer_rows_kernel(P p) {
  using A = typename Acc<T>::type;
  constexpr int U = 8;                               // rows a per lane and pass
  const T* x = static_cast<const T*>(p.in1);
  const T* y = static_cast<const T*>(p.in2);
  T* out = static_cast<T*>(p.out);
  const int C1 = (int)p.c1, C2 = (int)p.c2, lanes_b = C2 / 4;
  const int lane = threadIdx.x & 31, b = (lane % lanes_b) * 4, a_first = lane / lanes_b, a_step = 32 / lanes_b;
  const int num_out = (int)p.num_out;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5), total = p.n * p.num_out;
  int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  int64_t n = w / num_out;
  int o = (int)(w - n * num_out);
  const int64_t step_n = warps / num_out;
  const int step_o = (int)(warps - step_n * num_out);
  for (; w < total; w += warps) {
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    T* orow = out + (n * p.out_size + out_row(p, o)) * C1 * C2 + b;
    for (int a0 = a_first; a0 < C1; a0 += U * a_step) {
      A acc[U][4];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[u][k] = A(0);
      for (int64_t t = t0; t < t1; ++t) {
        const Entry e = entry(p, t);
        const Quad<T> yq = *reinterpret_cast<const Quad<T>*>(y + n * p.bs2 + e.r2 * C2 + b);
        const A s = scale_of<T>(p, e.tt);
        A yv[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) yv[k] = static_cast<A>(yq.v[k]) * s;
        const T* xr = x + n * p.bs1 + e.r1 * C1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int a = a0 + u * a_step;
          const A xv = a < C1 ? ld(xr + a) : A(0);
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[u][k] = fma(xv, yv[k], acc[u][k]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int a = a0 + u * a_step;
        if (a >= C1) break;
        Quad<T> q;
#pragma unroll
        for (int k = 0; k < 4; ++k) q.v[k] = static_cast<T>(acc[u][k]);
        *reinterpret_cast<Quad<T>*>(orow + (int64_t)a * C2) = q;
      }
    }
    n += step_n;
    o += step_o;
    if (o >= num_out) { o -= num_out; ++n; }
  }
}

// Batch-summed outer product = a GEMM whose reduction runs over (sample, table entry) pairs:
//   out[o, a, b] = sum_{n, t in seg[o]} s_t x[n, i1_t, a] y[n, i2_t, b].
// 64x64 output tile per block, 4x4 per thread, 8 pairs staged in shared memory per step.
// grid = (tiles_a * tiles_b, num_out, batch chunks); partial tiles are combined with atomicAdd.
template <typename T>
__global__ void __launch_bounds__(256) outer_acc_kernel(P p, int64_t chunk) {
  using A = typename Acc<T>::type;
  constexpr int TILE = 64, KK = 8;
  __shared__ A sa[KK][TILE];
  __shared__ A sb[KK][TILE];
  const T* x = static_cast<const T*>(p.in1);
  const T* y = static_cast<const T*>(p.in2);
  A* out = static_cast<A*>(p.out);
  const int64_t C1 = p.c1, C2 = p.c2;
  const int64_t tiles_b = ceil_div(C2, TILE);
  const int64_t a0 = (blockIdx.x / tiles_b) * TILE, b0 = (blockIdx.x % tiles_b) * TILE;
  const int64_t o = blockIdx.y;
  const int64_t n0 = blockIdx.z * chunk, n1 = min(n0 + chunk, p.n);
  int64_t t0, t1;
  seg_range(p, o, t0, t1);
  const int64_t len = t1 - t0;
  const int64_t pairs = (n1 - n0) * len;
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
  A acc[4][4] = {};
  for (int64_t k0 = 0; k0 < pairs; k0 += KK) {
    // 2 * KK * TILE = 1024 loads for 256 threads
    for (int q = tid; q < 2 * KK * TILE; q += 256) {
      const int which = q / (KK * TILE), r = (q / TILE) % KK, col = q % TILE;
      const int64_t k = k0 + r;
      A v = 0;
      if (k < pairs) {
        const int64_t n = n0 + k / len;
        const Entry e = entry(p, t0 + k % len);
        if (which == 0) {
          if (a0 + col < C1) v = ld(x + n * p.bs1 + e.r1 * C1 + a0 + col) * scale_of<T>(p, e.tt);
        } else {
          if (b0 + col < C2) v = ld(y + n * p.bs2 + e.r2 * C2 + b0 + col);
        }
      }
      (which == 0 ? sa : sb)[r][col] = v;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < KK; ++r) {
      A av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = sa[r][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = sb[r][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
    }
    __syncthreads();
  }
  const int64_t orow = out_row(p, o);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t a = a0 + ty * 4 + i, b = b0 + tx * 4 + j;
      if (a < C1 && b < C2 && pairs > 0) atomicAdd(out + (orow * C1 + a) * C2 + b, acc[i][j]);
    }
}

// The same for few channels (C1 and C2 multiples of four, float32; outer_few_wanted): a team of (C1 / 4) (C2 / 4) threads per sample, four
// by four products a thread, operands straight from global memory, of which tiles of 64 x 64 would use a sixteenth at 16 x 16
// channels.  Entries outside, samples inside, four of them in flight; the teams' sums meet in shared memory.  99 rows into 23 outputs,
// 20k samples, 16 x 16 1909 -> 195 us, 24 x 24 1933 -> 389; 5000 samples, 48 x 40 528 -> 367; 252 entries into 41 outputs, 5000 samples, 16 x 16
// 1096 -> 125.
__global__ void __launch_bounds__(256) outer_acc_few_kernel(P p, int64_t chunk, int team, int teams) {
  extern __shared__ __align__(16) float sums[];            // [teams][C1][C2]
  const float* x = static_cast<const float*>(p.in1);
  const float* y = static_cast<const float*>(p.in2);
  float* out = static_cast<float*>(p.out);
  const int c1 = (int)p.c1, c2 = (int)p.c2, q2 = c2 / 4, tid = threadIdx.x;
  const int which = tid / team, place = tid % team, a0 = place / q2 * 4, b0 = place % q2 * 4;
  const int64_t o = blockIdx.x, n0 = blockIdx.y * chunk, n1 = min(n0 + chunk, p.n);
  if (which < teams) {
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    float acc[4][4] = {};
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = entry(p, t);
      const float s = scale_of<float>(p, e.tt);
      const float* xt = x + e.r1 * c1 + a0;
      const float* yt = y + e.r2 * c2 + b0;
      float part[4][4] = {};
      int64_t n = n0 + which;
      for (; n + 3 * teams < n1; n += 4 * teams) {
        float4 a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = __ldg(reinterpret_cast<const float4*>(xt + (n + u * teams) * p.bs1));
          b[u] = __ldg(reinterpret_cast<const float4*>(yt + (n + u * teams) * p.bs2));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float av[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, bv[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) part[i][j] = fmaf(av[i], bv[j], part[i][j]);
        }
      }
      for (; n < n1; n += teams) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(xt + n * p.bs1)), b = __ldg(reinterpret_cast<const float4*>(yt + n * p.bs2));
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) part[i][j] = fmaf(av[i], bv[j], part[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(s, part[i][j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(sums + (which * c1 + a0 + i) * c2 + b0) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  }
  __syncthreads();
  const int64_t orow = out_row(p, o);
  for (int i = tid; i < c1 * c2; i += 256) {
    float v = sums[i];
    for (int w = 1; w < teams; ++w) v += sums[w * c1 * c2 + i];
    atomicAdd(out + orow * c1 * c2 + i, v);
  }
}


// ------------------------------------------------------------------------------------------
// INNER: one warp per (sample, output row)
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) inner_kernel(P p, int accumulated) {
  using A = typename Acc<T>::type;
  const T* x = static_cast<const T*>(p.in1);
  const T* y = static_cast<const T*>(p.in2);
  const int64_t C = p.c1;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t total = p.n * p.num_out;
  for (int64_t w = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); w < total; w += warps) {
    const int64_t o = w % p.num_out, n = w / p.num_out;
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    A acc = 0;
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = entry(p, t);
      const T* xr = x + n * p.bs1 + e.r1 * C;
      const T* yr = y + n * p.bs2 + e.r2 * C;
      A dot = 0;
      for (int64_t c = lane; c < C; c += 32) dot += ld(xr + c) * ld(yr + c);
      acc += dot * scale_of<T>(p, e.tt);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    if (lane == 0) {
      const int64_t orow = out_row(p, o);
      if (accumulated)
        atomicAdd(static_cast<A*>(p.out) + orow, acc);
      else
        st(static_cast<T*>(p.out) + n * p.out_size + orow, acc);
    }
  }
}

// ------------------------------------------------------------------------------------------
// VECMAT
// ------------------------------------------------------------------------------------------
// Weights shared by the batch, output per sample: a grouped GEMM.  Block = 64 samples x 64
// output channels of one output row; the reduction runs over (table entry, input channel).
template <typename T>
__global__ void __launch_bounds__(256) vecmat_shared_w_kernel(P p) {
  using A = typename Acc<T>::type;
  constexpr int BN = 64, BCO = 64, KC = 16, PAD = 4;
  __shared__ A sx[KC][BN + PAD];
  __shared__ A sw[KC][BCO];
  const T* x = static_cast<const T*>(p.in1);
  const T* w = static_cast<const T*>(p.in2);
  T* out = static_cast<T*>(p.out);
  const int64_t Cin = p.c1, Cout = p.c2;
  const int64_t cotiles = ceil_div(Cout, BCO);
  const int64_t n0 = (blockIdx.x / cotiles) * BN, co0 = (blockIdx.x % cotiles) * BCO;
  const int64_t o = blockIdx.y;
  int64_t t0, t1;
  seg_range(p, o, t0, t1);
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
  A acc[4][4] = {};
  for (int64_t t = t0; t < t1; ++t) {
    const Entry e = entry(p, t);
    const A s = scale_of<T>(p, e.tt);
    for (int64_t ci0 = 0; ci0 < Cin; ci0 += KC) {
      for (int q = tid; q < KC * BN; q += 256) {  // x tile, transposed on the way in
        const int nn = q / KC, k = q % KC;
        A v = 0;
        if (n0 + nn < p.n && ci0 + k < Cin) v = ld(x + (n0 + nn) * p.bs1 + e.r1 * Cin + ci0 + k) * s;
        sx[k][nn] = v;
      }
      for (int q = tid; q < KC * BCO; q += 256) {
        const int k = q / BCO, j = q % BCO;
        A v = 0;
        if (ci0 + k < Cin && co0 + j < Cout) v = ld(w + (e.r2 * Cin + ci0 + k) * Cout + co0 + j);
        sw[k][j] = v;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < KC; ++k) {
        A av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = sx[k][ty * 4 + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[j] = sw[k][tx * 4 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
      }
      __syncthreads();
    }
  }
  const int64_t orow = out_row(p, o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t n = n0 + ty * 4 + i;
    if (n >= p.n) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t co = co0 + tx * 4 + j;
      if (co < Cout) st(out + (n * p.out_size + orow) * Cout + co, acc[i][j]);
    }
  }
}

// The same for 16 or 32 output channels, where tiles of 64 would mostly be padding (C_in a multiple of four up to 64, float32): a
// thread owns SPT samples and sixteen output channels; the weights of eight entries at a time, scaled, come from shared memory as
// broadcasts, a sample's rows straight from global memory.  18k samples, 99 rows, 16 -> 16 channels, both products 432 -> 153 us; 70k
// samples, 252 entries 3807 -> 901; 20k samples, 99 rows, 64 -> 32 878 -> 393 (64 -> 64 a sixteenth at a time: 53 -> 63 at 450 samples).
template <int SPT>
__global__ void __launch_bounds__(128) vecmat_few_kernel(P p) {
  constexpr int ENTRIES = 8;
  extern __shared__ __align__(16) float sw[];              // [ENTRIES][C_in][16]
  __shared__ int64_t row[ENTRIES];
  const float* x = static_cast<const float*>(p.in1);
  const float* w = static_cast<const float*>(p.in2);
  float* out = static_cast<float*>(p.out);
  const int cin = (int)p.c1, cout = (int)p.c2, tiles = cout / 16, tid = threadIdx.x;
  const int64_t o = blockIdx.y / tiles, co = blockIdx.y % tiles * 16;
  const int64_t first = blockIdx.x * (int64_t)(128 * SPT) + tid;
  int64_t t0, t1;
  seg_range(p, o, t0, t1);
  float acc[SPT][16] = {};
  for (int64_t tb = t0; tb < t1; tb += ENTRIES) {
    const int count = (int)min((int64_t)ENTRIES, t1 - tb);
    __syncthreads();
    for (int i = tid; i < count * cin * 16; i += 128) {
      const int k = i / 16;
      const Entry e = entry(p, tb + k / cin);
      sw[i] = __ldg(w + (e.r2 * cin + k % cin) * cout + co + i % 16) * scale_of<float>(p, e.tt);
    }
    if (tid < count) row[tid] = entry(p, tb + tid).r1 * cin;
    __syncthreads();
    for (int t = 0; t < count; ++t) {
      const float* xt = x + row[t];
      for (int c = 0; c < cin; c += 4) {
        float4 v[SPT];
#pragma unroll
        for (int s = 0; s < SPT; ++s)
          v[s] = first + s * 128 < p.n ? __ldg(reinterpret_cast<const float4*>(xt + (first + s * 128) * p.bs1 + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4* wk = reinterpret_cast<const float4*>(sw + (t * cin + c + k) * 16);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 f = wk[q];
#pragma unroll
            for (int s = 0; s < SPT; ++s) {
              const float a = k == 0 ? v[s].x : k == 1 ? v[s].y : k == 2 ? v[s].z : v[s].w;
              acc[s][4 * q] = fmaf(a, f.x, acc[s][4 * q]);
              acc[s][4 * q + 1] = fmaf(a, f.y, acc[s][4 * q + 1]);
              acc[s][4 * q + 2] = fmaf(a, f.z, acc[s][4 * q + 2]);
              acc[s][4 * q + 3] = fmaf(a, f.w, acc[s][4 * q + 3]);
            }
          }
        }
      }
    }
  }
  const int64_t orow = out_row(p, o);
#pragma unroll
  for (int s = 0; s < SPT; ++s) {
    const int64_t n = first + s * 128;
    if (n >= p.n) continue;
    float4* to = reinterpret_cast<float4*>(out + (n * p.out_size + orow) * cout + co);
#pragma unroll
    for (int q = 0; q < 4; ++q) to[q] = make_float4(acc[s][4 * q], acc[s][4 * q + 1], acc[s][4 * q + 2], acc[s][4 * q + 3]);
  }
}


// Any other sharing pattern (per-sample matrices, shared vector, batch-summed output): one
// thread per output element; the matrix is streamed once, so this form is bandwidth bound.
template <typename T>
__global__ void __launch_bounds__(256) vecmat_direct_kernel(P p, int accumulated) {
  using A = typename Acc<T>::type;
  const T* x = static_cast<const T*>(p.in1);
  const T* w = static_cast<const T*>(p.in2);
  const int64_t Cin = p.c1, Cout = p.c2;
  const int64_t total = p.n * p.num_out * Cout;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t co = idx % Cout;
    const int64_t o = (idx / Cout) % p.num_out;
    const int64_t n = idx / (Cout * p.num_out);
    int64_t t0, t1;
    seg_range(p, o, t0, t1);
    A acc = 0;
    for (int64_t t = t0; t < t1; ++t) {
      const Entry e = entry(p, t);
      const T* xr = x + n * p.bs1 + e.r1 * Cin;
      const T* wr = w + n * p.bs2 + e.r2 * Cin * Cout + co;
      A dot = 0;
      for (int64_t ci = 0; ci < Cin; ++ci) dot += ld(xr + ci) * ld(wr + ci * Cout);
      acc += dot * scale_of<T>(p, e.tt);
    }
    const int64_t orow = out_row(p, o);
    if (accumulated)
      atomicAdd(static_cast<A*>(p.out) + orow * Cout + co, acc);
    else
      st(static_cast<T*>(p.out) + (n * p.out_size + orow) * Cout + co, acc);
  }
}

// ------------------------------------------------------------------------------------------
// dispatch
// ------------------------------------------------------------------------------------------
inline bool aligned16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; }

// Chunks of samples for outer_acc_few_kernel, at most `most` of them: one sum after the other of k terms adds k to the square of the rounding
// error (in units of 2^-24 and of half the result), which are here a thread's samples, the teams and the chunks' atomics, and
// with the tiles of outer_acc_kernel `tiled` chunks and their samples.  No more chunks than keep the error below the tiles' (1000 samples,
// one entry an output, 48 x 40 channels: tiles 1.5e-7, 125 chunks of two teams 2.1e-7).
int64_t few_chunks(int64_t n, int teams, int64_t tiled, int64_t most) {
  const double per_team = (double)n / teams, limit = 0.9 * ((double)tiled + (double)n / tiled) - teams, root = limit * limit - 4 * per_team;
  const double chunks = limit > 0 && root >= 0 ? (limit + std::sqrt(root)) / 2 : std::sqrt(per_team);
  return std::max<int64_t>(1, std::min<int64_t>({(int64_t)chunks, most, ceil_div(n, 4 * teams), 65535}));
}

// Whether teams are the faster kernel.  Up to 1024 products, or where tiles of 64 x 64 would be mostly padding, always.  One or two teams
// a block are worth it for sums of several entries, where the tiles' indexing costs as much as their products (48 x 40, 23 rows into 9
// outputs, 1000 samples 43 -> 35 us, 20k 438 -> 338), without sums only for few samples (4 rows, 1000 samples 23 -> 16, 20k 82 -> 100; segments
// of one entry each, which the tables here never have, are taken for sums: 30 rows, 1000 samples 40 -> 47),
// beyond 2048 products only for few in any case (64 x 64, 99 rows into 23 outputs, 200 samples 57 -> 41, 400 samples 68 -> 76).
bool outer_few_wanted(const P& p, int64_t tiles) {
  const int64_t products = p.c1 * p.c2;
  if (products > 2048) return products <= 4096 && p.n <= 512 && p.n * p.num_out <= 4608;
  return products <= 1024 || tiles > 1 || p.seg || p.n * p.num_out <= 8192;
}

template <typename T>
int launch(const eqt_product_args& a, P p, cudaStream_t s) {
  const int op = a.op;
  if (p.n == 0 || p.num_out == 0) return EQT_OK;
  if (op == EQT_OP_MUL || op == EQT_OP_VECSCA || op == EQT_OP_SCALE) {
    if (p.c1 == 0) return EQT_OK;
    if (a.accumulated && std::is_same<T, float>::value && p.c1 % 4 == 0 && aligned16(p.in1) && (op != EQT_OP_MUL || aligned16(p.in2))) {
      int lanes = 1;
      while (lanes < 32 && lanes < p.c1 / 4) lanes *= 2;
      const int64_t blocks_x = p.num_out * ceil_div(p.c1 / 4, lanes);
      int64_t chunks = ceil_div((int64_t)sm_count() * 8, blocks_x);
      chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, ceil_div(p.n, 4 * (256 / lanes))));
      chunks = std::min<int64_t>(chunks, 65535);
      const int64_t chunk = ceil_div(p.n, chunks);
      if (blocks_x <= INT32_MAX) {
        dim3 grid((unsigned)blocks_x, (unsigned)ceil_div(p.n, chunk)), block(lanes, 256 / lanes);
        if (op == EQT_OP_MUL) ew_acc_f4_kernel<EQT_OP_MUL><<<grid, block, 0, s>>>(p, chunk);
        if (op == EQT_OP_VECSCA) ew_acc_f4_kernel<EQT_OP_VECSCA><<<grid, block, 0, s>>>(p, chunk);
        if (op == EQT_OP_SCALE) ew_acc_f4_kernel<EQT_OP_SCALE><<<grid, block, 0, s>>>(p, chunk);
        return check_launch("ew_acc_f4_kernel");
      }
    }
    if (a.accumulated) {
      const int64_t blocks_x = p.num_out * ceil_div(p.c1, 32);
      int64_t chunks = ceil_div((int64_t)sm_count() * 8, blocks_x);
      chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, ceil_div(p.n, 64)));
      chunks = std::min<int64_t>(chunks, 65535);
      const int64_t chunk = ceil_div(p.n, chunks);
      dim3 grid((unsigned)blocks_x, (unsigned)ceil_div(p.n, chunk)), block(32, 8);
      if (op == EQT_OP_MUL) ew_acc_kernel<T, EQT_OP_MUL><<<grid, block, 0, s>>>(p, chunk);
      if (op == EQT_OP_VECSCA) ew_acc_kernel<T, EQT_OP_VECSCA><<<grid, block, 0, s>>>(p, chunk);
      if (op == EQT_OP_SCALE) ew_acc_kernel<T, EQT_OP_SCALE><<<grid, block, 0, s>>>(p, chunk);
      return check_launch("ew_acc_kernel");
    }
    if (std::is_same<T, float>::value && p.c1 % 4 == 0 && aligned16(p.in1) && aligned16(p.out) &&
        (op != EQT_OP_MUL || aligned16(p.in2))) {
      const int64_t items = p.num_out * (p.c1 / 4), blocks_x = ceil_div(items, EW_THREADS);
      const int sets = (int)std::max<int64_t>(1, EW_THREADS / items), step = 4 * sets;        // samples a block takes at a time
      int64_t chunks = std::max<int64_t>(1, std::min<int64_t>(ceil_div((int64_t)sm_count() * 32, blocks_x), ceil_div(p.n, step)));
      chunks = std::min<int64_t>(chunks, 65535);
      const int64_t chunk = ceil_div(ceil_div(p.n, chunks), step) * step;
      if (blocks_x > INT32_MAX) return fail(EQT_ERR_UNSUPPORTED, "too many output rows");
      const dim3 grid((unsigned)blocks_x, (unsigned)ceil_div(p.n, chunk));
      auto run = [&](auto* whole, auto* side) { (sets > 1 ? side : whole)<<<grid, EW_THREADS, 0, s>>>(p, chunk, sets); };
      if (op == EQT_OP_MUL) run(ew_kernel_f4<EQT_OP_MUL, false>, ew_kernel_f4<EQT_OP_MUL, true>);
      if (op == EQT_OP_VECSCA) run(ew_kernel_f4<EQT_OP_VECSCA, false>, ew_kernel_f4<EQT_OP_VECSCA, true>);
      if (op == EQT_OP_SCALE) run(ew_kernel_f4<EQT_OP_SCALE, false>, ew_kernel_f4<EQT_OP_SCALE, true>);
      return check_launch("ew_kernel_f4");
    }
    if (std::is_same<T, __nv_bfloat16>::value && p.c1 % 8 == 0 && aligned16(p.in1) && aligned16(p.out) &&
        (op != EQT_OP_MUL || aligned16(p.in2)) && p.n * p.num_out * (p.c1 / 8) < (int64_t(1) << 31)) {
      const unsigned grid = flat_grid(p.n * p.num_out * (p.c1 / 8), 256);
      if (op == EQT_OP_MUL) ew_kernel_b8<EQT_OP_MUL><<<grid, 256, 0, s>>>(p);
      if (op == EQT_OP_VECSCA) ew_kernel_b8<EQT_OP_VECSCA><<<grid, 256, 0, s>>>(p);
      if (op == EQT_OP_SCALE) ew_kernel_b8<EQT_OP_SCALE><<<grid, 256, 0, s>>>(p);
      return check_launch("ew_kernel_b8");
    }
    const unsigned grid = flat_grid(p.n * p.num_out * p.c1, 256);
    if (op == EQT_OP_MUL) ew_kernel<T, EQT_OP_MUL><<<grid, 256, 0, s>>>(p);
    if (op == EQT_OP_VECSCA) ew_kernel<T, EQT_OP_VECSCA><<<grid, 256, 0, s>>>(p);
    if (op == EQT_OP_SCALE) ew_kernel<T, EQT_OP_SCALE><<<grid, 256, 0, s>>>(p);
    return check_launch("ew_kernel");
  }
  if (op == EQT_OP_OUTER) {
    if (p.c1 == 0 || p.c2 == 0) return EQT_OK;
    if (a.accumulated) {
      const int64_t tiles = ceil_div(p.c1, 64) * ceil_div(p.c2, 64);
      if (p.num_out > 65535) return fail(EQT_ERR_UNSUPPORTED, "accumulated outer: more than 65535 output rows");
      int64_t chunks = ceil_div((int64_t)sm_count() * 4, tiles * p.num_out);
      chunks = std::max<int64_t>(1, std::min<int64_t>(chunks, ceil_div(p.n, 32)));
      chunks = std::min<int64_t>(chunks, 65535);
      if (std::is_same<T, float>::value && p.c1 % 4 == 0 && p.c2 % 4 == 0 && outer_few_wanted(p, tiles) &&
          aligned16(p.in1) && aligned16(p.in2)) {
        const int team = (int)(p.c1 * p.c2 / 16), teams = std::min<int>(16, 256 / team);
        chunks = few_chunks(p.n, teams, chunks, ceil_div((int64_t)sm_count() * 8, p.num_out));
        const int64_t chunk = ceil_div(p.n, chunks);
        outer_acc_few_kernel<<<dim3((unsigned)p.num_out, (unsigned)ceil_div(p.n, chunk)), 256, sizeof(float) * teams * p.c1 * p.c2, s>>>(p, chunk, team, teams);
        return check_launch("outer_acc_few_kernel");
      }
      const int64_t chunk = ceil_div(p.n, chunks);
      dim3 grid((unsigned)tiles, (unsigned)p.num_out, (unsigned)ceil_div(p.n, chunk));
      outer_acc_kernel<T><<<grid, 256, 0, s>>>(p, chunk);
      return check_launch("outer_acc_kernel");
    }
    // lanes own four columns each: 4, 8, ... 128 columns and operands whose rows allow 4-wide accesses; below 32 products a
    // row most lanes would idle (20k samples x 9 rows: 4 x 4 62 us, 34 us a thread per element; 4 x 8 62 and 64; 8 x 8 62 and 122)
    const int64_t q = p.c2 / 4;
    if (p.c2 % 4 == 0 && p.c1 * p.c2 >= 32 && q <= 32 && (q & (q - 1)) == 0 && p.c1 <= 0x7fffff && p.num_out <= 0x7fffffff &&
        ((reinterpret_cast<uintptr_t>(p.in2) | reinterpret_cast<uintptr_t>(p.out)) & (4 * sizeof(T) - 1)) == 0) {
      outer_rows_kernel<T><<<flat_grid(p.n * p.num_out, 8, 8), 256, 0, s>>>(p);
      return check_launch("outer_rows_kernel");
    }
    outer_kernel<T><<<flat_grid(p.n * p.num_out * p.c1 * p.c2, 256), 256, 0, s>>>(p);
    return check_launch("outer_kernel");
  }
  if (op == EQT_OP_INNER) {
    inner_kernel<T><<<flat_grid(p.n * p.num_out, 8), 256, 0, s>>>(p, a.accumulated);
    return check_launch("inner_kernel");
  }
  if (op == EQT_OP_VECMAT) {
    if (p.c2 == 0) return EQT_OK;
    if (std::is_same<T, float>::value && a.shared2 && !a.shared1 && !a.accumulated && (p.c2 == 16 || p.c2 == 32) && p.c1 % 4 == 0 && p.c1 <= 64 &&
        p.num_out * (p.c2 / 16) <= 65535 && aligned16(p.in1) && aligned16(p.out)) {
      const size_t bytes = sizeof(float) * 8 * p.c1 * 16;
      const unsigned rows = (unsigned)(p.num_out * (p.c2 / 16));
      // the more samples a thread the fewer reads of the weights, as long as every SM has two blocks
      const int64_t enough = 2 * (int64_t)sm_count();
      if (ceil_div(p.n, 512) * rows >= enough) vecmat_few_kernel<4><<<dim3((unsigned)ceil_div(p.n, 512), rows), 128, bytes, s>>>(p);
      else if (ceil_div(p.n, 256) * rows >= enough) vecmat_few_kernel<2><<<dim3((unsigned)ceil_div(p.n, 256), rows), 128, bytes, s>>>(p);
      else vecmat_few_kernel<1><<<dim3((unsigned)ceil_div(p.n, 128), rows), 128, bytes, s>>>(p);
      return check_launch("vecmat_few_kernel");
    }
    if (a.shared2 && !a.shared1 && !a.accumulated && p.num_out <= 65535) {
      dim3 grid((unsigned)(ceil_div(p.n, 64) * ceil_div(p.c2, 64)), (unsigned)p.num_out);
      vecmat_shared_w_kernel<T><<<grid, 256, 0, s>>>(p);
      return check_launch("vecmat_shared_w_kernel");
    }
    vecmat_direct_kernel<T><<<flat_grid(p.n * p.num_out * p.c2, 256), 256, 0, s>>>(p, a.accumulated);
    return check_launch("vecmat_direct_kernel");
  }
  return fail(EQT_ERR_BAD_ARGUMENT, "unknown op %d", op);
}

}  // namespace
}  // namespace eqt

extern "C" int eqt_sparse_product(const eqt_product_args* a, void* stream) {
  using namespace eqt;
  if (!a) return fail(EQT_ERR_BAD_ARGUMENT, "args is NULL");
  if (a->n < 0 || a->num_out < 0 || a->out_size < 0 || a->c1 < 0 || a->c2 < 0 || a->rows1 < 0 || a->rows2 < 0)
    return fail(EQT_ERR_BAD_ARGUMENT, "negative size");
  const bool empty = a->n == 0 || a->num_out == 0;
  if (!empty && (!a->in1 || !a->out || (a->op != EQT_OP_SCALE && !a->in2)))
    return fail(EQT_ERR_BAD_ARGUMENT, "NULL operand");
  if (!a->index_out && a->num_out > a->out_size) return fail(EQT_ERR_BAD_ARGUMENT, "more rows than the output has");
  if (!a->seg && !a->gather_index &&
      ((!a->index1 && a->num_out > a->rows1) || (a->op != EQT_OP_SCALE && !a->index2 && a->num_out > a->rows2)))
    return fail(EQT_ERR_BAD_ARGUMENT, "more entries than an operand without an index has rows");
  if (a->op == EQT_OP_SCALE && a->accumulated == 0 && a->shared1)
    return fail(EQT_ERR_BAD_ARGUMENT, "scale-segment needs a batched input");
  P p;
  p.in1 = a->in1; p.in2 = a->in2; p.out = a->out; p.scale = a->scale;
  p.i1 = a->index1; p.i2 = a->index2; p.seg = a->seg; p.gather = a->gather_index; p.iout = a->index_out;
  p.n = a->n; p.rows1 = a->rows1; p.rows2 = a->rows2; p.num_out = a->num_out; p.out_size = a->out_size;
  p.c1 = a->c1; p.c2 = a->c2;
  p.bs1 = a->shared1 ? 0 : a->rows1 * a->c1;
  switch (a->op) {
    case EQT_OP_MUL: case EQT_OP_INNER: p.bs2 = a->rows2 * a->c1; break;
    case EQT_OP_VECSCA: p.bs2 = a->rows2; break;
    case EQT_OP_OUTER: p.bs2 = a->rows2 * a->c2; break;
    case EQT_OP_VECMAT: p.bs2 = a->rows2 * a->c1 * a->c2; break;
    case EQT_OP_SCALE: p.bs2 = 0; break;
    default: return fail(EQT_ERR_BAD_ARGUMENT, "unknown op %d", a->op);
  }
  if (a->shared2) p.bs2 = 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (a->dtype) {
    case EQT_F32: return launch<float>(*a, p, s);
    case EQT_F64: return launch<double>(*a, p, s);
    case EQT_BF16: return launch<__nv_bfloat16>(*a, p, s);
    default: return fail(EQT_ERR_BAD_ARGUMENT, "unknown dtype %d", a->dtype);
  }
}

extern "C" const char* eqt_last_error(void) { return eqt::error_buffer(); }
extern "C" int eqt_version(void) { return 100; }
extern "C" int64_t eqt_launch_count(void) { return eqt::g_launches.load(); }
