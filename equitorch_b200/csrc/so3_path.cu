// Channel-wise tensor product with a channel-less second operand ('uu' SO3Linear), forward and backward in one pass
// each (float32 and bfloat16 storage, float32 arithmetic), for irreps of degree up to 3:
//
//   out[n, M, c] = sum_{t: M_t = M} s_t x[n, M1_t, c] y[n, M2_t] w[(n,) p_t, c]
//   gx [n, i, c] = sum_{t: M1_t = i} s_t g[n, M_t, c] y[n, M2_t] w[(n,) p_t, c]
//   gy [n, j]    = sum_{t: M2_t = j} s_t sum_c g[n, M_t, c] x[n, M1_t, c] w[(n,) p_t, c]
//   gw [(n,) p, c] = sum_{t: p_t = p} (sum_n) s_t g[n, M_t, c] x[n, M1_t, c] y[n, M2_t]
//
// The two-step form writes and reads the intermediate with one row per (M, path), 2.3 (l_max 2) to 6 (l_max 3) times
// the features, five to seven times over forward and backward.  Here a thread owns four channels of one sample and
// walks the paths; the Clebsch-Gordan block of a path is straight-line code on registers, chosen by a switch on its
// degrees that all threads take alike (a loop over table entries of shared memory was 2.5 times slower: every entry is
// a chain of four dependent shared-memory loads, and the columns below leave no more than eight warps per SM to hide
// it).  The forward kernel keeps the output block of an irrep in registers over its paths, the backward kernel the
// blocks of x and gx, so the paths are ordered by output irrep in one and by input irrep in the other.  The blocks of
// the other operand are re-read from the thread's own column of shared memory ([component][thread], conflict-free,
// filled by asynchronous copies); weights stream through a ring of such columns.  Bound: instruction issue (10 FMA-class instructions per CG entry in the backward
// kernel) for shared weights; with per-sample weights their traffic comes close.  20,480 samples, 54 paths, 32 bfloat16
// channels, per-sample weights: 54 us forward (1.9 TB/s) and 112 us backward (1.7 TB/s) where the two-step products took
// 514 us; 1024 samples, 11 paths, 16 float32 channels: 7 + 13 us (41 us).
#include <algorithm>

#include "common.cuh"

namespace eqt {
namespace {

constexpr int V = 4;                              // channels per thread

// P: two values at a time in packed instructions (fma.rn.f32x2).  Fewer instructions, but the scalar operand needs a pair of its own:
// 'uv' backward 279 -> 214 us (before its grid fitted the SMs; 20,011 samples, l_max 3, 64 channels), 'uu' forward 55 -> 52 us (20,480 samples, bfloat16, weights per
// sample); 'uu' backward, which is at its register limit without, 107 -> 114 us, so that one does without.
__device__ __forceinline__ unsigned long long two(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void apart(unsigned long long t, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(t)); }
template <int N, bool P> __device__ __forceinline__ void axpy(float (&o)[N], float s, const float (&x)[N]) {
  if constexpr (P) {
    const unsigned long long k = two(s, s);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      unsigned long long r;
      asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(k), "l"(two(x[i], x[i + 1])), "l"(two(o[i], o[i + 1])));
      apart(r, o[i], o[i + 1]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = fmaf(s, x[i], o[i]);
  }
}
template <int N, bool P> __device__ __forceinline__ float dot(const float (&a)[N], const float (&b)[N]) {
  if constexpr (P) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(two(a[0], a[1])), "l"(two(b[0], b[1])));
#pragma unroll
    for (int i = 2; i < N; i += 2) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(r) : "l"(two(a[i], a[i + 1])), "l"(two(b[i], b[i + 1])));
    float x, y;
    apart(r, x, y);
    return x + y;
  } else {
    float d = a[0] * b[0];
#pragma unroll
    for (int i = 1; i < N; ++i) d = fmaf(a[i], b[i], d);
    return d;
  }
}

#include "generated/path_specs.inc"

struct PathArgs {
  const void* x;            // (n, d1, c)
  const void* y;            // (n, d2)
  const void* w;            // (n, p, c) or (p, c)
  const void* g;            // (n, dout, c), backward only
  void* out;                // forward: (n, dout, c)
  void* gx;                 // backward; NULL = not wanted
  void* gy;
  void* gw;                 // (n, p, c) when the weights are per sample
  float* gw_partial;        // (gridDim.x, p, c) when they are shared
  const eqt_path_block* blocks;
  const eqt_path* paths;
  const int32_t* rows;      // UV_BACKWARD: rows of g in the order of their use
  int64_t n;
  int c, d1, d2, dout, p, num_blocks, num_paths, num_rows;
};

template <typename T> struct Chunk;
template <> struct Chunk<float> { using type = float4; };
template <> struct Chunk<__nv_bfloat16> { using type = uint2; };

template <typename T> __device__ __forceinline__ void load_v(const T* p, float (&v)[V]) {
  const typename Chunk<T>::type t = __ldg(reinterpret_cast<const typename Chunk<T>::type*>(p));
  const T* q = reinterpret_cast<const T*>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = static_cast<float>(q[i]);
}
template <typename T> __device__ __forceinline__ void store_v(T* p, const float (&v)[V]) {
  typename Chunk<T>::type t;
  T* q = reinterpret_cast<T*>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) q[i] = static_cast<T>(v[i]);
  *reinterpret_cast<typename Chunk<T>::type*>(p) = t;
}
// V storage elements of a shared-memory column
template <typename T> __device__ __forceinline__ void lds_v(const T* p, float (&v)[V]) {
  const typename Chunk<T>::type t = *reinterpret_cast<const typename Chunk<T>::type*>(p);
  const T* q = reinterpret_cast<const T*>(&t);
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = static_cast<float>(q[i]);
}
__device__ __forceinline__ void sts_v(float* p, const float (&v)[V]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }

// Asynchronous copy of this thread's V elements; the thread itself reads them after waiting for its own groups, so no
// barrier is involved.
template <typename T> __device__ __forceinline__ void copy_v(T* smem, const T* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
               "n"((int)sizeof(T) * V) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The weights of a sample in path order, AHEAD paths ahead of their use (a path is 60 to 300 instructions, a load from
// HBM over a thousand cycles: with the weights one path ahead the molecular layer spent four fifths of its time on them).
constexpr int AHEAD = 8;
template <typename T>
struct WeightStream {
  T* ring;                  // this thread's column, AHEAD rows
  const T* w;               // the thread's channels of weight 0; NULL: the weights are not wanted, what next() gives is not used
  const eqt_path* paths;
  int row, c, count, at;
  __device__ __forceinline__ void issue(int q) {
    if (q < count && w) copy_v(ring + (q % AHEAD) * row, w + (int64_t)paths[q].weight * c);
    copy_commit();
  }
  // everything committed before begin() - the sample's columns - is complete once the first weights are
  __device__ __forceinline__ void begin() {
    at = 0;
    for (int q = 0; q < AHEAD - 1; ++q) issue(q);
  }
  __device__ __forceinline__ void next(float (&v)[V]) {
    issue(at + AHEAD - 1);
    copy_wait<AHEAD - 1>();
    lds_v(ring + (at % AHEAD) * row, v);
    ++at;
  }
};

// The rows of the node-level gradient G (n, rows, c) of a sample in path order, a fixed number of rows ahead.
constexpr int ROWS_AHEAD = 16;
struct RowStream {
  float* ring;              // this thread's column, ROWS_AHEAD rows
  const float* g;           // the thread's channels of row 0 of its sample
  const int32_t* order;     // rows in the order of their use
  int row, c, count, at;
  __device__ __forceinline__ void issue(int q) {
    if (q < count) copy_v(ring + (q % ROWS_AHEAD) * row, g + (int64_t)order[q] * c);
    copy_commit();
  }
  __device__ __forceinline__ void begin() {
    at = 0;
    for (int q = 0; q < ROWS_AHEAD; ++q) issue(q);
  }
  template <int N> __device__ __forceinline__ void next(float (&v)[N][V]) {
    copy_wait<ROWS_AHEAD - N>();
#pragma unroll
    for (int m = 0; m < N; ++m) lds_v(ring + ((at + m) % ROWS_AHEAD) * row, v[m]);
#pragma unroll
    for (int m = 0; m < N; ++m) issue(at + m + ROWS_AHEAD);
    at += N;
  }
};

enum PathMode { UU_FORWARD, UU_BACKWARD, UV_EXPAND, UV_BACKWARD };

// Shared memory of a kernel; host and kernels agree on the sizes through this one description.
struct PathSmem {
  size_t blocks, paths, rows, ys, xcol, gcol, ring, gycol, gwcol, total;
  __host__ __device__ PathSmem(PathMode mode, bool shared_gw, int elem, int threads, int slots, int d1, int dout, int d2, int p, int num_blocks,
                               int num_paths, int num_rows) {
    const bool backward = mode == UU_BACKWARD || mode == UV_BACKWARD;
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t r = at; at = (at + bytes + 15) & ~size_t(15); return r; };
    const size_t row = (size_t)elem * V * threads;
    blocks = take(sizeof(eqt_path_block) * num_blocks);
    paths = take(sizeof(eqt_path) * num_paths);
    rows = take(mode == UV_BACKWARD ? sizeof(int32_t) * num_rows : 0);
    ys = take(sizeof(float) * slots * d2);
    xcol = take(mode == UV_BACKWARD ? 0 : row * d1);
    gcol = take(mode == UU_BACKWARD ? row * dout : 0);
    ring = take(mode == UV_EXPAND ? 0 : row * (mode == UV_BACKWARD ? ROWS_AHEAD : AHEAD));
    gycol = take(backward ? sizeof(float) * threads * d2 : 0);
    gwcol = take(shared_gw ? sizeof(float) * V * threads * p : 0);
    total = at;
  }
};

// A warp-uniform switch over the two degrees a path adds to the block's own.
#define EQT_PATH_CASES(CASE) \
  CASE(0, 0) CASE(0, 1) CASE(0, 2) CASE(0, 3) CASE(1, 0) CASE(1, 1) CASE(1, 2) CASE(1, 3) \
  CASE(2, 0) CASE(2, 1) CASE(2, 2) CASE(2, 3) CASE(3, 0) CASE(3, 1) CASE(3, 2) CASE(3, 3)
constexpr __host__ __device__ bool is_path(int a, int b, int c) { return a <= b + c && b <= a + c && c <= a + b; }

// o += w * (CG block of x and y): the weight meets the contraction in the addition to o, so that neither x * w nor the
// contraction is rounded a second time (with x * w first the output was at 1.04e-7 of its norm, l_max 3 and 64 channels;
// 7.7e-8 so, and the two-step products 7.5e-8)
template <typename T, int LO, int L1, int L2>
__device__ __forceinline__ void forward_path(float (&o)[2 * LO + 1][V], const T* xc, int row, const float* yr, const float (&w)[V]) {
  if constexpr (is_path(LO, L1, L2)) {
    float x[2 * L1 + 1][V], y[2 * L2 + 1], t[2 * LO + 1][V];
#pragma unroll
    for (int i = 0; i < 2 * L2 + 1; ++i) y[i] = yr[i];
#pragma unroll
    for (int m = 0; m < 2 * L1 + 1; ++m) lds_v(xc + m * row, x[m]);
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m)
#pragma unroll
      for (int i = 0; i < V; ++i) t[m][i] = 0.f;
    CgPath<LO, L1, L2>::template forward<V, true>(t, x, y);
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m)
#pragma unroll
      for (int i = 0; i < V; ++i) o[m][i] = fmaf(t[m][i], w[i], o[m][i]);
  }
}

template <typename T, int LO>
__device__ __forceinline__ void forward_block(const PathArgs& a, const eqt_path_block& b, WeightStream<T>& ws, const T* xc, int row,
                                              const float* yr, T* out) {
  float o[2 * LO + 1][V];
#pragma unroll
  for (int m = 0; m < 2 * LO + 1; ++m)
#pragma unroll
    for (int i = 0; i < V; ++i) o[m][i] = 0.f;
  for (int q = 0; q < b.count; ++q) {
    const eqt_path pd = ws.paths[ws.at];
    float wv[V];
    ws.next(wv);
#pragma unroll
    for (int i = 0; i < V; ++i) wv[i] *= pd.scale;
    const T* xb = xc + pd.offset * row;
    const float* yb = yr + pd.offset_y;
    switch (pd.code) {
#define EQT_CASE(L1, L2) case L1 * 4 + L2: forward_path<T, LO, L1, L2>(o, xb, row, yb, wv); break;
      EQT_PATH_CASES(EQT_CASE)
#undef EQT_CASE
    }
  }
#pragma unroll
  for (int m = 0; m < 2 * LO + 1; ++m) store_v<T>(out + (int64_t)(b.offset + m) * a.c, o[m]);
}

template <typename T>
__global__ void __launch_bounds__(128, 4) so3_uu_forward_kernel(PathArgs a, int per_sample) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, threads = blockDim.x, row = threads * V;
  const int tps = a.c / V, slots = threads / tps, slot = tid / tps, ch = (tid - slot * tps) * V;
  const PathSmem L(UU_FORWARD, false, sizeof(T), threads, slots, a.d1, a.dout, a.d2, a.p, a.num_blocks, a.num_paths, 0);
  eqt_path_block* blocks = reinterpret_cast<eqt_path_block*>(smem + L.blocks);
  eqt_path* paths = reinterpret_cast<eqt_path*>(smem + L.paths);
  float* ys = reinterpret_cast<float*>(smem + L.ys);
  T* xc = reinterpret_cast<T*>(smem + L.xcol) + tid * V;
  WeightStream<T> ws;
  ws.ring = reinterpret_cast<T*>(smem + L.ring) + tid * V;
  ws.row = row; ws.c = a.c;
  for (int i = tid; i < a.num_blocks; i += threads) blocks[i] = a.blocks[i];
  for (int i = tid; i < a.num_paths; i += threads) paths[i] = a.paths[i];
  const T* x = static_cast<const T*>(a.x);
  const T* y = static_cast<const T*>(a.y);
  // few samples: the output irreps (and with them the paths) are dealt to blockIdx.y in contiguous ranges
  const int b0 = a.num_blocks * (int)blockIdx.y / (int)gridDim.y, b1 = a.num_blocks * ((int)blockIdx.y + 1) / (int)gridDim.y;
  for (int64_t n0 = (int64_t)blockIdx.x * slots; n0 < a.n; n0 += (int64_t)gridDim.x * slots) {
    const int here = (int)min((int64_t)slots, a.n - n0);
    const int64_t n = n0 + slot;
    __syncthreads();                                   // tables loaded / the harmonics of the previous samples have been read
    if (slot < here) {
      for (int i = 0; i < a.d1; ++i) copy_v(xc + i * row, x + (n * a.d1 + i) * a.c + ch);
      ws.paths = paths + blocks[b0].first;
      ws.count = blocks[b1 - 1].first + blocks[b1 - 1].count - blocks[b0].first;
      ws.w = static_cast<const T*>(a.w) + (per_sample ? n * a.p * a.c : 0) + ch;
      ws.begin();
    }
    for (int i = tid; i < here * a.d2; i += threads) ys[i] = static_cast<float>(y[n0 * a.d2 + i]);
    __syncthreads();
    if (slot >= here) continue;
    T* out = static_cast<T*>(a.out) + n * a.dout * a.c + ch;
    const float* yr = ys + slot * a.d2;
    for (int b = b0; b < b1; ++b) {
      const eqt_path_block bd = blocks[b];
      switch (bd.l) {
        case 0: forward_block<T, 0>(a, bd, ws, xc, row, yr, out); break;
        case 1: forward_block<T, 1>(a, bd, ws, xc, row, yr, out); break;
        case 2: forward_block<T, 2>(a, bd, ws, xc, row, yr, out); break;
        case 3: forward_block<T, 3>(a, bd, ws, xc, row, yr, out); break;
      }
    }
  }
}

// gy of the CTA's samples from the threads' columns: the threads of a sample hold theirs side by side; the start is
// rotated to spread the banks
template <typename T>
__device__ __forceinline__ void sum_gy(const float* gy_all, T* gy, int64_t n0, int here, int d2, int threads, int tps) {
  for (int i = threadIdx.x; i < here * d2; i += threads) {
    const int sl = i / d2, k = i - sl * d2;
    const float* col = gy_all + k * threads + sl * tps;
    double v = 0.;
    int j = i % tps;
    for (int u = 0; u < tps; ++u) {
      v += col[j];
      if (++j == tps) j = 0;
    }
    gy[n0 * d2 + i] = static_cast<T>(static_cast<float>(v));
  }
}

// gw of the path without its factor, and what the last of its additions rounded off; gx and gyc (column of the thread, one
// float per y component) are added to, gyc once per path: a chain over all entries was at 1.36e-7 of the norm (l_max 3,
// 64 channels), sums per path and the factor in the addition at 8.9e-8, the two-step products at 9.9e-8
template <typename T, int LO, int L1, int L2>
__device__ __forceinline__ void backward_path(float (&gx)[2 * L1 + 1][V], const float (&x)[2 * L1 + 1][V], const T* gc, int row,
                                              const float* yr, float* gyc, int threads, const float (&w)[V], float scale,
                                              float (&gw)[V], float (&lost)[V]) {
  if constexpr (is_path(LO, L1, L2)) {
    float g[2 * LO + 1][V], y[2 * L2 + 1], r[2 * L1 + 1][V], gy[2 * L2 + 1];
#pragma unroll
    for (int i = 0; i < 2 * L2 + 1; ++i) { y[i] = yr[i]; gy[i] = 0.f; }
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m) lds_v(gc + m * row, g[m]);
#pragma unroll
    for (int m = 0; m < 2 * L1 + 1; ++m)
#pragma unroll
      for (int i = 0; i < V; ++i) r[m][i] = 0.f;
    CgPath<LO, L1, L2>::template adjoint<V>(r, g, y);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const float ws = w[i] * scale;
      gw[i] = 0.f;
#pragma unroll
      for (int m = 0; m < 2 * L1 + 1; ++m) {
        const float before = gw[i];
        gx[m][i] = fmaf(r[m][i], ws, gx[m][i]);
        gw[i] = fmaf(r[m][i], x[m][i], before);
        if (m == 2 * L1) lost[i] = fmaf(r[m][i], x[m][i], before - gw[i]);
      }
    }
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m)
#pragma unroll
      for (int i = 0; i < V; ++i) g[m][i] *= w[i];
    CgPath<LO, L1, L2>::template inner<V>(gy, g, x);
#pragma unroll
    for (int i = 0; i < 2 * L2 + 1; ++i) gyc[i * threads] = fmaf(gy[i], scale, gyc[i * threads]);
  }
}

template <typename T, int L1>
__device__ __forceinline__ void backward_block(const PathArgs& a, const eqt_path_block& b, WeightStream<T>& ws, const T* xc, const T* gc,
                                               int row, int threads, const float* yr, float* gyc, T* gxout, T* gw_out, float* gw_col) {
  float x[2 * L1 + 1][V], gx[2 * L1 + 1][V];
#pragma unroll
  for (int m = 0; m < 2 * L1 + 1; ++m) {
    lds_v(xc + (b.offset + m) * row, x[m]);
#pragma unroll
    for (int i = 0; i < V; ++i) gx[m][i] = 0.f;
  }
  for (int q = 0; q < b.count; ++q) {
    const eqt_path pd = ws.paths[ws.at];
    float wv[V], gw[V], lost[V];
    ws.next(wv);
    const T* gb = gc + pd.offset * row;
    switch (pd.code) {
#define EQT_CASE(LO, L2) \
  case LO * 4 + L2: backward_path<T, LO, L1, L2>(gx, x, gb, row, yr + pd.offset_y, gyc + pd.offset_y * threads, threads, wv, pd.scale, gw, lost); break;
      EQT_PATH_CASES(EQT_CASE)
#undef EQT_CASE
    }
    if (gw_col) {
      float v[V];
      lds_v(gw_col + pd.weight * row, v);
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = fmaf(gw[i], pd.scale, v[i]);
      sts_v(gw_col + pd.weight * row, v);
    } else if (gw_out) {
#pragma unroll
      for (int i = 0; i < V; ++i) gw[i] = fmaf(gw[i], pd.scale, lost[i] * pd.scale);
      store_v<T>(gw_out + (int64_t)pd.weight * a.c, gw);
    }
  }
  if (gxout)
#pragma unroll
    for (int m = 0; m < 2 * L1 + 1; ++m) store_v<T>(gxout + (int64_t)(b.offset + m) * a.c, gx[m]);
}

// An operand that none of the wanted gradients takes may be NULL: its columns are then left as they are and reach only
// gradients that are not stored.
template <typename T>
__global__ void __launch_bounds__(128, 3) so3_uu_backward_kernel(PathArgs a, int per_sample) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, threads = blockDim.x, row = threads * V;
  const int tps = a.c / V, slots = threads / tps, slot = tid / tps, ch = (tid - slot * tps) * V;
  const bool shared_gw = a.gw_partial != nullptr;
  const PathSmem L(UU_BACKWARD, shared_gw, sizeof(T), threads, slots, a.d1, a.dout, a.d2, a.p, a.num_blocks, a.num_paths, 0);
  eqt_path_block* blocks = reinterpret_cast<eqt_path_block*>(smem + L.blocks);
  eqt_path* paths = reinterpret_cast<eqt_path*>(smem + L.paths);
  float* ys = reinterpret_cast<float*>(smem + L.ys);
  T* xc = reinterpret_cast<T*>(smem + L.xcol) + tid * V;
  T* gc = reinterpret_cast<T*>(smem + L.gcol) + tid * V;
  float* gy_all = reinterpret_cast<float*>(smem + L.gycol);
  float* gw_all = reinterpret_cast<float*>(smem + L.gwcol);
  WeightStream<T> ws;
  ws.ring = reinterpret_cast<T*>(smem + L.ring) + tid * V;
  ws.paths = paths;
  ws.row = row; ws.c = a.c; ws.count = a.num_paths;
  for (int i = tid; i < a.num_blocks; i += threads) blocks[i] = a.blocks[i];
  for (int i = tid; i < a.num_paths; i += threads) paths[i] = a.paths[i];
  const float zero[V] = {};
  if (shared_gw)
    for (int q = 0; q < a.p; ++q) sts_v(gw_all + tid * V + q * row, zero);
  const T* x = static_cast<const T*>(a.x);
  const T* y = static_cast<const T*>(a.y);
  const T* g = static_cast<const T*>(a.g);
  for (int64_t n0 = (int64_t)blockIdx.x * slots; n0 < a.n; n0 += (int64_t)gridDim.x * slots) {
    const int here = (int)min((int64_t)slots, a.n - n0);
    const int64_t n = n0 + slot;
    __syncthreads();                                   // tables loaded / harmonics and partial gy of the previous samples have been read
    if (slot < here) {
      if (x)
        for (int i = 0; i < a.d1; ++i) copy_v(xc + i * row, x + (n * a.d1 + i) * a.c + ch);
      for (int i = 0; i < a.dout; ++i) copy_v(gc + i * row, g + (n * a.dout + i) * a.c + ch);
      ws.w = a.w ? static_cast<const T*>(a.w) + (per_sample ? n * a.p * a.c : 0) + ch : nullptr;
      ws.begin();
      for (int i = 0; i < a.d2; ++i) gy_all[i * threads + tid] = 0.f;
    }
    if (y)
      for (int i = tid; i < here * a.d2; i += threads) ys[i] = static_cast<float>(y[n0 * a.d2 + i]);
    __syncthreads();
    if (slot < here) {
      T* gx = a.gx ? static_cast<T*>(a.gx) + n * a.d1 * a.c + ch : nullptr;
      T* gw = a.gw ? static_cast<T*>(a.gw) + n * a.p * a.c + ch : nullptr;
      float* gwc = shared_gw ? gw_all + tid * V : nullptr;
      const float* yr = ys + slot * a.d2;
      copy_wait<AHEAD - 2>();                          // x and g: in the first group, with the first weights
      for (int b = 0; b < a.num_blocks; ++b) {
        const eqt_path_block bd = blocks[b];
        switch (bd.l) {
          case 0: backward_block<T, 0>(a, bd, ws, xc, gc, row, threads, yr, gy_all + tid, gx, gw, gwc); break;
          case 1: backward_block<T, 1>(a, bd, ws, xc, gc, row, threads, yr, gy_all + tid, gx, gw, gwc); break;
          case 2: backward_block<T, 2>(a, bd, ws, xc, gc, row, threads, yr, gy_all + tid, gx, gw, gwc); break;
          case 3: backward_block<T, 3>(a, bd, ws, xc, gc, row, threads, yr, gy_all + tid, gx, gw, gwc); break;
        }
      }
    }
    if (a.gy) {
      __syncthreads();
      sum_gy(gy_all, static_cast<T*>(a.gy), n0, here, a.d2, threads, tps);
    }
  }
  if (shared_gw) {
    __syncthreads();
    float* part = a.gw_partial + (int64_t)blockIdx.x * a.p * a.c;
    for (int i = tid; i < a.p * a.c; i += threads) {
      const int q = i / a.c, cc = i - q * a.c;
      const float* col = gw_all + q * row + cc;        // channel cc of slot 0; slots are c floats apart
      double v = 0.;
      for (int sl = 0; sl < slots; ++sl) v += col[sl * a.c];
      part[i] = static_cast<float>(v);
    }
  }
}

// ---- full channel mixing ('uv'): the channel-wise half of the layer ---------------------------------------------------
// S[n, row(p, M), c] = sum_{t: (p_t, M_t) = (p, M)} s_t x[n, M1_t, c] y[n, M2_t]: one row per (output component, path),
// which the GEMM with the C_in x C_out matrices consumes.  Bound: the rows written (6.2 times the features at l_max 3).
template <int LO>
__device__ __forceinline__ void expand_block(const PathArgs& a, const eqt_path_block& b, const eqt_path* paths, const float* xc, int row,
                                             const float* yr, float* out) {
  for (int q = b.first; q < b.first + b.count; ++q) {
    const eqt_path pd = paths[q];
    const float wv[V] = {pd.scale, pd.scale, pd.scale, pd.scale};
    float o[2 * LO + 1][V];
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m)
#pragma unroll
      for (int i = 0; i < V; ++i) o[m][i] = 0.f;
    const float* xb = xc + pd.offset * row;
    const float* yb = yr + pd.offset_y;
    switch (pd.code) {
#define EQT_CASE(L1, L2) case L1 * 4 + L2: forward_path<float, LO, L1, L2>(o, xb, row, yb, wv); break;
      EQT_PATH_CASES(EQT_CASE)
#undef EQT_CASE
    }
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m) store_v<float>(out + (int64_t)(pd.row + m * pd.row_stride) * a.c, o[m]);
  }
}

__global__ void __launch_bounds__(128, 4) so3_uv_expand_kernel(PathArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, threads = blockDim.x, row = threads * V;
  const int tps = a.c / V, slots = threads / tps, slot = tid / tps, ch = (tid - slot * tps) * V;
  const PathSmem L(UV_EXPAND, false, sizeof(float), threads, slots, a.d1, a.dout, a.d2, a.p, a.num_blocks, a.num_paths, 0);
  eqt_path_block* blocks = reinterpret_cast<eqt_path_block*>(smem + L.blocks);
  eqt_path* paths = reinterpret_cast<eqt_path*>(smem + L.paths);
  float* ys = reinterpret_cast<float*>(smem + L.ys);
  float* xc = reinterpret_cast<float*>(smem + L.xcol) + tid * V;
  for (int i = tid; i < a.num_blocks; i += threads) blocks[i] = a.blocks[i];
  for (int i = tid; i < a.num_paths; i += threads) paths[i] = a.paths[i];
  const float* x = static_cast<const float*>(a.x);
  const float* y = static_cast<const float*>(a.y);
  const int b0 = a.num_blocks * (int)blockIdx.y / (int)gridDim.y, b1 = a.num_blocks * ((int)blockIdx.y + 1) / (int)gridDim.y;
  for (int64_t n0 = (int64_t)blockIdx.x * slots; n0 < a.n; n0 += (int64_t)gridDim.x * slots) {
    const int here = (int)min((int64_t)slots, a.n - n0);
    const int64_t n = n0 + slot;
    __syncthreads();
    if (slot < here) {
      for (int i = 0; i < a.d1; ++i) copy_v(xc + i * row, x + (n * a.d1 + i) * a.c + ch);
      copy_commit();
    }
    for (int i = tid; i < here * a.d2; i += threads) ys[i] = y[n0 * a.d2 + i];
    copy_wait<0>();
    __syncthreads();
    if (slot >= here) continue;
    float* out = static_cast<float*>(a.out) + n * a.num_rows * a.c + ch;
    const float* yr = ys + slot * a.d2;
    for (int b = b0; b < b1; ++b) {
      const eqt_path_block bd = blocks[b];
      switch (bd.l) {
        case 0: expand_block<0>(a, bd, paths, xc, row, yr, out); break;
        case 1: expand_block<1>(a, bd, paths, xc, row, yr, out); break;
        case 2: expand_block<2>(a, bd, paths, xc, row, yr, out); break;
        case 3: expand_block<3>(a, bd, paths, xc, row, yr, out); break;
      }
    }
  }
}

// gx[n, M1, c] = sum_t s_t y[n, M2_t] G[n, row_t, c]  and  gy[n, M2] = sum_t s_t <x[n, M1_t], G[n, row_t]>  from one
// pass over G: a row is used by one path, so it goes from memory through the ring into registers once, and neither a
// second intermediate nor a second GEMM is needed for gx.  The straight-line blocks of a layer are more code than the
// instruction caches hold (4 k instructions a sample at l_max 3), and walking through them takes a CTA some 65 k cycles whatever its
// size, most of it waiting for instructions: what counts is the samples in flight.  x is therefore loaded a block at a time instead
// of kept in columns of shared memory, which leaves room for three CTAs: 294 -> 279 us (20,011
// samples, l_max 3, 64 channels); twelve warps in one CTA that keep together: 295 us.  Packed multiply-adds make the walk shorter: 214 us,
// and a grid of exactly the CTAs that fit: 182 us.
template <int LO, int L1, int L2>
__device__ __forceinline__ void uv_backward_path(float (&gx)[2 * L1 + 1][V], const float (&x)[2 * L1 + 1][V], RowStream& rs, const float* yr,
                                                 float* gyc, int threads, float scale) {
  if constexpr (is_path(LO, L1, L2)) {
    float g[2 * LO + 1][V], y[2 * L2 + 1], gy[2 * L2 + 1];
    rs.next<2 * LO + 1>(g);
#pragma unroll
    for (int i = 0; i < 2 * L2 + 1; ++i) { y[i] = yr[i]; gy[i] = 0.f; }
    CgPath<LO, L1, L2>::template inner<V, true>(gy, g, x);
#pragma unroll
    for (int i = 0; i < 2 * L2 + 1; ++i) gyc[i * threads] = fmaf(gy[i], scale, gyc[i * threads]);
#pragma unroll
    for (int m = 0; m < 2 * LO + 1; ++m)
#pragma unroll
      for (int i = 0; i < V; ++i) g[m][i] *= scale;
    CgPath<LO, L1, L2>::template adjoint<V, true>(gx, g, y);
  }
}

template <int L1>
__device__ __forceinline__ void uv_backward_block(const PathArgs& a, const eqt_path_block& b, const eqt_path* paths, RowStream& rs,
                                                  const float* x_from, int threads, const float* yr, float* gyc, float* gxout) {
  float x[2 * L1 + 1][V], gx[2 * L1 + 1][V];
#pragma unroll
  for (int m = 0; m < 2 * L1 + 1; ++m)
#pragma unroll
    for (int i = 0; i < V; ++i) x[m][i] = gx[m][i] = 0.f;
  if (x_from)
#pragma unroll
    for (int m = 0; m < 2 * L1 + 1; ++m) load_v(x_from + (int64_t)(b.offset + m) * a.c, x[m]);
  for (int q = b.first; q < b.first + b.count; ++q) {
    const eqt_path pd = paths[q];
    switch (pd.code) {
#define EQT_CASE(LO, L2) \
  case LO * 4 + L2: uv_backward_path<LO, L1, L2>(gx, x, rs, yr + pd.offset_y, gyc + pd.offset_y * threads, threads, pd.scale); break;
      EQT_PATH_CASES(EQT_CASE)
#undef EQT_CASE
    }
  }
  if (gxout)
#pragma unroll
    for (int m = 0; m < 2 * L1 + 1; ++m) store_v<float>(gxout + (int64_t)(b.offset + m) * a.c, gx[m]);
}

__global__ void __launch_bounds__(128, 3) so3_uv_backward_kernel(PathArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, threads = blockDim.x, row = threads * V;
  const int tps = a.c / V, slots = threads / tps, slot = tid / tps, ch = (tid - slot * tps) * V;
  const PathSmem L(UV_BACKWARD, false, sizeof(float), threads, slots, a.d1, a.dout, a.d2, a.p, a.num_blocks, a.num_paths, a.num_rows);
  eqt_path_block* blocks = reinterpret_cast<eqt_path_block*>(smem + L.blocks);
  eqt_path* paths = reinterpret_cast<eqt_path*>(smem + L.paths);
  int32_t* rows = reinterpret_cast<int32_t*>(smem + L.rows);
  float* ys = reinterpret_cast<float*>(smem + L.ys);
  float* gy_all = reinterpret_cast<float*>(smem + L.gycol);
  RowStream rs;
  rs.ring = reinterpret_cast<float*>(smem + L.ring) + tid * V;
  rs.order = rows;
  rs.row = row; rs.c = a.c; rs.count = a.num_rows;
  for (int i = tid; i < a.num_blocks; i += threads) blocks[i] = a.blocks[i];
  for (int i = tid; i < a.num_paths; i += threads) paths[i] = a.paths[i];
  for (int i = tid; i < a.num_rows; i += threads) rows[i] = a.rows[i];
  const float* x = static_cast<const float*>(a.x);
  const float* y = static_cast<const float*>(a.y);
  for (int64_t n0 = (int64_t)blockIdx.x * slots; n0 < a.n; n0 += (int64_t)gridDim.x * slots) {
    const int here = (int)min((int64_t)slots, a.n - n0);
    const int64_t n = n0 + slot;
    __syncthreads();                                   // tables loaded / harmonics and partial gy of the previous samples have been read
    if (slot < here) {
      rs.g = static_cast<const float*>(a.g) + n * a.num_rows * a.c + ch;
      rs.begin();
      for (int i = 0; i < a.d2; ++i) gy_all[i * threads + tid] = 0.f;
    }
    if (y)
      for (int i = tid; i < here * a.d2; i += threads) ys[i] = y[n0 * a.d2 + i];
    __syncthreads();
    if (slot < here) {
      float* gx = a.gx ? static_cast<float*>(a.gx) + n * a.d1 * a.c + ch : nullptr;
      const float* xn = x ? x + n * a.d1 * a.c + ch : nullptr;
      const float* yr = ys + slot * a.d2;
      for (int b = 0; b < a.num_blocks; ++b) {
        const eqt_path_block bd = blocks[b];
        switch (bd.l) {
          case 0: uv_backward_block<0>(a, bd, paths, rs, xn, threads, yr, gy_all + tid, gx); break;
          case 1: uv_backward_block<1>(a, bd, paths, rs, xn, threads, yr, gy_all + tid, gx); break;
          case 2: uv_backward_block<2>(a, bd, paths, rs, xn, threads, yr, gy_all + tid, gx); break;
          case 3: uv_backward_block<3>(a, bd, paths, rs, xn, threads, yr, gy_all + tid, gx); break;
        }
      }
    }
    if (a.gy) {
      __syncthreads();
      sum_gy(gy_all, static_cast<float*>(a.gy), n0, here, a.d2, threads, tps);
    }
  }
}

// out[i] = sum_b partial[b, i] in a fixed order: eight row lanes per block, then their sums in order
template <typename T>
__global__ void __launch_bounds__(256) so3_uu_reduce_kernel(const float* __restrict__ partial, T* __restrict__ out, int blocks, int count) {
  __shared__ double red[8][33];
  const int i = blockIdx.x * 32 + threadIdx.x;
  double v = 0.;
  if (i < count) {
#pragma unroll 4
    for (int b = threadIdx.y; b < blocks; b += 8) v += __ldg(partial + (int64_t)b * count + i);
  }
  red[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.y == 0 && i < count) {
#pragma unroll
    for (int k = 1; k < 8; ++k) v += red[k][threadIdx.x];
    out[i] = static_cast<T>(static_cast<float>(v));
  }
}

constexpr size_t PATH_SMEM_MAX = 220 * 1024;

struct PathShape { int threads, slots, grid, split; size_t smem; };

// 128 threads; fewer while that leaves SMs without a CTA (a sample's threads stay in one CTA)
bool path_shape(PathMode mode, bool shared_gw, int64_t n, int c, int dtype, const eqt_path_table* t, PathShape* s) {
  if (c < V || c % V || c / V > 128) return false;
  const bool backward = mode == UU_BACKWARD || mode == UV_BACKWARD;
  int threads = 128;
  while (threads > 32 && threads / 2 >= c / V && ceil_div(n, threads / (c / V)) < sm_count()) threads /= 2;
  for (; threads >= c / V && threads >= 32; threads /= 2) {
    const int slots = threads / (c / V);
    const PathSmem L(mode, shared_gw, dtype == EQT_F32 ? 4 : 2, threads, slots, t->d1, t->d_out, t->d2, t->num_weights,
                     backward ? t->num_bwd_blocks : t->num_fwd_blocks, t->num_paths, t->num_rows);
    if (L.total > PATH_SMEM_MAX) continue;
    // the gradients of the 'uv' rows take registers for three CTAs an SM: a grid of four leaves a quarter of them to a round of their
    // own, and every walk costs the same (20,011 samples, 64 channels, four -> three: l_max 3 214 -> 182 us, l_max 2 90 -> 74, l_max 1 38 -> 29)
    const int fit = (mode == UV_BACKWARD ? 384 : 512) / threads;
    const int per_sm = std::max<int>(1, std::min<int>(fit, (int)(PATH_SMEM_MAX / (L.total + 1024))));
    s->threads = threads; s->slots = slots; s->smem = L.total;
    s->grid = (int)std::min<int64_t>(ceil_div(n, slots), (int64_t)sm_count() * per_sm);
    s->split = backward ? 1 : std::max(1, std::min(t->num_fwd_blocks, sm_count() / std::max(1, s->grid)));
    return true;
  }
  return false;
}

int path_run(PathMode mode, const eqt_path_table* t, bool per_sample_w, bool shared_gw, int64_t n, int c, int dtype, PathArgs a,
             cudaStream_t st, int* grid) {
  a.n = n; a.c = c; a.d1 = t->d1; a.d2 = t->d2; a.dout = t->d_out; a.p = t->num_weights; a.num_paths = t->num_paths;
  a.rows = t->bwd_rows; a.num_rows = t->num_rows;
  const bool backward = mode == UU_BACKWARD || mode == UV_BACKWARD;
  a.num_blocks = backward ? t->num_bwd_blocks : t->num_fwd_blocks;
  a.blocks = backward ? t->bwd_blocks : t->fwd_blocks;
  a.paths = backward ? t->bwd_paths : t->fwd_paths;
  PathShape s;
  if (!path_shape(mode, shared_gw, n, c, dtype, t, &s))
    return fail(EQT_ERR_UNSUPPORTED, "paths and columns of %d channels do not fit shared memory", c);
  if (grid) *grid = s.grid;
  const uintptr_t mask = (uintptr_t)(V * (dtype == EQT_F32 ? 4 : 2)) - 1;
  if (((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.g) |
        reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.gx) | reinterpret_cast<uintptr_t>(a.gw)) & mask) != 0)
    return fail(EQT_ERR_UNSUPPORTED, "operands are not aligned to four elements");
  auto launch = [&](auto kern, auto... more) {
    if (s.smem > 48 * 1024)
      if (int rc = allow_shared(kern, PATH_SMEM_MAX)) return rc;
    kern<<<dim3((unsigned)s.grid, (unsigned)s.split), s.threads, s.smem, st>>>(a, more...);
    return check_launch("so3 path kernel");
  };
  const int per_sample = per_sample_w;
  switch (mode) {
    case UU_FORWARD: return dtype == EQT_F32 ? launch(so3_uu_forward_kernel<float>, per_sample) : launch(so3_uu_forward_kernel<__nv_bfloat16>, per_sample);
    case UU_BACKWARD: return dtype == EQT_F32 ? launch(so3_uu_backward_kernel<float>, per_sample) : launch(so3_uu_backward_kernel<__nv_bfloat16>, per_sample);
    case UV_EXPAND: return launch(so3_uv_expand_kernel);
    default: return launch(so3_uv_backward_kernel);
  }
}

int path_check(const eqt_path_table* t, int64_t n, int c, int dtype) {
  if (!t || !t->fwd_blocks || !t->bwd_blocks || !t->fwd_paths || !t->bwd_paths || !t->bwd_rows) return fail(EQT_ERR_BAD_ARGUMENT, "incomplete table");
  if (n < 0 || c <= 0 || t->d1 <= 0 || t->d2 <= 0 || t->d_out <= 0 || t->num_weights <= 0 || t->num_paths < 0 ||
      t->num_fwd_blocks < 0 || t->num_bwd_blocks < 0 || t->num_rows < 0)
    return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (dtype != EQT_F32 && dtype != EQT_BF16) return fail(EQT_ERR_UNSUPPORTED, "float32 or bfloat16 only");
  return EQT_OK;
}

}  // namespace
}  // namespace eqt

extern "C" int64_t eqt_so3_uu_scratch_floats(const eqt_path_table* table, int64_t n, int32_t channels, int32_t per_sample_weight, int32_t dtype) {
  using namespace eqt;
  if (!table || n < 0 || channels <= 0) return -1;
  PathShape s;
  if (!path_shape(UU_FORWARD, false, n, channels, dtype, table, &s) || !path_shape(UU_BACKWARD, !per_sample_weight, n, channels, dtype, table, &s)) return -1;
  return per_sample_weight ? 0 : (int64_t)s.grid * table->num_weights * channels;
}

extern "C" int eqt_so3_uu_forward(const eqt_path_table* table, const void* x, const void* y, const void* w, void* out, int64_t n,
                                  int32_t channels, int32_t per_sample_weight, int32_t dtype, void* stream) {
  using namespace eqt;
  if (int rc = path_check(table, n, channels, dtype)) return rc;
  if (n == 0) return EQT_OK;
  if (!x || !y || !w || !out) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  PathArgs a{};
  a.x = x; a.y = y; a.w = w; a.out = out;
  return path_run(UU_FORWARD, table, per_sample_weight != 0, false, n, channels, dtype, a, static_cast<cudaStream_t>(stream), nullptr);
}

extern "C" int eqt_so3_uu_backward(const eqt_path_table* table, const void* x, const void* y, const void* w, const void* g, void* gx,
                                   void* gy, void* gw, float* scratch, int64_t scratch_floats, int64_t n, int32_t channels,
                                   int32_t per_sample_weight, int32_t dtype, void* stream) {
  using namespace eqt;
  if (int rc = path_check(table, n, channels, dtype)) return rc;
  if (n == 0) return EQT_OK;
  if (!g || (gx && (!y || !w)) || (gy && (!x || !w)) || (gw && (!x || !y))) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  const bool shared_gw = gw && !per_sample_weight;
  if (shared_gw) {
    const int64_t need = eqt_so3_uu_scratch_floats(table, n, channels, 0, dtype);
    if (need < 0) return fail(EQT_ERR_UNSUPPORTED, "paths and columns of %d channels do not fit shared memory", (int)channels);
    if (!scratch || scratch_floats < need) return fail(EQT_ERR_BAD_ARGUMENT, "scratch too small: %lld floats needed", (long long)need);
  }
  PathArgs a{};
  a.x = x; a.y = y; a.w = w; a.g = g; a.gx = gx; a.gy = gy;
  a.gw = shared_gw ? nullptr : gw;
  a.gw_partial = shared_gw ? scratch : nullptr;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int blocks = 0;
  if (int rc = path_run(UU_BACKWARD, table, per_sample_weight != 0, shared_gw, n, channels, dtype, a, st, &blocks)) return rc;
  if (!shared_gw) return EQT_OK;
  const int count = table->num_weights * channels;
  const unsigned grid = (unsigned)ceil_div(count, 32);
  if (dtype == EQT_F32)
    so3_uu_reduce_kernel<float><<<grid, dim3(32, 8), 0, st>>>(scratch, static_cast<float*>(gw), blocks, count);
  else
    so3_uu_reduce_kernel<__nv_bfloat16><<<grid, dim3(32, 8), 0, st>>>(scratch, static_cast<__nv_bfloat16*>(gw), blocks, count);
  return check_launch("so3_uu_reduce_kernel");
}

extern "C" int eqt_so3_uv_supported(const eqt_path_table* table, int32_t channels) {
  using namespace eqt;
  PathShape s;
  return table && channels > 0 && path_shape(UV_EXPAND, false, 1 << 30, channels, EQT_F32, table, &s) &&
         path_shape(UV_BACKWARD, false, 1 << 30, channels, EQT_F32, table, &s);
}

extern "C" int eqt_so3_uv_expand(const eqt_path_table* table, const float* x, const float* y, float* rows, int64_t n, int32_t channels,
                                 void* stream) {
  using namespace eqt;
  if (int rc = path_check(table, n, channels, EQT_F32)) return rc;
  if (n == 0) return EQT_OK;
  if (!x || !y || !rows) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  PathArgs a{};
  a.x = x; a.y = y; a.out = rows;
  return path_run(UV_EXPAND, table, false, false, n, channels, EQT_F32, a, static_cast<cudaStream_t>(stream), nullptr);
}

extern "C" int eqt_so3_uv_backward(const eqt_path_table* table, const float* x, const float* y, const float* grad_rows, float* gx, float* gy,
                                   int64_t n, int32_t channels, void* stream) {
  using namespace eqt;
  if (int rc = path_check(table, n, channels, EQT_F32)) return rc;
  if (n == 0) return EQT_OK;
  if (!grad_rows || (gx && !y) || (gy && !x)) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  PathArgs a{};
  a.x = x; a.y = y; a.g = grad_rows; a.gx = gx; a.gy = gy;
  return path_run(UV_BACKWARD, table, false, false, n, channels, EQT_F32, a, static_cast<cudaStream_t>(stream), nullptr);
}
