// Block-diagonal Wigner-D matrices, float32: generation, gradient of the angles, rotation of features and gradient of the
// matrix.  Only the diagonal blocks carry arithmetic (455 of 2401 entries for l = 0..6); what bounds all four is HBM, and
// the work per sample is arranged so that few instructions stand between its loads and stores.
//
// Generation.  d(beta) = J Z(beta) J is a rotation about y, which commutes with the reflection y -> -y; the components with
// m < 0 are odd under it and those with m >= 0 even, so d[a][b] = 0 unless a and b are on the same side.  The four entries
// (+-p, +-q) of D (p, q >= 0: a quad) therefore need two values of d only,
//   u = d[p][q], v = d[-p][-q]:   D[ p][q] = cp cq u - sp sq v     D[ p][-q] = -cp sq u - sp cq v
//                                 D[-p][q] = sp cq u + cp sq v     D[-p][-q] = -sp sq u + cp cq v
// with cp, sp = cos, sin(p alpha) and cq, sq = cos, sin(q gamma).  A thread owns a quad of the block structure for the whole
// launch: the coefficients of u and v stay in registers, and a sample costs it 2 (l + 1) sines and cosines of beta from shared
// memory and about 4 (l + 1) + 12 multiply-adds.
#include "wigner_blocks.cuh"

#include <algorithm>

namespace eqt {
namespace {

constexpr int WQ_MAX_THREADS = 512;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async4(void* s, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async16(void* s, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// The image of a group of samples leaves shared memory as one bulk copy where address and size are multiples of 16 bytes
// (every whole group: it holds a multiple of four samples), else as ordinary stores.  Called by all threads of the block
// after they wrote the image; image_release before the image is written again.
__device__ __forceinline__ void image_store(float* dst, const float* img, int64_t floats) {
  const bool bulk = ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) && ((floats & 3) == 0);
  if (bulk) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  if (!bulk) {
    for (int64_t i = threadIdx.x; i < floats; i += blockDim.x) dst[i] = img[i];
  } else if (threadIdx.x == 0) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_addr(img)),
                 "r"((uint32_t)(floats * 4)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}
__device__ __forceinline__ void image_release() {      // followed by a barrier at the caller
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

struct Quads {
  const float* coef;
  const int32_t* blocks;
  const float* angle[3];
  float* d;            // forward: out; backward: grad_d
  float* grad[3];
  int64_t n;
  int dim, num_blocks, quads, group_threads, samples;   // threads per sample (quads rounded up to warps), samples per pass
};

template <int L1>
struct Quad {
  float ua[L1], ub[L1], va[L1], vb[L1];     // coefficients of cos(k beta), sin(k beta) in u and v
  int p, q, l, start;                       // l < 0: this thread has no quad
  __device__ void load(const Quads& a, int index) {
    l = -1;
    p = q = start = 0;
    int off = 0;
    for (int b = 0; b < a.num_blocks; ++b) {
      const int bl = __ldg(a.blocks + 3 * b + 1), count = (bl + 1) * (bl + 1);
      if (index < count) {
        start = __ldg(a.blocks + 3 * b);
        l = bl;
        off = __ldg(a.blocks + 3 * b + 2);
        p = index / (bl + 1);
        q = index - p * (bl + 1);
        break;
      }
      index -= count;
    }
    const int n = 2 * l + 1;
#pragma unroll
    for (int k = 0; k < L1; ++k) {
      ua[k] = ub[k] = va[k] = vb[k] = 0.f;
      if (k <= l) {
        const float* c = a.coef + off + k * n * n * 2;
        ua[k] = __ldg(c + ((p + l) * n + q + l) * 2);
        ub[k] = __ldg(c + ((p + l) * n + q + l) * 2 + 1);
        if (p > 0 && q > 0) {
          va[k] = __ldg(c + ((l - p) * n + l - q) * 2);
          vb[k] = __ldg(c + ((l - p) * n + l - q) * 2 + 1);
        }
      }
    }
  }
};

// trig[s][which][k] = (cos, sin)(k * angle), which = alpha, beta, gamma; the product is formed in float32 as the general
// kernel and the reference do
template <int L1>
__device__ __forceinline__ void fill_trig(const Quads& a, float2* trig, int64_t s0, int ns) {
  for (int i = threadIdx.x; i < ns * 3 * L1; i += blockDim.x) {
    const int s = i / (3 * L1), r = i - s * 3 * L1, which = r / L1, k = r - which * L1;
    float sn, cs;
    sincosf(__ldg(a.angle[which] + s0 + s) * (float)k, &sn, &cs);
    trig[i] = make_float2(cs, sn);
  }
}

// 100k samples of l = 0..6: 1255 us as one evaluation of d at four positions per entry, with the coefficients read from
// shared memory for each of them; 171 us so (5.7 TB/s written).
template <int L1>
__global__ void __launch_bounds__(WQ_MAX_THREADS) wigner_quads_forward_kernel(Quads a) {
  extern __shared__ __align__(16) float sm[];
  const int dd = a.dim * a.dim;
  float* img = sm;                                                        // [samples][dim][dim]
  float2* trig = reinterpret_cast<float2*>(img + a.samples * dd);         // samples is a multiple of 4: 16-byte aligned
  const int group = threadIdx.x / a.group_threads, groups = blockDim.x / a.group_threads;
  Quad<L1> quad;
  quad.load(a, threadIdx.x - group * a.group_threads);
  for (int i = threadIdx.x; i < a.samples * dd; i += blockDim.x) img[i] = 0.f;
  const int r1 = (quad.start + quad.l + quad.p) * a.dim, r0 = (quad.start + quad.l - quad.p) * a.dim;
  const int c1 = quad.start + quad.l + quad.q, c0 = quad.start + quad.l - quad.q;
  for (int64_t s0 = (int64_t)blockIdx.x * a.samples; s0 < a.n; s0 += (int64_t)gridDim.x * a.samples) {
    const int ns = (int)min((int64_t)a.samples, a.n - s0);
    image_release();
    __syncthreads();
    fill_trig<L1>(a, trig, s0, ns);
    __syncthreads();
    if (quad.l >= 0) {
      for (int s = group; s < ns; s += groups) {
        const float2* t = trig + s * 3 * L1;
        float u = 0.f, v = 0.f;
#pragma unroll
        for (int k = 0; k < L1; ++k) {
          const float2 b = t[L1 + k];
          u = fmaf(quad.ua[k], b.x, fmaf(quad.ub[k], b.y, u));
          v = fmaf(quad.va[k], b.x, fmaf(quad.vb[k], b.y, v));
        }
        const float2 pa = t[quad.p], qg = t[2 * L1 + quad.q];
        const float uc = u * qg.x, us = u * qg.y, vc = v * qg.x, vs = v * qg.y;
        float* o = img + s * dd;
        o[r1 + c1] = pa.x * uc - pa.y * vs;
        if (quad.q > 0) o[r1 + c0] = -pa.x * us - pa.y * vc;
        if (quad.p > 0) o[r0 + c1] = pa.y * uc + pa.x * vs;
        if (quad.p > 0 && quad.q > 0) o[r0 + c0] = pa.x * vc - pa.y * us;
      }
    }
    image_store(a.d + s0 * dd, img, (int64_t)ns * dd);
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// The transposed product per quad: with g the entries of grad_d at the four positions,
//   x = cp g[p][q] + sp g[-p][q]      y = cp g[p][-q] + sp g[-p][-q]
//   w = cp g[-p][q] - sp g[p][q]      z = cp g[-p][-q] - sp g[p][-q]
//   beta:  u' (x cq - y sq) + v' (w sq + z cq)
//   gamma: q (v (w cq - z sq) - u (x sq + y cq))      alpha: p (u (w cq - z sq) - v (x sq + y cq))
// 1130 us with four evaluations of d and of its derivative per entry; 224 us so.
template <int L1>
__global__ void __launch_bounds__(WQ_MAX_THREADS) wigner_quads_backward_kernel(Quads a) {
  extern __shared__ __align__(16) float sm[];
  const int dd = a.dim * a.dim, warps = a.group_threads / 32;
  float2* trig = reinterpret_cast<float2*>(sm);
  float* part = reinterpret_cast<float*>(trig + a.samples * 3 * L1);      // [samples][warps][3]
  const int group = threadIdx.x / a.group_threads, groups = blockDim.x / a.group_threads;
  const int in_group = threadIdx.x - group * a.group_threads, lane = threadIdx.x & 31;
  Quad<L1> quad;
  quad.load(a, in_group);
  const int r1 = (quad.start + quad.l + quad.p) * a.dim, r0 = (quad.start + quad.l - quad.p) * a.dim;
  const int c1 = quad.start + quad.l + quad.q, c0 = quad.start + quad.l - quad.q;
  for (int64_t s0 = (int64_t)blockIdx.x * a.samples; s0 < a.n; s0 += (int64_t)gridDim.x * a.samples) {
    const int ns = (int)min((int64_t)a.samples, a.n - s0);
    __syncthreads();
    fill_trig<L1>(a, trig, s0, ns);
    __syncthreads();
    // two samples at a time: eight loads in flight per thread
    for (int s = group; s < ns; s += 2 * groups) {
      float g[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool on = quad.l >= 0 && s + h * groups < ns;
        const float* gd = a.d + (s0 + s + h * groups) * dd;
        g[h][0] = on ? __ldg(gd + r1 + c1) : 0.f;
        g[h][1] = on && quad.q > 0 ? __ldg(gd + r1 + c0) : 0.f;
        g[h][2] = on && quad.p > 0 ? __ldg(gd + r0 + c1) : 0.f;
        g[h][3] = on && quad.p > 0 && quad.q > 0 ? __ldg(gd + r0 + c0) : 0.f;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int at = s + h * groups;
        if (at >= ns) break;                                              // the same for all threads of the group
        const float2* t = trig + at * 3 * L1;
        float u = 0.f, v = 0.f, du = 0.f, dv = 0.f;
#pragma unroll
        for (int k = 0; k < L1; ++k) {
          const float2 b = t[L1 + k];
          u = fmaf(quad.ua[k], b.x, fmaf(quad.ub[k], b.y, u));
          v = fmaf(quad.va[k], b.x, fmaf(quad.vb[k], b.y, v));
          du = fmaf((float)k, quad.ub[k] * b.x - quad.ua[k] * b.y, du);
          dv = fmaf((float)k, quad.vb[k] * b.x - quad.va[k] * b.y, dv);
        }
        const float2 pa = t[quad.p], qg = t[2 * L1 + quad.q];
        const float x = pa.x * g[h][0] + pa.y * g[h][2], y = pa.x * g[h][1] + pa.y * g[h][3];
        const float w = pa.x * g[h][2] - pa.y * g[h][0], z = pa.x * g[h][3] - pa.y * g[h][1];
        const float even = w * qg.x - z * qg.y, odd = x * qg.y + y * qg.x;
        float sum[3] = {(float)quad.p * (u * even - v * odd), du * (x * qg.x - y * qg.y) + dv * (w * qg.y + z * qg.x),
                        (float)quad.q * (v * even - u * odd)};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int i = 0; i < 3; ++i) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
        if (lane < 3) part[(at * warps + in_group / 32) * 3 + lane] = lane == 0 ? sum[0] : lane == 1 ? sum[1] : sum[2];
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ns * 3; i += blockDim.x) {
      const int s = i / 3, which = i - 3 * s;
      float sum = 0.f;
      for (int w = 0; w < warps; ++w) sum += part[(s * warps + w) * 3 + which];
      a.grad[which][s0 + s] = sum;
    }
  }
}

// ---- rotation of features --------------------------------------------------------------------------------------------
constexpr int BR_MAX_DIM = 128;

// Groups of up to four rows of one block.
struct RowTiles {
  int count, floats;                        // tiles, shared floats of one sample's matrix
  uint8_t row[BR_MAX_DIM], rows[BR_MAX_DIM], lo[BR_MAX_DIM], len[BR_MAX_DIM];
  uint16_t at[BR_MAX_DIM], first[BR_MAX_DIM + 1];   // first shared float; first entry in the list of block entries
};

// Two float32 values multiplied and added by one instruction (fma.rn.f32x2), each rounded as fmaf rounds it.
__device__ __forceinline__ void pair_fma(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r.x + r.y;
}
__device__ __forceinline__ uint64_t pair_of(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

// out[n, i, c] = sum_j M[n, i, j] x[n, j, c] (transposed: M[n, j, i]) over the block of row i.  A thread makes four rows of
// four channels: per contraction step one 16-byte load of features, one of four matrix entries (laid out [tile][j][row]) and
// 16 multiply-adds.  The entries of the blocks are copied by a list made once per launch (a shared-memory pair of offsets per
// entry) instead of row by row with mostly idle lanes, and the next samples are copied while these are multiplied.
// 100k samples of l = 0..6, 32 channels: 654 -> 350 us (4.1 TB/s).
constexpr int BR_THREADS = 256;
__global__ void __launch_bounds__(BR_THREADS) block_rotation_kernel(const float* __restrict__ mat, const float* __restrict__ x,
                                                                    float* __restrict__ out, int64_t n, int dim, int c, int transposed,
                                                                    int samples, const __grid_constant__ RowTiles given) {
  extern __shared__ __align__(16) float sm[];
  __shared__ RowTiles tiles;                                         // indexed by lane
  static_assert(sizeof(RowTiles) % 4 == 0 && sizeof(RowTiles) / 4 > BR_THREADS, "copied by words, more of them than threads");
  for (int i = threadIdx.x; i < (int)(sizeof(RowTiles) / 4); i += blockDim.x) reinterpret_cast<uint32_t*>(&tiles)[i] = reinterpret_cast<const uint32_t*>(&given)[i];
  __syncthreads();
  const int mat_room = tiles.floats, list_room = (tiles.first[tiles.count] + 3) & ~3;
  uint32_t* list = reinterpret_cast<uint32_t*>(sm);                  // (offset in the matrix << 16) | offset in shared memory
  const int sample_floats = mat_room + dim * c;
  float* stage = sm + list_room;                                     // [2][samples][mat_room + dim * c]
  for (int t = threadIdx.x; t < tiles.count; t += blockDim.x)
    for (int u = 0, k = tiles.first[t]; u < tiles.rows[t]; ++u)
      for (int j = 0; j < tiles.len[t]; ++j, ++k) {
        const int r = tiles.row[t] + u, q = tiles.lo[t] + j;
        list[k] = (uint32_t)(transposed ? q * dim + r : r * dim + q) << 16 | (uint32_t)(tiles.at[t] + j * 4 + u);
      }
  for (int i = threadIdx.x; i < 2 * samples * sample_floats; i += blockDim.x) stage[i] = 0.f;   // rows a tile does not have stay 0
  __syncthreads();
  const int entries = tiles.first[tiles.count], quads = dim * c / 4, cg = c / 4, items = tiles.count * cg;
  const int64_t step = (int64_t)gridDim.x * samples;
  auto fetch = [&](int64_t s0, int buf) {
    const int ns = (int)min((int64_t)samples, n - s0);
    for (int s = 0; s < ns; ++s) {
      float* to = stage + (buf * samples + s) * sample_floats;
      const float* m = mat + (s0 + s) * dim * dim;
      const float* xs = x + (s0 + s) * dim * c;
      for (int i = threadIdx.x; i < entries; i += blockDim.x) {
        const uint32_t e = list[i];
        cp_async4(to + (e & 0xffffu), m + (e >> 16));
      }
      for (int i = threadIdx.x; i < quads; i += blockDim.x) cp_async16(to + mat_room + 4 * i, xs + 4 * i);
    }
  };
  int64_t s0 = (int64_t)blockIdx.x * samples;
  if (s0 < n) fetch(s0, 0);
  cp_async_commit();
  for (int buf = 0; s0 < n; s0 += step, buf ^= 1) {
    if (s0 + step < n) fetch(s0 + step, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const int ns = (int)min((int64_t)samples, n - s0);
    for (int i = threadIdx.x; i < ns * items; i += blockDim.x) {
      const int s = i / items, r = i - s * items, t = r / cg, ch = (r - t * cg) * 4;
      const float* from = stage + (buf * samples + s) * sample_floats;
      const float4* mp = reinterpret_cast<const float4*>(from + tiles.at[t]);
      const float* xp = from + mat_room + tiles.lo[t] * c + ch;
      const int len = tiles.len[t], rows = tiles.rows[t];
      float acc[4][4] = {};
#pragma unroll 2
      for (int j = 0; j < len; ++j) {
        const float4 mv = mp[j], xv = *reinterpret_cast<const float4*>(xp + j * c);
        const float ma[4] = {mv.x, mv.y, mv.z, mv.w}, xa[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w = 0; w < 4; ++w) acc[u][w] = fmaf(ma[u], xa[w], acc[u][w]);
      }
      float* o = out + ((s0 + s) * dim + tiles.row[t]) * c + ch;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (u < rows) *reinterpret_cast<float4*>(o + u * c) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
    }
    __syncthreads();
  }
}

// The same product with the whole matrices copied, as one run per pass that begins at any float: where the blocks touch most
// of the matrix's cache lines anyway, that costs no traffic and takes the list away.  A thread makes four rows of V times
// four channels and keeps its tile and channels for the whole launch.
template <int V>
__global__ void __launch_bounds__(BR_THREADS) block_rotation_whole_kernel(const float* __restrict__ mat, const float* __restrict__ x,
                                                                          float* __restrict__ out, int64_t n, int dim, int c,
                                                                          int transposed, int samples,
                                                                          const __grid_constant__ RowTiles tiles) {
  extern __shared__ __align__(16) float sm[];                        // [2][3 + samples * dim * dim | samples * dim * c]
  const int dd = dim * dim, features = dim * c, mat_room = (samples * dd + 6) & ~3, buffer = mat_room + samples * features;
  const int cg = c / (4 * V), items = tiles.count * cg, sample = threadIdx.x / items, first = threadIdx.x - sample * items;
  const int64_t step = (int64_t)gridDim.x * samples;
  auto shift_of = [&](int64_t s0) { return (int)(reinterpret_cast<uintptr_t>(mat + s0 * dd) >> 2 & 3); };   // same place in 16 bytes
  auto fetch = [&](int64_t s0, int buf) {
    const int ns = (int)min((int64_t)samples, n - s0), floats = ns * dd, shift = shift_of(s0), head = min((4 - shift) & 3, floats);
    const int tail = head + ((floats - head) & ~3);
    const float* from = mat + s0 * dd;
    float* to = sm + buf * buffer;
    if ((int)threadIdx.x < head) cp_async4(to + shift + threadIdx.x, from + threadIdx.x);
    if ((int)threadIdx.x < floats - tail) cp_async4(to + shift + tail + threadIdx.x, from + tail + threadIdx.x);
    for (int i = head + 4 * threadIdx.x; i < tail; i += 4 * blockDim.x) cp_async16(to + shift + i, from + i);
    to += mat_room;
    from = x + s0 * features;
    for (int i = 4 * threadIdx.x; i < ns * features; i += 4 * blockDim.x) cp_async16(to + i, from + i);
  };
  int64_t s0 = (int64_t)blockIdx.x * samples;
  if (s0 < n) fetch(s0, 0);
  cp_async_commit();
  for (int buf = 0; s0 < n; s0 += step, buf ^= 1) {
    if (s0 + step < n) fetch(s0 + step, buf ^ 1);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    if (sample < (int)min((int64_t)samples, n - s0)) {
      for (int item = first; item < items; item += blockDim.x) {     // one, or one sample and several items
        const int t = item / cg, quad = (item - t * cg) * 4;
        const int lo = tiles.lo[t], row = tiles.row[t], rows = tiles.rows[t], len = tiles.len[t];
        // neighbouring tiles begin with different halves: the lanes of a phase then read different banks
        const int half = c / 2, ch = V == 2 && (t & 1) ? quad + half : quad, other = V == 2 && (t & 1) ? quad : quad + half;
        const int by_row = transposed ? 1 : dim, by_j = transposed ? dim : 1;
        const float* mp = sm + buf * buffer + shift_of(s0) + sample * dd + row * by_row + lo * by_j;
        const float* xp = sm + buf * buffer + mat_room + sample * features + lo * c;
        int at[4];                                                   // rows that the tile does not have: its last, not stored
#pragma unroll
        for (int u = 0; u < 4; ++u) at[u] = min(u, rows - 1) * by_row;
        uint64_t acc[4][2 * V] = {};
#pragma unroll 2
        for (int j = 0; j < len; ++j, xp += c, mp += by_j) {
          uint64_t m[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) m[u] = pair_of(mp[at[u]]);
#pragma unroll
          for (int h = 0; h < V; ++h) {
            const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(xp + (h ? other : ch));
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              pair_fma(acc[u][2 * h], m[u], xv.x);
              pair_fma(acc[u][2 * h + 1], m[u], xv.y);
            }
          }
        }
        float* o = out + (s0 + sample) * features + row * c;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < rows)
#pragma unroll
            for (int h = 0; h < V; ++h)
              *reinterpret_cast<ulonglong2*>(o + u * c + (h ? other : ch)) = make_ulonglong2(acc[u][2 * h], acc[u][2 * h + 1]);
      }
    }
    __syncthreads();
  }
}

// grad_M[n, i, j] = sum_c g[n, i, c] x[n, j, c] inside the blocks, zero outside.  Two neighbouring lanes make 4 x 4 entries of a
// block from rows that are ceil(size / 4) apart, one from the even and one from the odd groups of four channels, with 16-byte
// loads along the channels, so that neither operand is transposed on the way in; they exchange halves of their sums at the
// end.  Each lane begins with another group of channels: the lanes of a phase then read different banks although the rows are
// not padded, and a pass copies one run of each operand without a division.  Results go to an image of four samples whose
// zeros are written once, and the image leaves as one bulk copy.  Two lanes an item are twice the warps in the same shared
// memory: with one, on padded rows, eight warps an SM waited for their own chains and for barriers (issue 45 %).  An odd number of
// groups leaves the last to both lanes, two channels each (l = 0..6 of 36 channels, 40k samples 234 -> 207 us).
// 40k samples, one lane / two: l = 0..6 of 32 channels 232 / 177 us (5.0 TB/s), l = 0..4 of 64 channels 211 / 124, l = 0..2 of 32
// channels 45 / 35; a third pass in shared memory changes nothing (177, 124, 35).
constexpr int BG_THREADS = 256;
constexpr int BG_MAX_TILES = 512;
struct GradTiles {
  int count;
  uint32_t code[BG_MAX_TILES];                  // first row of the block, its size, tile row, tile column: eight bits each
};
enum GradForm { EVEN_GROUPS, ODD_GROUPS, ONE_LANE };      // two lanes an item, with an even or odd number of channel groups; one
template <GradForm FORM>
__global__ void __launch_bounds__(BG_THREADS) block_rotation_grad_kernel(const float* __restrict__ g, const float* __restrict__ x,
                                                                         float* __restrict__ gm, int64_t n, int dim, int c,
                                                                         int samples, int image_samples,
                                                                         const __grid_constant__ GradTiles tiles) {
  extern __shared__ __align__(16) float sm[];
  const int dd = dim * dim, features = dim * c, operand = samples * features, items = tiles.count;
  float* img = sm;                              // [image_samples][dim][dim]
  float* stage = img + image_samples * dd;      // [2][g, x][samples][dim][c]
  uint32_t* tile = reinterpret_cast<uint32_t*>(stage + 4 * operand);   // indexed by lane
  for (int i = threadIdx.x; i < items; i += blockDim.x) tile[i] = tiles.code[i];
  for (int i = threadIdx.x; i < image_samples * dd; i += blockDim.x) img[i] = 0.f;
  const int passes = image_samples / samples;   // per image
  const int64_t step = (int64_t)gridDim.x * image_samples;
  // the samples of one pass, and the pass after them: the next of the image or the first of the block's next image
  auto fetch = [&](int64_t base, int pass, int buf) {
    const int64_t s0 = base + pass * samples;
    const int floats = (int)max((int64_t)0, min((int64_t)samples, n - s0)) * features;
    float* to = stage + buf * 2 * operand;
    for (int i = 4 * threadIdx.x; i < floats; i += 4 * blockDim.x) {
      cp_async16(to + i, g + s0 * features + i);
      cp_async16(to + operand + i, x + s0 * features + i);
    }
    cp_async_commit();
  };
  int64_t ahead = (int64_t)blockIdx.x * image_samples;
  int ahead_pass = 0, buf = 0;
  auto fetch_next = [&](int to) {
    fetch(ahead, ahead_pass, to);
    if (++ahead_pass == passes) ahead_pass = 0, ahead += step;
  };
  fetch_next(0);
  constexpr int LANES = FORM == ONE_LANE ? 1 : 2;
  const int lane = threadIdx.x & 31, half = FORM == ONE_LANE ? 0 : lane & 1, groups = c / (4 * LANES);     // this lane's groups of channels
  const int first = FORM != ONE_LANE && groups ? (threadIdx.x >> 1) % groups : 0;
  for (int64_t base = (int64_t)blockIdx.x * image_samples; base < n; base += step) {
    const int total = (int)min((int64_t)image_samples, n - base);
    for (int pass = 0; pass < passes; ++pass) {
      const int part = pass * samples, ns = min(samples, total - part);
      if (pass == 0) image_release();
      cp_async_wait<0>();
      __syncthreads();                          // this pass has arrived; the place of the one before it is free
      fetch_next(buf ^ 1);
      for (int w = threadIdx.x - lane; w < LANES * ns * items; w += blockDim.x) {  // whole warps: the lanes exchange sums
        const bool made = w + lane < LANES * ns * items;
        const int i = made ? (w + lane) / LANES : 0, s = i / items;
        const uint32_t code = tile[i - s * items];
        const int lo = code & 255, size = code >> 8 & 255, np = (size + 3) / 4, pa = code >> 16 & 255, qa = code >> 24;
        const float* gp = stage + buf * 2 * operand + s * features + lo * c;
        const float* xp = gp + operand;
        int ro[4], co[4];                       // rows past the block read its last row and are not stored
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          ro[u] = min(pa + u * np, size - 1) * c;
          co[u] = min(qa + u * np, size - 1) * c;
        }
        uint64_t acc[4][4] = {};                // sums over even and odd channels
        for (int k = 0, at = first; k < groups; ++k, at = at + 1 == groups ? 0 : at + 1) {
          const int ch = 4 * LANES * at + 4 * half;
          ulonglong2 gv[4], xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            gv[u] = *reinterpret_cast<const ulonglong2*>(gp + ro[u] + ch);
            xv[u] = *reinterpret_cast<const ulonglong2*>(xp + co[u] + ch);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              pair_fma(acc[u][v], gv[u].x, xv[v].x);
              pair_fma(acc[u][v], gv[u].y, xv[v].y);
            }
        }
        if constexpr (FORM == ODD_GROUPS) {     // the last group: two channels each
          const int ch = c - 4 + 2 * half;
          uint64_t gv[4], xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            gv[u] = *reinterpret_cast<const uint64_t*>(gp + ro[u] + ch);
            xv[u] = *reinterpret_cast<const uint64_t*>(xp + co[u] + ch);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) pair_fma(acc[u][v], gv[u], xv[v]);
        }
        float* o = img + (part + s) * dd + lo * dim + lo;
        if constexpr (FORM == ONE_LANE) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v)
              if (made && pa + u * np < size && qa + v * np < size) o[(pa + u * np) * dim + qa + v * np] = pair_sum(acc[u][v]);
        } else {                                // the even lane keeps tile rows 0 and 1, the odd one 2 and 3
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int row = pa + (u + 2 * half) * np;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const float low = pair_sum(acc[u][v]), high = pair_sum(acc[u + 2][v]);
              const float sum = (half ? high : low) + __shfl_xor_sync(0xffffffffu, half ? low : high, 1);
              if (made && row < size && qa + v * np < size) o[row * dim + qa + v * np] = sum;
            }
          }
        }
      }
      buf ^= 1;
    }
    image_store(gm + base * dd, img, (int64_t)total * dd);
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

constexpr size_t SMEM_MOST = 200 * 1024;

template <typename K>
int resident_grid(K kernel, int threads, size_t bytes, int64_t want, unsigned* grid) {
  if (int rc = allow_shared(kernel, SMEM_MOST)) return rc;
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, bytes) != cudaSuccess || per_sm < 1) per_sm = 1;
  *grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sm_count() * per_sm));
  return EQT_OK;
}

bool on16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Quads of a table, from its component count alone: sum of (l + 1)^2 over blocks of 2 l + 1 components is bounded by
// dim * (max_l + 1) * (max_l + 1) / (2 max_l + 1); the exact list is on the device.
int quad_bound(const eqt_wigner_table* t) {
  const int l1 = t->max_l + 1;
  return (int)std::min<int64_t>((int64_t)t->dim * l1 * l1 / (2 * t->max_l + 1), INT32_MAX);
}

bool rotation_tiles(const int32_t* sizes, int blocks, RowTiles& t, int* dim) {
  t = RowTiles{};
  int start = 0, entries = 0;
  for (int b = 0; b < blocks; ++b) {
    if (sizes[b] <= 0 || sizes[b] > BR_MAX_DIM - start) return false;
    for (int u = 0; u < sizes[b]; u += 4) {
      const int rows = std::min(4, sizes[b] - u), i = t.count++;
      t.row[i] = (uint8_t)(start + u);
      t.rows[i] = (uint8_t)rows;
      t.lo[i] = (uint8_t)start;
      t.len[i] = (uint8_t)sizes[b];
      t.at[i] = (uint16_t)t.floats;
      t.first[i] = (uint16_t)entries;
      t.floats += 4 * sizes[b];
      entries += rows * sizes[b];
      t.first[t.count] = (uint16_t)entries;
    }
    start += sizes[b];
  }
  *dim = start;
  return true;                              // at most 128 * 128 entries and 128 * 128 + 3 * 128 floats: 16 bits hold both
}
size_t rotation_bytes(const RowTiles& t, int dim, int c, int samples) {
  return sizeof(float) * (((size_t)t.first[t.count] + 3) / 4 * 4 + 2 * (size_t)samples * (t.floats + (size_t)dim * c));
}
// Samples per pass: one item per thread, or as many as leave four blocks per SM their shared memory.
int rotation_samples(const RowTiles& t, int dim, int c) {
  int samples = std::max(1, std::min(16, BR_THREADS / std::max(1, t.count * (c / 4))));
  while (samples > 1 && rotation_bytes(t, dim, c, samples) > 56 * 1024) --samples;
  return rotation_bytes(t, dim, c, samples) <= SMEM_MOST ? samples : 0;
}


// Whole matrices where the rows of the blocks, in lines of 128 bytes, touch all of them (l = 0..5 and less; 81 % at l = 0..6, and
// HBM reads that share of them).  40k samples, by list / whole: l = 0..4 of 64 channels 145 / 120 us, l = 0..3 of 32 67 / 53,
// l = 0..2 of 32 54 / 38, l = 0..5 of 32 117 / 113; but l = 0..6 of 32 154 / 177, l = 0..7 of 32 186 / 218.
bool rotation_whole(const int32_t* sizes, int blocks, int dim) {
  int64_t touched = 124 * (int64_t)dim;
  for (int b = 0; b < blocks; ++b) touched += 4 * (int64_t)sizes[b] * sizes[b];
  return touched >= 4 * (int64_t)dim * dim;
}
// Not for operands far beyond L2 where a pass has one or two samples: a block then waits for what it copies, and the list leaves
// room for more of them (l = 0..4 of 128 channels, 20k samples 99 / 96 us, 40k 190 / 193, 80k 371 / 392; l = 0..5 of 64, 20k 83 / 78, 40k 157 /
// 161, 80k 306 / 326, of 192, 80k 758 / 847; l = 0..3 of 128, 80k 247 / 254; but l = 0..4 of 96, 80k 314 / 286).
bool whole_too_slow(int samples, int dim, int c, int64_t n) {
  const double bytes = 4. * n * ((double)dim * dim + 2. * dim * c);
  return bytes > 0.8e9 && (samples == 1 || (samples == 2 && (c >= 128 || dim >= 36)));
}
// Channels of a thread: twice four where they divide so (l = 0..4 of 64 channels: 134 us with four, 119 so).
int whole_quads(int c) { return c % 8 ? 1 : 2; }
size_t whole_bytes(int dim, int c, int samples) {
  return 2 * sizeof(float) * (((size_t)samples * dim * dim + 6) / 4 * 4 + (size_t)samples * dim * c);
}
// Samples per pass: one item per thread, or as many as leave three blocks per SM their shared memory; 0 if one does not fit.
int whole_samples(const RowTiles& t, int dim, int c) {
  int samples = std::max(1, std::min(16, BR_THREADS / std::max(1, t.count * (c / 4 / whole_quads(c)))));
  while (samples > 1 && whole_bytes(dim, c, samples) > 72 * 1024) --samples;
  return whole_bytes(dim, c, samples) <= SMEM_MOST ? samples : 0;
}

bool gradient_tiles(const int32_t* sizes, int blocks, GradTiles& t) {
  t.count = 0;
  for (int b = 0, start = 0; b < blocks; start += sizes[b++]) {
    const int np = (sizes[b] + 3) / 4;
    if (t.count + np * np > BG_MAX_TILES) return false;
    for (int i = 0; i < np * np; ++i)
      t.code[t.count++] = (uint32_t)start | (uint32_t)sizes[b] << 8 | (uint32_t)(i / np) << 16 | (uint32_t)(i % np) << 24;
  }
  return true;
}
// Samples per pass (a power of two, about two threads an item) and per image (a multiple of four and of the former); returns
// the shared memory, 0 where it does not fit.
size_t gradient_samples(const GradTiles& t, int dim, int c, int* samples, int* image) {
  int s = 16;
  while (s > 1 && 2 * s * t.count > BG_THREADS) s /= 2;
  for (;; s /= 2) {
    *samples = s;
    *image = std::max(4, s);
    const size_t bytes = sizeof(float) * ((size_t)*image * dim * dim + 4 * (size_t)s * dim * c + t.count);
    if (bytes <= 112 * 1024 || (s == 1 && bytes <= SMEM_MOST)) return bytes;
    if (s == 1) return 0;
  }
}

template <int L1>
int quads_forward(Quads a, int groups, cudaStream_t st) {
  const int threads = groups * a.group_threads, dd = a.dim * a.dim;
  const size_t bytes = sizeof(float) * a.samples * ((size_t)dd + 3 * L1 * 2);
  unsigned grid = 1;
  if (int rc = resident_grid(wigner_quads_forward_kernel<L1>, threads, bytes, ceil_div(a.n, a.samples), &grid)) return rc;
  wigner_quads_forward_kernel<L1><<<grid, threads, bytes, st>>>(a);
  return check_launch("wigner_quads_forward_kernel");
}
template <int L1>
int quads_backward(Quads a, int groups, cudaStream_t st) {
  const int threads = groups * a.group_threads;
  const size_t bytes = sizeof(float) * a.samples * ((size_t)3 * L1 * 2 + 3 * (a.group_threads / 32));
  unsigned grid = 1;
  if (int rc = resident_grid(wigner_quads_backward_kernel<L1>, threads, bytes, ceil_div(a.n, a.samples), &grid)) return rc;
  wigner_quads_backward_kernel<L1><<<grid, threads, bytes, st>>>(a);
  return check_launch("wigner_quads_backward_kernel");
}

// Threads per sample, samples per pass (a multiple of four, so that whole groups are multiples of 16 bytes) and thread groups.
bool quads_setup(const eqt_wigner_table* t, Quads& a, int* groups, bool image) {
  const int threads = (int)ceil_div(quad_bound(t), 32) * 32;
  if (threads > WQ_MAX_THREADS || t->max_l > 7) return false;
  a.coef = static_cast<const float*>(t->coef);
  a.blocks = t->blocks;
  a.dim = t->dim;
  a.num_blocks = t->num_blocks;
  a.group_threads = threads;
  *groups = std::max(1, 192 / threads);
  a.samples = (int)ceil_div(std::max(4, 2 * *groups), 4) * 4;
  return !image || sizeof(float) * a.samples * ((size_t)a.dim * a.dim + 48) <= SMEM_MOST;
}

}  // namespace

int wigner_quads_forward(const eqt_wigner_table* t, const float* alpha, const float* beta, const float* gamma, float* d, int64_t n,
                         cudaStream_t st) {
  Quads a{};
  int groups = 1;
  if (!quads_setup(t, a, &groups, true)) return NOT_TAKEN;
  a.angle[0] = alpha;
  a.angle[1] = beta;
  a.angle[2] = gamma;
  a.d = d;
  a.n = n;
  return t->max_l < 4 ? quads_forward<4>(a, groups, st) : t->max_l < 7 ? quads_forward<7>(a, groups, st) : quads_forward<8>(a, groups, st);
}

int wigner_quads_backward(const eqt_wigner_table* t, const float* alpha, const float* beta, const float* gamma, const float* grad_d,
                          float* ga, float* gb, float* gc, int64_t n, cudaStream_t st) {
  Quads a{};
  int groups = 1;
  if (!quads_setup(t, a, &groups, false)) return NOT_TAKEN;
  a.angle[0] = alpha;
  a.angle[1] = beta;
  a.angle[2] = gamma;
  a.d = const_cast<float*>(grad_d);
  a.grad[0] = ga;
  a.grad[1] = gb;
  a.grad[2] = gc;
  a.n = n;
  a.samples = 8 * groups;
  return t->max_l < 4 ? quads_backward<4>(a, groups, st) : t->max_l < 7 ? quads_backward<7>(a, groups, st) : quads_backward<8>(a, groups, st);
}

}  // namespace eqt

extern "C" int eqt_block_rotation_supported(const int32_t* block_sizes, int32_t num_blocks, int32_t channels) {
  using namespace eqt;
  if (!block_sizes || num_blocks <= 0 || channels <= 0 || channels % 4) return 0;
  RowTiles t;
  GradTiles g;
  int dim = 0, samples = 0, image = 0;
  if (!rotation_tiles(block_sizes, num_blocks, t, &dim) || !gradient_tiles(block_sizes, num_blocks, g)) return 0;
  return rotation_samples(t, dim, channels) > 0 && gradient_samples(g, dim, channels, &samples, &image) > 0;
}

extern "C" int eqt_block_rotation(const float* matrix, const float* x, float* out, int64_t n, const int32_t* block_sizes,
                                  int32_t num_blocks, int32_t channels, int32_t transposed, void* stream) {
  using namespace eqt;
  if (n < 0 || !eqt_block_rotation_supported(block_sizes, num_blocks, channels)) return fail(EQT_ERR_UNSUPPORTED, "blocks or channels");
  if (n == 0) return EQT_OK;
  if (!matrix || !x || !out) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (!on16(x) || !on16(out)) return fail(EQT_ERR_UNSUPPORTED, "features must be 16-byte aligned");
  RowTiles t;
  int dim = 0;
  rotation_tiles(block_sizes, num_blocks, t, &dim);
  unsigned grid = 1;
  const int whole = rotation_whole(block_sizes, num_blocks, dim) ? whole_samples(t, dim, channels) : 0;
  if (whole > 0 && !whole_too_slow(whole, dim, channels, n)) {
    const int samples = whole;
    const size_t bytes = whole_bytes(dim, channels, samples);
    const auto kernel = whole_quads(channels) == 2 ? block_rotation_whole_kernel<2> : block_rotation_whole_kernel<1>;
    const int items = samples * t.count * (channels / 4 / whole_quads(channels)), threads = std::min(BR_THREADS, (items + 31) / 32 * 32);
    if (int rc = resident_grid(kernel, threads, bytes, ceil_div(n, samples), &grid)) return rc;
    kernel<<<grid, threads, bytes, static_cast<cudaStream_t>(stream)>>>(matrix, x, out, n, dim, channels, transposed, samples, t);
    return check_launch("block_rotation_whole_kernel");
  }
  const int samples = rotation_samples(t, dim, channels);
  const size_t bytes = rotation_bytes(t, dim, channels, samples);
  if (int rc = resident_grid(block_rotation_kernel, BR_THREADS, bytes, ceil_div(n, samples), &grid)) return rc;
  block_rotation_kernel<<<grid, BR_THREADS, bytes, static_cast<cudaStream_t>(stream)>>>(matrix, x, out, n, dim, channels, transposed,
                                                                                       samples, t);
  return check_launch("block_rotation_kernel");
}

extern "C" int eqt_block_rotation_grad_matrix(const float* grad_out, const float* x, float* grad_matrix, int64_t n,
                                              const int32_t* block_sizes, int32_t num_blocks, int32_t channels, void* stream) {
  using namespace eqt;
  if (n < 0 || !eqt_block_rotation_supported(block_sizes, num_blocks, channels)) return fail(EQT_ERR_UNSUPPORTED, "blocks or channels");
  if (n == 0) return EQT_OK;
  if (!grad_out || !x || !grad_matrix) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (!on16(x) || !on16(grad_out)) return fail(EQT_ERR_UNSUPPORTED, "features must be 16-byte aligned");
  RowTiles t;
  GradTiles g;
  int dim = 0, samples = 0, image = 0;
  rotation_tiles(block_sizes, num_blocks, t, &dim);
  gradient_tiles(block_sizes, num_blocks, g);
  const size_t bytes = gradient_samples(g, dim, channels, &samples, &image);
  unsigned grid = 1;
  // few channels are soon multiplied, and then the exchange of sums costs more than the second lane saves, as long as the samples fill
  // the SMs (40k samples, two lanes / one: l = 0..2 of 4 channels 12.7 / 7.8 us, l = 0..6 of 4 105 / 82, of 12 125 / 105; 300 samples 5.1 /
  // 6.0; l = 0, 1 of 8 5.8 / 6.7)
  const bool one = channels <= 12 && dim >= 9 && n >= 16 * (int64_t)sm_count();
  const auto kernel = one ? block_rotation_grad_kernel<ONE_LANE>
                          : channels % 8 ? block_rotation_grad_kernel<ODD_GROUPS> : block_rotation_grad_kernel<EVEN_GROUPS>;
  const int threads = std::min(BG_THREADS, ((one ? 1 : 2) * samples * g.count + 31) / 32 * 32);
  if (int rc = resident_grid(kernel, threads, bytes, ceil_div(n, image), &grid)) return rc;
  kernel<<<grid, threads, bytes, static_cast<cudaStream_t>(stream)>>>(grad_out, x, grad_matrix, n, dim, channels,
                                                                                            samples, image, g);
  return check_launch("block_rotation_grad_kernel");
}
