// Clebsch-Gordan segment sums and their adjoint with one warp per (node, 32 lanes of channels), float32.
//
//   segment sum   S[d, r, c] = sum_{e in seg[d]} sum_{t in row r} scale[t] y[e, my[t]] feat[fidx[e], mf[t], c],
//                 with weights out[d, k, c] = sum_{r of k} w[path(r), c] S[d, r, c]  and, given x,
//                 gw[p, c] = sum_d sum_{r of p} x[d, k(r), c] S[d, r, c];  S itself is not written then
//   adjoint       gy[e, k] = sum_{t: my[t] = k} scale[t] sum_c feat[fidx[e], mf[t], c] G[node(e), row[t], c],
//                 with weights G[d, r, c] = w[path(r), c] g[d, k(r), c], which is not read from memory then
//
// The sum over a node's edges commutes with the Clebsch-Gordan contraction, so per edge only the outer product
// Q[m_y, m_feat] += y[m_y] x[m_feat] is accumulated, in a lane's registers: all cells of a channel (71 at l_max 2, several
// channels a lane at l_max 1), or half of them where registers end (l_max 3: two warps, 120 and 114 of the 234 cells).  A warp gathers
// its channels of the coming edges into a ring of its own (cp.async), so warps neither wait for each other nor share the
// staging of a row; they take contiguous ranges of nodes of equal work, found in the segment pointers at the start.
//
// What bounds it: instruction issue.  Per edge and 32 channels a warp needs 71 multiply-adds at l_max 2 (43 instructions: two cells
// m_y, m_y + 1 of a component share a packed one), 12 loads from shared memory and some 30 instructions of the ring; with four warps a
// node and two channels a lane the loads, the ring and the loop cost as much as the multiply-adds, in every one of the four.  20k
// nodes, 400k edges, 128 channels, l_max 2: a segment sum 581 -> 307 us (61 % of the issue slots used), the adjoint 751 -> 466; the same
// with channel-wise weights, a whole pass (the rows of 20k x 35 x 128 written and read five times less) 2322 -> 1072 us.
#include <algorithm>
#include <type_traits>

#include "tp_walk.cuh"

namespace eqt {
namespace {

template <int V> __device__ __forceinline__ void ld_lane(float (&x)[V], const float* p) {
  if constexpr (V == 4) { const float4 v = *reinterpret_cast<const float4*>(p); x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
  else if constexpr (V == 2) { const float2 v = *reinterpret_cast<const float2*>(p); x[0] = v.x; x[1] = v.y; }
  else x[0] = p[0];
}
template <int V> __device__ __forceinline__ void ldg_lane(float (&x)[V], const float* p) {
  if constexpr (V == 4) { const float4 v = __ldg(reinterpret_cast<const float4*>(p)); x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w; }
  else if constexpr (V == 2) { const float2 v = __ldg(reinterpret_cast<const float2*>(p)); x[0] = v.x; x[1] = v.y; }
  else x[0] = __ldg(p);
}
template <int V> __device__ __forceinline__ void st_lane(float* p, const float (&v)[V]) {
  if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if constexpr (V == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else p[0] = v[0];
}
template <int V> __device__ __forceinline__ void fma_lane(float (&acc)[V], const float (&a)[V], const float (&b)[V]) {
#pragma unroll
  for (int k = 0; k < V; ++k) acc[k] = fmaf(a[k], b[k], acc[k]);
}
// (a, b) += x (u, v): packed where a lane holds one channel (fma.rn.f32x2 takes one issue slot instead of two)
template <int V> __device__ __forceinline__ void fma_pair(float (&a)[V], float (&b)[V], const float (&x)[V], float u, float v) {
  if constexpr (V == 1) {
    asm("{\n\t.reg .b64 s, t, r;\n\tmov.b64 s, {%2, %2};\n\tmov.b64 t, {%3, %4};\n\tmov.b64 r, {%0, %1};\n\t"
        "fma.rn.f32x2 r, s, t, r;\n\tmov.b64 {%0, %1}, r;\n\t}" : "+f"(a[0]), "+f"(b[0]) : "f"(x[0]), "f"(u), "f"(v));
  } else {
#pragma unroll
    for (int k = 0; k < V; ++k) { a[k] = fmaf(x[k], u, a[k]); b[k] = fmaf(x[k], v, b[k]); }
  }
}
template <int V> __device__ __forceinline__ void dot_pair(float& a, float& b, const float (&x)[V], const float (&u)[V], const float (&v)[V]) {
  if constexpr (V == 1) {
    asm("{\n\t.reg .b64 s, t, r;\n\tmov.b64 s, {%2, %2};\n\tmov.b64 t, {%3, %4};\n\tmov.b64 r, {%0, %1};\n\t"
        "fma.rn.f32x2 r, s, t, r;\n\tmov.b64 {%0, %1}, r;\n\t}" : "+f"(a), "+f"(b) : "f"(x[0]), "f"(u[0]), "f"(v[0]));
  } else {
#pragma unroll
    for (int k = 0; k < V; ++k) { a = fmaf(x[k], u[k], a); b = fmaf(x[k], v[k], b); }
  }
}
#define EQT_LDX(X, P) ld_lane<V>(X, P)
#define EQT_FMA(ACC, A, S) do { _Pragma("unroll") for (int k_ = 0; k_ < V; ++k_) (ACC)[k_] = fmaf((A)[k_], (S), (ACC)[k_]); } while (0)
#define EQT_FMA2(A, B, X, S, T) fma_pair<V>(A, B, X, S, T)
#define EQT_MUL(ACC, A, S) do { _Pragma("unroll") for (int k_ = 0; k_ < V; ++k_) (ACC)[k_] = (A)[k_] * (S); } while (0)
#define EQT_ZERO(X) do { _Pragma("unroll") for (int k_ = 0; k_ < V; ++k_) (X)[k_] = 0.f; } while (0)
#define EQT_DOT(ACC, X, H) do { _Pragma("unroll") for (int k_ = 0; k_ < V; ++k_) (ACC) = fmaf((X)[k_], (H)[k_], (ACC)); } while (0)
#define EQT_DOT2(A, B, X, G, H) dot_pair<V>(A, B, X, G, H)
#include "generated/walk_specs.inc"
#undef EQT_LDX
#undef EQT_FMA
#undef EQT_FMA2
#undef EQT_MUL
#undef EQT_ZERO
#undef EQT_DOT
#undef EQT_DOT2

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void copy16(uint32_t dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

constexpr int DEPTH = 4;      // ring slots of a warp

// A warp handles CW = V 32 / EPW channels of EPW edges at a time: V channels a lane, and with 16 channels (EPW = 2) a half-warp
// an edge.  CC: the layer's channels, or 0 where only a.C tells.
template <class S, int V, int EPW, int CC, bool WITH_Y>
struct Ring {
  static constexpr int LPE = 32 / EPW, CW = LPE * V, XF = S::NX * CW, YF = WITH_Y ? S::YF : 0, SLOT = EPW * (XF + YF);
  static constexpr int CHUNKS = S::NX * CW / 4, PASSES = (CHUNKS + LPE - 1) / LPE;       // 16-byte pieces of an edge; per lane
  static constexpr int STEP = LPE / (CW / 4);                                            // components between a lane's pieces
  const WalkArgs& a;
  uint32_t dst;                 // this lane's place in slot 0 (shared-memory address)
  float* ring;
  int lane, sub, ne;
  int64_t e0;
  const float* src;             // this lane's piece of feature row 0, its place in row 0 of y
  const float* ysrc;
  int delta;                    // two halves: from there to the lane's second piece (floats)
  uint32_t fi, nfi, yi, nyi;    // gather indices of edge 32 block + lane of this block of 32 edges and of the next

  __device__ __forceinline__ Ring(const WalkArgs& a_, float* ring_, int lane_, int half, int channel0, int64_t e0_, int ne_)
      : a(a_), ring(ring_), lane(lane_), sub(lane_ / LPE), ne(ne_), e0(e0_), delta(0) {
    const int C = CC ? CC : a.C, piece = lane % LPE, at = piece / (CW / 4);
    src = a.feat + S::comp(half, at) * C + channel0 + piece % (CW / 4) * 4;
    if (S::HALVES == 2) delta = (S::comp(half, at + STEP) - S::comp(half, at)) * C;
    static_assert(S::HALVES == 1 || (PASSES == 2 && CHUNKS % LPE == 0), "a half's pieces are two to a lane");
    if (WITH_Y) ysrc = a.y + lane % LPE;
    dst = smem_addr(ring + sub * (XF + YF) + piece * 4);
    fetch(0);
    fi = nfi; yi = nyi;
    fetch(1);
  }
  __device__ __forceinline__ void fetch(int block) {
    const int e = block * 32 + lane;
    const bool in = e < ne;
    nfi = in ? (uint32_t)(a.fidx ? __ldg(a.fidx + e0 + e) : e0 + e) : 0;
    if (WITH_Y) nyi = in ? (uint32_t)(a.yidx ? __ldg(a.yidx + e0 + e) : e0 + e) : 0;
  }
  // request the edges EPW t, EPW t + 1 .. (nothing past the end); always closes a group
  __device__ __forceinline__ void issue(int t) {
    const int first = t * EPW;
    if (first < ne) {
      const int C = CC ? CC : a.C;
      if (first % 32 == 0 && t) { fi = nfi; yi = nyi; fetch(first / 32 + 1); }
      const uint32_t row = __shfl_sync(0xffffffffu, fi, (first + sub) % 32), to = dst + (uint32_t)(t % DEPTH) * (SLOT * 4);
      const bool in = EPW == 1 || first + sub < ne;
      const float* p = src + (uint64_t)row * (uint32_t)(S::DF * C);
#pragma unroll
      for (int i = 0; i < PASSES; ++i) {
        if (in && ((i + 1) * LPE <= CHUNKS || lane % LPE + i * LPE < CHUNKS))
          copy16(to + i * LPE * 16, S::HALVES == 2 ? (i ? p + delta : p) : p + i * STEP * C);
      }
      if (WITH_Y) {
        const uint32_t yrow = __shfl_sync(0xffffffffu, yi, (first + sub) % 32);
        if (in && lane % LPE < S::DY) copy4(to + XF * 4 - (lane % LPE) * 12, ysrc + (uint64_t)yrow * S::DY);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void start() {
    for (int t = 0; t < DEPTH - 1; ++t) issue(t);
  }
  // stage t has landed for every lane of the warp; the slot of stage t - 1 is refilled
  __device__ __forceinline__ const float* stage(int t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 2) : "memory");
    __syncwarp();
    issue(t + DEPTH - 1);
    return ring + (t % DEPTH) * SLOT + sub * (XF + YF);
  }
};

// First node whose work, cost(d) = edge_cost ptr[d] + node_cost d, is at least total * part / parts: lanes 0-15 search for
// `part`, lanes 16-31 for `part + 1`, sixteen probes a round.  Returns (first node, nodes) of this part.
template <int EDGE_COST, int NODE_COST>
__device__ __forceinline__ int2 share_of_nodes(const int64_t* ptr, int64_t n, int part, int parts, int lane) {
  if (parts >= n) return make_int2(min(part, (int)n), part < n ? 1 : 0);
  const int64_t base = ptr ? __ldg(ptr) : 0, total = EDGE_COST * ((ptr ? __ldg(ptr + n) : n) - base) + NODE_COST * n;
  const int64_t target = total * (part + (lane >> 4)) / parts;
  int64_t lo = 0, len = n;
  while (__any_sync(0xffffffffu, len > 0)) {
    const int64_t step = (len + 15) >> 4, end = min((int64_t)((lane & 15) + 1) * step, len);
    const int64_t p = lo + end - 1;
    const bool yes = len > 0 && EDGE_COST * ((ptr ? __ldg(ptr + p) : p) - base) + NODE_COST * p >= target;
    const uint32_t votes = (__ballot_sync(0xffffffffu, yes) >> (lane & 16)) & 0xffffu;
    if (len > 0) {
      if (votes == 0) {
        lo += len;
        len = 0;
      } else {
        const int f = __ffs(votes) - 1;
        const int64_t skip = f * step, last = min((int64_t)(f + 1) * step, len) - 1;
        lo += skip;
        len = last - skip;
      }
    }
  }
  const int first = (int)__shfl_sync(0xffffffffu, lo, 0);
  return make_int2(first, (int)__shfl_sync(0xffffffffu, lo, 16) - first);
}

enum WalkMode { ROWS, MIX, MIX_GRAD };     // rows as they are; mixed by weights; that and the weights' gradient

template <int V, int EPW> __device__ __forceinline__ void over_edges(float (&v)[V]) {     // lanes of different edges hold parts of a sum
#pragma unroll
  for (int k = 0; k < V; ++k)
    if constexpr (EPW == 2) v[k] += __shfl_xor_sync(0xffffffffu, v[k], 16);
}

template <int V, int EPW, int CC>
struct RowSink {
  float* o;
  int channels;
  bool store;
  template <int K> __device__ __forceinline__ void open() {}
  template <int R, int K, int P, int L> __device__ __forceinline__ void row(float (&v)[V]) {
    over_edges<V, EPW>(v);
    if (EPW == 1 || store) st_lane<V>(o + R * (CC ? CC : channels), v);
  }
  template <int K> __device__ __forceinline__ void close() {}
};

template <class S, int V, int EPW, int CC, bool GRAD>
struct MixSink {
  static constexpr int CW = 32 / EPW * V, OWN = S::HALVES == 2 ? (S::K + 1) / 2 : 1;
  float* o;
  const float* ws;                     // weights of the warp's channels, paths CW floats apart
  const float* x;
  int channels, half;
  float* give;                         // where the other half finds this half's part of its components
  float (&gw)[S::NP][V];
  float acc[V], xv[V];
  float own[OWN][V];
  template <int K> __device__ __forceinline__ void open() {
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = 0.f;
    if (GRAD) ldg_lane<V>(xv, x + K * (CC ? CC : channels));
  }
  template <int R, int K, int P, int L> __device__ __forceinline__ void row(const float (&v)[V]) {
    float w[V];
    ld_lane<V>(w, ws + P * CW);
    fma_lane<V>(acc, w, v);
    if (GRAD) fma_lane<V>(gw[L], xv, v);
  }
  template <int K> __device__ __forceinline__ void close() {
    over_edges<V, EPW>(acc);
    if constexpr (S::HALVES == 1) {
      if (EPW == 1 || (threadIdx.x & 16) == 0) st_lane<V>(o + K * (CC ? CC : channels), acc);
    } else {                           // even components are finished by half 0, odd ones by half 1
      if ((K & 1) == half) {
#pragma unroll
        for (int k = 0; k < V; ++k) own[K / 2][k] = acc[k];
      } else if (EPW == 1 || (threadIdx.x & 16) == 0) {
        st_lane<V>(give + (K / 2) * CW, acc);
      }
    }
  }
};

template <class S, int V> constexpr int sum_ctas(int mode) {     // of four warps an SM, by the registers of a lane
  return S::NC * V > 96 ? 3 : S::NC * V > 64 ? (mode == MIX_GRAD ? 3 : 4) : 5;
}

// Nodes whose part of the weights' gradient a lane adds up in registers before it goes to the group's sums in shared memory.  One
// chain over all nodes of a warp grows with the graph (l_max 3, 128 channels, error of the norm: 20k nodes 3.6e-7, 100k 7.9e-7; in sixteens
// 1.6e-7 at either, in eights 1.25e-7).  A pass of few edges a node takes 1-2 % longer, one of thirty under 1 %.
constexpr int FOLD_NODES = 16;

template <class S, int V, int EPW, int CC, int MODE>
struct SumShared {
  using R = Ring<S, V, EPW, CC, true>;
  static constexpr int GROUPS = 4 / S::HALVES, CW = R::CW;
  static constexpr int SC = S::HALVES * S::TH, WS = MODE == ROWS ? 0 : S::P * CW;
  static constexpr int XCH = MODE != ROWS && S::HALVES == 2 ? GROUPS * 2 * 2 * ((S::K + 1) / 2) * CW : 0;
  static constexpr int RINGS = 4 * DEPTH * R::SLOT;
  // weight gradients of a group: 64 bits where five CTAs an SM have room for them (not with four channels a lane)
  using Sum = std::conditional_t<V == 4, float, double>;
  static constexpr int GW = MODE == MIX_GRAD ? GROUPS * S::P * 32 * V : 0;
  static constexpr size_t BYTES = sizeof(float) * (SC + WS + XCH + RINGS) + sizeof(Sum) * GW;
};

template <class S, int V, int EPW, int CC, int MODE>
__global__ void __launch_bounds__(128, (sum_ctas<S, V>(MODE))) walk_sum_kernel(WalkArgs a) {
  using SH = SumShared<S, V, EPW, CC, MODE>;
  using R = typename SH::R;
  constexpr int CW = R::CW;
  extern __shared__ __align__(16) float shared[];
  float* sc = shared;
  float* ws = sc + SH::SC;
  float* xch = ws + SH::WS;
  float* rings = xch + SH::XCH;
  using Sum = typename SH::Sum;
  Sum* sums = reinterpret_cast<Sum*>(rings + SH::RINGS);             // [group][path][lane][V]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = S::HALVES == 2 ? warp & 1 : 0, group = S::HALVES == 2 ? warp >> 1 : warp;
  const int C = CC ? CC : a.C, channel0 = blockIdx.y * CW, ch = lane % R::LPE * V;

  for (int i = tid; i < SH::SC; i += 128) {
    const int t = S::order(i);
    sc[i] = t >= 0 ? __ldg(a.scale + t) : 0.f;
  }
  if (MODE != ROWS)
    for (int i = tid; i < SH::WS; i += 128) ws[i] = __ldg(a.w + (int64_t)(i / CW) * C + channel0 + i % CW);
  const int2 share = share_of_nodes<S::NC * V + 30, S::TH * V + 100>(a.ptr, a.n_out, blockIdx.x * SH::GROUPS + group, gridDim.x * SH::GROUPS, lane);
  const int64_t d0 = share.x;
  const int nd = share.y;
  __syncthreads();

  float gw[S::NP][V];
#pragma unroll
  for (int i = 0; i < S::NP; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) gw[i][k] = 0.f;
  auto fold = [&](bool first) __attribute__((always_inline)) {       // a path's rows, and so its sums, belong to one half
#pragma unroll
    for (int i = 0; i < S::NP; ++i) {
      const int p = S::path(half, i);
      if (p < 0) continue;
      Sum* to = sums + ((group * S::P + p) * 32 + lane) * V;
#pragma unroll
      for (int k = 0; k < V; ++k) {
        to[k] = (first ? Sum(0) : to[k]) + gw[i][k];
        gw[i][k] = 0.f;
      }
    }
  };
  if (nd > 0) {
    const int64_t* ptr = a.ptr ? a.ptr + d0 : nullptr;
    const int64_t e0 = ptr ? __ldg(ptr) : d0;
    const int ne = ptr ? (int)(__ldg(ptr + nd) - e0) : nd;
    R ring(a, rings + warp * (DEPTH * R::SLOT), lane, half, channel0, e0, ne);
    ring.start();

    float q[S::NC][V];
#pragma unroll
    for (int i = 0; i < S::NC; ++i)
#pragma unroll
      for (int k = 0; k < V; ++k) q[i][k] = 0.f;
    const float4* scales = reinterpret_cast<const float4*>(sc + half * S::TH);
    int d = 0;
    auto edge_end = [&](int i) { return i < nd ? ptr ? (int)(__ldg(ptr + i + 1) - e0) : i + 1 : 0; };
    int boundary = edge_end(0), next = edge_end(1);       // first edge of the nodes behind this one and behind the next
    auto flush = [&]() __attribute__((always_inline)) {   // a node without edges flushes a zero Q, i.e. zero rows
      if constexpr (MODE == ROWS) {
        RowSink<V, EPW, CC> sink{a.out + (d0 + d) * S::R * C + channel0 + ch, a.C, EPW == 1 || lane < 16};
        if (half == 0) S::template rows0<V>(q, scales, sink);
        else S::template rows1<V>(q, scales, sink);
      } else {
        float* o = a.out + (d0 + d) * S::K * C + channel0 + ch;
        constexpr int PART = (S::K + 1) / 2 * CW;
        float* buffers = xch + (group * 2 + (d & 1)) * 2 * PART + ch;      // of this node: one from each half
        MixSink<S, V, EPW, CC, MODE == MIX_GRAD> sink{o, ws + ch, MODE == MIX_GRAD ? a.x + (d0 + d) * S::K * C + channel0 + ch : nullptr,
                                                  a.C, half, buffers + half * PART, gw};
        if (half == 0) S::template rows0<V>(q, scales, sink);
        else S::template rows1<V>(q, scales, sink);
        if constexpr (S::HALVES == 2) {
          // the pair meets once a node; two sets of buffers, so a half is at most one node ahead of what the other still reads
          asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory");
          const float* take = buffers + (half ^ 1) * PART;
#pragma unroll
          for (int i = 0; i < (S::K + 1) / 2; ++i) {
            float v[V];
            ld_lane<V>(v, take + i * CW);
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] += sink.own[i][k];
            if (2 * i + half < S::K && (EPW == 1 || lane < 16)) st_lane<V>(o + (2 * i + half) * C, v);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < S::NC; ++i)
#pragma unroll
        for (int k = 0; k < V; ++k) q[i][k] = 0.f;
      ++d;
      if (MODE == MIX_GRAD && d % FOLD_NODES == 0) fold(d == FOLD_NODES);
      boundary = next;
      next = edge_end(d + 1);
    };

    // the round behind the last stage only flushes, so that the code of a flush is there once
    const int stages = (ne + EPW - 1) / EPW;
    for (int t = 0; t <= stages; ++t) {
      if (EPW == 1 || t == stages) {
        while (t == stages ? d < nd : t >= boundary) flush();
        if (t == stages) break;
      }
      const float* xs = ring.stage(t);
      auto add = [&]() __attribute__((always_inline)) {
        float y[S::YF];
#pragma unroll
        for (int k = 0; k < S::YF; k += 4) {
          const float4 v = *reinterpret_cast<const float4*>(xs + R::XF + k);
          y[k] = v.x; y[k + 1] = v.y; y[k + 2] = v.z; y[k + 3] = v.w;
        }
        if (half == 0) S::template outer0<V, CW>(q, xs + ch, y);
        else S::template outer1<V, CW>(q, xs + ch, y);
      };
      if constexpr (EPW == 1) {
        add();
      } else {                            // the two edges of a stage may belong to different nodes
        const int mine = t * EPW + ring.sub, end = min(t * EPW + EPW, ne);
        for (int e = t * EPW; e < end;) {
          while (e >= boundary) flush();
          const int to = min(boundary, end);
          if (mine >= e && mine < to) add();
          __syncwarp();
          e = to;
        }
      }
    }
  }

  if constexpr (MODE == MIX_GRAD) {        // the warps' sums in a fixed order; the rest of them is walk_gw_kernel's
    fold(nd < FOLD_NODES);
    __syncthreads();
    for (int i = tid; i < S::P * CW; i += 128) {
      const int p = i / CW, c = i % CW;
      Sum v = 0;
#pragma unroll
      for (int g = 0; g < SH::GROUPS; ++g)
#pragma unroll
        for (int e = 0; e < EPW; ++e) v += sums[(g * S::P + p) * 32 * V + e * CW + c];
      a.scratch[((int64_t)blockIdx.x * S::P + p) * C + channel0 + c] = static_cast<float>(v);
    }
  }
}

// gw[i] = sum of the CTAs' parts, added up in 64 bits in a fixed order
__global__ void __launch_bounds__(256) walk_gw_kernel(const float* __restrict__ part, float* __restrict__ out, int parts, int count) {
  __shared__ double red[8][33];
  const int i = blockIdx.x * 32 + threadIdx.x;
  double v = 0.;
  if (i < count) {
#pragma unroll 4
    for (int b = threadIdx.y; b < parts; b += 8) v += __ldg(part + (int64_t)b * count + i);
  }
  red[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.y == 0 && i < count) {
#pragma unroll
    for (int k = 1; k < 8; ++k) v += red[k][threadIdx.x];
    out[i] = static_cast<float>(v);
  }
}

// ---- adjoint -------------------------------------------------------------------------------------------------------------
// A CTA is the warps of a node's channels and halves.  H[cell] = sum_t scale[t] G[row[t]] in registers once per node, per edge
// a dot product over the lane's cells; the lanes' parts of BATCH stages go through shared memory and are added up by the CTA.
constexpr int BATCH = 4;

template <int V, int CC, bool MIXED>
struct GradSource {
  const float* g;
  const float* ws;
  float gv[V];
  template <int K> __device__ __forceinline__ void open() {
    if (MIXED) ldg_lane<V>(gv, g + K * CC);
  }
  template <int R, int K, int P> __device__ __forceinline__ void row(float (&v)[V]) {
    if constexpr (MIXED) {
      ld_lane<V>(v, ws + P * CC);
#pragma unroll
      for (int k = 0; k < V; ++k) v[k] *= gv[k];
    } else {
      ldg_lane<V>(v, g + R * CC);
    }
  }
};

template <class S, int V, int EPW, int CC, bool MIXED>
struct InnerShared {
  using R = Ring<S, V, EPW, CC, false>;
  static constexpr int NW = CC / R::CW * S::HALVES;                                      // warps of a CTA
  static constexpr int SC = S::HALVES * S::TH, WS = MIXED ? S::P * CC : 0;
  static constexpr int RINGS = NW * DEPTH * R::SLOT, PART = S::DY * 36, RED = BATCH * NW * PART;
  static constexpr size_t BYTES = sizeof(float) * (SC + WS + RINGS + RED);
  static constexpr int WARPS = S::NC * V > 96 ? 12 : S::NC * V > 64 ? 16 : 20, CTAS = WARPS / NW > 0 ? WARPS / NW : 1;
};

template <class S, int V, int EPW, int CC, bool MIXED>
__global__ void __launch_bounds__((32 * InnerShared<S, V, EPW, CC, MIXED>::NW), (InnerShared<S, V, EPW, CC, MIXED>::CTAS)) walk_inner_kernel(WalkArgs a) {
  using SH = InnerShared<S, V, EPW, CC, MIXED>;
  using R = typename SH::R;
  constexpr int CW = R::CW, NW = SH::NW, NT = 32 * NW;
  extern __shared__ __align__(16) float shared[];
  float* sc = shared;
  float* ws = sc + SH::SC;
  float* rings = ws + SH::WS;
  float* red = rings + SH::RINGS;       // [BATCH][NW][DY][36]: lanes' parts, rows of 32 padded so that eight rows' pieces of 16 bytes differ in banks
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = S::HALVES == 2 ? warp & 1 : 0, chunk = S::HALVES == 2 ? warp >> 1 : warp;
  const int channel0 = chunk * CW, ch = lane % R::LPE * V;

  for (int i = tid; i < SH::SC; i += NT) {
    const int t = S::order(i);
    sc[i] = t >= 0 ? __ldg(a.scale + t) : 0.f;
  }
  for (int i = tid; i < SH::WS; i += NT) ws[i] = __ldg(a.w + i);
  const int2 share = share_of_nodes<S::NC * V + 60, S::TH * V + 100>(a.ptr, a.n_out, blockIdx.x, gridDim.x, lane);
  const int64_t d0 = share.x;
  const int nd = share.y;
  __syncthreads();
  if (nd == 0) return;
  const int64_t* ptr = a.ptr + d0;
  const int64_t e0 = __ldg(ptr);
  const int ne = (int)(__ldg(ptr + nd) - e0);
  R ring(a, rings + warp * (DEPTH * R::SLOT), lane, half, channel0, e0, ne);
  ring.start();

  float h[S::NC][V];
#pragma unroll
  for (int i = 0; i < S::NC; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) h[i][k] = 0.f;
  const float4* scales = reinterpret_cast<const float4*>(sc + half * S::TH);
  int d = -1, boundary = 0, next = (int)(__ldg(ptr + 1) - e0);
  auto next_node = [&]() __attribute__((always_inline)) {
    ++d;
    const int begin = boundary;
    boundary = next;
    next = d + 1 < nd ? (int)(__ldg(ptr + d + 2) - e0) : 0;
    if (boundary > begin) {
      GradSource<V, CC, MIXED> source{a.g + (d0 + d) * ((MIXED ? S::K : S::R) * CC) + channel0 + ch, ws + channel0 + ch};
      if (half == 0) S::template cells0<V>(h, scales, source);
      else S::template cells1<V>(h, scales, source);
    }
  };

  const int stages = (ne + EPW - 1) / EPW;
  for (int t0 = 0; t0 < stages; t0 += BATCH) {
    const int count = min(BATCH, stages - t0);
    for (int s = 0; s < count; ++s) {
      const int t = t0 + s;
      const float* xs = ring.stage(t);
      float ay[S::DY];
      auto dot = [&]() __attribute__((always_inline)) {
        if (half == 0) S::template dot0<V, CW>(ay, xs + ch, h);
        else S::template dot1<V, CW>(ay, xs + ch, h);
      };
      if constexpr (EPW == 1) {
        while (t >= boundary) next_node();
        dot();
      } else {
#pragma unroll
        for (int k = 0; k < S::DY; ++k) ay[k] = 0.f;
        const int mine = t * EPW + ring.sub, end = min(t * EPW + EPW, ne);
        for (int e = t * EPW; e < end;) {
          while (e >= boundary) next_node();
          const int to = min(boundary, end);
          if (mine >= e && mine < to) dot();
          __syncwarp();
          e = to;
        }
      }
      float* rd = red + (s * NW + warp) * SH::PART + lane;
#pragma unroll
      for (int k = 0; k < S::DY; ++k) rd[k * 36] = ay[k];
    }
    if (NW > 1) __syncthreads(); else __syncwarp();
    // two lanes an (edge, component), half the lanes' parts of every warp each; with half-warps an edge, each has its own
    constexpr int ROUND = S::DY <= 4 ? 4 : S::DY <= 8 ? 2 : 1, SLOTS = 16 / ROUND;
    for (int i = warp * ROUND; i < count; i += NW * ROUND) {
      const int s = i + lane / 2 / SLOTS, k = lane / 2 % SLOTS, part = lane & 1, edge = (t0 + s) * EPW + (EPW == 2 ? part : 0);
      const bool mine = s < count && k < S::DY && (EPW == 1 || edge < ne);
      float v = 0.f;
      if (mine) {
        const float* rd = red + s * NW * SH::PART + k * 36 + part * 16;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
          float4 q[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) q[j] = *reinterpret_cast<const float4*>(rd + w * SH::PART + 4 * j);
          v += (((q[0].x + q[0].y) + (q[0].z + q[0].w)) + ((q[1].x + q[1].y) + (q[1].z + q[1].w))) +
               (((q[2].x + q[2].y) + (q[2].z + q[2].w)) + ((q[3].x + q[3].y) + (q[3].z + q[3].w)));
        }
      }
      if (EPW == 1) v += __shfl_xor_sync(0xffffffffu, v, 1);
      if (mine && (EPW == 2 || part == 0)) a.out[(a.yidx ? __ldg(a.yidx + e0 + edge) : e0 + edge) * S::DY + k] = v;
    }
    if (NW > 1) __syncthreads(); else __syncwarp();
  }
}

// ---- launches ------------------------------------------------------------------------------------------------------------
// CTAs in x: one wave of those that fit the SMs, but no more groups of warps than nodes
template <class S, int V, int EPW, int MODE> int64_t sum_grid(int64_t n_out, int channels) {
  constexpr int CW = 32 / EPW * V, GROUPS = 4 / S::HALVES;
  const int64_t most = std::max<int64_t>(1, (int64_t)sm_count() * sum_ctas<S, V>(MODE) / (channels / CW));
  return std::max<int64_t>(1, std::min<int64_t>(most, ceil_div(n_out, GROUPS)));
}

template <class S, int V, int EPW, int CC, int MODE> int launch_sum(const WalkArgs& a, cudaStream_t s) {
  using SH = SumShared<S, V, EPW, CC, MODE>;
  auto kern = walk_sum_kernel<S, V, EPW, CC, MODE>;
  if (int rc = allow_shared(kern, SH::BYTES)) return rc;
  const unsigned grid = (unsigned)sum_grid<S, V, EPW, MODE>(a.n_out, a.C);
  kern<<<dim3(grid, a.C / SH::CW), 128, SH::BYTES, s>>>(a);
  if (int rc = check_launch("walk_sum_kernel")) return rc;
  if (MODE != MIX_GRAD) return EQT_OK;
  const int count = S::P * a.C;
  walk_gw_kernel<<<(unsigned)ceil_div(count, 32), dim3(32, 8), 0, s>>>(a.scratch, a.gw, (int)grid, count);
  return check_launch("walk_gw_kernel");
}

template <class S, int V, int EPW, int CC, bool MIXED> int launch_inner(const WalkArgs& a, cudaStream_t s) {
  using SH = InnerShared<S, V, EPW, CC, MIXED>;
  auto kern = walk_inner_kernel<S, V, EPW, CC, MIXED>;
  if (int rc = allow_shared(kern, SH::BYTES)) return rc;
  constexpr int64_t per_sm = std::min<int64_t>(SH::CTAS, 227 * 1024 / (SH::BYTES + 1024));
  static_assert(per_sm > 0, "a CTA's shared memory");
  const int64_t grid = std::min<int64_t>(a.n_out, sm_count() * per_sm);
  kern<<<(unsigned)grid, 32 * SH::NW, SH::BYTES, s>>>(a);
  return check_launch("walk_inner_kernel");
}

inline bool walk_channels(int c) { return c == 16 || (c > 0 && c % 32 == 0); }

// f(channels of a lane, edges of a warp, channels or 0) for a channel count
template <class S, class F> auto by_channels(int c, F f) {
  using std::integral_constant;
  constexpr bool narrow = S::NC <= 16;      // a lane has room for several channels' cells
  integral_constant<int, 1> one;
  if (c == 16) return f(one, integral_constant<int, 2>{}, integral_constant<int, 16>{});
  if (c == 32) return f(one, one, integral_constant<int, 32>{});
  if (c == 64) return f(integral_constant<int, narrow ? 2 : 1>{}, one, integral_constant<int, 64>{});
  if (c == 128) return f(integral_constant<int, narrow ? 4 : 1>{}, one, integral_constant<int, 128>{});
  return f(one, one, integral_constant<int, 0>{});
}

template <class S> int run_sum(const WalkArgs& a, cudaStream_t s) {
  return by_channels<S>(a.C, [&](auto v, auto epw, auto c) {
    if (!a.w) return launch_sum<S, v(), epw(), c(), ROWS>(a, s);
    return a.x ? launch_sum<S, v(), epw(), c(), MIX_GRAD>(a, s) : launch_sum<S, v(), epw(), c(), MIX>(a, s);
  });
}

template <class S> int run_inner(const WalkArgs& a, cudaStream_t s) {
  return by_channels<S>(a.C, [&](auto v, auto epw, auto c) {
    if constexpr (c() == 0) return fail(EQT_ERR_UNSUPPORTED, "%d channels", a.C);
    else return a.w ? launch_inner<S, v(), epw(), c(), true>(a, s) : launch_inner<S, v(), epw(), c(), false>(a, s);
  });
}

}  // namespace

bool walk_supported(uint64_t key, bool with_weights, bool adjoint, int channels) {
  if (!walk_channels(channels) || (adjoint && channels != 16 && channels != 32 && channels != 64 && channels != 128)) return false;
#define EQT_TRY(S) if (key && key == (with_weights ? S::MIX_KEY : S::KEY)) return true;
  EQT_FOR_EACH_WALK(EQT_TRY)
#undef EQT_TRY
  return false;
}

bool walk_sizes(uint64_t key, bool with_weights, int entries, int rows, int d_feat, int d_y) {
#define EQT_TRY(S) \
  if (key && key == (with_weights ? S::MIX_KEY : S::KEY)) return entries == S::T && rows == S::R && d_feat == S::DF && d_y == S::DY;
  EQT_FOR_EACH_WALK(EQT_TRY)
#undef EQT_TRY
  return false;
}

int64_t walk_scratch_floats(uint64_t mix_key, int64_t n_out, int channels) {
  if (!walk_supported(mix_key, true, false, channels)) return -1;
#define EQT_TRY(S) \
  if (mix_key == S::MIX_KEY) \
    return by_channels<S>(channels, [&](auto v, auto epw, auto) { return sum_grid<S, v(), epw(), MIX_GRAD>(n_out, channels) * S::P * channels; });
  EQT_FOR_EACH_WALK(EQT_TRY)
#undef EQT_TRY
  return -1;
}

int walk_segment_sum(uint64_t key, const WalkArgs& a, cudaStream_t s) {
#define EQT_TRY(S) if (key == (a.w ? S::MIX_KEY : S::KEY)) return run_sum<S>(a, s);
  EQT_FOR_EACH_WALK(EQT_TRY)
#undef EQT_TRY
  return fail(EQT_ERR_UNSUPPORTED, "no straight-line code for this structure");
}

int walk_inner(uint64_t key, const WalkArgs& a, cudaStream_t s) {
#define EQT_TRY(S) if (key == (a.w ? S::MIX_KEY : S::KEY)) return run_inner<S>(a, s);
  EQT_FOR_EACH_WALK(EQT_TRY)
#undef EQT_TRY
  return fail(EQT_ERR_UNSUPPORTED, "no straight-line code for this structure");
}

}  // namespace eqt
