// Product of two channelled operands with full channel mixing ('uvw' TensorProduct), float32, weights shared by the batch,
// degrees up to 2, 16 or 32 channels a side:
//
//   out[n, M, w] = sum_p sum_(M1, M2) cg_p[M, M1, M2] sum_(u, v) x1[n, M1, u] x2[n, M2, v] W[p, u, v, w]
//
// The two-step form writes an intermediate of one (C1 x C2) block per sample and row (290 MB for 2000 samples, l_max 2, 32
// channels) and reads it five more times over forward and backward.  Nothing of it is needed: per path the sum over one
// operand's channels is a GEMM whose other side are the weights alone,
//
//   Z[n, c, (i, j)] = sum_k f[n, c, k] W[p, i, k, j]        rows (sample, component of f), N = (i, j), K = channels of f
//   out[n, a, j]   += sum_i (sum_b cg[a, b, c] s[n, b, i]) Z[n, c, (i, j)]
//
// and the second line is a handful of multiply-adds per accumulator element that the epilogue does on the way out of tensor
// memory.  Every derivative is of the same kind with the roles of the three operands exchanged:
//   output        s = x1 (i = u), f = x2 (k = v), j = w          gradient of x1   s = x2 (i = v), f = g (k = w), j = u
//   gradient of x2   s = x1 (i = u), f = g (k = w), j = v
// so one kernel serves all three; the weight gradient is a GEMM over the samples with a generated operand (below).
//
// uvw_contract_kernel: a CTA takes 128 samples, one irrep of f and a range of the channels i (in groups of 128 / J, so that an
// MMA is 128 columns wide), for all paths of that irrep.  f is split into TF32 big / small tiles in shared memory once, the
// packed weights stream through two stages, and the accumulators are four slots of 128 columns (one component of one path and
// channel group each), which lets the MMAs run ahead of the contraction.  Every path's sums over i meet in registers; the CTAs of a
// sample tile write partial outputs that a second launch adds up in a fixed order.
//   warps 0-7   split f, then contraction: a thread is one sample and half of the columns j
//   warp 8      bulk copies of the packed weights     warp 9   TMEM allocation and MMA issue
// Bound: the tensor array (three TF32 products, K = 8 per instruction) and, for the paths into l = 2, the multiply-adds.
// All waits are bounded; on expiry the abort flag is raised, every role leaves its loop, TMEM is freed and the status is set.
#include <algorithm>
#include <vector>

#include "tc_common.cuh"

namespace eqt {
namespace {
using namespace tc;

// Two float32 values in one 64-bit register pair: packed multiply-adds (fma.rn.f32x2) take half the issue slots.
struct Two { unsigned long long v; };
__device__ __forceinline__ Two two(float x, float y) {
  Two r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void apart(const Two& t, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(t.v)); }
__device__ __forceinline__ Two fma2(const Two& a, const Two& b, const Two& c) {
  Two r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ Two mul2(const Two& a, const Two& b) {
  Two r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
template <int N> __device__ __forceinline__ void axpy(Two (&o)[N], float s, const Two (&x)[N]) {
  const Two k = two(s, s);
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = fma2(k, x[i], o[i]);
}
template <int N> __device__ __forceinline__ void times(Two (&o)[N], const Two (&a)[N], const Two (&b)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = mul2(a[i], b[i]);
}
template <int N> __device__ __forceinline__ void scaled(Two (&o)[N], float s, const Two (&x)[N]) {
  const Two k = two(s, s);
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = mul2(k, x[i]);
}

#include "generated/triple_specs.inc"

constexpr int COLS = 128;                  // columns of an accumulator slot: channels i of a group x J
constexpr int SLOTS = 4;
constexpr int MAX_GROUPS = 16;             // irreps of the contracted operand
constexpr int MAX_SEGMENTS = 128;
constexpr int CONTRACT_THREADS = 10 * 32;
constexpr int B_STAGES = 2;
constexpr int CHAIN = 160;                 // multiply-adds in a row into one output element (cut())

__host__ __device__ constexpr bool couples(int a, int b, int c) { return a <= b + c && b <= a + c && c <= a + b; }
// bytes of 128 rows split into big and small: two tiles of 128-byte rows, or [big | small] side by side in one
__host__ __device__ constexpr int split_bytes(int k) { return k > 16 ? 2 * 128 * 128 : 128 * 128; }
// byte offset of chunk c (four floats) of row r, big or small, inside such an image
__device__ __forceinline__ uint32_t split_at(int k, int r, int c, bool small) {
  const int chunk = k > 16 ? c : c + (small ? 4 : 0);
  return (k > 16 && small ? 128 * 128 : 0) + r * 128 + ((chunk ^ (r & 7)) << 4);
}
// The pairs of split_tf32 by the conversion instruction.  The contraction splits one tile while nothing else runs on the SM, so its
// quarter rate costs nothing there, and the loop is shorter: 1-2 us less a pass than in integer arithmetic, the same bits (32
// channels, contractions of 100 samples, l_max 1 29.5 -> 28.3 us, 511 samples, l_max 2 75.3 -> 73.1, 8000 samples 489 -> 479).  The
// weight gradient's row makers issue without a pause and are better off with split_tf32 (2000 samples, l_max 2 170 -> 167).
__device__ __forceinline__ void split_by_cvt(const float4 v, float4& hi, float4& lo) {
  hi = make_float4(rn_tf32(v.x), rn_tf32(v.y), rn_tf32(v.z), rn_tf32(v.w));
  lo = make_float4(rn_tf32(v.x - hi.x), rn_tf32(v.y - hi.y), rn_tf32(v.z - hi.z), rn_tf32(v.w - hi.w));
}

struct ContractJob {
  const float* s;                  // (ds, ci, padded n): transposed, so that the samples of a warp are one run
  const float* f;                  // (n, df, ck)
  float* out;                      // (slices, n, d_out, J): partial sums, or the output itself with one slice
  float* sum;                      // (n, d_out, J)
  const unsigned char* packed;     // (num_paths, ci / group, split_bytes(ck))
  const eqt_uvw_path* paths;
  int ds, df, d_out, ci, ck, slices;
  int first[MAX_GROUPS], count[MAX_GROUPS], offset[MAX_GROUPS], degree[MAX_GROUPS];   // per irrep of f: its paths, first component, l
};
struct Segment { short job, group, q0, q1; int slice; };       // channel groups [q0, q1) of one irrep of f
struct ContractLaunch {
  ContractJob job[2];
  Segment seg[MAX_SEGMENTS];
  int64_t n, pad;                  // samples, and that rounded up to whole tiles
  int segments, tiles;
  int* status;
};

// N columns of this thread's TMEM lane, not waited for
template <int N> __device__ __forceinline__ void tmem_request(uint32_t taddr, uint32_t (&r)[N]);
template <> __device__ __forceinline__ void tmem_request<8>(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
template <> __device__ __forceinline__ void tmem_request<16>(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// values of earlier requests, behind one wait
template <int N> __device__ __forceinline__ void tmem_arrived(uint32_t (&r)[N]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]) :: "memory");
}

struct Ring {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++s == stages) {
      s = 0;
      ph ^= 1;
    }
  }
};

struct ContractBars {
  uint64_t b_full[B_STAGES], b_empty[B_STAGES], full[SLOTS], empty[SLOTS];
};

// The contraction of one thread: one sample, columns [half * J / 2, (half + 1) * J / 2) of every channel, two side by side.
template <int J> struct Contraction {
  static constexpr int JH = J / 2, IQ = COLS / J;
  const ContractJob& job;
  ContractBars& bars;
  volatile int* ab;
  uint32_t taddr;            // TMEM lane of the thread's sample, first column of its half
  const float* s;            // the sample in the transposed operand
  int64_t pad;
  int q0, q1, lane;
  Ring slot;
  bool ok = true;

  // The accumulator of channel i + 1 and its coefficients are on their way while those of channel i are used.
  template <int LO, int LS, int LF, int C>
  __device__ __forceinline__ void column(Two (&acc)[2 * LO + 1][JH / 2], const float* sp) {
    if (!ok || !bar_wait(&bars.full[slot.s], slot.ph, ab)) { ok = false; return; }
    tc_fence_after();
    const uint32_t at = taddr + (uint32_t)(slot.s * COLS);
    const int64_t step = job.ci * pad;
    uint32_t z[JH];
    float next[2 * LS + 1];
    tmem_request<JH>(at, z);
#pragma unroll
    for (int b = 0; b < 2 * LS + 1; ++b) next[b] = __ldg(sp + b * step);
#pragma unroll
    for (int i = 0; i < IQ; ++i) {
      tmem_arrived<JH>(z);
      Two v[JH / 2];
      float now[2 * LS + 1];
#pragma unroll
      for (int j = 0; j < JH / 2; ++j) v[j] = two(__uint_as_float(z[2 * j]), __uint_as_float(z[2 * j + 1]));
#pragma unroll
      for (int b = 0; b < 2 * LS + 1; ++b) now[b] = next[b];
      if (i + 1 < IQ) {
        tmem_request<JH>(at + (i + 1) * J, z);
#pragma unroll
        for (int b = 0; b < 2 * LS + 1; ++b) next[b] = __ldg(sp + b * step + (i + 1) * pad);
      }
      CgTriple<LO, LS, LF>::template column<C, JH / 2>(acc, now, v);
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) bar_arrive(&bars.empty[slot.s]);
    slot.next(SLOTS);
  }

  template <int LO, int LS, int LF> __device__ __forceinline__ void path(Two (&acc)[2 * LO + 1][JH / 2], int offset_s) {
    if constexpr (couples(LO, LS, LF)) {
      const float* sp = s + ((int64_t)offset_s * job.ci + q0 * IQ) * pad;
      for (int q = q0; q < q1; ++q, sp += IQ * pad) {
        column<LO, LS, LF, 0>(acc, sp);
        if constexpr (LF > 0) {
          column<LO, LS, LF, 1>(acc, sp);
          column<LO, LS, LF, 2>(acc, sp);
        }
        if constexpr (LF > 1) {
          column<LO, LS, LF, 3>(acc, sp);
          column<LO, LS, LF, 4>(acc, sp);
        }
      }
    }
  }

  // all paths of an irrep of f into one output irrep; returns the path behind them
  template <int LO, int LF> __device__ __forceinline__ int block(int q, int end, float* out, bool store) {
    Two acc[2 * LO + 1][JH / 2];
#pragma unroll
    for (int a = 0; a < 2 * LO + 1; ++a)
#pragma unroll
      for (int j = 0; j < JH / 2; ++j) acc[a][j] = two(0.f, 0.f);
    const int offset_o = __ldg(&job.paths[q].offset_o);
    for (; q < end && ok && __ldg(&job.paths[q].offset_o) == offset_o; ++q) {
      const int offset_s = __ldg(&job.paths[q].offset_s);
      switch (__ldg(&job.paths[q].l_s)) {
        case 0: path<LO, 0, LF>(acc, offset_s); break;
        case 1: path<LO, 1, LF>(acc, offset_s); break;
        case 2: path<LO, 2, LF>(acc, offset_s); break;
      }
    }
    if (store && ok)
#pragma unroll
      for (int a = 0; a < 2 * LO + 1; ++a)
#pragma unroll
        for (int j = 0; j < JH; j += 4)
          *reinterpret_cast<ulonglong2*>(out + (offset_o + a) * J + j) = make_ulonglong2(acc[a][j / 2].v, acc[a][j / 2 + 1].v);
    return q;
  }

  template <int LF> __device__ __forceinline__ void run(int first, int end, float* out, bool store) {
    uint64_t written = 0;                      // components of the output that a path of this irrep reaches
    for (int q = first; q < end && ok;) {
      const int lo = __ldg(&job.paths[q].l_o);
      written |= ((uint64_t(1) << (2 * lo + 1)) - 1) << __ldg(&job.paths[q].offset_o);
      switch (lo) {
        case 0: q = block<0, LF>(q, end, out, store); break;
        case 1: q = block<1, LF>(q, end, out, store); break;
        default: q = block<2, LF>(q, end, out, store); break;
      }
    }
    if (store && ok)
      for (int a = 0; a < job.d_out; ++a)
        if (!((written >> a) & 1))
          for (int j = 0; j < JH; j += 4) *reinterpret_cast<float4*>(out + a * J + j) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
};

// The MMAs of a CTA, issued by one thread: `items` (path, channel group) images, `nf` components of f each.  Two components' slots take
// their MMAs in turn, because MMAs into one accumulator execute one after the other.
template <int K>
__device__ __forceinline__ void contract_issue(ContractBars& bars, volatile int* ab, unsigned char* base, unsigned char* b_base,
                                               uint32_t tmem, int items, int nf) {
  constexpr uint32_t SMALL = (K > 16 ? 128 * 128 : 64) / 16, STEP = 32 / 16, BYTES = split_bytes(K);
  const uint32_t idesc = umma_idesc_tf32(COLS);
  Ring st, slot;
  for (int it = 0; it < items; ++it, st.next(B_STAGES)) {
    if (!bar_wait(&bars.b_full[st.s], st.ph, ab)) return;
    const uint32_t b = umma_lo(s32(b_base + st.s * BYTES));
    for (int c = 0; c < nf; c += 2) {
      const bool two = c + 1 < nf;
      const Ring first = slot;
      Ring second = slot;
      second.next(SLOTS);
      if (!bar_wait(&bars.empty[first.s], first.ph ^ 1, ab)) return;
      if (two && !bar_wait(&bars.empty[second.s], second.ph ^ 1, ab)) return;
      tc_fence_after();
      const uint32_t d0 = tmem + (uint32_t)(first.s * COLS), d1 = tmem + (uint32_t)(second.s * COLS);
      const uint32_t a0 = umma_lo(s32(base + c * BYTES)), a1 = a0 + BYTES / 16;
      // the corrections first: the adder inside the tensor core truncates, and their sum is 2^-11 of the whole
#pragma unroll
      for (int q = 0; q < K / 8; ++q) {
        if (q == 0) umma_tf32_lo<false>(d0, a0, b + SMALL, idesc);
        else umma_tf32_lo<true>(d0, a0 + q * STEP, b + SMALL + q * STEP, idesc);
        if (two) {
          if (q == 0) umma_tf32_lo<false>(d1, a1, b + SMALL, idesc);
          else umma_tf32_lo<true>(d1, a1 + q * STEP, b + SMALL + q * STEP, idesc);
        }
        umma_tf32_lo<true>(d0, a0 + SMALL + q * STEP, b + q * STEP, idesc);
        if (two) umma_tf32_lo<true>(d1, a1 + SMALL + q * STEP, b + q * STEP, idesc);
      }
#pragma unroll
      for (int q = 0; q < K / 8; ++q) {
        umma_tf32_lo<true>(d0, a0 + q * STEP, b + q * STEP, idesc);
        if (two) umma_tf32_lo<true>(d1, a1 + q * STEP, b + q * STEP, idesc);
      }
      umma_commit(&bars.full[first.s]);
      if (two) umma_commit(&bars.full[second.s]);
      slot = second;
      if (two) slot.next(SLOTS);
    }
    umma_commit(&bars.b_empty[st.s]);
  }
}

template <int J>
__global__ void __launch_bounds__(CONTRACT_THREADS, 1) uvw_contract_kernel(const __grid_constant__ ContractLaunch p) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ ContractBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Segment seg = p.seg[blockIdx.x / p.tiles];
  const int64_t tile = blockIdx.x % p.tiles;
  const ContractJob& job = p.job[seg.job];
  const int k = job.ck, first = job.first[seg.group], count = job.count[seg.group];
  const int lf = job.degree[seg.group], nf = 2 * lf + 1;
  const uint32_t a_bytes = split_bytes(k), b_bytes = split_bytes(k);
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* b_base = base + (size_t)nf * a_bytes;

  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < B_STAGES; ++i) { bar_init(&bars.b_full[i], 1); bar_init(&bars.b_empty[i], 1); }
    for (int i = 0; i < SLOTS; ++i) { bar_init(&bars.full[i], 1); bar_init(&bars.empty[i], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&tmem_slot)), "r"(SLOTS * COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp < 8) {      // f of the tile, component by component: rows are samples, rows past the batch are zero
    const int quads = k / 4, per_row = nf * quads;
    const float* f = job.f + (int64_t)job.offset[seg.group] * k;
    for (int i = tid; i < 128 * per_row; i += 256) {
      const int r = i / per_row, rest = i - r * per_row, c = rest / quads, ch = rest - c * quads;
      const int64_t n = tile * 128 + r;
      float4 hi, lo;
      split_by_cvt(n < p.n ? __ldg(reinterpret_cast<const float4*>(f + n * job.df * k) + rest) : make_float4(0.f, 0.f, 0.f, 0.f), hi, lo);
      *reinterpret_cast<float4*>(base + c * a_bytes + split_at(k, r, ch, false)) = hi;
      *reinterpret_cast<float4*>(base + c * a_bytes + split_at(k, r, ch, true)) = lo;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic writes -> visible to tcgen05.mma
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* ab = &abort_flag;
  const int groups = job.ci * J / COLS;          // channel groups of a path

  if (warp == 8) {
    // ---------------- packed weights ----------------
    if (lane == 0) {
      Ring st;
      bool ok = true;
      for (int q = first; q < first + count && ok; ++q)
        for (int g = seg.q0; g < seg.q1; ++g, st.next(B_STAGES)) {
          if (!bar_wait(&bars.b_empty[st.s], st.ph ^ 1, ab)) { ok = false; break; }
          bar_expect_tx(&bars.b_full[st.s], b_bytes);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           s32(b_base + st.s * b_bytes)), "l"(job.packed + ((int64_t)q * groups + g) * b_bytes), "r"(b_bytes),
                       "r"(s32(&bars.b_full[st.s])) : "memory");
        }
    }
  } else if (warp == 9) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const int items = count * (seg.q1 - seg.q0);
      if (k > 16) contract_issue<32>(bars, ab, base, b_base, tmem, items, nf);
      else contract_issue<16>(bars, ab, base, b_base, tmem, items, nf);
    }
  } else {
    // ---------------- contraction ----------------
    const int quarter = warp & 3, half = warp >> 2;
    const int64_t n = tile * 128 + quarter * 32 + lane;
    Contraction<J> w{job, bars, ab, tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * (J / 2)), job.s + n, p.pad,
                     seg.q0, seg.q1, lane};
    float* out = job.out + (((int64_t)seg.slice * p.n + min(n, p.n - 1)) * job.d_out) * J + half * (J / 2);
    switch (lf) {
      case 0: w.template run<0>(first, first + count, out, n < p.n); break;
      case 1: w.template run<1>(first, first + count, out, n < p.n); break;
      default: w.template run<2>(first, first + count, out, n < p.n); break;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(SLOTS * COLS) : "memory");
  }
  if (abort_flag && tid == 0) {
    atomicExch(p.status, 2);
    let_copies_land(bars.b_full, B_STAGES);
  }
}

// What a contraction reads, one slice of the grid per job and kind.  Weights of every (path, channel group) as the image that a
// stage holds: row (i, j) of the group, K = k, scaled, split and swizzled; a thread writes four k of one row.  And s with the
// samples last, through shared memory in blocks of 32 x 32 (rows past the batch are zero).
struct PackJob {
  const eqt_uvw_path* paths;
  unsigned char* packed;
  int64_t si, sk, sj, sp;          // strides of the weights: i, k, j, path
  int ci, ck, cj, num_paths;
  const float* s;                  // (n, columns)
  float* st;                       // (columns, pad)
  int columns;
};
struct PackLaunch { PackJob job[2]; const float* w; int64_t n, pad; };
__global__ void __launch_bounds__(256) uvw_pack_kernel(const __grid_constant__ PackLaunch p) {
  const PackJob& job = p.job[blockIdx.y / 2];
  if (blockIdx.y & 1) {
    __shared__ float block[32][33];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t across = ceil_div(job.columns, 32), blocks = across * (p.pad / 32);
    for (int64_t t = blockIdx.x; t < blocks; t += gridDim.x) {
      const int64_t n0 = t / across * 32;
      const int c0 = (int)(t % across) * 32;
      __syncthreads();
      for (int r = y; r < 32; r += 8) block[r][x] = n0 + r < p.n && c0 + x < job.columns ? __ldg(job.s + (n0 + r) * job.columns + c0 + x) : 0.f;
      __syncthreads();
      for (int r = y; r < 32; r += 8)
        if (c0 + r < job.columns) job.st[(int64_t)(c0 + r) * p.pad + n0 + x] = block[x][r];
    }
    return;
  }
  const int quads = job.ck / 4, iq = COLS / job.cj, groups = job.ci / iq;
  const int64_t total = (int64_t)job.num_paths * groups * quads * COLS;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int row = (int)(t % COLS), ch = (int)(t / COLS % quads);
    const int64_t image = t / COLS / quads;
    const int q = (int)(image / groups), g = (int)(image % groups), i = g * iq + row / job.cj, j = row % job.cj;
    const float scale = __ldg(&job.paths[q].scale);
    const float* w = p.w + __ldg(&job.paths[q].weight) * job.sp + i * job.si + j * job.sj + (int64_t)ch * 4 * job.sk;
    float4 hi, lo;
    split_tf32(make_float4(__ldg(w) * scale, __ldg(w + job.sk) * scale, __ldg(w + 2 * job.sk) * scale, __ldg(w + 3 * job.sk) * scale), hi, lo);
    unsigned char* to = job.packed + image * split_bytes(job.ck);
    *reinterpret_cast<float4*>(to + split_at(job.ck, row, ch, false)) = hi;
    *reinterpret_cast<float4*>(to + split_at(job.ck, row, ch, true)) = lo;
  }
}

struct SumLaunch { const float* from[2]; float* to[2]; int64_t quads[2]; int slices[2]; };
__global__ void __launch_bounds__(256) uvw_sum_kernel(const __grid_constant__ SumLaunch p) {
  const int job = blockIdx.y;
  const float4* from = reinterpret_cast<const float4*>(p.from[job]);
  const int64_t quads = p.quads[job];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < quads; i += (int64_t)gridDim.x * blockDim.x) {
    float4 v = __ldg(from + i);
    for (int s = 1; s < p.slices[job]; ++s) {
      const float4 u = __ldg(from + s * quads + i);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    reinterpret_cast<float4*>(p.to[job])[i] = v;
  }
}

bool channels_fit(int c) { return c == 16 || c == 32; }

int check_role(const eqt_uvw_role& r) {
  if (!r.paths || r.num_paths <= 0 || !r.groups || r.num_groups <= 0 || r.ds <= 0 || r.df <= 0 || r.d_out <= 0)
    return fail(EQT_ERR_BAD_ARGUMENT, "incomplete role");
  if (!channels_fit(r.ci) || !channels_fit(r.ck) || !channels_fit(r.cj)) return fail(EQT_ERR_UNSUPPORTED, "16 or 32 channels a side");
  if (r.num_groups > MAX_GROUPS || r.d_out > 64) return fail(EQT_ERR_UNSUPPORTED, "too many irreps");
  int at = 0;
  for (int g = 0; g < r.num_groups; ++g) {
    const eqt_uvw_group& e = r.groups[g];
    if (e.l < 0 || e.l > TRIPLE_MAX_L || e.count < 0 || e.longest < (e.count > 0) || e.longest > e.count || e.offset < 0 || e.offset + 2 * e.l + 1 > r.df) return fail(EQT_ERR_BAD_ARGUMENT, "bad irrep %d", g);
    at += e.count;
  }
  return at == r.num_paths ? EQT_OK : fail(EQT_ERR_BAD_ARGUMENT, "the irreps list %d of %d paths", at, r.num_paths);
}

// Channel groups of an irrep are dealt to CTAs so that the longest CTA is as short as the SMs allow: the smallest bound on the
// accumulator slots of a CTA (components x paths x channel groups) whose CTAs fit one wave, or one CTA per irrep where
// the sample tiles alone fill the chip.  The multiply-adds into an output element are one chain, of which a CTA takes CHAIN at most (32
// channels, l_max 2, error of the operand gradients against 64 bits: chains of 320 2.6e-7, of 160 2.1e-7, the two-step form 2.25e-7;
// 20k samples 2840 -> 2980 us).  Longest first.  -1: one channel group alone is more than that, or too many CTAs a tile.
int cut(const eqt_uvw_role* roles, int jobs, int64_t tiles, ContractLaunch* L, int (&slices)[2]) {
  struct Item { int job, group, unit, quads, most; };        // most: channel groups of a CTA
  std::vector<Item> items;
  for (int j = 0; j < jobs; ++j)
    for (int g = 0; g < roles[j].num_groups; ++g) {
      const eqt_uvw_group& e = roles[j].groups[g];
      if (!e.count) continue;
      items.push_back({j, g, e.count * (2 * e.l + 1), roles[j].ci * roles[j].cj / COLS, CHAIN / (e.longest * (2 * e.l + 1) * (COLS / roles[j].cj))});
      if (items.back().most < 1) return -1;
    }
  const int64_t room = std::max<int64_t>((int64_t)items.size(), std::min<int64_t>(MAX_SEGMENTS, sm_count() / tiles));
  int bound = 0, worst = 0;
  for (const Item& i : items) { bound = std::max(bound, i.unit); worst = std::max(worst, i.unit * i.quads); }
  auto per = [&](const Item& i, int b) { return std::max(1, std::min({i.quads, i.most, b / i.unit})); };
  for (; bound < worst; ++bound) {
    int64_t need = 0;
    for (const Item& i : items) need += (i.quads + per(i, bound) - 1) / per(i, bound);
    if (need <= room) break;
  }
  int64_t need = 0;
  for (const Item& i : items) need += (i.quads + per(i, bound) - 1) / per(i, bound);
  if (need > MAX_SEGMENTS) return -1;
  slices[0] = slices[1] = 0;
  int count = 0;
  std::vector<std::pair<int, Segment>> segs;
  for (const Item& i : items) {
    const int parts = (i.quads + per(i, bound) - 1) / per(i, bound);
    for (int t = 0; t < parts; ++t) {
      const int q0 = i.quads * t / parts, q1 = i.quads * (t + 1) / parts;
      segs.push_back({(q1 - q0) * i.unit, Segment{(short)i.job, (short)i.group, (short)q0, (short)q1, slices[i.job]++}});
    }
  }
  std::stable_sort(segs.begin(), segs.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
  for (const auto& s : segs) {
    if (L) L->seg[count] = s.second;
    ++count;
  }
  return count;
}

int64_t packed_floats(const eqt_uvw_role& r) { return (int64_t)r.num_paths * (r.ci * r.cj / COLS) * split_bytes(r.ck) / 4; }

template <int J> int launch_contract(const ContractLaunch& L, size_t smem, cudaStream_t st) {
  if (int rc = allow_shared(uvw_contract_kernel<J>, 227 * 1024 - 1024)) return rc;
  uvw_contract_kernel<J><<<(unsigned)(L.segments * L.tiles), CONTRACT_THREADS, smem, st>>>(L);
  return check_launch("uvw_contract_kernel");
}

}  // namespace
}  // namespace eqt

extern "C" int64_t eqt_uvw_scratch_floats(const eqt_uvw_role* roles, int32_t jobs, int64_t n) {
  using namespace eqt;
  if (!roles || jobs < 1 || jobs > 2 || n <= 0) return -1;
  for (int j = 0; j < jobs; ++j)
    if (check_role(roles[j])) return -1;
  int slices[2];
  if (ceil_div(n, 128) * MAX_SEGMENTS > 0x7fffffffll || cut(roles, jobs, ceil_div(n, 128), nullptr, slices) < 0) return -1;
  int64_t need = 0;
  for (int j = 0; j < jobs; ++j)
    need += packed_floats(roles[j]) + ceil_div(n, 128) * 128 * roles[j].ds * roles[j].ci + (slices[j] > 1 ? slices[j] * n * roles[j].d_out * roles[j].cj : 0);
  return need;
}

extern "C" int eqt_uvw_contract(const eqt_uvw_role* roles, int32_t jobs, const float* const* s, const float* const* f, float* const* out,
                                const float* w, float* scratch, int64_t scratch_floats, int64_t n, int32_t* status, void* stream) {
  using namespace eqt;
  if (!roles || jobs < 1 || jobs > 2 || n < 0 || !s || !f || !out || !w || !status) return fail(EQT_ERR_BAD_ARGUMENT, "bad arguments");
  if (n == 0) return EQT_OK;
  const int64_t need = eqt_uvw_scratch_floats(roles, jobs, n);
  if (need < 0) return EQT_ERR_UNSUPPORTED;
  if (!scratch || scratch_floats < need) return fail(EQT_ERR_BAD_ARGUMENT, "scratch of %lld floats needed", (long long)need);
  if (jobs == 2 && roles[0].cj != roles[1].cj) return fail(EQT_ERR_UNSUPPORTED, "both products need the same number of output channels");
  uintptr_t bits = reinterpret_cast<uintptr_t>(scratch);
  for (int j = 0; j < jobs; ++j) {
    if (!s[j] || !f[j] || !out[j]) return fail(EQT_ERR_BAD_ARGUMENT, "NULL operand");
    bits |= reinterpret_cast<uintptr_t>(s[j]) | reinterpret_cast<uintptr_t>(f[j]) | reinterpret_cast<uintptr_t>(out[j]);
  }
  if (bits & 15u) return fail(EQT_ERR_UNSUPPORTED, "operands must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ContractLaunch L{};
  PackLaunch P{};
  SumLaunch S{};
  int slices[2];
  L.n = P.n = n; L.tiles = (int)ceil_div(n, 128); L.pad = P.pad = (int64_t)L.tiles * 128; L.status = status;
  L.segments = cut(roles, jobs, L.tiles, &L, slices);
  P.w = w;
  size_t smem = 0;
  int64_t at = 0, widest = 0, rows = 0;
  for (int j = 0; j < jobs; ++j) {
    const eqt_uvw_role& r = roles[j];
    ContractJob& c = L.job[j];
    c.f = f[j]; c.sum = out[j]; c.paths = r.paths;
    c.ds = r.ds; c.df = r.df; c.d_out = r.d_out; c.ci = r.ci; c.ck = r.ck; c.slices = slices[j];
    c.packed = reinterpret_cast<unsigned char*>(scratch + at);
    P.job[j] = PackJob{r.paths, reinterpret_cast<unsigned char*>(scratch + at), r.stride_i, r.stride_k, r.stride_j, r.stride_p,
                       r.ci, r.ck, r.cj, r.num_paths, s[j], nullptr, r.ds * r.ci};
    at += packed_floats(r);
    c.s = P.job[j].st = scratch + at;
    at += L.pad * r.ds * r.ci;
    widest = std::max({widest, (int64_t)r.num_paths * r.ci * r.cj * (r.ck / 4), L.pad * r.ds * r.ci / 4});
    int q = 0;
    for (int g = 0; g < r.num_groups; ++g) {
      c.first[g] = q; c.count[g] = r.groups[g].count; c.offset[g] = r.groups[g].offset; c.degree[g] = r.groups[g].l;
      q += r.groups[g].count;
      if (r.groups[g].count) smem = std::max(smem, (size_t)(2 * r.groups[g].l + 1 + B_STAGES) * split_bytes(r.ck));
    }
  }
  for (int j = 0; j < jobs; ++j) {
    ContractJob& c = L.job[j];
    S.quads[j] = n * roles[j].d_out * roles[j].cj / 4;
    S.slices[j] = slices[j];
    S.to[j] = c.sum;
    if (slices[j] > 1) {
      c.out = scratch + at;
      at += slices[j] * S.quads[j] * 4;
      rows = std::max(rows, S.quads[j]);
    } else {
      c.out = c.sum;
      S.quads[j] = 0;
    }
    S.from[j] = c.out;
  }
  uvw_pack_kernel<<<dim3(flat_grid(widest, 256), 2 * jobs), 256, 0, st>>>(P);
  if (int rc = check_launch("uvw_pack_kernel")) return rc;
  if (int rc = roles[0].cj == 32 ? launch_contract<32>(L, smem + 1024, st) : launch_contract<16>(L, smem + 1024, st)) return rc;
  if (rows) {
    uvw_sum_kernel<<<dim3(flat_grid(rows, 256), jobs), 256, 0, st>>>(S);
    if (int rc = check_launch("uvw_sum_kernel")) return rc;
  }
  return EQT_OK;
}

// ------------------------------------------------------------------------------------------
// Weight gradient
// ------------------------------------------------------------------------------------------
//   gW[p, i, k, j] = sum_(n, c) Q[(i, j), (n, c)] f[n, c, k],     Q = sum_(a, b) cg[a, b, c] s[n, b, i] g[n, a, j]
//
// A GEMM whose reduction runs over samples and components of f, with M = 128 pairs (i, j) of one path, N = channels of f.  A
// thread is one pair: it computes its row of Q from the two operands in shared memory, eight samples at a time, splits it and
// stores it to tensor memory, where the MMA reads it; f arrives as [big | small] tiles of 32 samples, so that one MMA of 2 K
// columns makes big * big and big * small, and one of K columns small * big.  An MMA waits for the one
// before it into the same accumulator, so even and odd k-steps and the two kinds of MMA have accumulators of their own, folded into
// float32 registers every 16 to 24 k-steps each (the adder of the tensor core truncates); and every instruction of the issuing
// thread counts, so the MMAs of a stage are straight-line code by the degree of f (one accumulator and a loop: 211 us at 2000 samples,
// l_max 2, 32 channels; four: 201 us; without the loop 167 us; a third stage changes nothing).  The work - (path, channel group) x chunks of 32 samples -
// is one line that is cut into equal costs, one range per SM; a range that ends inside a (path, channel group) leaves a partial sum,
// and a second launch adds the partial sums of each in order.
//   warps 0-7   rows of Q (two sets of four, alternating groups of eight samples)
//   warps 8-11  accumulators -> registers -> partial sums; warp 8 also TMEM allocation and MMA issue
//   warps 12-15 operands -> shared memory
// Bound: the multiply-adds of Q and its split.
namespace eqt {
namespace {

constexpr int CHUNK = 32;                  // samples of a stage
constexpr int W_STAGES = 2;
constexpr int W_LOADERS = 4;
constexpr int W_THREADS = (12 + W_LOADERS) * 32;
constexpr int MAX_UNITS = 640;             // (path, channel group) and one CTA an SM
constexpr int MAX_PIECES = 1024;

// Rows of 32 samples of s and g in shared memory: the 16-byte chunks of a row are permuted so that eight neighbouring rows (a
// phase of 16-byte reads) as well as rows 4 l + t for eight l (a store of the loaders) lie on different banks.
__device__ __forceinline__ int chunk_of(int row, int chunk) { return chunk ^ ((row ^ row >> 2) & 7); }
// Row of the tiles of f that holds channel ch: r & 7 differs between the float4 that a store spreads over the banks.
__host__ __device__ constexpr int f_row(int k, int ch) { return (ch >> 2) + (ch & 3) * (k / 4); }

struct WPiece { int unit, chunk0, chunk1; };                 // unit = path x channel group
struct WLaunch {
  const float *s, *f, *g;                  // (n, ds, ci), (n, df, ck), (n, d_out, J)
  float* partial;                          // (pieces, 128, ck)
  const eqt_uvw_path* paths;               // with offset_f and l_f
  int64_t n;
  int ds, df, d_out, ci, ck, groups;
  int* status;
  short cta[MAX_PIECES + 1];               // pieces [cta[b], cta[b + 1]) of CTA b
  WPiece piece[MAX_PIECES];
};

struct WBars { uint64_t full[W_STAGES], empty[W_STAGES], a_ready[4], a_free[4], d_full, d_free; };

__device__ __forceinline__ void tmem_put16(uint32_t taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
        "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
}

__host__ __device__ constexpr int fold_every(int lf) { return lf == 2 ? 2 : lf == 1 ? 4 : 8; }      // stages between folds
constexpr int A_COL0 = 192;                // TMEM: [even | odd k-steps: big, corrections][small * big, even | odd], then the A slots

struct WSmem {
  int s, g, b, stage;                      // byte offsets inside a stage; the tiles of f first (1024-byte aligned)
  __host__ __device__ WSmem(int k, int cj) {
    const int iq = COLS / cj;
    b = 0;
    s = 5 * 2 * k * 128;
    g = s + 5 * iq * CHUNK * 4;
    stage = (g + 5 * cj * CHUNK * 4 + 1023) / 1024 * 1024;
  }
};

template <int J> struct RowMaker {
  WBars& bars;
  volatile int* ab;
  const unsigned char* base;
  int stage_bytes, s_off, g_off;           // operands of a stage
  int i, j;                                // this thread's pair of channels
  uint32_t tmem;                           // TMEM lane of the warp, first column of the A slots
  int set, lane;
  Ring st;
  uint32_t a_phase = 0;                    // the set's two slots advance together

  template <int LO, int LS, int LF> __device__ __forceinline__ bool rows(int chunks) {
    if constexpr (couples(LO, LS, LF)) {
      constexpr int NO = 2 * LO + 1, NS = 2 * LS + 1, NF = 2 * LF + 1, IQ = COLS / J;
      for (int t = 0; t < chunks; ++t, st.next(W_STAGES), a_phase ^= 1) {
        if (!bar_wait(&bars.full[st.s], st.ph, ab)) return false;
        const unsigned char* stage = base + st.s * stage_bytes;
#pragma unroll 1
        for (int u = set; u < 4; u += 2) {
          if (!bar_wait(&bars.a_free[u], a_phase ^ 1, ab)) return false;
          tc_fence_after();
          Two q[2][NF][2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            Two s[NS][2], g[NO][2];
            const float4* sp = reinterpret_cast<const float4*>(stage + s_off);
            const float4* gp = reinterpret_cast<const float4*>(stage + g_off);
#pragma unroll
            for (int b = 0; b < NS; ++b) {
              const float4 v = sp[(b * IQ + i) * 8 + chunk_of(b * IQ + i, u * 2 + h)];
              s[b][0] = two(v.x, v.y); s[b][1] = two(v.z, v.w);
            }
#pragma unroll
            for (int a = 0; a < NO; ++a) {
              const float4 v = gp[(a * J + j) * 8 + chunk_of(a * J + j, u * 2 + h)];
              g[a][0] = two(v.x, v.y); g[a][1] = two(v.z, v.w);
            }
            CgTriple<LO, LS, LF>::template pair<2>(q[h], s, g);
          }
#pragma unroll
          for (int c = 0; c < NF; ++c) {
            float v[16];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 4; e += 2) {       // the MMA drops what of the small part is past TF32
                float x, y;
                apart(q[h][c][e / 2], x, y);
                v[h * 4 + e] = hi_tf32(x);
                v[h * 4 + e + 1] = hi_tf32(y);
                apart(fma2(two(v[h * 4 + e], v[h * 4 + e + 1]), two(-1.f, -1.f), q[h][c][e / 2]), v[8 + h * 4 + e], v[8 + h * 4 + e + 1]);
              }
            tmem_put16(tmem + (uint32_t)(u * 80 + c * 16), v);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
          __syncwarp();
          if (lane == 0) bar_arrive(&bars.a_ready[u]);
        }
        if (lane == 0) bar_arrive(&bars.empty[st.s]);
      }
    }
    return true;
  }
};

template <int J, int K>
__global__ void __launch_bounds__(W_THREADS, 1) uvw_wgrad_kernel(const __grid_constant__ WLaunch p) {
  constexpr int IQ = COLS / J;
  extern __shared__ unsigned char smem_raw[];
  __shared__ WBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int k = K;
  const WSmem L(k, J);
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (tid == 0) {
    abort_flag = 0;
    for (int i = 0; i < W_STAGES; ++i) { bar_init(&bars.full[i], W_LOADERS); bar_init(&bars.empty[i], 9); }      // makers + the MMAs' commit
    for (int i = 0; i < 4; ++i) { bar_init(&bars.a_ready[i], 4); bar_init(&bars.a_free[i], 1); }
    bar_init(&bars.d_full, 1);
    bar_init(&bars.d_free, 4);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* ab = &abort_flag;
  const int p0 = p.cta[blockIdx.x], p1 = p.cta[blockIdx.x + 1];

  if (warp < 8) {
    // ---------------- rows of Q ----------------
    const int quarter = warp & 3, row = quarter * 32 + lane;
    RowMaker<J> w{bars, ab, base, L.stage, L.s, L.g, row / J, row % J,
                  tmem + ((uint32_t)(quarter * 32) << 16) + A_COL0, warp >> 2, lane};
    for (int x = p0; x < p1; ++x) {
      const WPiece pc = p.piece[x];
      const eqt_uvw_path* path = p.paths + pc.unit / p.groups;
      const int chunks = pc.chunk1 - pc.chunk0;
      bool ok = true;
      switch (__ldg(&path->l_o) * 9 + __ldg(&path->l_s) * 3 + __ldg(&path->l_f)) {
#define EQT_CASE(LO, LS, LF) case LO * 9 + LS * 3 + LF: ok = w.template rows<LO, LS, LF>(chunks); break;
        EQT_CASE(0, 0, 0) EQT_CASE(0, 1, 1) EQT_CASE(0, 2, 2) EQT_CASE(1, 0, 1) EQT_CASE(1, 1, 0) EQT_CASE(1, 1, 1) EQT_CASE(1, 1, 2)
        EQT_CASE(1, 2, 1) EQT_CASE(1, 2, 2) EQT_CASE(2, 0, 2) EQT_CASE(2, 1, 1) EQT_CASE(2, 1, 2) EQT_CASE(2, 2, 0) EQT_CASE(2, 2, 1)
        EQT_CASE(2, 2, 2)
#undef EQT_CASE
      }
      if (!ok) break;
    }
  } else if (warp < 12) {
    // ---------------- MMA issue and accumulators -> partial sums ----------------
    // A fold covers up to fold_every() stages of one piece.
    const int quarter = warp & 3;
    const uint32_t wide = umma_idesc_tf32(2 * k), narrow = umma_idesc_tf32(k);
    Ring st;
    uint32_t a_phase = 0, d_phase = 0;
    // MMAs of a stage, issued by one thread; nf is odd, so that a stage begins with an even k-step again
    auto stage = [&](auto count, bool first) __attribute__((always_inline)) {
      constexpr int NF = decltype(count)::value;
      const uint32_t tiles = umma_lo(s32(base + st.s * L.stage));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!bar_wait(&bars.a_ready[u], a_phase, ab)) return false;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < NF; ++c) {
          const int step = u * NF + c, odd = step & 1;
          const uint32_t a = tmem + A_COL0 + u * 80 + c * 16, b = tiles + c * 2 * k * 128 / 16 + u * 2;
          const uint32_t more = step > 1 ? 1 : !first;
          umma_tf32_ta_lo(tmem + odd * (2 * k), a, b, wide, more);                 // big * [big | small]
          umma_tf32_ta_lo(tmem + 4 * k + odd * k, a + 8, b, narrow, more);         // small * big
        }
        umma_commit(&bars.a_free[u]);
      }
      umma_commit(&bars.empty[st.s]);
      return true;
    };
    auto issue = [&](int stages, int nf) {
      if (!bar_wait(&bars.d_free, d_phase ^ 1, ab)) return false;
      tc_fence_after();
      for (int t = 0; t < stages; ++t, st.next(W_STAGES), a_phase ^= 1) {
        if (!bar_wait(&bars.full[st.s], st.ph, ab)) return false;
        const bool done = nf == 5   ? stage(std::integral_constant<int, 5>(), t == 0)
                          : nf == 3 ? stage(std::integral_constant<int, 3>(), t == 0)
                                    : stage(std::integral_constant<int, 1>(), t == 0);
        if (!done) return false;
      }
      umma_commit(&bars.d_full);
      return true;
    };
    bool ok = true;
    for (int x = p0; x < p1 && ok; ++x) {
      const WPiece pc = p.piece[x];
      const int lf = __ldg(&p.paths[pc.unit / p.groups].l_f), every = fold_every(lf);
      float sum[k];
#pragma unroll
      for (int i = 0; i < k; ++i) sum[i] = 0.f;
      for (int t = pc.chunk0; t < pc.chunk1; t += every) {
        if (warp == 8) {
          int issued = lane == 0 ? (int)issue(min(every, pc.chunk1 - t), 2 * lf + 1) : 1;
          issued = __shfl_sync(0xffffffffu, issued, 0);
          if (!issued) { ok = false; break; }
        }
        if (!bar_wait(&bars.d_full, d_phase, ab)) { ok = false; break; }
        d_phase ^= 1;
        tc_fence_after();
        // every fold has at least four k-steps, so that all accumulators are written
        const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
        for (int o = 0; o < 6 * k; o += 32) {
          float v[32];
          tmem_ld32(at + o, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) sum[(o + i) % k] += v[i];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(&bars.d_free);
      }
      if (!ok) break;
      float* out = p.partial + ((int64_t)x * 128 + quarter * 32 + lane) * k;
#pragma unroll
      for (int i = 0; i < k; i += 4) *reinterpret_cast<float4*>(out + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
    }
  } else {
    // ---------------- operands -> shared memory ----------------
    // A lane has one float4 of every component for FP (GP) samples of f (g): neighbouring lanes a run of channels of few samples.
    constexpr int FQ = K / 4, GQ = J / 4, FP = FQ / 4, GP = GQ / 4, FN = 32 / FQ, GN = 32 / GQ, IV = IQ / 4;
    const int me = warp - 12;
    Ring st;
    bool ok = true;
    for (int x = p0; x < p1 && ok; ++x) {
      const WPiece pc = p.piece[x];
      const eqt_uvw_path* path = p.paths + pc.unit / p.groups;
      const int i0 = pc.unit % p.groups * IQ;
      const int ns = 2 * __ldg(&path->l_s) + 1, no = 2 * __ldg(&path->l_o) + 1, nf = 2 * __ldg(&path->l_f) + 1;
      const float* fp = p.f + (int64_t)__ldg(&path->offset_f) * K + lane % FQ * 4;
      const float* gp = p.g + (int64_t)__ldg(&path->offset_o) * J + lane % GQ * 4;
      const float* sp = p.s + (int64_t)__ldg(&path->offset_s) * p.ci + i0;
      for (int t = pc.chunk0; t < pc.chunk1; ++t, st.next(W_STAGES)) {
        const int64_t n0 = (int64_t)t * CHUNK;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 fv[FP][5], gv[GP][5], sv[2 * IV];
        // the loads of a stage are in flight before the wait for its buffer
#pragma unroll
        for (int h = 0; h < FP; ++h) {
          const int64_t n = n0 + (me * FP + h) * FN + lane / FQ;
          const float* from = fp + n * p.df * K;
#pragma unroll
          for (int c = 0; c < 5; ++c) fv[h][c] = n < p.n && c < nf ? __ldg(reinterpret_cast<const float4*>(from + c * K)) : zero;
        }
#pragma unroll
        for (int h = 0; h < GP; ++h) {
          const int64_t n = n0 + (me * GP + h) * GN + lane / GQ;
          const float* from = gp + n * p.d_out * J;
#pragma unroll
          for (int a = 0; a < 5; ++a) gv[h][a] = n < p.n && a < no ? __ldg(reinterpret_cast<const float4*>(from + a * J)) : zero;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {          // components me, me + 4 of s for the sample of the lane
          const int b = me + h * 4;
#pragma unroll
          for (int v = 0; v < IV; ++v)
            sv[h * IV + v] = n0 + lane < p.n && b < ns ? __ldg(reinterpret_cast<const float4*>(sp + ((n0 + lane) * p.ds + b) * p.ci) + v) : zero;
        }
        if (!bar_wait(&bars.empty[st.s], st.ph ^ 1, ab)) { ok = false; break; }
        unsigned char* stage = base + st.s * L.stage;
#pragma unroll
        for (int h = 0; h < FP; ++h) {
          const int n = (me * FP + h) * FN + lane / FQ;
#pragma unroll
          for (int c = 0; c < 5; ++c) {
            if (c >= nf) break;
            float4 hi, lo;
            split_tf32(fv[h][c], hi, lo);
            const float big[4] = {hi.x, hi.y, hi.z, hi.w}, small[4] = {lo.x, lo.y, lo.z, lo.w};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
              const int r = f_row(K, lane % FQ * 4 + m);             // rows [0, K) big, [K, 2 K) small; K is a multiple of 8
              float* to = reinterpret_cast<float*>(stage + c * 2 * K * 128 + r * 128 + (((n >> 2) ^ (r & 7)) << 4) + (n & 3) * 4);
              to[0] = big[m];
              to[K * 32] = small[m];
            }
          }
        }
        auto put = [&](int off, int row, int n, const float4& v) {
          float* to = reinterpret_cast<float*>(stage + off) + (n & 3);
          const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int m = 0; m < 4; ++m) to[(row + m) * CHUNK + chunk_of(row + m, n >> 2) * 4] = w[m];
        };
#pragma unroll
        for (int h = 0; h < GP; ++h)
#pragma unroll
          for (int a = 0; a < 5; ++a)
            if (a < no) put(L.g, a * J + lane % GQ * 4, (me * GP + h) * GN + lane / GQ, gv[h][a]);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int v = 0; v < IV; ++v)
            if (me + h * 4 < ns) put(L.s, (me + h * 4) * IQ + v * 4, lane, sv[h * IV + v]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // tiles of f: generic writes -> visible to tcgen05.mma
        __syncwarp();
        if (lane == 0) bar_arrive(&bars.full[st.s]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (abort_flag && tid == 0) atomicExch(p.status, 2);
}

// The same sums by float32 multiply-adds: a thread is a pair (i, j), with its Q in a register per component of f, K accumulators, and K
// totals that take the accumulators every F_CHUNK samples, so that no chain of additions is long.  Operands arrive as they lie
// in memory, a chunk ahead of their use.  Error of the norm against 64 bits, l_max 2, 32 channels, this | TF32 pairs | the two-step form:
// 1 sample 0.6 | 1.0 | 0.6e-7, 200 samples 1.5 | 3.6 | 2.6e-7, 511 samples 1.6 | 4.1 | 4.0e-7.
// Bound: multiply-adds and the broadcast reads of f (one of 16 bytes per two packed multiply-adds).  us, l_max 2, this | TF32 pairs: 511
// samples, 32 channels 61 | 51, 16 channels 13 | 15; 2000 samples, 32 channels 212 | 170, 16 channels 35 | 41.  Two pairs a thread,
// which halve those reads, spill: 227.
constexpr int F_CHUNK = 16;
constexpr int F_STAGES = 2;
constexpr int f_ctas(int k) { return k > 16 ? 3 : 4; }                  // an SM; four with 32 accumulators spill
__host__ __device__ constexpr int f_stage_bytes(int k, int cj) { return F_CHUNK * 5 * (COLS / cj + cj + k) * 4; }

template <int J, int K> struct PairSums {
  static constexpr int IQ = COLS / J;
  const WLaunch& p;
  unsigned char* smem;
  int tid, i0;
  Two total[K / 2];

  template <int LO, int LS, int LF> __device__ __forceinline__ void run(const eqt_uvw_path* path, int chunk0, int chunk1) {
    if constexpr (couples(LO, LS, LF)) {
      constexpr int NO = 2 * LO + 1, NS = 2 * LS + 1, NF = 2 * LF + 1;
      constexpr int SQ = NS * IQ / 4, GQ = NO * J / 4, FQ = NF * K / 4, PER = SQ + GQ + FQ;      // 16-byte pieces of a sample
      const float* sp = p.s + (int64_t)__ldg(&path->offset_s) * p.ci + i0;
      const float* gp = p.g + (int64_t)__ldg(&path->offset_o) * J;
      const float* fp = p.f + (int64_t)__ldg(&path->offset_f) * K;
      auto load = [&](int chunk) {               // samples past the batch are zero
        if (chunk < chunk1) {
          const uint32_t to = s32(smem + (chunk - chunk0) % F_STAGES * f_stage_bytes(K, J));
          for (int t = tid; t < F_CHUNK * PER; t += COLS) {
            const int u = t / PER, r = t - u * PER;
            const int64_t n = (int64_t)chunk * F_CHUNK + u, m = min(n, p.n - 1);
            const float* from = r < SQ ? sp + (m * p.ds + r / (IQ / 4)) * p.ci + r % (IQ / 4) * 4
                                : r < SQ + GQ ? gp + m * p.d_out * J + (r - SQ) * 4 : fp + m * p.df * K + (r - SQ - GQ) * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + t * 16), "l"(from), "r"(n < p.n ? 16 : 0) : "memory");
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      for (int c = 0; c < F_STAGES - 1; ++c) load(chunk0 + c);
      const int i = tid / J, j = tid % J;
      for (int chunk = chunk0; chunk < chunk1; ++chunk) {
        load(chunk + F_STAGES - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(F_STAGES - 1) : "memory");
        __syncthreads();
        const float* at = reinterpret_cast<const float*>(smem + (chunk - chunk0) % F_STAGES * f_stage_bytes(K, J));
        Two acc[K / 2];
#pragma unroll
        for (int m = 0; m < K / 2; ++m) acc[m] = two(0.f, 0.f);
#pragma unroll 1
        for (int u = 0; u < F_CHUNK; u += 2, at += 2 * PER * 4) {          // two samples side by side
          Two s[NS][1], g[NO][1], q[NF][1];
#pragma unroll
          for (int b = 0; b < NS; ++b) s[b][0] = two(at[b * IQ + i], at[PER * 4 + b * IQ + i]);
#pragma unroll
          for (int a = 0; a < NO; ++a) g[a][0] = two(at[SQ * 4 + a * J + j], at[PER * 4 + SQ * 4 + a * J + j]);
          CgTriple<LO, LS, LF>::template pair<1>(q, s, g);
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < NF; ++c) {
              float x, y;
              apart(q[c][0], x, y);
              const Two qq = h ? two(y, y) : two(x, x);
              const float4* f = reinterpret_cast<const float4*>(at + (h * PER + SQ + GQ) * 4 + c * K);
#pragma unroll
              for (int m = 0; m < K / 4; ++m) {
                const float4 v = f[m];
                acc[2 * m] = fma2(qq, two(v.x, v.y), acc[2 * m]);
                acc[2 * m + 1] = fma2(qq, two(v.z, v.w), acc[2 * m + 1]);
              }
            }
        }
#pragma unroll
        for (int m = 0; m < K / 2; ++m) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(total[m].v) : "l"(acc[m].v));
        __syncthreads();                         // the stage may be written again
      }
    }
  }
};

template <int J, int K>
__global__ void __launch_bounds__(COLS, f_ctas(K)) uvw_wgrad_f32_kernel(const __grid_constant__ WLaunch p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int p0 = p.cta[blockIdx.x], p1 = p.cta[blockIdx.x + 1];
  for (int x = p0; x < p1; ++x) {
    const WPiece pc = p.piece[x];
    const eqt_uvw_path* path = p.paths + pc.unit / p.groups;
    PairSums<J, K> w{p, smem_raw, (int)threadIdx.x, pc.unit % p.groups * (COLS / J)};
#pragma unroll
    for (int m = 0; m < K / 2; ++m) w.total[m] = two(0.f, 0.f);
    switch (__ldg(&path->l_o) * 9 + __ldg(&path->l_s) * 3 + __ldg(&path->l_f)) {
#define EQT_CASE(LO, LS, LF) case LO * 9 + LS * 3 + LF: w.template run<LO, LS, LF>(path, pc.chunk0, pc.chunk1); break;
      EQT_CASE(0, 0, 0) EQT_CASE(0, 1, 1) EQT_CASE(0, 2, 2) EQT_CASE(1, 0, 1) EQT_CASE(1, 1, 0) EQT_CASE(1, 1, 1) EQT_CASE(1, 1, 2)
      EQT_CASE(1, 2, 1) EQT_CASE(1, 2, 2) EQT_CASE(2, 0, 2) EQT_CASE(2, 1, 1) EQT_CASE(2, 1, 2) EQT_CASE(2, 2, 0) EQT_CASE(2, 2, 1)
      EQT_CASE(2, 2, 2)
#undef EQT_CASE
    }
    float sum[K];                                // columns in the order of the tensor-core kernel's
#pragma unroll
    for (int m = 0; m < K / 2; ++m) apart(w.total[m], sum[f_row(K, 2 * m)], sum[f_row(K, 2 * m + 1)]);
    float* out = p.partial + ((int64_t)x * COLS + threadIdx.x) * K;
#pragma unroll
    for (int m = 0; m < K; m += 4) *reinterpret_cast<float4*>(out + m) = make_float4(sum[m], sum[m + 1], sum[m + 2], sum[m + 3]);
  }
}

struct WSumLaunch {
  const float* partial;
  float* gw;                               // (paths, i, k, j) with the strides below
  const eqt_uvw_path* paths;
  int64_t si, sk, sj, sp;
  int ck, cj, groups, units;
  short first[MAX_UNITS + 1];              // pieces of unit u: [first[u], first[u + 1])
};
// gw of 32 pairs (i, j) of a unit: its pieces, each 32 K floats in a row, are dealt to lanes of 8 K threads and added up in 64 bits, the
// lanes' sums in order; through shared memory, so that the writes run along j.
__global__ void __launch_bounds__(1024) uvw_wgrad_sum_kernel(const __grid_constant__ WSumLaunch p) {
  extern __shared__ double red[];                // 4 values of every thread (one lane: none)
  __shared__ float tile[32][33];
  const int tid = threadIdx.x, quads = p.ck / 4, per = 32 * quads, lanes = blockDim.x / per, lane = tid / per, e = tid % per;
  const int unit = blockIdx.x / 4, row0 = blockIdx.x % 4 * 32, iq = COLS / p.cj;
  double v[4] = {0., 0., 0., 0.};
#pragma unroll 4
  for (int t = p.first[unit] + lane; t < p.first[unit + 1]; t += lanes) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(p.partial) + ((int64_t)t * COLS + row0) * quads + e);
    v[0] += u.x; v[1] += u.y; v[2] += u.z; v[3] += u.w;
  }
  if (lanes > 1) {
#pragma unroll
    for (int m = 0; m < 4; ++m) red[m * blockDim.x + tid] = v[m];
    __syncthreads();
  }
  const int q = unit / p.groups;
  if (lane == 0) {
    const double scale = __ldg(&p.paths[q].scale);
#pragma unroll
    for (int m = 0; m < 4; ++m) {                // column r of the accumulator: channel 4 (r % (K / 4)) + r / (K / 4)
      for (int t = 1; t < lanes; ++t) v[m] += red[m * blockDim.x + t * per + e];
      const int r = e % quads * 4 + m;
      tile[4 * (r % quads) + r / quads][e / quads] = (float)(v[m] * scale);
    }
  }
  __syncthreads();
  float* to = p.gw + __ldg(&p.paths[q].weight) * p.sp;
  for (int t = tid; t < 32 * p.ck; t += blockDim.x) {
    const int k = t / 32, row = row0 + t % 32, i = unit % p.groups * iq + row / p.cj, j = row % p.cj;
    to[i * p.si + k * p.sk + j * p.sj] = tile[k][t % 32];
  }
}

// Float32 multiply-adds where TF32 pairs would be further from 64 bits than the two-step form was: below 512 samples, and with 16 output
// channels, whose sums that form took on multiply-adds at any size (16 channels: 2.3e-7 against 3.4e-7 at 512 samples).  And where f
// has 16 channels, whose MMAs are half as wide: 2000 samples, l_max 2, 32 x 16 -> 32 channels 152 us on tensor cores, 1.7e-7 instead of 4.5e-7.
bool wgrad_f32(const eqt_uvw_role& r, int64_t n) { return n < 512 || r.cj == 16 || r.ck == 16; }

// The line of (path, channel group, chunk), cut into ranges of equal cost.  Cost of a chunk: instructions of a thread that makes rows.
// Returns the number of pieces, or (without L) the most that there can be.
int cut_wgrad(const eqt_uvw_role& r, const int32_t* degrees, int64_t n, WLaunch* L, WSumLaunch* S, int* ctas) {
  const bool f32 = wgrad_f32(r, n);
  const int64_t chunks = ceil_div(n, f32 ? F_CHUNK : CHUNK);
  const int groups = r.ci * r.cj / COLS, units = r.num_paths * groups;
  if (chunks > 0x7fffffff || units + std::min<int64_t>(sm_count(), units * ceil_div(n, CHUNK)) > MAX_UNITS) return -1;
  const int want = (int)std::min<int64_t>(std::min(sm_count() * (f32 ? f_ctas(r.ck) : 1), MAX_PIECES - units), units * chunks);
  if (!L) return units + want;
  auto cost = [&](int q) {
    const int no = 2 * degrees[3 * q] + 1, ns = 2 * degrees[3 * q + 1] + 1, nf = 2 * degrees[3 * q + 2] + 1;
    return (int64_t)(f32 ? 8 * no * ns + 2 * (no + ns) + nf * (6 * r.ck / 4 + 4) : 16 + 20 * nf + 6 * no * ns);
  };
  int64_t total = 0;
  for (int q = 0; q < r.num_paths; ++q) total += cost(q) * groups * chunks;
  // the current CTA ends where its share of the total does (steps of total / want without a division each); the last one takes what is left
  const int64_t share = total / want, rest = total % want;
  int64_t end = share, carry = rest, before = 0;       // before: cost of the units before the current one
  int pieces = 0, cta = 0;
  L->cta[0] = 0;
  for (int u = 0; u < units; ++u) {
    S->first[u] = (short)pieces;
    const int64_t c = cost(u / groups);
    for (int64_t at = 0; at < chunks;) {
      const int64_t upto = cta + 1 >= want ? chunks : std::min(chunks, (end - before + c / 2) / c);
      if (upto <= at) {                    // nothing of this unit fits the current CTA any more
        L->cta[++cta] = (short)pieces;
        end += share;
        carry += rest;
        if (carry >= want) {
          carry -= want;
          ++end;
        }
        continue;
      }
      L->piece[pieces++] = WPiece{u, (int)at, (int)upto};
      at = upto;
    }
    before += c * chunks;
  }
  S->first[units] = (short)pieces;
  while (cta < want) L->cta[++cta] = (short)pieces;
  *ctas = want;
  return pieces;
}

template <int J, int K> int launch_wgrad_tc(const WLaunch& L, int ctas, cudaStream_t st) {
  if (int rc = allow_shared(uvw_wgrad_kernel<J, K>, 160 * 1024)) return rc;
  uvw_wgrad_kernel<J, K><<<ctas, W_THREADS, (size_t)W_STAGES * WSmem(K, J).stage + 1024, st>>>(L);
  return check_launch("uvw_wgrad_kernel");
}
template <int J, int K> int launch_wgrad_f32(const WLaunch& L, int ctas, cudaStream_t st) {
  if (int rc = allow_shared(uvw_wgrad_f32_kernel<J, K>, 160 * 1024)) return rc;
  uvw_wgrad_f32_kernel<J, K><<<ctas, COLS, F_STAGES * f_stage_bytes(K, J), st>>>(L);
  return check_launch("uvw_wgrad_f32_kernel");
}

}  // namespace
}  // namespace eqt

extern "C" int64_t eqt_uvw_wgrad_scratch_floats(const eqt_uvw_role* role, const int32_t* degrees, int64_t n) {
  using namespace eqt;
  if (!role || !degrees || n <= 0 || check_role(*role)) return -1;
  const int pieces = cut_wgrad(*role, degrees, n, nullptr, nullptr, nullptr);
  return pieces < 0 ? -1 : (int64_t)pieces * 128 * role->ck;
}

extern "C" int eqt_uvw_wgrad(const eqt_uvw_role* role, const int32_t* degrees, const float* s, const float* f, const float* g, float* gw,
                             float* scratch, int64_t scratch_floats, int64_t n, int32_t* status, void* stream) {
  using namespace eqt;
  if (!role || !degrees || n <= 0 || !s || !f || !g || !gw || !scratch || !status) return fail(EQT_ERR_BAD_ARGUMENT, "bad arguments");
  if (int rc = check_role(*role)) return rc;
  for (int q = 0; q < 3 * role->num_paths; ++q)
    if (degrees[q] < 0 || degrees[q] > TRIPLE_MAX_L) return fail(EQT_ERR_BAD_ARGUMENT, "bad degree");
  if ((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(f) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(scratch)) & 15u)
    return fail(EQT_ERR_UNSUPPORTED, "operands must be 16-byte aligned");
  const eqt_uvw_role& r = *role;
  WLaunch L{};
  WSumLaunch S{};
  int ctas = 0;
  const int pieces = cut_wgrad(r, degrees, n, &L, &S, &ctas);
  if (pieces < 0) return fail(EQT_ERR_UNSUPPORTED, "too many paths");
  if (scratch_floats < (int64_t)pieces * 128 * r.ck) return fail(EQT_ERR_BAD_ARGUMENT, "scratch too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  L.s = s; L.f = f; L.g = g; L.partial = scratch; L.paths = r.paths; L.n = n;
  L.ds = r.ds; L.df = r.df; L.d_out = r.d_out; L.ci = r.ci; L.ck = r.ck; L.groups = r.ci * r.cj / COLS; L.status = status;
  const int rc = !wgrad_f32(r, n) ? launch_wgrad_tc<32, 32>(L, ctas, st)
                 : r.cj == 32     ? (r.ck == 32 ? launch_wgrad_f32<32, 32>(L, ctas, st) : launch_wgrad_f32<32, 16>(L, ctas, st))
                                  : (r.ck == 32 ? launch_wgrad_f32<16, 32>(L, ctas, st) : launch_wgrad_f32<16, 16>(L, ctas, st));
  if (rc) return rc;
  S.partial = scratch; S.gw = gw; S.paths = r.paths;
  S.si = r.stride_i; S.sk = r.stride_k; S.sj = r.stride_j; S.sp = r.stride_p;
  S.ck = r.ck; S.cj = r.cj; S.groups = L.groups; S.units = r.num_paths * L.groups;
  const int per = 8 * r.ck;                      // about three pieces a lane
  int lanes = 1;
  while (2 * lanes * per <= 1024 && 3 * lanes * S.units < pieces) lanes *= 2;
  uvw_wgrad_sum_kernel<<<(unsigned)(S.units * (COLS / 32)), per * lanes, lanes > 1 ? per * lanes * 32 : 0, st>>>(S);
  return check_launch("uvw_wgrad_sum_kernel");
}
