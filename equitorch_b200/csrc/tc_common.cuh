// Shared pieces of the tcgen05 kernels: mbarrier / TMA / UMMA / TMEM wrappers and tensor-map creation.
#pragma once

#include <cuda.h>

#include <mutex>

#include "common.cuh"

namespace eqt {
namespace tc {

constexpr int TC_THREADS = 320;
constexpr int KB = 32;                 // floats per k-block = one 128-byte swizzle row
constexpr int TILE_M = 128;
constexpr int TC_WAIT_SPINS = 1 << 21;

__device__ __forceinline__ uint32_t s32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void bar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(b)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(s32(b)), "r"(parity) : "memory");
  return ok != 0;
}
// Bounded wait that also gives up as soon as another role has raised the abort flag.
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, volatile int* abort_flag) {
  for (int i = 0; i < TC_WAIT_SPINS; ++i) {
    if (bar_try(b, parity)) return true;
    if ((i & 63) == 63) {
      if (*abort_flag) return false;
      __nanosleep(128);
    }
  }
  *abort_flag = 1;
  return false;
}

// After an expired wait: copies that may still be in flight to the buffers behind `bars` get a bounded chance to land before the
// CTA's shared memory is released (one of the two parities is the phase before, which is complete).
__device__ __forceinline__ void let_copies_land(uint64_t* bars, int count) {
  for (int i = 0; i < count; ++i)
    for (int ph = 0; ph < 2; ++ph)
      for (int t = 0; t < 1024 && !bar_try(&bars[i], ph); ++t) __nanosleep(256);
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(s32(dst)), "l"(map), "r"(s32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(s32(dst)), "l"(map), "r"(s32(bar)), "r"(c0), "r"(c1) : "memory");
}

// K-major, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart; descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_byte_addr) {
  return (uint64_t)((smem_byte_addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// kind::tf32, D = f32, A and B K-major, M = 128, N = n
__host__ __device__ inline uint32_t umma_idesc_tf32(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);
}
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// the same with the A operand in tensor memory (128 lanes x 8 columns of 32 bits, K along the columns)
__device__ __forceinline__ void umma_tf32_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// The same from the low words of K-major descriptors (address / 16; the high words are those of umma_desc), so that an issuing
// thread steps along K with one 32-bit addition of an immediate instead of building 64-bit words per MMA.
constexpr uint32_t UMMA_DESC_HI = (1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t umma_lo(uint32_t smem_byte_addr) { return ((smem_byte_addr & 0x3FFFF) >> 4) | (1u << 16); }
template <bool ACCUMULATE>
__device__ __forceinline__ void umma_tf32_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %4};\n\tmov.b64 b, {%2, %4};\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], a, b, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "n"(UMMA_DESC_HI), "n"(ACCUMULATE ? 1 : 0) : "memory");
}
__device__ __forceinline__ void umma_tf32_ta_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tmov.b64 b, {%2, %5};\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], b, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(UMMA_DESC_HI) : "memory");
}
// Operands MN-major, 128-byte swizzle with 32-byte atoms (layout type 1, the only swizzled layout tcgen05 takes for 32-bit MN-major
// operands): 32 floats of M/N per 128-byte row, 4 reduction rows per 512-byte group (stride byte offset), the next 32 floats of M/N
// `lbo` bytes further.  The low words carry the leading byte offset.
constexpr uint32_t UMMA_DESC_MN32_HI = (512 >> 4) | (1u << 14) | (1u << 29);
__device__ __forceinline__ uint32_t umma_lo_mn32(uint32_t smem_byte_addr, uint32_t lbo_bytes) {
  return ((smem_byte_addr & 0x3FFFF) >> 4) | (((lbo_bytes >> 4) & 0x3FFF) << 16);
}
// A in tensor memory (128 lanes x 8 columns), B MN-major as above
__device__ __forceinline__ void umma_tf32_ta_mn32_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tmov.b64 b, {%2, %5};\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], b, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(UMMA_DESC_MN32_HI) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// round to nearest TF32 (10 mantissa bits); the result is a float whose 13 low mantissa bits are zero
__device__ __forceinline__ float rn_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

// x as two TF32 values, hi and what is left of it, both rounded to nearest, ties away, as cvt.rna.tf32 does, which runs at a quarter of
// the rate: with two of them per element the splitter warps were as long about a tile as its bytes took to arrive.  hi in integer
// arithmetic (a NaN that wraps around there keeps its lo); lo has at most 12 significant bits, the MMA reads the first 11, and lo (1 + 2^-11)
// is exact and carries into those whenever the twelfth is set.  Against the conversions, in otherwise the same kernels: weight gradient of
// 100k nodes 991 -> 872 us, its three products 2094 -> 2032, both segment sums 3877 -> 3740, the same values bit for bit.
__device__ __forceinline__ float hi_tf32(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }
__device__ __forceinline__ void split_tf32(float x, float& hi, float& lo) {
  hi = hi_tf32(x);
  lo = (x - hi) * 1.00048828125f;
}
__device__ __forceinline__ void split_tf32(const float4& v, float4& hi, float4& lo) {
  split_tf32(v.x, hi.x, lo.x);
  split_tf32(v.y, hi.y, lo.y);
  split_tf32(v.z, hi.z, lo.z);
  split_tf32(v.w, hi.w, lo.w);
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Epilogue store of a 32 x 32 accumulator block held one row per lane.  Written directly, every store instruction
// would touch 32 rows with 16 bytes each; the block goes through the warp's shared-memory patch (32 rows, pitch
// EPI_PITCH floats: 16-byte aligned rows, conflict-free in both directions) and leaves as eight instructions of four
// full 128-byte row segments.  Lane l then serves columns 4 (l % 8) .. +3 of rows 4 i + l / 8, i = 0..7: `orow[i]`
// points at that row's first served column (column offset included), bit i of `vmask` says whether the row exists.
constexpr int EPI_PITCH = 36;
constexpr int EPI_PATCH_BYTES = 4 * 32 * EPI_PITCH * 4;      // four epilogue warps
// `add`: onto what this thread stored there before
__device__ __forceinline__ void store_block_rows(float* patch, const float (&v)[32], int lane, float* const (&orow)[8],
                                                 unsigned vmask, int c0, int n_cols, bool add = false) {
  __syncwarp();                                 // the previous block has been read out of the patch
#pragma unroll
  for (int c = 0; c < 32; c += 4)
    *reinterpret_cast<float4*>(patch + lane * EPI_PITCH + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float4 t = *reinterpret_cast<const float4*>(patch + (i * 4 + (lane >> 3)) * EPI_PITCH + (lane & 7) * 4);
    if (!((vmask >> i) & 1) || c0 + (lane & 7) * 4 >= n_cols) continue;
    float4* to = reinterpret_cast<float4*>(orow[i] + c0);
    if (add) {
      const float4 o = *to;
      t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
    }
    *to = t;
  }
}

// lane i of the warp stores its 32 values to TMEM lane (base lane + i), columns [col, col + 32); the caller
// issues tcgen05.wait::st before signalling anybody
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
        "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])),
        "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])),
        "r"(__float_as_uint(v[11])), "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
        "r"(__float_as_uint(v[15])), "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])),
        "r"(__float_as_uint(v[19])), "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])),
        "r"(__float_as_uint(v[23])), "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])),
        "r"(__float_as_uint(v[27])), "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])),
        "r"(__float_as_uint(v[31]))
      : "memory");
}

// the same with 16 values
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
        "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
        "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
        "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
}

// ---- host side ---------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  });
  return fn;
}

inline int make_map(CUtensorMap* map, const float* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
             const cuuint32_t* box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return fail(EQT_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  // The encoder is a driver call and needs a current context; on a thread that has made no runtime call yet (an
  // autograd worker whose first operation is this one) there is none until the runtime binds the primary context.
  // cudaSetDevice does that and, unlike cudaFree(0), is legal while a stream is being captured.
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
  cuuint32_t ones[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<float*>(base), dims,
                   strides_bytes, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(EQT_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return EQT_OK;
}

using ::eqt::sm_count;   // per-device SM count (common.cuh)

}  // namespace tc
}  // namespace eqt
