// Node-level channel mixing on the 5th-generation tensor cores (tcgen05, accumulators in TMEM).
//
// For one output irrep (a "block": `dim` components, `paths` coupling paths into it) the weight
// step of the layer is a plain GEMM
//
//     out[(node, m), co] = sum_{kk} A[(node, m), kk] * Bt[co, kk],      kk = (path, ci)
//
// because the intermediate rows of a fixed output component are contiguous in memory: row
// (node, m) of A is the slice S[node, in_row0 + m*paths : in_row0 + (m+1)*paths, :] of the
// per-node intermediate, K = paths * C_in floats long.  A is described to TMA as a 3-D tensor
// (kk, m, node) so that one box of (32 floats, dim, nodes_per_tile) lands in shared memory as up
// to 128 consecutive 128-byte rows in the 128B-swizzled K-major layout tcgen05.mma reads.
//
// Precision: float32 results are required to 1e-5, which a single TF32 product (10 mantissa
// bits) cannot give.  Each operand is split as x = big + small with big = x rounded to the 10
// mantissa bits of TF32 and small = x - big rounded to as many (split_tf32), and three
// kind::tf32 MMAs accumulate big*big + big*small + small*big in float32 in TMEM; the dropped
// small*small term is below 2^-22 relative.  The weights are split once on the host side of the
// call, the activations by four "splitter" warps between the TMA arrival and the MMA issue.
//
// Roles inside a CTA of 10 warps (one persistent CTA per SM, tiles of up to 128 (node, m) rows):
//   warp 0      TMA producer (one elected lane), ring of `stages` k-blocks of 32 floats
//   warp 1      TMEM allocation, MMA issue (one elected lane), tcgen05.commit to free stages
//   warps 2-5   split A in place (big) and into a second buffer (small), fence to the async proxy
//   warps 6-9   epilogue: tcgen05.ld of the finished accumulator (double buffered in TMEM),
//               float4 stores of the valid rows
// Every wait on an mbarrier is bounded; on expiry the kernel raises the status flag, stops
// issuing work, frees its TMEM and returns.
#include <algorithm>
#include <initializer_list>
#include <vector>

#include "tc_common.cuh"

namespace eqt {
namespace {
using namespace tc;

constexpr int MAX_JOBS = 8;

struct alignas(64) JobDev {
  CUtensorMap map_a, map_bb, map_bs;        // A (3-D: k, m, node), B big / small (2-D: k, column)
  float* out;                               // first output element of (node 0, m 0)
  int64_t out_node_stride, out_m_stride;    // in floats; a row holds n_cols contiguous floats
  int64_t tile_begin;                       // position of the job's first tile in the launch's work list
  int dim;                                  // rows per node
  int npt;                                  // nodes per tile (npt * dim <= 128)
  int kblocks;                              // K / 32
  int n_cols;                               // N of this job
};

struct MixLaunch {
  JobDev job[MAX_JOBS];
  int64_t n;            // nodes
  int64_t total_tiles;
  int num_jobs;
  int max_cols;         // largest N among the jobs: fixes the stage layout and the TMEM split
  int stages;
  int tmem_cols;        // power of two >= 2 * max_cols (+ 64 per stage with a_in_tmem)
  int a_in_tmem;        // split A operand lives in tensor memory instead of shared memory
  int issuers;          // MMA issuer warps (2 when two accumulators per tile fit tensor memory)
  int* status;
};

}  // namespace
}  // namespace eqt

#include "mix_tc_kernel.inc"
#include "wgrad_tc_kernel.inc"
#include "vecmat_tc_kernel.inc"

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
namespace eqt {
namespace {

struct GemmJob {
  const float* a;            // first element of (node 0, m 0, k 0)
  int64_t K;                 // reduction length (multiple of 32); row (node, m) holds K contiguous floats
  int dim;                   // rows per node
  int64_t a_m_stride, a_node_stride;       // floats
  const float* b_big;        // (N, K) row-major
  const float* b_small;
  int N;                     // multiple of 16, <= 256
  float* out;
  int64_t out_node_stride, out_m_stride;   // floats
};

int launch_jobs(const GemmJob* jobs, int count, int64_t n, int* status, cudaStream_t st) {
  auto* kernel = mix_tc_kernel<false>;
  for (int q = 0; q < count; ++q)
    if (jobs[q].K / KB > MIX_CHUNK_KB) kernel = mix_tc_kernel<true>;
  if (int rc = allow_shared(kernel, 220 * 1024)) return rc;      // per device / context, so set on every call (a cheap host-side call)
  for (int first = 0; first < count; first += MAX_JOBS) {
    const int m = std::min(MAX_JOBS, count - first);
    MixLaunch L{};
    L.n = n; L.num_jobs = m; L.status = status;
    for (int q = 0; q < m; ++q) L.max_cols = std::max(L.max_cols, jobs[first + q].N);
    const uint32_t a_bytes = TILE_M * KB * 4, b_bytes = (uint32_t)L.max_cols * KB * 4;
    uint32_t stage_bytes = 2 * a_bytes + 2 * b_bytes;
    const size_t epi_bytes = EPI_PATCH_BYTES;                  // the epilogue warps' transpose patches behind the ring
    const size_t ring_budget = 220 * 1024 - 1024 - epi_bytes;
    L.stages = (int)std::min<size_t>(8, ring_budget / stage_bytes);
    {   // A through tensor memory when at least four stages of 64 columns fit beside the two accumulators
      const uint32_t sb = a_bytes + 2 * b_bytes;
      const int st = (int)std::min<size_t>(std::min<size_t>(8, ring_budget / sb), (512 - 2 * L.max_cols) / 64);
      if (st >= 4) {
        L.a_in_tmem = 1;
        L.stages = st;
        stage_bytes = sb;
      }
    }
    L.issuers = 1;
    if (L.a_in_tmem && 4 * L.max_cols + 64 * 4 <= 512) {      // two accumulators per tile and at least four A slots
      L.issuers = 2;
      L.stages = std::min(L.stages, (512 - 4 * L.max_cols) / 64);
    }
    if (L.stages < 2) return fail(EQT_ERR_UNSUPPORTED, "tile too wide for the shared-memory ring");
    // the epilogue reads accumulators in groups of 32 columns, so the second one is padded to a multiple of 32
    const int acc_cols = (2 * L.issuers - 1) * L.max_cols + (L.max_cols + 31) / 32 * 32;
    L.tmem_cols = 32;
    while (L.tmem_cols < std::max(acc_cols, 2 * L.issuers * L.max_cols + (L.a_in_tmem ? 64 * L.stages : 0))) L.tmem_cols <<= 1;
    int64_t total = 0;
    for (int q = 0; q < m; ++q) {
      const GemmJob& j = jobs[first + q];
      JobDev& d = L.job[q];
      d.out = j.out; d.out_node_stride = j.out_node_stride; d.out_m_stride = j.out_m_stride;
      d.dim = j.dim; d.npt = TILE_M / j.dim; d.kblocks = (int)(j.K / KB); d.n_cols = j.N;
      d.tile_begin = total;
      total += ceil_div(n, d.npt);
      {
        cuuint64_t dims[3] = {(cuuint64_t)j.K, (cuuint64_t)j.dim, (cuuint64_t)n};
        cuuint64_t strides[2] = {(cuuint64_t)j.a_m_stride * 4, (cuuint64_t)j.a_node_stride * 4};
        cuuint32_t box[3] = {KB, (cuuint32_t)j.dim, (cuuint32_t)d.npt};
        if (int rc = make_map(&d.map_a, j.a, 3, dims, strides, box)) return rc;
      }
      {
        cuuint64_t dims[2] = {(cuuint64_t)j.K, (cuuint64_t)j.N};
        cuuint64_t strides[1] = {(cuuint64_t)j.K * 4};
        cuuint32_t box[2] = {KB, (cuuint32_t)j.N};
        if (int rc = make_map(&d.map_bb, j.b_big, 2, dims, strides, box)) return rc;
        if (int rc = make_map(&d.map_bs, j.b_small, 2, dims, strides, box)) return rc;
      }
    }
    L.total_tiles = total;
    const unsigned grid = (unsigned)std::min<int64_t>(total, sm_count());
    kernel<<<grid, TC_THREADS + 32, (size_t)L.stages * stage_bytes + 1024 + epi_bytes, st>>>(L);
    if (int rc = check_launch("mix_tc_kernel")) return rc;
  }
  return EQT_OK;
}

int check_common(const void* a, const void* b, const void* c, const void* d, const eqt_mix_block* blocks, int32_t* status,
                 int64_t n, int32_t rows, int32_t comps, int32_t cin, int32_t cout, int32_t num_blocks) {
  if (n < 0 || rows <= 0 || comps <= 0 || cin <= 0 || cout <= 0 || num_blocks < 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (n == 0 || num_blocks == 0) return -1;
  if (!a || !b || !c || !d || !blocks || !status) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
       reinterpret_cast<uintptr_t>(d)) & 15u)
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core mix needs 16-byte aligned operands");
  if (n > 0x7fffffffll) return fail(EQT_ERR_UNSUPPORTED, "too many nodes for one TMA coordinate");
  return EQT_OK;
}

}  // namespace
}  // namespace eqt

extern "C" int eqt_mix_tc(const float* s, const float* w_big, const float* w_small, float* out, int64_t n,
                          int32_t rows, int32_t comps, int32_t cin, int32_t cout, const eqt_mix_block* blocks,
                          int32_t num_blocks, int32_t* status, void* stream) {
  using namespace eqt;
  if (int rc = check_common(s, w_big, w_small, out, blocks, status, n, rows, comps, cin, cout, num_blocks))
    return rc < 0 ? EQT_OK : rc;
  if (cin % KB != 0 || cout % 16 != 0 || cout > 256)
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core mix needs C_in %% 32 == 0 and C_out %% 16 == 0, C_out <= 256");
  std::vector<GemmJob> jobs;
  for (int b = 0; b < num_blocks; ++b) {
    const eqt_mix_block& blk = blocks[b];
    if (blk.dim <= 0 || blk.dim > TILE_M || blk.paths <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad block %d", b);
    GemmJob j{};
    j.K = (int64_t)blk.paths * cin; j.dim = blk.dim;
    j.a = s + (int64_t)blk.in_row0 * cin; j.a_m_stride = j.K; j.a_node_stride = (int64_t)rows * cin;
    j.b_big = w_big + blk.w_offset; j.b_small = w_small + blk.w_offset; j.N = cout;
    j.out = out + (int64_t)blk.out_row0 * cout; j.out_node_stride = (int64_t)comps * cout; j.out_m_stride = cout;
    jobs.push_back(j);
  }
  return launch_jobs(jobs.data(), (int)jobs.size(), n, status, static_cast<cudaStream_t>(stream));
}

extern "C" int eqt_mix_tc_transposed(const float* g, const float* w_big, const float* w_small, float* g_inter,
                                     int64_t n, int32_t rows, int32_t comps, int32_t cin, int32_t cout,
                                     const eqt_mix_block* blocks, int32_t num_blocks, int32_t* status, void* stream) {
  using namespace eqt;
  if (int rc = check_common(g, w_big, w_small, g_inter, blocks, status, n, rows, comps, cin, cout, num_blocks))
    return rc < 0 ? EQT_OK : rc;
  if (cout % KB != 0 || cin % 16 != 0)
    return fail(EQT_ERR_UNSUPPORTED, "transposed tensor-core mix needs C_out %% 32 == 0 and C_in %% 16 == 0");
  std::vector<GemmJob> jobs;
  for (int b = 0; b < num_blocks; ++b) {
    const eqt_mix_block& blk = blocks[b];
    if (blk.dim <= 0 || blk.dim > TILE_M || blk.paths <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad block %d", b);
    const int64_t width = (int64_t)blk.paths * cin;        // floats per (node, m) row of g_inter
    const int chunk_max = (256 / cin) > 0 ? (256 / cin) * cin : 0;
    if (chunk_max == 0) return fail(EQT_ERR_UNSUPPORTED, "C_in > 256");
    for (int64_t c0 = 0; c0 < width; c0 += chunk_max) {
      GemmJob j{};
      j.K = cout; j.dim = blk.dim;
      j.a = g + (int64_t)blk.out_row0 * cout; j.a_m_stride = cout; j.a_node_stride = (int64_t)comps * cout;
      j.b_big = w_big + blk.w_offset + c0 * cout; j.b_small = w_small + blk.w_offset + c0 * cout;
      j.N = (int)std::min<int64_t>(chunk_max, width - c0);
      j.out = g_inter + (int64_t)blk.in_row0 * cin + c0; j.out_node_stride = (int64_t)rows * cin; j.out_m_stride = width;
      jobs.push_back(j);
    }
  }
  return launch_jobs(jobs.data(), (int)jobs.size(), n, status, static_cast<cudaStream_t>(stream));
}

namespace eqt {
namespace {

// Launch of the weight-gradient kernel instance for the batch's output columns: one CTA per (block, split, M slice).
int launch_wgrad(const WgradBatch& b, size_t smem, cudaStream_t st) {
  cudaError_t e = b.n_cols <= 64
                      ? cudaFuncSetAttribute(wgrad_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)
                      : cudaFuncSetAttribute(wgrad_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  if (e != cudaSuccess) return fail(EQT_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  const WgradBlock& last = b.blk[b.count - 1];
  const unsigned grid = (unsigned)(last.cta_begin + last.splits * last.m_tiles);
  if (b.n_cols <= 64)
    wgrad_tc_kernel<64><<<grid, WgradCfg<64>::THREADS, smem, st>>>(b);
  else
    wgrad_tc_kernel<128><<<grid, WgradCfg<128>::THREADS, smem, st>>>(b);
  return check_launch("wgrad_tc_kernel");
}

// Launch shape of the weight-gradient GEMM of one block: reduction rows per tile, M tiles, node splits and the
// floats of scratch the per-CTA partial sums need.  Returns an error code for blocks that do not fit.
struct WgradShape {
  int npt, rows_pad, m_tiles, splits, issuers;
  size_t smem;
  int64_t K, tiles, need;
  void split(int s, int cout) { splits = s; need = (int64_t)s * m_tiles * 128 * cout; }
};
// Tiles of an accumulator before it is folded into registers: 320 terms.  A single issuer's accumulator has every tile of its CTA, and one of
// few tiles folds them in thirds, which keeps its error at that of two issuers with half of them each (l = 0..4, 128 channels, 1500
// nodes, six tiles: 7.0e-7 of the norm in one, 5.2e-7 with two issuers).
int wgrad_chunk(int rows_pad, int issuers, int64_t tiles) {
  const int64_t most = std::max(1, 320 / rows_pad);
  return (int)(issuers == 1 ? std::min<int64_t>(most, ceil_div(tiles, 3)) : most);
}

// Rows of a tile: no more than leave every SM one, but 32.
int wgrad_rows(const eqt_mix_block* blocks, int count, int64_t n, int cin) {
  int64_t rows = 0;
  for (int b = 0; b < count; ++b) rows += n * blocks[b].dim * ceil_div((int64_t)blocks[b].paths * cin, 128);
  return (int)std::min<int64_t>(96, std::max<int64_t>(32, ceil_div(ceil_div(rows, sm_count()), 8) * 8));
}
int wgrad_shape(const eqt_mix_block& blk, int b, int64_t n, int cin, int cout, int rows, WgradShape* w) {
  if (blk.dim <= 0 || blk.dim > TILE_M || blk.paths <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad block %d", b);
  WgradTile tile;
  if (!wgrad_tile(blk.dim, cout, &tile, rows) && !wgrad_tile(blk.dim, cout, &tile)) return fail(EQT_ERR_UNSUPPORTED, "irrep with %d components does not fit a reduction tile", blk.dim);
  w->npt = tile.npt; w->rows_pad = tile.rows_pad; w->smem = tile.smem; w->issuers = tile.issuers;
  w->K = (int64_t)blk.paths * cin;                               // M extent of this GEMM
  w->m_tiles = (int)ceil_div(w->K, 128);
  w->tiles = ceil_div(n, w->npt);
  w->split((int)std::max<int64_t>(1, std::min<int64_t>(w->tiles, sm_count() / w->m_tiles)), cout);
  return EQT_OK;
}

// Blocks of one launch share the SMs: another split for the block whose CTAs have the most tiles, while there are SMs.  A launch is then
// one wave of CTAs with about as many tiles each, where every block on all SMs made a wave a block: each with its own fill and
// drain, of one or two tiles a CTA on small batches (10k nodes, l_max 3, 64 channels 100 -> 82 us, 1000 nodes, l_max 2 22.3 -> 10.7).
// A wide layer has so many slices of M that its high degrees, with the fewest nodes a tile, would not get a second split in one wave and
// run alone at its end: two to four waves where that makes CTAs more even than it costs, each wave's fill and drain counted as six tiles.
void wgrad_share(WgradShape* w, int count, int cout) {
  const int sms = sm_count();
  int ctas = 0, best[WGRAD_MAX_BLOCKS];
  double even = 6;                                                  // tiles of a CTA if all were alike
  for (int b = 0; b < count; ++b) {
    w[b].split(1, cout);
    ctas += w[b].m_tiles;
    even += (double)w[b].tiles * w[b].m_tiles / sms;
  }
  double least = 1e300;
  for (int waves = 1; waves <= 4; ++waves) {
    int64_t longest = 0;
    for (;;) {
      int most = 0;
      for (int b = 1; b < count; ++b)
        if (w[b].tiles * w[most].splits > w[most].tiles * w[b].splits) most = b;
      longest = ceil_div(w[most].tiles, w[most].splits);
      if (ctas + w[most].m_tiles > waves * sms || w[most].splits >= w[most].tiles) break;
      ctas += w[most].m_tiles;
      w[most].split(w[most].splits + 1, cout);
    }
    const double cost = (double)ceil_div(ctas, sms) * (double)(longest + 6);
    if (cost < 0.97 * least) {
      least = cost;
      for (int b = 0; b < count; ++b) best[b] = w[b].splits;
    }
    if (cost < 1.13 * even) break;
  }
  for (int b = 0; b < count; ++b) w[b].split(best[b], cout);
}

// Tile of the indexed form: no more rows than leave every SM a tile, but 48 (600 samples, 32 columns, 7 tiles of 96 rows 7.8 us, 13 of 48 6.5).
bool outer_tile(int64_t n, int cols, int m_tiles, WgradTile* t) {
  const int64_t rows = ceil_div(ceil_div(n * std::max(m_tiles, 1), sm_count()), 8) * 8;
  return wgrad_tile(1, cols, t, (int)std::min<int64_t>(96, std::max<int64_t>(48, rows)));
}

// Splits of a product whose slices all have `tiles` tiles: as many waves of CTAs as leave the SMs least idle (32 slices: 4 splits are 128
// CTAs, 9 are 288 of 296: 100k samples 712 -> 654 us), a wave's fill and drain counted as six tiles.
int outer_splits(int64_t tiles, int m_tiles) {
  const int sms = sm_count();
  int best = 1;
  double least = 1e300;
  for (int waves = 1; waves <= 4; ++waves) {
    const int64_t s = std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)waves * sms / m_tiles));
    const double cost = (double)ceil_div(s * m_tiles, sms) * (double)(ceil_div(tiles, s) + 6);
    if (cost < least) { least = cost; best = (int)s; }
  }
  return best;
}

}  // namespace
}  // namespace eqt

extern "C" int64_t eqt_wgrad_tc_scratch_floats(int64_t n, int32_t cin, int32_t cout, const eqt_mix_block* blocks,
                                               int32_t num_blocks) {
  using namespace eqt;
  if (n < 0 || cin <= 0 || cout <= 0 || cin % 32 || cout % 32 || num_blocks < 0 || (num_blocks && !blocks)) return -1;
  // the sum over the blocks: with that much scratch all blocks run in one launch; eqt_wgrad_tc also works with the
  // largest block's need alone (one launch per block then)
  int64_t together = 0, alone = 0;
  std::vector<WgradShape> shapes(num_blocks);
  const int tile_rows = wgrad_rows(blocks, num_blocks, n, cin);
  for (int b = 0; b < num_blocks; ++b) {
    if (wgrad_shape(blocks[b], b, std::max<int64_t>(n, 1), cin, cout, tile_rows, &shapes[b])) return -1;
    alone = std::max(alone, shapes[b].need);
  }
  for (int b0 = 0; b0 < num_blocks; b0 += WGRAD_MAX_BLOCKS) wgrad_share(&shapes[b0], std::min(WGRAD_MAX_BLOCKS, num_blocks - b0), cout);
  for (const WgradShape& w : shapes) together += w.need;
  return std::max(together, alone);
}

extern "C" int eqt_wgrad_tc(const float* s, const float* g, float* gw_packed, float* scratch, int64_t scratch_floats,
                            int64_t n, int32_t rows, int32_t comps, int32_t cin, int32_t cout,
                            const eqt_mix_block* blocks, int32_t num_blocks, int32_t* status, void* stream) {
  using namespace eqt;
  if (int rc = check_common(s, g, gw_packed, scratch, blocks, status, n, rows, comps, cin, cout, num_blocks))
    return rc < 0 ? EQT_OK : rc;
  if (cin % 32 != 0 || cout % 32 != 0 || cout > 128)
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core weight gradient needs C_in %% 32 == 0, C_out %% 32 == 0, C_out <= 128");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // every block is checked before the first launch, so a refusal leaves gw_packed untouched
  std::vector<WgradShape> shapes(num_blocks);
  const int tile_rows = wgrad_rows(blocks, num_blocks, n, cin);
  for (int b = 0; b < num_blocks; ++b) {
    if (int rc = wgrad_shape(blocks[b], b, n, cin, cout, tile_rows, &shapes[b])) return rc;
    if (shapes[b].need > scratch_floats)
      return fail(EQT_ERR_BAD_ARGUMENT, "scratch too small: block %d needs %lld floats, %lld given", b,
                  (long long)shapes[b].need, (long long)scratch_floats);
  }
  // With scratch for every block at once, up to WGRAD_MAX_BLOCKS blocks share a launch (and one reduction launch);
  // otherwise the blocks run one after the other and reuse the scratch.
  std::vector<WgradShape> shared = shapes;
  int64_t total_need = 0;
  for (int b0 = 0; b0 < num_blocks; b0 += WGRAD_MAX_BLOCKS) wgrad_share(&shared[b0], std::min(WGRAD_MAX_BLOCKS, num_blocks - b0), cout);
  for (const WgradShape& w : shared) total_need += w.need;
  const int per_launch = total_need <= scratch_floats ? WGRAD_MAX_BLOCKS : 1;
  if (per_launch > 1) shapes = shared;
  for (int b0 = 0; b0 < num_blocks; b0 += per_launch) {
    const int count = std::min(per_launch, num_blocks - b0);
    WgradBatch B{};
    ReduceBatch R{};
    B.count = R.count = count;
    B.n = n; B.n_cols = R.cols = cout; B.status = status;
    size_t smem = 0;
    int cta = 0, most_splits = 0;
    int64_t scratch_at = 0, quads = 0;
    for (int q = 0; q < count; ++q) {
      const eqt_mix_block& blk = blocks[b0 + q];
      const WgradShape& w = shapes[b0 + q];
      WgradBlock& a = B.blk[q];
      a.dim = blk.dim; a.npt = w.npt; a.rows_pad = w.rows_pad; a.chunk_tiles = wgrad_chunk(w.rows_pad, w.issuers, ceil_div(w.tiles, w.splits));
      a.m_tiles = w.m_tiles; a.splits = w.splits; a.cta_begin = cta;
      a.partial = scratch + scratch_at;
      cta += w.splits * w.m_tiles;
      most_splits = std::max(most_splits, w.splits);
      smem = std::max(smem, w.smem);
      a.issuers = w.issuers;
      {
        cuuint64_t dims[3] = {(cuuint64_t)w.K, (cuuint64_t)blk.dim, (cuuint64_t)n};
        cuuint64_t strides[2] = {(cuuint64_t)w.K * 4, (cuuint64_t)rows * cin * 4};
        cuuint32_t box[3] = {128, (cuuint32_t)blk.dim, (cuuint32_t)w.npt};
        if (int rc = make_map(&a.map_s, s + (int64_t)blk.in_row0 * cin, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
      }
      {
        cuuint64_t dims[3] = {(cuuint64_t)cout, (cuuint64_t)blk.dim, (cuuint64_t)n};
        cuuint64_t strides[2] = {(cuuint64_t)cout * 4, (cuuint64_t)comps * cout * 4};
        cuuint32_t box[3] = {KB, (cuuint32_t)blk.dim, (cuuint32_t)w.npt};
        if (int rc = make_map(&a.map_g, g + (int64_t)blk.out_row0 * cout, 3, dims, strides, box,
                              CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B)) return rc;
      }
      R.blk[q].partial = a.partial; R.blk[q].out = gw_packed + blk.w_offset; R.blk[q].splits = w.splits;
      R.blk[q].padded_rows = (int64_t)w.m_tiles * 128; R.blk[q].begin = quads;
      quads += w.K * cout / 4;
      scratch_at += w.need;
    }
    R.total = quads;
    if (int rc = launch_wgrad(B, smem, st)) return rc;
    auto reduce = [&](auto* kernel, int warps) {
      kernel<<<(unsigned)ceil_div(quads, 32 * (REDUCE_WARPS / warps)), 32 * REDUCE_WARPS, 0, st>>>(R);
    };
    if (most_splits == 1) reduce(wgrad_reduce_batched_kernel<1>, 1);
    else if (most_splits == 2) reduce(wgrad_reduce_batched_kernel<2>, 2);
    else if (most_splits <= 4) reduce(wgrad_reduce_batched_kernel<4>, 4);
    else reduce(wgrad_reduce_batched_kernel<REDUCE_WARPS>, REDUCE_WARPS);
    if (int rc = check_launch("wgrad_reduce_batched_kernel")) return rc;
  }
  return EQT_OK;
}

// ------------------------------------------------------------------------------------------
// The reference's indexed products with shared weights on the same machinery
// ------------------------------------------------------------------------------------------
extern "C" int eqt_vecmat_tc_grouped(const float* x, const float* w, const int64_t* index2, const float* scale, float* w_big,
                                     float* w_small, float* out, int64_t n, int32_t rows1, int32_t cin, int32_t cout,
                                     int32_t num_out, int64_t slots, int32_t group, int32_t num_groups, const int32_t* group_rows,
                                     const int32_t* slot_entry, const int32_t* kb_begin, const int32_t* a_col, int32_t longest,
                                     int32_t* status, void* stream) {
  using namespace eqt;
  if (n < 0 || rows1 <= 0 || cin <= 0 || cout <= 0 || num_out < 0 || slots < 0 || group <= 0 || num_groups < 0)
    return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (n == 0 || num_out == 0 || num_groups == 0) return EQT_OK;
  if (!x || !w || !w_big || !w_small || !out || !kb_begin || !a_col || !status) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (group > 1 && (!group_rows || !slot_entry)) return fail(EQT_ERR_BAD_ARGUMENT, "groups of rows need their tables");
  if (!group_rows && num_groups != num_out) return fail(EQT_ERR_BAD_ARGUMENT, "one group per output row without a row table");
  if (cin % KB != 0 || cout % 16 != 0 || cout > 128 || (group > 1 && (cout % 32 != 0 || group * cout > 128)))
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core vecmat needs C_in %% 32 == 0, C_out %% 16 == 0, C_out <= 128 (all rows of a group)");
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(w_big) |
       reinterpret_cast<uintptr_t>(w_small)) & 15u)
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core vecmat needs 16-byte aligned operands");
  if (n > 0x7fffffffll || (int64_t)rows1 * cin > 0x7fffffffll || slots * cin > 0x7fffffffll)
    return fail(EQT_ERR_UNSUPPORTED, "operands too large for one TMA coordinate");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t ktot = slots * cin;
  const int n_cols = group * cout;
  if (slots > 0) {
    pack_vecmat_weights_kernel<<<flat_grid(ktot * n_cols, 256), 256, 0, st>>>(w, index2, scale, slot_entry, w_big, w_small, slots, group,
                                                                              cin, cout);
    if (int rc = check_launch("pack_vecmat_weights_kernel")) return rc;
  }
  VecmatLaunch L{};
  L.out = out; L.kb_begin = kb_begin; L.rows = group_rows; L.a_col = a_col; L.n = n; L.num_out = num_out; L.status = status;
  L.num_groups = num_groups; L.group = group; L.cout = cout; L.n_cols = n_cols;
  L.total_items = (int64_t)num_groups * ceil_div(n, TILE_M);
  const uint32_t stage_bytes = TILE_M * KB * 4 + 2u * (uint32_t)n_cols * KB * 4;
  L.bigs = group == 1 ? 2 : 1;
  L.chunk_kb = group == 1 ? VM_SHORT_CHUNK_KB : VM_CHUNK_KB;
  L.acc_sets = (L.bigs + 1) * n_cols <= 128 ? 2 : 1;       // at least four A slots stay free (two at 128 columns)
  const int acc_cols = L.acc_sets * (L.bigs + 1) * n_cols;
  constexpr size_t patches = std::max(VecmatCfg<true>::PATCH_BYTES, VecmatCfg<false>::PATCH_BYTES);
  L.stages = (int)std::min<size_t>(std::min<size_t>(8, (220 * 1024 - 1024 - patches) / stage_bytes), (512 - acc_cols) / 64);
  if (L.stages < 2) return fail(EQT_ERR_UNSUPPORTED, "tile too wide for the shared-memory ring");
  L.tmem_cols = 32;
  while (L.tmem_cols < acc_cols + 64 * L.stages) L.tmem_cols <<= 1;
  {
    cuuint64_t dims[3] = {(cuuint64_t)rows1 * cin, 1, (cuuint64_t)n};
    cuuint64_t strides[2] = {(cuuint64_t)rows1 * cin * 4, (cuuint64_t)rows1 * cin * 4};
    cuuint32_t box[3] = {KB, 1, TILE_M};
    if (int rc = make_map(&L.map_a, x, 3, dims, strides, box)) return rc;
  }
  {
    // an empty table still needs valid maps: describe at least one k-block
    cuuint64_t dims[2] = {(cuuint64_t)std::max<int64_t>(ktot, KB), (cuuint64_t)n_cols};
    cuuint64_t strides[1] = {(cuuint64_t)std::max<int64_t>(ktot, KB) * 4};
    cuuint32_t box[2] = {KB, (cuuint32_t)n_cols};
    if (int rc = make_map(&L.map_bb, w_big, 2, dims, strides, box)) return rc;
    if (int rc = make_map(&L.map_bs, w_small, 2, dims, strides, box)) return rc;
  }
  // Resident weights: one-row groups of short sums over rows of x that are read about once (an output row's items run one after
  // the other, so a row that several output rows read would come from memory each time), 128 columns with two A slots.  Only
  // where the ring kernel has one accumulator set (more than 42 columns: with two its epilogue overlaps as well, and it is 7-10 %
  // faster: 50k nodes of 4 rows, 64 -> 32 channels, 23.9 against 26.0 us) and where CTAs have more than one item to overlap: with at
  // most one, loading the weights first costs 2-8 % (48 and 64 columns; 160 items: 3-5 % gained, 640: 10-20 %, 6256: 17-32 %).  Two units of two
  // k-blocks hold both A slots to the end, so they take three items a CTA to gain (376 items: 16.0 -> 16.3 us, 640: 24.0 -> 22.2, 6256:
  // 180 -> 154).
  const int b_bytes = longest * n_cols * KB * 8;
  if (group == 1 && longest >= 1 && longest <= VM_SHORT_CHUNK_KB && slots <= rows1 + rows1 / 2 && b_bytes <= 96 * 1024 &&
      L.acc_sets == 1 && (n_cols <= 64 || (n_cols == 128 && longest <= 2)) &&
      L.total_items > (int64_t)sm_count() * (n_cols == 128 && longest == 2 ? 3 : 1)) {
    ResidentLaunch R{};
    R.map_a = L.map_a; R.map_bb = L.map_bb; R.map_bs = L.map_bs;
    R.out = out; R.kb_begin = kb_begin; R.rows = group_rows; R.a_col = a_col; R.status = status;
    R.n = n; R.tiles = ceil_div(n, TILE_M); R.total_items = L.total_items;
    R.num_out = num_out; R.n_cols = n_cols; R.units = n_cols > 64 ? 2 : 1; R.unit_cols = n_cols / R.units;
    R.slots = std::min(4, (512 - 6 * R.unit_cols) / 64);
    R.b_bytes = b_bytes; R.longest = longest;
    R.raw_stages = (int)std::min<size_t>(8, (220 * 1024 - 1024 - EPI_PATCH_BYTES - b_bytes) / (TILE_M * KB * 4));
    auto* resident = longest == 1 ? vecmat_resident_kernel<true> : vecmat_resident_kernel<false>;
    if (int rc = allow_shared(resident, 220 * 1024)) return rc;
    resident<<<(unsigned)std::min<int64_t>(R.total_items, sm_count()), TC_THREADS,
               (size_t)b_bytes + (size_t)R.raw_stages * TILE_M * KB * 4 + 1024 + EPI_PATCH_BYTES, st>>>(R);
    return check_launch("vecmat_resident_kernel");
  }
  const bool wide = group > 1;
  auto* kernel = wide ? vecmat_tc_kernel<false, true> : longest == 1 ? vecmat_tc_kernel<true, false> : vecmat_tc_kernel<false, false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  if (e != cudaSuccess) return fail(EQT_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  const unsigned grid = (unsigned)std::min<int64_t>(L.total_items, sm_count());
  kernel<<<grid, wide ? VecmatCfg<true>::THREADS : VecmatCfg<false>::THREADS,
           (size_t)L.stages * stage_bytes + 1024 + (wide ? VecmatCfg<true>::PATCH_BYTES : VecmatCfg<false>::PATCH_BYTES), st>>>(L);
  return check_launch("vecmat_tc_kernel");
}

extern "C" int eqt_vecmat_tc(const float* x, const float* w, const int64_t* index2, const float* scale, float* w_big,
                             float* w_small, float* out, int64_t n, int32_t rows1, int32_t cin, int32_t cout,
                             int32_t num_out, int64_t entries, const int32_t* kb_begin, const int32_t* a_col,
                             int32_t* status, void* stream) {
  return eqt_vecmat_tc_grouped(x, w, index2, scale, w_big, w_small, out, n, rows1, cin, cout, num_out, entries, 1, num_out, nullptr,
                               nullptr, kb_begin, a_col, 0, status, stream);
}

extern "C" int64_t eqt_outer_tc_scratch_floats(int64_t n, int32_t columns, int32_t m_tiles) {
  using namespace eqt;
  if (n < 0 || columns <= 0 || columns % 32 || m_tiles <= 0) return -1;
  WgradTile tile;
  if (columns > 128 || !outer_tile(n, columns, m_tiles, &tile)) return -1;
  return (int64_t)outer_splits(std::max<int64_t>(1, ceil_div(n, tile.npt)), m_tiles) * m_tiles * 128 * columns;
}

extern "C" int eqt_outer_tc_grouped(const float* in1, const float* in2, float* out, float* scratch, int64_t scratch_floats, int64_t n,
                                    int32_t rows1, int32_t c1, int32_t rows2, int32_t c2, int32_t group, const int32_t* a_cols,
                                    const int32_t* b_cols, int32_t m_tiles, const int32_t* red_ptr, const int32_t* red_slot,
                                    const float* red_scale, int32_t num_w, int32_t transposed, int32_t* status, void* stream) {
  using namespace eqt;
  if (n < 0 || rows1 <= 0 || rows2 <= 0 || c1 <= 0 || c2 <= 0 || group <= 0 || m_tiles < 0 || num_w < 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (num_w == 0) return EQT_OK;
  if (!in1 || !in2 || !out || !scratch || !a_cols || !b_cols || !red_ptr || !red_slot || !red_scale || !status)
    return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (c1 % 32 != 0 || c2 % 32 != 0 || c2 > 128 || group > 128 / c2)
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core outer product needs C1 %% 32 == 0, C2 %% 32 == 0, C2 <= 128 (all rows of a group)");
  if ((reinterpret_cast<uintptr_t>(in1) | reinterpret_cast<uintptr_t>(in2) | reinterpret_cast<uintptr_t>(out) |
       reinterpret_cast<uintptr_t>(scratch)) & 15u)
    return fail(EQT_ERR_UNSUPPORTED, "tensor-core outer product needs 16-byte aligned operands");
  if (n > 0x7fffffffll || (int64_t)rows1 * c1 > 0x7fffffffll || (int64_t)rows2 * c2 > 0x7fffffffll || m_tiles >= (1 << 22))
    return fail(EQT_ERR_UNSUPPORTED, "operands too large for one TMA coordinate");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int columns = group * c2;
  int splits = 1;
  if (n > 0 && m_tiles > 0) {
    WgradTile tile;
    if (!outer_tile(n, columns, m_tiles, &tile)) return fail(EQT_ERR_UNSUPPORTED, "tile does not fit shared memory");
    const int npt = tile.npt;                                                        // reduction rows per tile
    WgradBatch B{};
    B.count = 1; B.n = n; B.n_cols = columns; B.status = status;
    WgradBlock& a = B.blk[0];
    a.dim = 1; a.npt = npt; a.rows_pad = tile.rows_pad; a.issuers = tile.issuers;
    a.a_cols = a_cols; a.b_cols = b_cols; a.b_row_boxes = c2 / 32;
    const int64_t tiles = ceil_div(n, npt);
    splits = outer_splits(tiles, m_tiles);
    a.chunk_tiles = wgrad_chunk(a.rows_pad, a.issuers, ceil_div(tiles, splits));
    const int64_t need = (int64_t)splits * m_tiles * 128 * columns;
    if (need > scratch_floats) return fail(EQT_ERR_BAD_ARGUMENT, "scratch too small: %lld floats needed", (long long)need);
    a.partial = scratch;
    a.m_tiles = m_tiles; a.splits = splits; a.cta_begin = 0;
    {
      cuuint64_t dims[3] = {(cuuint64_t)rows1 * c1, 1, (cuuint64_t)n};
      cuuint64_t strides[2] = {(cuuint64_t)rows1 * c1 * 4, (cuuint64_t)rows1 * c1 * 4};
      cuuint32_t box[3] = {KB, 1, (cuuint32_t)npt};
      if (int rc = make_map(&a.map_s, in1, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
    }
    {
      cuuint64_t dims[3] = {(cuuint64_t)rows2 * c2, 1, (cuuint64_t)n};
      cuuint64_t strides[2] = {(cuuint64_t)rows2 * c2 * 4, (cuuint64_t)rows2 * c2 * 4};
      cuuint32_t box[3] = {KB, 1, (cuuint32_t)npt};
      if (int rc = make_map(&a.map_g, in2, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B)) return rc;
    }
    if (int rc = launch_wgrad(B, tile.smem, st)) return rc;
  }
  // with no samples or no entries every unit list is read as empty only if m_tiles == 0; otherwise the partial sums
  // above were written by this call
  if (n == 0 || m_tiles == 0) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(float) * (size_t)num_w * c1 * c2, st);
    if (e != cudaSuccess) return fail(EQT_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    return EQT_OK;
  }
  const auto reduce = [&](auto* kernel, int warps) {
    kernel<<<(unsigned)ceil_div((int64_t)num_w * c1 * c2 / 4, 32 * (REDUCE_WARPS / warps)), 32 * REDUCE_WARPS, 0, st>>>(
        scratch, out, red_ptr, red_slot, red_scale, splits, (int64_t)m_tiles * 128, num_w, c1, c2, columns);
  };
  // eight warps a result from nine splits on, fewer where the results alone fill the SMs (30 x 96 x 96 weights, 512 samples: the sum with eight
  // warps 8.1 us, with two some 5; but 8 x 32 x 32, 4000 samples, both kernels 17.4 and 19.8)
  const bool fill = (int64_t)num_w * c1 * c2 / 4 > 32 * 4 * (int64_t)sm_count();
  const auto by_warps = [&](auto t) {
    constexpr bool T = t();
    if (splits > 8 && (!fill || splits >= 32)) reduce(outer_reduce_kernel<T, 8, 2>, 8);
    else if (splits >= 16) reduce(outer_reduce_kernel<T, 4, 4>, 4);
    else if (splits > 8) reduce(outer_reduce_kernel<T, 2, 4>, 2);
    else if (splits >= 4) reduce(outer_reduce_kernel<T, 1, 4>, 1);
    else reduce(outer_reduce_kernel<T, 1, 2>, 1);
  };
  if (transposed) by_warps(std::true_type{}); else by_warps(std::false_type{});
  return check_launch("outer_reduce_kernel");
}

extern "C" int eqt_outer_tc(const float* in1, const float* in2, float* out, float* scratch, int64_t scratch_floats, int64_t n,
                            int32_t rows1, int32_t c1, int32_t rows2, int32_t c2, const int32_t* a_cols, const int32_t* b_cols,
                            int32_t m_tiles, const int32_t* red_ptr, const int32_t* red_slot, const float* red_scale,
                            int32_t num_w, int32_t* status, void* stream) {
  return eqt_outer_tc_grouped(in1, in2, out, scratch, scratch_floats, n, rows1, c1, rows2, c2, 1, a_cols, b_cols, m_tiles, red_ptr,
                              red_slot, red_scale, num_w, 0, status, stream);
}

// ------------------------------------------------------------------------------------------
// Weight gradient without any caller-side or library-side allocation
// ------------------------------------------------------------------------------------------
namespace eqt {
namespace {

// Scratch for the per-CTA partial sums of eqt_wgrad_tc_static: 148 SMs x 128 rows x 64 columns of
// float32 = 4,849,664 bytes, resident on every GPU that loads this library until the process exits.
constexpr int64_t kStaticScratchFloats = 148ll * 128 * 64;
static __device__ __align__(256) float g_wgrad_scratch[kStaticScratchFloats];

constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
float* g_static_ptr[kMaxDevices] = {};

// Device address of g_wgrad_scratch on the current device.  In host code the symbol itself is only a
// handle; the address a kernel can use comes from cudaGetSymbolAddress, once per device.
int static_scratch(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail(EQT_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return fail(EQT_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_wgrad_scratch);
    if (e != cudaSuccess || !p) return fail(EQT_ERR_CUDA, "cudaGetSymbolAddress(g_wgrad_scratch): %s", cudaGetErrorString(e));
    g_static_ptr[dev] = static_cast<float*>(p);
  }
  *out = g_static_ptr[dev];
  return EQT_OK;
}

}  // namespace
}  // namespace eqt

extern "C" int64_t eqt_wgrad_tc_static_capacity(void) { return eqt::kStaticScratchFloats; }

extern "C" int eqt_wgrad_tc_static(const float* s, const float* g, float* gw_packed, int64_t n, int32_t rows,
                                   int32_t comps, int32_t cin, int32_t cout, const eqt_mix_block* blocks,
                                   int32_t num_blocks, int32_t* status, void* stream) {
  using namespace eqt;
  if (cout > 64)
    return fail(EQT_ERR_UNSUPPORTED,
                "eqt_wgrad_tc_static: C_out = %d exceeds the limit of 64 output channels of the built-in scratch "
                "(%lld floats); use eqt_wgrad_tc with a caller-provided scratch buffer", (int)cout,
                (long long)kStaticScratchFloats);
  if ((int64_t)sm_count() * 128 * cout > kStaticScratchFloats)
    return fail(EQT_ERR_UNSUPPORTED,
                "eqt_wgrad_tc_static: %d SMs x 128 x %d floats exceed the built-in scratch of %lld floats; use "
                "eqt_wgrad_tc with a caller-provided scratch buffer", sm_count(), (int)cout,
                (long long)kStaticScratchFloats);
  if (n > 0 && num_blocks > 0 && blocks && cin > 0 && cin % 32 == 0 && cout > 0 && cout % 32 == 0) {
    const int tile_rows = wgrad_rows(blocks, num_blocks, n, cin);
    for (int b = 0; b < num_blocks; ++b) {   // the real need of every block, before anything is launched
      WgradShape w{};
      if (int rc = wgrad_shape(blocks[b], b, n, cin, cout, tile_rows, &w)) return rc;
      if (w.need > kStaticScratchFloats)
        return fail(EQT_ERR_UNSUPPORTED,
                    "eqt_wgrad_tc_static: block %d (%d paths x %d input channels) needs %lld floats of scratch, the "
                    "built-in scratch holds %lld; use eqt_wgrad_tc with a caller-provided scratch buffer", b,
                    (int)blocks[b].paths, (int)cin, (long long)w.need, (long long)kStaticScratchFloats);
    }
  }
  float* scratch = nullptr;
  if (int rc = static_scratch(&scratch)) return rc;
  return eqt_wgrad_tc(s, g, gw_packed, scratch, kStaticScratchFloats, n, rows, comps, cin, cout, blocks, num_blocks,
                      status, stream);
}

// ------------------------------------------------------------------------------------------
// Packing and splitting of the weights for the GEMMs above (one launch instead of a dozen tensor ops)
// ------------------------------------------------------------------------------------------
namespace eqt {
namespace {

struct PackArgs {
  int first[16], paths[16];      // per block: first gathered path, number of paths
  int num_blocks, cin, cout, k_major;
  int64_t total;
};

// k_major = 1: per block Bt[co, p*cin + ci] (operand of eqt_mix_tc);  0: [p*cin + ci, co] (stacked paths)
__global__ void __launch_bounds__(256) pack_weights_kernel(const float* __restrict__ w, const int64_t* __restrict__ gather,
                                                           float* __restrict__ big, float* __restrict__ small, PackArgs a) {
  const int64_t per_path = (int64_t)a.cin * a.cout;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.total; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t g = i / per_path;              // gathered path this element belongs to (blocks are contiguous runs)
    const int64_t r = i % per_path;
    int ci, co;
    if (a.k_major) {
      int b = 0;
      while (b + 1 < a.num_blocks && g >= a.first[b + 1]) ++b;
      const int64_t local = i - (int64_t)a.first[b] * per_path;      // offset inside the block's (cout, paths*cin) matrix
      const int64_t kk = local % ((int64_t)a.paths[b] * a.cin);
      co = (int)(local / ((int64_t)a.paths[b] * a.cin));
      g = a.first[b] + kk / a.cin;
      ci = (int)(kk % a.cin);
    } else {
      ci = (int)(r / a.cout);
      co = (int)(r % a.cout);
    }
    const float v = __ldg(w + __ldg(gather + g) * per_path + (int64_t)ci * a.cout + co);
    const float hi = rn_tf32(v);
    big[i] = hi;
    small[i] = rn_tf32(v - hi);
  }
}

}  // namespace
}  // namespace eqt

extern "C" int eqt_pack_weights(const float* w, const int64_t* path_gather, int32_t cin, int32_t cout,
                                const eqt_mix_block* blocks, int32_t num_blocks, int32_t k_major, float* big,
                                float* small, void* stream) {
  using namespace eqt;
  if (!w || !path_gather || !blocks || !big || !small) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (num_blocks <= 0 || num_blocks > 16 || cin <= 0 || cout <= 0) return fail(EQT_ERR_UNSUPPORTED, "1..16 blocks supported");
  PackArgs a{};
  a.num_blocks = num_blocks; a.cin = cin; a.cout = cout; a.k_major = k_major;
  int total_paths = 0;
  for (int b = 0; b < num_blocks; ++b) {
    a.first[b] = (int)(blocks[b].w_offset / ((int64_t)cin * cout));
    a.paths[b] = blocks[b].paths;
    if (a.first[b] != total_paths) return fail(EQT_ERR_BAD_ARGUMENT, "blocks must be packed back to back");
    total_paths += blocks[b].paths;
  }
  a.total = (int64_t)total_paths * cin * cout;
  pack_weights_kernel<<<flat_grid(a.total, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(w, path_gather, big, small, a);
  return check_launch("pack_weights_kernel");
}
