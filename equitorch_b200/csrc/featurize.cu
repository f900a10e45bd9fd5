// Edge featurisation: radius graph over a cell list, and per edge - in the same pass that writes the edge - the
// edge vector, its length, real spherical harmonics, the Bessel radial basis and a cutoff envelope.
//
// The caller bins the points into cubic cells of side >= r (one slab of cells per graph of the batch), sorts them by
// cell and passes the sorted order and the first sorted position of every cell.  One warp owns one target node:
// its lanes walk the points of the 27 surrounding cells, compact the ones closer than r into a list in shared
// memory (ballot + prefix count), and the list is ordered by source index with a rank count so that the result does
// not depend on how the points were binned.  `eqt_radius_count` stores min(#neighbours, max_neighbors) per target;
// after an exclusive scan of those counts `eqt_radius_edges` repeats the search and writes, for the neighbours of
// smallest index, source, target, vec = pos[target] - pos[source], |vec| and the features.
//
// replaces (see include/eqt_b200.h): the chain RadiusGraph -> AddSphericalHarmonics -> AddVectorLengthEmbedding(BesselBasis)
// -> cutoff of the reference's transforms, which calls a third-party neighbour search and then one elementwise
// kernel per operation.
#include <algorithm>

#include "common.cuh"

namespace eqt {
namespace {

#include "generated/sh_specs.inc"

constexpr int RG_WARPS = 4;
constexpr int RG_LIST = 512;        // candidates per target held in shared memory

struct RadiusArgs {
  const float* pos;               // (n, 3)
  const int64_t* batch;           // (n) graph of every point, or NULL
  const int32_t* cell_start;      // (num_cells + 1) into the sorted order
  const int32_t* sorted_index;    // (n) original index of the k-th point in cell order
  const int32_t* point_cell;      // (n) cell of every point (graph slab included), as binned by the caller
  int dims[3];                    // cells per axis (per graph)
  float r2;
  int loop, max_neighbors;
  int64_t n;
  int32_t* degree;                // count pass: (n)
  int32_t* status;                // set to 1 if a target had more than RG_LIST candidates
  // edge pass
  const int64_t* ptr;             // (n + 1)
  int64_t* src;
  int64_t* dst;
  float* vec;                     // (E, 3) or NULL
  float* len;                     // (E) or NULL
  float* sh;                      // (E, (l_max + 1)^2) or NULL
  float* bessel;                  // (E, num_basis) or NULL
  float* cutoff;                  // (E) or NULL
  const float* bessel_w;          // (num_basis) frequencies (n pi by default)
  int l_max, num_basis, cutoff_kind;
  float sh_scale, r_max, cut_min, cut_range, cut_p, cut_eps;
};

// neighbours of target i into list[0 .. count), unsorted; returns the number found (may exceed RG_LIST: the caller flags it)
__device__ __forceinline__ int collect(const RadiusArgs& a, int64_t i, int* list, int lane) {
  const float px = __ldg(a.pos + 3 * i), py = __ldg(a.pos + 3 * i + 1), pz = __ldg(a.pos + 3 * i + 2);
  // the caller's binning is authoritative: the target's cell is read, not recomputed
  const int per_graph = a.dims[0] * a.dims[1] * a.dims[2];
  const int cell = __ldg(a.point_cell + i), local = cell % per_graph;
  if (cell < 0) return 0;         // a graph index out of range
  const int64_t slab = cell - local;
  const int cx = local % a.dims[0], cy = (local / a.dims[0]) % a.dims[1], cz = local / (a.dims[0] * a.dims[1]);
  int count = 0;
  for (int dz = -1; dz <= 1; ++dz) {
    const int z = cz + dz;
    if (z < 0 || z >= a.dims[2]) continue;
    for (int dy = -1; dy <= 1; ++dy) {
      const int y = cy + dy;
      if (y < 0 || y >= a.dims[1]) continue;
      // the three cells x - 1, x, x + 1 are consecutive in the linear order: one range
      const int x0 = max(cx - 1, 0), x1 = min(cx + 1, a.dims[0] - 1);
      const int64_t c0 = slab + ((int64_t)z * a.dims[1] + y) * a.dims[0] + x0;
      const int k0 = __ldg(a.cell_start + c0), k1 = __ldg(a.cell_start + c0 + (x1 - x0) + 1);
      for (int kb = k0; kb < k1; kb += 32) {
        const int k = kb + lane;
        bool hit = false;
        int j = 0;
        if (k < k1) {
          j = __ldg(a.sorted_index + k);
          const float ex = __ldg(a.pos + 3 * (int64_t)j) - px, ey = __ldg(a.pos + 3 * (int64_t)j + 1) - py,
                      ez = __ldg(a.pos + 3 * (int64_t)j + 2) - pz;
          hit = ex * ex + ey * ey + ez * ez < a.r2 && (a.loop || j != i);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
          const int at = count + __popc(m & ((1u << lane) - 1u));
          if (at < RG_LIST) list[at] = j;
        }
        count += __popc(m);
      }
    }
  }
  __syncwarp();
  return count;
}

__global__ void __launch_bounds__(RG_WARPS * 32) radius_count_kernel(RadiusArgs a) {
  __shared__ int lists[RG_WARPS][RG_LIST];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t i = (int64_t)blockIdx.x * RG_WARPS + warp; i < a.n; i += (int64_t)gridDim.x * RG_WARPS) {
    const int count = collect(a, i, lists[warp], lane);
    if (lane == 0) {
      if (count > RG_LIST) atomicExch(a.status, 1);
      a.degree[i] = min(count, a.max_neighbors);
    }
    __syncwarp();
  }
}

template <int LMAX>
__device__ __forceinline__ void write_sh(const RadiusArgs& a, int64_t e, const float (&u)[3]) {
  constexpr int K = (LMAX + 1) * (LMAX + 1);
  float y[K];
  ShUnrolled<float, LMAX>::forward(u, y);
#pragma unroll
  for (int k = 0; k < K; ++k) a.sh[e * K + k] = y[k] * a.sh_scale;
}

__device__ __forceinline__ float cutoff_value(const RadiusArgs& a, float r) {
  const float u = fminf(fmaxf((r - a.cut_min) / a.cut_range, 0.f), 1.f);
  float c;
  if (a.cutoff_kind == EQT_CUTOFF_POLYNOMIAL) {
    const float p = a.cut_p;
    c = 1.f - ((p + 1.f) * (p + 2.f) / 2.f) * powf(u, p) + (p * (p + 2.f)) * powf(u, p + 1.f) - (p * (p + 1.f) / 2.f) * powf(u, p + 2.f);
  } else if (a.cutoff_kind == EQT_CUTOFF_COSINE) {
    c = 0.5f * (1.f + cosf(3.14159265358979323846f * u));
  } else {
    c = expf(1.f - 1.f / (1.f - u * u + a.cut_eps));
  }
  return c;
}

__global__ void __launch_bounds__(RG_WARPS * 32) radius_edges_kernel(RadiusArgs a) {
  __shared__ int lists[RG_WARPS][RG_LIST];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t i = (int64_t)blockIdx.x * RG_WARPS + warp; i < a.n; i += (int64_t)gridDim.x * RG_WARPS) {
    const int* list = lists[warp];
    const int count = min(collect(a, i, lists[warp], lane), RG_LIST);
    const int64_t e0 = __ldg(a.ptr + i);
    const int keep = (int)(__ldg(a.ptr + i + 1) - e0);
    const float px = __ldg(a.pos + 3 * i), py = __ldg(a.pos + 3 * i + 1), pz = __ldg(a.pos + 3 * i + 2);
    for (int q = lane; q < count; q += 32) {
      const int j = list[q];
      int rank = 0;
      for (int k = 0; k < count; ++k) rank += list[k] < j;      // sources are distinct
      if (rank >= keep) continue;                               // beyond max_neighbors
      const int64_t e = e0 + rank;
      a.src[e] = j;
      a.dst[e] = i;
      const float vx = px - __ldg(a.pos + 3 * (int64_t)j), vy = py - __ldg(a.pos + 3 * (int64_t)j + 1),
                  vz = pz - __ldg(a.pos + 3 * (int64_t)j + 2);
      const float r = sqrtf(vx * vx + vy * vy + vz * vz);
      if (a.vec) { a.vec[3 * e] = vx; a.vec[3 * e + 1] = vy; a.vec[3 * e + 2] = vz; }
      if (a.len) a.len[e] = r;
      if (a.sh) {
        const float inv = 1.f / fmaxf(r, 1e-12f);
        const float u[3] = {vx * inv, vy * inv, vz * inv};
        switch (a.l_max) {
          case 0: a.sh[e] = a.sh_scale; break;
          case 1: write_sh<1>(a, e, u); break;
          case 2: write_sh<2>(a, e, u); break;
          case 3: write_sh<3>(a, e, u); break;
          default: write_sh<4>(a, e, u); break;
        }
      }
      if (a.bessel) {
        const float pre = 2.f / a.r_max;
        for (int b = 0; b < a.num_basis; ++b) a.bessel[e * a.num_basis + b] = pre * (sinf(__ldg(a.bessel_w + b) * r / a.r_max) / r);
      }
      if (a.cutoff) {
        a.cutoff[e] = cutoff_value(a, r);
      }
    }
    __syncwarp();
  }
}

// ---- cell list and neighbour lists in few passes ---------------------------------------------------------------------------
// The order of the points within a cell does not matter (neighbour lists are ordered by index), so the cells are filled by a
// counting sort: every point takes a number in its cell (atomic), an exclusive scan of the cell counts gives the places.
// A radix sort of 64-bit cell numbers with its index arithmetic took some forty launches, 170 us of kernels per 100k points;
// this one takes 14 us.
struct BinArgs {
  const float* pos;
  const int64_t* batch;
  float lo[3], inv_cell;
  int dims[3], graphs;
  int64_t n;
  int32_t* point_cell;    // -1: a graph index out of range, no neighbours
  int32_t* rank;
  int32_t* cell_count;    // zeroed by the caller
};
__global__ void __launch_bounds__(256) radius_bin_kernel(BinArgs a) {
  const int per_graph = a.dims[0] * a.dims[1] * a.dims[2];
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
    int c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = min(max((int)floorf((__ldg(a.pos + 3 * i + k) - a.lo[k]) * a.inv_cell), 0), a.dims[k] - 1);
    const int64_t graph = a.batch ? __ldg(a.batch + i) : 0;
    const bool inside = graph >= 0 && graph < a.graphs;
    const int cell = inside ? (int)graph * per_graph + (c[2] * a.dims[1] + c[1]) * a.dims[0] + c[0] : -1;
    a.point_cell[i] = cell;
    a.rank[i] = inside ? atomicAdd(a.cell_count + cell, 1) : 0;
  }
}
// sorted[place] = (x, y, z, index): the search then reads a candidate with one 16-byte load next to its neighbours' instead of
// an index and three scattered floats
__global__ void __launch_bounds__(256) radius_place_kernel(const float* __restrict__ pos, const int32_t* __restrict__ point_cell,
                                                           const int32_t* __restrict__ rank, const int32_t* __restrict__ cell_start,
                                                           float4* __restrict__ sorted, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int cell = point_cell[i];
    if (cell >= 0)
      sorted[cell_start[cell] + rank[i]] =
          make_float4(__ldg(pos + 3 * i), __ldg(pos + 3 * i + 1), __ldg(pos + 3 * i + 2), __int_as_float((int)i));
  }
}

struct SearchArgs {
  const float* pos;
  const float4* sorted;
  const int32_t* cell_start;
  const int32_t* point_cell;
  int dims[3];
  float r2;
  int loop, most;               // most = min(max_neighbors, RG_LIST): row length of `list`
  int64_t n;
  int32_t* degree;
  int32_t* list;                // (n, most) neighbours, ascending
  int32_t* status;
};
// One warp per target.  The nine ranges of candidates (three consecutive cells each) are read by nine lanes at once and walked
// as one sequence, so that the lanes are full and no range waits for the one before it: range by range, 12 of 32 lanes had a
// candidate and each of the nine steps was a chain of four dependent loads (103 us per 100k points and 18 neighbours for the
// count, and the same again in the pass that wrote the edges; 73 us here, once, with the sorted list kept).
__global__ void __launch_bounds__(RG_WARPS * 32) radius_search_kernel(SearchArgs a) {
  __shared__ int lists[RG_WARPS][RG_LIST];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_graph = a.dims[0] * a.dims[1] * a.dims[2];
  int* found = lists[warp];
  for (int64_t i = (int64_t)blockIdx.x * RG_WARPS + warp; i < a.n; i += (int64_t)gridDim.x * RG_WARPS) {
    const int cell = __ldg(a.point_cell + i);
    if (cell < 0) {
      if (lane == 0) a.degree[i] = 0;
      continue;
    }
    const float px = __ldg(a.pos + 3 * i), py = __ldg(a.pos + 3 * i + 1), pz = __ldg(a.pos + 3 * i + 2);
    const int local = cell % per_graph, slab = cell - local;
    const int cx = local % a.dims[0], cy = (local / a.dims[0]) % a.dims[1], cz = local / (a.dims[0] * a.dims[1]);
    int first = 0, len = 0;
    if (lane < 9) {
      const int z = cz + lane / 3 - 1, y = cy + lane % 3 - 1;
      if (z >= 0 && z < a.dims[2] && y >= 0 && y < a.dims[1]) {
        const int x0 = max(cx - 1, 0), x1 = min(cx + 1, a.dims[0] - 1);
        const int32_t* c = a.cell_start + slab + (z * a.dims[1] + y) * a.dims[0] + x0;
        first = __ldg(c);
        len = __ldg(c + x1 - x0 + 1) - first;
      }
    }
    int begin[9], shift[9], total = 0;          // candidate f of range q is at sorted position f + shift[q]
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      begin[q] = total;
      shift[q] = __shfl_sync(0xffffffffu, first, q) - total;
      total += __shfl_sync(0xffffffffu, len, q);
    }
    int count = 0;
    for (int f0 = 0; f0 < total; f0 += 32) {
      const int f = f0 + lane;
      int at = shift[0];
#pragma unroll
      for (int q = 1; q < 9; ++q) at = f >= begin[q] ? shift[q] : at;
      bool hit = false;
      int j = 0;
      if (f < total) {
        const float4 c = __ldg(a.sorted + f + at);
        j = __float_as_int(c.w);
        const float ex = c.x - px, ey = c.y - py, ez = c.z - pz;
        hit = ex * ex + ey * ey + ez * ez < a.r2 && (a.loop || j != i);
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int to = count + __popc(m & ((1u << lane) - 1u));
        if (to < RG_LIST) found[to] = j;
      }
      count += __popc(m);
    }
    __syncwarp();
    if (lane == 0) {
      if (count > RG_LIST) atomicExch(a.status, 1);
      a.degree[i] = min(count, a.most);
    }
    count = min(count, RG_LIST);
    for (int q = lane; q < count; q += 32) {
      const int j = found[q];
      int rank = 0;
      for (int k = 0; k < count; ++k) rank += found[k] < j;      // sources are distinct
      if (rank < a.most) a.list[i * a.most + rank] = j;
    }
    __syncwarp();
  }
}

// Edges and their features from the neighbour lists: a block takes 32 consecutive targets, whose edges are consecutive, and a
// thread an edge, so that no lane idles over a target with few neighbours; harmonics go through shared memory and radial
// functions are computed per (edge, function), so that both leave as whole rows of addresses.  One warp per target with one
// store per component took 262 us for 1.8M edges (l_max 3, 8 functions); 99 us so.
constexpr int LE_TARGETS = 32, LE_THREADS = 128;
template <int LMAX>
__global__ void __launch_bounds__(LE_THREADS) radius_list_edges_kernel(RadiusArgs a, const int32_t* __restrict__ list, int most) {
  constexpr int K = LMAX < 0 ? 1 : (LMAX + 1) * (LMAX + 1);
  constexpr int PITCH = K | 1;
  __shared__ float stage[LMAX < 0 ? 1 : LE_THREADS * PITCH];
  __shared__ float radius[LE_THREADS];
  __shared__ int64_t first[LE_TARGETS + 1];
  const int64_t blocks = (a.n + LE_TARGETS - 1) / LE_TARGETS;
  for (int64_t blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
    const int64_t i0 = blk * LE_TARGETS;
    const int targets = (int)min((int64_t)LE_TARGETS, a.n - i0);
    __syncthreads();
    if (threadIdx.x <= targets) first[threadIdx.x] = __ldg(a.ptr + i0 + threadIdx.x);
    __syncthreads();
    const int64_t last = first[targets];
    for (int64_t e0 = first[0]; e0 < last; e0 += LE_THREADS) {
      const int64_t e = e0 + threadIdx.x;
      const int here = (int)min((int64_t)LE_THREADS, last - e0);
      if (e < last) {
        int lo = 0, hi = targets;                       // first[lo] <= e < first[hi]
        while (hi - lo > 1) {
          const int mid = (lo + hi) / 2;
          if (first[mid] <= e) lo = mid; else hi = mid;
        }
        const int64_t i = i0 + lo;
        const int j = __ldg(list + i * most + (e - first[lo]));
        a.src[e] = j;
        a.dst[e] = i;
        const float vx = __ldg(a.pos + 3 * i) - __ldg(a.pos + 3 * (int64_t)j), vy = __ldg(a.pos + 3 * i + 1) - __ldg(a.pos + 3 * (int64_t)j + 1),
                    vz = __ldg(a.pos + 3 * i + 2) - __ldg(a.pos + 3 * (int64_t)j + 2);
        const float r = sqrtf(vx * vx + vy * vy + vz * vz);
        if (a.vec) { a.vec[3 * e] = vx; a.vec[3 * e + 1] = vy; a.vec[3 * e + 2] = vz; }
        if (a.len) a.len[e] = r;
        radius[threadIdx.x] = r;
        if constexpr (LMAX == 0) stage[threadIdx.x] = a.sh_scale;
        if constexpr (LMAX > 0) {
          const float inv = 1.f / fmaxf(r, 1e-12f);
          const float u[3] = {vx * inv, vy * inv, vz * inv};
          float y[K];
          ShUnrolled<float, LMAX>::forward(u, y);
#pragma unroll
          for (int k = 0; k < K; ++k) stage[threadIdx.x * PITCH + k] = y[k] * a.sh_scale;
        }
        if (a.cutoff) a.cutoff[e] = cutoff_value(a, r);
      }
      __syncthreads();
      if constexpr (LMAX >= 0)
        for (int t = threadIdx.x; t < here * K; t += LE_THREADS) a.sh[e0 * K + t] = stage[t / K * PITCH + t % K];
      if (a.bessel) {
        const float pre = 2.f / a.r_max;
        for (int t = threadIdx.x; t < here * a.num_basis; t += LE_THREADS) {
          const int q = t / a.num_basis;
          const float r = radius[q];
          a.bessel[e0 * a.num_basis + t] = pre * (sinf(__ldg(a.bessel_w + t - q * a.num_basis) * r / a.r_max) / r);
        }
      }
      __syncthreads();
    }
  }
}

int fill_args(const eqt_radius_grid* g, const float* pos, const int64_t* batch, int64_t n, float r, int loop, int max_neighbors,
              int32_t* status, RadiusArgs& a) {
  if (!g || !g->cell_start || !g->sorted_index || !g->point_cell) return fail(EQT_ERR_BAD_ARGUMENT, "incomplete cell list");
  if (n < 0 || r <= 0.f || max_neighbors <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (g->dims[0] <= 0 || g->dims[1] <= 0 || g->dims[2] <= 0 || !(g->cell_size >= r))
    return fail(EQT_ERR_BAD_ARGUMENT, "cells must be at least r wide");
  if (n > 0x7fffffffll) return fail(EQT_ERR_UNSUPPORTED, "too many points");
  if (n > 0 && (!pos || !status)) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  a.pos = pos; a.batch = batch; a.cell_start = g->cell_start; a.sorted_index = g->sorted_index; a.point_cell = g->point_cell;
  for (int k = 0; k < 3; ++k) a.dims[k] = g->dims[k];
  a.r2 = r * r; a.loop = loop; a.max_neighbors = max_neighbors; a.n = n; a.status = status;
  return EQT_OK;
}

int fill_features(const eqt_edge_features* f, RadiusArgs& a) {
  if (f) {
    if (f->sh && (f->l_max < 0 || f->l_max > 4)) return fail(EQT_ERR_UNSUPPORTED, "fused harmonics take l_max <= 4");
    if (f->bessel && (!f->bessel_weights || f->num_basis <= 0 || !(f->r_max > 0.f))) return fail(EQT_ERR_BAD_ARGUMENT, "bad radial basis");
    if (f->cutoff && (f->cutoff_kind < EQT_CUTOFF_POLYNOMIAL || f->cutoff_kind > EQT_CUTOFF_MOLLIFIER || !(f->cutoff_r_max > f->cutoff_r_min)))
      return fail(EQT_ERR_BAD_ARGUMENT, "bad cutoff");
    a.vec = f->vec; a.len = f->length; a.sh = f->sh; a.bessel = f->bessel; a.cutoff = f->cutoff; a.bessel_w = f->bessel_weights;
    a.l_max = f->l_max; a.num_basis = f->num_basis; a.cutoff_kind = f->cutoff_kind;
    a.sh_scale = f->integral_normalize ? 0.28209479177387814f : 1.f;
    a.r_max = f->r_max; a.cut_min = f->cutoff_r_min; a.cut_range = f->cutoff_r_max - f->cutoff_r_min;
    a.cut_p = f->cutoff_p; a.cut_eps = f->cutoff_eps;
  }
  return EQT_OK;
}

}  // namespace
}  // namespace eqt

extern "C" int eqt_radius_bin(const float* pos, const int64_t* batch, int64_t n, const float* lo, float cell_size, const int32_t* dims,
                              int32_t graphs, int32_t* point_cell, int32_t* rank, int32_t* cell_count, void* stream) {
  using namespace eqt;
  if (!lo || !dims || n < 0 || graphs < 0 || !(cell_size > 0.f)) return fail(EQT_ERR_BAD_ARGUMENT, "bad cell grid");
  if (dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad cell grid");
  if (n > 0x7fffffffll || (double)dims[0] * dims[1] * dims[2] * graphs > 2147483647.0) return fail(EQT_ERR_UNSUPPORTED, "too many points or cells");
  if (n == 0) return EQT_OK;
  if (!pos || !point_cell || !rank || !cell_count) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  BinArgs a{pos, batch, {lo[0], lo[1], lo[2]}, 1.f / cell_size, {dims[0], dims[1], dims[2]}, graphs, n, point_cell, rank, cell_count};
  radius_bin_kernel<<<flat_grid(n, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return check_launch("radius_bin_kernel");
}

extern "C" int eqt_radius_place(const float* pos, const int32_t* point_cell, const int32_t* rank, const int32_t* cell_start, float* sorted,
                                int64_t n, void* stream) {
  using namespace eqt;
  if (n < 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (n == 0) return EQT_OK;
  if (!pos || !point_cell || !rank || !cell_start || !sorted) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (reinterpret_cast<uintptr_t>(sorted) & 15u) return fail(EQT_ERR_UNSUPPORTED, "sorted points must be 16-byte aligned");
  radius_place_kernel<<<flat_grid(n, 256, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(pos, point_cell, rank, cell_start,
                                                                                         reinterpret_cast<float4*>(sorted), n);
  return check_launch("radius_place_kernel");
}

extern "C" int eqt_radius_search(const float* pos, const float* sorted, const int32_t* cell_start, const int32_t* point_cell, int64_t n,
                                 const int32_t* dims, float r, int32_t loop, int32_t row, int32_t* degree, int32_t* list, int32_t* status,
                                 void* stream) {
  using namespace eqt;
  if (!dims || n < 0 || r <= 0.f || row <= 0 || row > RG_LIST || dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0)
    return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (n == 0) return EQT_OK;
  if (!pos || !sorted || !cell_start || !point_cell || !degree || !list || !status) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  if (reinterpret_cast<uintptr_t>(sorted) & 15u) return fail(EQT_ERR_UNSUPPORTED, "sorted points must be 16-byte aligned");
  SearchArgs a{pos, reinterpret_cast<const float4*>(sorted), cell_start, point_cell, {dims[0], dims[1], dims[2]}, r * r, loop, row, n,
               degree, list, status};
  radius_search_kernel<<<flat_grid(ceil_div(n, RG_WARPS), 1, 16), RG_WARPS * 32, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return check_launch("radius_search_kernel");
}

extern "C" int eqt_radius_list_edges(const float* pos, int64_t n, const int64_t* ptr, const int32_t* list, int32_t row, int64_t* src,
                                     int64_t* dst, const eqt_edge_features* f, void* stream) {
  using namespace eqt;
  if (n < 0 || row <= 0) return fail(EQT_ERR_BAD_ARGUMENT, "bad sizes");
  if (n == 0) return EQT_OK;
  if (!pos || !ptr || !list || !src || !dst) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  RadiusArgs a{};
  a.pos = pos; a.n = n; a.ptr = ptr; a.src = src; a.dst = dst;
  if (int rc = fill_features(f, a)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = flat_grid(ceil_div(n, LE_TARGETS), 1, 16);
  switch (a.sh ? a.l_max : -1) {
    case -1: radius_list_edges_kernel<-1><<<grid, LE_THREADS, 0, st>>>(a, list, row); break;
    case 0: radius_list_edges_kernel<0><<<grid, LE_THREADS, 0, st>>>(a, list, row); break;
    case 1: radius_list_edges_kernel<1><<<grid, LE_THREADS, 0, st>>>(a, list, row); break;
    case 2: radius_list_edges_kernel<2><<<grid, LE_THREADS, 0, st>>>(a, list, row); break;
    case 3: radius_list_edges_kernel<3><<<grid, LE_THREADS, 0, st>>>(a, list, row); break;
    default: radius_list_edges_kernel<4><<<grid, LE_THREADS, 0, st>>>(a, list, row); break;
  }
  return check_launch("radius_list_edges_kernel");
}

extern "C" int eqt_radius_count(const eqt_radius_grid* grid, const float* pos, const int64_t* batch, int64_t n, float r,
                                int32_t loop, int32_t max_neighbors, int32_t* degree, int32_t* status, void* stream) {
  using namespace eqt;
  RadiusArgs a{};
  if (int rc = fill_args(grid, pos, batch, n, r, loop, max_neighbors, status, a)) return rc;
  if (n == 0) return EQT_OK;
  if (!degree) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  a.degree = degree;
  radius_count_kernel<<<flat_grid(ceil_div(n, RG_WARPS), 1, 16), RG_WARPS * 32, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return check_launch("radius_count_kernel");
}

extern "C" int eqt_radius_edges(const eqt_radius_grid* grid, const float* pos, const int64_t* batch, int64_t n, float r,
                                int32_t loop, int32_t max_neighbors, const int64_t* ptr, int64_t* src, int64_t* dst,
                                const eqt_edge_features* f, int32_t* status, void* stream) {
  using namespace eqt;
  RadiusArgs a{};
  if (int rc = fill_args(grid, pos, batch, n, r, loop, max_neighbors, status, a)) return rc;
  if (n == 0) return EQT_OK;
  if (!ptr || !src || !dst) return fail(EQT_ERR_BAD_ARGUMENT, "NULL pointer");
  a.ptr = ptr; a.src = src; a.dst = dst;
  if (int rc = fill_features(f, a)) return rc;
  radius_edges_kernel<<<flat_grid(ceil_div(n, RG_WARPS), 1, 16), RG_WARPS * 32, 0, static_cast<cudaStream_t>(stream)>>>(a);
  return check_launch("radius_edges_kernel");
}
