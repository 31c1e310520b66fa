// grid_rays.cuh - 3-D grids with one thread per sub-ray.
//
// A cell of a supersampled grid receives the node values of ss^2 sub-rays, and
// the reference adds them sub-ray by sub-ray, each in walk order
// (src/dtfe.c:710-729).  One thread per column keeps that order by walking its
// ss^2 rays one after the other, which leaves most of the GPU idle below a few
// hundred columns a side: 120^2 columns at ss = 2 are 450 warps, each waiting
// through four walks.  Here every sub-ray has its thread and writes its node
// values to a row of its own; a second kernel adds each cell's values in the
// reference's order, so the cells are the same to the bit.  A ray says from
// where to where its row is written; a node in between that no chord holds is
// written as -0.0, which changes no sum.  A ray that comes back to a node it
// has passed (after a turn-around or a perturbation) has no place for the
// second value: its column is marked and walked by the one-thread kernel.
#pragma once

#include "mesh.h"

namespace sdtfe {
namespace {

// where a column's node values go: its cells directly ...  Several: grids with
// more than one sub-ray a column, whose reductions are written as the
// instruction itself (FP64, 32k uniform points, 512^3 at ss 2: 10.1 -> 8.4 ms;
// grids of one ray a column lose by that, 256^3 0.35 -> 0.56).
template <bool Several>
struct CellSink {
  static constexpr bool kShortChain = false;  // reciprocal_near, walk64.cuh
  double* col;
  int ss;
  __device__ __forceinline__ void begin(int, int) {}
  __device__ __forceinline__ void put(int is, double v) {
    double* const cell = col + (int)((unsigned)is / (unsigned)ss);
    if constexpr (Several)
      asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(cell)), "d"(v));
    else
      cell_add(cell, v);
  }
};

// ... or the ray's row of nodes
struct NodeSink {
  static constexpr bool kShortChain = true;
  double* row;
  int first;       // the row is written from here (-1: nothing yet)
  int done;        // to here
  bool irregular;  // came back to a node it had passed
  // (a value put on a node passed before is lost, with its column's rows)
  __device__ __forceinline__ void begin(int i0, int i1) {
    if (first < 0) first = done = i0;
    if (i0 < done) irregular = true;
    for (; done < i0; ++done) put(done, -0.0);
    done = max(done, i1);
  }
  __device__ __forceinline__ void put(int is, double v) const {
    asm volatile("st.global.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(row + is)), "d"(v));
  }
};

// A grid's sub-rays.
struct GridRays {
  int G, ss, lanes;  // lanes: rays a warp walks
  double* nodes;  // row (i*G + j)*ss^2 + is*ss + js of G*ss nodes
  int2* range;    // per ray: the nodes its row holds, [x, y)
  int* col;       // per column: bit k for a ray of status k, and the two marks
};
constexpr int kIrregular = 1 << 8, kHasNodes = 1 << 9;

__device__ __forceinline__ int worst_status(int marks) {
  return 31 - __clz((marks & (kIrregular - 1)) | 1);
}

// This thread's sub-ray, (column i, j; sub-ray is, js), in a launch over
// ray_warps(): warps cover compact patches of the fine grid.
__device__ __forceinline__ bool ray_of_grid(const GridRays& a, int* i, int* j, int* is, int* js) {
  const int nf = a.G * a.ss;  // fine columns a side
  const int warp = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  const int pi = patch_rows(a.lanes), pj = patch_cols(a.lanes);
  const int tiles_j = (nf + pj - 1) / pj;
  const int lane = (int)threadIdx.x & 31;
  const int fi = (warp / tiles_j) * pi + lane / pj, fj = (warp % tiles_j) * pj + lane % pj;
  *i = fi / a.ss;
  *j = fj / a.ss;
  *is = fi % a.ss;
  *js = fj % a.ss;
  return lane < a.lanes && fi < nf && fj < nf;
}
inline long long ray_warps(long long nf, int lanes) {
  const int pi = patch_rows(lanes), pj = patch_cols(lanes);
  return ((nf + pi - 1) / pi) * ((nf + pj - 1) / pj);
}
inline long long ray_warps(const GridRays& a) { return ray_warps((long long)a.G * a.ss, a.lanes); }

__device__ __forceinline__ size_t ray_index(const GridRays& a, int i, int j, int is, int js) {
  return (((size_t)i * a.G + j) * a.ss + is) * a.ss + js;
}
__device__ __forceinline__ NodeSink ray_nodes(const GridRays& a, int i, int j, int is, int js) {
  return {a.nodes + ray_index(a, i, j, is, js) * ((size_t)a.G * a.ss), -1, 0, false};
}

__device__ __forceinline__ void ray_done(const GridRays& a, int i, int j, int is, int js,
                                         const NodeSink& out, int status) {
  const bool any = out.first >= 0;
  a.range[ray_index(a, i, j, is, js)] = make_int2(any ? out.first : 0, any ? out.done : 0);
  atomicOr(a.col + (size_t)i * a.G + j,
           1 << status | (any ? kHasNodes : 0) | (out.irregular ? kIrregular : 0));
}

// One thread per cell: its ss^3 node values, sub-ray by sub-ray.  SS: the usual
// supersamplings, whose loads are all in flight together (0: any).
template <int SS>
__global__ void __launch_bounds__(256) k_grid_sum(const GridRays a, double* __restrict__ grid) {
  const long long cell = blockIdx.x * 256LL + threadIdx.x;
  if (cell >= (long long)a.G * a.G * a.G) return;
  const int iz = (int)(cell % a.G);
  const long long c = cell / a.G;
  if ((a.col[c] & (kHasNodes | kIrregular)) != kHasNodes) return;
  const int ss = SS > 0 ? SS : a.ss, nzs = a.G * ss;
  const double* v = a.nodes + (size_t)c * ss * ss * nzs + iz * ss;
  const int2* range = a.range + (size_t)c * ss * ss;
  double sum = grid[cell];
  if constexpr (SS > 0) {
#pragma unroll 1
    for (int is = 0; is < SS; ++is, v += SS * nzs, range += SS) {
      double node[SS][SS];
#pragma unroll
      for (int js = 0; js < SS; ++js) {
        const int2 held = range[js];
#pragma unroll
        for (int k = 0; k < SS; ++k) {
          const int n = iz * SS + k;
          node[js][k] = n >= held.x && n < held.y ? v[js * nzs + k] : -0.0;
        }
      }
#pragma unroll
      for (int js = 0; js < SS; ++js)
#pragma unroll
        for (int k = 0; k < SS; ++k) sum += node[js][k];
    }
  } else {
    for (int r = 0; r < ss * ss; ++r, v += nzs) {
      const int2 held = range[r];
      const int k1 = min(held.y - iz * ss, ss);
      for (int k = max(held.x - iz * ss, 0); k < k1; ++k) sum += v[k];
    }
  }
  grid[cell] = sum;
}

// Which grids are walked by sub-rays: all with several a column (but for dense FP64
// grids, walk.cu), as long as the rows of nodes (8 B times the fine grid) stay within
// 4 GiB - up to 406^3 cells at ss = 2, 268^3 at 3, 203^3 at 4.  One thread a column is
// slower below and, measured, still at that size (83k-point lattice, mixed / FP64, one
// thread a column -> sub-rays): 128^3 ss 4 6.9 / 10.9 -> 1.9 / 2.0 ms, 200^3 ss 2 3.0 /
// 2.8 -> 1.3 / 1.4, 256^3 ss 3 9.2 / 7.7 -> 4.4 / 4.3, 384^3 ss 2 6.6 / 6.0 -> 4.5 / 4.4.
// Batches of the rows lose that again to one tail each.
constexpr size_t kNodeBytes = size_t(4) << 30;
inline bool grid_takes_rays(int G, unsigned ss) {
  const double n = (double)G * ss;
  return ss > 1 && 8.0 * n * n * n <= (double)kNodeBytes;
}

// The grid by sub-rays: rays(GridRays) launches the walks, serial(GridRays) the
// one-thread columns, which counts the columns' outcomes and walks those that are
// marked irregular.  *taken is false when the grid is not for this, or its
// scratch is not to be had: nothing has been done.
template <class Rays, class Serial>
dtfe_status_t grid_by_rays(int G, unsigned ss, int lanes, double* d_grid, cudaStream_t s,
                           bool* taken, Rays&& rays, Serial&& serial) {
  *taken = false;
  if (!grid_takes_rays(G, ss)) return DTFE_OK;
  const size_t n = (size_t)G * ss, col_bytes = sizeof(int) * (size_t)G * G;
  void *nodes = nullptr, *range = nullptr, *col = nullptr;
  if (scratch_alloc_async(&nodes, sizeof(double) * n * n * n, s) != DTFE_OK ||
      scratch_alloc_async(&range, sizeof(int2) * n * n, s) != DTFE_OK ||
      scratch_alloc_async(&col, col_bytes, s) != DTFE_OK) {
    scratch_free_async(nodes, s);
    scratch_free_async(range, s);
    cudaGetLastError();
    dtfe_clear_error();
    return DTFE_OK;
  }
  *taken = true;
  const GridRays a{G, (int)ss, lanes, static_cast<double*>(nodes), static_cast<int2*>(range),
                   static_cast<int*>(col)};
  cudaError_t e = cudaMemsetAsync(col, 0, col_bytes, s);
  if (e == cudaSuccess) {
    rays(a);
    const auto sum = ss == 2 ? k_grid_sum<2> : (ss == 3 ? k_grid_sum<3> : (ss == 4 ? k_grid_sum<4> : k_grid_sum<0>));
    sum<<<(unsigned)(((long long)G * G * G + 255) / 256), 256, 0, s>>>(a, d_grid);
    serial(a);
    count_launch(3);
    e = cudaGetLastError();
  }
  scratch_free_async(nodes, s);
  scratch_free_async(range, s);
  scratch_free_async(col, s);
  SDTFE_CUDA(e);
  return DTFE_OK;
}

}  // namespace
}  // namespace sdtfe
