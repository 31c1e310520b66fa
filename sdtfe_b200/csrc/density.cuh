// density.cuh - a vertex's density from the volumes of its tets, in the
// reference's order (mesh.cu and noalloc.cu).
//
// The vertex -> tet lists are filled in the order the atomics happen to run;
// the reference adds the volumes in increasing tet order (src/triangulate.c:
// 190-221), so each list is put in that order first.
#pragma once

#include <cstdint>

namespace sdtfe {

// a3 part 1: per-tet volume |V| in the reference's operation order
// (src/triangulate.c:191-215), and the tets of each vertex counted.  Checked:
// a tet with a vertex id outside [0, n) sets *flags' kOutOfRange and is passed
// over, here and by k_tet_fill.  One that lists a vertex twice sets kRepeated.
constexpr int kOutOfRange = 1, kRepeated = 2;
__device__ __forceinline__ bool vertices_in(const int4& v, int n) {
  return (unsigned)v.x < (unsigned)n && (unsigned)v.y < (unsigned)n && (unsigned)v.z < (unsigned)n &&
         (unsigned)v.w < (unsigned)n;
}

template <bool Checked>
__global__ void k_volume_count(const double4* __restrict__ pos, const int4* __restrict__ rows,
                               int nt, int n, double* __restrict__ vol, int* __restrict__ cnt,
                               int* __restrict__ flags) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const int4 v = rows[2 * (size_t)t];
  if (Checked && !vertices_in(v, n)) {
    atomicOr(flags, kOutOfRange);
    return;
  }
  if (v.x == v.y || v.x == v.z || v.x == v.w || v.y == v.z || v.y == v.w || v.z == v.w)
    atomicOr(flags, kRepeated);
  const double4 a = pos[v.x], b = pos[v.y], c = pos[v.z], d = pos[v.w];
  const double r0 = (a.x - d.x) * ((b.y - d.y) * (c.z - d.z) - (b.z - d.z) * (c.y - d.y));
  const double r1 = (a.y - d.y) * ((b.z - d.z) * (c.x - d.x) - (b.x - d.x) * (c.z - d.z));
  const double r2 = (a.z - d.z) * ((b.x - d.x) * (c.y - d.y) - (b.y - d.y) * (c.x - d.x));
  vol[t] = fabs((r0 + r1 + r2) / 6);
  atomicAdd(cnt + v.x, 1);
  atomicAdd(cnt + v.y, 1);
  atomicAdd(cnt + v.z, 1);
  atomicAdd(cnt + v.w, 1);
}

// The vertex -> tet lists: off holds the scanned counts, cnt counts down.
template <bool Checked>
__global__ void k_tet_fill(const int4* __restrict__ rows, int nt, int n, const int* __restrict__ off,
                           int* __restrict__ cnt, int* __restrict__ idx) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  const int4 v = rows[2 * (size_t)t];
  if (Checked && !vertices_in(v, n)) return;
  idx[off[v.x] + atomicSub(cnt + v.x, 1) - 1] = t;
  idx[off[v.y] + atomicSub(cnt + v.y, 1) - 1] = t;
  idx[off[v.z] + atomicSub(cnt + v.z, 1) - 1] = t;
  idx[off[v.w] + atomicSub(cnt + v.w, 1) - 1] = t;
}

// A warp takes a vertex.  Lists of up to kRankedTets tets (27 in the mean) are
// not sorted: each lane counts, for up to four of the tets, how many ids are
// smaller, and puts the tet's volume in that place of a row in shared memory,
// which one lane adds up.  Longer lists are sorted by one lane where they are.
//
// What bounds it: latency of the list, its volumes and the serial sum, hidden by
// the other warps.  One thread a vertex sorted its list in memory, three
// dependent accesses an exchange, and summed gathers one by one: 4k clustered
// points 76 + 10 us, 131k 113 + 21 us.  The whole dtfe_density_noalloc: 4k
// points 136 -> 51 us, 30k 170 -> 76, 131k 240 -> 151 (of these 10, 17 and 18 us
// by validating, measuring and counting in one kernel and waiting once).
constexpr int kRankedTets = 128;
constexpr int kDensityWarps = 8;  // warps a block

// Shell sort over a diminishing gap sequence (Ciura's gaps, then x2.25):
// O(d^1.3) for the rare hub vertex with hundreds or thousands of tets.  (A tet
// that lists a vertex twice is in its list twice; the sorted order is the same
// whichever comes first.)
__device__ inline void shell_sort(int* a, int d) {
  constexpr int kGaps[] = {1, 4, 10, 23, 57, 132, 301, 701, 1577, 3548, 7983, 17961, 40412};
  int g = 0;
  while (g + 1 < (int)(sizeof(kGaps) / sizeof(kGaps[0])) && kGaps[g + 1] < d) ++g;
  for (; g >= 0; --g) {
    const int gap = kGaps[g];
    for (int i = gap; i < d; ++i) {
      const int key = a[i];
      int j = i;
      while (j >= gap && a[j - gap] > key) {
        a[j] = a[j - gap];
        j -= gap;
      }
      a[j] = key;
    }
  }
}

// The places of K tets a lane, at list positions lane, lane + 32, ...  A tet that
// lists the vertex several times is in the list as often: where there are such tets
// (repeated), equal ids take their places in list order, so that every place is taken.
template <int K>
__device__ __forceinline__ void rank_volumes(const int* __restrict__ list, int d,
                                             const double* __restrict__ vol, int lane,
                                             bool repeated, double* row) {
  unsigned id[K];
  int rank[K];
  double v[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = 32 * k + lane;
    id[k] = i < d ? (unsigned)list[i] : 0u;  // (no place is taken from d on)
    v[k] = i < d ? vol[id[k]] : 0.0;
    rank[k] = 0;
    if (repeated) {
      const unsigned same = __match_any_sync(0xffffffffu, i < d ? id[k] : 0xffffffffu);
      rank[k] = __popc(same & ((1u << lane) - 1u));
    }
  }
  const unsigned tie = repeated ? 1u : 0u;  // an equal id of an earlier 32 comes first
#pragma unroll
  for (int c = 0; c < K; ++c) {
    const int m = min(32, d - 32 * c);
    for (int j = 0; j < m; ++j) {
      const unsigned other = __shfl_sync(0xffffffffu, id[c], j);
#pragma unroll
      for (int k = 0; k < K; ++k) rank[k] += other < (c < k ? id[k] + tie : id[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (32 * k + lane < d) row[rank[k]] = v[k];
}

// The sum of a vertex's tet volumes, taken from 0 in increasing tet order (the
// reference's in-place scatter-add, to the bit); valid in lane 0.  The whole
// warp calls it; row: kRankedTets doubles of shared memory, the warp's own.
__device__ inline double volume_sum(int* __restrict__ list, int d, const double* __restrict__ vol,
                                    bool repeated, double* row) {
  const int lane = (int)(threadIdx.x & 31u);
  double s = 0;
  if (d <= kRankedTets) {
    if (d <= 32) rank_volumes<1>(list, d, vol, lane, repeated, row);
    else if (d <= 64) rank_volumes<2>(list, d, vol, lane, repeated, row);
    else rank_volumes<4>(list, d, vol, lane, repeated, row);
    __syncwarp();
    if (lane == 0)
      for (int i = 0; i < d; ++i) s += row[i];
  } else if (lane == 0) {
    shell_sort(list, d);
    for (int i = 0; i < d; ++i) s += vol[list[i]];
  }
  return s;
}

}  // namespace sdtfe
