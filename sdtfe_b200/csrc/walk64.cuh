// walk64.cuh - FP64 ray walk through a device-resident Delaunay mesh.
//
// The arithmetic here repeats the reference's FP64 operations in the same
// order (src/dtfe.c:19-374, 518-552), and the translation units that include
// this header are compiled with -fmad=false, so each product and sum is
// rounded on its own exactly as the reference's x86-64 build rounds it.  With
// the same mesh, the same sample positions and the same perturbation stream
// the walk therefore visits the same tets and returns the same doubles.
//
// Data layout (built by mesh.cu):
//   TetRec64  160 B per tet: its four vertices in the projected frame, rho_A
//             and the gradient; three 256-bit loads a step (the vertex not yet
//             seen, vertex A and the field).
//   links     16 B per (tet, entry face, rotation): tet_links.cuh.
//   TriRec64   64 B per projected hull triangle: (x, y) of its corners, the
//             three edge neighbours and the tet under it.
#pragma once

#include <cstdint>

#include "sdtfe_rng.h"
#include "tet_links.cuh"

namespace sdtfe {

// src/constants.h:6-8
constexpr double kZero = 1e4 * 2.220446049250313080847263336181640625e-16;
constexpr int kPerturbMax = 1000;

enum RayStatus : int {
  kRayOk = 0,
  kRayMiss = 1,
  kRayNoExit = 2,
  kRayPerturbMax = 3,
  kRayBudget = 4,
  kRayLocBudget = 5,
};

struct __align__(32) TetRec64 {
  double4 v[4];  // vertices A..D in the projected frame (w unused)
  double4 f;     // rho_A, grad_x, grad_y, grad_z
};
static_assert(sizeof(TetRec64) == 160, "TetRec64 layout");

struct __align__(16) TriRec64 {
  double2 a, b, c;  // projected corners
  int4 nb;          // (n_CB, n_AC, n_BA, tet)
};
static_assert(sizeof(TriRec64) == 64, "TriRec64 layout");

// 32 B in one load
__device__ __forceinline__ double4 load256(const double4* p) {
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
      : "l"(p));
  return v;
}

template <class T>
__host__ __device__ __forceinline__ T sel4(int k, T a, T b, T c, T d) {
  return k == 0 ? a : (k == 1 ? b : (k == 2 ? c : d));
}

__device__ __forceinline__ int sign_eps(double x) {
  return x > kZero ? 1 : (x < -kZero ? -1 : 0);
}

__device__ __forceinline__ int nb_at(const int4& n, int k) { return sel4(k, n.x, n.y, n.z, n.w); }

// ---------------------------------------------------------------------------
// a8: Plücker test for a ray along +z (src/dtfe.c:29-215).
//
// For the edge P->Q the permuted product with the ray (lz, -lz*oy, lz*ox) is
//   lz*(Px*Qy - Py*Qx) + (Px - Qx)*(-lz*oy) + (Py - Qy)*(lz*ox)
// (src/dtfe.c:24-26, 44-47).  Edges in side_t order: CB, AC, BA, DC, BD, DA.
struct Ray64 {
  double lz, m_oy, ox_l;  // lz, -lz*oy, lz*ox
};

__device__ __forceinline__ double edge_u64(const Ray64& r, double2 p, double2 q) {
  double v0 = p.x - q.x;
  double v1 = p.y - q.y;
  double v5 = p.x * q.y - p.y * q.x;
  return r.lz * v5 + v0 * r.m_oy + v1 * r.ox_l;
}

struct Hit64 {
  int enter, leave;
  bool ok, special;
};

// The four faces BDC, ACD, ADB, ABC each carry three signed edge terms; a face
// whose three edge signs are all zero is skipped, a face is entered when its
// signed terms are all >= 0 and left when all are <= 0 (the two are exclusive
// once the all-zero case is skipped).  The first entered and the first left
// face in that order are chosen; the test fails unless both exist.
__device__ __forceinline__ Hit64 plucker_faces(const int s[6]) {
  // signed sign terms per face (the reference's conditions, src/dtfe.c:66-213)
  const int f0a = -s[0], f0b = s[3], f0c = -s[4];   // BDC: -CB, +DC, -BD
  const int f1a = s[1], f1b = -s[3], f1c = -s[5];   // ACD: +AC, -DC, -DA
  const int f2a = s[5], f2b = s[4], f2c = -s[2];    // ADB: +DA, +BD, -BA
  const int f3a = s[2], f3b = s[0], f3c = -s[1];    // ABC: +BA, +CB, -AC
  auto live = [](int a, int b, int c) { return (a | b | c) != 0; };
  auto ent = [&](int a, int b, int c) { return live(a, b, c) && a >= 0 && b >= 0 && c >= 0; };
  auto lea = [&](int a, int b, int c) { return live(a, b, c) && a <= 0 && b <= 0 && c <= 0; };
  auto zer = [](int a, int b, int c) { return a == 0 || b == 0 || c == 0; };
  const bool e0 = ent(f0a, f0b, f0c), e1 = ent(f1a, f1b, f1c), e2 = ent(f2a, f2b, f2c),
             e3 = ent(f3a, f3b, f3c);
  const bool l0 = lea(f0a, f0b, f0c), l1 = lea(f1a, f1b, f1c), l2 = lea(f2a, f2b, f2c),
             l3 = lea(f3a, f3b, f3c);
  Hit64 h;
  h.enter = e0 ? 0 : (e1 ? 1 : (e2 ? 2 : (e3 ? 3 : -1)));
  h.leave = l0 ? 0 : (l1 ? 1 : (l2 ? 2 : (l3 ? 3 : -1)));
  h.ok = h.enter >= 0 && h.leave >= 0;
  const bool z0 = zer(f0a, f0b, f0c), z1 = zer(f1a, f1b, f1c), z2 = zer(f2a, f2b, f2c),
             z3 = zer(f3a, f3b, f3c);
  h.special = h.ok && (sel4(h.enter, z0, z1, z2, z3) || sel4(h.leave, z0, z1, z2, z3));
  return h;
}

// z of the point where the ray crosses face f: the face normaliser is summed
// in the reference's order, then ((1 - w1) - w2)*z0 + w1*z1 + w2*z2.
__host__ __device__ __forceinline__ double face_z64(int f, const double u[6], const double z[4]) {
  const double a0 = sel4(f, -u[0], u[1], u[5], u[2]);
  const double a1 = sel4(f, u[3], -u[3], u[4], u[0]);
  const double a2 = sel4(f, -u[4], -u[5], -u[2], -u[1]);
  const double w1n = sel4(f, -u[4], u[1], u[4], -u[1]);
  const double w2n = sel4(f, u[3], -u[3], -u[2], u[2]);
  const double z0 = sel4(f, z[3], z[2], z[1], z[0]);
  const double z1 = sel4(f, z[2], z[3], z[0], z[1]);
  const double z2 = sel4(f, z[1], z[0], z[3], z[2]);
  const double inv = 1.0 / (a0 + a1 + a2);
  const double w1 = w1n * inv;
  const double w2 = w2n * inv;
  return (1 - w1 - w2) * z0 + w1 * z1 + w2 * z2;
}

__device__ __forceinline__ Hit64 ray_tet64(const Ray64& r, const double2 xy[4], double u[6]) {
  u[0] = edge_u64(r, xy[2], xy[1]);  // CB
  u[1] = edge_u64(r, xy[2], xy[0]);  // AC
  u[2] = edge_u64(r, xy[1], xy[0]);  // BA
  u[3] = edge_u64(r, xy[2], xy[3]);  // DC
  u[4] = edge_u64(r, xy[1], xy[3]);  // BD
  u[5] = edge_u64(r, xy[3], xy[0]);  // DA
  int s[6];
#pragma unroll
  for (int e = 0; e < 6; ++e) s[e] = sign_eps(u[e]);
  return plucker_faces(s);
}

// ---------------------------------------------------------------------------
// a7: visibility walk on the projected hull, from triangle `start`
// (src/dtfe.c:518-552).  Returns the tet under the query point or -1.
// Returns the tet under the hull triangle containing (qx, qy); *tri_out (if
// given) receives the triangle.
__device__ __forceinline__ int locate64(const TriRec64* __restrict__ tri, int start, double qx,
                                        double qy, int max_steps, int* status,
                                        int* tri_out = nullptr) {
  int cur = start;
  int steps = 0;
  *status = kRayOk;
  do {
    if (++steps > max_steps) {
      *status = kRayLocBudget;
      return -1;
    }
    const TriRec64* t = tri + cur;
    const double2 a = __ldg(&t->a), b = __ldg(&t->b), c = __ldg(&t->c);
    const int4 nb = __ldg(&t->nb);
    double s_in, s_q;
    s_in = (c.x - a.x) * (b.y - a.y) - (c.y - a.y) * (b.x - a.x);
    s_q = (qx - a.x) * (b.y - a.y) - (qy - a.y) * (b.x - a.x);
    if (s_in * s_q < 0.0) {
      cur = nb.z;  // across a-b
      continue;
    }
    s_in = (a.x - b.x) * (c.y - b.y) - (a.y - b.y) * (c.x - b.x);
    s_q = (qx - b.x) * (c.y - b.y) - (qy - b.y) * (c.x - b.x);
    if (s_in * s_q < 0.0) {
      cur = nb.x;  // across b-c
      continue;
    }
    s_in = (b.x - c.x) * (a.y - c.y) - (b.y - c.y) * (a.x - c.x);
    s_q = (qx - c.x) * (a.y - c.y) - (qy - c.y) * (a.x - c.x);
    if (s_in * s_q < 0.0) {
      cur = nb.y;  // across c-a
      continue;
    }
    if (tri_out) *tri_out = cur;
    return nb.w;
  } while (cur != -1);
  *status = kRayMiss;
  return -1;
}

// One of locate64's edge tests (edge o->p, opposite vertex opp: s_in * s_q <
// 0) decided for every query point of the rectangle [xlo, xhi] x [ylo, yhi]
// at once: 1 when it holds for all of them, 0 when it fails for all, -1 when
// the outcome may differ inside.  s_in is the reference's own value.  The
// FP64 s_q = (qx - o.x) dy - (qy - o.y) dx (dy, dx the rounded edge
// differences) is within 3.0001 u M(q) of the linear form L(q) = (qx - o.x) dy
// - (qy - o.y) dx, M(q) = |qx - o.x| |dy| + |qy - o.y| |dx| (u = 2^-53; the
// operations are not contracted).  L and M take their extremes at the
// corners, so every s_q lies within 6.0002 u max M of the corners' FP64
// values; 16 u covers that and the rounding of the bound, and 2^-1000 any
// underflow.  The product s_in * s_q is then of one sign for all queries,
// and well clear of underflow to zero.
__host__ __device__ inline int edge_region(double2 o, double2 p, double2 opp, double xlo,
                                           double xhi, double ylo, double yhi) {
  const double s_in = (opp.x - o.x) * (p.y - o.y) - (opp.y - o.y) * (p.x - o.x);
  if (s_in == 0.0) return 0;  // the product is (signed) zero for every query
  const double dy = p.y - o.y, dx = p.x - o.x;
  const double qx[4] = {xlo, xhi, xlo, xhi}, qy[4] = {ylo, ylo, yhi, yhi};
  double lo = 0.0, hi = 0.0, mag = 0.0;
  for (int k = 0; k < 4; ++k) {
    const double tx = qx[k] - o.x, ty = qy[k] - o.y;
    const double s = tx * dy - ty * dx;
    lo = k == 0 ? s : (s < lo ? s : lo);
    hi = k == 0 ? s : (s > hi ? s : hi);
    const double m = (tx < 0.0 ? -tx : tx) * (dy < 0.0 ? -dy : dy) +
                     (ty < 0.0 ? -ty : ty) * (dx < 0.0 ? -dx : dx);
    mag = m > mag ? m : mag;
  }
  const double err = 16.0 * 0x1p-53 * mag + 0x1p-1000;
  const double a_in = s_in < 0.0 ? -s_in : s_in;
  if (lo > err) {  // s_q > 0 throughout
    if (a_in * (lo - err) < 0x1p-1000) return -1;
    return s_in < 0.0 ? 1 : 0;
  }
  if (hi < -err) {  // s_q < 0 throughout
    if (a_in * (-err - hi) < 0x1p-1000) return -1;
    return s_in > 0.0 ? 1 : 0;
  }
  return -1;
}

enum LocKind : int {
  kLocResume = 0,  // each query continues locate64 from *start with max_steps - *steps
  kLocFound = 1,   // every query's walk ends in triangle *start
  kLocMiss = 2,    // every query's walk leaves the hull
};

// The reference's location walk from triangle 0 (locate64), run once for a
// whole rectangle of query points while each edge test has one outcome for
// all of them.  Where the rectangle straddles a test, the walk stops and each
// query resumes it on its own at that triangle, with the steps taken so far
// counted against its budget: every query then makes exactly the moves, and
// ends with exactly the result, of its own walk from triangle 0.
__host__ __device__ inline int locate_region(const TriRec64* tri, double xlo, double xhi,
                                             double ylo, double yhi, int max_steps, int* start,
                                             int* steps_out) {
  int cur = 0, steps = 0;
  for (;;) {
    if (steps >= max_steps) break;  // each query's next step exceeds its budget
    const TriRec64& t = tri[cur];
    int nx = -1;
    int r = edge_region(t.a, t.b, t.c, xlo, xhi, ylo, yhi);  // edge a-b
    if (r == 1) {
      nx = t.nb.z;
    } else if (r == 0) {
      r = edge_region(t.b, t.c, t.a, xlo, xhi, ylo, yhi);  // edge b-c
      if (r == 1) {
        nx = t.nb.x;
      } else if (r == 0) {
        r = edge_region(t.c, t.a, t.b, xlo, xhi, ylo, yhi);  // edge c-a
        if (r == 1) {
          nx = t.nb.y;
        } else if (r == 0) {
          *start = cur;
          *steps_out = steps;
          return kLocFound;
        }
      }
    }
    if (r < 0) break;
    ++steps;
    if (nx == -1) {
      *start = -1;
      *steps_out = steps;
      return kLocMiss;
    }
    cur = nx;
  }
  *start = cur;
  *steps_out = steps;
  return kLocResume;
}

// The rectangle holding every sample position of a map tile (Args: the FP64
// or the mixed map's kernel arguments).  A ray's position is x(col) + u *
// scale with u in [0, 1), x(col) the expression below (the same as the
// rays'); each is monotone in col and u, so the tile's positions lie in
// [x(tx0), x(c1) + scale], and the same for y.
template <class Args>
__device__ __forceinline__ void tile_rect(const Args& a, int tile, double* xlo, double* xhi,
                                          double* ylo, double* yhi) {
  const int tx0 = (tile % a.tiles_x) * a.TW, ty0 = (tile / a.tiles_x) * a.TH;
  const int c1 = min(tx0 + a.TW, a.G) - 1, r1 = min(ty0 + a.TH, a.G) - 1;
  *xlo = tx0 * a.dxy + a.offx - a.soff;
  *xhi = (c1 * a.dxy + a.offx - a.soff) + a.scale;
  *ylo = ty0 * a.dxy + a.offy - a.soff;
  *yhi = (r1 * a.dxy + a.offy - a.soff) + a.scale;
}

// A tile's shared point location (locate_region), packed for the map kernel:
// (kind | steps << 2 as unsigned bits, start triangle).  steps <= loc_budget
// = 4 n_tri + 64 < 2^29 + 64 (the launchers cap n_tri below 2^27), so the
// packed value fits in 32 unsigned bits; it is unpacked with unsigned shifts.
template <class Args>
__device__ __forceinline__ int2 tile_location(const Args& a, int tile) {
  int kind = kLocMiss, start = -1, steps = 0;
  if (a.n_tri > 0) {
    double xlo, xhi, ylo, yhi;
    tile_rect(a, tile, &xlo, &xhi, &ylo, &yhi);
    kind = locate_region(a.tri, xlo, xhi, ylo, yhi, a.loc_budget, &start, &steps);
  }
  return make_int2((int)((unsigned)kind | ((unsigned)steps << 2)), start);
}

// One ray's point location from its tile's shared walk l (tile_location):
// where the tile's rectangle straddled a test, the ray resumes the walk from
// triangle 0 at that triangle with the steps already taken counted against
// its budget, so it reaches exactly the tet, triangle and status of its own
// locate64(tri, 0, ...).  A tile that left the hull leaves every ray a miss.
__device__ __forceinline__ int locate_from_tile(const TriRec64* __restrict__ tri, int2 l,
                                                double qx, double qy, int loc_budget,
                                                int* status, int* tri_out = nullptr) {
  const int lk = (int)((unsigned)l.x & 3u);
  if (lk == kLocFound) {
    if (tri_out) *tri_out = l.y;
    *status = kRayOk;
    return __ldg(&tri[l.y].nb.w);
  }
  if (lk == kLocResume)
    return locate64(tri, l.y, qx, qy, loc_budget - (int)((unsigned)l.x >> 2), status, tri_out);
  *status = kRayMiss;
  return -1;
}

// ---------------------------------------------------------------------------
// Accumulators: what a walk does with each crossed tet.

// a10: surface density, src/dtfe.c:356-369.  The chord midpoint must lie
// strictly inside (z0, z1); the linear field there times the chord length is
// added.
struct SurfaceAcc64 {
  static constexpr bool kShortChain = false;
  double z0, z1;
  double rho;
  // what visit() reads of a tet's record, loaded ahead of it
  struct Field {
    double4 A, f;
    __device__ __forceinline__ explicit Field(const TetRec64* __restrict__ t)
        : A(load256(&t->v[0])), f(load256(&t->f)) {}
  };
  __device__ __forceinline__ void visit(double ox, double oy, const Field& t, double z_in,
                                        double z_out) {
    const double d = z_out - z_in;
    const double zm = d / 2 + z_in;
    if (zm > z0 && zm < z1) {
      const double fixed = t.f.x + (t.f.y * (ox - t.A.x)) + (t.f.z * (oy - t.A.y)) - (t.f.w * t.A.z);
      rho += (fixed + t.f.w * zm) * d;
    }
  }
};

// One node's value added into its grid cell, *cell += v, as a reduction
// performed at L2: the thread does not wait for the cell's old value.  Each
// grid column belongs to one thread, and one thread's reductions to one
// address are performed in its program order, so every cell receives exactly
// the additions, in the order and with the roundings, of the reference's
// loop (src/dtfe.c:505-511).  The address space is named: the pointer travels
// through memory with the accumulator (general_step64), where the compiler loses
// it and turns an atomicAdd into a generic atomic that returns the old value.
__device__ __forceinline__ void cell_add(double* cell, double v) {
  __builtin_assume(__isGlobal(cell));
  atomicAdd(cell, v);
}

// The patch of neighbouring columns or rays that a warp walks on its first
// `lanes` lanes: 4 x 8, 4 x 4 or 2 x 4.  (A launch too small for the GPU takes
// fewer of them a warp: grid_lanes32 in walk32.cu, grid_lanes64 in walk.cu.)
__host__ __device__ constexpr int patch_rows(int lanes) { return lanes <= 8 ? 2 : 4; }
__host__ __device__ constexpr int patch_cols(int lanes) { return lanes <= 16 ? 4 : 8; }

// This thread's grid column (i: x index, j: y index) in a launch of
// grid_warps(G, lanes) warps: each warp covers a patch and four in a row two by
// two of them, so that a warp's columns are neighbours and cross many of the
// same tets.  False for the columns past the grid and the lanes past the patch.
__device__ __forceinline__ bool grid_column(int G, int lanes, int* i, int* j) {
  const int warp = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  const int tile = warp >> 2, wq = warp & 3;
  const int pi = patch_rows(lanes), pj = patch_cols(lanes);
  const int tiles_j = (G + 2 * pj - 1) / (2 * pj);
  const int ti = tile / tiles_j, tj = tile - ti * tiles_j;
  const int lane = (int)threadIdx.x & 31;
  *i = (2 * ti + (wq >> 1)) * pi + lane / pj;
  *j = (2 * tj + (wq & 1)) * pj + lane % pj;
  return lane < lanes && *i < G && *j < G;
}
inline unsigned grid_warps(int G, int lanes) {
  const int pi = 2 * patch_rows(lanes), pj = 2 * patch_cols(lanes);
  return 4u * (unsigned)(((G + pi - 1) / pi) * ((G + pj - 1) / pj));
}

// a12: 3-D column, src/dtfe.c:489-513.  The field is sampled at the fine z
// nodes inside the chord and added, with weight 1/ss^3, to the column cell.
template <class Sink>  // grid_rays.cuh
struct ColumnAcc64 {
  static constexpr bool kShortChain = Sink::kShortChain;
  Sink out;
  double z0, dzs, w;
  int nzs;
  // most chords of a fine mesh hold no node: the record is read when one does
  struct Field {
    const TetRec64* __restrict__ t;
    __device__ __forceinline__ explicit Field(const TetRec64* __restrict__ p) : t(p) {}
  };
  __device__ __forceinline__ void visit(double ox, double oy, const Field& r, double z_in,
                                        double z_out) {
    int i0 = (int)ceil((z_in - z0 - dzs / 2.) / dzs);
    i0 = i0 < 0 ? 0 : i0;
    int i1 = (int)ceil((z_out - z0 - dzs / 2.) / dzs);
    i1 = i1 > nzs ? nzs : i1;
    if (i1 > i0) {
      const double4 A = load256(&r.t->v[0]), f = load256(&r.t->f);
      const double fixed = f.x + f.y * (ox - A.x) + f.z * (oy - A.y) - f.w * A.z;
      out.begin(i0, i1);
      for (int is = i0; is < i1; ++is) {
        const double zi = z0 + dzs * is + dzs / 2.;
        out.put(is, (fixed + f.w * zi) * w);
      }
    }
  }
};

struct WalkConf64 {
  double lz;        // slab depth, the ray's direction length
  double dist;      // perturbation step (delta_xy/2)/PERTURB_MAX
  uint64_t seed;    // perturbation stream key
  int max_visits;   // visit budget
  const TetRec64* __restrict__ rec;
  const int4* __restrict__ rows;             // tetra_data rows (vertex ids, neighbours)
  const uint4* __restrict__ link;            // links (NULL: general steps only)
  const signed char* __restrict__ tri_face;  // the tet face under each hull triangle
};

// ---------------------------------------------------------------------------
// a9 + a10: the tet walk (src/dtfe.c:247-374).  On failure the crossing count
// stays 0 and the status says why; column accumulators keep what they already
// added, as evaluate_3d_ray_on_grid does.  The walk follows the neighbour
// across the leave face, turns around (swaps enter and leave) when that
// neighbour is the tet it came from, and perturbs the ray towards a
// generator-chosen corner while a chosen face has a zero edge sign.
//
// Two kinds of step, as in the mixed walk (walk32.cu).  The fast step knows the
// face the ray came in through and carries its triangle; the general step
// takes a tet in the mesh's vertex order and decides everything from its six
// products.

constexpr int kWalk64On = -1;  // the walk continues

// A walk between steps, for the general step.
template <class Acc>
struct Walk64 {
  double ox, oy;
  uint64_t ray, ctr;  // perturbation stream and draws so far
  Acc acc;
  int crossed, cur, prev;
  int rec;            // cur's record for its entry face (-1: not known)
};

template <class Acc>
__device__ __noinline__ int general_step64(const WalkConf64& W, Walk64<Acc>& w, int* visits,
                                           int max_record) {
  if (w.crossed >= W.max_visits) return kRayBudget;
  const TetRec64* rec = W.rec + w.cur;
  double2 xy[4];
  double z[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double4 v = load256(&rec->v[k]);
    xy[k] = make_double2(v.x, v.y);
    z[k] = v.z;
  }
  const int4 nb = __ldg(&W.rows[2 * (size_t)w.cur + 1]);
  Ray64 ry{W.lz, -W.lz * w.oy, W.lz * w.ox};
  double u[6];
  Hit64 h = ray_tet64(ry, xy, u);
  if (!h.ok) return kRayNoExit;
  int np = 0;
  while (h.special) {  // src/dtfe.c:329-349, perturb_ray at :219-245
    const int r = sdtfe_rand31(W.seed, w.ray, w.ctr++) % 4;
    const double2 vr = sel4(r, xy[0], xy[1], xy[2], xy[3]);
    double dx = vr.x - w.ox;
    double dy = vr.y - w.oy;
    const double mag = sqrt(dx * dx + dy * dy);
    if (mag > W.dist) {
      dx = dx / mag;
      dy = dy / mag;
      dx = dx * W.dist;
      dy = dy * W.dist;
    }
    w.ox = w.ox + dx;
    w.oy = w.oy + dy;
    ry.m_oy = -W.lz * w.oy;
    ry.ox_l = W.lz * w.ox;
    if (++np > kPerturbMax) return kRayPerturbMax;
    h = ray_tet64(ry, xy, u);
    if (!h.ok) return kRayNoExit;
  }
  const double z_in = face_z64(h.enter, u, z);
  const double z_out = face_z64(h.leave, u, z);
  if (visits != nullptr && w.crossed < max_record) visits[w.crossed] = w.cur;
  ++w.crossed;
  w.acc.visit(w.ox, w.oy, typename Acc::Field(rec), z_in, z_out);
  int m = h.leave;
  int nx = nb_at(nb, m);
  if (nx == -1) return kRayOk;
  if (nx == w.prev) {  // turn around
    m = h.enter;
    nx = nb_at(nb, m);
    if (nx == -1) return kRayOk;
  }
  w.rec = -1;
  if (W.link) {
    const int G = m == 0 ? 1 : 0;  // a record of cur whose entry face is not m
    const uint4 lk = __ldg(W.link + 3 * (4 * (size_t)w.cur + G));
    const int k = rot_inv(G, m);
    const uint32_t L = k == 0 ? lk.x : (k == 1 ? lk.y : lk.z);
    if (L <= kLinkLast) w.rec = (int)(L / 3u);
  }
  w.prev = w.cur;
  w.cur = nx;
  return kWalk64On;
}

// The triangle a fast walk carries: the face the ray last crossed and its
// cyclic products U(0,1), U(1,2), U(2,0) (edge_u64), all below -kZero.
struct Tri64 {
  double x0, y0, z0, x1, y1, z1, x2, y2, z2;
  double e01, e12, e20;
};

// z where the ray crosses a carried triangle, as the face_z64 of the face in
// the given roles (tet_links.cuh): n0..n2 are the products opposite slots
// 0..2, sum their sum with the right one added last (product_sums), and the
// corners follow in state order (an entry) or against it (an exit).  The sign
// of all three products cancels.  The point is formed for each slot as corner 0
// and then picked: 12 FP64 operations more than picking the five operands, but
// 16 selects and a dozen registers less.
struct ProductSums {
  double last0, last1, last2;  // by the slot whose product is added last
};
__host__ __device__ __forceinline__ ProductSums product_sums(double n0, double n1, double n2) {
  return {n1 + n2 + n0, n0 + n2 + n1, n0 + n1 + n2};
}

template <bool Exit>
__host__ __device__ __forceinline__ double crossing_by(double n0, double n1, double n2, double z0,
                                                       double z1, double z2, double inv, bool f0,
                                                       bool f1) {
  const double w0 = n0 * inv, w1 = n1 * inv, w2 = n2 * inv;
  const double m0 = w0 * z0, m1 = w1 * z1, m2 = w2 * z2;
  const double c0 = Exit ? (1 - w2 - w1) * z0 + m2 + m1 : (1 - w1 - w2) * z0 + m1 + m2;
  const double c1 = Exit ? (1 - w0 - w2) * z1 + m0 + m2 : (1 - w2 - w0) * z1 + m2 + m0;
  const double c2 = Exit ? (1 - w1 - w0) * z2 + m1 + m0 : (1 - w0 - w1) * z2 + m0 + m1;
  return f0 ? c0 : (f1 ? c1 : c2);
}

template <bool Exit>
__host__ __device__ __forceinline__ double crossing64(double n0, double n1, double n2, double z0,
                                                      double z1, double z2, const ProductSums& s,
                                                      unsigned roles) {
  const bool f0 = (roles & 3u) == 0u, f1 = (roles & 3u) == 1u;   // corner 0's slot (else 2)
  const bool l0 = (roles & 12u) == 0u, l2 = (roles & 12u) == 8u;  // the last added (else 1)
  const double sum = l0 ? s.last0 : (l2 ? s.last2 : s.last1);
  const double inv = 1.0 / sum;
  return crossing_by<Exit>(n0, n1, n2, z0, z1, z2, inv, f0, f1);
}

// the same with the reciprocal of role_sum in hand
__device__ __forceinline__ double role_sum(const ProductSums& s, unsigned roles) {
  const bool l0 = (roles & 12u) == 0u, l2 = (roles & 12u) == 8u;
  return l0 ? s.last0 : (l2 ? s.last2 : s.last1);
}
template <bool Exit>
__device__ __forceinline__ double crossing64(double n0, double n1, double n2, double z0, double z1,
                                             double z2, double inv, unsigned roles) {
  return crossing_by<Exit>(n0, n1, n2, z0, z1, z2, inv, (roles & 3u) == 0u, (roles & 3u) == 1u);
}

// 1/s, correctly rounded, from y = 1/s' of an s' within a few ulps of s.  A
// Newton step with exact remainders takes y, itself a few ulps off, to within
// one ulp of 1/s, and a second one rounds it correctly unless s has a mantissa
// of all ones (P. Markstein, IBM J. Res. Dev. 34, 1990, theorem 7); s and 1/s
// far from over- and underflow.  Four operations for a division's dozen: the
// sub-rays of grids, which wait for their own chain of operations, gain (32k
// clustered points, 120^3 at ss 2: 0.579 -> 0.528 ms; 48^3 at ss 3 0.380 ->
// 0.360); maps (-0.4 to +2.3 %) and one-thread columns (0 to +1 %) do not, so
// only accumulators with kShortChain use it.
__host__ __device__ __forceinline__ double reciprocal_near(double s, double y) {
  y = fma(fma(-s, y, 1.0), y, y);
  return fma(fma(-s, y, 1.0), y, y);
}
__device__ __forceinline__ bool mantissa_all_ones(double s) {
  return ((uint32_t)__double2loint(s) & ((uint32_t)__double2hiint(s) | 0xFFF00000u)) == 0xFFFFFFFFu;
}

// Whether three products are all above kZero in magnitude, and below 2^512 (no
// sum of them, or its reciprocal, is then near over- or underflow).  From the
// high words alone: what lies within 2^-20 of kZero is left to the general step.
constexpr uint32_t kZeroHigh = 0x3D838800u;
static_assert(kZero == 0x1.388p-39, "kZeroHigh is kZero's high word, its low word is 0");
__device__ __forceinline__ bool all_clear(double a, double b, double c) {
  constexpr uint32_t lo = 2u * (kZeroHigh + 1u), span = 2u * 0x5FF00000u - lo;
  const uint32_t u = 2u * (uint32_t)__double2hiint(a) - lo, v = 2u * (uint32_t)__double2hiint(b) - lo,
                 w = 2u * (uint32_t)__double2hiint(c) - lo;
  return max(max(u, v), w) < span;
}

// The face left through, from the apex' products with the vertices of a triangle
// of three negative products: the one without vertex k, where a_{k+1} < 0 <
// a_{k+2} (k = 0 if k0, 1 if k1, else 2).  False when the three, none of them
// zero, have one sign: the reference finds no such face.  Exact products never
// do, but the reference's are rounded by about lz*x*y*2^-53, which passes kZero in
// boxes of side 100 and more: the signs at an apex on the ray are then noise.
// Signs come from the high words: compared as doubles they take the FP64 pipe, which
// is near half of its rate (131k clustered points, 512^2 x 16: 1 to 2 %).
__host__ __device__ __forceinline__ bool negative(double a) {
#ifdef __CUDA_ARCH__
  return __double2hiint(a) < 0;
#else
  return a < 0.0;
#endif
}
__host__ __device__ __forceinline__ bool exit_slot(double a0, double a1, double a2, bool* k0,
                                                   bool* k1) {
  const bool p0 = !negative(a0), n1 = negative(a1), p2 = !negative(a2);
  *k0 = p2 & n1;
  *k1 = !p2 & p0;
  return *k0 | *k1 | !(p0 | n1);
}

// The triangle of record rec's entry face, in the record's order, and the
// ray's crossing of it.  False when its products are not all below -kZero:
// the general step takes the tet.
template <bool ShortChain>
__device__ __forceinline__ bool entry_triangle64(const WalkConf64& W, const Ray64& r, int rec,
                                                 Tri64* s, double* z_in) {
  const int F = rec & 3;
  const TetRec64* t = W.rec + (rec >> 2);
  const double4 a = load256(&t->v[rot_slot(F, 0)]), b = load256(&t->v[rot_slot(F, 1)]),
                c = load256(&t->v[rot_slot(F, 2)]);
  s->x0 = a.x;
  s->y0 = a.y;
  s->z0 = a.z;
  s->x1 = b.x;
  s->y1 = b.y;
  s->z1 = b.z;
  s->x2 = c.x;
  s->y2 = c.y;
  s->z2 = c.z;
  s->e01 = edge_u64(r, make_double2(a.x, a.y), make_double2(b.x, b.y));
  s->e12 = edge_u64(r, make_double2(b.x, b.y), make_double2(c.x, c.y));
  s->e20 = edge_u64(r, make_double2(c.x, c.y), make_double2(a.x, a.y));
  *z_in = crossing64<false>(s->e12, s->e20, s->e01, a.z, b.z, c.z,
                             product_sums(s->e12, s->e20, s->e01), entry_roles(F, 0));
  return s->e01 < -kZero && s->e12 < -kZero && s->e20 < -kZero &&
         (!ShortChain || all_clear(s->e01, s->e12, s->e20));
}

// The walk of one ray from the tet ft, located under hull triangle ft_tri (-1:
// not known), whose face the ray comes in through.
//
// The fast step.  Of the tet's six products (src/dtfe.c:44-64) the entry
// face's three are the previous step's, up to the exact sign that the
// reference's formula gives a reversed edge; the apex V adds a_k = U(V, P_k).
// When all three are clear of kZero and not of one sign the reference enters
// through the known face and leaves through the one without P_k, a_{k+1} < 0 <
// a_{k+2} (walk32.cu proves the rule for all 64 combinations of signs, rounded
// ones too).  Else the general step decides, on all six products.  The exit crossing and the next tet's entry crossing are
// the same point of the same triangle, each computed in the order the
// reference computes it for that face of that tet (crossing64).
//
// What bounds it: latency, with the FP64 and the ALU pipe each near half of
// their rate (66 % issue at 19 warps per SM; about 250 warp instructions a visit,
// a third of them FP64).  All six products in the mesh's order, the
// face rule on their signs and each face's operands picked by its index took
// 456, at 24 of 32 lanes.  131k clustered points, 512^2 x 16: 15.7 -> 8.8 ms;
// 32k uniform points, 256^2 x 4: 0.864 -> 0.549 ms.  Measured and not kept: the
// field's record read only when the midpoint is known (2 to 8 % slower), its
// constant part formed before the crossing (5 % slower), the next vertex and
// links fetched a step ahead in grids (1 to 6 % slower).
template <class Acc>
__device__ __forceinline__ int walk64(const WalkConf64& W, int ft, int ft_tri, double ox, double oy,
                                      uint64_t ray, Acc& acc, int* crossed_out, int* visits,
                                      int max_record) {
  *crossed_out = 0;
  if (ft < 0) return kRayMiss;
  Walk64<Acc> w;
  w.ox = ox;
  w.oy = oy;
  w.ray = ray;
  w.ctr = 0;
  w.crossed = 0;
  w.cur = ft;
  w.prev = ft;  // (the reference's walk starts as if it had come from ft itself)
  w.rec = W.link && ft_tri >= 0 ? 4 * ft + W.tri_face[ft_tri] : -1;
  Ray64 r{W.lz, -W.lz * oy, W.lz * ox};
  Tri64 s;
  double z_in = 0.0;
  uint32_t L = 3u * (uint32_t)w.rec;
  int crossed = 0, status = kWalk64On;
  bool fast = w.rec >= 0 && entry_triangle64<Acc::kShortChain>(W, r, w.rec, &s, &z_in);
  while (status == kWalk64On) {
    if (fast) {
      const uint32_t rec = L / 3u;
      const TetRec64* t = W.rec + (rec >> 2);
      const double4 V = load256(&t->v[rec & 3u]);
      const uint4 lk = __ldg(W.link + L);
      const typename Acc::Field field(t);
      const double2 v = make_double2(V.x, V.y);
      const double a0 = edge_u64(r, v, make_double2(s.x0, s.y0));
      const double a1 = edge_u64(r, v, make_double2(s.x1, s.y1));
      const double a2 = edge_u64(r, v, make_double2(s.x2, s.y2));
      bool k0, k1;
      const bool found = exit_slot(a0, a1, a2, &k0, &k1);
      const bool sure = found & (Acc::kShortChain ? all_clear(a0, a1, a2)
                                                  : (fabs(a0) > kZero) & (fabs(a1) > kZero) &
                                                        (fabs(a2) > kZero));
      const auto pick = [k0, k1](auto a, auto b, auto c) { return k0 ? a : (k1 ? b : c); };
      const uint32_t next = pick(lk.x, lk.y, lk.z);
      if (sure & (next != kLinkGeneral) & (crossed < W.max_visits)) {
        const unsigned roles = lk.w >> pick(0u, 8u, 16u);
        // the exit face: slots i = k+1, j = k+2 (mod 3) and the apex
        const double xi = pick(s.x1, s.x2, s.x0), yi = pick(s.y1, s.y2, s.y0);
        const double xj = pick(s.x2, s.x0, s.x1), yj = pick(s.y2, s.y0, s.y1);
        const double zi = pick(s.z1, s.z2, s.z0), zj = pick(s.z2, s.z0, s.z1);
        const double ei = pick(a1, a2, a0), ej = -pick(a2, a0, a1);
        s.e01 = pick(s.e12, s.e20, s.e01);
        s.e12 = ej;
        s.e20 = ei;
        s.x0 = xi;
        s.y0 = yi;
        s.z0 = zi;
        s.x1 = xj;
        s.y1 = yj;
        s.z1 = zj;
        s.x2 = V.x;
        s.y2 = V.y;
        s.z2 = V.z;
        const ProductSums sums = product_sums(s.e12, s.e20, s.e01);
        double inv = 0.0, z_out;
        if constexpr (Acc::kShortChain) {
          inv = 1.0 / role_sum(sums, roles);
          z_out = crossing64<true>(s.e12, s.e20, s.e01, s.z0, s.z1, s.z2, inv, roles);
        } else {
          z_out = crossing64<true>(s.e12, s.e20, s.e01, s.z0, s.z1, s.z2, sums, roles);
        }
        if (visits != nullptr && crossed < max_record) visits[crossed] = (int)(rec >> 2);
        ++crossed;
        acc.visit(ox, oy, field, z_in, z_out);
        if (next == kLinkHull) {
          status = kRayOk;
          break;
        }
        if constexpr (Acc::kShortChain) {
          const double sum = role_sum(sums, roles >> 4);
          const double y = mantissa_all_ones(sum) ? 1.0 / sum : reciprocal_near(sum, inv);
          z_in = crossing64<false>(s.e12, s.e20, s.e01, s.z0, s.z1, s.z2, y, roles >> 4);
        } else {
          z_in = crossing64<false>(s.e12, s.e20, s.e01, s.z0, s.z1, s.z2, sums, roles >> 4);
        }
        L = next;
        continue;
      }
      w.cur = (int)(rec >> 2);
      w.prev = crossed > 0 ? nb_at(__ldg(&W.rows[2 * (size_t)w.cur + 1]), (int)(rec & 3u)) : w.cur;
    }
    w.acc = acc;
    w.crossed = crossed;
    status = general_step64(W, w, visits, max_record);
    acc = w.acc;
    crossed = w.crossed;
    if (status != kWalk64On) break;
    ox = w.ox;
    oy = w.oy;
    r.m_oy = -W.lz * oy;
    r.ox_l = W.lz * ox;
    fast = w.rec >= 0 && entry_triangle64<Acc::kShortChain>(W, r, w.rec, &s, &z_in);
    L = 3u * (uint32_t)w.rec;
  }
  if (status != kRayOk) return status;
  *crossed_out = crossed;
  return kRayOk;
}

}  // namespace sdtfe
