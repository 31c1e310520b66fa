// walk32.cuh - record layout of the mixed-precision walk.
#pragma once

#include <cstdint>

namespace sdtfe {

// The mixed walk's records.  A ray inside a tet knows the face it came in
// through, the "entry face" F; the step needs the one vertex it has not seen
// yet (the apex, opposite F), the tet's field, and what lies behind each of
// the three other faces.  So there is one record per (tet, entry face), at
// index 4*t + F, and the apex of record 4*t + F is vertex F of the tet.
//
// 32 B, one aligned 256-bit load:
struct __align__(32) TetGeo32 {
  float x, y, z, rho;  // the apex (projected frame) and its density
  float gx, gy, gz;    // gradient of the tet's linear field, projected frame
  float ext;           // extent of the tet's projection (largest x or y difference of
                       // two vertices, rounded up), a bound on |vertex - origin| for any
                       // ray that crossed one of its faces; +inf when the FP32 field
                       // value is not trusted (kFieldCond)
};
static_assert(sizeof(TetGeo32) == 32, "TetGeo32 layout");

// Links: which record comes next.  The walk keeps the three vertices of the
// face it last crossed in an order of its own (the two that stay, then the
// newest), which is one of three rotations of the face's listed order; a link
// names record and rotation together, L = 3*(4*n + F') + r with state slot s
// holding record slot (s + r) mod 3.  The links of (record, rotation) are one
// 16 B row at index L: x, y, z for an exit through the face opposite state
// slot 0, 1, 2.  Rotating the rows instead of the choice keeps index
// arithmetic out of the step: both loads follow from L alone.
constexpr uint32_t kLinkHull = 0xFFFFFFFFu;     // the ray leaves the mesh
constexpr uint32_t kLinkGeneral = 0xFFFFFFFEu;  // not a face shared vertex by vertex with
                                                // one orientation: general step
constexpr uint32_t kLinkLast = 0xFFFFFFFDu;     // largest L
// meshes with more tets than L can name have no links (general steps only)
constexpr long long kMaxLinkedTets = ((long long)kLinkLast + 1) / 12;

// largest field condition (magnitudes over least vertex value) the FP32
// field value is used for
constexpr double kFieldCond = 4096.0;

// device bytes of the mixed walk's records per tet and in all
constexpr size_t mixed_record_bytes(long long nt) {
  return (size_t)nt * (4 * sizeof(TetGeo32) + (nt <= kMaxLinkedTets ? 12 * 4 * sizeof(uint32_t) : 0));
}

// Original vertex slot of slot k (0..2: the entry face's vertices in the order
// the face is listed in, BDC, ACD, ADB, ABC; 3: the apex) for entry face F,
// and its inverse; two bits per entry, one byte per F.
constexpr uint32_t kRotSlots = 0xE49C782Du;
constexpr uint32_t kRotInverse = 0xE4789C63u;
__host__ __device__ constexpr int rot_slot(int F, int k) { return (int)((kRotSlots >> (8 * F + 2 * k)) & 3u); }
__host__ __device__ constexpr int rot_inv(int F, int v) { return (int)((kRotInverse >> (8 * F + 2 * v)) & 3u); }

// The rotation r of a face's three vertices u[0..2] (state order) against a
// record's slots w[0..2]: u[s] == w[(s + r) % 3], or -1 if they are not a
// rotation of one another (other vertices, or the other orientation).
__host__ __device__ inline int link_rotation(const int u[3], const int w[3]) {
  for (int r = 0; r < 3; ++r)
    if (u[0] == w[r] && u[1] == w[(r + 1) % 3] && u[2] == w[(r + 2) % 3]) return r;
  return -1;
}

}  // namespace sdtfe
