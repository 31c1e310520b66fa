// tet_links.cuh - the links between walk records, shared by the FP64 and the
// mixed walk.
//
// A ray inside a tet knows the face it came in through.  Both walks carry that
// face's three vertices in an order of their own (the two that stay from step
// to step, then the newest); what a step needs to know is which (tet, entry
// face) lies behind each of the three other faces, and how the carried order
// stands to the orders the mesh lists those faces in.
#pragma once

#include <cstdint>

namespace sdtfe {

// Record of (tet t, entry face F): 4*t + F.  Its slots 0..2 are the entry
// face's vertices in the order the face is listed in (BDC, ACD, ADB, ABC),
// slot 3 the apex, which is vertex F.  Original vertex of slot k for entry
// face F, and its inverse; two bits per entry, one byte per F.
constexpr uint32_t kRotSlots = 0xE49C782Du;
constexpr uint32_t kRotInverse = 0xE4789C63u;
__host__ __device__ constexpr int rot_slot(int F, int k) { return (int)((kRotSlots >> (8 * F + 2 * k)) & 3u); }
__host__ __device__ constexpr int rot_inv(int F, int v) { return (int)((kRotInverse >> (8 * F + 2 * v)) & 3u); }

// A link names record and rotation together, L = 3*(4*n + F') + r, with state
// slot s holding record slot (s + r) mod 3.  The links of (record, rotation)
// are one 16 B row at index L: x, y, z for an exit through the face opposite
// state slot 0, 1, 2, and in w one byte each of roles (below).  Rotating the
// rows instead of the choice keeps index arithmetic out of the step: its loads
// follow from L alone.
constexpr uint32_t kLinkHull = 0xFFFFFFFFu;     // the ray leaves the mesh
constexpr uint32_t kLinkGeneral = 0xFFFFFFFEu;  // not a face shared vertex by vertex with
                                                // one orientation: general step
constexpr uint32_t kLinkLast = 0xFFFFFFFDu;     // largest L
// meshes with more tets than L can name have no links (general steps only)
constexpr long long kMaxLinkedTets = ((long long)kLinkLast + 1) / 12;
constexpr int kLinkRowsPerTet = 12;

// The rotation r of a face's three vertices u[0..2] (state order) against a
// record's slots w[0..2]: u[s] == w[(s + r) % 3], or -1 if they are not a
// rotation of one another (other vertices, or the other orientation).
__host__ __device__ inline int link_rotation(const int u[3], const int w[3]) {
  for (int r = 0; r < 3; ++r)
    if (u[0] == w[r] && u[1] == w[(r + 1) % 3] && u[2] == w[(r + 2) % 3]) return r;
  return -1;
}

// Roles.  The reference computes where a ray crosses a face of a tet from the
// face's corners in an order that depends on the face's place in the tet
// (src/dtfe.c:66-211): three signed products are added, one of them last, and
// the point is ((1 - w1) - w2) z0 + w1 z1 + w2 z2.  Corner 0 is listed slot
// role_first(F), corners 1 and 2 follow in the listed order, and the product
// added last is the one opposite corner role_last(F).  (face_z64 is the same
// per face; tests/test_tet_links.py compares the two.)
__host__ __device__ constexpr int role_first(int F) { return F == 3 ? 0 : (F == 2 ? 2 : 1); }
__host__ __device__ constexpr int role_last(int F) { return F == 1 ? 0 : (F == 2 ? 2 : 1); }

// The same in state slots, two bits each: the slot of corner 0 and the slot
// whose product is added last.  For the entry face of record (., F) carried
// with rotation r the corners follow in state order.
__host__ __device__ constexpr unsigned entry_roles(int F, int r) {
  const int first = (role_first(F) - r + 3) % 3;
  return (unsigned)(first | ((first + role_last(F)) % 3) << 2);
}
// For the exit of a tet entered through F, leaving behind record slot kappa,
// on the state after the step: slots 0, 1, 2 = record slots kappa + 1,
// kappa + 2 and the apex.  Seen from this tet the face is listed the other way
// round, so the corners follow in descending state order.
__host__ __device__ constexpr unsigned exit_roles(int F, int kappa) {
  const int m = rot_slot(F, kappa);  // the face left through
  const int state[3] = {rot_slot(F, (kappa + 1) % 3), rot_slot(F, (kappa + 2) % 3), F};
  const int c0 = rot_slot(m, role_first(m));
  const int first = state[0] == c0 ? 0 : (state[1] == c0 ? 1 : 2);
  return (unsigned)(first | ((first - role_last(m) + 3) % 3) << 2);
}
constexpr bool exit_corners_descend() {
  for (int F = 0; F < 4; ++F)
    for (int kappa = 0; kappa < 3; ++kappa) {
      const int m = rot_slot(F, kappa);
      const int state[3] = {rot_slot(F, (kappa + 1) % 3), rot_slot(F, (kappa + 2) % 3), F};
      const int first = (int)(exit_roles(F, kappa) & 3u);
      for (int c = 0; c < 3; ++c)
        if (state[(first - c + 3) % 3] != rot_slot(m, (role_first(m) + c) % 3)) return false;
    }
  return true;
}
static_assert(exit_corners_descend(), "an exit face's corners do not descend in state order");

}  // namespace sdtfe
