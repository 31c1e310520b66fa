// Host build of the carried triangle's crossings (crossing64 in
// sdtfe_b200/csrc/walk64.cuh and the roles of tet_links.cuh) for
// tests/test_tet_links.py.  Test scaffolding only.
#include "walk64.cuh"

using namespace sdtfe;

namespace {
double product(const double* o, double lz, const double* p, const double* q) {
  // src/dtfe.c:24-26, 44-47
  const double v0 = p[0] - q[0], v1 = p[1] - q[1], v5 = p[0] * q[1] - p[1] * q[0];
  return lz * v5 + v0 * (-lz * o[1]) + v1 * (lz * o[0]);
}
}  // namespace

// Tet v[4][3], line through o along z.  out[0..3]: face_z64 of each face.
// in[F*3 + r]: the crossing of face F carried with rotation r, as an entry.
// ex[F*3 + k]: the crossing of the face left through, entered through F and
// leaving record slot k behind, on the state after the step.
extern "C" void tl_crossings(const double* v, const double* o, double lz, double* out, double* in,
                             double* ex) {
  const auto U = [&](int p, int q) { return product(o, lz, v + 3 * p, v + 3 * q); };
  const double z[4] = {v[2], v[5], v[8], v[11]};
  const double u[6] = {U(2, 1), U(2, 0), U(1, 0), U(2, 3), U(1, 3), U(3, 0)};
  for (int f = 0; f < 4; ++f) out[f] = face_z64(f, u, z);
  for (int F = 0; F < 4; ++F)
    for (int r = 0; r < 3; ++r) {
      const int s[3] = {rot_slot(F, r), rot_slot(F, (r + 1) % 3), rot_slot(F, (r + 2) % 3)};
      const double n0 = U(s[1], s[2]), n1 = U(s[2], s[0]), n2 = U(s[0], s[1]);
      in[3 * F + r] = crossing64<false>(n0, n1, n2, z[s[0]], z[s[1]], z[s[2]],
                                        product_sums(n0, n1, n2), entry_roles(F, r));
      // slots kappa + 1, kappa + 2 and the apex; the last two products with the
      // exact sign of the reversed edge, as the walk has them
      const int e[3] = {rot_slot(F, (r + 1) % 3), rot_slot(F, (r + 2) % 3), F};
      const double m0 = -U(e[2], e[1]), m1 = U(e[2], e[0]), m2 = U(e[0], e[1]);
      ex[3 * F + r] = crossing64<true>(m0, m1, m2, z[e[0]], z[e[1]], z[e[2]],
                                       product_sums(m0, m1, m2), exit_roles(F, r));
    }
}

extern "C" int tl_exit_face(int F, int k) { return rot_slot(F, k); }
extern "C" int tl_rotation(const int* u, const int* w) { return link_rotation(u, w); }

// The slot left behind for apex products a[0..2], or -1.
extern "C" int tl_exit_slot(const double* a) {
  bool k0, k1;
  if (!exit_slot(a[0], a[1], a[2], &k0, &k1)) return -1;
  return k0 ? 0 : (k1 ? 1 : 2);
}
