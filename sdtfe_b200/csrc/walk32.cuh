// walk32.cuh - record layout of the mixed-precision walk.
#pragma once

#include <cstdint>

#include "tet_links.cuh"

namespace sdtfe {

// The mixed walk's records, one per (tet, entry face) at index 4*t + F: the one
// vertex a ray that came in through face F has not seen yet, the apex (vertex
// F), and the tet's field.  32 B, one aligned 256-bit load.
struct __align__(32) TetGeo32 {
  float x, y, z, rho;  // the apex (projected frame) and its density
  float gx, gy, gz;    // gradient of the tet's linear field, projected frame
  float ext;           // extent of the tet's projection (largest x or y difference of
                       // two vertices, rounded up), a bound on |vertex - origin| for any
                       // ray that crossed one of its faces; +inf when the FP32 field
                       // value is not trusted (kFieldCond)
};
static_assert(sizeof(TetGeo32) == 32, "TetGeo32 layout");

// largest field condition (magnitudes over least vertex value) the FP32
// field value is used for
constexpr double kFieldCond = 4096.0;

}  // namespace sdtfe
