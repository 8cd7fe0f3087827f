// Velocity of a grid node from its momentum, mass and external force (host +
// device), with one reciprocal for the three components.
#pragma once

#include <cfloat>

#include "../../include/fsi_b200.h"

#if defined(__CUDACC__)
#define FSI_HD3 __host__ __device__ __forceinline__
#else
#define FSI_HD3 inline
#endif

namespace fsi {

// A particle one rounding off a cell centre on all three axes gives its corner
// node a weight of 1e-43.  The reciprocal of such a mass may be infinite, and its
// product with a momentum of zero no number; scaled by 2^64 both are exact.
// (Atomic adds to FP32 in global memory flush sums below FLT_MIN to zero, so that
// the substep's own grids hold no such mass; a node written another way may.)
struct NodeMass {
  float scale, inv;  // inv = 1 / (scale m)
};

FSI_HD3 NodeMass node_mass(float m) {  // m > 0
  NodeMass r;
  r.scale = m < FLT_MIN ? 1.8446744073709552e19f : 1.0f;
  r.inv = 1.0f / (m * r.scale);
  return r;
}

// one component after the grid update and the sticky walls (solid.py:97-111,
// 251-259): momentum and dt times the external force over the mass
FSI_HD3 float grid_node_component(float P, const NodeMass& m, float f, float gravity, int idx, int G,
                                  const FsiMpmParams& mp) {
  float u = ((P + mp.dt * f) * m.scale) * m.inv + mp.dt * gravity;
  if (idx < mp.bound && u < 0.0f) u = 0.0f;
  if (idx > G - mp.bound && u > 0.0f) u = 0.0f;
  return u;
}

}  // namespace fsi
