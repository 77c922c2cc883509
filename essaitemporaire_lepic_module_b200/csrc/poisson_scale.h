// The scale of the Poisson solves' residual norm (Src/pdesolver.f90:91-111):
// the nodes 1..n+1 times the centre coefficient.  The product is formed in
// double, exact below 2^53 nodes: the solves take grids of up to 4.2e9 nodes,
// and in 32-bit integers it wraps from 2^31.
#pragma once
#include <cmath>

namespace lepic {
inline double residual_scale(const int n[3], double ac) {
  return std::fabs((n[0] + 1.0) * (n[1] + 1.0) * (n[2] + 1.0) * ac);
}
}  // namespace lepic
