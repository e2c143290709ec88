// When the two first-order steps that orthonormalise the kept vectors (k_gs_apply) do not suffice.
#ifndef TRL_ORTHONORMAL_LIMIT_H
#define TRL_ORTHONORMAL_LIMIT_H

#include <cmath>

namespace trl_detail {

// The largest |E|, E = Z Z^T - I of K vectors, that the second step may be given. A step leaves at
// most K E^2 (each overlap is a sum over the K vectors), so it reaches eps, as Gram-Schmidt twice
// does, from overlaps up to sqrt(eps / K): 2.4e-9 for 40 vectors, 9e-10 for 256.
inline double gs_limit(int K) { return std::sqrt(0x1p-52 / K); }

} // namespace trl_detail

#endif
