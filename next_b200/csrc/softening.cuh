// The reference's softening law, split into the part a node fixes and the part
// a target adds (shared by the upward pass, which stores the node's part, and
// the plain walk).  Compiled with -fmad=false wherever it is used, so every
// operation rounds as src/dt/softening.h:21-35 and src/gravity/octree.h:145-148.
#pragma once

namespace nb {

__device__ __forceinline__ double dmax_like_std(double a, double b) { return (a < b) ? b : a; }

// eps_size + eps_mass of nextSoftening: cell size and mass only.
__device__ __forceinline__ double softening_base(double size, double mass) {
    const double eps_size = size * 0.015;
    const double eps_mass = cbrt(mass) * 0.002;
    return eps_size + eps_mass;
}

// nextSoftening from that base and the distance.
__device__ __forceinline__ double softening_at(double base, double dist) {
    const double taper = 1.0 / (1.0 + dist * 10.0);
    return dmax_like_std(base * taper, 1e-4);
}

// The dark-matter rule's softening of a target of mass mi (type 1).
__device__ __forceinline__ double softening_dark(double size, double mass, double mi) {
    return 2.0 * size / pow(mass / mi, 0.333333333);
}

}  // namespace nb
