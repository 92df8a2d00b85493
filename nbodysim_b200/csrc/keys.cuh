// Morton key words of a particle by exact descent from its root cube.
#pragma once

#include "common.cuh"

namespace nbody {

// Octant digits by descent from the root cube, rounding every child centre
// exactly as allocate_child does (src/octree.cpp:65-84: center + (+-1 * half) / 2
// with half = side / 2), and choosing the octant with strict '>' as
// add_particle does (src/octree.cpp:153-165). Digits are (z<<2)|(y<<1)|x so
// that Morton order equals the reference's child order 0..7. T is the
// reference build's datatype: double, or float for its FLOAT build.
__device__ inline double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ inline float add_rn(float a, float b) { return __fadd_rn(a, b); }

template <typename T>
__device__ inline uint64_t descend_word(T x, T y, T z, T &cx, T &cy, T &cz, T &side) {
    uint64_t key = 0;
#pragma unroll 3
    for (int l = 0; l < kLevelsPerWord; l++) {
        const T half = side / T(2);
        const T q = half / T(2);
        int bx = x > cx, by = y > cy, bz = z > cz;
        key = (key << 3) | (uint64_t)((bz << 2) | (by << 1) | bx);
        cx = add_rn(cx, bx ? q : -q);
        cy = add_rn(cy, by ? q : -q);
        cz = add_rn(cz, bz ? q : -q);
        side = half;
    }
    return key;
}

// `words` key words of one particle from the root cube (center, side).
template <typename T>
__device__ inline void descend_words(const double *p, const double *root, int words, uint64_t *out) {
    T cx = (T)root[0], cy = (T)root[1], cz = (T)root[2], s = (T)root[3];
    const T x = (T)p[0], y = (T)p[1], z = (T)p[2];
    for (int w = 0; w < words; w++) out[w] = descend_word<T>(x, y, z, cx, cy, cz, s);
}

}  // namespace nbody
