// FP64 direct-sum accelerations for error reports: every result of the
// Barnes-Hut path can be compared with the exact (all-pairs) sum on the same
// positions. A warp takes kTargets targets; each lane sums a stride of the sources
// for all of them with Neumaier compensation, and the 32 partial sums are combined
// in a fixed butterfly with exact two-sums, so the result does not depend on
// scheduling. The sources are cut into as many chunks as n alone says, and the
// chunks' sums are combined in order the same way.
// The pair term follows gravity (src/main.cpp:306-333): normalize(d) * M * G * r^-2,
// or 1 / (r^2 + e^-r) with damping.
//
// Bound: the FP64 pipe, at about 39 FP64 instructions a pair. One target per warp
// over all sources, with the pair term as written above, took 137 warp instructions a
// pair, 70 of them FP64 (a square root, four divides, three Neumaier sums), waited on
// its loads and used 44% of the pipe; with few targets most of the chip was idle.
// 100,000 particles: 3.39 -> 1.31 ms for 4096 targets (damped 4.35 -> 2.72), 2.05 ->
// 0.12 ms for 100. A pair's terms with the products of the offset and G M r^-3 have a root
// mean square error of 1.50e-16 against an 80-bit one (with a square root and divides: 1.57e-16).
#include "direct.cuh"
#include "fp64.cuh"

namespace nbody {

namespace {

__device__ inline void neumaier(double &sum, double &comp, double g) {
    const double t = sum + g;
    comp += fabs(sum) >= fabs(g) ? (sum - t) + g : (g - t) + sum;
    sum = t;
}

// (s, c) += (s2, c2) with the rounding error of s + s2 kept exactly (TwoSum).
__device__ inline void combine(double &s, double &c, double s2, double c2) {
    const double t = s + s2;
    const double bp = t - s;
    const double err = (s - (t - bp)) + (s2 - bp);
    s = t;
    c = c + c2 + err;
}

constexpr int kTargets = 2;       // targets per warp (1, 2, 3 and 4 within 6%; fewer keep more warps for few targets)
constexpr int kDirectWarps = 4;   // warps per block, on the same sources
constexpr uint32_t kDirectChunk = 8192;   // sources per chunk, until there are
constexpr uint32_t kDirectMaxChunks = 16;  // this many chunks
constexpr uint32_t kDirectSlab = 65536;   // targets per launch: bounds the chunk sums

// G M r^-3, by which a pair's offset is multiplied. The products are taken in an order in
// which none leaves the exponent range unless r^2 or the result does.
__device__ inline double pair_factor(double r2, double gm) {
    double e;
    const double y = approx_inverse(r2, e);
    const double p = __dmul_rn(__dmul_rn(gm, y), __dmul_rn(y, y));
    return fma(p, __dmul_rn(e, fma(e, 1.875, 1.5)), p);
}
// With damping: G M / (r (r^2 + e^-r)).
__device__ inline double damped_factor(double r2, double gm) {
    const double r = __dsqrt_rn(r2);
    return __ddiv_rn(__ddiv_rn(gm, r2 + exp(-r)), r);
}

// Whether a factor is well inside the exponent range (false for zero, infinities, NaN).
// One that is not may belong to an ordinary force: G M r^-3 of a mass of 1e11 at 1e-105.
__device__ inline bool ordinary(double f) { return 2u * (uint32_t)__double2hiint(f) - (123u << 21) < (1800u << 21); }

// The term as the reference forms it. A call, so that the loop's registers need not hold
// it (inlined: 1.31 -> 1.32 ms, damped 2.72 -> 3.02).
template <bool kDamp>
__device__ __noinline__ double3 reference_term(double dx, double dy, double dz, double r2, double gm) {
    const double r = __dsqrt_rn(r2);
    const double g = __dmul_rn(gm, __ddiv_rn(1.0, kDamp ? r2 + exp(-r) : r2));
    return make_double3(__dmul_rn(__ddiv_rn(dx, r), g), __dmul_rn(__ddiv_rn(dy, r), g), __dmul_rn(__ddiv_rn(dz, r), g));
}

__device__ inline void combine_lanes(double &s, double &c, int lane) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const double s2 = __shfl_xor_sync(0xffffffffu, s, o);
        const double c2 = __shfl_xor_sync(0xffffffffu, c, o);
        // both partners combine in the same order (lower lane first) so they agree
        if (lane & o) {
            double a = s2, b = c2;
            combine(a, b, s, c);
            s = a; c = b;
        } else {
            combine(s, c, s2, c2);
        }
    }
}

// Block (x, y): kDirectWarps * kTargets targets against chunk y of the sources. With
// one chunk the results go to out, otherwise each target's (sum, compensation) of
// x, y, z to part[y][target].
template <bool kDamp>
__global__ void __launch_bounds__(kDirectWarps * 32)
    k_direct(const double *__restrict__ pos, const double *__restrict__ mass, uint32_t n, uint32_t chunk,
             const uint32_t *__restrict__ targets, uint32_t first, uint32_t m, double *__restrict__ out,
             double *__restrict__ part) {
    const uint32_t w0 = (blockIdx.x * kDirectWarps + (threadIdx.x >> 5)) * kTargets;
    const int lane = threadIdx.x & 31;
    if (w0 >= m) return;
    uint32_t ti[kTargets];
    double xi[kTargets], yi[kTargets], zi[kTargets];
    double s[kTargets][3], c[kTargets][3];
#pragma unroll
    for (int q = 0; q < kTargets; q++) {
        const uint32_t w = first + min(w0 + q, m - 1);  // past the end: the last target again, not stored
        ti[q] = targets ? targets[w] : w;
        xi[q] = pos[3 * (size_t)ti[q]]; yi[q] = pos[3 * (size_t)ti[q] + 1]; zi[q] = pos[3 * (size_t)ti[q] + 2];
#pragma unroll
        for (int d = 0; d < 3; d++) s[q][d] = c[q][d] = 0.0;
    }
    const uint32_t k0 = blockIdx.y * chunk, k1 = min(n - k0, chunk) + k0;
    for (uint32_t k = k0 + lane; k < k1; k += 32) {
        const double x = pos[3 * (size_t)k], y = pos[3 * (size_t)k + 1], z = pos[3 * (size_t)k + 2];
        const double gm = __dmul_rn(mass[k], kG);
        double f[kTargets], dx[kTargets], dy[kTargets], dz[kTargets], r2[kTargets];
        bool rare = false;
#pragma unroll
        for (int q = 0; q < kTargets; q++) {
            dx[q] = __dsub_rn(x, xi[q]); dy[q] = __dsub_rn(y, yi[q]); dz[q] = __dsub_rn(z, zi[q]);
            r2[q] = __dadd_rn(__dadd_rn(__dmul_rn(dx[q], dx[q]), __dmul_rn(dy[q], dy[q])), __dmul_rn(dz[q], dz[q]));
            f[q] = kDamp ? damped_factor(r2[q], gm) : pair_factor(r2[q], gm);
            rare |= !ordinary(f[q]);
        }
        if (!rare) {
#pragma unroll
            for (int q = 0; q < kTargets; q++) {
                neumaier(s[q][0], c[q][0], __dmul_rn(dx[q], f[q]));
                neumaier(s[q][1], c[q][1], __dmul_rn(dy[q], f[q]));
                neumaier(s[q][2], c[q][2], __dmul_rn(dz[q], f[q]));
            }
        } else {
#pragma unroll
            for (int q = 0; q < kTargets; q++) {
                if (k == ti[q]) continue;  // a particle exerts no force on itself
                double3 t = make_double3(__dmul_rn(dx[q], f[q]), __dmul_rn(dy[q], f[q]), __dmul_rn(dz[q], f[q]));
                if (!ordinary(f[q]) && !(gm == 0.0 && f[q] == 0.0)) t = reference_term<kDamp>(dx[q], dy[q], dz[q], r2[q], gm);
                neumaier(s[q][0], c[q][0], t.x);
                neumaier(s[q][1], c[q][1], t.y);
                neumaier(s[q][2], c[q][2], t.z);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kTargets; q++) {
#pragma unroll
        for (int d = 0; d < 3; d++) combine_lanes(s[q][d], c[q][d], lane);
        if (lane == 0 && w0 + q < m) {
            const size_t w = w0 + q;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (gridDim.y == 1) {
                    out[3 * w + d] = s[q][d] + c[q][d];
                } else {
                    double *p = part + 6 * ((size_t)blockIdx.y * m + w) + 2 * d;
                    p[0] = s[q][d];
                    p[1] = c[q][d];
                }
            }
        }
    }
}

// One thread per target component: the chunks' sums in order.
__global__ void k_direct_sum(const double *__restrict__ part, uint32_t chunks, uint32_t m, double *__restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * m) return;
    const uint32_t w = i / 3, d = i - 3 * w;
    double s = 0.0, c = 0.0;
    for (uint32_t k = 0; k < chunks; k++) {
        const double *p = part + 6 * ((size_t)k * m + w) + 2 * d;
        combine(s, c, p[0], p[1]);
    }
    out[i] = s + c;
}

uint32_t direct_chunks(uint32_t n) {
    const uint32_t want = n / kDirectChunk + (n % kDirectChunk ? 1u : 0u);
    return want < 1u ? 1u : want < kDirectMaxChunks ? want : kDirectMaxChunks;
}

}  // namespace

size_t direct_scratch_bytes(uint32_t n, uint32_t m) {
    const uint32_t chunks = direct_chunks(n);
    return chunks > 1 ? 48 * (size_t)chunks * (m < kDirectSlab ? m : kDirectSlab) : 0;
}

cudaError_t launch_direct(const double *pos, const double *mass, uint32_t n, int damping, const uint32_t *targets,
                          uint32_t m, double *out, double *part, cudaStream_t st, unsigned *launches) {
    const uint32_t chunks = direct_chunks(n);
    const uint32_t chunk = (n / chunks + (n % chunks ? 1u : 0u) + 31u) & ~31u;
    for (uint32_t first = 0; first < m; first += kDirectSlab) {
        const uint32_t cnt = m - first < kDirectSlab ? m - first : kDirectSlab;
        const uint32_t per_block = kDirectWarps * kTargets;
        // whole chunks of `chunk` sources; rounding up may leave fewer of them
        const dim3 grid((cnt + per_block - 1) / per_block, (n + chunk - 1) / chunk);
        double *o = out + 3 * (size_t)first;
        if (damping) k_direct<true><<<grid, kDirectWarps * 32, 0, st>>>(pos, mass, n, chunk, targets, first, cnt, o, part);
        else k_direct<false><<<grid, kDirectWarps * 32, 0, st>>>(pos, mass, n, chunk, targets, first, cnt, o, part);
        *launches += 1;
        if (grid.y > 1) {
            k_direct_sum<<<(3 * cnt + 255) / 256, 256, 0, st>>>(part, grid.y, cnt, o);
            *launches += 1;
        }
    }
    return cudaGetLastError();
}

}  // namespace nbody
