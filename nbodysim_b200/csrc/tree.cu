// Octree construction on the GPU: root cube, Morton-order keys, radix sort,
// binary radix tree, chain-free octree, bottom-up mass / centre of mass.
//
// The tree is the reference's octree (src/octree.cpp:54-196, src/main.cpp:887-927)
// with single-child chains collapsed: a node exists here iff the reference
// node at the same cell has two or more non-empty children (or is the root's
// first branching descendant). Chains carry the same mass and, up to rounding
// emulated below, the same centre of mass as their bottom node, so every
// particle's walk accepts the same bodies (see walk.cu).
#include "tree.cuh"
#include "keys.cuh"
#include "sort.cuh"

#include <cstdio>

namespace nbody {

// ---------------------------------------------------------------------------
// Root cube from the extrema: bbox midpoint; side = largest extent + 2.0, a tie
// for the largest extent falls through to the z extent (src/main.cpp:898-920).
// The FLOAT build computes it from float extrema (the extrema of the rounded
// positions are the rounded extrema): center = float(lo + hi) / 2.0 rounded to
// float, extents in float, side = float(extent + 2.0).
__device__ inline void root_from_extrema(const double *lo, const double *hi, bool single, double *center,
                                         double *side) {
    if (single) {
        float l[3], h[3];
        for (int k = 0; k < 3; k++) {
            l[k] = __double2float_rn(lo[k]);
            h[k] = __double2float_rn(hi[k]);
            center[k] = (double)__double2float_rn(__dmul_rn((double)__fadd_rn(l[k], h[k]), 0.5));
        }
        const float ex = __fsub_rn(h[0], l[0]), ey = __fsub_rn(h[1], l[1]), ez = __fsub_rn(h[2], l[2]);
        float e;
        if (ex > ey && ex > ez) e = ex;
        else if (ey > ex && ey > ez) e = ey;
        else e = ez;
        *side = (double)__double2float_rn(__dadd_rn((double)e, 2.0));
        return;
    }
    for (int k = 0; k < 3; k++) center[k] = (lo[k] + hi[k]) / 2.0;
    const double ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
    if (ex > ey && ex > ez) *side = ex + 2.0;
    else if (ey > ex && ey > ez) *side = ey + 2.0;
    else *side = ez + 2.0;
}

// Root cube (root_from_extrema) over all particles. Also flags
// non-finite positions (masses are checked where the bodies are gathered), and
// (optionally) reduces max |v| for the adaptive step.
// The first kernel of a build, so it also zeroes the sort's counters and, with
// reset, gives the pass's scalars their starting values. Those two, the digit counts
// (k_keys), their scan (each sort tile) and the full sort's 22 were launches of their
// own: a step of 97 particles 130 -> 114 us, of 5000 212 -> 191 us.
__global__ void k_bbox(const double *__restrict__ pos, const double *__restrict__ vel, uint32_t n,
                       double *__restrict__ partial, DevScalars *sc, int keep_root, int single,
                       uint4 *__restrict__ zero, size_t zero_quads, int reset) {
    griddep();
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < zero_quads; i += (size_t)gridDim.x * blockDim.x)
        zero[i] = make_uint4(0u, 0u, 0u, 0u);
    __shared__ double s_red[7][32];
    __shared__ bool s_last;
    double mn[3] = {INFINITY, INFINITY, INFINITY};
    double mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    double vmax = 0.0;
    bool bad = false;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double x = pos[3 * (size_t)i], y = pos[3 * (size_t)i + 1], z = pos[3 * (size_t)i + 2];
        bad |= !(isfinite(x) && isfinite(y) && isfinite(z));
        mn[0] = fmin(mn[0], x); mx[0] = fmax(mx[0], x);
        mn[1] = fmin(mn[1], y); mx[1] = fmax(mx[1], y);
        mn[2] = fmin(mn[2], z); mx[2] = fmax(mx[2], z);
        if (vel) {
            double vx = vel[3 * (size_t)i], vy = vel[3 * (size_t)i + 1], vz = vel[3 * (size_t)i + 2];
            vmax = fmax(vmax, vx * vx + vy * vy + vz * vz);  // |v|^2; the square root of the maximum at the end
        }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&sc->status, kStatusNonFinite);
    double v[7] = {mn[0], mn[1], mn[2], -mx[0], -mx[1], -mx[2], -vmax};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = 0; k < 7; k++) {
        double r = warp_min(v[k]);
        if (lane == 0) s_red[k][wid] = r;
    }
    __syncthreads();
    if (wid == 0) {
        for (int k = 0; k < 7; k++) {
            double r = lane < nw ? s_red[k][lane] : INFINITY;
            r = warp_min(r);
            if (lane == 0) partial[7 * blockIdx.x + k] = r;
        }
        if (lane == 0) {
            __threadfence();
            s_last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (!s_last) return;
    // The last block reduces every block's partials: each thread takes whole
    // rows (seven independent loads), then a block reduction.
    __threadfence();
    double acc[7];
#pragma unroll
    for (int k = 0; k < 7; k++) acc[k] = INFINITY;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
#pragma unroll
        for (int k = 0; k < 7; k++) acc[k] = fmin(acc[k], __ldcg(&partial[7 * b + k]));
    }
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const double m = warp_min(acc[k]);
        if (lane == 0) s_red[k][wid] = m;
    }
    __syncthreads();
    if (wid != 0) return;
    double r[7];
#pragma unroll
    for (int k = 0; k < 7; k++) r[k] = warp_min(lane < nw ? s_red[k][lane] : INFINITY);
    if (lane == 0 && reset) reset_pass(sc);
    if (lane == 0 && keep_root) {
        sc->max_vel_bits = (unsigned long long)__double_as_longlong(sqrt(-r[6]));
        sc->ticket = 0;
    } else if (lane == 0) {
        double lo[3] = {r[0], r[1], r[2]}, hi[3] = {-r[3], -r[4], -r[5]};
        for (int k = 0; k < 3; k++) {
            sc->bbox_min[k] = lo[k];
            sc->bbox_max[k] = hi[k];
        }
        double center[3], side;
        root_from_extrema(lo, hi, single != 0, center, &side);
        for (int k = 0; k < 3; k++) sc->root_center[k] = center[k];
        sc->root_side = side;
        sc->max_vel_bits = (unsigned long long)__double_as_longlong(sqrt(-r[6]));
        sc->ticket = 0;
    }
}

// Root cube per system (several independent systems): one block per system.
__global__ void k_bbox_systems(const double *__restrict__ pos, const double *__restrict__ mass,
                               const uint32_t *__restrict__ sys_start, double *__restrict__ sys_root,
                               DevScalars *sc, int single) {
    griddep();
    __shared__ double s_red[6][32];
    const uint32_t b0 = sys_start[blockIdx.x], b1 = sys_start[blockIdx.x + 1];
    double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool bad = false;
    for (uint32_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
        const double x = pos[3 * (size_t)i], y = pos[3 * (size_t)i + 1], z = pos[3 * (size_t)i + 2];
        bad |= !(isfinite(x) && isfinite(y) && isfinite(z) && isfinite(mass[i]));
        mn[0] = fmin(mn[0], x); mx[0] = fmax(mx[0], x);
        mn[1] = fmin(mn[1], y); mx[1] = fmax(mx[1], y);
        mn[2] = fmin(mn[2], z); mx[2] = fmax(mx[2], z);
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&sc->status, kStatusNonFinite);
    double v[6] = {mn[0], mn[1], mn[2], -mx[0], -mx[1], -mx[2]};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = 0; k < 6; k++) {
        const double r = warp_min(v[k]);
        if (lane == 0) s_red[k][wid] = r;
    }
    __syncthreads();
    if (wid != 0) return;
    double r[6];
    for (int k = 0; k < 6; k++) r[k] = warp_min(lane < nw ? s_red[k][lane] : INFINITY);
    if (lane == 0) {
        const double lo[3] = {r[0], r[1], r[2]}, hi[3] = {-r[3], -r[4], -r[5]};
        double *o = sys_root + 4 * (size_t)blockIdx.x;
        root_from_extrema(lo, hi, single != 0, o, o + 3);
    }
}

// ---------------------------------------------------------------------------
// Key words per particle: levels 1..21 (k1) and 22..42 (k2). Escaped
// particles can make the root cube many orders of magnitude larger than the
// bulk of the system, so the first 21 levels alone do not separate it. With
// k2_user null only k1 is computed (a sort plan that needs no second word).
// The sort key goes to `sortkey`, the identity to `idx`: the second word, or
// without it the first, or with sys_id the system's number (sys_bits) above the
// first word's top bits. The digits of the sort's passes are counted on the way,
// per block in shared memory: `passes` of the sort key (shift of the first one:
// `shift`) into slots 0.. and, with k2_user, the 8 of k1 into slots 8...
__global__ void __launch_bounds__(256)
    k_keys(const double *__restrict__ pos, uint32_t n, const DevScalars *sc, uint64_t *__restrict__ k1_user,
           uint64_t *__restrict__ sortkey, uint64_t *__restrict__ k2_user, uint32_t *__restrict__ idx,
           const uint32_t *__restrict__ sys_id, const double *__restrict__ sys_root, int sys_bits, int single,
           int passes, int shift, uint32_t *__restrict__ hist) {
    griddep();
    __shared__ uint32_t s_h[16 * 256];
    const int both = k2_user ? 8 : 0, words = k2_user ? 2 : 1;
    for (int k = threadIdx.x; k < (both ? 16 : passes) * 256; k += blockDim.x) s_h[k] = 0u;
    __syncthreads();
    double root[4] = {0.0, 0.0, 0.0, 0.0};
    if (!sys_id) {
        root[0] = sc->root_center[0]; root[1] = sc->root_center[1]; root[2] = sc->root_center[2];
        root[3] = sc->root_side;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint64_t sys = 0;
        if (sys_id) {
            sys = sys_id[i];
            const double *r = sys_root + 4 * (size_t)sys;
            root[0] = r[0]; root[1] = r[1]; root[2] = r[2]; root[3] = r[3];
        }
        const double p[3] = {pos[3 * (size_t)i], pos[3 * (size_t)i + 1], pos[3 * (size_t)i + 2]};
        uint64_t w[2] = {0, 0};
        if (single) descend_words<float>(p, root, words, w);
        else descend_words<double>(p, root, words, w);
        k1_user[i] = w[0];
        const uint64_t key = sys_id ? (sys << (64 - sys_bits)) | (w[0] >> (sys_bits - 1)) : k2_user ? w[1] : w[0];
        sortkey[i] = key;
        if (k2_user) k2_user[i] = w[1];
        idx[i] = i;
        for (int q = 0; q < passes; q++) atomicAdd(&s_h[q * 256 + ((key >> (shift + 8 * q)) & 255u)], 1u);
        for (int q = 0; q < both; q++) atomicAdd(&s_h[(8 + q) * 256 + ((w[0] >> (8 * q)) & 255u)], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < (both ? 16 : passes) * 256; k += blockDim.x)
        if (s_h[k]) atomicAdd(&hist[k], s_h[k]);
}

// dst[j] = src[idx[j]], and the systems likewise (sys_id null: none).
__global__ void k_gather_key(const uint64_t *__restrict__ src, const uint32_t *__restrict__ idx,
                             uint64_t *__restrict__ dst, uint32_t n, const uint32_t *__restrict__ sys_id,
                             uint32_t *__restrict__ sys_sorted) {
    griddep();
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t i = idx[j];
    dst[j] = src[i];
    if (sys_id) sys_sorted[j] = sys_id[i];
}

// Runs of neighbours that the sort plan left equal over its bits, (k1 >> s1)
// and, when the plan sorted part of the second word, (k2 >> s2), are put in
// order here: each run of at most kMaxTieRun particles is sorted in place by
// the full keys (k1, then k2; k2 in key_a, computed here for the run when the
// plan had no second words), with a stable insertion sort, so that equal keys
// keep the user order as the full LSD sort keeps it. Runs are disjoint and a
// permutation inside a run leaves every prefix of the run unchanged, so the
// runs are found and sorted concurrently. A longer run sets the flag of the
// full sort. Runs of several systems lie within one system.
constexpr uint32_t kMaxTieRun = 64;

__global__ void k_fix_ties(uint64_t *__restrict__ k1_sorted, uint64_t *__restrict__ k2_sorted,
                           uint32_t *__restrict__ idx, const double *__restrict__ pos, int have_k2, int s1, int s2,
                           uint32_t n, int single, const uint32_t *__restrict__ sys,
                           const double *__restrict__ sys_root, DevScalars *sc) {
    griddep();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    auto same = [&](uint32_t a, uint32_t b) {
        bool t = (k1_sorted[a] >> s1) == (k1_sorted[b] >> s1);
        if (t && have_k2) t = (k2_sorted[a] >> s2) == (k2_sorted[b] >> s2);
        if (t && sys) t = sys[a] == sys[b];
        return t;
    };
    if (j + 1 >= n || !same(j, j + 1) || (j > 0 && same(j - 1, j))) return;  // not the first of a run
    uint32_t e = j + 1;
    while (e + 1 < n && same(e, e + 1)) {
        if (++e - j + 1 > kMaxTieRun) {
            atomicOr(&sc->word_ties, 1u);
            return;
        }
    }
    atomicAdd(&sc->tie_runs, 1u);
    if (!have_k2) {
        // The plan sorted top bits of the first word only: the run is sorted by its
        // first words, and only a stretch of equal first words needs the second
        // word, computed for it here (stable sorts both, as the full sort is).
        for (uint32_t q = j + 1; q <= e; q++) {
            const uint64_t a1 = k1_sorted[q];
            const uint32_t ai = idx[q];
            uint32_t p = q;
            while (p > j && k1_sorted[p - 1] > a1) {
                k1_sorted[p] = k1_sorted[p - 1];
                idx[p] = idx[p - 1];
                p--;
            }
            k1_sorted[p] = a1;
            idx[p] = ai;
        }
        double root[4] = {sc->root_center[0], sc->root_center[1], sc->root_center[2], sc->root_side};
        if (sys) {
            const double *r = sys_root + 4 * (size_t)sys[j];
            root[0] = r[0]; root[1] = r[1]; root[2] = r[2]; root[3] = r[3];
        }
        for (uint32_t a = j; a < e;) {
            uint32_t b = a;
            while (b < e && k1_sorted[b + 1] == k1_sorted[a]) b++;
            if (b > a) {
                for (uint32_t q = a; q <= b; q++) {
                    const size_t u = 3 * (size_t)idx[q];
                    const double p[3] = {pos[u], pos[u + 1], pos[u + 2]};
                    uint64_t w[2];
                    if (single) descend_words<float>(p, root, 2, w);
                    else descend_words<double>(p, root, 2, w);
                    k2_sorted[q] = w[1];
                }
                for (uint32_t q = a + 1; q <= b; q++) {
                    const uint64_t a2 = k2_sorted[q];
                    const uint32_t ai = idx[q];
                    uint32_t p = q;
                    while (p > a && k2_sorted[p - 1] > a2) {
                        k2_sorted[p] = k2_sorted[p - 1];
                        idx[p] = idx[p - 1];
                        p--;
                    }
                    k2_sorted[p] = a2;
                    idx[p] = ai;
                }
            }
            a = b + 1;
        }
        return;
    }
    for (uint32_t q = j + 1; q <= e; q++) {
        const uint64_t a1 = k1_sorted[q], a2 = k2_sorted[q];
        const uint32_t ai = idx[q];
        uint32_t p = q;
        while (p > j && (k1_sorted[p - 1] > a1 || (k1_sorted[p - 1] == a1 && k2_sorted[p - 1] > a2))) {
            k1_sorted[p] = k1_sorted[p - 1];
            k2_sorted[p] = k2_sorted[p - 1];
            idx[p] = idx[p - 1];
            p--;
        }
        k1_sorted[p] = a1;
        k2_sorted[p] = a2;
        idx[p] = ai;
    }
}

// Exclusive prefix sum of u32 values in place: tiles of 4096 scanned per
// block, tile totals scanned by one block, then added back.
constexpr int kScanThreads = 1024;
constexpr int kScanTile = 4 * kScanThreads;

__device__ inline uint32_t block_exclusive_scan(uint32_t x, uint32_t *s_warp, uint32_t *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t incl = x;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0;
        uint32_t wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        s_warp[lane] = wi - w;
        if (lane == 31) s_warp[32] = wi;
    }
    __syncthreads();
    uint32_t r = s_warp[wid] + incl - x;
    if (total) *total = s_warp[32];
    return r;
}

__global__ void k_scan_tiles(uint32_t *__restrict__ v, uint32_t len, uint32_t *__restrict__ tile_sums) {
    griddep();
    __shared__ uint32_t s_warp[33];
    const uint32_t base = blockIdx.x * kScanTile + 4 * threadIdx.x;
    uint32_t x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = base + k < len ? v[base + k] : 0u;
    uint32_t s = x[0] + x[1] + x[2] + x[3];
    uint32_t tot;
    uint32_t run = block_exclusive_scan(s, s_warp, &tot);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (base + k < len) v[base + k] = run;
        run += x[k];
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = tot;
}

// One block: exclusive scan of up to a few thousand tile totals; writes the grand total.
__global__ void k_scan_small(uint32_t *__restrict__ v, uint32_t len, uint32_t *total) {
    griddep();
    __shared__ uint32_t s_warp[33];
    uint32_t carry = 0;
    for (uint32_t b = 0; b < len; b += blockDim.x) {
        uint32_t i = b + threadIdx.x;
        uint32_t x = i < len ? v[i] : 0u;
        uint32_t tot;
        uint32_t r = block_exclusive_scan(x, s_warp, &tot);
        if (i < len) v[i] = r + carry;
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void k_scan_add(uint32_t *__restrict__ v, uint32_t len, const uint32_t *__restrict__ tile_sums) {
    griddep();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < len) v[i] += tile_sums[i / kScanTile];
}

unsigned scan_exclusive(uint32_t *v, uint32_t len, uint32_t *tile_sums, uint32_t *total, cudaStream_t st) {
    const uint32_t tiles = (len + kScanTile - 1) / kScanTile;
    launch_pdl(k_scan_tiles, dim3(tiles), dim3(kScanThreads), 0, st, v, len, tile_sums);
    launch_pdl(k_scan_small, dim3(1), dim3(kScanThreads), 0, st, tile_sums, tiles, total);
    if (tiles > 1) launch_pdl(k_scan_add, dim3((len + 255) / 256), dim3(256), 0, st, v, len, tile_sums);
    return tiles > 1 ? 3u : 2u;
}

// ---------------------------------------------------------------------------
// Bodies in sorted order (as floats in the FLOAT build); flags non-finite masses.
__global__ void k_gather_bodies(const uint32_t *__restrict__ idx, const double *__restrict__ pos,
                                const double *__restrict__ mass, double4 *__restrict__ body,
                                uint32_t n, DevScalars *sc, int single) {
    griddep();
    uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t i = idx[j];
    double m = mass[i];
    if (!isfinite(m)) atomicOr(&sc->status, kStatusNonFinite);
    double4 b = make_double4(pos[3 * (size_t)i], pos[3 * (size_t)i + 1], pos[3 * (size_t)i + 2], m);
    if (single) {
        b.x = (double)__double2float_rn(b.x); b.y = (double)__double2float_rn(b.y);
        b.z = (double)__double2float_rn(b.z); b.w = (double)__double2float_rn(b.w);
    }
    body[j] = b;
}

// Groups of particles whose 42-level keys agree get a third key word (levels
// 43..63) and are re-sorted among themselves. Identical keys over all 63
// levels mean coincident particles (the reference recurses without bound).
constexpr int kMaxDeepGroup = 64;

// Position i: the first of such a group handles it. `root`: center, side (one system).
__device__ inline void deep_group_at(uint32_t i, const uint64_t *key1, const uint64_t *key2, uint64_t *key3,
                                     uint32_t *idx, double4 *body, uint32_t n, const uint32_t *sys,
                                     const double *sys_root, const double *one_root, DevScalars *sc, int single) {
    if (i + 1 >= n) return;
    const uint64_t k = key1[i], kk = key2[i];
    const uint32_t ss = sys ? sys[i] : 0u;
    auto same = [&](uint32_t q) { return key1[q] == k && key2[q] == kk && (!sys || sys[q] == ss); };
    if (!same(i + 1)) return;
    if (i > 0 && same(i - 1)) return;  // not the first of its group
    uint32_t e = i + 1;
    while (e + 1 < n && same(e + 1)) e++;
    const uint32_t g = e - i + 1;
    atomicAdd(&sc->deep_groups, 1u);
    atomicOr(&sc->status, kStatusDeepGroup);
    if (g > kMaxDeepGroup) {
        // More than 64 particles inside one cell of side 2^-42 of the root:
        // reported as coincident. Zero third words keep the radix tree well
        // formed (ties then break on sorted position).
        for (uint32_t j = i; j <= e; j++) key3[j] = 0;
        atomicOr(&sc->status, kStatusCoincident);
        return;
    }
    const double *r = sys ? sys_root + 4 * (size_t)ss : one_root;
    const double root[4] = {r[0], r[1], r[2], r[3]};
    for (uint32_t j = i; j <= e; j++) {
        const double4 b = body[j];
        const double p[3] = {b.x, b.y, b.z};
        uint64_t w[3];
        if (single) descend_words<float>(p, root, 3, w);
        else descend_words<double>(p, root, 3, w);
        key3[j] = w[2];
    }
    // insertion sort of the group by its third word
    for (uint32_t j = i + 1; j <= e; j++) {
        const uint64_t a3 = key3[j];
        const uint32_t ai = idx[j];
        const double4 ab = body[j];
        uint32_t p = j;
        while (p > i && key3[p - 1] > a3) {
            key3[p] = key3[p - 1]; idx[p] = idx[p - 1]; body[p] = body[p - 1];
            p--;
        }
        key3[p] = a3; idx[p] = ai; body[p] = ab;
    }
    for (uint32_t j = i; j < e; j++)
        if (key3[j] == key3[j + 1]) atomicOr(&sc->status, kStatusCoincident);
}

__global__ void k_deep_groups(const uint64_t *__restrict__ key1, const uint64_t *__restrict__ key2,
                              uint64_t *__restrict__ key3, uint32_t *__restrict__ idx,
                              double4 *__restrict__ body, uint32_t n, const uint32_t *__restrict__ sys,
                              const double *__restrict__ sys_root, DevScalars *sc, int single) {
    griddep();
    const double root[4] = {sc->root_center[0], sc->root_center[1], sc->root_center[2], sc->root_side};
    deep_group_at(blockIdx.x * blockDim.x + threadIdx.x, key1, key2, key3, idx, body, n, sys, sys_root, root, sc, single);
}

// ---------------------------------------------------------------------------
// Binary radix tree (Karras 2012, "Maximizing parallelism in the construction
// of BVHs, octrees and k-d trees"), prefix lengths in key bits over up to
// three 63-bit words; exact duplicates fall back to index bits so the tree
// stays well formed while the coincident status reports the error.
struct KeyView {
    const uint64_t *k1, *k2, *k3;
    int n;
    const uint32_t *sys;  // system per sorted position, or null (one system)
    __device__ int delta(int i, int j) const {
        if (j < 0 || j >= n) return -1;
        if (sys && sys[i] != sys[j]) return -1;  // separate systems: separate trees
        uint64_t a = k1[i], b = k1[j];
        if (a != b) return __clzll(a ^ b) - 1;
        a = k2[i]; b = k2[j];
        if (a != b) return 63 + __clzll(a ^ b) - 1;
        a = k3[i]; b = k3[j];
        if (a != b) return 126 + __clzll(a ^ b) - 1;
        return 189 + __clz((unsigned)i ^ (unsigned)j);
    }
};

__device__ inline int level_of(int delta) { return min(delta / 3, kMaxLevels); }

// KeyView::delta(i, j) for one i, with i's first key word and system held in
// registers (the kernel's stores could alias the keys, so the compiler would
// load them again for every call); the deeper words only where first words agree.
struct DeltaFrom {
    const KeyView &kv;
    int i;
    uint64_t a1;
    uint32_t si;
    __device__ DeltaFrom(const KeyView &v, int at) : kv(v), i(at), a1(v.k1[at]), si(v.sys ? v.sys[at] : 0u) {}
    __device__ int operator()(int j) const {
        if (j < 0 || j >= kv.n) return -1;
        if (kv.sys && kv.sys[j] != si) return -1;
        const uint64_t b1 = kv.k1[j];
        if (a1 != b1) return __clzll(a1 ^ b1) - 1;
        return kv.delta(i, j);
    }
};

// Binary node i, whose first pair of neighbours shares dn bits: its children, encoded
// >= 0 internal binary node, < 0 leaf ~index. Returns its prefix length.
__device__ inline int radix_node(const KeyView &kv, int i, int dn, int &left, int &right) {
    const DeltaFrom di(kv, i);
    const int dprev = di(i - 1);
    int d = (dn - dprev) >= 0 ? 1 : -1;
    int dmin = d > 0 ? dprev : dn;  // delta(i, i - d)
    int lmax = 2;
    while (di(i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (di(i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = di(j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (di(i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int lo = min(i, j), hi = max(i, j);
    left = (lo == gamma) ? ~gamma : gamma;
    right = (hi == gamma + 1) ? ~(gamma + 1) : gamma + 1;
    return dnode;
}

__global__ void k_radix_tree(KeyView kv, int32_t *__restrict__ bleft, int32_t *__restrict__ bright,
                             int32_t *__restrict__ bparent, int32_t *__restrict__ bdelta, uint32_t *max_prefix_bits,
                             uint32_t *pair_passes, uint32_t sys_bits) {
    __shared__ uint32_t hist[kPassBins];
    griddep();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = kv.n;
    // the deepest split: key bits that separate every pair of neighbours
    const int dn = i < n - 1 ? DeltaFrom(kv, i)(i + 1) : -1;
    const int wmax = __reduce_max_sync(0xffffffffu, dn);
    if ((threadIdx.x & 31) == 0 && wmax >= 0) atomicMax(max_prefix_bits, (uint32_t)wmax + 1u);
    // the pairs by the sort passes that separate them (the next build's plan):
    // per warp one shared-memory add per distinct pass count, per block one
    // global add per nonzero bin
    if (threadIdx.x < kPassBins) hist[threadIdx.x] = 0u;
    __syncthreads();
    {
        const int bin = dn >= 0 ? passes_for_bits((uint32_t)dn + 1u, sys_bits) : -1;
        const uint32_t same = __match_any_sync(0xffffffffu, bin);
        if (bin >= 0 && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&hist[bin], (uint32_t)__popc(same));
    }
    __syncthreads();
    if (threadIdx.x < kPassBins && hist[threadIdx.x]) atomicAdd(&pair_passes[threadIdx.x], hist[threadIdx.x]);
    if (i >= n - 1) return;
    // With several systems, the internal nodes of the system [s, e) are s..e-2:
    // the last particle of a system indexes no internal node.
    if (kv.sys && kv.sys[i] != kv.sys[i + 1]) {
        bdelta[i] = -1;
        return;
    }
    const bool seg_root = i == 0 || (kv.sys && kv.sys[i - 1] != kv.sys[i]);
    int left, right;
    const int dnode = radix_node(kv, i, dn, left, right);
    bleft[i] = left;
    bright[i] = right;
    bdelta[i] = dnode;
    if (left >= 0) bparent[left] = i;
    if (right >= 0) bparent[right] = i;
    if (seg_root) bparent[i] = -1;
}

// A binary node heads an octree node iff it is the root or its parent sits
// at a shallower octree level.
// Also the starting values of the collapse and the COM climb: a copy of the
// flags to be scanned in place (head_id), parents "none" (so that a child the
// collapse could not attach, reported as an error, is never followed) and zero
// arrival counts. One thread per particle (n = m + 1).
__global__ void k_head_flags(const int32_t *__restrict__ bparent, const int32_t *__restrict__ bdelta,
                             uint32_t m, uint32_t *__restrict__ flag, uint32_t *__restrict__ head_id,
                             int32_t *__restrict__ oparent, int32_t *__restrict__ leaf_oparent,
                             uint32_t *__restrict__ ocount) {
    griddep();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > m) return;
    leaf_oparent[i] = -1;
    if (i == m) return;
    oparent[i] = -1;
    ocount[i] = 0u;
    uint32_t f = 0u;  // not an internal node (the last particle of a system)
    if (bdelta[i] >= 0) {
        const int p = bparent[i];
        f = (p < 0 || level_of(bdelta[p]) < level_of(bdelta[i])) ? 1u : 0u;
    }
    flag[i] = f;
    head_id[i] = f;
}

// Octree root of every system: the head of the binary node at the system's
// first particle (none for a system of fewer than two particles).
__global__ void k_sys_roots(const uint32_t *__restrict__ sys_start, const uint32_t *__restrict__ flag,
                            const uint32_t *__restrict__ head_id, uint32_t nsys, int32_t *__restrict__ root_node) {
    griddep();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsys) return;
    const uint32_t a = sys_start[s], b = sys_start[s + 1];
    root_node[s] = (b - a >= 2 && flag[a]) ? (int32_t)head_id[a] : -1;
}

// Visits, left to right, the exits of the same-level (L) binary subtree of head i.
template <class Emit>
__device__ inline void collapse_node(int i, int L, const int32_t *bleft, const int32_t *bright, const int32_t *bdelta,
                                     Emit &&emit, uint32_t *status) {
    auto same_level = [&](int ch) { return ch >= 0 && level_of(bdelta[ch]) == L; };
    if (L >= kMaxLevels) {
        // The capped level (keys equal over every word: coincident particles,
        // reported as such) can nest deeper: an in-order walk with a stack, a
        // frame visiting its left child, then its right child.
        int fnode[8], fstate[8];
        int fs = 1;
        fnode[0] = i;
        fstate[0] = 0;
        while (fs > 0) {
            const int x = fnode[fs - 1];
            if (fstate[fs - 1] == 2) { fs--; continue; }
            const int ch = fstate[fs - 1] == 0 ? bleft[x] : bright[x];
            fstate[fs - 1]++;
            if (same_level(ch)) {
                if (fs < 8) { fnode[fs] = ch; fstate[fs] = 0; fs++; }
                else atomicOr(status, kStatusCapacity);
            } else {
                emit(ch);
            }
        }
    } else {
        // In-order walk over the same-level binary nodes. Their prefix lengths grow
        // strictly downwards and stay within the level's 3 key bits, so the walk is
        // at most 3 binary nodes deep: unrolled, with nothing in local memory.
        const int c1[2] = {bleft[i], bright[i]};
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const int x = c1[a];
            if (!same_level(x)) {
                emit(x);
                continue;
            }
            const int c2[2] = {bleft[x], bright[x]};
#pragma unroll
            for (int b = 0; b < 2; b++) {
                const int y = c2[b];
                if (!same_level(y)) {
                    emit(y);
                    continue;
                }
                const int c3[2] = {bleft[y], bright[y]};
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    if (same_level(c3[c])) atomicOr(status, kStatusCapacity);  // deeper than 3: malformed
                    else emit(c3[c]);
                }
            }
        }
    }
}

// Each head gathers, left to right, the exits of its same-level binary
// subtree: leaves and deeper heads. Left-to-right is Morton order, i.e. the
// reference's child order 0..7.
__global__ void k_collapse(const int32_t *__restrict__ bleft, const int32_t *__restrict__ bright,
                           const int32_t *__restrict__ bdelta, const uint32_t *__restrict__ head_id,
                           const uint32_t *__restrict__ flag, uint32_t m, int32_t *__restrict__ ochild,
                           int32_t *__restrict__ ometa, int32_t *__restrict__ oparent,
                           int32_t *__restrict__ leaf_oparent, DevScalars *sc) {
    griddep();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m || !flag[i]) return;
    const int id = (int)head_id[i];
    const int L = level_of(bdelta[i]);
    int nch = 0, nint = 0;
    // A child that is no binary node of this octree level becomes a child of
    // the octree node, in order.
    auto emit = [&](int ch) {
        if (nch >= 8) {
            atomicOr(&sc->status, kStatusCapacity);
            return;
        }
        if (ch < 0) {
            ochild[8 * id + nch] = ch;
            leaf_oparent[~ch] = id;
        } else {
            const int cid = (int)head_id[ch];
            ochild[8 * id + nch] = cid;
            oparent[cid] = id;
            nint++;
        }
        nch++;
    };
    collapse_node((int)i, L, bleft, bright, bdelta, emit, &sc->status);
    ometa[id] = L | (min(nch, 8) << 8) | (min(nint, 8) << 12);
    if (id == 0) oparent[0] = -1;
    // the deepest level: one atomic per group of converged lanes
    const unsigned am = __activemask();
    const uint32_t lmax = __reduce_max_sync(am, (uint32_t)L);
    if ((threadIdx.x & 31) == (unsigned)(__ffs(am) - 1)) atomicMax(&sc->depth, lmax);
}

// ---------------------------------------------------------------------------
// Bottom-up mass and centre of mass (src/octree.cpp:203-221, 252-278): the
// climb starts at the nodes whose children are all bodies, and a node is
// computed by the thread of its last node child to finish. Sums run in
// child order with explicit round-to-nearest operations (no FMA contraction),
// as the reference computes them. A child separated from its parent by k
// single-child chain nodes enters with its centre of mass passed k times
// through the chain's (c * m) / m, the value the reference's chain top holds.
constexpr int kComLanes = 4;
constexpr uint32_t kComGroupsMax = 131072;

__device__ inline double3 load_node_com(const double4 *p, double &m) {
    const double2 *q = reinterpret_cast<const double2 *>(p);
    double2 a = __ldcg(q), b = __ldcg(q + 1);
    m = b.y;
    return make_double3(a.x, a.y, b.x);
}

// Round-to-nearest arithmetic of the reference build's datatype.
__device__ inline double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ inline float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ inline double div_rn(double a, double b) { return __ddiv_rn(a, b); }
__device__ inline float div_rn(float a, float b) { return __fdiv_rn(a, b); }

// One node's mass and centre of mass from its children, in the arithmetic of
// T (double, or float for the reference's FLOAT build): child(k) is the k-th child,
// body_at(j) a body, node_at(c, mass, level) a node child's centre, mass and level.
template <typename T, class Child, class BodyAt, class NodeAt>
__device__ inline double4 node_com(int L, int nch, Child &&child, BodyAt &&body_at, NodeAt &&node_at) {
    T m = 0, sx = 0, sy = 0, sz = 0;
    for (int k = 0; k < nch; k++) {
        const int c = child(k);
        T cmk, cx, cy, cz;
        if (c < 0) {
            const double4 b = body_at(~c);
            cmk = (T)b.w;
            cx = (T)b.x; cy = (T)b.y; cz = (T)b.z;
        } else {
            double dm;
            int level;
            const double3 cc = node_at(c, dm, level);
            cmk = (T)dm;
            cx = (T)cc.x; cy = (T)cc.y; cz = (T)cc.z;
            const int chain = level - L - 1;
            for (int t = 0; t < chain; t++) {
                if (cmk == T(0)) {
                    cx = cy = cz = T(0);
                } else {
                    cx = div_rn(mul_rn(cx, cmk), cmk);
                    cy = div_rn(mul_rn(cy, cmk), cmk);
                    cz = div_rn(mul_rn(cz, cmk), cmk);
                }
            }
        }
        m = add_rn(m, cmk);
        sx = add_rn(sx, mul_rn(cx, cmk));
        sy = add_rn(sy, mul_rn(cy, cmk));
        sz = add_rn(sz, mul_rn(cz, cmk));
    }
    double4 out;
    out.w = (double)m;
    if (m == T(0)) {
        out.x = out.y = out.z = 0.0;
    } else {
        out.x = (double)div_rn(sx, m);
        out.y = (double)div_rn(sy, m);
        out.z = (double)div_rn(sz, m);
    }
    return out;
}

// (launch bounds: 4 resident blocks of 256 threads, 64 registers)
template <typename T>
__global__ void __launch_bounds__(256, 4)
    k_com(const double4 *__restrict__ body, const int32_t *__restrict__ oparent, const int32_t *__restrict__ ochild,
          const int32_t *__restrict__ ometa, double4 *onode, uint32_t *ocount, uint32_t n, DevScalars *sc) {
    griddep();
    // One thread per node; the climb starts at nodes whose children are all
    // bodies, and a node is computed by the last of its node children to finish.
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n - 1 || q >= sc->n_onodes) return;
    int p = (int)q;
    if (meta_ninternal(ometa[p]) != 0) return;
    // A well-formed tree is at most kMaxLevels + 1 internal levels deep; the
    // bound only guards against a malformed tree after a reported error.
    for (int hops = 0; p >= 0; hops++) {
        if (hops > kMaxLevels + 1 || p >= (int)(n - 1)) {
            atomicOr(&sc->status, kStatusCapacity);
            return;
        }
        // The node's structure is final (the collapse wrote it): its metadata, child
        // list and parent load before the arrival count, so that after it only the
        // children's values remain to be read.
        const int32_t meta = ometa[p];
        const int nch = meta_nchild(meta);
        const int4 *cp = reinterpret_cast<const int4 *>(ochild + 8 * (size_t)p);
        const int4 c0 = __ldg(cp), c1 = __ldg(cp + 1);
        const int up = oparent[p];
        if (hops > 0) {
            // One acquire-release count: it publishes the node this thread wrote on
            // the previous hop, and the last node child to arrive sees every
            // other child's result.
            uint32_t old;
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(&ocount[p]) : "memory");
            if (old != (uint32_t)(meta_ninternal(meta) - 1)) return;
        }
        // The reference sums the masses, then the mass-weighted centres, each in
        // child order; both sums run here in one pass over the children.
        const int L = meta_level(meta);
        const double4 out = node_com<T>(
            L, nch,
            [&](int k) {  // selects, not an indexed array (which would live in local memory)
                const int4 h = k < 4 ? c0 : c1;
                return (k & 2) ? ((k & 1) ? h.w : h.z) : ((k & 1) ? h.y : h.x);
            },
            [&](int j) { return body[j]; },
            [&](int c, double &m, int &level) {
                const double3 v = load_node_com(&onode[c], m);
                level = meta_level(ometa[c]);
                return v;
            });
        double2 *q = reinterpret_cast<double2 *>(&onode[p]);
        __stcg(q, make_double2(out.x, out.y));
        __stcg(q + 1, make_double2(out.z, out.w));
        p = up;
    }
}

// A node is computed by kComLanes lanes: each loads the children k = lane, lane +
// kComLanes, ... at once, passes them through their chains and forms the products;
// the sums then run over the children in order, every lane taking each term by
// shuffle, and the three quotients are taken by three lanes.
//
// Bound: latency of a hop (count, structure, children), of which a climb has as many
// as the octree has levels. One thread per node (k_com) loads the children one after
// another, up to 8 round trips to L2 a hop; with many nodes, whose hops overlap, its
// fewer instructions win. This against k_com: 1000 particles 16 / 29 us, 5000 18 / 39,
// 65,536 25 / 43, 100,000 33 / 47, 200,000 63 / 54, 1,048,576 231 / 154 (2 lanes: 20,
// 25, -, 33, 63, 223; 8 lanes: 16, 16, -, 33, 74, 293).
template <typename T>
__device__ inline T group_value(T v, int k) { return __shfl_sync(0xffffffffu, v, k, kComLanes); }

template <typename T>
__global__ void __launch_bounds__(256)
    k_com_groups(const double4 *__restrict__ body, const int32_t *__restrict__ oparent,
                 const int32_t *__restrict__ ochild, const int32_t *__restrict__ ometa, double4 *onode, uint32_t *ocount,
                 uint32_t n, DevScalars *sc) {
    griddep();
    constexpr int kEach = 8 / kComLanes;  // children per lane
    const unsigned FULL = 0xffffffffu;
    // The climb starts at nodes whose children are all bodies; a node is computed
    // by the group of its last node child to finish.
    const uint32_t q = (blockIdx.x * blockDim.x + threadIdx.x) / kComLanes;
    const int l = threadIdx.x % kComLanes;
    int p = -1;
    if (q < n - 1 && q < sc->n_onodes && meta_ninternal(ometa[q]) == 0) p = (int)q;
    // A well-formed tree is at most kMaxLevels + 1 internal levels deep; the
    // bound only guards against a malformed tree after a reported error.
    for (int hops = 0; __any_sync(FULL, p >= 0); hops++) {
        if (hops > kMaxLevels + 1 || p >= (int)(n - 1)) {
            atomicOr(&sc->status, kStatusCapacity);
            p = -1;
            if (hops > kMaxLevels + 1) return;  // (the same hop for the whole warp)
        }
        // The node's structure is final (the collapse wrote it): it loads before the
        // arrival count, so that after it only the children's values remain to be read.
        int meta = 0, up = -1;
        int32_t ch[kEach];
        if (p >= 0) {
            meta = ometa[p];
            up = oparent[p];
#pragma unroll
            for (int i = 0; i < kEach; i++) ch[i] = __ldg(&ochild[8 * (size_t)p + l + i * kComLanes]);
        }
        const int nch = meta_nchild(meta), L = meta_level(meta);
        if (hops > 0) {
            // One acquire-release count per node: it publishes the node this group wrote
            // on the previous hop, and the last node child to arrive sees every other
            // child's result. (The only node child needs none.)
            __syncwarp();
            uint32_t old = 0;
            if (p >= 0 && l == 0 && meta_ninternal(meta) > 1)
                asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(&ocount[p]) : "memory");
            old = group_value(old, 0);
            __syncwarp();
            if (old != (uint32_t)(meta_ninternal(meta) - 1)) p = -1;
        }
        T cm[kEach], px[kEach], py[kEach], pz[kEach];
#pragma unroll
        for (int i = 0; i < kEach; i++) {
            cm[i] = px[i] = py[i] = pz[i] = T(0);
            if (p < 0 || l + i * kComLanes >= nch) continue;
            const int c = ch[i];
            T cmk, cx, cy, cz;
            int chain = 0;
            if (c < 0) {
                const double4 b = body[~c];
                cmk = (T)b.w;
                cx = (T)b.x; cy = (T)b.y; cz = (T)b.z;
            } else {
                double dm;
                const double3 cc = load_node_com(&onode[c], dm);
                cmk = (T)dm;
                cx = (T)cc.x; cy = (T)cc.y; cz = (T)cc.z;
                chain = meta_level(ometa[c]) - L - 1;
            }
            for (int t = 0; t < chain; t++) {
                if (cmk == T(0)) {
                    cx = cy = cz = T(0);
                } else {
                    cx = div_rn(mul_rn(cx, cmk), cmk);
                    cy = div_rn(mul_rn(cy, cmk), cmk);
                    cz = div_rn(mul_rn(cz, cmk), cmk);
                }
            }
            cm[i] = cmk;
            px[i] = mul_rn(cx, cmk); py[i] = mul_rn(cy, cmk); pz[i] = mul_rn(cz, cmk);
        }
        // The reference sums the masses, then the mass-weighted centres, each in
        // child order; the terms past the last child are +0 and change nothing.
        T m = 0, sx = 0, sy = 0, sz = 0;
        const int most = (int)__reduce_max_sync(FULL, p >= 0 ? (unsigned)nch : 0u);
#pragma unroll
        for (int i = 0; i < kEach; i++) {
            if (i * kComLanes >= most) break;
#pragma unroll
            for (int k = 0; k < kComLanes; k++) {
                m = add_rn(m, group_value(cm[i], k));
                sx = add_rn(sx, group_value(px[i], k));
                sy = add_rn(sy, group_value(py[i], k));
                sz = add_rn(sz, group_value(pz[i], k));
            }
        }
        if (p >= 0) {
            double *out = reinterpret_cast<double *>(&onode[p]);
#pragma unroll
            for (int d = l; d < 4; d += kComLanes) {
                const T num = d == 0 ? sx : d == 1 ? sy : sz;
                __stcg(out + d, d == 3 ? (double)m : m == T(0) ? 0.0 : (double)div_rn(num, m));
            }
        }
        p = p >= 0 ? up : -1;
    }
}

// ---------------------------------------------------------------------------
// The whole build of a small system (root cube to mass and centre of mass) in one
// block, with keys, trees and node values in shared memory: one thread per particle,
// per binary node and per octree node.
//
// Bound of the general chain at these sizes: the latency of a dozen dependent
// kernels (3 to 6 us each, whatever they do). A step of 97 particles takes 84 us
// against 107 with the chain, of 600 109 against 134, of 1000 121 against 137. One
// thread per particle keeps every phase one pass; 1024 is the largest block.
struct SmallTree {
    uint64_t k1[kSmallTree], k2[kSmallTree], k3[kSmallTree];
    double4 body[kSmallTree], node[kSmallTree];
    int32_t child[kSmallTree][8];
    uint32_t idx[kSmallTree], head_id[kSmallTree];
    int32_t left[kSmallTree], right[kSmallTree], parent[kSmallTree], delta[kSmallTree];
    int32_t meta[kSmallTree], opar[kSmallTree], pending[kSmallTree];
    double red[7][32], root[4];
    uint32_t scan[33], most_bits, depth;
    int32_t root_done;
};

// Sorts (a, b, id) over the block, one triple per thread, ascending (b only with kTwo):
// a bitonic network, through shared memory where partners are in other warps.
template <bool kTwo>
__device__ inline void small_sort(uint64_t &a, uint64_t &b, uint32_t &id, SmallTree &s) {
    const unsigned FULL = 0xffffffffu;
    const uint32_t t = threadIdx.x;
    for (uint32_t size = 2; size <= blockDim.x; size <<= 1) {
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            uint64_t pa, pb = 0;
            uint32_t pid;
            if (stride < 32) {
                pa = __shfl_xor_sync(FULL, a, stride);
                if constexpr (kTwo) pb = __shfl_xor_sync(FULL, b, stride);
                pid = __shfl_xor_sync(FULL, id, stride);
            } else {
                s.k1[t] = a;
                if constexpr (kTwo) s.k2[t] = b;
                s.idx[t] = id;
                __syncthreads();
                pa = s.k1[t ^ stride];
                if constexpr (kTwo) pb = s.k2[t ^ stride];
                pid = s.idx[t ^ stride];
                __syncthreads();
            }
            const bool low = ((t & stride) == 0) == ((t & size) == 0);  // keeps the smaller
            bool less = pa < a;
            if (pa == a) less = kTwo ? pb < b || (pb == b && pid < id) : pid < id;
            if (less == low) {
                a = pa;
                b = pb;
                id = pid;
            }
        }
    }
    s.k1[t] = a;
    if constexpr (kTwo) s.k2[t] = b;
    s.idx[t] = id;
    __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(kSmallTree)
    k_small_tree(const double *__restrict__ pos, const double *__restrict__ vel, const double *__restrict__ mass, uint32_t n,
                 int keep_root, int reset, uint32_t *__restrict__ sidx, double4 *__restrict__ body,
                 double4 *__restrict__ onode, int32_t *__restrict__ ochild, int32_t *__restrict__ ometa,
                 int32_t *__restrict__ oparent, int32_t *__restrict__ leaf_oparent, DevScalars *sc) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    SmallTree &s = *reinterpret_cast<SmallTree *>(small_raw);
    griddep();
    constexpr bool single = sizeof(T) == 4;
    const uint32_t t = threadIdx.x;
    const int lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
    const bool mine = t < n;
    // ---- root cube, as k_bbox
    double v[7] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, -0.0};
    double p[3] = {0.0, 0.0, 0.0};
    uint32_t bad = 0;
    if (mine) {
        double4 b = make_double4(pos[3 * t], pos[3 * t + 1], pos[3 * t + 2], mass[t]);
        bad = !(isfinite(b.x) && isfinite(b.y) && isfinite(b.z) && isfinite(b.w));
        p[0] = b.x; p[1] = b.y; p[2] = b.z;
        v[0] = b.x; v[1] = b.y; v[2] = b.z; v[3] = -b.x; v[4] = -b.y; v[5] = -b.z;
        if (vel) {
            const double vx = vel[3 * t], vy = vel[3 * t + 1], vz = vel[3 * t + 2];
            v[6] = -(vx * vx + vy * vy + vz * vz);
        }
        if (single) {
            b.x = (double)__double2float_rn(b.x); b.y = (double)__double2float_rn(b.y);
            b.z = (double)__double2float_rn(b.z); b.w = (double)__double2float_rn(b.w);
        }
        s.node[t] = b;  // in user order, until the nodes need the room
        leaf_oparent[t] = -1;
    }
    for (int k = 0; k < 7; k++) {
        const double r = warp_min(v[k]);
        if (lane == 0) s.red[k][wid] = r;
    }
    if (t == 0) {
        s.most_bits = 0u;
        s.depth = 0u;
        s.root_done = 0;
        if (reset) reset_pass(sc);
    }
    bad = __syncthreads_or(bad);
    if (wid == 0) {
        double r[7];
        for (int k = 0; k < 7; k++) r[k] = warp_min(lane < nw ? s.red[k][lane] : INFINITY);
        if (lane == 0) {
            if (bad) atomicOr(&sc->status, kStatusNonFinite);
            if (!keep_root) {
                const double lo[3] = {r[0], r[1], r[2]}, hi[3] = {-r[3], -r[4], -r[5]};
                for (int k = 0; k < 3; k++) {
                    sc->bbox_min[k] = lo[k];
                    sc->bbox_max[k] = hi[k];
                }
                double center[3], side;
                root_from_extrema(lo, hi, single, center, &side);
                for (int k = 0; k < 3; k++) sc->root_center[k] = center[k];
                sc->root_side = side;
            }
            sc->max_vel_bits = (unsigned long long)__double_as_longlong(sqrt(-r[6]));
            for (int k = 0; k < 3; k++) s.root[k] = sc->root_center[k];
            s.root[3] = sc->root_side;
        }
    }
    __syncthreads();
    // ---- keys and order: by the first word, then, where two agree, by both
    uint64_t w[2] = {~0ull, ~0ull};
    uint32_t id = t;
    if (mine) descend_words<T>(p, s.root, 1, w);
    small_sort<false>(w[0], w[1], id, s);
    bool tie = t + 1 < n && s.k1[t] == s.k1[t + 1];
    if (__syncthreads_or(tie)) {
        w[1] = ~0ull;
        if (mine) {  // (the first n places hold the particles)
            const double4 b = s.node[id];
            const double q[3] = {b.x, b.y, b.z};
            descend_words<T>(q, s.root, 2, w);
        }
        small_sort<true>(w[0], w[1], id, s);
        tie = t + 1 < n && s.k1[t] == s.k1[t + 1] && s.k2[t] == s.k2[t + 1];
    } else {
        tie = false;
    }
    if (mine) s.body[t] = s.node[id];
    if (__syncthreads_or(tie)) {
        deep_group_at(t, s.k1, s.k2, s.k3, s.idx, s.body, n, nullptr, nullptr, s.root, sc, single);
        __syncthreads();
    }
    if (mine) {
        sidx[t] = s.idx[t];
        body[t] = s.body[t];
    }
    if (n < 2) return;
    // ---- binary radix tree
    const int m = (int)n - 1, i = (int)t;
    const KeyView kv{s.k1, s.k2, s.k3, (int)n, nullptr};
    const bool node = i < m;
    if (node) {
        const int dn = kv.delta(i, i + 1);
        atomicMax(&s.most_bits, (uint32_t)dn + 1u);
        int left, right;
        s.delta[i] = radix_node(kv, i, dn, left, right);
        s.left[i] = left;
        s.right[i] = right;
        if (left >= 0) s.parent[left] = i;
        if (right >= 0) s.parent[right] = i;
        if (i == 0) s.parent[0] = -1;
        s.opar[i] = -1;
    }
    __syncthreads();
    // ---- octree heads, numbered, and their children
    bool head = false;
    if (node) {
        const int q = s.parent[i];
        head = q < 0 || level_of(s.delta[q]) < level_of(s.delta[i]);
    }
    uint32_t nodes;
    const uint32_t number = block_exclusive_scan(head ? 1u : 0u, s.scan, &nodes);
    if (node) s.head_id[i] = number;
    __syncthreads();
    if (head) {
        const int L = level_of(s.delta[i]);
        int nch = 0, nint = 0;
        collapse_node(i, L, s.left, s.right, s.delta, [&](int ch) {
            if (nch >= 8) {
                atomicOr(&sc->status, kStatusCapacity);
                return;
            }
            if (ch < 0) {
                leaf_oparent[~ch] = (int)number;
            } else {
                ch = (int)s.head_id[ch];
                s.opar[ch] = (int)number;
                nint++;
            }
            s.child[number][nch++] = ch;
        }, &sc->status);
        s.meta[number] = L | (nch << 8) | (nint << 12);
        s.pending[number] = nint;
        atomicMax(&s.depth, (uint32_t)L);
    }
    __syncthreads();
    // ---- mass and centre of mass: each round, the nodes whose node children are done
    const bool onod = t < nodes;
    const int meta = onod ? s.meta[t] : 0, nch = meta_nchild(meta);
    bool done = !onod;
    for (int round = 0; round <= kMaxLevels + 1; round++) {
        const bool now = !done && *(volatile int32_t *)&s.pending[t] == 0;
        if (now) {
            s.node[t] = node_com<T>(
                meta_level(meta), nch, [&](int k) { return s.child[t][k]; }, [&](int j) { return s.body[j]; },
                [&](int c, double &cm, int &level) {
                    const double4 q = s.node[c];
                    cm = q.w;
                    level = meta_level(s.meta[c]);
                    return make_double3(q.x, q.y, q.z);
                });
            done = true;
        }
        __syncthreads();
        if (now) {
            const int up = s.opar[t];
            if (up >= 0) atomicSub(&s.pending[up], 1);
            else s.root_done = 1;
        }
        __syncthreads();
        if (s.root_done) break;
    }
    if (onod) {
        if (!done) atomicOr(&sc->status, kStatusCapacity);  // (never in a well-formed tree)
        onode[t] = s.node[t];
        ometa[t] = meta;
        oparent[t] = s.opar[t];
        for (int k = 0; k < nch; k++) ochild[8 * (size_t)t + k] = s.child[t][k];
    }
    if (t == 0) {
        sc->n_onodes = nodes;
        sc->depth = s.depth;
        sc->max_prefix_bits = s.most_bits;
    }
}

cudaError_t small_tree(const TreeBuild &tb, cudaStream_t st) {
    unsigned threads = 64;
    while (threads < tb.n) threads <<= 1;
    auto *k = tb.single ? k_small_tree<float> : k_small_tree<double>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallTree));
    if (e != cudaSuccess) return e;
    return launch_pdl(k, dim3(1), dim3(threads), sizeof(SmallTree), st, tb.pos, tb.vel_for_max, tb.mass, tb.n, tb.keep_root,
                      tb.reset, tb.idx_a, tb.body, tb.onode, tb.ochild, tb.ometa, tb.oparent, tb.leaf_oparent, tb.sc);
}

// ---------------------------------------------------------------------------
static inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

cudaError_t build_octree(const TreeBuild &tb, cudaStream_t st, unsigned *launches) {
    const uint32_t n = tb.n;
    unsigned L = 0;
    if (n == 0) return tb.reset ? launch_reset_pass(tb.sc, st) : cudaSuccess;
    const bool multi = tb.nsys > 1;
    if (is_small_tree(tb)) {
        if (tb.mass_ready) cudaStreamWaitEvent(st, tb.mass_ready, 0);
        *launches += 1;
        return small_tree(tb, st);
    }
    // The plan's passes: on the second word, on the first, or (several systems) on the
    // system's number and the first word together.
    const int p2 = multi ? 0 : tb.sort_p2, p1 = multi ? 0 : tb.sort_p1, pm = multi ? tb.sort_pm : 0;
    const int passes_used = multi ? pm : p2 > 0 ? 8 + 8 : p1;
    // root cube (+ max |v| when requested); one per system when there are several
    const unsigned bbox_blocks = std::max(1u, std::min(tb.bbox_blocks, blocks_for(n, 1024)));
    launch_pdl(k_bbox, dim3(bbox_blocks), dim3(256), 0, st, tb.pos, tb.vel_for_max, n, tb.bbox_partial, tb.sc,
               multi ? 0 : tb.keep_root, tb.single, reinterpret_cast<uint4 *>(tb.sort_scratch),
               sort_zero_words(n, passes_used) / 4, tb.reset);
    L += 1;
    if (multi) {
        if (tb.mass_ready) cudaStreamWaitEvent(st, tb.mass_ready, 0);
        launch_pdl(k_bbox_systems, dim3(tb.nsys), dim3(256), 0, st, tb.pos, tb.mass, tb.sys_start, tb.sys_root, tb.sc, tb.single);
        L += 1;
    }
    uint32_t *err = &tb.sc->status;
    const uint32_t *sys_id = multi ? tb.sys_id : nullptr, *sys_sorted = multi ? tb.sys_sorted : nullptr;
    // `count` LSD passes with shifts from `shift`, slots from `slot`, ping-ponging
    // (kin, iin) and (kout, iout): an even count leaves the result in (kin, iin),
    // an odd one in (kout, iout).
    auto passes = [&](uint64_t *kin, uint64_t *kout, uint32_t *iin, uint32_t *iout, int count, int shift, int slot) {
        for (int q = 0; q < count; q++) {
            sort_pass(kin, iin, kout, iout, n, slot + q, shift + 8 * q, tb.sort_scratch, err, kStatusSortStall, st, &L);
            uint64_t *tk = kin; kin = kout; kout = tk;
            uint32_t *ti = iin; iin = iout; iout = ti;
        }
    };
    auto gather = [&](const uint64_t *src, uint64_t *dst, const uint32_t *sid) {
        launch_pdl(k_gather_key, dim3(blocks_for(n, 256)), dim3(256), 0, st, src, tb.idx_a, dst, n, sid, tb.sys_sorted);
        L += 1;
    };
    auto keys = [&](uint64_t *sortkey, uint64_t *k2, uint32_t *idx, int count, int shift) {
        launch_pdl(k_keys, dim3(std::min(1184u, blocks_for(n, 256))), dim3(256), 0, st, tb.pos, n, tb.sc, tb.key3, sortkey,
                   k2, idx, sys_id, tb.sys_root, tb.sys_bits, tb.single, count, shift, tb.sort_scratch);
        L += 1;
    };
    FullSort full{tb.key_a, tb.key_b, tb.key3, tb.key2, tb.idx_a, tb.idx_b, sys_id, tb.sys_sorted, n, tb.sort_scratch, err,
                  kStatusSortStall, &tb.sc->word_ties, p2 > 0, tb.pos, tb.sc, tb.sys_root, tb.single};
    // Every plan leaves k1 in sorted order in key_b and the permutation in idx_a
    // (a plan with an odd pass count starts in the other buffers). The user-order
    // words: k1 in key3, k2 in key2.
    bool checked = true;
    int s1 = 0, s2 = 0;  // the tie check's shifts of the first and second words
    if (multi && pm == 0) {
        keys(tb.key_a, nullptr, tb.idx_a, 0, 0);
        full.run_if = nullptr;
        checked = false;
        sort_full(full, st, &L);
    } else if (multi) {
        const int shift = digit_shift64(pm, 0);
        uint64_t *k0 = (pm & 1) ? tb.key_b : tb.key_a, *k0o = (pm & 1) ? tb.key_a : tb.key_b;
        uint32_t *i0 = (pm & 1) ? tb.idx_b : tb.idx_a, *i0o = (pm & 1) ? tb.idx_a : tb.idx_b;
        keys(k0, nullptr, i0, pm, shift);
        passes(k0, k0o, i0, i0o, pm, shift, 0);  // result: idx_a
        gather(tb.key3, tb.key_b, sys_id);
        s1 = std::min(63, std::max(0, 63 - (8 * pm - tb.sys_bits)));
    } else if (p2 > 0) {
        uint64_t *k0 = (p2 & 1) ? tb.key_b : tb.key_a, *k0o = (p2 & 1) ? tb.key_a : tb.key_b;
        uint32_t *i0 = (p2 & 1) ? tb.idx_b : tb.idx_a, *i0o = (p2 & 1) ? tb.idx_a : tb.idx_b;
        keys(k0, tb.key2, i0, p2, digit_shift(p2, 0));
        passes(k0, k0o, i0, i0o, p2, digit_shift(p2, 0), 0);              // result: key_a, idx_a
        gather(tb.key3, tb.key_b, nullptr);                               // k1 in that order
        passes(tb.key_b, tb.key_a, tb.idx_a, tb.idx_b, 8, 0, 8);          // result: key_b, idx_a
        gather(tb.key2, tb.key_a, nullptr);                               // k2 in sorted order
        checked = p2 < 8;
        s2 = digit_shift(p2, 0);
    } else {
        uint64_t *k0 = (p1 & 1) ? tb.key_a : tb.key_b, *k0o = (p1 & 1) ? tb.key_b : tb.key_a;
        uint32_t *i0 = (p1 & 1) ? tb.idx_b : tb.idx_a, *i0o = (p1 & 1) ? tb.idx_a : tb.idx_b;
        keys(k0, nullptr, i0, p1, digit_shift(p1, 0));
        passes(k0, k0o, i0, i0o, p1, digit_shift(p1, 0), 0);  // result: key_b, idx_a
        s1 = digit_shift(p1, 0);
    }
    if (checked) {
        // Equal neighbours over the bits the plan sorted mean it did not separate
        // every particle: short runs of them are sorted in place (k2 is read, or
        // computed, only where k1 is equal), and a long one makes the full sort run,
        // a launch that otherwise returns at once.
        launch_pdl(k_fix_ties, dim3(blocks_for(n, 256)), dim3(256), 0, st, tb.key_b, tb.key_a, tb.idx_a, tb.pos,
                   p2 > 0 ? 1 : 0, s1, s2, n, tb.single, sys_sorted, tb.sys_root, tb.sc);
        L += 1;
        sort_full(full, st, &L);
    }
    if (tb.mass_ready && !multi) cudaStreamWaitEvent(st, tb.mass_ready, 0);  // the first reader of the masses
    launch_pdl(k_gather_bodies, dim3(blocks_for(n, 256)), dim3(256), 0, st, tb.idx_a, tb.pos, tb.mass, tb.body, n, tb.sc, tb.single);
    L += 1;
    *launches += L;
    if (n < 2) return cudaGetLastError();
    L = 0;
    launch_pdl(k_deep_groups, dim3(blocks_for(n, 256)), dim3(256), 0, st, tb.key_b, tb.key_a, tb.key3, tb.idx_a, tb.body, n,
                                                       sys_sorted, tb.sys_root, tb.sc, tb.single);
    KeyView kv{tb.key_b, tb.key_a, tb.key3, (int)n, sys_sorted};
    const uint32_t m = n - 1;
    launch_pdl(k_radix_tree, dim3(blocks_for(m, 256)), dim3(256), 0, st, kv, tb.bleft, tb.bright, tb.bparent, tb.bdelta,
               &tb.sc->max_prefix_bits, tb.sc->pair_passes, multi ? (uint32_t)tb.sys_bits : 0u);
    launch_pdl(k_head_flags, dim3(blocks_for(n, 256)), dim3(256), 0, st, tb.bparent, tb.bdelta, m, tb.head_flag,
               tb.head_id, tb.oparent, tb.leaf_oparent, tb.ocount);
    L += 3 + scan_exclusive(tb.head_id, m, tb.scan_tmp, &tb.sc->n_onodes, st);
    launch_pdl(k_collapse, dim3(blocks_for(m, 256)), dim3(256), 0, st, tb.bleft, tb.bright, tb.bdelta, tb.head_id, tb.head_flag,
                                                    m, tb.ochild, tb.ometa, tb.oparent, tb.leaf_oparent,
                                                    tb.sc);
    L += 1;
    if (multi) {
        launch_pdl(k_sys_roots, dim3(blocks_for(tb.nsys, 256)), dim3(256), 0, st, tb.sys_start, tb.head_flag, tb.head_id, tb.nsys,
                                                               tb.sys_root_node);
        L += 1;
    }
    *launches += L;
    return cudaGetLastError();
}

cudaError_t compute_com(const TreeBuild &tb, cudaStream_t st, unsigned *launches) {
    const uint32_t n = tb.n;
    if (n < 2 || is_small_tree(tb)) return cudaSuccess;  // (a small system's build has done it)
    // (the arrival counts were zeroed by the build's k_head_flags)
    const bool groups = n <= kComGroupsMax;
    const dim3 grid(blocks_for((uint64_t)(n - 1) * (groups ? kComLanes : 1), 256));
    launch_pdl(groups ? (tb.single ? k_com_groups<float> : k_com_groups<double>) : tb.single ? k_com<float> : k_com<double>,
               grid, dim3(256), 0, st, tb.body, tb.oparent, tb.ochild, tb.ometa, tb.onode, tb.ocount, n, tb.sc);
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace nbody
