// Particle merging on the GPU: the reference's minimum node size pass
// (apply_minimum_size, src/main.cpp:1001-1060) and its collision capture and
// merge (src/main.cpp:386-396, 423-430, 475-516, 521-550).
//
// Both produce, per particle, a label: the user index of the particle that
// represents its merged group (itself when it is not merged). The merged
// values are stored at the representative, and a compaction keeps the
// representatives and the untouched particles in user order.
//
// Minimum size: the reference folds, bottom-up, every node whose side is below
// min_size into one particle (each node's children in child order,
// new = collide(new, child)). After the fold only the topmost such cells
// matter: a cell at the first level L* whose side is below min_size keeps one
// particle, the fold of its subtree. A chain node passes its one child's
// particle up unchanged, so the fold over the chain-free octree below the
// topmost branching node inside the cell is the reference's fold, bit for bit.
//
// Collisions: a particle records a pair with every leaf its walk accepts that
// lies closer than the collision range. A separate search finds the leaves within
// range and replays the reference's FP64 opening test exactly on their ancestors.
// Pairs become connected components
// (union-find, root = smallest user index). The reference merges the pairs in
// the iteration order of an unordered_set, so its result for a group of three
// or more depends on pointer hashes; here each component is folded in
// ascending user index. For a single pair the order does not matter
// (IEEE addition commutes), so the merged particle is the reference's bit for bit.
#include "merge.cuh"
#include "sort.cuh"
#include "tree.cuh"

namespace nbody {

namespace {

constexpr uint32_t kUnionRetries = 1u << 20;
constexpr int kFrames = kMaxLevels + 2;


struct Val {
    double x, y, z, vx, vy, vz, m;
};

// collide(a, b) (src/main.cpp:423-430) with weighted_average
// (src/vector.cpp:129-132): (a*ma + b*mb) / (ma + mb), mass ma + mb.
__device__ inline void collide_into(Val &a, const Val &b) {
    const double w = __dadd_rn(a.m, b.m);
    a.x = __ddiv_rn(__dadd_rn(__dmul_rn(a.x, a.m), __dmul_rn(b.x, b.m)), w);
    a.y = __ddiv_rn(__dadd_rn(__dmul_rn(a.y, a.m), __dmul_rn(b.y, b.m)), w);
    a.z = __ddiv_rn(__dadd_rn(__dmul_rn(a.z, a.m), __dmul_rn(b.z, b.m)), w);
    a.vx = __ddiv_rn(__dadd_rn(__dmul_rn(a.vx, a.m), __dmul_rn(b.vx, b.m)), w);
    a.vy = __ddiv_rn(__dadd_rn(__dmul_rn(a.vy, a.m), __dmul_rn(b.vy, b.m)), w);
    a.vz = __ddiv_rn(__dadd_rn(__dmul_rn(a.vz, a.m), __dmul_rn(b.vz, b.m)), w);
    a.m = w;
}

__device__ inline Val user_val(const double *pos, const double *vel, const double *mass, uint32_t u) {
    const size_t o = 3 * (size_t)u;
    return {pos[o], pos[o + 1], pos[o + 2], vel[o], vel[o + 1], vel[o + 2], mass[u]};
}

__device__ inline void store_merged(const MergeBufs &m, uint32_t r, const Val &v) {
    const size_t o = 3 * (size_t)r;
    m.mpos[o] = v.x; m.mpos[o + 1] = v.y; m.mpos[o + 2] = v.z;
    m.mvel[o] = v.vx; m.mvel[o + 1] = v.vy; m.mvel[o + 2] = v.vz;
    m.mmass[r] = v.m;
    m.rep[r] = 1u;
}

// distance() of src/vector.cpp:99-102 on (a - b), every operation rounded alone.
__device__ inline double exact_dist(double ax, double ay, double az, double bx, double by, double bz) {
    const double dx = __dsub_rn(ax, bx), dy = __dsub_rn(ay, by), dz = __dsub_rn(az, bz);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

__global__ void k_merge_init(MergeBufs m, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMcCount) m.counters[i] = 0u;
    if (i >= n) return;
    m.label[i] = i;
    m.rep[i] = 0u;
    m.flag[i] = 0u;
}

// One thread per octree node; the topmost nodes at or below level L* fold their subtree.
__global__ void k_min_size(Tree t, const int32_t *__restrict__ oparent, const double *__restrict__ vel,
                           double min_size, MergeBufs m) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (t.n < 2 || p >= t.sc->n_onodes) return;
    const double S = t.sc->root_side;
    int ls = 0;  // first level whose cells are smaller than min_size (sides halve exactly)
    while (ls <= kMaxLevels && !(S * exp2_neg(ls) < min_size)) ls++;
    if (meta_level(t.ometa[p]) < ls) return;
    if (p != 0) {
        const int32_t par = oparent[p];
        if (par < 0 || meta_level(t.ometa[par]) >= ls) return;
    }
    // post-order fold with an explicit stack of frames (levels strictly increase downwards)
    int node[kFrames], next[kFrames];
    bool has[kFrames];
    Val acc[kFrames];
    int top = 0;
    node[0] = (int)p; next[0] = 0; has[0] = false;
    uint32_t jmin = 0xffffffffu, jmax = 0, umin = 0xffffffffu;
    Val out{};
    bool done = false;
    for (uint32_t guard = 0; guard < 4 * t.n + 64 && !done; guard++) {
        const int q = node[top];
        if (next[top] >= meta_nchild(t.ometa[q])) {
            const Val v = acc[top];
            if (top == 0) {
                out = v;
                done = true;
                break;
            }
            top--;
            if (!has[top]) { acc[top] = v; has[top] = true; }
            else collide_into(acc[top], v);
            continue;
        }
        const int32_t ch = t.ochild[8 * q + next[top]++];
        if (ch < 0) {
            const uint32_t j = ~(uint32_t)ch;
            const double4 b = t.body[j];
            const uint32_t u = t.sidx[j];
            const size_t o = 3 * (size_t)u;
            const Val v{b.x, b.y, b.z, vel[o], vel[o + 1], vel[o + 2], b.w};
            jmin = min(jmin, j); jmax = max(jmax, j); umin = min(umin, u);
            if (!has[top]) { acc[top] = v; has[top] = true; }
            else collide_into(acc[top], v);
        } else if (top + 1 < kFrames) {
            top++;
            node[top] = ch; next[top] = 0; has[top] = false;
        } else {
            break;
        }
    }
    if (!done || umin == 0xffffffffu) {
        atomicOr(&m.counters[kMcStatus], kMergeStatusTree);
        return;
    }
    store_merged(m, umin, out);
    for (uint32_t j = jmin; j <= jmax; j++) m.label[t.sidx[j]] = umin;
    atomicAdd(&m.counters[kMcGroups], 1u);
}

// Collision search: one warp per 32 Morton-consecutive particles.
//
// Bound: instruction issue. A stackless walk per particle with the exact opening
// test (FP64 square root and divide) at every node took 385 M warp instructions and
// 1.62 ms on a cube of 60,000 (range 0.5); this search takes 0.124 ms. There, lanes of a warp sit in different
// subtrees, and a node's test costs ~100 instructions. Here a lane takes one stacked
// node or leaf and asks whether it can hold a particle within range of the group's
// box (every particle of a node lies within side * sqrt(3) of its centre of mass);
// what is left is asked of every particle of the group by squared distances (without
// that, a group that straddles a large cell has a box full of nodes near no particle,
// and the few such groups take 1.2 ms). The few pairs within range then climb the
// leaf's ancestors with the exact opening test, which is what decides whether the
// reference's walk reaches the leaf.
constexpr int kFindWarps = 4;
// The stack keeps room for a depth-first descent of one entry at a time (at most 7
// more entries per level); tiles get narrower as it fills up to that reserve.
constexpr int kFindReserve = 7 * (kMaxLevels + 1) + 8;
constexpr int kFindStack = 1152;
static_assert(kFindStack - kFindReserve >= 2 * 32 * 8, "room for full tiles above the reserve");

// Whether the walk of the particle at b opens every ancestor of the leaf j (src/main.cpp:377).
__device__ inline bool opens_to_leaf(const Tree &t, const int32_t *oparent, const int32_t *leaf_oparent, uint32_t j,
                                     const double4 &b, double S, double theta, uint32_t *status) {
    int p = leaf_oparent[j];
    for (int hops = 0; p >= 0; hops++) {
        if (hops > kMaxLevels + 1 || p >= (int)(t.n - 1)) {
            atomicOr(status, kMergeStatusTree);
            return false;
        }
        const double4 nd = t.onode[p];
        const double side = S * exp2_neg(meta_level(t.ometa[p]));
        if (!(__ddiv_rn(side, exact_dist(nd.x, nd.y, nd.z, b.x, b.y, b.z)) > theta)) return false;
        p = oparent[p];
    }
    return true;
}

__global__ void __launch_bounds__(kFindWarps * 32)
    k_collide_find(Tree t, const int32_t *__restrict__ oparent, const int32_t *__restrict__ leaf_oparent, double theta,
                   double range, MergeBufs m) {
    __shared__ int32_t s_stack[kFindWarps][kFindStack];
    __shared__ double4 s_tile[kFindWarps][32];  // centre of mass or body, squared reach
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t g0 = 32 * (blockIdx.x * kFindWarps + wid);
    if (g0 >= t.n || t.n < 2) return;
    int32_t *stack = s_stack[wid];
    const unsigned FULL = 0xffffffffu;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t i = g0 + lane;
    const bool valid = i < t.n;
    const double4 bi = t.body[valid ? i : g0];
    const double lox = warp_min(bi.x), hix = warp_max(bi.x), loy = warp_min(bi.y), hiy = warp_max(bi.y),
                 loz = warp_min(bi.z), hiz = warp_max(bi.z);
    const double S = t.sc->root_side;
    int top = 1;
    if (lane == 0) stack[0] = 0;
    __syncwarp();
    uint64_t seen = 0;
    while (top > 0) {
        const int take = max(1, min(min(top, 32), (kFindStack - kFindReserve - top) / 8));
        top -= take;
        seen += take;
        if (seen > 4ull * t.n + 64) {  // more entries than a well-formed octree holds
            if (lane == 0) atomicOr(&m.counters[kMcStatus], kMergeStatusTree);
            return;
        }
        int32_t ref = -1;
        int nch = 0;
        int4 c0 = make_int4(0, 0, 0, 0), c1 = c0;
        bool near = false;
        double4 q = make_double4(0.0, 0.0, 0.0, 0.0);
        if (lane < take) {
            ref = stack[top + lane];
            double reach = range;
            if (ref >= 0) {
                q = t.onode[ref];
                const int32_t meta = t.ometa[ref];
                nch = meta_nchild(meta);
                const int4 *cp = reinterpret_cast<const int4 *>(t.ochild + 8 * (size_t)ref);
                c0 = cp[0];
                c1 = cp[1];
                reach = range + S * exp2_neg(meta_level(meta)) * 1.7320508075688772;
            } else {
                q = t.body[~ref];
            }
            const double reach2 = reach * reach * (1.0 + 4e-9);
            const double dx = fmax(fmax(lox - q.x, q.x - hix), 0.0), dy = fmax(fmax(loy - q.y, q.y - hiy), 0.0),
                         dz = fmax(fmax(loz - q.z, q.z - hiz), 0.0);
            near = !(dx * dx + dy * dy + dz * dz > reach2);
            s_tile[wid][lane] = make_double4(q.x, q.y, q.z, reach2);
        }
        __syncwarp();
        const uint32_t leaves = __ballot_sync(FULL, ref < 0);
        for (uint32_t left = __ballot_sync(FULL, near); left; left &= left - 1) {
            const int k = __ffs(left) - 1;
            const double4 e = s_tile[wid][k];
            const double dx = e.x - bi.x, dy = e.y - bi.y, dz = e.z - bi.z;
            const bool in = valid && !(dx * dx + dy * dy + dz * dz > e.w);
            if (!((leaves >> k) & 1u)) {
                const uint32_t any = __ballot_sync(FULL, in);
                if (lane == k) near = any != 0u;
                continue;
            }
            const uint32_t j = ~(uint32_t)__shfl_sync(FULL, ref, k);
            if (!in || j == i) continue;  // a particle's own leaf is never accepted
            if (!(exact_dist(e.x, e.y, e.z, bi.x, bi.y, bi.z) < range)) continue;  // src/main.cpp:386
            if (!opens_to_leaf(t, oparent, leaf_oparent, j, bi, S, theta, &m.counters[kMcStatus])) continue;
            const uint32_t ui = t.sidx[i], uj = t.sidx[j];
            const uint32_t slot = atomicAdd(&m.counters[kMcPairs], 1u);
            if (slot < m.pair_cap) m.pairs[slot] = make_uint2(min(ui, uj), max(ui, uj));
        }
        __syncwarp();
        // children of the nodes in reach
        const int myn = near && ref >= 0 ? nch : 0;
        const uint32_t q0 = __ballot_sync(FULL, myn & 1), q1 = __ballot_sync(FULL, myn & 2),
                       q2 = __ballot_sync(FULL, myn & 4), q3 = __ballot_sync(FULL, myn & 8);
        const int pre = __popc(q0 & lt) + 2 * __popc(q1 & lt) + 4 * __popc(q2 & lt) + 8 * __popc(q3 & lt);
        int32_t *dst = stack + top + pre;
        if (myn > 0) dst[0] = c0.x;
        if (myn > 1) dst[1] = c0.y;
        if (myn > 2) dst[2] = c0.z;
        if (myn > 3) dst[3] = c0.w;
        if (myn > 4) dst[4] = c1.x;
        if (myn > 5) dst[5] = c1.y;
        if (myn > 6) dst[6] = c1.z;
        if (myn > 7) dst[7] = c1.w;
        top += __popc(q0) + 2 * __popc(q1) + 4 * __popc(q2) + 8 * __popc(q3);
        __syncwarp();
    }
}

// Root of x. Links only ever point to a smaller index, so the chase ends
// within x steps; stale reads of concurrent links are still ancestors.
__device__ inline uint32_t uf_find(const uint32_t *label, uint32_t x) {
    for (;;) {
        const uint32_t y = *(const volatile uint32_t *)&label[x];
        if (y >= x) return x;
        x = y;
    }
}

__global__ void k_uf_union(MergeBufs m, uint32_t np) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= np) return;
    const uint2 pr = m.pairs[k];
    m.flag[pr.x] = 1u;
    m.flag[pr.y] = 1u;
    for (uint32_t it = 0; it < kUnionRetries; it++) {
        const uint32_t ra = uf_find(m.label, pr.x), rb = uf_find(m.label, pr.y);
        if (ra == rb) return;
        const uint32_t lo = min(ra, rb), hi = max(ra, rb);
        if (atomicCAS(&m.label[hi], hi, lo) == hi) return;  // hi was still a root: linked
    }
    atomicOr(&m.counters[kMcStatus], kMergeStatusUnion);
}

// Flattens the endpoints' labels to their roots and copies the endpoint flags for the scan.
__global__ void k_uf_flatten(MergeBufs m, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t f = m.flag[i];
    if (f) m.label[i] = uf_find(m.label, i);
    m.offs[i] = f;
}

__global__ void k_endpoint_keys(MergeBufs m, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !m.flag[i]) return;
    const uint32_t k = m.offs[i];
    m.skey_a[k] = m.label[i];
    m.sidx_a[k] = i;
}

// One thread per component (segment of equal roots, ascending user index; the
// root is the smallest index, so it comes first).
__global__ void k_fold_components(MergeBufs m, uint32_t k, const double *__restrict__ pos,
                                  const double *__restrict__ vel, const double *__restrict__ mass) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= k) return;
    const uint64_t r = m.skey_a[q];
    if (q > 0 && m.skey_a[q - 1] == r) return;
    Val acc = user_val(pos, vel, mass, m.sidx_a[q]);
    for (uint32_t s = q + 1; s < k && m.skey_a[s] == r; s++) collide_into(acc, user_val(pos, vel, mass, m.sidx_a[s]));
    store_merged(m, (uint32_t)r, acc);
}

__global__ void k_keep_flags(MergeBufs m, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) m.offs[i] = m.label[i] == i ? 1u : 0u;
}

template <typename AccT>
__global__ void k_compact(MergeBufs m, uint32_t n, const double *__restrict__ pos, const double *__restrict__ vel,
                          const double *__restrict__ mass, const AccT *__restrict__ acc) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || m.label[i] != i) return;
    const uint32_t j = m.offs[i];
    AccT *acc2 = (AccT *)m.acc2;
    const size_t o = 3 * (size_t)i, p = 3 * (size_t)j;
    if (m.rep[i]) {  // a new particle: merged state, zero acceleration
        for (int c = 0; c < 3; c++) {
            m.pos2[p + c] = m.mpos[o + c];
            m.vel2[p + c] = m.mvel[o + c];
            acc2[p + c] = (AccT)0;
        }
        m.mass2[j] = m.mmass[i];
    } else {
        for (int c = 0; c < 3; c++) {
            m.pos2[p + c] = pos[o + c];
            m.vel2[p + c] = vel[o + c];
            acc2[p + c] = acc[o + c];
        }
        m.mass2[j] = mass[i];
    }
}

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

cudaError_t merge_begin(const MergeBufs &m, uint32_t n, cudaStream_t st, unsigned *launches) {
    k_merge_init<<<blocks_for(std::max<uint32_t>(n, kMcCount), 256), 256, 0, st>>>(m, n);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t merge_min_size(const MergeBufs &m, const Tree &t, const int32_t *oparent, const double *vel,
                           double min_size, cudaStream_t st, unsigned *launches) {
    if (t.n < 2) return cudaSuccess;
    k_min_size<<<blocks_for(t.n - 1, 128), 128, 0, st>>>(t, oparent, vel, min_size, m);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t collide_find(const MergeBufs &m, const Tree &t, const int32_t *oparent, const int32_t *leaf_oparent,
                         double theta, double range, cudaStream_t st, unsigned *launches) {
    if (t.n < 2) return cudaSuccess;
    k_collide_find<<<blocks_for(t.n, kFindWarps * 32), kFindWarps * 32, 0, st>>>(t, oparent, leaf_oparent, theta, range, m);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t collide_components(const MergeBufs &m, uint32_t n, uint32_t npairs, cudaStream_t st, unsigned *launches) {
    if (npairs == 0 || n == 0) return cudaSuccess;
    k_uf_union<<<blocks_for(npairs, 256), 256, 0, st>>>(m, npairs);
    k_uf_flatten<<<blocks_for(n, 256), 256, 0, st>>>(m, n);
    *launches += 2 + scan_exclusive(m.offs, n, m.scan_tmp, &m.counters[kMcInvolved], st);
    k_endpoint_keys<<<blocks_for(n, 256), 256, 0, st>>>(m, n);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t collide_fold(const MergeBufs &m, uint32_t k, const double *pos, const double *vel, const double *mass,
                         cudaStream_t st, unsigned *launches) {
    if (k == 0) return cudaSuccess;
    // stable LSD sort of the endpoints (ascending user index) by their 32-bit root
    cudaError_t e = sort_reset(m.sort_scratch, k, 4, st);
    if (e == cudaSuccess) e = sort_histograms(m.skey_a, 0, k, m.sort_scratch, st, launches);
    if (e != cudaSuccess) return e;
    uint64_t *kin = m.skey_a, *kout = m.skey_b;
    uint32_t *iin = m.sidx_a, *iout = m.sidx_b;
    for (int q = 0; q < 4; q++) {
        e = sort_pass(kin, iin, kout, iout, k, q, digit_shift(8, q), m.sort_scratch, &m.counters[kMcStatus], kMergeStatusSort,
                      st, launches);
        if (e != cudaSuccess) return e;
        uint64_t *tk = kin; kin = kout; kout = tk;
        uint32_t *ti = iin; iin = iout; iout = ti;
    }
    // four passes: the result is back in skey_a / sidx_a
    k_fold_components<<<blocks_for(k, 256), 256, 0, st>>>(m, k, pos, vel, mass);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t merge_compact(const MergeBufs &m, uint32_t n, const double *pos, const double *vel, const double *mass,
                          const void *acc, bool acc_double, cudaStream_t st, unsigned *launches) {
    if (n == 0) return cudaSuccess;
    k_keep_flags<<<blocks_for(n, 256), 256, 0, st>>>(m, n);
    *launches += 1 + scan_exclusive(m.offs, n, m.scan_tmp, &m.counters[kMcKept], st);
    if (acc_double) k_compact<double><<<blocks_for(n, 256), 256, 0, st>>>(m, n, pos, vel, mass, (const double *)acc);
    else k_compact<float><<<blocks_for(n, 256), 256, 0, st>>>(m, n, pos, vel, mass, (const float *)acc);
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace nbody
