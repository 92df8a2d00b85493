// Fused Barnes-Hut walk + gravity, one warp per 32 Morton-consecutive particles.
//
// Semantics are the reference's per-particle BFS (src/main.cpp:368-400): a
// particle opens a node iff side / |com - x| > theta and the node is not a
// leaf, otherwise it accepts the node unless the node is its own leaf; an
// accepted node adds G M (com - x) / r^3 (src/main.cpp:306-333). Every lane
// keeps exactly its own decisions: the warp walks the union of the 32 walks,
// carrying with every queued node the mask of lanes that reached it (opened
// all its ancestors). Lanes outside the mask ignore the node, so each lane's
// accepted set is the reference's set for that particle.
//
// The octree here has no single-child chains (tree.cu). A reference chain
// above a branching node K has K's mass and K's centre of mass (to rounding),
// and a larger side; a particle that opens K opens the whole chain, and one
// that does not accepts exactly one chain node -- the same body. So the
// accepted bodies and their count match the reference.
//
// MIXED precision: coordinates enter the inner loop as FP32 offsets from the
// group's bbox centre, pair forces and accumulation are FP32. The opening test
// r^2 < (side/theta)^2 is evaluated in FP32 with a proven error band; a lane
// whose value falls inside the band re-evaluates the reference's expression
// exactly (side / sqrt(dx^2 + dy^2 + dz^2) > theta on the original values, in
// the arithmetic of the reference build: FP64, or the FLOAT build's float), so
// decisions are those of the reference.
// Accepted bodies go to one of three lists, each stored as pairs of entries
// for the packed FP32 instructions (two entries per instruction): entries that
// every lane of the group takes (no mask), entries some lanes take (a lane mask
// each), and bodies close to the group's box, whose offsets carry an FP32
// remainder so that close pairs keep FP32 accuracy of the offset itself.
// FP64 ("plain form"): the same walk with every quantity in FP64 and the
// reference's opening test evaluated directly.
#include "walk.cuh"
#include "fp64.cuh"

#include <algorithm>
#include <type_traits>

namespace nbody {

namespace {

constexpr float kU = 5.9604644775390625e-8f;  // 2^-24, FP32 unit roundoff
// Band half-width (see walk_band in the comments of k_walk): 32u q + 20u Pm sqrt(q),
// plus every r^2 below (64 u Pm)^2.
constexpr float kTolRel = 32.0f * kU;
constexpr float kTolPm = 20.0f * kU;
constexpr float kTiny = 64.0f * kU;

// 1/sqrt(x) in one special-function instruction (flush-to-zero; squared pair
// distances are never subnormal), the same ~2 ulp accuracy as rsqrtf without
// rsqrtf's subnormal fix-up instructions.
__device__ inline float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}


// Values that are the same for every lane of a group, kept in shared memory
// rather than in one register per lane.
struct GroupConsts {
    double ref[3];      // reference point: centre of the group's bounding box
    double S, s_theta;  // root side, root side / theta
    float box[6];       // group box of the FP32 offsets: lo x, hi x, lo y, hi y, lo z, hi z
    float pm_tol, tiny, near_r2, pad;
    uint32_t st[6];     // per-group statistics: entries, tiles, decisions, list, near, longest queue
};

// Floats from one pair of mixed nodes to the next: 20 and not 16, so that the stores of
// a tile's pairs spread over 16 banks instead of 4 (1M bodies: -0.8% walk time).
constexpr int kPair = 20;

// Shared memory of one warp: the tile's nodes that are decided lane by lane.
template <bool kFp64>
struct TileSmem;
template <>
struct TileSmem<false> {
    // The tile's mixed nodes, compacted and stored in pairs: pair j holds
    // x0 x1 y0 y1 z0 z1 -q0 -q1 band0 band1 reach0 reach1 ref0 ref1 - - at kPair j
    // ((com - ref).xyz, q = (side/theta)^2, the half-width of its error band, the
    // mask of lanes that reached the node, the node). Once a pair is decided,
    // its first two words hold the two open masks.
    alignas(16) float mx[16 * kPair];
};
template <>
struct TileSmem<true> {
    alignas(16) double4 tc[32];  // com.xyz (absolute), side
    double tq[32];               // (side/theta)^2
    uint32_t tr[32];             // reach mask
};

// Shared memory of one group: its interaction lists, rings of kCap entries that
// are summed in batches of 32, and the sums so far. Which lists there are:
//   MIXED forward: entries every lane takes, entries some lanes take (a lane mask
//   each), and bodies near the group's box; MIXED adjoint: the last two; FP64: one,
//   with masks.
// MIXED lists are stored in pairs of entries, so that the packed FP32
// instructions (two lanes of arithmetic each) read their operands straight from
// two 16-byte loads: entries 2j and 2j+1 occupy 8 floats
// (x0, x1, y0, y1, z0, z1, Gm0, Gm1) at 8j. The adjoint's near list is FP64.
template <bool kFp64, bool kAdj, int kCap>
struct GroupSmem;

template <int kCap>
struct GroupSmem<false, false, kCap> {
    GroupConsts gc;
    alignas(16) float lf[4 * kCap];
    alignas(16) float lp[4 * kCap];
    alignas(16) float nhi[4 * kCap];  // near: offsets rounded to FP32, G m
    alignas(16) float nlo[4 * kCap];  // and what the rounding left (x, y, z; the fourth slot is 0)
    alignas(8) uint32_t lm[kCap];
    alignas(8) uint32_t nm[kCap];
    float acc[3][3][32];              // per list and component: sums of the batches so far
};
template <int kCap>
struct GroupSmem<false, true, kCap> {
    GroupConsts gc;
    alignas(16) float lp[4 * kCap];
    alignas(16) double4 nc[kCap];     // near: com.xyz (absolute), G m
    alignas(8) uint32_t lm[kCap];
    uint32_t nm[kCap];
    int lr[kCap], nr[kCap];           // node refs
    float acc[2][3][32];
};
template <bool kAdj, int kCap>
struct GroupSmem<true, kAdj, kCap> {
    GroupConsts gc;
    alignas(16) double4 lc[kCap];     // com.xyz (absolute), G m
    uint32_t lm[kCap];
    int lr[kAdj ? kCap : 1];
    double acc[1][4][32];             // x, y, z, potential
};

// A team's block: its group, the queue, the batches summed in one turn, and what
// each warp's tile adds.
constexpr int kTeamSlots = kTeamMaxWarps + 3;
template <bool kFp64, bool kAdj>
struct TeamSmem {
    GroupSmem<kFp64, kAdj, kTeamList> g;
    TileSmem<kFp64> tile[kTeamMaxWarps];
    int2 queue[kQueueCap];
    std::conditional_t<kFp64, double, float> slot[kTeamSlots][kFp64 ? 4 : 3][32];
    alignas(16) uint32_t add[kTeamMaxWarps][4];  // entries for the three lists, children
    uint32_t cnt[32];                 // accepted nodes per lane
    uint32_t group;
};

// Shared memory of a warp that walks a group by itself; its queue is in global memory.
template <bool kFp64, bool kAdj>
struct SoloSmem {
    GroupSmem<kFp64, kAdj, kSoloList> g;
    TileSmem<kFp64> tile;
};

// The reference's FP64 opening test on the original doubles
// (src/main.cpp:377 with distance() of src/vector.cpp:99-102).
__device__ inline bool exact_open(double cx, double cy, double cz, double px, double py, double pz,
                                  double side, double theta) {
    double dx = __dsub_rn(cx, px), dy = __dsub_rn(cy, py), dz = __dsub_rn(cz, pz);
    double d = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
    return __ddiv_rn(side, d) > theta;
}

// The same test as the reference's FLOAT build evaluates it: float
// differences, their squares summed in double (pow(float, 2) promotes), the
// double square root rounded to float, then float side / float distance
// against float theta (src/main.cpp:377, src/vector.cpp:99-102, datatype float).
__device__ inline bool exact_open_f32(double cx, double cy, double cz, double px, double py, double pz,
                                      double side, float theta) {
    const float dx = __fsub_rn((float)cx, (float)px), dy = __fsub_rn((float)cy, (float)py),
                dz = __fsub_rn((float)cz, (float)pz);
    const double s = __dadd_rn(__dadd_rn(__dmul_rn((double)dx, (double)dx), __dmul_rn((double)dy, (double)dy)),
                               __dmul_rn((double)dz, (double)dz));
    const float d = __double2float_rn(__dsqrt_rn(s));
    return __fdiv_rn(__double2float_rn(side), d) > theta;
}

// The reference's opening test in the build's datatype.
__device__ inline bool ref_open(bool single, double cx, double cy, double cz, double px, double py, double pz,
                                double side, double theta, float theta_f) {
    return single ? exact_open_f32(cx, cy, cz, px, py, pz, side, theta_f)
                  : exact_open(cx, cy, cz, px, py, pz, side, theta);
}

// ---- packed FP32 pairs (sm_100 f32x2: one instruction, two FP32 lanes of work)
__device__ inline uint64_t f2pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ inline void f2unpack(uint64_t r, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ inline uint64_t f2add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ inline uint64_t f2mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ inline uint64_t f2fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Writes entry k of a paired list.
__device__ inline void put_pair_entry(float *l, int k, float x, float y, float z, float gm) {
    float *e = l + 8 * (k >> 1) + (k & 1);
    e[0] = x; e[2] = y; e[4] = z; e[6] = gm;
}

// An offset o (FP64) as hi + lo in FP32: hi = o rounded, lo = what it left, rounded.
__device__ inline float lo_part(double o, float hi) { return (float)(o - (double)hi); }

// Gravity of a batch of a paired list on this lane's particle, two entries per
// packed instruction. kMasked: entry k is taken iff `bit` is set in lm[k]; an
// entry not taken enters with inverse distance 0, so it adds exactly 0 even when
// it is the lane's own leaf (distance 0). Without kMasked every entry is taken.
// An odd count is padded with a far, massless entry. The batch's sums are returned
// in v.
//
// kComp (the near list): the entry offsets are hi + lo pairs (`lo` holds the lo
// parts in the same layout) and so is the particle's (plx, ply, plz): the
// difference is (hi - phi) + (lo - plo). When hi and phi are within a factor
// two of each other their difference is exact (Sterbenz), so a body close to
// the particle gets its offset to FP32 accuracy of the offset itself.
template <bool kDamp, bool kMasked, bool kComp = false>
__device__ inline void force_pairs_f32(float *l, const uint32_t *lm, int count, uint32_t bit, float px, float py,
                                       float pz, float (&v)[3], float *lo = nullptr, float plx = 0.f, float ply = 0.f,
                                       float plz = 0.f) {
    if (count & 1) {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) {
            put_pair_entry(l, count, 1e18f, 1e18f, 1e18f, 0.f);
            if constexpr (kComp) put_pair_entry(lo, count, 0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
    }
    const uint64_t npx = f2pack(-px, -px), npy = f2pack(-py, -py), npz = f2pack(-pz, -pz);
    uint64_t nlx = 0, nly = 0, nlz = 0;
    if constexpr (kComp) { nlx = f2pack(-plx, -plx); nly = f2pack(-ply, -ply); nlz = f2pack(-plz, -plz); }
    uint64_t sx = f2pack(0.f, 0.f), sy = sx, sz = sx;
    const int pairs = (count + 1) >> 1;
#pragma unroll 2
    for (int j = 0; j < pairs; j++) {
        const float4 A = *reinterpret_cast<const float4 *>(l + 8 * j);      // x0 x1 y0 y1
        const float4 B = *reinterpret_cast<const float4 *>(l + 8 * j + 4);  // z0 z1 g0 g1
        const float g0 = B.z, g1 = B.w;
        uint64_t dx = f2add(f2pack(A.x, A.y), npx);
        uint64_t dy = f2add(f2pack(A.z, A.w), npy);
        uint64_t dz = f2add(f2pack(B.x, B.y), npz);
        if constexpr (kComp) {
            const float4 C = *reinterpret_cast<const float4 *>(lo + 8 * j);
            const float4 D = *reinterpret_cast<const float4 *>(lo + 8 * j + 4);
            dx = f2add(dx, f2add(f2pack(C.x, C.y), nlx));
            dy = f2add(dy, f2add(f2pack(C.z, C.w), nly));
            dz = f2add(dz, f2add(f2pack(D.x, D.y), nlz));
        }
        const uint64_t r2 = f2fma(dz, dz, f2fma(dy, dy, f2mul(dx, dx)));
        float r0, r1;
        f2unpack(r2, r0, r1);
        float i0 = rsqrt_ftz(r0), i1 = rsqrt_ftz(r1);
        if constexpr (kMasked) {
            const uint2 m = *reinterpret_cast<const uint2 *>(lm + 2 * j);
            i0 = (m.x & bit) ? i0 : 0.f;
            i1 = (m.y & bit) ? i1 : 0.f;
        }
        uint64_t f;
        if constexpr (kDamp) {
            const float q0 = r0 * i0, q1 = r1 * i1;
            f = f2pack(g0 * i0 / (r0 + expf(-q0)), g1 * i1 / (r1 + expf(-q1)));
        } else {
            const uint64_t inv = f2pack(i0, i1);
            f = f2mul(f2mul(f2mul(inv, inv), inv), f2pack(g0, g1));
        }
        sx = f2fma(f, dx, sx);
        sy = f2fma(f, dy, sy);
        sz = f2fma(f, dz, sz);
    }
    float a0, a1;
    f2unpack(sx, a0, a1); v[0] = a0 + a1;
    f2unpack(sy, a0, a1); v[1] = a0 + a1;
    f2unpack(sz, a0, a1); v[2] = a0 + a1;
}

// Per-particle accepted-body counts of a list (only when counts are requested).
__device__ inline uint32_t count_list(const uint32_t *lm, int count, uint32_t bit) {
    uint32_t c = 0;
    for (int k = 0; k < count; k++) c += (lm[k] & bit) ? 1u : 0u;
    return c;
}

// ---- adjoint pair terms (frozen decisions) --------------------------------
// For a taken pair with offset d = com - x and cotangent la = dL/da_i:
//   F = G M g(r) d,  dF/dd = G M (g I + h d d^T),  h = g'(r) / r,  dF/dM = G g d
//   undamped g = r^-3, h = -3 r^-5; damped g = 1 / (r (r^2 + e^-r)).
// v = (dF/dd) la goes to the node's centre-of-mass cotangent and, negated, to
// the particle's own position; G g (d . la) goes to the node's mass cotangent.
template <bool kDamp, typename T>
__device__ inline void pair_adjoint(T dx, T dy, T dz, T r2, T gm, T lax, T lay, T laz, T &vx, T &vy, T &vz,
                                    T &mterm) {
    if constexpr (sizeof(T) == 4) {
        // FP32: the same terms written with the unit offset u = d / r, so that no
        // factor grows faster than the force itself (h alone, ~ r^-5, overflows
        // FP32 below r ~ 2e-8): h s d = (h r^2) (u . la) u, G g s = G (g r) (u . la).
        const float inv = rsqrt_ftz(r2);
        const float ux = dx * inv, uy = dy * inv, uz = dz * inv;
        const float sh = ux * lax + uy * lay + uz * laz;
        float g, gr, hr2;
        if constexpr (kDamp) {
            const float r = r2 * inv;
            const float e = expf(-r);
            const float den = r2 + e;
            g = inv / den;
            gr = 1.f / den;
            hr2 = -(3.f * r2 + e - r * e) * inv / (den * den);
        } else {
            gr = inv * inv;
            g = gr * inv;
            hr2 = -3.f * g;
        }
        const float c = hr2 * sh;
        vx = gm * (g * lax + c * ux);
        vy = gm * (g * lay + c * uy);
        vz = gm * (g * laz + c * uz);
        mterm = float(kG) * gr * sh;
    } else {
        const T inv = plain_range(r2) ? inverse_root(r2) : 1.0 / sqrt(r2);
        const T inv2 = inv * inv;
        T g, h;
        if constexpr (kDamp) {
            const T r = r2 * inv;
            const T e = exp(-r);
            const T den = r2 + e;
            g = inv / den;
            h = -(T(3) * r2 + e - r * e) * inv2 * inv / (den * den);
        } else {
            g = inv * inv2;
            h = T(-3) * g * inv2;
        }
        const T s = dx * lax + dy * lay + dz * laz;
        const T hs = h * s;
        vx = gm * (g * lax + hs * dx);
        vy = gm * (g * lay + hs * dy);
        vz = gm * (g * laz + hs * dz);
        mterm = T(kG) * g * s;
    }
}

// Sums 32 per-lane values over the warp: lane l returns the sum over lanes of
// v[l]. Five butterfly stages (16 + 8 + 4 + 2 + 1 shuffles); at each stage a
// lane keeps the half of its values whose index has its own lane bit and sends
// the other half to its partner, so the 32 sums come out one per lane with
// only five dependent shuffles.
template <typename T>
__device__ inline T warp_transpose_sum32(T (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool h = lane & o;
#pragma unroll
        for (int i = 0; i < o; i++) {
            const T send = h ? v[i] : v[i + o];
            const T keep = h ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

// Lane l holds the warp sum of component (l & 3) of entry (l >> 2) of a chunk of
// eight: adds it to that node's (or leaf's) cotangent (x, y, z, mass).
__device__ inline void scatter_adj8(double *adj_node, double *adj_leaf, const int *lr, int k0, int count, double z,
                                    int lane) {
    const int k = k0 + (lane >> 2);
    if (k < count) {
        const int ref = lr[k];
        double *dst = ref >= 0 ? adj_node + 4 * (size_t)ref : adj_leaf + 4 * (size_t)(~ref);
        atomicAdd(dst + (lane & 3), z);
    }
}

// The list in chunks of eight entries: every lane's pair terms for the chunk,
// one transposed warp reduction, one atomic per lane. The terms are those of
// pair_adjoint, without damping two entries per packed instruction, where an entry not
// taken enters with inverse distance 0, which makes every one of its terms 0. What is
// missing of the last chunk is padded with far, massless entries that no lane takes.
//
// Bound: instruction issue, most of it these terms and the reduction (125 a chunk).
// Packed terms: adjoint walk of 65,536 bodies 470 to 435 us, 100,000 633 to 582,
// 500,000 2600 to 2300 (5000, where a team waits for one group's chain: 90 to 92).
// Damped terms are scalar, but read the same pairs: with entries of four floats 65,536
// takes 884 us instead of 893 and 5000 164 instead of 160.
template <bool kDamp>
__device__ inline void adj_list_f32(float *l, uint32_t *lm, const int *lr, int count, int lane, float px, float py,
                                    float pz, float lax, float lay, float laz, float &gx, float &gy, float &gz,
                                    double *adj_node, double *adj_leaf) {
    if (count & 7) {
        const int k = count + lane;
        __syncwarp();
        if (k < ((count + 7) & ~7)) {
            put_pair_entry(l, k, 1e18f, 1e18f, 1e18f, 0.f);
            lm[k] = 0u;
        }
        __syncwarp();
    }
    const uint32_t bit = 1u << lane;
    const uint64_t npx = f2pack(-px, -px), npy = f2pack(-py, -py), npz = f2pack(-pz, -pz);
    const uint64_t lx = f2pack(lax, lax), ly = f2pack(lay, lay), lz = f2pack(laz, laz);
    const uint64_t g2 = f2pack((float)kG, (float)kG);
    uint64_t sx = f2pack(0.f, 0.f), sy = sx, sz = sx;
    for (int k0 = 0; k0 < count; k0 += 8) {
        float v[32];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const float4 A = *reinterpret_cast<const float4 *>(l + 4 * (k0 + j));      // x0 x1 y0 y1
            const float4 B = *reinterpret_cast<const float4 *>(l + 4 * (k0 + j) + 4);  // z0 z1 g0 g1
            const uint2 m = *reinterpret_cast<const uint2 *>(lm + k0 + j);
            if constexpr (kDamp) {  // an exponential and three divides an entry: nothing to gain by packing
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float *w = v + 4 * (j + h);
                    const float dx = (h ? A.y : A.x) - px, dy = (h ? A.w : A.z) - py, dz = (h ? B.y : B.x) - pz;
                    const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                    pair_adjoint<true, float>(dx, dy, dz, r2, h ? B.w : B.z, lax, lay, laz, w[0], w[1], w[2], w[3]);
                    if (!((h ? m.y : m.x) & bit)) w[0] = w[1] = w[2] = w[3] = 0.f;
                    gx -= w[0]; gy -= w[1]; gz -= w[2];
                }
            } else {
                const uint64_t dx = f2add(f2pack(A.x, A.y), npx), dy = f2add(f2pack(A.z, A.w), npy),
                               dz = f2add(f2pack(B.x, B.y), npz);
                const uint64_t r2 = f2fma(dz, dz, f2fma(dy, dy, f2mul(dx, dx)));
                float r0, r1;
                f2unpack(r2, r0, r1);
                const uint64_t inv = f2pack((m.x & bit) ? rsqrt_ftz(r0) : 0.f, (m.y & bit) ? rsqrt_ftz(r1) : 0.f);
                const uint64_t ux = f2mul(dx, inv), uy = f2mul(dy, inv), uz = f2mul(dz, inv);
                const uint64_t sh = f2fma(uz, lz, f2fma(uy, ly, f2mul(ux, lx)));
                const uint64_t gr = f2mul(inv, inv), g = f2mul(gr, inv);
                const uint64_t gm = f2pack(B.z, B.w), c = f2mul(f2mul(g, f2pack(-3.f, -3.f)), sh);
                const uint64_t vx = f2mul(gm, f2fma(c, ux, f2mul(g, lx))), vy = f2mul(gm, f2fma(c, uy, f2mul(g, ly))),
                               vz = f2mul(gm, f2fma(c, uz, f2mul(g, lz)));
                const uint64_t mt = f2mul(f2mul(g2, gr), sh);
                sx = f2add(sx, vx); sy = f2add(sy, vy); sz = f2add(sz, vz);
                f2unpack(vx, v[4 * j], v[4 * j + 4]);
                f2unpack(vy, v[4 * j + 1], v[4 * j + 5]);
                f2unpack(vz, v[4 * j + 2], v[4 * j + 6]);
                f2unpack(mt, v[4 * j + 3], v[4 * j + 7]);
            }
        }
        const float z = warp_transpose_sum32(v, lane);
        scatter_adj8(adj_node, adj_leaf, lr, k0, count, (double)z, lane);
    }
    float a0, a1;
    f2unpack(sx, a0, a1); gx -= a0 + a1;
    f2unpack(sy, a0, a1); gy -= a0 + a1;
    f2unpack(sz, a0, a1); gz -= a0 + a1;
}

template <bool kDamp>
__device__ inline void adj_near_f32(const double4 *nc, const uint32_t *nm, const int *nr, int count, int lane,
                                    double bx, double by, double bz, float lax, float lay, float laz, float &gx,
                                    float &gy, float &gz, double *adj_node, double *adj_leaf) {
    for (int k0 = 0; k0 < count; k0 += 8) {
        float v[32];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k = k0 + j;
            float vx = 0.f, vy = 0.f, vz = 0.f, mt = 0.f;
            if (k < count && ((nm[k] >> lane) & 1u)) {
                const double4 c = nc[k];
                const float dx = (float)(c.x - bx), dy = (float)(c.y - by), dz = (float)(c.z - bz);
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                pair_adjoint<kDamp, float>(dx, dy, dz, r2, (float)c.w, lax, lay, laz, vx, vy, vz, mt);
            }
            gx -= vx; gy -= vy; gz -= vz;
            v[4 * j] = vx; v[4 * j + 1] = vy; v[4 * j + 2] = vz; v[4 * j + 3] = mt;
        }
        const float z = warp_transpose_sum32(v, lane);
        scatter_adj8(adj_node, adj_leaf, nr, k0, count, (double)z, lane);
    }
}

template <bool kDamp>
__device__ inline void adj_list_f64(const double4 *lc, const uint32_t *lm, const int *lr, int count, int lane,
                                    double bx, double by, double bz, double lax, double lay, double laz, double &gx,
                                    double &gy, double &gz, double *adj_node, double *adj_leaf) {
    for (int k0 = 0; k0 < count; k0 += 8) {
        double v[32];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k = k0 + j;
            double vx = 0.0, vy = 0.0, vz = 0.0, mt = 0.0;
            if (k < count && ((lm[k] >> lane) & 1u)) {
                const double4 c = lc[k];
                const double dx = c.x - bx, dy = c.y - by, dz = c.z - bz;
                const double r2 = dx * dx + dy * dy + dz * dz;
                pair_adjoint<kDamp, double>(dx, dy, dz, r2, c.w, lax, lay, laz, vx, vy, vz, mt);
            }
            gx -= vx; gy -= vy; gz -= vz;
            v[4 * j] = vx; v[4 * j + 1] = vy; v[4 * j + 2] = vz; v[4 * j + 3] = mt;
        }
        const double z = warp_transpose_sum32(v, lane);
        scatter_adj8(adj_node, adj_leaf, lr, k0, count, z, lane);
    }
}

// FP64 pair terms. Bound: the FP64 pipe and its dependent chains. A square root and a
// divide per pair (and per opening test of a mixed node) were most of the walk; the
// corrected inverse roots (fp64.cuh) and the test on squares take 16,384 particles from
// 227 to 147 us, 200,000 from 1750 to 1107, 60,001 damped (which keeps a divide and an
// exponential) from 890 to 790, the adjoint of 16,384 from 302 to 255 (139, 1092,
// 745 and 245 since the queue is taken in batches).
template <bool kDamp, bool kPot>
__device__ inline void force_list_f64(const double4 *lc, const uint32_t *lm, int count, int lane, double bx,
                                      double by, double bz, double &ax, double &ay, double &az, double &pot) {
#pragma unroll 2
    for (int k = 0; k < count; k++) {
        const bool take = (lm[k] >> lane) & 1u;
        const double4 c = lc[k];
        const double dx = c.x - bx, dy = c.y - by, dz = c.z - bz;
        const double r2 = dx * dx + dy * dy + dz * dz;
        double f, inv = 0.0;
        if constexpr (kDamp || kPot) inv = inverse_root(r2);
        if constexpr (kDamp) f = c.w * inv / (r2 + exp(-(r2 * inv)));
        else f = inverse_cube(r2, c.w);
        if (!plain_range(r2)) {  // the lane's own leaf (not taken), or an extreme distance
            const double d = sqrt(r2);
            inv = 1.0 / d;
            if constexpr (kDamp) f = c.w * inv / (r2 + exp(-d));
            else f = c.w * inv * inv * inv;
        }
        f = take ? f : 0.0;
        ax = fma(f, dx, ax); ay = fma(f, dy, ay); az = fma(f, dz, az);
        if constexpr (kPot) pot += take ? c.w * inv : 0.0;
    }
}

// Sums one batch (count <= 32 entries from ring position `start`, a multiple of 32)
// of list `list` on this lane's particle into v; cnt grows by the accepted bodies.
template <bool kFp64, bool kDamp, bool kPot, bool kAdj, int kList, class G, typename Acc, int NC>
__device__ inline void sum_batch(G &s, int start, int count, int lane, const WalkArgs &a, const double4 &b, float px,
                                 float py, float pz, float plx, float ply, float plz, double lax, double lay,
                                 double laz, Acc (&v)[NC], uint32_t &cnt) {
    const uint32_t bit = 1u << lane;
#pragma unroll
    for (int c = 0; c < NC; c++) v[c] = Acc(0);
    if constexpr (kFp64) {
        if constexpr (kAdj) {
            adj_list_f64<kDamp>(s.lc + start, s.lm + start, s.lr + start, count, lane, b.x, b.y, b.z, lax, lay, laz,
                                v[0], v[1], v[2], a.adj_node, a.adj_leaf);
        } else {
            double pot = 0.0;
            force_list_f64<kDamp, kPot>(s.lc + start, s.lm + start, count, lane, b.x, b.y, b.z, v[0], v[1], v[2], pot);
            if constexpr (NC > 3) v[3] = pot;
        }
        if (a.counts) cnt += count_list(s.lm + start, count, bit);
    } else if constexpr (kAdj) {
        if constexpr (kList == 0) {
            adj_list_f32<kDamp>(s.lp + 4 * start, s.lm + start, s.lr + start, count, lane, px, py, pz, (float)lax,
                                (float)lay, (float)laz, v[0], v[1], v[2], a.adj_node, a.adj_leaf);
            if (a.counts) cnt += count_list(s.lm + start, count, bit);
        } else {
            adj_near_f32<kDamp>(s.nc + start, s.nm + start, s.nr + start, count, lane, b.x, b.y, b.z, (float)lax,
                                (float)lay, (float)laz, v[0], v[1], v[2], a.adj_node, a.adj_leaf);
            if (a.counts) cnt += count_list(s.nm + start, count, bit);
        }
    } else {
        if constexpr (kList == 0) {
            force_pairs_f32<kDamp, false>(s.lf + 4 * start, nullptr, count, 0u, px, py, pz, v);
            cnt += count;
        } else if constexpr (kList == 1) {
            force_pairs_f32<kDamp, true>(s.lp + 4 * start, s.lm + start, count, bit, px, py, pz, v);
            if (a.counts) cnt += count_list(s.lm + start, count, bit);
        } else {
            force_pairs_f32<kDamp, true, true>(s.nhi + 4 * start, s.nm + start, count, bit, px, py, pz, v,
                                               s.nlo + 4 * start, plx, ply, plz);
            if (a.counts) cnt += count_list(s.nm + start, count, bit);
        }
    }
}

// The walk of one group of up to 32 particles, by one warp (kTeam false) or by the
// warps of a block together (kTeam true).
//
// Both do the same arithmetic in the same order. The entries still to be examined wait
// in a queue, which is taken in batches of a team's four tiles. Which entries come next
// (walk.cuh) is decided when a batch is done, and children queue up in the order of their
// parents, so the sequence in which entries are examined, and with it the sequence of
// every interaction list, does not depend on how many are examined at a time. Each list
// is summed in batches of 32 consecutive entries, the batches' sums are added in order,
// and the lists' sums last.
//
// Nodes, bodies and children are gathered, one 32-byte load each. Many groups keep the
// load pipe of the L1 and shared memory at 76% beside 69% of the issue slots (1M bodies,
// with two 16-byte loads each), so there a node's children are loaded once it is known
// that it is opened, as about one in three is: 981 to 946 us, and 931 with 32-byte loads;
// a collapsed system 3585 to 3470 and 3415 (945 and 3460 since the queue is taken in
// batches, which small opening angles need). The other forms wait for their loads instead
// (teams) or have too few warps an SM to cover a second one (FP64, adjoint) and take the
// children along with the node (20,011 bodies: 53 us, 56 with the later load; FP64 of
// 200,000: 1117, 1150; adjoint of 100,000: 629, 693).
//
// Bound of few groups: the serial chain of one group's tiles (~3 us each at one warp
// per scheduler; 11% of issue slots used on a shell of 20,011), which a team of four
// cuts to a third; of many: instruction issue (73% of slots), where one warp each
// needs no barriers. Teams of 2, 6 and 8 warps were slower (5000 particles: 79, 51,
// 55 us against 51 with four; 65,536: 291, 330, 446 against 258). A stack cut into
// parts for several warps, last in first out, was as fast for few groups, but one
// warp that has to repeat its order of sums for an ensemble took 12 to 30% longer.
template <bool kFp64, bool kDamp, bool kPot, bool kAdj, bool kStats, bool kTeam>
__global__ void __launch_bounds__((kTeam ? kTeamMaxWarps : kWalkMaxWarps) * 32) k_walk(WalkArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    griddep();
    // A walk ends, within its queue, on a well-formed octree only. Where the build has
    // reported that it is not (a sort that gave up, a node with too many children), the
    // pass stops here and the host reports the error.
    if (a.t.sc->status & (kStatusSortStall | kStatusCapacity)) return;
    using Acc = std::conditional_t<kFp64, double, float>;
    using Team = TeamSmem<kFp64, kAdj>;
    using Solo = SoloSmem<kFp64, kAdj>;
    constexpr int kLists = kFp64 ? 1 : kAdj ? 2 : 3;
    constexpr int NC = kPot ? 4 : 3;
    constexpr uint32_t kCap = kTeam ? kTeamList : kSoloList;
    constexpr bool kLate = !kTeam && !kFp64 && !kAdj;  // children loaded for opened nodes only
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Team &tm = *reinterpret_cast<Team *>(smem_raw);
    Solo &solo = reinterpret_cast<Solo *>(smem_raw)[kTeam ? 0 : wid];
    auto &s = [&]() -> auto & {
        if constexpr (kTeam) return tm.g;
        else return solo.g;
    }();
    auto &tile = [&]() -> auto & {
        if constexpr (kTeam) return tm.tile[wid];
        else return solo.tile;
    }();
    int2 *const queue = kTeam ? tm.queue : a.queue + (size_t)(blockIdx.x * (blockDim.x >> 5) + wid) * kQueueCap;
    const uint32_t w = kTeam ? wid : 0, W = kTeam ? blockDim.x >> 5 : 1;  // this warp within the team
    auto sync = [] {
        if constexpr (kTeam) __syncthreads();
        else __syncwarp();
    };
    const Tree &t = a.t;
    const uint32_t n = t.n;
    const bool single = a.single != 0;
    const float theta_f = __double2float_rn(a.theta);
    const double theta = single ? (double)theta_f : a.theta;
    // relative width of the FP64 form's group-level band: its own rounding, or
    // the FLOAT build's (~6.3 float ulps of (side/theta)^2)
    const double grp_rel = single ? 1e-6 : 1e-12;
    const double S1 = t.sc->root_side;
    const unsigned FULL = 0xffffffffu;
    const uint32_t lt = (1u << lane) - 1u;

    for (;;) {
        uint32_t g = 0;
        if constexpr (kTeam) {
            __syncthreads();  // the last group's shared memory is no longer read
            if (threadIdx.x == 0) tm.group = atomicAdd(&t.sc->group_counter, 1u);
            __syncthreads();
            g = tm.group;
        } else {
            if (lane == 0) g = atomicAdd(&t.sc->group_counter, 1u);
            g = __shfl_sync(FULL, g, 0);
        }
        if (g >= a.n_groups) break;

        uint32_t g0, gcount;
        int root = 0;
        double S = S1;
        if (a.groups) {
            const int4 gr = a.groups[g];
            g0 = (uint32_t)gr.x;
            gcount = (uint32_t)gr.y;
            root = a.sys_root_node[gr.z];
            S = a.sys_root[4 * (size_t)gr.z + 3];
        } else {
            g0 = g * 32;
            gcount = min(32u, n - g0);
            root = n >= 2 ? 0 : -1;
        }
        const double s_theta = S / theta;
        const uint32_t j = g0 + lane;
        const bool valid = (uint32_t)lane < gcount;
        const double4 b = t.body[valid ? j : g0];
        const uint32_t vmask = __ballot_sync(FULL, valid);
        // adjoint mode: this particle's cotangent dL/da
        double lax = 0.0, lay = 0.0, laz = 0.0;
        if constexpr (kAdj) {
            if (valid) {
                const size_t u3 = 3 * (size_t)t.sidx[j];
                if constexpr (kFp64) { lax = a.lamd[u3]; lay = a.lamd[u3 + 1]; laz = a.lamd[u3 + 2]; }
                else { lax = a.lamf[u3]; lay = a.lamf[u3 + 1]; laz = a.lamf[u3 + 2]; }
            }
        }

        // Reference point: centre of the group's bounding box.
        const double rx = 0.5 * (warp_min(b.x) + warp_max(b.x));
        const double ry = 0.5 * (warp_min(b.y) + warp_max(b.y));
        const double rz = 0.5 * (warp_min(b.z) + warp_max(b.z));
        const float px = (float)(b.x - rx), py = (float)(b.y - ry), pz = (float)(b.z - rz);
        // what the FP32 offsets left out (the forward near list adds it back)
        const float plx = lo_part(b.x - rx, px), ply = lo_part(b.y - ry, py), plz = lo_part(b.z - rz, pz);
        // Error band of the FP32 opening test. With u = 2^-24 and Pm the largest
        // |offset| from the reference point in the group, every lane has
        // |r2_f32 - r2| <= 7.1u r2 + 7u Pm sqrt(r2) and |q_f32 - q| <= 1.01u q;
        // outside |r2 - q| <= 32u q + 20u Pm sqrt(q), and for r2 > (64u Pm)^2,
        // the FP32 decision equals the exact one. Inside, the lane re-tests in FP64.
        const float pm_g = warp_maxf(fmaxf(fabsf(px), fmaxf(fabsf(py), fabsf(pz))));
        const float pm_tol = kTolPm * pm_g;
        const float tiny = (kTiny * pm_g) * (kTiny * pm_g);
        const float near_r2 = (pm_g * 0x1p-9f) * (pm_g * 0x1p-9f);
        // Group bounding box of the offsets (lanes past n repeat lane 0): FP32
        // for the MIXED form, FP64 for the FP64 form (group-level test only).
        float lox = 0.f, hix = 0.f, loy = 0.f, hiy = 0.f, loz = 0.f, hiz = 0.f;
        double dlox = 0.0, dhix = 0.0, dloy = 0.0, dhiy = 0.0, dloz = 0.0, dhiz = 0.0, dpm = 0.0;
        if constexpr (kFp64) {
            dlox = warp_min(b.x) - rx; dhix = warp_max(b.x) - rx;
            dloy = warp_min(b.y) - ry; dhiy = warp_max(b.y) - ry;
            dloz = warp_min(b.z) - rz; dhiz = warp_max(b.z) - rz;
            dpm = fmax(fmax(fmax(-dlox, dhix), fmax(-dloy, dhiy)), fmax(-dloz, dhiz));
        } else {
            lox = warp_minf(px); hix = warp_maxf(px);
            loy = warp_minf(py); hiy = warp_maxf(py);
            loz = warp_minf(pz); hiz = warp_maxf(pz);
        }

        if (w == 0) {
            if (lane == 0) {
                s.gc.ref[0] = rx; s.gc.ref[1] = ry; s.gc.ref[2] = rz;
                s.gc.S = S; s.gc.s_theta = s_theta;
                s.gc.box[0] = lox; s.gc.box[1] = hix; s.gc.box[2] = loy;
                s.gc.box[3] = hiy; s.gc.box[4] = loz; s.gc.box[5] = hiz;
                s.gc.pm_tol = pm_tol; s.gc.tiny = tiny; s.gc.near_r2 = near_r2;
                if constexpr (kStats)
                    for (int q = 0; q < 6; q++) s.gc.st[q] = 0u;
                queue[0] = make_int2(root, (int)vmask);
            }
#pragma unroll
            for (int l = 0; l < kLists; l++)
#pragma unroll
                for (int c = 0; c < NC; c++) s.acc[l][c][lane] = Acc(0);
            if constexpr (kTeam) tm.cnt[lane] = 0u;
        }
        uint32_t cnt = 0, nint = 0, nfallback = 0;
        uint32_t head = 0, qn = root >= 0 ? 1u : 0u;       // the queue: first entry, entries
        uint32_t lstart[3] = {0, 0, 0}, lcount[3] = {0, 0, 0};  // each list's ring: first entry, entries
        // One warp examines a batch tile by tile: the tiles still to come (they are at the
        // queue's front), and the tile's entries, which are loaded a tile early where the
        // queue (in global memory) holds them all already (else their masks are 0).
        uint32_t left = 0;
        int2 ahead = make_int2(0, 0);
        sync();

        while (qn > 0) {
            uint32_t base = head, take = 32;
            if (!kTeam && left > 0) {
                left--;
                head += 32;
            } else {
                const bool newest = qn > a.wide;
                take = min(qn, kQueueBatch);
                if (newest) {
                    const int room = ((int)(kQueueCap - kQueueReserve) - (int)qn) / 8;
                    take = (uint32_t)max(1, min(room, (int)kQueueBatch));
                }
                if (take > 32u) take &= ~31u;
                if (newest) base = head + qn - take;
                else head += kTeam ? take : min(take, 32u);
                if constexpr (!kTeam) {
                    left = (take - 1u) / 32u;
                    if (newest) {
                        // the other tiles move to the front, as children take their place
                        for (uint32_t q = 32u + lane; q < take; q += 32u)
                            queue[(head - take + q) & (kQueueCap - 1)] = queue[(base + q) & (kQueueCap - 1)];
                        head -= 32u * left;
                    }
                    take = min(take, 32u);
                    if (newest || ahead.y == 0) ahead = queue[(base + min((uint32_t)lane, take - 1u)) & (kQueueCap - 1)];
                    __syncwarp();  // all read before any lane writes there
                }
            }
            qn -= take;
            const int cntt = take > 32u * w ? (int)min(32u, take - 32u * w) : 0;
            if (kStats && lane == 0 && cntt > 0) {
                atomicAdd(&s.gc.st[0], (uint32_t)cntt);
                atomicAdd(&s.gc.st[1], 1u);
            }

            // ---- stage: lane k takes the tile's entry k
            bool is_int = false;
            int4 ch0 = make_int4(0, 0, 0, 0), ch1 = make_int4(0, 0, 0, 0);
            uint32_t reach = 0;
            int nch = 0, ref = 0;
            double cx = 0, cy = 0, cz = 0, m = 0, so = 0;
            if (lane < cntt) {
                const int2 e = kTeam ? queue[(base + 32u * w + lane) & (kQueueCap - 1)] : ahead;
                ref = e.x;
                reach = (uint32_t)e.y;
                if (ref >= 0) {
                    const double4 nd = load32(t.onode + ref);
                    const int meta = t.ometa[ref];
                    cx = nd.x; cy = nd.y; cz = nd.z; m = nd.w;
                    nch = meta_nchild(meta);
                    so = exp2_neg(meta_level(meta));  // 2^-level
                    if constexpr (!kLate) load32(t.ochild + 8 * (size_t)ref, ch0, ch1);
                    is_int = true;
                } else {
                    const double4 bd = load32(t.body + ~ref);
                    cx = bd.x; cy = bd.y; cz = bd.z; m = bd.w;
                    const uint32_t own = (uint32_t)(~ref) - g0;  // a leaf of this group: not its own lane
                    if (own < 32u) reach &= ~(1u << own);
                }
            }
            if constexpr (!kTeam) ahead = qn >= 32u ? queue[(head + lane) & (kQueueCap - 1)] : make_int2(0, 0);
            float fcx = 0.f, fcy = 0.f, fcz = 0.f;
            if constexpr (!kFp64) {
                fcx = (float)(cx - s.gc.ref[0]); fcy = (float)(cy - s.gc.ref[1]); fcz = (float)(cz - s.gc.ref[2]);
            }

            // ---- group-level test, one node per lane: when every point of the
            // group's box (widened by twice the FP32 error band) lies beyond the
            // opening radius side/theta, no lane opens the node; when every point
            // lies within it, every lane that reached it opens it. Only the
            // remaining nodes are decided lane by lane below.
            uint32_t my_open = 0;
            bool mixed = false;
            float r2box = 0.f;  // squared distance of the node from the group's box (MIXED form)
            double qd = 0.0;             // (side/theta)^2 (FP64 form)
            float qf = 0.f, band = 0.f;  // (side/theta)^2 in FP32 and the half-width of its error band
            if (is_int) {
                if constexpr (kFp64) {
                    const double sq = s.gc.S * so / theta;
                    qd = sq * sq;
                    const double ox = cx - s.gc.ref[0], oy = cy - s.gc.ref[1], oz = cz - s.gc.ref[2];
                    const double ax_ = fmax(fmax(dlox - ox, ox - dhix), 0.0), ay_ = fmax(fmax(dloy - oy, oy - dhiy), 0.0),
                                 az_ = fmax(fmax(dloz - oz, oz - dhiz), 0.0);
                    const double bx_ = fmax(fabs(ox - dlox), fabs(ox - dhix)), by_ = fmax(fabs(oy - dloy), fabs(oy - dhiy)),
                                 bz_ = fmax(fabs(oz - dloz), fabs(oz - dhiz));
                    const double r2min = ax_ * ax_ + ay_ * ay_ + az_ * az_;
                    const double r2max = bx_ * bx_ + by_ * by_ + bz_ * bz_;
                    const double tol = grp_rel * (qd + dpm * sq) + 1e-300;
                    if (r2min - qd > tol) my_open = 0;
                    else if (qd - r2max > tol) my_open = reach;
                    else mixed = true;
                } else {
                    const double sqd = s.gc.s_theta * so;
                    qf = (float)(sqd * sqd);
                    band = fmaf(s.gc.pm_tol, (float)sqd, kTolRel * qf);
                    const float tol = 2.f * band;
                    const float ax_ = fmaxf(fmaxf(s.gc.box[0] - fcx, fcx - s.gc.box[1]), 0.f), ay_ = fmaxf(fmaxf(s.gc.box[2] - fcy, fcy - s.gc.box[3]), 0.f),
                                az_ = fmaxf(fmaxf(s.gc.box[4] - fcz, fcz - s.gc.box[5]), 0.f);
                    const float bx_ = fmaxf(fabsf(fcx - s.gc.box[0]), fabsf(fcx - s.gc.box[1])), by_ = fmaxf(fabsf(fcy - s.gc.box[2]), fabsf(fcy - s.gc.box[3])),
                                bz_ = fmaxf(fabsf(fcz - s.gc.box[4]), fabsf(fcz - s.gc.box[5]));
                    const float r2min = fmaf(az_, az_, fmaf(ay_, ay_, ax_ * ax_));
                    const float r2max = fmaf(bz_, bz_, fmaf(by_, by_, bx_ * bx_));
                    r2box = r2min;
                    if (r2min <= 4.f * s.gc.tiny) mixed = true;
                    else if (r2min - qf > tol) my_open = 0;
                    else if (qf - r2max > tol) my_open = reach;
                    else mixed = true;
                }
            }

            // ---- decide the mixed nodes of the tile, lane by lane
            const uint32_t intm = __ballot_sync(FULL, mixed);
            if (kStats && lane == 0) atomicAdd(&s.gc.st[2], (uint32_t)__popc(intm));
            if (intm) {
                if constexpr (kFp64) {
                    tile.tc[lane] = make_double4(cx, cy, cz, s.gc.S * so);
                    tile.tq[lane] = qd;
                    tile.tr[lane] = reach;
                    __syncwarp();
                }
                if constexpr (kFp64) {
                    // The FP64 form compares squares, which settles all but distances within
                    // their rounding (the FLOAT build's: grp_rel) of the opening radius; those
                    // take the reference's own test, a square root and a divide.
                    uint32_t mm = intm;
                    while (mm) {
                        const int k = __ffs(mm) - 1;
                        mm &= mm - 1;
                        const double4 c = tile.tc[k];
                        const double q_k = tile.tq[k];
                        const uint32_t rk = tile.tr[k];
                        const double dx = c.x - b.x, dy = c.y - b.y, dz = c.z - b.z;
                        const double over = dx * dx + dy * dy + dz * dz - q_k;
                        bool open = over < 0.0;
                        if (!(fabs(over) > grp_rel * q_k))
                            open = ref_open(single, c.x, c.y, c.z, b.x, b.y, b.z, c.w, theta, theta_f);
                        const uint32_t om = __ballot_sync(FULL, open) & rk;
                        if (lane == k) my_open = om;
                    }
                } else {
                    // The mixed nodes, compacted into pairs, are decided two per round
                    // with packed FP32 arithmetic (the same roundings as the scalar
                    // expressions: dx = c.x + (-px), r2 = fma(dz, dz, fma(dy, dy, dx dx)),
                    // d = r2 + (-q)). Lane 0 stores each pair's open masks over the
                    // pair's first two words; each mixed lane then reads its own.
                    const int nmix = __popc(intm);
                    const int mpos = __popc(intm & lt);
                    if (mixed) {
                        float *e = tile.mx + kPair * (mpos >> 1) + (mpos & 1);
                        e[0] = fcx; e[2] = fcy; e[4] = fcz; e[6] = -qf;
                        e[8] = band; e[10] = __uint_as_float(reach); e[12] = __int_as_float(ref);
                    }
                    if (lane == 0 && (nmix & 1)) {
                        // pad an odd count with an entry no lane reached
                        float *e = tile.mx + kPair * (nmix >> 1) + 1;
                        e[0] = 0.f; e[2] = 0.f; e[4] = 0.f; e[6] = 0.f;
                        e[8] = 0.f; e[10] = 0.f; e[12] = 0.f;
                    }
                    __syncwarp();
                    const float tiny_ = s.gc.tiny;
                    const uint64_t npx = f2pack(-px, -px), npy = f2pack(-py, -py), npz = f2pack(-pz, -pz);
                    const uint32_t bit = 1u << lane;
                    for (int k = 0; k < nmix; k += 2) {
                        float *pr = tile.mx + (kPair / 2) * k;
                        const float4 A = *reinterpret_cast<const float4 *>(pr);      // x0 x1 y0 y1
                        const float4 B = *reinterpret_cast<const float4 *>(pr + 4);  // z0 z1 -q0 -q1
                        const float4 C = *reinterpret_cast<const float4 *>(pr + 8);  // band0 band1 reach0 reach1
                        const uint64_t dx = f2add(f2pack(A.x, A.y), npx);
                        const uint64_t dy = f2add(f2pack(A.z, A.w), npy);
                        const uint64_t dz = f2add(f2pack(B.x, B.y), npz);
                        const uint64_t r2 = f2fma(dz, dz, f2fma(dy, dy, f2mul(dx, dx)));
                        const uint64_t dd = f2add(r2, f2pack(B.z, B.w));
                        float r21, r22, d1, d2;
                        f2unpack(r2, r21, r22);
                        f2unpack(dd, d1, d2);
                        const uint32_t rk1 = __float_as_uint(C.z), rk2 = __float_as_uint(C.w);
                        bool open1 = d1 < 0.f, open2 = d2 < 0.f;
                        const bool amb1 = (rk1 & bit) && (fabsf(d1) <= C.x || r21 <= tiny_);
                        const bool amb2 = (rk2 & bit) && (fabsf(d2) <= C.y || r22 <= tiny_);
                        if (__any_sync(FULL, amb1 || amb2)) {
                            const float2 R = *reinterpret_cast<const float2 *>(pr + 12);  // ref0 ref1
                            if (amb1) {
                                const int node = __float_as_int(R.x);
                                const double4 nd = t.onode[node];
                                const double side = s.gc.S * exp2_neg(meta_level(t.ometa[node]));
                                open1 = ref_open(single, nd.x, nd.y, nd.z, b.x, b.y, b.z, side, theta, theta_f);
                                nfallback++;
                            }
                            if (amb2) {
                                const int node = __float_as_int(R.y);
                                const double4 nd = t.onode[node];
                                const double side = s.gc.S * exp2_neg(meta_level(t.ometa[node]));
                                open2 = ref_open(single, nd.x, nd.y, nd.z, b.x, b.y, b.z, side, theta, theta_f);
                                nfallback++;
                            }
                        }
                        const uint32_t om1 = __ballot_sync(FULL, open1) & rk1;
                        const uint32_t om2 = __ballot_sync(FULL, open2) & rk2;
                        // every lane has read the pair before the ballots complete
                        if (lane == 0) *reinterpret_cast<uint2 *>(pr) = make_uint2(om1, om2);
                    }
                    __syncwarp();
                    if (mixed) my_open = __float_as_uint(tile.mx[kPair * (mpos >> 1) + (mpos & 1)]);
                }
                __syncwarp();
            }

            // ---- accepted bodies -> interaction lists (compacted across lanes).
            // MIXED: a body closer to the group's box than 2^-9 of the group's
            // extent would lose too many bits in FP32 offsets (and could give a
            // zero r^2); it goes to the near list, whose offsets keep FP32 accuracy
            // of the offset itself.
            const uint32_t accm = reach & ~my_open;
            nint += __popc(accm);
            bool near = false;
            if constexpr (!kFp64) {
                if (accm) {
                    if (!is_int) {  // internal nodes have it from the group test
                        const float ax_ = fmaxf(fmaxf(s.gc.box[0] - fcx, fcx - s.gc.box[1]), 0.f),
                                    ay_ = fmaxf(fmaxf(s.gc.box[2] - fcy, fcy - s.gc.box[3]), 0.f),
                                    az_ = fmaxf(fmaxf(s.gc.box[4] - fcz, fcz - s.gc.box[5]), 0.f);
                        r2box = fmaf(az_, az_, fmaf(ay_, ay_, ax_ * ax_));
                    }
                    near = r2box < s.gc.near_r2;
                }
            }
            // entries every lane of the group takes go to a list without masks (MIXED forward)
            const bool take_it = accm != 0 && !near;
            const bool all = !kFp64 && !kAdj && take_it && accm == vmask;
            const uint32_t amk = !kFp64 && !kAdj ? __ballot_sync(FULL, all) : 0u;
            const uint32_t pmk = __ballot_sync(FULL, take_it && !all);
            const uint32_t nmk = !kFp64 ? __ballot_sync(FULL, near) : 0u;
            // exclusive prefix of the child counts (0..8) from four independent ballots of their bits
            const int myn = my_open ? nch : 0;
            if (kLate && myn > 0) load32(t.ochild + 8 * (size_t)ref, ch0, ch1);
            const uint32_t q0 = __ballot_sync(FULL, myn & 1), q1 = __ballot_sync(FULL, myn & 2),
                           q2 = __ballot_sync(FULL, myn & 4), q3 = __ballot_sync(FULL, myn & 8);
            const uint32_t pre = __popc(q0 & lt) + 2 * __popc(q1 & lt) + 4 * __popc(q2 & lt) + 8 * __popc(q3 & lt);
            uint32_t add_a = __popc(amk), add_p = __popc(pmk), add_n = __popc(nmk);
            uint32_t add_c = __popc(q0) + 2 * __popc(q1) + 4 * __popc(q2) + 8 * __popc(q3);
            if (kStats && lane == 0) {
                atomicAdd(&s.gc.st[3], add_a + add_p);
                atomicAdd(&s.gc.st[4], add_n);
            }
            // a team's warps append in the order of their tiles
            uint32_t off_a = 0, off_p = 0, off_n = 0, off_c = 0;
            if constexpr (kTeam) {
                if (lane == 0) *reinterpret_cast<uint4 *>(tm.add[w]) = make_uint4(add_a, add_p, add_n, add_c);
                __syncthreads();
                add_a = add_p = add_n = add_c = 0;
                for (uint32_t q = 0; q < W; q++) {
                    const uint4 u = *reinterpret_cast<const uint4 *>(tm.add[q]);
                    if (q == w) { off_a = add_a; off_p = add_p; off_n = add_n; off_c = add_c; }
                    add_a += u.x; add_p += u.y; add_n += u.z; add_c += u.w;
                }
            }
            auto slot_of = [&](int l, uint32_t off, uint32_t mk) -> int {
                const uint32_t q = lstart[l] + lcount[l] + off + __popc(mk & lt);
                return (int)(q >= kCap ? q - kCap : q);
            };
            if constexpr (kFp64) {
                if (take_it) {
                    const int pos = slot_of(0, off_p, pmk);
                    s.lc[pos] = make_double4(cx, cy, cz, kG * m);
                    s.lm[pos] = accm;
                    if constexpr (kAdj) s.lr[pos] = ref;
                }
                lcount[0] += add_p;
            } else if constexpr (kAdj) {
                if (take_it) {
                    const int pos = slot_of(0, off_p, pmk);
                    put_pair_entry(s.lp, pos, fcx, fcy, fcz, (float)(kG * m));
                    s.lm[pos] = accm;
                    s.lr[pos] = ref;
                } else if (near) {
                    const int pos = slot_of(1, off_n, nmk);
                    s.nc[pos] = make_double4(cx, cy, cz, kG * m);
                    s.nm[pos] = accm;
                    s.nr[pos] = ref;
                }
                lcount[0] += add_p;
                lcount[1] += add_n;
            } else {
                const float gmf = (float)(kG * m);
                if (all) {
                    put_pair_entry(s.lf, slot_of(0, off_a, amk), fcx, fcy, fcz, gmf);
                } else if (take_it) {
                    const int pos = slot_of(1, off_p, pmk);
                    put_pair_entry(s.lp, pos, fcx, fcy, fcz, gmf);
                    s.lm[pos] = accm;
                }
                if (nmk && near) {
                    const int pos = slot_of(2, off_n, nmk);
                    const double ox = cx - s.gc.ref[0], oy = cy - s.gc.ref[1], oz = cz - s.gc.ref[2];
                    put_pair_entry(s.nhi, pos, fcx, fcy, fcz, gmf);
                    put_pair_entry(s.nlo, pos, lo_part(ox, fcx), lo_part(oy, fcy), lo_part(oz, fcz), 0.f);
                    s.nm[pos] = accm;
                }
                lcount[0] += add_a;
                lcount[1] += add_p;
                lcount[2] += add_n;
            }

            // ---- children of opened nodes -> queue
            if (myn > 0) {
                const uint32_t at = head + qn + off_c + pre;
                const int om = (int)my_open;
                queue[at & (kQueueCap - 1)] = make_int2(ch0.x, om);
                if (myn > 1) queue[(at + 1) & (kQueueCap - 1)] = make_int2(ch0.y, om);
                if (myn > 2) queue[(at + 2) & (kQueueCap - 1)] = make_int2(ch0.z, om);
                if (myn > 3) queue[(at + 3) & (kQueueCap - 1)] = make_int2(ch0.w, om);
                if (myn > 4) queue[(at + 4) & (kQueueCap - 1)] = make_int2(ch1.x, om);
                if (myn > 5) queue[(at + 5) & (kQueueCap - 1)] = make_int2(ch1.y, om);
                if (myn > 6) queue[(at + 6) & (kQueueCap - 1)] = make_int2(ch1.z, om);
                if (myn > 7) queue[(at + 7) & (kQueueCap - 1)] = make_int2(ch1.w, om);
            }
            qn += add_c;
            if (kStats && lane == 0) atomicMax(&s.gc.st[5], qn);
            sync();

            // ---- the lists' full batches
            if constexpr (!kTeam) {
                Acc v[NC];
                auto solo_batch = [&](auto L) {
                    constexpr int l = decltype(L)::value;
                    if (lcount[l] < 32u) return;
                    sum_batch<kFp64, kDamp, kPot, kAdj, l>(s, (int)lstart[l], 32, lane, a, b, px, py, pz, plx, ply, plz,
                                                           lax, lay, laz, v, cnt);
#pragma unroll
                    for (int c = 0; c < NC; c++) s.acc[l][c][lane] += v[c];
                    lstart[l] = lstart[l] + 32u >= kCap ? lstart[l] + 32u - kCap : lstart[l] + 32u;
                    lcount[l] -= 32u;
                    __syncwarp();
                };
                solo_batch(std::integral_constant<int, 0>{});
                if constexpr (kLists > 1) solo_batch(std::integral_constant<int, 1>{});
                if constexpr (kLists > 2) solo_batch(std::integral_constant<int, 2>{});
            } else {
                uint32_t nb = 0;
#pragma unroll
                for (int l = 0; l < kLists; l++) nb += lcount[l] >> 5;
                if (nb > 0) {
                    // batch q of the round (list by list) goes to warp q mod W
                    uint32_t q0_ = 0;
                    auto team_batches = [&](auto L) {
                        constexpr int l = decltype(L)::value;
                        const uint32_t k = lcount[l] >> 5;
                        for (uint32_t i = (w + W - q0_ % W) % W; i < k; i += W) {
                            const uint32_t q = lstart[l] + 32u * i;
                            Acc v[NC];
                            sum_batch<kFp64, kDamp, kPot, kAdj, l>(s, (int)(q >= kCap ? q - kCap : q), 32, lane, a, b, px,
                                                                   py, pz, plx, ply, plz, lax, lay, laz, v, cnt);
#pragma unroll
                            for (int c = 0; c < NC; c++) tm.slot[q0_ + i][c][lane] = v[c];
                        }
                        q0_ += k;
                    };
                    team_batches(std::integral_constant<int, 0>{});
                    if constexpr (kLists > 1) team_batches(std::integral_constant<int, 1>{});
                    if constexpr (kLists > 2) team_batches(std::integral_constant<int, 2>{});
                    __syncthreads();
                    q0_ = 0;
#pragma unroll
                    for (int l = 0; l < kLists; l++) {
                        const uint32_t k = lcount[l] >> 5;
                        if ((uint32_t)l % W == w) {
                            for (uint32_t i = 0; i < k; i++)
#pragma unroll
                                for (int c = 0; c < NC; c++) s.acc[l][c][lane] += tm.slot[q0_ + i][c][lane];
                        }
                        q0_ += k;
                        lstart[l] += 32u * k;
                        if (lstart[l] >= kCap) lstart[l] -= kCap;
                        lcount[l] &= 31u;
                    }
                }
            }
        }

        // ---- what is left in the lists
        {
            Acc v[NC];
            auto rest = [&](auto L) {
                constexpr int l = decltype(L)::value;
                if (lcount[l] == 0u || (kTeam && (uint32_t)l % W != w)) return;
                sum_batch<kFp64, kDamp, kPot, kAdj, l>(s, (int)lstart[l], (int)lcount[l], lane, a, b, px, py, pz, plx, ply,
                                                       plz, lax, lay, laz, v, cnt);
#pragma unroll
                for (int c = 0; c < NC; c++) s.acc[l][c][lane] += v[c];
            };
            rest(std::integral_constant<int, 0>{});
            if constexpr (kLists > 1) rest(std::integral_constant<int, 1>{});
            if constexpr (kLists > 2) rest(std::integral_constant<int, 2>{});
        }
        if constexpr (kTeam) {
            if (a.counts) atomicAdd(&tm.cnt[lane], cnt);
            __syncthreads();
            cnt = tm.cnt[lane];
        }

        // ---- epilogue: results in the caller's particle order
        double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll
        for (int l = 0; l < kLists; l++) {
            ax += (double)s.acc[l][0][lane];
            ay += (double)s.acc[l][1][lane];
            az += (double)s.acc[l][2][lane];
        }
        const float fax = (float)ax, fay = (float)ay, faz = (float)az;
        if constexpr (!kFp64) { ax = fax; ay = fay; az = faz; }
        if (valid && w == 0) {
            const uint32_t ui = t.sidx[j];
            if constexpr (kAdj) {
                if constexpr (kFp64) {
                    a.gdird[3 * (size_t)ui] = ax; a.gdird[3 * (size_t)ui + 1] = ay; a.gdird[3 * (size_t)ui + 2] = az;
                } else {
                    a.gdirf[3 * (size_t)ui] = fax; a.gdirf[3 * (size_t)ui + 1] = fay; a.gdirf[3 * (size_t)ui + 2] = faz;
                }
            } else if constexpr (kFp64) {
                a.accd[3 * (size_t)ui] = ax; a.accd[3 * (size_t)ui + 1] = ay; a.accd[3 * (size_t)ui + 2] = az;
            } else {
                a.accf[3 * (size_t)ui] = fax; a.accf[3 * (size_t)ui + 1] = fay; a.accf[3 * (size_t)ui + 2] = faz;
            }
            if (a.counts) a.counts[ui] = cnt;
            if constexpr (kPot) {
                if (a.pot) a.pot[ui] = -s.acc[0][3][lane];
            }
        }
        unsigned long long wc = nint;
        for (int o = 16; o; o >>= 1) wc += __shfl_xor_sync(FULL, wc, o);
        uint32_t wf = nfallback;
        for (int o = 16; o; o >>= 1) wf += __shfl_xor_sync(FULL, wf, o);
        double amag = valid ? sqrt(ax * ax + ay * ay + az * az) : 0.0;
        if (!kAdj && a.track_max_acc) amag = warp_max(amag);
        if (lane == 0) {
            atomicAdd(&t.sc->interactions, wc);
            atomicAdd(&t.sc->interactions_total, wc);
            if (wf) atomicAdd(&t.sc->fallback_tests, wf);
            if (w == 0) {
                if constexpr (kStats) {
                    atomicAdd(&t.sc->walk_entries, (unsigned long long)s.gc.st[0]);
                    atomicAdd(&t.sc->walk_tiles, (unsigned long long)s.gc.st[1]);
                    atomicAdd(&t.sc->walk_decisions, (unsigned long long)s.gc.st[2]);
                    atomicAdd(&t.sc->walk_list, (unsigned long long)s.gc.st[3]);
                    if (s.gc.st[4]) atomicAdd(&t.sc->walk_near, (unsigned long long)s.gc.st[4]);
                    atomicMax(&t.sc->max_stack, s.gc.st[5]);
                }
                if (!kAdj && a.track_max_acc) atomic_max_nonneg(&t.sc->max_acc_bits, amag);
            }
        }
        if constexpr (!kTeam) __syncwarp();
    }
}

// Potentials (diagnostics) are summed by the FP64 form only. The walk's
// statistics (entries, tiles, decisions, list and near entries, longest queue)
// are collected by their own instances of the forward kernel (kStats), so that
// the others carry none of that bookkeeping; the adjoint collects none.
template <bool kFp64, bool kStats, bool kTeam>
const void *forward_kernel(int damping, bool pot) {
    if constexpr (!kFp64) {
        (void)pot;
        return damping ? (const void *)k_walk<false, true, false, false, kStats, kTeam>
                       : (const void *)k_walk<false, false, false, false, kStats, kTeam>;
    } else {
        if (damping)
            return pot ? (const void *)k_walk<true, true, true, false, kStats, kTeam>
                       : (const void *)k_walk<true, true, false, false, kStats, kTeam>;
        return pot ? (const void *)k_walk<true, false, true, false, kStats, kTeam>
                   : (const void *)k_walk<true, false, false, false, kStats, kTeam>;
    }
}

template <bool kTeam>
const void *walk_kernel(bool fp64, bool adj, int damping, bool pot, bool stats) {
    if (adj) {
        if (fp64)
            return damping ? (const void *)k_walk<true, true, false, true, false, kTeam>
                           : (const void *)k_walk<true, false, false, true, false, kTeam>;
        return damping ? (const void *)k_walk<false, true, false, true, false, kTeam>
                       : (const void *)k_walk<false, false, false, true, false, kTeam>;
    }
    if (fp64) return stats ? forward_kernel<true, true, kTeam>(damping, pot) : forward_kernel<true, false, kTeam>(damping, pot);
    return stats ? forward_kernel<false, true, kTeam>(damping, pot) : forward_kernel<false, false, kTeam>(damping, pot);
}

const void *any_walk_kernel(bool team, bool fp64, bool adj, int damping, bool pot, bool stats) {
    return team ? walk_kernel<true>(fp64, adj, damping, pot, stats) : walk_kernel<false>(fp64, adj, damping, pot, stats);
}

// No instance needs more dynamic shared memory than a launch gets without asking.
constexpr size_t kPlainSmem = 48 << 10;
static_assert(sizeof(SoloSmem<true, true>) * kWalkMaxWarps <= kPlainSmem && sizeof(SoloSmem<true, false>) * kWalkMaxWarps <= kPlainSmem &&
                  sizeof(SoloSmem<false, true>) * kWalkMaxWarps <= kPlainSmem && sizeof(SoloSmem<false, false>) * kWalkMaxWarps <= kPlainSmem &&
                  sizeof(TeamSmem<true, true>) <= kPlainSmem && sizeof(TeamSmem<true, false>) <= kPlainSmem &&
                  sizeof(TeamSmem<false, true>) <= kPlainSmem && sizeof(TeamSmem<false, false>) <= kPlainSmem,
              "larger ones need cudaFuncAttributeMaxDynamicSharedMemorySize");

size_t solo_smem(bool fp64, bool adj) {
    if (fp64) return adj ? sizeof(SoloSmem<true, true>) : sizeof(SoloSmem<true, false>);
    return adj ? sizeof(SoloSmem<false, true>) : sizeof(SoloSmem<false, false>);
}
size_t team_smem(bool fp64, bool adj) {
    if (fp64) return adj ? sizeof(TeamSmem<true, true>) : sizeof(TeamSmem<true, false>);
    return adj ? sizeof(TeamSmem<false, true>) : sizeof(TeamSmem<false, false>);
}

cudaError_t launch(const void *k, const WalkArgs &a, unsigned blocks, unsigned warps, size_t smem, cudaStream_t st) {
    WalkArgs args = a;
    void *params[] = {&args};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, k, params);
}

}  // namespace

// The grid is sized by the forward walk's instances. The adjoint's FP64 ones take
// more registers: fewer of their blocks are resident, and the rest start as those
// end and find the work counter drained (groups wait for nothing). Sizing every
// launch by the largest instance kept the FP64 forward walk at 3 resident blocks of
// the 5 that fit: 1.295 -> 1.161 ms (sphere of 60,001, damped).
cudaError_t walk_max_blocks_per_sm(bool fp64, unsigned warps, int *out) {
    int minblocks = 1 << 30;
    for (int q = 0; q < 8; q++) {
        const bool damp = q & 1, pot = q & 2, stats = q & 4;
        if (pot && !fp64) continue;
        int nb = 0;
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &nb, any_walk_kernel(false, fp64, false, damp, pot, stats), (int)warps * 32, solo_smem(fp64, false) * warps);
        if (e != cudaSuccess) return e;
        minblocks = nb < minblocks ? nb : minblocks;
    }
    *out = minblocks;
    return cudaSuccess;
}

cudaError_t walk_launch_shape(bool fp64, int device, unsigned warps, unsigned blocks_per_sm, WalkLaunch *out) {
    int maxb = 0;
    cudaError_t e = walk_max_blocks_per_sm(fp64, warps, &maxb);
    if (e != cudaSuccess) return e;
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    if (maxb < 1) maxb = 1;
    const int per_sm = blocks_per_sm ? (int)blocks_per_sm < maxb ? (int)blocks_per_sm : maxb : maxb;
    out->blocks = (unsigned)(sms * per_sm);
    out->warps = warps;
    out->sms = (unsigned)sms;
    return cudaSuccess;
}

bool walk_by_teams(bool fp64, bool adjoint, double theta, uint32_t n, uint32_t n_groups, uint32_t systems,
                   const WalkLaunch &l) {
    return n_groups <= team_groups_per_sm(fp64, adjoint, theta) * l.sms && n >= kTeamMinSize * systems;
}

// One block per group, as many as fit; the rest take the groups left.
unsigned team_blocks(uint32_t n_groups, const WalkLaunch &l) { return std::min(n_groups, kTeamBlocksPerSm * l.sms); }

cudaError_t launch_walk(const WalkArgs &a, bool fp64, const WalkLaunch &l, cudaStream_t st) {
    const bool adj = a.adjoint != 0;
    const bool team = walk_by_teams(fp64, adj, a.theta, a.t.n, a.n_groups, a.systems, l);
    const void *k = any_walk_kernel(team, fp64, adj, a.damping, a.pot != nullptr, a.stats != 0);
    if (team) return launch(k, a, team_blocks(a.n_groups, l), kTeamMaxWarps, team_smem(fp64, adj), st);
    const unsigned need = (a.n_groups + l.warps - 1) / l.warps;
    return launch(k, a, need < l.blocks ? need : l.blocks, l.warps, solo_smem(fp64, adj) * l.warps, st);
}

}  // namespace nbody
