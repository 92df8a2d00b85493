// Fused tree walk + gravity (walk.cu).
#pragma once

#include "common.cuh"

namespace nbody {

constexpr int kWalkWarps = 4;       // default warps per block (the autotuner may pick 1 or 2)
constexpr int kWalkMaxWarps = 4;    // largest block the walk kernel is compiled for
constexpr int kTeamMaxWarps = 4;    // warps of a block that walk one group together
// Queue of the nodes a walk has still to examine (per warp in global memory, per team
// in shared memory), taken in batches of kQueueBatch: a team's turn. While no more than
// queue_wide(theta) wait, the oldest go first; beyond, the newest, in batches that get
// smaller until a depth-first descent of one entry at a time (at most 7 more entries per
// level) fits in the reserve.
//
// Oldest first keeps tiles full and reads nodes level by level; newest first bounds the
// queue. A small opening angle opens so many nodes that the queue is at its limit for most
// of the walk, and a low one leaves room for whole batches (MIXED cube / sphere of 20,000,
// us: theta 0.1 limit 256: 868 / 789, 640: 1356 / 1108; 0.3: 195 / 205 and 231 / 268;
// 0.5: 82 / 90 both). At ordinary angles few walks pass 640 (collapsed system of 1,048,576:
// 3530 with 256, 3468 with 640). One tile at a time past 1280 left a team's other warps
// idle and made tiles narrow: 40,000 at theta 0.05 8.9 ms, at 0.3 0.75, now 3.7 and 0.41.
constexpr uint32_t kQueueCap = 2048;
constexpr uint32_t kQueueWide = 640, kQueueWideSmallTheta = 256;
constexpr uint32_t queue_wide(double theta) { return theta < 0.45 ? kQueueWideSmallTheta : kQueueWide; }
constexpr uint32_t kQueueBatch = 32 * kTeamMaxWarps;
constexpr uint32_t kQueueReserve = 7 * (kMaxLevels + 1) + 8;
static_assert((kQueueCap & (kQueueCap - 1)) == 0, "ring index");
static_assert(kQueueWide + 7 * kQueueBatch <= kQueueCap - kQueueReserve, "a batch's pushes fit before batches get smaller");
static_assert(kQueueWideSmallTheta >= kQueueBatch && kQueueWide >= kQueueBatch, "past the limit there is a whole batch");
static_assert(kQueueBatch <= kQueueReserve, "room for a batch moved to the front");
// Interaction lists: less than a batch of 32 left over, and what a tile (a team's tiles) adds.
constexpr int kSoloList = 64;
constexpr int kTeamList = 32 + 32 * kTeamMaxWarps;
// Teams walk while there are at most this many groups per SM. Fewer groups leave
// walk warps idle, and time is the chain of one group's tiles; with more, barriers
// cost more than the last wave of single warps. Where that is depends on the state: a
// shell's short lists suit single warps sooner than a sphere's long ones. Walk times,
// teams against single warps (us):
//   MIXED: 5000 particles 51 / 98, shell of 20,011 53 / 82; 40,000: shell 90 / 100,
//   sphere 168 / 203; 48,000: shell 113 / 100, cube 162 / 186, sphere 188 / 215,
//   collapsed 244 / 268; 56,000: 127 / 104, 190 / 195, 219 / 225, 274 / 266. Below a
//   theta of 0.25 the teams' second wave costs more, at 0.1: 25,000 cube 1165 / 1540,
//   sphere 1231 / 1619; 35,000: 2019 / 1955, 1942 / 2060; 40,000: 2412 / 2186, 2237 / 2293.
//   Its adjoint: 5000 94 / 172; spheres of 60,000 381 / 414, 72,000 455 / 461, 85,000
//   532 / 524, 100,000 606 / 582.
//   FP64: 5000 94 / 225, 16,384 139 / 315, 60,001 (damped) 743 / 920; 85,000: sphere
//   532 / 567, shell 293 / 242; 112,000: sphere 657 / 707, collapsed 858 / 836, shell
//   375 / 326; 150,000: sphere 870 / 881.
//   Its adjoint: 16,384 242 / 547, 100,000 1196 / 1380, 113,000 1346 / 1448.
// Systems of fewer than kTeamMinSize particles have a few short tiles per group, for
// which the barriers cost more (a step of 97: 133 us with teams, 125 without; 150:
// the same; 300: 147 and 151).
constexpr uint32_t kTeamMinSize = 160;
constexpr unsigned team_groups_per_sm(bool fp64, bool adjoint, double theta) {
    return fp64 ? 24 : adjoint ? 16 : theta < 0.25 ? 7 : 10;
}
// Blocks per SM of a team grid: as many as are resident (at most 96 registers, 36 KB of
// shared memory). The FP64 adjoint's take 128 and 168 registers: three or four are
// resident, and the others start as those end and find the groups drained.
constexpr unsigned kTeamBlocksPerSm = 5;

struct WalkArgs {
    Tree t;
    double theta;
    int damping;
    // The reference's FLOAT build: node values are floats and the opening test
    // is its float expression (float theta, float side / float distance).
    int single;
    float *accf;        // MIXED: user order, 3 floats per particle
    double *accd;       // FP64: user order, 3 doubles per particle
    uint32_t *counts;   // optional: accepted nodes per particle (user order)
    double *pot;        // optional: potential phi_i per particle (user order)
    int2 *queue;        // kQueueCap entries per warp of the grid (walks by one warp)
    uint32_t wide;      // queue_wide(theta)
    uint32_t n_groups;  // ceil(n / 32)
    uint32_t systems;   // independent systems (1: a single one)
    int track_max_acc;  // reduce max |a| (adaptive dt)
    int stats;          // collect the walk statistics (DevScalars walk_* and max_stack)
    // Adjoint mode (frozen decisions): the walk computes, for the cotangent
    // lam (dL/da per particle, user order), the direct term
    // gdir_i = -sum_n K_in lam_i and the node sums adj[n] = (sum_i K_in lam_i,
    // sum_i G g_in (d_in . lam_i)), internal nodes in adj_node, leaves (by
    // sorted index) in adj_leaf. K = dF/d(com) of the pair force.
    int adjoint;
    const float *lamf;  // MIXED
    const double *lamd; // FP64
    float *gdirf;       // MIXED: user order, 3 per particle
    double *gdird;      // FP64
    double *adj_node;   // 4 doubles per internal node
    double *adj_leaf;   // 4 doubles per sorted particle
    // Several independent systems: the work queue is a table of groups
    // (first sorted particle, count <= 32, system); each system has its own
    // octree root and root side. Null for a single system (groups of 32 from 0).
    const int4 *groups;
    const int32_t *sys_root_node;
    const double *sys_root;     // 4 per system: center xyz, side
};

// Launch shape of the persistent walk: `warps` per block, `blocks` in the grid
// (a whole number of resident blocks per SM) of `sms` SMs.
struct WalkLaunch {
    unsigned blocks;
    unsigned warps;
    unsigned sms;
};
// blocks_per_sm = 0: as many as fit. Returns the shape for that block size.
cudaError_t walk_launch_shape(bool fp64, int device, unsigned warps, unsigned blocks_per_sm, WalkLaunch *out);
// Resident blocks per SM that fit for `warps` per block (all forward instances).
cudaError_t walk_max_blocks_per_sm(bool fp64, unsigned warps, int *out);
// Whether teams walk n particles in n_groups groups, and their grid (blocks of kTeamMaxWarps).
bool walk_by_teams(bool fp64, bool adjoint, double theta, uint32_t n, uint32_t n_groups, uint32_t systems,
                   const WalkLaunch &l);
unsigned team_blocks(uint32_t n_groups, const WalkLaunch &l);
cudaError_t launch_walk(const WalkArgs &a, bool fp64, const WalkLaunch &l, cudaStream_t st);

}  // namespace nbody
