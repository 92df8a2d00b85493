// LSD radix sort of (u64 key, u32 index) pairs, one kernel per 8-bit pass.
//
// The global digit counts of every pass do not depend on the order of the
// keys, so they are taken for all passes where the keys are made. Each pass then
// is a single kernel: a block takes the next tile (4096 keys) in ticket order,
// ranks its keys stably (per warp, 16 rounds of 32 keys; the lanes that share
// a digit are found with eight ballots, one per digit bit),
// publishes its per-digit count, adds the counts of all earlier tiles by
// decoupled look-back (a tile only ever waits for tiles that started before
// it, so the wait always ends; it is still bounded, and a timeout is reported
// as an error), and scatters: the tile is first laid out in digit order in
// shared memory, so that each digit's run goes out in coalesced writes.
#include "sort.cuh"
#include "keys.cuh"

namespace nbody {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 16;
static_assert(kThreads * kItems == kSortTile, "a tile is one load of the block");
constexpr uint32_t kFlagAgg = 1u << 30, kFlagInc = 2u << 30, kValue = (1u << 30) - 1;
constexpr uint32_t kSpinLimit = 1u << 20;

// Digit counts of the 8 passes of w into slots slot...
__global__ void k_hist(const uint64_t *__restrict__ w, int slot, uint32_t n, uint32_t *__restrict__ ghist) {
    griddep();
    __shared__ uint32_t s_h[8 * 256];
    for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) s_h[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t a = w[i];
        for (int k = 0; k < 8; k++) atomicAdd(&s_h[k * 256 + ((a >> (8 * k)) & 255u)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x)
        if (s_h[i]) atomicAdd(&ghist[slot * 256 + i], s_h[i]);
}

// Zeroes `words` 32-bit words (16-byte aligned), four per thread and step.
__global__ void k_zero_words(uint32_t *__restrict__ p, size_t words) {
    griddep();
    const size_t q = words / 4, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < q; i += stride)
        reinterpret_cast<uint4 *>(p)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (size_t i = 4 * q + blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) p[i] = 0u;
}

struct SweepSmem {
    uint32_t wc[kWarps][256];  // per-warp digit counts, then per-warp offsets
    uint32_t base[256];        // global position of the tile's first key of each digit
    uint32_t lstart[256];      // position of each digit's first key within the tile
    uint32_t wsum[2][kWarps];
    uint64_t buf[kSortTile];   // the tile in digit order: keys, then indices
};

// One tile of one pass. kShared: the inputs were written by other blocks of this
// launch (read past L1).
template <bool kShared>
__device__ inline void sweep_tile(SweepSmem &s, uint32_t tile, const uint64_t *kin, const uint32_t *iin, uint64_t *kout,
                                  uint32_t *iout, uint32_t n, int shift, const uint32_t *hist, uint32_t *status,
                                  uint32_t *err, uint32_t err_bit) {
    auto &s_wc = s.wc;
    auto &s_base = s.base;
    auto &s_lstart = s.lstart;
    auto &s_buf = s.buf;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const uint32_t in_all = kShared ? __ldcg(&hist[t]) : hist[t];  // keys with digit t, over all tiles
    for (int k = 0; k < kWarps; k++) s_wc[k][t] = 0;
    __syncthreads();
    const uint32_t base = tile * kSortTile + (uint32_t)w * (32 * kItems);
    const uint32_t lt = (1u << lane) - 1u;
    uint64_t key[kItems];
    uint32_t idx[kItems], rank[kItems];
    // ---- load, then rank: warp w owns keys [base, base + 512) in order
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const uint32_t i = base + r * 32 + lane;
        const bool valid = i < n;
        key[r] = valid ? (kShared ? __ldcg(&kin[i]) : __ldcs(&kin[i])) : 0ull;
        idx[r] = valid ? (kShared ? __ldcg(&iin[i]) : __ldcs(&iin[i])) : 0u;
    }
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const uint32_t i = base + r * 32 + lane;
        const bool valid = i < n;
        const uint32_t d = (uint32_t)((key[r] >> shift) & 255u);
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const uint32_t bb = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= ((d >> b) & 1u) ? bb : ~bb;
        }
        if (!valid) peers = 1u << lane;
        const uint32_t before = valid ? s_wc[w][d] : 0u;
        rank[r] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (peers & lt) == 0) s_wc[w][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // ---- per digit (thread t = digit): offsets of each warp, tile total
    uint32_t total = 0;
#pragma unroll
    for (int k = 0; k < kWarps; k++) {
        const uint32_t c = s_wc[k][t];
        s_wc[k][t] = total;
        total += c;
    }
    // ---- exclusive scans over the digits: start within the tile, start of the digit
    // in the whole output (every block scans the 256 counts itself: a launch less per
    // sort than one scan kernel, and the counts are in L2)
    uint32_t first = 0;
    {
        uint32_t x = total, y = in_all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t p = __shfl_up_sync(0xffffffffu, x, o), q = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) {
                x += p;
                y += q;
            }
        }
        if (lane == 31) {
            s.wsum[0][w] = x;
            s.wsum[1][w] = y;
        }
        __syncthreads();
        uint32_t off = 0;
        for (int k = 0; k < w; k++) {
            off += s.wsum[0][k];
            first += s.wsum[1][k];
        }
        s_lstart[t] = off + x - total;
        first += y - in_all;
    }
    // ---- decoupled look-back over earlier tiles
    uint32_t *st = status + (size_t)tile * 256 + t;
    uint32_t excl = 0;
    if (tile == 0) {
        atomicExch(st, kFlagInc | total);
    } else {
        atomicExch(st, kFlagAgg | total);
        // read up to 8 predecessors per round trip, newest first
        const volatile uint32_t *vs = status;
        int64_t p = (int64_t)tile - 1;
        uint32_t spins = 0;
        bool done = false;
        while (!done) {
            uint32_t v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = p - k >= 0 ? vs[(size_t)(p - k) * 256 + t] : kFlagInc;
            int used = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (done || used < k) continue;  // stop at the first entry not yet published
                const uint32_t flag = v[k] & ~kValue;
                if (flag == 0u) continue;
                excl += v[k] & kValue;
                used = k + 1;
                if (flag == kFlagInc) done = true;
            }
            p -= used;
            if (!done && used == 0 && ++spins > kSpinLimit) {
                atomicOr(err, err_bit);
                break;
            }
        }
        __threadfence();
        atomicExch(st, kFlagInc | (excl + total));
    }
    s_base[t] = first + excl;
    __syncthreads();
    // ---- scatter through shared memory: the tile is laid out in digit order,
    // then consecutive threads write consecutive positions of each digit's run
    const uint32_t tcount = min(kSortTile, n - tile * kSortTile);
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const uint32_t i = base + r * 32 + lane;
        if (i < n) {
            const uint32_t d = (uint32_t)((key[r] >> shift) & 255u);
            s_buf[s_lstart[d] + s_wc[w][d] + rank[r]] = key[r];
        }
    }
    __syncthreads();
    uint32_t dslot[kItems];
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const uint32_t q = (uint32_t)t + r * kThreads;
        dslot[r] = 0;
        if (q < tcount) {
            const uint64_t k = s_buf[q];
            const uint32_t d = (uint32_t)((k >> shift) & 255u);
            dslot[r] = d;
            kout[s_base[d] + (q - s_lstart[d])] = k;
        }
    }
    __syncthreads();
    uint32_t *s_idx = reinterpret_cast<uint32_t *>(s_buf);
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const uint32_t i = base + r * 32 + lane;
        if (i < n) {
            const uint32_t d = (uint32_t)((key[r] >> shift) & 255u);
            s_idx[s_lstart[d] + s_wc[w][d] + rank[r]] = idx[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kItems; r++) {
        const uint32_t q = (uint32_t)t + r * kThreads;
        if (q < tcount) iout[s_base[dslot[r]] + (q - s_lstart[dslot[r]])] = s_idx[q];
    }
}

__global__ void __launch_bounds__(kThreads) k_onesweep(const uint64_t *__restrict__ kin,
                                                       const uint32_t *__restrict__ iin, uint64_t *__restrict__ kout,
                                                       uint32_t *__restrict__ iout, uint32_t n, int shift,
                                                       const uint32_t *__restrict__ hist, uint32_t *status,
                                                       uint32_t *ticket, uint32_t *err, uint32_t err_bit) {
    griddep();
    __shared__ SweepSmem s;
    __shared__ uint32_t s_tile;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    sweep_tile<false>(s, s_tile, kin, iin, kout, iout, n, shift, hist, status, err, err_bit);
}

// The second key word of particle i.
__device__ inline uint64_t second_word(const FullSort &f, uint32_t i) {
    double root[4] = {f.sc->root_center[0], f.sc->root_center[1], f.sc->root_center[2], f.sc->root_side};
    if (f.sys_id) {
        const double *r = f.sys_root + 4 * (size_t)f.sys_id[i];
        root[0] = r[0]; root[1] = r[1]; root[2] = r[2]; root[3] = r[3];
    }
    const double p[3] = {f.pos[3 * (size_t)i], f.pos[3 * (size_t)i + 1], f.pos[3 * (size_t)i + 2]};
    uint64_t w[2];
    if (f.single) descend_words<float>(p, root, 2, w);
    else descend_words<double>(p, root, 2, w);
    return w[1];
}

// The full sort in one launch. Work items are (phase, tile), taken in order from one
// counter; an item first waits until every tile of the phase before has finished.
// Those were taken earlier, by blocks already running, so the wait always ends (it is
// still bounded). As 22 launches (16 passes and what lies between) that returned at once
// when the sort was not needed, it cost 40 us of a force pass outside a captured graph
// (60,001 particles: 1034 -> 999 us a call), and a conditional node inside one.
__global__ void __launch_bounds__(kThreads) k_full_sort(FullSort f) {
    griddep();
    __shared__ SweepSmem s;
    __shared__ uint32_t s_item, s_stop;
    if (f.run_if && *f.run_if == 0u) return;
    const uint32_t tiles = (f.n + kSortTile - 1) / kSortTile;
    const bool multi = f.sys_id != nullptr;
    const uint32_t phases = multi ? 22 : 19;
    uint32_t *hist = f.scratch + 256 * kFullSlot;
    uint32_t *item = f.scratch + kSortCounters + kFullCounters, *done = item + 1;
    uint32_t *status0 = f.scratch + kSortStatus + (size_t)kFullSlot * tiles * 256;
    const int t = threadIdx.x;
    for (;;) {
        if (t == 0) {
            s_stop = 0u;
            s_item = atomicAdd(item, 1u);
            const uint32_t ph = s_item / tiles;
            if (ph > 0 && ph < phases) {
                const volatile uint32_t *d = done + (ph - 1);
                uint32_t spins = 0;
                while (*d < tiles) {
                    if (++spins > kSpinLimit) {
                        atomicOr(f.err, f.err_bit);
                        s_stop = 1u;
                        break;
                    }
                    __nanosleep(100);
                }
                __threadfence();
            }
        }
        __syncthreads();
        const uint32_t ph = s_item / tiles, tile = s_item % tiles;
        if (ph >= phases || s_stop) return;
        const uint32_t b = tile * kSortTile, e = min(f.n, b + kSortTile);
        // passes 0-7 on the second word, 8-15 on the first, 16-17 on the system
        int pass = -1;
        if (ph >= 1 && ph <= 8) pass = (int)ph - 1;
        else if (ph >= 10 && ph <= 17) pass = (int)ph - 2;
        else if (multi && (ph == 19 || ph == 20)) pass = (int)ph - 3;
        if (ph == 0) {
            // digit counts (in the buffer of the tile), identity, status words of this tile's row
            uint32_t *h = reinterpret_cast<uint32_t *>(s.buf);
            for (int k = 0; k < 18; k++) status0[((size_t)k * tiles + tile) * 256 + t] = 0u;
            for (int w = 0; w < 2; w++) {
                __syncthreads();
                for (int k = t; k < 10 * 256; k += kThreads) h[k] = 0u;
                __syncthreads();
                for (uint32_t i = b + t; i < e; i += kThreads) {
                    uint64_t k;
                    if (w) k = f.k1[i];
                    else if (f.have_k2) k = f.k2[i];
                    else f.k2[i] = k = second_word(f, i);
                    if (!w) {
                        f.key_a[i] = k;
                        f.idx_a[i] = i;
                    }
                    for (int q = 0; q < 8; q++) atomicAdd(&h[q * 256 + ((k >> (8 * q)) & 255u)], 1u);
                    if (w && multi) {
                        const uint32_t sy = f.sys_id[i];
                        atomicAdd(&h[8 * 256 + (sy & 255u)], 1u);
                        atomicAdd(&h[9 * 256 + ((sy >> 8) & 255u)], 1u);
                    }
                }
                __syncthreads();
                for (int k = t; k < (w && multi ? 10 : 8) * 256; k += kThreads)
                    if (h[k]) atomicAdd(&hist[w * 8 * 256 + k], h[k]);
            }
        } else if (pass >= 0) {
            const bool on_k1 = pass >= 8 && pass < 16, odd = pass & 1;
            uint64_t *ka = on_k1 ? f.key_b : f.key_a, *kb = on_k1 ? f.key_a : f.key_b;
            sweep_tile<true>(s, tile, odd ? kb : ka, odd ? f.idx_b : f.idx_a, odd ? ka : kb, odd ? f.idx_a : f.idx_b, f.n,
                             8 * (pass < 16 ? pass & 7 : pass - 16), hist + 256 * pass,
                             status0 + (size_t)pass * tiles * 256, f.err, f.err_bit);
        } else {
            for (uint32_t j = b + t; j < e; j += kThreads) {
                const uint32_t i = __ldcg(&f.idx_a[j]);
                if (ph == 9) f.key_b[j] = f.k1[i];
                else if (ph == 18 && multi) f.key_a[j] = f.sys_id[i];
                else if (ph == 18) f.key_a[j] = f.k2[i];
                else {
                    f.key_b[j] = f.k1[i];
                    f.key_a[j] = f.k2[i];
                    f.sys_sorted[j] = f.sys_id[i];
                }
            }
        }
        __threadfence();
        __syncthreads();
        if (t == 0) atomicAdd(done + ph, 1u);
    }
}

}  // namespace

size_t sort_scratch_bytes(uint32_t n) {
    const size_t tiles = (n + kSortTile - 1) / kSortTile;
    return 4 * (kSortStatus + kSortSlots * tiles * 256);
}

size_t sort_zero_words(uint32_t n, int passes) {
    const size_t tiles = (n + kSortTile - 1) / kSortTile;
    return kSortStatus + (size_t)passes * tiles * 256;
}

cudaError_t sort_reset(uint32_t *scratch, uint32_t n, int passes, cudaStream_t st) {
    const size_t words = sort_zero_words(n, passes);
    const unsigned blocks = (unsigned)std::min<size_t>(1184, (words / 4 + 255) / 256);
    return launch_pdl(k_zero_words, dim3(blocks ? blocks : 1), dim3(256), 0, st, scratch, words);
}

cudaError_t sort_histograms(const uint64_t *w, int slot, uint32_t n, uint32_t *scratch, cudaStream_t st,
                            unsigned *launches) {
    const unsigned blocks = (unsigned)std::min<size_t>(1184, (n + 255) / 256);
    *launches += 1;
    return launch_pdl(k_hist, dim3(blocks ? blocks : 1), dim3(256), 0, st, w, slot, n, scratch);
}

cudaError_t sort_pass(const uint64_t *kin, const uint32_t *iin, uint64_t *kout, uint32_t *iout, uint32_t n, int slot,
                      int shift, uint32_t *scratch, uint32_t *err, uint32_t err_bit, cudaStream_t st,
                      unsigned *launches) {
    const size_t tiles = (n + kSortTile - 1) / kSortTile;
    *launches += 1;
    return launch_pdl(k_onesweep, dim3((unsigned)tiles), dim3(kThreads), 0, st, kin, iin, kout, iout, n, shift,
                      scratch + 256 * slot, scratch + kSortStatus + (size_t)slot * tiles * 256,
                      scratch + kSortCounters + slot, err, err_bit);
}

cudaError_t sort_full(const FullSort &f, cudaStream_t st, unsigned *launches) {
    const size_t tiles = (f.n + kSortTile - 1) / kSortTile;
    *launches += 1;
    return launch_pdl(k_full_sort, dim3((unsigned)std::min<size_t>(296, tiles)), dim3(kThreads), 0, st, f);
}

}  // namespace nbody
