// Individual particles on a lattice: Brownian step, binning by radix sort and
// cell offsets, in-cell A + B -> 0 pairing, compaction.
//
// The reference keeps individuals as 64-bit (cell, id) keys, moves them one
// lattice cell at a time (individual_diffuseX/Y, IndividualSolver.cl:750-1014),
// re-sorts after every move (IndividualSolver::computeDiffusionConstants ->
// sortSpecies, IndividualSolver.cpp:1100-1153, :673-712) and handles births and
// deaths by scans and compaction (maintainPopulation, IndividualSolver.cpp:458-671).
// This path keeps continuous positions (one float2 each, so that a gather is one access) and a
// species byte per particle;
// a step is
//   move:    x += vx dt + sqrt(2 D dt) z (Box-Muller normals from the particle's
//            Philox stream), reflecting walls, key = floor(y) G + floor(x);
//   bin:     stable radix sort of (key, index) (the move counts the digits, the
//            sort's last pass the particles per cell);
//   react:   in each cell the k-th A (in sorted order) pairs with the k-th B and the
//            pair is removed with probability p (one 32-bit draw per pair against
//            floor(p 2^32));
//   compact: survivors in sorted order.
// In long lists react and compact go by the sorted list (k_pairs, k_compact); in short ones
// they are one kernel over the cells, which also scans the counts into the cell starts
// (k_react_compact).
// Compiled with -fmad=false: positions must round as the CPU replay does.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "lookback.cuh"
#include "host_common.h"
#include "sort_kernels.h"
#include "../../include/gpgmp_c.h"

using namespace gpgmp;

namespace {

__device__ __forceinline__ float reflect_into(float x, float L) {
    if (x < 0.0f) x = -x;
    if (x >= L) x = (L + L) - x;
    if (x < 0.0f) x = 0.0f;
    if (x >= L) x = nextafterf(L, 0.0f);
    return x;
}

// The move also counts the radix digits of the new keys for every sort pass (the
// histogram the sort would otherwise read the keys again for).  Bound by its instructions
// (a Philox block, a logarithm, sine and cosine, a square root): one block of draws without
// the stream's buffer, the passes unrolled, the next position loaded a round ahead, and no
// index written (the sort's first pass makes it).  4.2M particles on 1024 x 1024: 52 us
// before, 37 now.
template <int RB, int PASSES>
__global__ void __launch_bounds__(256, 6) k_move(float2* __restrict__ pos, const uint32_t* __restrict__ np, int G,
                                                 float sig, float ax, float ay, uint32_t seed, uint32_t step,
                                                 uint32_t* __restrict__ keys, uint32_t* __restrict__ hist) {
    constexpr int DIG = 1 << RB;
    __shared__ uint32_t s_h[PASSES * DIG];
    for (int i = threadIdx.x; i < PASSES * DIG; i += blockDim.x) s_h[i] = 0;
    __syncthreads();
    const int n = (int)*np;
    const float L = (float)G;
    const int lane = threadIdx.x & 31;
    const int stride = (int)(gridDim.x * blockDim.x);
    int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    float2 at = make_float2(0.0f, 0.0f);
    if (i < n) at = pos[i];
    // whole warps step together (the digit counts below are warp-collective)
    for (; i - lane < n; i += stride) {
        const bool valid = i < n;
        const float2 from = at;
        if (i + stride < n) at = pos[i + stride];      // n < 2^30, the grid has fewer threads than that
        uint32_t w[4];
        philox4x32_10(0u, step, (uint32_t)i, PH_PART, seed, 0u, w);
        float z0, z1;
        normal2(w[0], w[1], &z0, &z1);
        float xn = from.x + ax;
        xn = xn + sig * z0;
        float yn = from.y + ay;
        yn = yn + sig * z1;
        xn = reflect_into(xn, L);
        yn = reflect_into(yn, L);
        const uint32_t k = (uint32_t)(int)yn * (uint32_t)G + (uint32_t)(int)xn;
        if (valid) {
            pos[i] = make_float2(xn, yn);
            keys[i] = k;
        }
        // The particles come in the last step's cell order, so a warp's upper digits
        // are mostly all the same: one add for the warp then, one per lane otherwise.
        const unsigned vmask = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            const uint32_t d = (k >> (RB * p)) & (DIG - 1u);
            const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);      // lane 0 is in range
            if (__all_sync(0xffffffffu, !valid || d == d0)) {
                if (lane == 0) atomicAdd(&s_h[p * DIG + d0], (uint32_t)__popc(vmask));
            } else if (valid) {
                atomicAdd(&s_h[p * DIG + d], 1u);
            }
        }
    }
    __syncthreads();
    for (int i2 = threadIdx.x; i2 < PASSES * DIG; i2 += blockDim.x) {
        const uint32_t c = s_h[i2];
        if (c) atomicAdd(&hist[i2], c);
    }
}

// React and compact in one pass over the cells, with two decoupled look-back scans
// (lookback.cuh).  A tile of 1024 cells (four per thread) takes its cells' starts
// from the scan of the counts; its particles are then one contiguous range of the
// sorted list, whose species bytes the block stages in shared memory.  Each thread
// pairs the A's and B's of its cells there: the k-th A in sorted order with the k-th
// B, a pair going with probability thresh / 2^32 (one 32-bit draw per pair from the
// cell's stream), from species bit masks in a cell of up to 32 particles and by
// walking the staged bytes in a larger one.  Then the tile takes its survivors' output offset from the scan of the
// survivor counts, and each warp writes the survivors of its own threads' cells
// (position and species) with ballot-ranked, coalesced stores: the order of
// compacting the sorted list by alive flags.  The last tile writes the total.  A tile
// with more particles than the staging holds walks each cell in global memory with
// alive flags instead.
constexpr int kRcThreads = 256;
constexpr int kRcCells = 4;
constexpr int kRcTile = kRcThreads * kRcCells;
constexpr int kRcWarps = kRcThreads / 32;
constexpr uint8_t kRcDead = 0xffu;

// exclusive sum over the block (kRcThreads threads); *total = the block's sum
__device__ __forceinline__ uint32_t block_excl_sum(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kRcWarps ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < kRcWarps) s_warp[lane] = w;
    }
    __syncthreads();
    *total = s_warp[kRcWarps - 1];
    return (warp == 0 ? 0u : s_warp[warp - 1]) + incl - v;
}

// Pairs one cell's A's and B's in order; dead(place) is called for both of a pair that goes.
// Returns the number of pairs removed.
template <class SP, class DEAD>
__device__ __forceinline__ uint32_t pair_cell(uint32_t b, uint32_t f, const SP& species, uint32_t seed, uint32_t step,
                                              uint32_t cell, uint32_t thresh, const DEAD& dead) {
    Stream st;
    st.init(seed, 1u, step, cell, PH_PAIR);
    uint32_t ia = b, ib = b, removed = 0;
    for (;;) {
        while (ia < f && species(ia) != 0) ia++;
        while (ib < f && species(ib) != 1) ib++;
        if (ia >= f || ib >= f) break;
        if (st.next() < thresh) {
            dead(ia);
            dead(ib);
            removed++;
        }
        ia++;
        ib++;
    }
    return removed;
}

// scratch (uint64 words): [0] tile counter (u32), error word (u32 at byte 8), two unused,
// then the status words of the two scans, ntiles each.
// Dynamic shared memory: cap bytes (species of the staged particles).
// (at most 32 registers: eight tiles per SM, so the 1024 tiles of a 1024 x 1024 grid
// are resident in one wave)
__global__ void __launch_bounds__(kRcThreads, 8) k_react_compact(
    const uint32_t* __restrict__ count, uint32_t* __restrict__ start, int64_t ncells,
    const uint32_t* __restrict__ svals, const float2* __restrict__ pos, const uint8_t* __restrict__ sp,
    uint32_t seed, uint32_t step, uint32_t thresh, uint32_t* __restrict__ alive, float2* __restrict__ pos2, uint8_t* __restrict__ sp2, uint64_t* __restrict__ scratch,
    uint32_t ntiles, uint32_t cap, uint32_t* __restrict__ total) {
    extern __shared__ uint8_t s_sp[];          // [cap] species, kRcDead = removed
    __shared__ uint32_t s_tile, s_prefix;
    __shared__ uint32_t s_warp[kRcWarps];
    unsigned int* counter = reinterpret_cast<unsigned int*>(scratch);
    int* err = reinterpret_cast<int*>(scratch) + 2;
    uint64_t* status_start = scratch + 4;
    uint64_t* status_out = status_start + ntiles;
    if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t c0 = (int64_t)tile * kRcTile + (int64_t)threadIdx.x * kRcCells;
    uint32_t cnt[kRcCells];
    if (c0 + kRcCells <= ncells) {
        const uint4 w = *reinterpret_cast<const uint4*>(count + c0);
        cnt[0] = w.x; cnt[1] = w.y; cnt[2] = w.z; cnt[3] = w.w;
    } else {
#pragma unroll
        for (int j = 0; j < kRcCells; ++j) cnt[j] = c0 + j < ncells ? count[c0 + j] : 0u;
    }
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < kRcCells; ++j) sum += cnt[j];
    uint32_t agg;
    const uint32_t ex = block_excl_sum(sum, s_warp, &agg);
    if (warp == 0) {
        const uint32_t p = warp_lookback_u32(status_start, tile, agg, err);
        if (lane == 0) s_prefix = p;
    }
    __syncthreads();
    const uint32_t S = s_prefix;               // the tile's first particle in the sorted list
    uint32_t o[kRcCells + 1];                  // the cells' offsets within the tile
    o[0] = ex;
#pragma unroll
    for (int j = 0; j < kRcCells; ++j) o[j + 1] = o[j] + cnt[j];
    if (c0 + kRcCells <= ncells) {
        *reinterpret_cast<uint4*>(start + c0) = make_uint4(S + o[0], S + o[1], S + o[2], S + o[3]);
    } else {
#pragma unroll
        for (int j = 0; j < kRcCells; ++j)
            if (c0 + j < ncells) start[c0 + j] = S + o[j];
    }
    const bool staged = agg <= cap;            // the same in every thread of the block
    // the part of the staged range that holds this warp's threads' cells
    const uint32_t w0 = __shfl_sync(0xffffffffu, o[0], 0);
    const uint32_t w1 = __shfl_sync(0xffffffffu, o[kRcCells], 31);
    uint32_t removed = 0;
    if (staged) {
        for (uint32_t p0 = 0; p0 < agg; p0 += 4 * kRcThreads) {
            uint32_t src[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t p = p0 + u * kRcThreads + threadIdx.x;
                src[u] = p < agg ? svals[S + p] : 0u;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t p = p0 + u * kRcThreads + threadIdx.x;
                if (p < agg) s_sp[p] = sp[src[u]];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kRcCells; ++j) {
            if (cnt[j] >= 2) {
                if (cnt[j] <= 32) {
                    Stream st;
                    st.init(seed, 1u, step, (uint32_t)(c0 + j), PH_PAIR);
                    // species masks of the cell; the k-th set bits of the two masks pair
                    uint32_t am = 0, bm = 0;
                    for (uint32_t q = 0; q < cnt[j]; ++q) {
                        const uint8_t t = s_sp[o[j] + q];
                        am |= (uint32_t)(t == 0) << q;
                        bm |= (uint32_t)(t == 1) << q;
                    }
                    while (am && bm) {
                        const int ia = __ffs(am) - 1, ib = __ffs(bm) - 1;
                        am &= am - 1u;
                        bm &= bm - 1u;
                        if (st.next() < thresh) {
                            s_sp[o[j] + ia] = kRcDead;
                            s_sp[o[j] + ib] = kRcDead;
                            removed++;
                        }
                    }
                } else {
                    removed += pair_cell(o[j], o[j + 1], [&](uint32_t q) { return s_sp[q]; }, seed, step,
                                         (uint32_t)(c0 + j), thresh, [&](uint32_t q) { s_sp[q] = kRcDead; });
                }
            }
        }
    } else {
        const auto global_sp = [&](uint32_t q) { return sp[svals[q]]; };
        for (uint32_t q = S + o[0]; q < S + o[kRcCells]; ++q) alive[q] = 1u;
#pragma unroll
        for (int j = 0; j < kRcCells; ++j) {
            if (cnt[j] >= 2) {
                removed += pair_cell(S + o[j], S + o[j + 1], global_sp, seed, step, (uint32_t)(c0 + j), thresh,
                                     [&](uint32_t q) { alive[q] = 0u; });
            }
        }
    }
    const uint32_t surv = sum - 2 * removed;
    uint32_t agg2;
    const uint32_t ex2 = block_excl_sum(surv, s_warp, &agg2);
    if (warp == 0) {
        const uint32_t p = warp_lookback_u32(status_out, tile, agg2, err);
        if (lane == 0) {
            s_prefix = p;
            if (tile == ntiles - 1) *total = p + agg2;
        }
    }
    __syncthreads();
    if (staged) {
        // warp w writes the particles of its own threads' cells -- one contiguous part
        // [w0, w1) of the staged range -- in rows of 32; its survivors start where its
        // first lane's exclusive survivor count says
        uint32_t d = s_prefix + __shfl_sync(0xffffffffu, ex2, 0);
        for (uint32_t r = w0; r < w1; r += 32) {
            const uint32_t p = r + lane;
            const bool live = p < w1 && s_sp[p] != kRcDead;
            const unsigned m = __ballot_sync(0xffffffffu, live);
            if (live) {
                const uint32_t dd = d + __popc(m & ((1u << lane) - 1u));
                const uint32_t src = svals[S + p];
                pos2[dd] = pos[src];
                sp2[dd] = s_sp[p];
            }
            d += __popc(m);
        }
    } else {
        uint32_t d = s_prefix + ex2;
        for (uint32_t q = S + o[0]; q < S + o[kRcCells]; ++q) {
            if (removed && !alive[q]) continue;
            const uint32_t src = svals[q];
            pos2[d] = pos[src];
            sp2[d] = sp[src];
            d++;
        }
    }
}

// The same from the sorted keys, for long lists (particles_step_one), as two
// kernels that wait for no other tile: k_pairs marks the removed places of the sorted list,
// a bit each, and counts them per tile and per group of tiles; k_compact adds up the counts
// before its tile and writes the survivors.  A tile is kRrTile places and owns the cells that
// begin there.  Cells' starts and counts come from the places where the key changes, so the
// sort need not count the cells; the cell after a gap of empty ones writes theirs.  A tile's
// last cell may reach up to 256 places into the next tile; one that goes on after that is
// paired in global memory.
// Bound by the loads' latency and the instructions around them, so k_pairs takes eight places
// per thread with 16-byte loads and keeps heads and species as bits (a place per lane and a
// ballot per row: 33 us, now 26).  4.2M particles on 1024 x 1024, both kernels: 57 us, with
// which k_react_compact and the counting in the sort are level (60); 16.8M on 1024 x 1024 a
// step of 543 us against 674, 1M 90 against 101, 4.2M on 2000 x 2000 227 against 276.  As one
// kernel with a look-back between pairs and survivors it took 84 to 94 us: 2048 tiles in
// four waves, each waiting for its slowest.
constexpr int kRrThreads = 256, kRrWarps = kRrThreads / 32, kRrRows = 8;
constexpr int kRrTile = kRrThreads * kRrRows, kRrGroup = 1024;      // places of a tile, tiles of a group
constexpr int kRrGroups = (1 << 30) / (kRrTile * kRrGroup);
// Runs of empty cells: up to 4 are written by the thread of the cell after them, then by its
// warp, from kRrBigGap by its block, from kRrHugeGap by all blocks of k_compact.
constexpr uint32_t kRrBigGap = 512, kRrGaps = 16, kRrHugeGap = 16384;
// what k_pairs leaves for k_compact, zeroed before: the number of huge gaps, the removed
// places' counts per group and tile, and their bits; then the gaps (first cell, cell after,
// start), which need no zeroing
struct Removed {
    uint32_t *ngaps, *groups, *tile, *bits, *gaps;
    __host__ __device__ Removed(uint32_t* p, uint32_t tiles)
        : ngaps(p), groups(p + 1), tile(p + 1 + kRrGroups), bits(p + 1 + kRrGroups + tiles),
          gaps(p + zeroed(tiles)) {}
    __host__ __device__ static size_t zeroed(uint32_t tiles) {
        return 1 + kRrGroups + (size_t)tiles * (1 + kRrTile / 32);
    }
    static size_t words(uint32_t tiles, int64_t ncells) { return zeroed(tiles) + 3 * (size_t)(ncells / kRrHugeGap + 1); }
    __device__ __forceinline__ void gap(uint32_t a, uint32_t b, uint32_t q) const {
        uint32_t* g = gaps + 3 * (size_t)atomicAdd(ngaps, 1u);
        g[0] = a;
        g[1] = b;
        g[2] = q;
    }
    __device__ __forceinline__ void add(uint32_t t, uint32_t count) const {
        atomicAdd(&tile[t], count);
        atomicAdd(&groups[t / kRrGroup], count);
    }
};
// Every warp sums up the bits of words 0 .. W - 1 by itself: the total, and at(r), the bits
// before this warp's word of row r.
struct WordSums {
    uint32_t v[3], all;
    template <class WORD>
    __device__ __forceinline__ WordSums(int words, const WORD& word) {
        const int lane = threadIdx.x & 31;
        uint32_t c[3], mine = 0;
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            c[u] = 3 * lane + u < words ? __popc(word(3 * lane + u)) : 0u;
            mine += c[u];
        }
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        v[0] = incl - mine;
        v[1] = v[0] + c[0];
        v[2] = v[1] + c[1];
        all = __shfl_sync(0xffffffffu, incl, 31);
    }
    __device__ __forceinline__ uint32_t at(int r) const {
        const int w = r * kRrWarps + (threadIdx.x >> 5), u = w % 3;
        return __shfl_sync(0xffffffffu, u == 0 ? v[0] : u == 1 ? v[1] : v[2], w / 3);
    }
};

__global__ void __launch_bounds__(kRrThreads, 6) k_pairs(
    const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ svals, const uint32_t* __restrict__ np, uint32_t ncells,
    const uint8_t* __restrict__ sp, uint32_t seed, uint32_t step, uint32_t thresh, uint32_t* __restrict__ start,
    uint32_t* __restrict__ count, Removed removed) {
    constexpr int kSpan = kRrTile + kRrThreads;     // places a tile looks at
    constexpr int kWords = kSpan / 32;              // a bit per place: a thread's eight are a byte
    __shared__ __align__(16) uint32_t s_key[kRrTile];
    __shared__ uint16_t s_head[kRrTile + 1];        // the tile's cells: their first places, then the end
    __shared__ uint32_t s_dead[kWords];             // removed places
    __shared__ uint32_t s_a[kWords + 1], s_b[kWords + 1];      // places of species 0 and 1
    __shared__ uint32_t s_cnt[kRrWarps];
    __shared__ uint32_t s_end, s_ngaps;
    __shared__ uint32_t s_gap[kRrGaps][3];          // long gaps: first cell, cell after, start
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n = *np, tile = blockIdx.x, i0 = tile * kRrTile;
    // the cells a .. b - 1 are empty and would start at place q
    const auto fill = [&](uint32_t a, uint32_t b, uint32_t q, uint32_t from, uint32_t by) {
        for (uint32_t c = a + from; c < b; c += by) {
            start[c] = q;
            count[c] = 0u;
        }
    };
    if (i0 >= n) {
        if (tile == 0 && tid == 0) removed.gap(0, ncells, 0);
        return;
    }
    const uint32_t m = min(n - i0, (uint32_t)kSpan);          // places there are
    const uint32_t own = min(m, (uint32_t)kRrTile);
    // eight places from p on: keys and species bits (places past the list: key 2^32 - 1)
    uint32_t key[8], abits, bbits;
    const auto load = [&](uint32_t p) {
        uint32_t src[8];
        if (p + 8 <= m) {
            const uint4* k = reinterpret_cast<const uint4*>(skeys + i0 + p);
            const uint4* v = reinterpret_cast<const uint4*>(svals + i0 + p);
            const uint4 k0 = k[0], k1 = k[1], v0 = v[0], v1 = v[1];
            key[0] = k0.x; key[1] = k0.y; key[2] = k0.z; key[3] = k0.w;
            key[4] = k1.x; key[5] = k1.y; key[6] = k1.z; key[7] = k1.w;
            src[0] = v0.x; src[1] = v0.y; src[2] = v0.z; src[3] = v0.w;
            src[4] = v1.x; src[5] = v1.y; src[6] = v1.z; src[7] = v1.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                key[j] = p + j < m ? skeys[i0 + p + j] : 0xffffffffu;
                src[j] = p + j < m ? svals[i0 + p + j] : 0u;
            }
        }
        uint8_t t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = sp[src[j]];
        abits = bbits = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            abits |= (uint32_t)(t[j] == 0) << j;
            bbits |= (uint32_t)(t[j] == 1) << j;
        }
    };
    // which of the eight begin a cell; before: the key of the place before them
    const auto begins = [&](uint32_t before) {
        uint32_t h = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) h |= (uint32_t)(key[j] != (j ? key[j - 1] : before)) << j;
        return h;
    };
    uint8_t* a8 = reinterpret_cast<uint8_t*>(s_a);
    uint8_t* b8 = reinterpret_cast<uint8_t*>(s_b);
    const uint32_t p0 = 8 * tid;
    if (tid < kWords) s_dead[tid] = 0;
    if (tid == 0) {
        s_ngaps = 0;
        s_a[kWords] = s_b[kWords] = 0;
    }
    if (warp == 0) {
        // the places after the tile's own: where its last cell ends, if in sight
        load(kRrTile + p0);
        uint32_t before = __shfl_up_sync(0xffffffffu, key[7], 1);
        if (lane == 0) before = m > kRrTile ? skeys[i0 + kRrTile - 1] : 0xffffffffu;
        const uint32_t h = begins(before);
        const unsigned any = __ballot_sync(0xffffffffu, h != 0);
        const uint32_t mine = kRrTile + p0 + __ffs(h) - 1;
        const uint32_t e = __shfl_sync(0xffffffffu, mine, any ? __ffs(any) - 1 : 0);
        if (lane == 0) s_end = any ? e : (uint32_t)kSpan;
        a8[kRrTile / 8 + tid] = (uint8_t)abits;
        b8[kRrTile / 8 + tid] = (uint8_t)bbits;
    }
    load(p0);
    uint32_t heads;
    {
        uint32_t before = __shfl_up_sync(0xffffffffu, key[7], 1);
        if (lane == 0) before = i0 + p0 && p0 < m ? skeys[i0 + p0 - 1] : 0xffffffffu;
        heads = begins(before);
        // the list's end is not a cell's beginning
        if (p0 + 8 > m) heads &= p0 < m ? (1u << (m - p0)) - 1u : 0u;
    }
    a8[tid] = (uint8_t)abits;
    b8[tid] = (uint8_t)bbits;
    reinterpret_cast<uint4*>(s_key)[2 * tid] = make_uint4(key[0], key[1], key[2], key[3]);
    reinterpret_cast<uint4*>(s_key)[2 * tid + 1] = make_uint4(key[4], key[5], key[6], key[7]);
    uint32_t incl = __popc(heads);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_cnt[warp] = incl;
    __syncthreads();
    uint32_t at = incl - __popc(heads), nheads = 0;
#pragma unroll
    for (int w = 0; w < kRrWarps; ++w) {
        at += w < warp ? s_cnt[w] : 0u;
        nheads += s_cnt[w];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (heads >> j & 1u) s_head[at++] = (uint16_t)(p0 + j);
    // the last cell ends at a beginning in sight, at the list's end, or out of sight
    const uint32_t head_end = s_end;
    const bool big = nheads > 0 && head_end == kSpan && n - i0 > kSpan;
    if (tid == 0) s_head[nheads] = (uint16_t)(m <= kRrTile ? m : min(head_end, m));
    __syncthreads();
    const uint32_t cells = nheads - (big ? 1u : 0u);           // cells to pair here
    const auto dead = [&](uint32_t q) { atomicOr(&s_dead[q >> 5], 1u << (q & 31u)); };
    for (uint32_t c0 = warp * 32; c0 < nheads; c0 += kRrThreads) {
        const uint32_t c = c0 + lane;
        uint32_t cell = 0, gap0 = 0, p = 0;
        if (c < nheads) {
            p = s_head[c];
            cell = s_key[p];
            gap0 = p ? s_key[p - 1] + 1u : i0 ? skeys[i0 - 1] + 1u : 0u;
            start[cell] = i0 + p;
        }
        if (c < cells) {
            const uint32_t f = s_head[c + 1], cnt = f - p;
            count[cell] = cnt;
            if (cnt <= 32) {
                // species masks of the cell; the k-th set bits of the two masks pair
                const uint32_t w = p >> 5, mask = 0xffffffffu >> (32 - cnt);
                uint32_t am = __funnelshift_r(s_a[w], s_a[w + 1], p) & mask;
                uint32_t bm = __funnelshift_r(s_b[w], s_b[w + 1], p) & mask;
                if (am && bm) {
                    Stream st;
                    st.init(seed, 1u, step, cell, PH_PAIR);
                    do {
                        uint32_t d[4];
                        st.block(d);
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (am && bm && d[u] < thresh) {
                                dead(p + __ffs(am) - 1);
                                dead(p + __ffs(bm) - 1);
                            }
                            am &= am - 1u;
                            bm &= bm - 1u;
                        }
                    } while (am && bm);
                }
            } else {
                pair_cell(p, f, [&](uint32_t q) {
                    const uint32_t bit = q & 31u;
                    return s_a[q >> 5] >> bit & 1u ? 0 : s_b[q >> 5] >> bit & 1u ? 1 : 2;
                }, seed, step, cell, thresh, dead);
            }
        }
        // empty cells before this one: a few by the thread, more by the warp, many by the
        // block below
        const uint32_t gap = c < nheads ? cell - gap0 : 0u;
        bool wide = gap > 4;
        if (gap >= kRrHugeGap) {
            removed.gap(gap0, cell, i0 + p);
            wide = false;
        } else if (gap >= kRrBigGap) {
            const uint32_t slot = atomicAdd(&s_ngaps, 1u);
            if (slot < kRrGaps) {
                s_gap[slot][0] = gap0;
                s_gap[slot][1] = cell;
                s_gap[slot][2] = i0 + p;
                wide = false;
            }
        } else if (!wide) {
            fill(gap0, cell, i0 + p, 0, 1);
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1u) {
            const int l = __ffs(todo) - 1;
            fill(__shfl_sync(0xffffffffu, gap0, l), __shfl_sync(0xffffffffu, cell, l),
                 i0 + __shfl_sync(0xffffffffu, p, l), lane, 32);
        }
    }
    __syncthreads();
    // the tile's bits are words 0 .. 63 (warps 0 and 1), the next tile's the rest (warp 2)
    if (warp < 3) {
        const uint32_t w = tid < kWords ? s_dead[tid] : 0u;
        if (w) atomicOr(&removed.bits[(size_t)tile * (kRrTile / 32) + tid], w);
        const uint32_t sum = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(w));
        if (sum && lane == 0) removed.add(tile + (warp == 2 ? 1u : 0u), sum);
    }
    const uint32_t gaps = min(s_ngaps, (uint32_t)kRrGaps);
    for (uint32_t g = 0; g < gaps; ++g) fill(s_gap[g][0], s_gap[g][1], s_gap[g][2], tid, kRrThreads);
    if (n - i0 <= kRrTile) {
        const uint32_t after = s_key[own - 1] + 1u;
        if (ncells - after < kRrHugeGap) fill(after, ncells, n, tid, kRrThreads);
        else if (tid == 0) removed.gap(after, ncells, n);
    }
    if (big && tid == 0) {
        const uint32_t p = i0 + s_head[cells], cell = s_key[s_head[cells]];
        uint32_t lo = i0 + kSpan, hi = n;      // every place before lo that is not before p is the cell's
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (skeys[mid] == cell) lo = mid + 1;
            else hi = mid;
        }
        count[cell] = lo - p;
        pair_cell(p, lo, [&](uint32_t q) { return sp[svals[q]]; }, seed, step, cell, thresh, [&](uint32_t q) {
            atomicOr(&removed.bits[q >> 5], 1u << (q & 31u));
            removed.add(q / kRrTile, 1u);
        });
    }
}

__global__ void __launch_bounds__(kRrThreads, 6) k_compact(
    const uint32_t* __restrict__ svals, const uint32_t* __restrict__ np, const float2* __restrict__ pos, const uint8_t* __restrict__ sp,
    Removed removed, uint32_t* __restrict__ start, uint32_t* __restrict__ count, float2* __restrict__ pos2,
    uint8_t* __restrict__ sp2, uint32_t* __restrict__ total) {
    __shared__ uint32_t s_sum[kRrWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t n = *np, tile = blockIdx.x, i0 = tile * kRrTile;
    for (uint32_t g = 0, gaps = *removed.ngaps; g < gaps; ++g) {
        const uint32_t* gap = removed.gaps + 3 * (size_t)g;
        const uint32_t after = gap[1], q = gap[2];
        for (uint32_t c = gap[0] + tile * kRrThreads + tid; c < after; c += gridDim.x * kRrThreads) {
            start[c] = q;
            count[c] = 0u;
        }
    }
    if (i0 >= n) {
        if (tile == 0 && tid == 0) *total = 0u;
        return;
    }
    const uint32_t m = min(n - i0, (uint32_t)kRrTile);
    uint32_t src[kRrRows], word[kRrRows];
#pragma unroll
    for (int r = 0; r < kRrRows; ++r) {
        const uint32_t p = r * kRrThreads + tid;
        src[r] = p < m ? svals[i0 + p] : 0u;
        word[r] = removed.bits[(size_t)tile * (kRrTile / 32) + r * kRrWarps + warp];
    }
    // removed places before the tile
    const uint32_t group = tile / kRrGroup;
    uint32_t sum = 0;
    for (uint32_t g = tid; g < group; g += kRrThreads) sum += removed.groups[g];
    for (uint32_t t = group * kRrGroup + tid; t < tile; t += kRrThreads) sum += removed.tile[t];
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) s_sum[warp] = sum;
    const WordSums gone(kRrTile / 32, [&](int w) { return removed.bits[(size_t)tile * (kRrTile / 32) + w]; });
    float2 at[kRrRows];
    uint8_t sv[kRrRows];
#pragma unroll
    for (int r = 0; r < kRrRows; ++r) {
        if ((uint32_t)(r * kRrThreads + tid) < m) {
            at[r] = pos[src[r]];
            sv[r] = sp[src[r]];
        }
    }
    __syncthreads();
    uint32_t base = i0;
#pragma unroll
    for (int w = 0; w < kRrWarps; ++w) base -= s_sum[w];
    if (n - i0 <= kRrTile && tid == 0) *total = base + m - gone.all;
#pragma unroll
    for (int r = 0; r < kRrRows; ++r) {
        const uint32_t p = r * kRrThreads + tid;
        const uint32_t d = base + p - gone.at(r) - __popc(word[r] & ((1u << lane) - 1u));
        if (p < m && !(word[r] >> lane & 1u)) {
            pos2[d] = at[r];
            sp2[d] = sv[r];
        }
    }
}

// positions between the caller's two arrays and the steps' one
__global__ void k_join(const float* __restrict__ x, const float* __restrict__ y, float2* __restrict__ pos, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        pos[i] = make_float2(x[i], y[i]);
}
__global__ void k_split(const float2* __restrict__ pos, float* __restrict__ x, float* __restrict__ y, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float2 p = pos[i];
        x[i] = p.x;
        y[i] = p.y;
    }
}
inline unsigned grid_of(int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8); }

}  // namespace

struct gpgmp_particles {
    int64_t cap = 0, n = 0;
    int grid = 0;
    float D = 0, vx = 0, vy = 0, dt = 1, p = 0;
    uint32_t seed = 0, thresh = 0;
    int32_t step = 0;
    int key_bits = 32;
    cudaStream_t stream = nullptr;
    float2 *pos = nullptr, *pos2 = nullptr;      // pos2: the next step's, and free between steps
    uint8_t *sp = nullptr, *sp2 = nullptr;
    uint32_t *keys = nullptr, *skeys = nullptr, *svals = nullptr;
    uint32_t *start = nullptr, *count = nullptr, *alive = nullptr;
    void* sort_scratch = nullptr;
    uint32_t* removed = nullptr;     // k_pairs: counts and bits of the removed places
    uint64_t* rc_scratch = nullptr;  // react + compact: tile counter, error word, total, scan status words
    uint32_t rc_tiles = 0;
    uint32_t* dn = nullptr;          // the number of particles before and after a step, by the step's parity
    uint32_t* host_tail = nullptr;   // pinned: that number read back, and as a call starts with it
};

#define CK(expr)                                                                                              \
    do {                                                                                                      \
        cudaError_t e_ = (expr);                                                                              \
        if (e_ != cudaSuccess) return set_error(GPGMP_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e_));    \
    } while (0)

extern "C" {

int gpgmp_particles_destroy(gpgmp_particles* h) {
    if (!h) return GPGMP_OK;
    cudaStreamSynchronize(h->stream);
    void* ptrs[] = {h->pos, h->pos2, h->sp, h->sp2, h->keys, h->skeys, h->svals, h->start,
                    h->count, h->alive, h->sort_scratch, h->removed, h->rc_scratch, h->dn};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (h->host_tail) cudaFreeHost(h->host_tail);
    delete h;
    return GPGMP_OK;
}

int gpgmp_particles_create(int64_t capacity, int32_t grid, float D, float vx, float vy, float dt, float p_react,
                           uint32_t seed, gpgmp_particles** out) {
    if (!out || capacity <= 0 || capacity >= ((int64_t)1 << 30) || grid <= 0 || grid > 32768 || !(dt > 0) ||
        !(D >= 0) || !(p_react >= 0) || !(p_react <= 1))
        return set_error(GPGMP_ERR_INVALID, "bad particle system parameters");
    auto* h = new gpgmp_particles();
    h->cap = capacity;
    h->grid = grid;
    h->D = D; h->vx = vx; h->vy = vy; h->dt = dt; h->p = p_react;
    h->seed = seed;
    h->thresh = (uint32_t)std::floor((double)p_react * 4294967296.0 < 4294967295.0
                                         ? (double)p_react * 4294967296.0 : 4294967295.0);
    const int64_t ncells = (int64_t)grid * grid;
    int bits = 1;
    while (((int64_t)1 << bits) < ncells) ++bits;
    h->key_bits = bits;
    const size_t n4 = sizeof(uint32_t) * (size_t)capacity;
    cudaError_t e = cudaSuccess;
    auto A = [&](void** p, size_t b) { if (e == cudaSuccess) e = cudaMalloc(p, b); };
    A((void**)&h->pos, sizeof(float2) * capacity); A((void**)&h->pos2, sizeof(float2) * capacity);
    A((void**)&h->sp, capacity); A((void**)&h->sp2, capacity);
    A((void**)&h->keys, n4); A((void**)&h->skeys, n4); A((void**)&h->svals, n4);
    A((void**)&h->alive, n4);
    A((void**)&h->start, sizeof(uint32_t) * (size_t)ncells); A((void**)&h->count, sizeof(uint32_t) * (size_t)ncells);
    A(&h->sort_scratch, sort_layout(capacity, bits).bytes);
    h->rc_tiles = (uint32_t)((ncells + kRcTile - 1) / kRcTile);
    A((void**)&h->rc_scratch, sizeof(uint64_t) * (4 + 2 * (size_t)h->rc_tiles));
    A((void**)&h->dn, 2 * sizeof(uint32_t));
    A((void**)&h->removed, sizeof(uint32_t) * Removed::words((uint32_t)((capacity + kRrTile - 1) / kRrTile), ncells));
    if (e == cudaSuccess) e = cudaMemset(h->rc_scratch, 0, 4 * sizeof(uint64_t));     // the error word
    if (e == cudaSuccess) e = cudaMallocHost((void**)&h->host_tail, 2 * sizeof(uint32_t));
    if (e != cudaSuccess) {
        int c = set_error(e == cudaErrorMemoryAllocation ? GPGMP_ERR_NOMEM : GPGMP_ERR_CUDA, "allocation: %s",
                          cudaGetErrorString(e));
        gpgmp_particles_destroy(h);
        return c;
    }
    *out = h;
    return GPGMP_OK;
}

int gpgmp_particles_set_stream(gpgmp_particles* h, void* stream) {
    if (!h) return set_error(GPGMP_ERR_INVALID, "handle is NULL");
    h->stream = (cudaStream_t)stream;
    return GPGMP_OK;
}

int gpgmp_particles_set(gpgmp_particles* h, const float* x, const float* y, const uint8_t* species, int64_t n,
                        int32_t step) {
    if (!h || n < 0 || n > h->cap || (n > 0 && (!x || !y || !species))) return set_error(GPGMP_ERR_INVALID, "bad argument");
    float *dx = reinterpret_cast<float*>(h->pos2), *dy = dx + h->cap;
    CK(cudaMemcpyAsync(dx, x, sizeof(float) * n, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(dy, y, sizeof(float) * n, cudaMemcpyHostToDevice, h->stream));
    if (n > 0) {
        k_join<<<grid_of(n), 256, 0, h->stream>>>(dx, dy, h->pos, n);
        CK(cudaGetLastError());
    }
    CK(cudaMemcpyAsync(h->sp, species, n, cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->n = n;
    h->step = step;
    return GPGMP_OK;
}

int gpgmp_particles_get(gpgmp_particles* h, float* x, float* y, uint8_t* species, int64_t* n) {
    if (!h || !n) return set_error(GPGMP_ERR_INVALID, "bad argument");
    float *dx = reinterpret_cast<float*>(h->pos2), *dy = dx + h->cap;
    if ((x || y) && h->n > 0) {
        k_split<<<grid_of(h->n), 256, 0, h->stream>>>(h->pos, dx, dy, h->n);
        CK(cudaGetLastError());
    }
    if (x) CK(cudaMemcpyAsync(x, dx, sizeof(float) * h->n, cudaMemcpyDeviceToHost, h->stream));
    if (y) CK(cudaMemcpyAsync(y, dy, sizeof(float) * h->n, cudaMemcpyDeviceToHost, h->stream));
    if (species) CK(cudaMemcpyAsync(species, h->sp, h->n, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    *n = h->n;
    return GPGMP_OK;
}

// One step of a list of at most h->n particles, whose number the device holds in one of
// h->dn's two words and which leaves its own number in the other.
static int particles_step_one(gpgmp_particles* h) {
    cudaStream_t st = h->stream;
    const uint32_t* np = h->dn + (h->step & 1);
    uint32_t* next = h->dn + (~h->step & 1);
    const int64_t n = h->n;
    const int64_t ncells = (int64_t)h->grid * h->grid;
    const float sig = sqrtf(2.0f * h->D * h->dt);
    const float ax = h->vx * h->dt, ay = h->vy * h->dt;
    const uint32_t step = (uint32_t)h->step;
    // k_pairs goes by the particles, k_react_compact by the cells: the first wins by much
    // where cells are many (a step of 262144 particles on 8192 x 8192: 194 us against 1051, on
    // 2048 x 2048: 108 against 141, on 1024 x 1024: 77 against 82; 65536 on 4096 x 4096: 162
    // against 323; 600000 on 1024 x 1024: 72 against 82), the second where the tiles of the
    // list are too few for the empty cells (131072 on 1024 x 1024: 73 against 83, 2000 on
    // 128 x 128: 41 against 70) or for the SMs (4000 on 64 x 64: 43 against 47).
    const bool rows = n >= 65536 && (n >= 262144 || 2 * n >= ncells || ncells >= (int64_t)1 << 22);
    if (!rows) CK(cudaMemsetAsync(h->count, 0, sizeof(uint32_t) * (size_t)ncells, st));
    if (n > 0) {
        CK(radix_sort_begin(n, h->key_bits, h->sort_scratch, st));
        const SortLayout L = sort_layout(n, h->key_bits);
        const unsigned blocks = (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 6);
        const auto move = [&](auto kernel) {
            kernel<<<blocks, 256, 0, st>>>(h->pos, np, h->grid, sig, ax, ay, h->seed, step, h->keys,
                                           radix_sort_hist(n, h->key_bits, h->sort_scratch));
        };
        if (L.digit_bits == 10) {
            if (L.passes == 2) move(k_move<10, 2>);
            else move(k_move<10, 3>);
        } else {
            if (L.passes == 1) move(k_move<8, 1>);
            else if (L.passes == 2) move(k_move<8, 2>);
            else move(k_move<8, 3>);      // at most 30 bits: four passes of 8 are three of 10
        }
        CK(cudaGetLastError());
        // where k_react_compact follows, the last pass also counts the particles per cell
        CK(radix_sort_finish(h->keys, nullptr, h->skeys, h->svals, n, h->key_bits, h->sort_scratch, st,
                             rows ? nullptr : h->count, ncells, np));
    }
    if (rows) {
        const uint32_t tiles = (uint32_t)((n + kRrTile - 1) / kRrTile);
        const Removed removed(h->removed, tiles);
        CK(cudaMemsetAsync(h->removed, 0, sizeof(uint32_t) * Removed::zeroed(tiles), st));
        k_pairs<<<tiles, kRrThreads, 0, st>>>(h->skeys, h->svals, np, (uint32_t)ncells, h->sp, h->seed, step,
                                              h->thresh, h->start, h->count, removed);
        CK(cudaGetLastError());
        k_compact<<<tiles, kRrThreads, 0, st>>>(h->svals, np, h->pos, h->sp, removed, h->start, h->count, h->pos2, h->sp2,
                                                next);
        CK(cudaGetLastError());
    } else {
        CK(cudaMemsetAsync(h->rc_scratch, 0, sizeof(uint64_t) * (4 + 2 * (size_t)h->rc_tiles), st));
        // staging for twice the mean number of particles per tile (+ 1024), up to 47 KB
        // (with the static shared memory, within the 48 KB a launch gets without opting in)
        uint64_t want = (uint64_t)(2.0 * (double)n * kRcTile / (double)ncells) + 1024;
        if (want > 47 * 1024) want = 47 * 1024;
        const uint32_t cap = (uint32_t)want;
        k_react_compact<<<h->rc_tiles, kRcThreads, cap, st>>>(
            h->count, h->start, ncells, h->svals, h->pos, h->sp, h->seed, step, h->thresh, h->alive, h->pos2, h->sp2,
            h->rc_scratch, h->rc_tiles, cap, next);
        CK(cudaGetLastError());
    }
    {
        float2* t = h->pos; h->pos = h->pos2; h->pos2 = t;
        uint8_t* ts = h->sp; h->sp = h->sp2; h->sp2 = ts;
    }
    h->step++;
    return GPGMP_OK;
}

int gpgmp_particles_step(gpgmp_particles* h, int32_t nsteps) {
    if (!h || nsteps < 0) return set_error(GPGMP_ERR_INVALID, "bad argument");
    if (nsteps == 0) return GPGMP_OK;
    cudaStream_t st = h->stream;
    h->host_tail[1] = (uint32_t)h->n;
    CK(cudaMemcpyAsync(h->dn + (h->step & 1), &h->host_tail[1], sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    // The number of particles only falls, so the launches of a step may be made for an older
    // one: it is read back every kSyncSteps steps and at the end, not at each (a step of 4.2M
    // particles: 199 us with, 186 without; of 20000: 63 and 50).
    constexpr int kSyncSteps = 16;
    for (int s = 0; s < nsteps; ++s) {
        const int rc = particles_step_one(h);
        if (s + 1 == nsteps || s % kSyncSteps == kSyncSteps - 1 || rc) {
            CK(cudaMemcpyAsync(&h->host_tail[0], h->dn + (h->step & 1), sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            h->n = (int64_t)h->host_tail[0];
        }
        if (rc) return rc;
    }
    return GPGMP_OK;
}

// start/count of the last step's binning (before the reaction removed pairs), the
// sorted keys and the index permutation of that step
int gpgmp_particles_bins(gpgmp_particles* h, uint32_t* start, uint32_t* count, uint32_t* sorted_keys,
                         uint32_t* sorted_index, int64_t* n_binned) {
    if (!h) return set_error(GPGMP_ERR_INVALID, "handle is NULL");
    const int64_t ncells = (int64_t)h->grid * h->grid;
    if (start) CK(cudaMemcpyAsync(start, h->start, sizeof(uint32_t) * ncells, cudaMemcpyDeviceToHost, h->stream));
    if (count) CK(cudaMemcpyAsync(count, h->count, sizeof(uint32_t) * ncells, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    int64_t nb = 0;
    if (count) for (int64_t c = 0; c < ncells; ++c) nb += count[c];
    if (sorted_keys && nb) CK(cudaMemcpy(sorted_keys, h->skeys, sizeof(uint32_t) * nb, cudaMemcpyDeviceToHost));
    if (sorted_index && nb) CK(cudaMemcpy(sorted_index, h->svals, sizeof(uint32_t) * nb, cudaMemcpyDeviceToHost));
    if (n_binned) *n_binned = nb;
    return GPGMP_OK;
}

int gpgmp_particles_status(gpgmp_particles* h, int32_t* status) {
    if (!h || !status) return set_error(GPGMP_ERR_INVALID, "bad argument");
    const SortLayout L = sort_layout(h->cap, h->key_bits);
    int a = 0, b = 0;
    CK(cudaMemcpy(&a, (const char*)h->sort_scratch + L.off_counters + 16, sizeof(int), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(&b, (const char*)h->rc_scratch + 8, sizeof(int), cudaMemcpyDeviceToHost));
    *status = (a || b) ? GPGMP_ERR_TIMEOUT : GPGMP_OK;
    return GPGMP_OK;
}

}  // extern "C"
