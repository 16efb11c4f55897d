// Scan, radix sort and cell offsets of the individual-particle path.
//
// Reference: IndividualSolver sorts (cell, id) pairs with an LSD radix sort of
// 4-bit digits built from block sort / radix offsets / 3-kernel exclusive scan /
// reorder, 6 synchronous launches per pass and 8 passes (IndividualSolver.cpp:673-808,
// kernels IndividualSolver.cl:36-369, 493-553), then derives each cell's first and
// last particle (computeCellIndices, IndividualSolver.cl:564-619).  The result is
// the stable sort by cell.
//
// Here, from the published methods (not from the reference's SDK-derived code):
//  - exclusive scan: single pass with decoupled look-back (Merrill & Garland 2016);
//  - radix sort: onesweep (Adinets & Merrill 2022): one histogram kernel for every
//    digit position, then one kernel per digit (8 bits, or 10 where that saves a
//    pass: 17-20 and 25-30 key bits) that ranks its tile (peer masks from shared-memory
//    atomicOr on the digit's low 8 bits, ballots for the rest),
//    publishes per-digit tile counts, looks back for the prefix and scatters through
//    shared memory; tile 0 scans the pass's digit counts into the digits' global
//    starts and publishes them inside its inclusive prefix, so no other tile (and no
//    separate launch) turns counts into offsets; stable;
//  - cell offsets: key histogram + exclusive scan (start), count; the reference's
//    left/right indices follow from them.
// Every look-back spin has an iteration limit; exceeding it sets the error word
// (GPGMP_ERR_TIMEOUT for the caller) and the kernel continues without waiting.
#include <type_traits>
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <cuda_runtime.h>
#include "lookback.cuh"
#include "sort_kernels.h"
#include "host_common.h"
#include "../../include/gpgmp_c.h"

namespace gpgmp {
namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 32;
constexpr int kScanTile = kScanThreads * kScanItems;   // 16384

// ---- exclusive scan ------------------------------------------------------------
// scratch: [0] tile counter, [1] error word, then one status word per tile:
// (flag << 32) | value, flag 0 = not ready, 1 = tile aggregate, 2 = inclusive prefix.
// A tile is 16384 values, 1024 consecutive ones per warp, which a warp holds in registers as
// eight rows of 32 16-byte quads: every load and store is one coalesced 512-byte row, and
// the exclusive sums come from shuffles over the eight rows at once, so nothing but the
// warps' totals passes through shared memory (partial tiles and unaligned pointers take
// element loads in the same places).
// A scan of one tile needs neither the counter nor status words (tiles == 1): it clears the
// error word itself and the scratch is not cleared before.
// A warp's 128 ROWS values in registers, as rows of 32 quads, and their exclusive sums.
template <int ROWS>
struct ScanTile {
    static constexpr int kValues = 128 * ROWS;
    uint4 v[ROWS];
    uint32_t ex[ROWS];           // sum of the warp's values before the lane's quad of row j
    // row: 128 words of shared memory of the warp's own, for the element loads and stores
    __device__ __forceinline__ void load(const uint32_t* __restrict__ in, int64_t wbase, int64_t n, int vec, int lane,
                                         uint32_t* row) {
        if (vec && wbase + kValues <= n) {      // the same in every lane
            const uint4* src = reinterpret_cast<const uint4*>(in + wbase) + lane;
#pragma unroll
            for (int j = 0; j < ROWS; ++j) v[j] = src[j * 32];
            return;
        }
        const auto at = [&](int64_t i) { return i < n ? in[i] : 0u; };
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const int64_t i = wbase + j * 128 + lane;
            v[j] = make_uint4(at(i), at(i + 32), at(i + 64), at(i + 96));
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            row[lane] = v[j].x;
            row[lane + 32] = v[j].y;
            row[lane + 64] = v[j].z;
            row[lane + 96] = v[j].w;
            __syncwarp();
            v[j] = reinterpret_cast<const uint4*>(row)[lane];
            __syncwarp();
        }
    }
    // returns the warp's total
    __device__ __forceinline__ uint32_t sum(int lane) {
#pragma unroll
        for (int j = 0; j < ROWS; ++j) ex[j] = (v[j].x + v[j].y) + (v[j].z + v[j].w);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, ex[j], o);
                if (lane >= o) ex[j] += t;
            }
        }
        uint32_t total = 0;
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            const uint32_t row = __shfl_sync(0xffffffffu, ex[j], 31);
            ex[j] += total - ((v[j].x + v[j].y) + (v[j].z + v[j].w));
            total += row;
        }
        return total;
    }
    __device__ __forceinline__ void store(uint32_t* __restrict__ out, int64_t wbase, int64_t n, int vec, int lane,
                                          uint32_t base, uint32_t* row) const {
        const bool full = vec && wbase + kValues <= n;
        uint4* dst = reinterpret_cast<uint4*>(out + wbase) + lane;
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            uint4 w;
            w.x = base + ex[j];
            w.y = w.x + v[j].x;
            w.z = w.y + v[j].y;
            w.w = w.z + v[j].z;
            if (full) {
                dst[j * 32] = w;
                continue;
            }
            reinterpret_cast<uint4*>(row)[lane] = w;
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 128; c += 32) {
                const int64_t i = wbase + j * 128 + c + lane;
                if (i < n) out[i] = row[c + lane];
            }
            __syncwarp();
        }
    }
};

// exclusive sums of W warps' totals (called by one warp): returns lane w's warp's, *sum all
template <int W>
__device__ __forceinline__ uint32_t scan_warps(uint32_t mine, int lane, uint32_t* sum) {
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    *sum = __shfl_sync(0xffffffffu, incl, W - 1);
    return incl - mine;
}

constexpr int kScanWarps = kScanThreads / 32;
__global__ void __launch_bounds__(kScanThreads, 2) k_scan_exclusive(const uint32_t* __restrict__ in,
                                                                    uint32_t* __restrict__ out, int64_t n,
                                                                    uint64_t* __restrict__ scratch, int vec,
                                                                    uint32_t tiles) {
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp[kScanWarps], s_base[kScanWarps];
    __shared__ __align__(16) uint32_t s_row[kScanWarps][128];
    unsigned int* counter = reinterpret_cast<unsigned int*>(scratch);
    int* err = reinterpret_cast<int*>(scratch) + 2;
    uint64_t* status = scratch + 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_tile = tiles > 1 ? atomicAdd(counter, 1u) : 0u;
        if (tiles == 1) *err = 0;
    }
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t wbase = (int64_t)tile * kScanTile + warp * (32 * kScanItems);
    ScanTile<kScanItems / 4> t;
    t.load(in, wbase, n, vec, lane, s_row[warp]);
    const uint32_t total = t.sum(lane);
    if (lane == 0) s_warp[warp] = total;
    __syncthreads();
    if (warp == 0) {
        uint32_t aggregate;
        const uint32_t ex = scan_warps<kScanWarps>(lane < kScanWarps ? s_warp[lane] : 0u, lane, &aggregate);
        const uint32_t prefix = tiles > 1 ? warp_lookback_u32(status, tile, aggregate, err) : 0u;
        if (lane < kScanWarps) s_base[lane] = prefix + ex;
    }
    __syncthreads();
    t.store(out, wbase, n, vec, lane, s_base[warp], s_row[warp]);
}

// Large scans: one CTA per SM, each with a ring of tiles that it takes by number as it goes.  A
// CTA publishes its tile's sum and adds up the sums of all tiles since its last one, so there
// is no chain of look-backs.  A sum takes 2 to 4 us to reach the other SMs while memory is
// busy, longer than a tile's share of the bandwidth (3 us), so a CTA keeps three tiles in
// shared memory: one loading (bulk copy), one whose sum is published, one whose prefix is
// complete and which is written.  A tile waits only for tiles of lower numbers, which running
// CTAs have taken, and a CTA publishes a tile's sum before it waits for that tile's prefix: the
// CTAs need not run at once, so a scan beside another kernel's makes do with the SMs it
// finds.  2^27 values: 187 us, 5.7 TB/s (306 us with every tile staged in shared memory by
// its own CTA and chained look-backs; 214 us with the CTAs in rounds of fixed tiles, which had
// to run all at once; HBM's floor is 166).
constexpr int kStreamThreads = 1024, kStreamWarps = kStreamThreads / 32, kStreamStages = 3;
constexpr int kStreamRows = kScanTile / (128 * kStreamWarps);
constexpr int kStreamSmem = kStreamStages * kScanTile * (int)sizeof(uint32_t);
__device__ __forceinline__ uint32_t scan_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__global__ void __launch_bounds__(kStreamThreads, 1) k_scan_stream(const uint32_t* __restrict__ in,
                                                                   uint32_t* __restrict__ out, int64_t n,
                                                                   uint64_t* __restrict__ scratch, uint32_t tiles) {
    extern __shared__ __align__(128) uint32_t s_ring[];      // [stage][kScanTile]
    __shared__ __align__(8) uint64_t s_full[kStreamStages];
    __shared__ uint32_t s_tile[kStreamStages];               // the tiles of the ring, past the last: >= tiles
    __shared__ uint32_t s_warp[kStreamWarps], s_base[kStreamWarps];
    __shared__ __align__(16) uint32_t s_row[kStreamWarps][128];
    int* err = reinterpret_cast<int*>(scratch) + 2;
    uint64_t* status = scratch + 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int* counter = reinterpret_cast<unsigned int*>(scratch);
    const auto tile_of = [&](uint32_t i) { return s_tile[i % kStreamStages]; };
    const auto first = [&](uint32_t i) { return (int64_t)tile_of(i) * kScanTile; };
    const auto whole = [&](uint32_t i) { return first(i) + kScanTile <= n; };  // all but the last tile of all
    const auto issue = [&](uint32_t i) {
        const uint32_t bar = scan_smem(&s_full[i % kStreamStages]);
        constexpr uint32_t bytes = kScanTile * sizeof(uint32_t);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                         scan_smem(s_ring + (i % kStreamStages) * kScanTile)),
                     "l"(in + first(i)), "r"(bytes), "r"(bar)
                     : "memory");
    };
    const auto wait = [&](uint32_t i) {
        const uint32_t bar = scan_smem(&s_full[i % kStreamStages]), parity = (i / kStreamStages) & 1u;
        for (uint32_t spins = 0;; ++spins) {
            uint32_t ok;
            asm volatile(
                "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                : "=r"(ok)
                : "r"(bar), "r"(parity)
                : "memory");
            if (ok) return;
            if (spins == kSpinLimit) {
                atomicExch(err, 1);
                return;
            }
        }
    };
    ScanTile<kStreamRows> t;
    const auto read = [&](uint32_t i) {
        const uint4* q = reinterpret_cast<const uint4*>(s_ring + (i % kStreamStages) * kScanTile) +
                         warp * (32 * kStreamRows) + lane;
#pragma unroll
        for (int j = 0; j < kStreamRows; ++j) t.v[j] = q[j * 32];
    };
    // the sums of tile i's warps into s_warp (the caller syncs)
    const auto sums = [&](uint32_t i) {
        if (whole(i)) {
            wait(i);
        } else {
            uint32_t* q = s_ring + (i % kStreamStages) * kScanTile;
            for (int k = threadIdx.x; k < kScanTile; k += kStreamThreads) q[k] = first(i) + k < n ? in[first(i) + k] : 0u;
            __syncthreads();       // the same in every thread of the block
        }
        read(i);
        uint32_t x = 0;
#pragma unroll
        for (int j = 0; j < kStreamRows; ++j) x += (t.v[j].x + t.v[j].y) + (t.v[j].z + t.v[j].w);
        x = __reduce_add_sync(0xffffffffu, x);
        if (lane == 0) s_warp[warp] = x;
    };
    // thread 0 takes tile numbers a tile ahead of their loads (next), so that no load waits for one
    uint32_t next = 0;
    const auto take = [&](uint32_t i) {
        s_tile[i % kStreamStages] = next;
        if (next < tiles) {
            if (whole(i)) issue(i);
            next = atomicAdd(counter, 1u);
        }
    };
    if (threadIdx.x == 0) {
        next = atomicAdd(counter, 1u);
        for (int b = 0; b < kStreamStages; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(scan_smem(&s_full[b])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (uint32_t i = 0; i < kStreamStages; ++i) take(i);
    }
    __syncthreads();
    uint32_t carry = 0, from = 0, ex = 0;       // warp 0: the sum of tiles 0 .. from - 1; the tile's sums before each warp
    if (tile_of(0) < tiles) {
        sums(0);
        __syncthreads();
        if (warp == 0) {
            uint32_t aggregate;
            ex = scan_warps<kStreamWarps>(s_warp[lane], lane, &aggregate);
            if (lane == 0) st_relaxed_u64(&status[tile_of(0)], kScanFlagA | aggregate);
        }
        __syncthreads();
    }
    for (uint32_t i = 0; tile_of(i) < tiles; ++i) {      // the same in every thread of the block
        const bool more = tile_of(i + 1) < tiles;
        if (more) sums(i + 1);
        __syncthreads();
        if (warp == 0) {
            uint32_t ex_next = 0;
            if (more) {
                uint32_t aggregate;
                ex_next = scan_warps<kStreamWarps>(s_warp[lane], lane, &aggregate);
                if (lane == 0) st_relaxed_u64(&status[tile_of(i + 1)], kScanFlagA | aggregate);
            }
            const uint32_t tile = tile_of(i);
            uint32_t before = 0, spins = 0;
            constexpr int kWords = 6;             // 192 tiles, a round of the SMs and some more, in one go
            for (uint32_t q0 = from; q0 < tile; q0 += 32 * kWords) {
                uint64_t w[kWords];
                bool ready;
                do {
                    ready = true;
#pragma unroll
                    for (int u = 0; u < kWords; ++u) {
                        const uint32_t q = q0 + 32 * u + lane;
                        w[u] = q < tile ? ld_volatile_u64(&status[q]) : kScanFlagA;
                        ready = ready && (w[u] >> 32) != 0;
                    }
                    if (!ready && ++spins > kSpinLimit) {
                        atomicExch(err, 1);
                        ready = true;
                    }
                } while (!__all_sync(0xffffffffu, ready));
#pragma unroll
                for (int u = 0; u < kWords; ++u) before += (uint32_t)w[u];
            }
            carry += __reduce_add_sync(0xffffffffu, before);
            from = tile;
            s_base[lane] = carry + ex;
            ex = ex_next;
        }
        __syncthreads();
        read(i);
        t.sum(lane);
        t.store(out, first(i) + warp * t.kValues, n, 1, lane, s_base[warp], s_row[warp]);
        __syncthreads();
        if (threadIdx.x == 0) take(i + kStreamStages);
    }
}

// ---- radix sort ------------------------------------------------------------------
// A tile is kThreads threads x kItems keys, kItems as many as the registers hold: 16.8M pairs
// of 32 bits took 446 us with tiles of 15 keys per thread, 440 with 18 (6 four-CTA shapes of
// 256 to 384 threads: 445 to 490).
template <int RB>
struct SortShape {
    static constexpr int kThreads = 512;
    static constexpr int kMinBlocks = 2;
    static constexpr int kItems = RB == 8 ? 18 : 15;
    static constexpr int kTile = kThreads * kItems;
    static constexpr int kWarps = kThreads / 32;
    // keys and values of a tile in sorted order (dynamic shared memory)
    static constexpr int kStagingBytes = 2 * kTile * (int)sizeof(uint32_t);
    static_assert(kTile < 65536, "positions in a tile fit 16 bits");
};
constexpr uint32_t kFlagA = 1u << 30, kFlagP = 2u << 30, kValMask = (1u << 30) - 1;
constexpr int kMatchItems = 3;   // items of a lane ranked together
constexpr int kLookWindow = 4;   // predecessor tiles read per look-back step
constexpr int kHistWords = 3 * 1024;   // digit counts of every pass: 4 x 256 or up to 3 x 1024

// Digits of RB bits: DIG values, owned two at a time by the first kDigitThreads threads in
// the digit phases (two 16-bit counts are one word of shared memory, two look-back words
// one 8-byte access).
template <int RB>
struct Radix {
    static constexpr int DIG = 1 << RB;
    static constexpr uint32_t MASK = (uint32_t)DIG - 1u;
    static constexpr int kDigitThreads = DIG / 2;
    static constexpr int kDigitWarps = kDigitThreads / 32;
    static_assert(kDigitThreads <= SortShape<RB>::kThreads, "a thread per two digits");
};

// One pass over the keys counts every digit position: hist[pass][DIG].  A CTA per SM
// counts into shared memory, where every lane has counters of its own (a word of lane l in
// bank l), so that neither equal digits nor digits of one bank make a warp's additions wait
// for one another: with counters shared by the lanes an addition took 3.5 cycles of the
// shared-memory pipe on random keys and 32 on equal ones.  10-bit digits have two counters
// to a word (three passes of words of their own are 384 KB), which go to the global
// histogram before one of 16 bits can overflow: after kHistFlush rounds of 512 keys per
// lane.  The passes are a constant because the instructions bound this kernel next: a shift,
// a mask and an addition per digit.
// 16.8M keys, four digits: 33 us with shared counters, 17.6 now.
constexpr int kHistThreads = 1024, kHistFlush = 96;
template <int RB>
constexpr int kHistPair = RB == 8 ? 1 : 2;   // counters per word
template <int RB, int PASSES>
constexpr int kHistSmem = PASSES * Radix<RB>::DIG / kHistPair<RB> * 32 * (int)sizeof(uint32_t);
template <int RB, int PASSES>
__global__ void __launch_bounds__(kHistThreads, 1) k_radix_histogram(const uint32_t* __restrict__ keys, int64_t n,
                                                                     uint32_t* __restrict__ hist) {
    using R = Radix<RB>;
    constexpr int PAIR = kHistPair<RB>, ROWS = R::DIG / PAIR, words = PASSES * ROWS;
    extern __shared__ __align__(16) uint32_t s_h[];
    const int lane = threadIdx.x & 31;
    const auto clear = [&] {
        for (int i = threadIdx.x; i < words * 8; i += kHistThreads)
            reinterpret_cast<uint4*>(s_h)[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
    };
    const auto count = [&](uint32_t k) {
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            // byte offset: 128 * (row of the digit) + 4 * lane
            constexpr int down = PAIR - 1 - 7;
            const int s = RB * p + down;
            const uint32_t row = (s >= 0 ? k >> (s & 31) : k << (-s & 31)) & (uint32_t)((ROWS - 1) << 7);
            uint32_t* w = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(s_h) + p * ROWS * 128 + (row | lane << 2));
            atomicAdd(w, PAIR == 2 && (k >> (RB * p) & 1u) ? 0x10000u : 1u);
        }
    };
    const auto flush = [&] {
        __syncthreads();
        for (int w = threadIdx.x; w < words; w += kHistThreads) {
            uint32_t lo = 0, hi = 0;
#pragma unroll 8
            for (int l = 0; l < 32; ++l) {
                const uint32_t c = s_h[w * 32 + ((w + l) & 31)];
                lo += PAIR == 2 ? c & 0xffffu : c;
                if (PAIR == 2) hi += c >> 16;
            }
            if (lo) atomicAdd(&hist[PAIR * w], lo);
            if (hi) atomicAdd(&hist[PAIR * w + 1], hi);
        }
        __syncthreads();
    };
    clear();
    const int64_t stride = (int64_t)gridDim.x * kHistThreads;
    const int64_t t0 = blockIdx.x * (int64_t)kHistThreads + threadIdx.x;
    // 16-byte loads where the pointer allows them; the head before the first 16-byte
    // boundary and the tail after the last whole quad take single loads
    const int head = (int)((16 - ((uintptr_t)keys & 15)) & 15) / 4;
    const int64_t h = head < n ? head : n;
    const uint4* q = reinterpret_cast<const uint4*>(keys + h);
    const int64_t nq = ((uintptr_t)keys & 3) ? 0 : (n - h) / 4;
    int since = 0;   // rounds since the last flush (the same in every thread)
    for (int64_t base = 0; base < nq; base += 4 * stride) {
        if (PAIR == 2 && since++ == kHistFlush) {
            flush();
            clear();
            since = 1;
        }
        uint4 a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (base + u * stride + t0 < nq) a[u] = __ldg(q + base + u * stride + t0);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (base + u * stride + t0 < nq) {
                count(a[u].x); count(a[u].y); count(a[u].z); count(a[u].w);
            }
    }
    // at most 3 + 3 keys, or the whole of a list whose pointer is not a multiple of 4
    const int64_t done = nq > 0 ? h + 4 * nq : 0;
    if (nq > 0 && t0 < h) count(keys[t0]);
    for (int64_t base = done; base < n; base += stride) {
        if (PAIR == 2 && since++ == kHistFlush) {
            flush();
            clear();
            since = 1;
        }
        if (base + t0 < n) count(keys[base + t0]);
    }
    flush();
}

// the lanes of `mask` whose digit agrees with d in bits LO..HI-1, by a ballot per bit
template <int LO, int HI>
__device__ __forceinline__ unsigned match_bits(uint32_t d, unsigned mask) {
#pragma unroll
    for (int b = LO; b < HI; ++b) {
        const bool bit = (d >> b) & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, bit);
        mask &= bit ? bal : ~bal;
    }
    return mask;
}
// N positions in a tile, two to a register (indexes are constants after unrolling)
template <int N>
struct Positions {
    uint32_t p[(N + 1) / 2];
    __device__ __forceinline__ void set(int i, uint32_t v) {
        p[i / 2] = __byte_perm(p[i / 2], v, i & 1 ? 0x5410 : 0x3254);
    }
    __device__ __forceinline__ uint32_t get(int i) const { return i & 1 ? p[i / 2] >> 16 : p[i / 2] & 0xffffu; }
};

// One onesweep pass.  Warp w of a tile owns keys [w*32*IT, (w+1)*32*IT) of the tile
// in a warp-striped layout (item j of lane l is key j*32 + l), so processing items in
// order and lanes in order is index order: the ranks are stable.
// Bound by shared-memory accesses (63-70 % of their pipe; the arithmetic at 26 %): each
// scattered one costs 3.3 wavefronts per warp (32 random digits on 32 banks).  So the
// tile's digit counts come out of the ranking instead of a pass of atomics of their own,
// one atomic of a group's leader reads and advances the warp's count, and the values
// travel through registers, loaded before the look-back and staged after it.  Equal digits
// are found by words of lane bits; ballots take 10 wavefronts fewer and 50 instructions
// more per 32 keys: 548 us for 16.8M pairs of 32 bits against 460.  Three items are ranked
// together, so that the chain of an item (bits, read, count, shuffle) has company.
// A pass over 16.8M pairs: 116 us before, 95 now.
template <int RB>
__global__ void __launch_bounds__(SortShape<RB>::kThreads, SortShape<RB>::kMinBlocks) k_onesweep(const uint32_t* __restrict__ kin,
                                                           const uint32_t* __restrict__ vin,
                                                           uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                           int64_t n, int shift, const uint32_t* __restrict__ bins,
                                                           uint32_t* __restrict__ look, unsigned int* tile_counter,
                                                           int* err, uint32_t* __restrict__ cell_count,
                                                           uint32_t ncells, const uint32_t* __restrict__ count) {
    using R = Radix<RB>;
    constexpr int kThreads = SortShape<RB>::kThreads, kItems = SortShape<RB>::kItems;
    constexpr int kTile = SortShape<RB>::kTile;
    constexpr int kWarps = SortShape<RB>::kWarps;
    constexpr int DIG = R::DIG;
    // per warp and digit, two digits to a word: the warp's count, then the tile-local
    // position of the warp's first key of that digit
    __shared__ uint32_t s_warp_hist[kWarps][DIG / 2];
    __shared__ uint32_t s_delta[DIG];        // global start minus tile-local start of each digit
    __shared__ uint32_t s_w[R::kDigitWarps];
    __shared__ uint32_t s_hw[R::kDigitWarps];
    extern __shared__ uint32_t s_staging[];  // keys, values in tile-sorted order
    uint32_t* s_keys = s_staging;
    uint32_t* s_vals = s_staging + kTile;
    __shared__ uint32_t s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
    for (int i = threadIdx.x; i < kWarps * DIG / 2; i += kThreads) (&s_warp_hist[0][0])[i] = 0;
    // ranking: per warp and value of a digit's low 8 bits, the lanes holding it (in the
    // keys' staging area, which is free until the staging step)
    static_assert(kItems % kMatchItems == 0 && kMatchItems * kWarps * 256 <= 2 * kTile, "match words fit in the staging area");
    uint32_t* s_match = s_staging + warp * kMatchItems * 256;
    for (int i = threadIdx.x; i < kMatchItems * kWarps * 256; i += kThreads) s_staging[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t tbase = (int64_t)tile * kTile;
    if (count) {      // the list may be shorter than the launch; no tile waits for a later one
        n = *count;
        if (tbase >= n) return;
    }
    const int64_t wbase = tbase + (int64_t)warp * 32 * kItems;
    // a tile with every key in range needs no tests of the items
    const auto run = [&](auto all) {
        constexpr bool FULL = decltype(all)::value;
        // item j of this lane is in range iff j * 32 < rem
        const int64_t rem64 = n - (wbase + lane);
        const int rem = FULL ? kTile : rem64 < kTile ? (int)rem64 : kTile;
        uint32_t key[kItems];
        Positions<kItems> pos;
#pragma unroll
        for (int j = 0; j < kItems; ++j) key[j] = j * 32 < rem ? kin[wbase + j * 32 + lane] : 0xffffffffu;
        // warp-level ranking (stable): the lowest lane of each group of equal digits adds the
        // group to the warp's count of the digit, and the count before it comes back to the
        // whole group by one shuffle
        const unsigned lt = (1u << lane) - 1u;
        uint32_t* hist = s_warp_hist[warp];
#pragma unroll
        for (int j0 = 0; j0 < kItems; j0 += kMatchItems) {
            uint32_t d[kMatchItems], prior[kMatchItems];
            unsigned peers[kMatchItems];
            bool ok[kMatchItems];
#pragma unroll
            for (int u = 0; u < kMatchItems; ++u) {
                ok[u] = (j0 + u) * 32 < rem;
                d[u] = (key[j0 + u] >> shift) & R::MASK;
                if (ok[u]) atomicOr(&s_match[u * 256 + (d[u] & 255u)], 1u << lane);
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < kMatchItems; ++u)
                peers[u] = ok[u] ? s_match[u * 256 + (d[u] & 255u)] : 0u;
            __syncwarp();
#pragma unroll
            for (int u = 0; u < kMatchItems; ++u) {
                // cleared for the next items
                if (ok[u] && lane == __ffs(peers[u]) - 1) s_match[u * 256 + (d[u] & 255u)] = 0u;
                peers[u] = match_bits<8, RB>(d[u], peers[u]);
                prior[u] = 0;
                if (ok[u] && lane == __ffs(peers[u]) - 1)
                    prior[u] = atomicAdd(&hist[d[u] >> 1], (uint32_t)__popc(peers[u]) << ((d[u] & 1u) * 16)) >>
                               ((d[u] & 1u) * 16);
                __syncwarp();
            }
#pragma unroll
            for (int u = 0; u < kMatchItems; ++u) {
                const int leader = ok[u] ? __ffs(peers[u]) - 1 : lane;
                pos.set(j0 + u, (__shfl_sync(0xffffffffu, prior[u], leader) & 0xffffu) + __popc(peers[u] & lt));
            }
        }
        __syncthreads();
        // digit thread t owns digits 2t and 2t + 1: the tile's counts of them, published so that
        // the look-back of later tiles can pass over this one
        const bool digit_thread = threadIdx.x < R::kDigitThreads;
        const int w0 = threadIdx.x, d0 = 2 * threadIdx.x;
        uint64_t* lk = reinterpret_cast<uint64_t*>(look) + (size_t)tile * (DIG / 2) + w0;
        const auto pair = [](uint32_t flag, uint32_t a, uint32_t b) {
            return (uint64_t)(flag | (b & kValMask)) << 32 | (flag | (a & kValMask));
        };
        // exclusive scan over the digit threads: within the warp here, the warps' totals in tot
        const auto scan = [&](uint32_t mine, uint32_t* tot) {
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) tot[warp] = incl;
            return incl - mine;
        };
        uint32_t count0 = 0, count1 = 0, first = 0, excl0 = 0, excl1 = 0;
        if (digit_thread) {
            uint32_t c = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) c += s_warp_hist[w][w0];
            count0 = c & 0xffffu;
            count1 = c >> 16;
            if (tile > 0) st_relaxed_u64(lk, pair(kFlagA, count0, count1));
            first = scan(count0 + count1, s_w);
            // tile 0 alone scans the pass's digit counts into the digits' global starts and
            // publishes start + its own count as its inclusive prefix, so every later tile's
            // look-back sum already holds its digit's global start
            if (tile == 0) {
                const uint32_t b0 = bins[d0], b1 = bins[d0 + 1];
                excl0 = scan(b0 + b1, s_hw);
                excl1 = excl0 + b0;
            }
        }
        __syncthreads();
        if (digit_thread) {
            for (int w = 0; w < warp; ++w) first += s_w[w];
            // the start of each warp's keys of the two digits, in place of the warp's counts
            uint32_t run = first | (first + count0) << 16;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = s_warp_hist[w][w0];
                s_warp_hist[w][w0] = run;
                run += c;
            }
            if (tile == 0) {
                for (int w = 0; w < warp; ++w) {
                    excl0 += s_hw[w];
                    excl1 += s_hw[w];
                }
            }
        }
        __syncthreads();
        // stage the keys in tile-sorted order; the values are on their way during the look-back
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            if (j * 32 < rem) {
                const uint32_t d = (key[j] >> shift) & R::MASK;
                const uint32_t q = pos.get(j) + ((hist[d >> 1] >> ((d & 1u) * 16)) & 0xffffu);
                pos.set(j, q);
                s_keys[q] = key[j];
                key[j] = vin ? vin[wbase + j * 32 + lane] : (uint32_t)(wbase + j * 32 + lane);
            }
        }
        // look back for the prefix of the two digits: kLookWindow tiles at a time, summing the
        // counts up to and including the nearest inclusive prefix (a tile publishes both digits'
        // words in one store, so both reach it together)
        if (digit_thread) {
            if (tile > 0) {
                int64_t t = (int64_t)tile - 1;
                uint32_t spins = 0;
                bool done = false;
                while (!done) {
                    uint64_t w[kLookWindow];
                    bool ready = true;
#pragma unroll
                    for (int j = 0; j < kLookWindow; ++j) {
                        w[j] = t - j >= 0 ? ld_volatile_u64(lk - (size_t)(tile - (t - j)) * (DIG / 2)) : pair(kFlagP, 0, 0);
                        ready = ready && ((uint32_t)w[j] & ~kValMask) != 0;
                    }
                    if (!ready) {
                        if (++spins > kSpinLimit) {
                            atomicExch(err, 1);
                            break;
                        }
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < kLookWindow; ++j) {
                        if (!done) {
                            excl0 += (uint32_t)w[j] & kValMask;
                            excl1 += (uint32_t)(w[j] >> 32) & kValMask;
                            done = ((uint32_t)w[j] & ~kValMask) == kFlagP;
                        }
                    }
                    t -= kLookWindow;
                }
            }
            st_relaxed_u64(lk, pair(kFlagP, excl0 + count0, excl1 + count1));
            s_delta[d0] = excl0 - first;
            s_delta[d0 + 1] = excl1 - (first + count0);
        }
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (j * 32 < rem) s_vals[pos.get(j)] = key[j];
        __syncthreads();
        const int valid = FULL ? kTile : (int)(n - tbase);
        if (!cell_count) {
#pragma unroll (FULL ? 5 : 1)
            for (int i = threadIdx.x; i < valid; i += kThreads) {
                const uint32_t k = s_keys[i];
                const uint32_t g = s_delta[(k >> shift) & R::MASK] + (uint32_t)i;
                kout[g] = k;
                vout[g] = s_vals[i];
            }
            return;
        }
        // last pass with cell counts: the staged keys are the tile's keys in full order, so
        // a warp's 32 consecutive keys form a few runs of equal cells; the last lane of each
        // run adds the run's length (whole warps step together for the shuffles)
        for (int b = threadIdx.x - lane; b < valid; b += kThreads) {
            const int i = b + lane;
            const bool ok = i < valid;
            const uint32_t k = ok ? s_keys[i] : 0xffffffffu;
            if (ok) {
                const uint32_t g = s_delta[(k >> shift) & R::MASK] + (uint32_t)i;
                kout[g] = k;
                vout[g] = s_vals[i];
            }
            const uint32_t prev = __shfl_up_sync(0xffffffffu, k, 1);
            const uint32_t next = __shfl_down_sync(0xffffffffu, k, 1);
            const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || k != prev);
            if (ok && k < ncells && (lane == 31 || k != next)) {
                const int first = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
                atomicAdd(&cell_count[k], (uint32_t)(lane - first + 1));
            }
        }
    };
    if (n - tbase >= kTile) run(std::true_type());
    else run(std::false_type());
}

// ---- small lists ----------------------------------------------------------------
// Up to 8192 pairs in one CTA: LSD passes of 5-bit digits between registers and shared
// memory, so that a sort of a short list is one launch instead of a clear, a histogram and a
// kernel per 8-bit digit, whose latencies add up (4096 pairs, 10-bit keys: 23 us a call, now 12,
// 9 of them the kernel).
// A warp owns 32 ITEMS consecutive pairs; five ballots give each lane the lanes that share
// its item's digit and the count of the digit whose number it bears, so a lane keeps one
// digit's running count in a register.  The counts of all warps (32 x 32, digit-major) are
// scanned once per pass.
constexpr int kSmallThreads = 1024, kSmallMax = 8 * kSmallThreads;
template <int ITEMS>
__global__ void __launch_bounds__(kSmallThreads) k_sort_small(const uint32_t* __restrict__ kin,
                                                              const uint32_t* __restrict__ vin,
                                                              uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                              int n, int key_bits, int* __restrict__ err) {
    extern __shared__ uint32_t s_pairs[];                     // keys, then values
    __shared__ uint32_t s_count[32 * 32], s_warp[32];
    uint32_t* s_k = s_pairs;
    uint32_t* s_v = s_pairs + ITEMS * kSmallThreads;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int base = warp * 32 * ITEMS + lane;
    if (threadIdx.x == 0) *err = 0;
    uint32_t key[ITEMS], val[ITEMS], pos[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = base + 32 * j;
        key[j] = i < n ? kin[i] : 0xffffffffu;      // past the end: digit 31 of every pass, after the rest
        val[j] = i < n ? vin[i] : 0u;
    }
    for (int shift = 0; shift < key_bits; shift += 5) {
        const uint32_t mask = key_bits - shift >= 5 ? 31u : (1u << (key_bits - shift)) - 1u;
        uint32_t mine = 0;                          // pairs of digit `lane` so far in this warp
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t d = base + 32 * j < n || shift > 0 ? (key[j] >> shift) & mask : mask;
            uint32_t peers = 0xffffffffu, own = 0xffffffffu;
#pragma unroll
            for (int b = 0; b < 5; ++b) {
                const uint32_t bal = __ballot_sync(0xffffffffu, (d >> b) & 1u);
                peers &= (d >> b) & 1u ? bal : ~bal;
                own &= (lane >> b) & 1 ? bal : ~bal;
            }
            pos[j] = __shfl_sync(0xffffffffu, mine, (int)d) + __popc(peers & ((1u << lane) - 1u));
            mine += __popc(own);
        }
        s_count[lane * 32 + warp] = mine;
        __syncthreads();
        // exclusive scan in (digit, warp) order: thread 32 d + w holds digit d of warp w
        const uint32_t c = s_count[threadIdx.x];
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t before = lane < warp ? s_warp[lane] : 0u;
        before = __reduce_add_sync(0xffffffffu, before);
        s_count[threadIdx.x] = before + incl - c;
        __syncthreads();
        const uint32_t start = s_count[lane * 32 + warp];      // of digit `lane` in this warp
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t d = base + 32 * j < n || shift > 0 ? (key[j] >> shift) & mask : mask;
            const uint32_t p = pos[j] + __shfl_sync(0xffffffffu, start, (int)d);
            s_k[p] = key[j];
            s_v[p] = val[j];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            key[j] = s_k[base + 32 * j];
            val[j] = s_v[base + 32 * j];
        }
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = base + 32 * j;
        if (i < n) {
            kout[i] = key[j];
            vout[i] = val[j];
        }
    }
}

// Cell starts and counts of a short list over few cells in one CTA: a histogram in shared
// memory and its scan, instead of two clears, a histogram and a scan.
constexpr int64_t kSmallCells = 16384, kSmallKeys = 32768;
__global__ void __launch_bounds__(kSmallThreads) k_cells_small(const uint32_t* __restrict__ keys, int n, int ncells,
                                                               uint32_t* __restrict__ start,
                                                               uint32_t* __restrict__ count, int* __restrict__ err) {
    extern __shared__ uint32_t s_cells[];          // kSmallThreads * per words
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (ncells + kSmallThreads - 1) / kSmallThreads;
    if (threadIdx.x == 0) *err = 0;
    for (int c = threadIdx.x; c < per * kSmallThreads; c += kSmallThreads) s_cells[c] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSmallThreads) {
        const uint32_t k = keys[i];
        if (k < (uint32_t)ncells) atomicAdd(&s_cells[k], 1u);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < ncells; c += kSmallThreads) count[c] = s_cells[c];
    uint32_t sum = 0;
    for (int q = 0; q < per; ++q) sum += s_cells[threadIdx.x * per + q];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t run = __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u) + incl - sum;
    for (int q = 0; q < per; ++q) {
        const int c = threadIdx.x * per + q;
        const uint32_t k = s_cells[c];
        s_cells[c] = run;
        run += k;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < ncells; c += kSmallThreads) start[c] = s_cells[c];
}

// Counts per cell.  Equal neighbours within a warp are added as one run (the keys come
// sorted, so a warp holds a few runs): the last lane of each run adds its length.
__global__ void k_histogram_cells(const uint32_t* __restrict__ keys, int64_t n, uint32_t ncells,
                                  uint32_t* __restrict__ count) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; base < n; base += stride) {
        const int64_t i = base + lane;
        const uint32_t k = i < n ? keys[i] : 0xffffffffu;   // past the end: no cell
        const uint32_t prev = __shfl_up_sync(0xffffffffu, k, 1);
        const uint32_t next = __shfl_down_sync(0xffffffffu, k, 1);
        const unsigned starts = __ballot_sync(0xffffffffu, lane == 0 || k != prev);
        const bool last = lane == 31 || k != next;
        if (last && k < ncells) {
            const int first = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
            atomicAdd(&count[k], (uint32_t)(lane - first + 1));
        }
    }
}

__global__ void k_left_right(const uint32_t* __restrict__ start, const uint32_t* __restrict__ count, int64_t ncells,
                             uint32_t* __restrict__ left, uint32_t* __restrict__ right) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < ncells;
         c += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t s = start[c], k = count[c];
        left[c] = s;
        right[c] = k ? s + k - 1 : s;
    }
}

inline unsigned grid_cap(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 16) b = 148 * 16;
    return (unsigned)b;
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

size_t scan_scratch_bytes(int64_t n) {
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    return (size_t)(2 + tiles) * sizeof(uint64_t);
}

// Scans of more than one tile per SM stream (us, look-back -> stream: 2^22 values 14.7 ->
// 13.7, 2^24 47 -> 35, 2^27 325 -> 187; below, both wait for the launch), where the pointers
// are 16-byte aligned as the bulk copies want them.
constexpr int64_t kStreamMinTiles = 64;

cudaError_t scan_exclusive_u32(const uint32_t* in, uint32_t* out, int64_t n, void* scratch, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles > 1) {
        cudaError_t e = cudaMemsetAsync(scratch, 0, scan_scratch_bytes(n), st);
        if (e != cudaSuccess) return e;
    }
    const int vec = (((uintptr_t)in | (uintptr_t)out) & 15u) == 0 ? 1 : 0;
    if (vec && tiles > kStreamMinTiles) {
        int dev = 0, sms = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k_scan_stream, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem);
        if (e != cudaSuccess) return e;
        if (tiles > sms) {
            k_scan_stream<<<sms, kStreamThreads, kStreamSmem, st>>>(in, out, n, (uint64_t*)scratch, (uint32_t)tiles);
            return cudaGetLastError();
        }
    }
    k_scan_exclusive<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, (uint64_t*)scratch, vec, (uint32_t)tiles);
    return cudaGetLastError();
}

int scan_error_flag_offset() { return 8; }   // byte offset of the error word inside the scan scratch

SortLayout sort_layout(int64_t n, int key_bits) {
    SortLayout L{};
    if (key_bits < 1) key_bits = 1;
    if (key_bits > 32) key_bits = 32;
    const int p8 = (key_bits + 7) / 8, p10 = (key_bits + 9) / 10;
    // 10-bit digits where they save a pass (17-20 and 25-30 key bits)
    L.digit_bits = (key_bits > 16 && key_bits <= 30 && p10 < p8) ? 10 : 8;
    L.passes = L.digit_bits == 10 ? p10 : p8;
    const int tile = L.digit_bits == 10 ? SortShape<10>::kTile : SortShape<8>::kTile;
    L.tiles = (n + tile - 1) / tile;
    size_t off = 0;
    L.off_hist = off;    off += align256(sizeof(uint32_t) * kHistWords);
    L.off_counters = off; off += align256(sizeof(uint32_t) * 8);     // tile counters [4], error word [4]
    // look-back words for the widest layout (4 passes x 256 digits of SortShape<8>'s tiles, or
    // 3 x 1024 of SortShape<10>'s), so that the scratch size does not depend on key_bits
    const int64_t t8 = (n + SortShape<8>::kTile - 1) / SortShape<8>::kTile;
    const int64_t t10 = (n + SortShape<10>::kTile - 1) / SortShape<10>::kTile;
    const int64_t look_words = std::max<int64_t>(std::max<int64_t>(4 * 256 * t8, 3 * 1024 * t10), 3 * 1024);
    L.off_look = off;    off += align256(sizeof(uint32_t) * (size_t)look_words);
    L.off_alt_keys = off; off += align256(sizeof(uint32_t) * (size_t)(n > 0 ? n : 1));
    L.off_alt_vals = off; off += align256(sizeof(uint32_t) * (size_t)(n > 0 ? n : 1));
    L.bytes = off;
    return L;
}

cudaError_t radix_sort_begin(int64_t n, int key_bits, void* scratch, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const SortLayout L = sort_layout(n, key_bits);
    cudaError_t e = L.digit_bits == 10
                        ? cudaFuncSetAttribute(k_onesweep<10>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               SortShape<10>::kStagingBytes)
                        : cudaFuncSetAttribute(k_onesweep<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               SortShape<8>::kStagingBytes);
    if (e != cudaSuccess) return e;
    return cudaMemsetAsync(scratch, 0,
                           L.off_look + sizeof(uint32_t) * ((size_t)1 << L.digit_bits) * (size_t)L.tiles * L.passes, st);
}

uint32_t* radix_sort_hist(int64_t n, int key_bits, void* scratch) {
    return (uint32_t*)((char*)scratch + sort_layout(n, key_bits).off_hist);
}

cudaError_t radix_sort_finish(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, int64_t n,
                              int key_bits, void* scratch, cudaStream_t st, uint32_t* cell_count, int64_t ncells,
                              const uint32_t* count) {
    if (n <= 0) return cudaSuccess;
    const SortLayout L = sort_layout(n, key_bits);
    const int rb = L.digit_bits, dig = 1 << rb;
    char* base = (char*)scratch;
    uint32_t* hist = (uint32_t*)(base + L.off_hist);
    uint32_t* counters = (uint32_t*)(base + L.off_counters);
    uint32_t* look = (uint32_t*)(base + L.off_look);
    uint32_t* ak = (uint32_t*)(base + L.off_alt_keys);
    uint32_t* av = (uint32_t*)(base + L.off_alt_vals);
    // ping-pong so that the last pass lands in (kout, vout)
    const uint32_t* sk = kin;
    const uint32_t* sv = vin;
    for (int p = 0; p < L.passes; ++p) {
        const bool to_out = ((L.passes - 1 - p) % 2) == 0;
        uint32_t* dk = to_out ? kout : ak;
        uint32_t* dv = to_out ? vout : av;
        uint32_t* lp = look + (size_t)dig * L.tiles * p;
        uint32_t* cc = p == L.passes - 1 ? cell_count : nullptr;
        if (rb == 10)
            k_onesweep<10><<<(unsigned)L.tiles, SortShape<10>::kThreads, SortShape<10>::kStagingBytes, st>>>(
                sk, sv, dk, dv, n, rb * p, hist + dig * p, lp, counters + p, (int*)(counters + 4), cc,
                (uint32_t)ncells, count);
        else
            k_onesweep<8><<<(unsigned)L.tiles, SortShape<8>::kThreads, SortShape<8>::kStagingBytes, st>>>(
                sk, sv, dk, dv, n, rb * p, hist + dig * p, lp, counters + p, (int*)(counters + 4), cc,
                (uint32_t)ncells, count);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        sk = dk;
        sv = dv;
    }
    return cudaSuccess;
}

static cudaError_t sort_small(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, int n,
                              int key_bits, int* err, cudaStream_t st) {
    const auto launch = [&](auto kernel, int items) -> cudaError_t {
        const int smem = 2 * items * kSmallThreads * (int)sizeof(uint32_t);
        if (smem > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
        }
        kernel<<<1, kSmallThreads, smem, st>>>(kin, vin, kout, vout, n, key_bits, err);
        return cudaGetLastError();
    };
    if (n <= kSmallThreads) return launch(k_sort_small<1>, 1);
    if (n <= 2 * kSmallThreads) return launch(k_sort_small<2>, 2);
    if (n <= 4 * kSmallThreads) return launch(k_sort_small<4>, 4);
    return launch(k_sort_small<8>, 8);
}

cudaError_t radix_sort_pairs_u32(const uint32_t* kin, const uint32_t* vin, uint32_t* kout, uint32_t* vout, int64_t n,
                                 int key_bits, void* scratch, cudaStream_t st, uint32_t* cell_count, int64_t ncells) {
    if (n <= 0) return cudaSuccess;
    const SortLayout L = sort_layout(n, key_bits);
    if (n <= kSmallMax && !cell_count)
        return sort_small(kin, vin, kout, vout, (int)n, key_bits, (int*)((char*)scratch + L.off_counters) + 4, st);
    cudaError_t e = radix_sort_begin(n, key_bits, scratch, st);
    if (e != cudaSuccess) return e;
    uint32_t* hist = radix_sort_hist(n, key_bits, scratch);
    const unsigned hb = (unsigned)std::min<int64_t>((n + 16 * kHistThreads - 1) / (16 * kHistThreads), 148);
    const auto histogram = [&](auto kernel, int smem) -> cudaError_t {
        cudaError_t a = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (a != cudaSuccess) return a;
        kernel<<<hb, kHistThreads, smem, st>>>(kin, n, hist);
        return cudaGetLastError();
    };
    if (L.digit_bits == 10)
        e = L.passes == 2 ? histogram(k_radix_histogram<10, 2>, kHistSmem<10, 2>)
                          : histogram(k_radix_histogram<10, 3>, kHistSmem<10, 3>);
    else
        e = L.passes == 1   ? histogram(k_radix_histogram<8, 1>, kHistSmem<8, 1>)
            : L.passes == 2 ? histogram(k_radix_histogram<8, 2>, kHistSmem<8, 2>)
            : L.passes == 3 ? histogram(k_radix_histogram<8, 3>, kHistSmem<8, 3>)
                            : histogram(k_radix_histogram<8, 4>, kHistSmem<8, 4>);
    if (e != cudaSuccess) return e;
    return radix_sort_finish(kin, vin, kout, vout, n, key_bits, scratch, st, cell_count, ncells);
}

cudaError_t cell_counts_u32(const uint32_t* sorted_keys, int64_t n, int64_t ncells, uint32_t* count, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(uint32_t) * (size_t)ncells, st);
    if (e != cudaSuccess) return e;
    if (n > 0) k_histogram_cells<<<grid_cap(n, 256), 256, 0, st>>>(sorted_keys, n, (uint32_t)ncells, count);
    return cudaGetLastError();
}

cudaError_t cell_offsets_u32(const uint32_t* sorted_keys, int64_t n, int64_t ncells, uint32_t* start, uint32_t* count,
                             void* scan_scratch, cudaStream_t st) {
    if (n <= kSmallKeys && ncells <= kSmallCells) {
        const int smem = (int)((ncells + kSmallThreads - 1) / kSmallThreads * kSmallThreads * sizeof(uint32_t));
        if (smem > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(k_cells_small, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
        }
        k_cells_small<<<1, kSmallThreads, smem, st>>>(sorted_keys, (int)n, (int)ncells, start, count,
                                                      (int*)scan_scratch + 2);
        return cudaGetLastError();
    }
    cudaError_t e = cell_counts_u32(sorted_keys, n, ncells, count, st);
    if (e != cudaSuccess) return e;
    return scan_exclusive_u32(count, start, ncells, scan_scratch, st);
}

cudaError_t left_right_u32(const uint32_t* start, const uint32_t* count, int64_t ncells, uint32_t* left,
                           uint32_t* right, cudaStream_t st) {
    k_left_right<<<grid_cap(ncells, 256), 256, 0, st>>>(start, count, ncells, left, right);
    return cudaGetLastError();
}

}  // namespace gpgmp

// ---- exclusive scan without allocation -----------------------------------------
// For callers that must not call cudaMalloc: the scan's scratch (tile counter,
// error word, one status word per 16384-value tile) lives in a fixed file-scope
// device array instead of a caller buffer.  Every device that loads this library
// holds the array (32 KiB) until the process exits; it serves scans of up to
// kNoAllocMaxN values.
namespace gpgmp {
namespace {
constexpr int64_t kNoAllocMaxN = (int64_t)1 << 26;
constexpr size_t kNoAllocWords = 2 + (size_t)(kNoAllocMaxN / kScanTile);
static __device__ __align__(256) uint64_t g_noalloc_scan_scratch[kNoAllocWords];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_addr[kNoAllocMaxDevices] = {};

// Device address of the array on the current device.  In host code the array's
// name only stands in for the symbol, so the address comes from
// cudaGetSymbolAddress, once per device, with that device current.
int noalloc_scratch(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return set_error(GPGMP_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return set_error(GPGMP_ERR_UNSUPPORTED, "device %d", dev);
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scan_scratch);
        if (e != cudaSuccess || !p)
            return set_error(GPGMP_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_noalloc_addr[dev] = p;
    }
    *out = g_noalloc_addr[dev];
    return GPGMP_OK;
}
}  // namespace
}  // namespace gpgmp

extern "C" int gpgmp_exclusive_scan_u32_noalloc(const uint32_t* in, uint32_t* out, int64_t n, void* stream) {
    using namespace gpgmp;
    if (n < 0 || (n > 0 && (!in || !out))) return set_error(GPGMP_ERR_INVALID, "bad argument");
    if (n > kNoAllocMaxN)
        return set_error(GPGMP_ERR_INVALID, "n = %lld exceeds the %lld values the built-in scratch serves",
                         (long long)n, (long long)kNoAllocMaxN);
    if (n == 0) return GPGMP_OK;
    void* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    // zeroes the counter, the error word and the status words this scan uses, then scans
    cudaError_t e = scan_exclusive_u32(in, out, n, scratch, (cudaStream_t)stream);
    if (e != cudaSuccess) return set_error(GPGMP_ERR_CUDA, "scan: %s", cudaGetErrorString(e));
    return GPGMP_OK;
}

// Waits for `stream` and reads the error word of the built-in scratch: GPGMP_ERR_TIMEOUT
// in *status when the last scan's look-back gave up (its output is then wrong).  The
// next no-allocation scan clears the word, so this is read before it.
extern "C" int gpgmp_exclusive_scan_u32_noalloc_status(void* stream, int32_t* status) {
    using namespace gpgmp;
    if (!status) return set_error(GPGMP_ERR_INVALID, "bad argument");
    void* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    if (e != cudaSuccess) return set_error(GPGMP_ERR_CUDA, "cudaStreamSynchronize: %s", cudaGetErrorString(e));
    uint32_t word = 0;
    e = cudaMemcpy(&word, (const char*)scratch + scan_error_flag_offset(), sizeof(word), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return set_error(GPGMP_ERR_CUDA, "cudaMemcpy: %s", cudaGetErrorString(e));
    *status = word ? GPGMP_ERR_TIMEOUT : GPGMP_OK;
    return GPGMP_OK;
}
