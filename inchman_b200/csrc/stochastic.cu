// Wide kernels of the stochastic and reference-compatible deterministic solvers.
// One launch covers every realisation of a solver (grid z or the flattened
// index runs over realisations); the host event loop drives them.
//
// Compiled with -fmad=false: the sampling code must round exactly as its CPU
// replay does.
#include <cstdio>
#include <utility>
#include "kernels.h"
#include "stoch_device.cuh"

namespace gpgmp {

namespace {

constexpr int kIncMinReactions = 6;   // networks above this size keep per-reaction hazards
constexpr int NT = 256;               // threads of a diffusion tile block

// Launch shapes the autotuner chooses from (GridDesc::tile, GridDesc::ssa_threads; the
// drift-diffusion sweeps have one shape):
// diffusion tiles of TW x TH cells for 256 threads (1, 2 or 4 cells per thread in the
// gather; the one-cell halo is recomputed, so wider tiles recompute less), and SSA
// blocks of 64, 128 or 256 threads (one cell per thread).  Every draw is keyed by its
// cell, so all shapes give the same bits.
constexpr int kTileW[kNumDiffusionTiles] = {32, 32, 64, 16, 64, 32};
constexpr int kTileH[kNumDiffusionTiles] = {16, 8, 8, 16, 16, 32};
constexpr int kSsaThreadChoices[kNumSsaThreadChoices] = {128, 64, 256};

// n / d for n < 2^31 by one multiplication: with s = ceil(log2 d) and m = ceil(2^(31+s) / d)
// < 2^32 the error of m is below 2^s, so n m / 2^(31+s) exceeds n / d by less than 1 / d
// (Granlund & Montgomery 1994).
struct FastDiv {
    uint32_t d, m;
    int s;
    __host__ explicit FastDiv(uint32_t div) : d(div), m(0), s(0) {
        while ((1ull << s) < d) ++s;
        m = (uint32_t)((((1ull << 31) << s) + d - 1) / d);
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const {
        return (uint32_t)(((uint64_t)n * m) >> (31 + s));
    }
};

// realisation and cell of index i of all the cells (a 64-bit division costs as much as a
// random block, so it is left to totals of 2^31 cells and more)
__device__ __forceinline__ void split_cell(int64_t i, int64_t total, const FastDiv& area, int* r, int* c) {
    *r = total < ((int64_t)1 << 31) ? (int)area((uint32_t)i) : (int)(i / area.d);
    *c = (int)(i - (int64_t)*r * area.d);
}

__global__ void k_init_poisson(Planes planes, int S, FastDiv area_div, int R, uint32_t seed,
                               const float* __restrict__ lam) {
    const int area = (int)area_div.d;
    const int64_t total = (int64_t)R * area;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        int r, c;
        split_cell(i, total, area_div, &r, &c);
        for (int s = 0; s < S; ++s) {
            Stream st;
            st.init(seed, (uint32_t)r, 0u, (uint32_t)c, PH_INIT | ((uint32_t)s << 8));
            planes.p[s][((int64_t)r * S + s) * area + c] = poisson(st, lam[s]);
        }
    }
}

// MASKED: localised reactions, rmask as GridDesc::rmask (the unmasked form is the
// same code with every reaction on)
template <bool MASKED, int kSsaThreads>
__global__ void __launch_bounds__(kSsaThreads) k_ssa(Planes planes, int S, int area, int R,
                                                     const gpgmp_reaction* __restrict__ reactions, int nreac,
                                                     uint32_t seed, uint32_t step_seed, float window,
                                                     int32_t* __restrict__ status,
                                                     const uint32_t* __restrict__ rmask, int rmask_words) {
    extern __shared__ __align__(16) unsigned char smem[];
    gpgmp_reaction* rt = reinterpret_cast<gpgmp_reaction*>(smem);
    uint32_t* deps = reinterpret_cast<uint32_t*>(smem + sizeof(gpgmp_reaction) * nreac);
    float* hs = reinterpret_cast<float*>(deps + 4 * nreac);
    int* xs = reinterpret_cast<int*>(hs + (size_t)nreac * kSsaThreads);
    for (int i = threadIdx.x; i < nreac; i += blockDim.x) rt[i] = reactions[i];
    __syncthreads();
    build_deps(rt, nreac, deps);
    const int64_t total = (int64_t)R * area;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int r = (int)(i / area);
    const int c = (int)(i - (int64_t)r * area);
    int* x = xs + threadIdx.x;
    for (int s = 0; s < S; ++s) x[s * kSsaThreads] = planes.p[s][((int64_t)r * S + s) * area + c];
    Stream st;
    st.init(seed, (uint32_t)r, step_seed, (uint32_t)c, PH_SSA);
    // both forms give the same bits; the incremental one pays off for larger networks
    int e;
    if (MASKED) {
        CellReactions on;
        on.load(rmask, rmask_words, area, c);
        e = nreac > kIncMinReactions ? ssa_cell_inc(rt, deps, nreac, x, kSsaThreads, hs + threadIdx.x, st, window, on)
                                     : ssa_cell_h(rt, nreac, x, kSsaThreads, st, window,
                                                  GatedHazard<MassActionHazard>{MassActionHazard{}, on});
    } else {
        e = nreac > kIncMinReactions ? ssa_cell_inc(rt, deps, nreac, x, kSsaThreads, hs + threadIdx.x, st, window)
                                     : ssa_cell(rt, nreac, x, kSsaThreads, st, window);
    }
    for (int s = 0; s < S; ++s) planes.p[s][((int64_t)r * S + s) * area + c] = x[s * kSsaThreads];
    if (e) atomicOr(&status[r], e);
}

// The same windows for a network in the packed form: NR reactions as kernel parameters,
// their running sums in registers (ssa_small), or any number in shared memory (ssa_packed).
template <int NR, int kSsaThreads>
__global__ void __launch_bounds__(kSsaThreads) k_ssa_small(Planes planes, int S, FastDiv area_div, int R,
                                                           const gpgmp_reaction* __restrict__ reactions,
                                                           const __grid_constant__ SmallNet<NR> net, uint32_t seed,
                                                           uint32_t step_seed, float window,
                                                           int32_t* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint4 s_net[NR];
    if (threadIdx.x < NR) s_net[threadIdx.x] = net.net[threadIdx.x];
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int area = (int)area_div.d;
    const int64_t total = (int64_t)R * area;
    if (i >= total) return;
    int r, c;
    split_cell(i, total, area_div, &r, &c);
    const int64_t first = (int64_t)r * S * area + c;
    const auto at = [&](int s) -> int32_t& { return planes.p[s][first + (int64_t)s * area]; };
    Stream st;
    st.init(seed, (uint32_t)r, step_seed, (uint32_t)c, PH_SSA);
    const int e = packed_window<kSsaThreads>(
        reactions, NR, at, S, reinterpret_cast<float*>(smem) + threadIdx.x, st, window,
        [&](float* x, Stream& q, SsaPos& pos) { return ssa_small<NR, kSsaThreads>(net, s_net, x, q, window, pos); });
    if (e) atomicOr(&status[r], e);
}

template <int kSsaThreads>
__global__ void __launch_bounds__(kSsaThreads) k_ssa_packed(Planes planes, int S, FastDiv area_div, int R,
                                                            const gpgmp_reaction* __restrict__ reactions, int nreac,
                                                            const PackedReaction* __restrict__ packed, int nnet,
                                                            uint32_t seed, uint32_t step_seed, float window,
                                                            int32_t* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smem[];
    float4* ent = reinterpret_cast<float4*>(smem);
    uint4* nets = reinterpret_cast<uint4*>(ent + nreac);
    float* cs = reinterpret_cast<float*>(nets + nreac);
    float* xs = cs + (size_t)nreac * kSsaThreads;
    packed_tables<kSsaThreads>(packed, nreac, ent, nets);
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int area = (int)area_div.d;
    const int64_t total = (int64_t)R * area;
    if (i >= total) return;
    int r, c;
    split_cell(i, total, area_div, &r, &c);
    const int64_t first = (int64_t)r * S * area + c;
    const auto at = [&](int s) -> int32_t& { return planes.p[s][first + (int64_t)s * area]; };
    Stream st;
    st.init(seed, (uint32_t)r, step_seed, (uint32_t)c, PH_SSA);
    const int e = packed_window<kSsaThreads>(
        reactions, nreac, at, S, xs + threadIdx.x, st, window, [&](float* x, Stream& q, SsaPos& pos) {
            return ssa_packed<kSsaThreads>(ent, nets, nnet, nreac, x, cs + threadIdx.x, q, window, pos);
        });
    if (e) atomicOr(&status[r], e);
}

// 2-D homogeneous jumps.  A block owns a TW x TH tile, samples the lost counts of the tile
// and of its one-cell halo (recomputed, the streams are keyed by cell) into shared memory,
// then gathers.  Reads `in`, writes `out`: no block reads what another writes.
template <int TW, int TH>
__global__ void __launch_bounds__(NT) k_diffuse_tile(const int* __restrict__ in, int* __restrict__ out, int W, int H,
                                                     int S, int species, uint32_t seed, uint32_t step_seed,
                                                     float pmove, int4 bm4) {
    constexpr int RW = TW + 2, RH = TH + 2;
    __shared__ int s_lost[RH * RW * 4];
    __shared__ int s_n[TH * TW];
    const int area = W * H;
    const int r = blockIdx.z;
    const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;
    const int64_t plane = ((int64_t)r * S + species) * area;
    const int bm[4] = {bm4.x, bm4.y, bm4.z, bm4.w};
    const uint32_t phase = PH_DIFF | ((uint32_t)species << 8);
    BinomialSetup<7> jump;
    jump.init(pmove);
    for (int i = threadIdx.x; i < RW * RH; i += NT) {
        const int lx = i % RW, ly = i / RW;
        const int gx = x0 + lx - 1, gy = y0 + ly - 1;
        int l[4] = {0, 0, 0, 0};
        if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
            const int c = gy * W + gx;
            const int n = in[plane + c];
            Stream st;
            st.init(seed, (uint32_t)r, step_seed, (uint32_t)c, phase);
            homog_lost(n, jump, st, gx, gy, W, H, bm, l);
            if (lx >= 1 && lx < 1 + TW && ly >= 1 && ly < 1 + TH) s_n[(ly - 1) * TW + (lx - 1)] = n;
        }
#pragma unroll
        for (int d = 0; d < 4; ++d) s_lost[i * 4 + d] = l[d];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < TW * TH; i += NT) {
        const int lx = i % TW, ly = i / TW;
        const int gx = x0 + lx, gy = y0 + ly;
        if (gx >= W || gy >= H) continue;
        const int o = (ly + 1) * RW + (lx + 1);
        int v = s_n[i];
        v -= s_lost[o * 4] + s_lost[o * 4 + 1] + s_lost[o * 4 + 2] + s_lost[o * 4 + 3];
        if (gx > 0) v += s_lost[(o - 1) * 4 + 1];
        if (gx < W - 1) v += s_lost[(o + 1) * 4 + 0];
        if (gy > 0) v += s_lost[(o - RW) * 4 + 3];
        if (gy < H - 1) v += s_lost[(o + RW) * 4 + 2];
        out[plane + gy * W + gx] = v;
    }
}

// Drift-diffusion sweep in x (DIR 0) or y (DIR 1), written out of place.  A thread owns one
// cell of a 32 x 8 (x) or 8 x 32 (y) tile, works out its probabilities and draw set-ups
// once and samples it in up to kSweepReal realisations; the tile is 32 cells long in the
// sweep's direction so that its 16 halo cells, sampled again here, are 1/16 of the work,
// and one barrier serves all the realisations.  Issue slots bound it (the random block and
// the two searches), not its 8 bytes per cell:
// 8.4M cells 140 us (67 MB; 198 us with one realisation and one set-up per cell and tile,
// whose quarter-tile of halo rows was sampled again).  tall: the grid's first dimension, which
// alone may exceed 65535, counts the rows of tiles instead of the columns.
constexpr int kSweepReal = 8;
template <int DIR>
__global__ void __launch_bounds__(NT, 4) k_sweep(const int* __restrict__ in, int* __restrict__ out, int W, int H, int S,
                                              int R, int species, uint32_t seed, uint32_t step_seed, int wall_lo,
                                              int wall_hi, const float* __restrict__ Df, const float* __restrict__ rf,
                                              float dt, float dx, int fpe, int tall) {
    constexpr int TW = DIR == 0 ? 32 : 8, TH = DIR == 0 ? 8 : 32;
    constexpr int LINE = 34;                       // cells along the sweep with both halo cells
    constexpr int STEP = DIR == 0 ? 1 : TW;        // to the next cell along the sweep
    constexpr int CELLS = LINE * 8;
    static_assert(TW * TH == NT && CELLS == NT + 16, "a thread per cell and 16 halo cells");
    __shared__ int s_minus[kSweepReal][CELLS], s_plus[kSweepReal][CELLS], s_kept[kSweepReal][NT];
    const int64_t area = (int64_t)W * H;
    const int r0 = blockIdx.z * kSweepReal;
    const int nr = min(kSweepReal, R - r0);
    const int x0 = (tall ? blockIdx.y : blockIdx.x) * TW, y0 = (tall ? blockIdx.x : blockIdx.y) * TH;
    const uint32_t phase = PH_DIFF | ((uint32_t)species << 8) | (uint32_t)(DIR + 1);
    const int64_t plane0 = ((int64_t)r0 * S + species) * area, plane_step = (int64_t)S * area;
    const auto set_up = [&](SweepCell& cell, int gx, int gy) {
        const int64_t fi = (int64_t)species * area + (int64_t)gy * W + gx;
        const int p = DIR == 0 ? gx : gy, last = (DIR == 0 ? W : H) - 1;
        cell.init(Df[fi], rf[fi], dt, dx, p == 0 && wall_lo == 0, p == last && wall_hi == 0, fpe != 0);
    };
    // the halo: cell i & 1 ? after : before the tile's line i >> 1, of realisation h >> 4
    for (int h = threadIdx.x; h < 16 * nr; h += NT) {
        const int i = h & 15, k = h >> 4, line = i >> 1, after = i & 1;
        const int gx = x0 + (DIR == 0 ? (after ? TW : -1) : line);
        const int gy = y0 + (DIR == 0 ? line : (after ? TH : -1));
        int minus = 0, plus = 0;
        if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
            SweepCell cell;
            set_up(cell, gx, gy);
            const int c = gy * W + gx;
            Stream st;
            st.init(seed, (uint32_t)(r0 + k), step_seed, (uint32_t)c, phase);
            cell.draw(in[plane0 + k * plane_step + c], st, &minus, &plus);
        }
        const int o = DIR == 0 ? line * LINE + (after ? TW + 1 : 0) : (after ? TH + 1 : 0) * TW + line;
        s_minus[k][o] = minus;
        s_plus[k][o] = plus;
    }
    const int lx = threadIdx.x % TW, ly = threadIdx.x / TW;
    const int gx = x0 + lx, gy = y0 + ly;
    const int o = DIR == 0 ? ly * LINE + lx + 1 : (ly + 1) * TW + lx;
    const bool own = gx < W && gy < H;
    const int c = gy * W + gx;
    if (own) {
        SweepCell cell;
        set_up(cell, gx, gy);
        int next = in[plane0 + c];
#pragma unroll 1
        for (int k = 0; k < nr; ++k) {
            const int n = next;
            if (k + 1 < nr) next = in[plane0 + (k + 1) * plane_step + c];
            Stream st;
            st.init(seed, (uint32_t)(r0 + k), step_seed, (uint32_t)c, phase);
            int minus, plus;
            cell.draw(n, st, &minus, &plus);
            s_minus[k][o] = minus;
            s_plus[k][o] = plus;
            s_kept[k][threadIdx.x] = n - minus - plus;
        }
    }
    __syncthreads();
    if (!own) return;
    const int p = DIR == 0 ? gx : gy, last = (DIR == 0 ? W : H) - 1;
    for (int k = 0; k < nr; ++k) {
        int v = s_kept[k][threadIdx.x];
        if (p > 0) v += s_plus[k][o - STEP];
        if (p < last) v += s_minus[k][o + STEP];
        out[plane0 + k * plane_step + c] = v;
    }
}

__global__ void k_source(int* plane_base, int W, int H, int S, int R, int species, uint32_t seed,
                         uint32_t step_seed, int boundary, int count, float pi) {
    const int total = R * W;
    const int area = W * H;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int r = i / W, dev = i % W;
        int gid;
        switch (boundary) {
            case 0: gid = dev * W; break;
            case 1: gid = (W - 1) + dev * W; break;
            case 2: gid = dev; break;
            default: gid = dev + (H - 1) * W; break;
        }
        if (gid >= area) continue;
        Stream st;
        st.init(seed, (uint32_t)r, step_seed, (uint32_t)gid,
                PH_SOURCE | ((uint32_t)species << 8) | (uint32_t)boundary);
        plane_base[((int64_t)r * S + species) * area + gid] += binomial(st, count, pi);
    }
}

__device__ __forceinline__ uint32_t float_key(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__global__ void k_timestep(int area, const float* __restrict__ D, const float* __restrict__ r, float dx,
                           uint32_t* min_key, int kind, float stay) {
    uint32_t best = 0xffffffffu;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < area; c += gridDim.x * blockDim.x)
    {
        const float ts = kind == kTsFpe             ? fpe_timestep(D[c], r[c], dx, stay)
                         : kind == kTsDeterministic ? det_timestep(D[c], r[c], dx)
                                                    : cell_timestep(D[c], r[c], dx);
        if (ts == ts) best = min(best, float_key(ts));   // NaN is skipped, as fminf does
    }
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0) atomicMin(min_key, best);
}

struct DriftParams { float p[8]; };

__global__ void k_diffusivity_drift(int W, int H, int species, int method, DriftParams prm, float L,
                                    float* dx, float* dy, float* rx, float* ry) {
    const int area = W * H;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < area; c += gridDim.x * blockDim.x) {
        const int x = c % W, y = c / W;
        const int64_t i = (int64_t)species * area + c;
        const float px = L / (float)W * ((float)x - (float)W * 0.5f);
        const float py = L / (float)H * ((float)y - (float)H * 0.5f);
        const float* p = prm.p;
        if (method == GPGMP_DRIFT_HOMOGENEOUS) {
            dx[i] = p[0]; dy[i] = p[1]; rx[i] = p[2]; ry[i] = p[3];
        } else if (method == GPGMP_DRIFT_MULTIPLICATIVE_NOISE) {
            const float sx = px + L, sy = py + L;
            dx[i] = (p[0] * p[0]) * (sx * sx) * 0.5f;
            dy[i] = (p[1] * p[1]) * (sy * sy) * 0.5f;
            rx[i] = p[2] * sx;
            ry[i] = p[3] * sy;
        } else if (method == GPGMP_DRIFT_ORNSTEIN_UHLENBECK) {
            dx[i] = p[0]; dy[i] = p[1];
            rx[i] = -(p[2] * px + p[3] * py);
            ry[i] = -(p[4] * px + p[5] * py);
        }
    }
}

// ---- deterministic, reference-compatible ------------------------------------
// Deterministic.cl:17-65 (mirror neighbours), written out of place.
__global__ void k_det_diffuse(const float* __restrict__ in, float* __restrict__ out, int W, int H, int S, int R,
                              const float* __restrict__ D, float dt, float dx2) {
    const int area = W * H;
    const int64_t total = (int64_t)R * S * area;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % area);
        const int s = (int)((i / area) % S);
        const int x = c % W, y = c / W;
        const float* p = in + (i - c);
        const float sl = x > 0 ? p[c - 1] : p[c + 1];
        const float sr = x < W - 1 ? p[c + 1] : p[c - 1];
        const float st = y > 0 ? p[c - W] : p[c + W];
        const float sb = y < H - 1 ? p[c + W] : p[c - W];
        const float sh = p[c];
        const float lap = st + sb + sl + sr - 4.0f * sh;
        out[i] = sh + dt * D[s] * lap / dx2;
    }
}

// Deterministic.cl:143-238: 20 classical RK4 substeps per window, clamp at 0.
__global__ void k_rk4(float* state, int S, int area, int R, const gpgmp_reaction* __restrict__ reactions, int nreac,
                      float deltat, const uint32_t* __restrict__ rmask, int rmask_words) {
    extern __shared__ unsigned char smem[];
    gpgmp_reaction* rt = reinterpret_cast<gpgmp_reaction*>(smem);
    float* buf = reinterpret_cast<float*>(smem + sizeof(gpgmp_reaction) * nreac);
    for (int i = threadIdx.x; i < nreac; i += blockDim.x) rt[i] = reactions[i];
    __syncthreads();
    const int64_t total = (int64_t)R * area;
    const int64_t gi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (gi >= total) return;
    const int r = (int)(gi / area), c = (int)(gi % area);
    const int B = blockDim.x;
    float* x = buf + threadIdx.x;           // [S] stride B
    float* k = buf + (size_t)S * B + threadIdx.x;   // 4 x [S]
    float* y = buf + (size_t)5 * S * B + threadIdx.x;
    float* sp = state + (int64_t)r * S * area + c;
    for (int s = 0; s < S; ++s) x[s * B] = sp[(int64_t)s * area];
    CellReactions on;           // localised reactions contribute nothing where they are off
    on.load(rmask, rmask_words, area, c);
    const int nmax = 20;
    const float h = deltat / (float)nmax;
    for (int it = 0; it < nmax; ++it) {
        for (int stage = 0; stage < 4; ++stage) {
            const float off = stage == 0 ? 0.0f : (stage == 3 ? h : 0.5f * h);
            float* kin = k + (size_t)(stage == 0 ? 0 : stage - 1) * S * B;
            float* kout = k + (size_t)stage * S * B;
            for (int s = 0; s < S; ++s) {
                y[s * B] = stage == 0 ? x[s * B] : x[s * B] + off * kin[s * B];
                kout[s * B] = 0.0f;
            }
            for (int q = 0; q < nreac; ++q) {
                if (!on(q)) continue;
                const gpgmp_reaction& rc = rt[q];
                float law = rc.rate;
                for (int j = 0; j < rc.num_reactants; ++j)
                    for (int m = 0; m < rc.reactant_stoich[j]; ++m) law *= y[rc.reactant_species[j] * B];
                for (int j = 0; j < rc.num_reactants; ++j)
                    kout[rc.reactant_species[j] * B] -= (float)rc.reactant_stoich[j] * law;
                for (int j = 0; j < rc.num_products; ++j)
                    kout[rc.product_species[j] * B] += (float)rc.product_stoich[j] * law;
            }
        }
        for (int s = 0; s < S; ++s) {
            float v = x[s * B] + h / 6.0f * (k[s * B] + 2.0f * k[(S + s) * B] + 2.0f * k[(2 * S + s) * B] +
                                              k[(3 * S + s) * B]);
            x[s * B] = v < 0.0f ? 0.0f : v;
        }
    }
    for (int s = 0; s < S; ++s) sp[(int64_t)s * area] = x[s * B];
}

// Deterministic.cl:71-136 (inhomogeneous drift-diffusion, one direction, one
// species, mirror neighbours): s' = s + dt (D_l s_l + D_r s_r - 2 D s) / dx^2
// - dt (r_r s_r - r_l s_l) / (2 dx), written out of place; the other species'
// planes are copied so that `out` is a whole state.
template <int DIR>
__global__ void k_det_sweep(const float* __restrict__ in, float* __restrict__ out, int W, int H, int S, int R,
                            int species, const float* __restrict__ D, const float* __restrict__ rv, float dt,
                            float dx) {
    const int area = W * H;
    const int64_t total = (int64_t)R * S * area;
    const float dx2 = dx * dx;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % area);
        const int s = (int)((i / area) % S);
        if (s != species) {
            out[i] = in[i];
            continue;
        }
        const int x = c % W, y = c / W;
        int lo, hi;
        if (DIR == 0) {
            lo = x > 0 ? c - 1 : c + 1;
            hi = x < W - 1 ? c + 1 : c - 1;
        } else {
            lo = y > 0 ? c - W : c + W;
            hi = y < H - 1 ? c + W : c - W;
        }
        const float* p = in + (i - c);
        const float* Dp = D + (int64_t)species * area;
        const float* rp = rv + (int64_t)species * area;
        const float sl = p[lo] * Dp[lo], sr = p[hi] * Dp[hi], sh = p[c] * Dp[c];
        const float lap = sl + sr - 2.0f * sh;
        const float drift = rp[hi] * p[hi] - rp[lo] * p[lo];
        out[i] = p[c] + dt * lap / dx2 - dt * drift / (2.0f * dx);
    }
}

// ---- alpha-QSS (Mott & Oran 2001), Deterministic.cl:240-522 ------------------------
constexpr int kAqssMaxSpecies = kMaxSpecies;
constexpr int kAqssMaxIter = 100000;    // corrector passes per cell and window before giving up

// production q and destruction d of every species: law = rate * prod x^nu
// (Reaction.cpp:145-162); a reaction adds |net| law to q (net > 0) or d (net < 0)
// of each species whose net stoichiometry it changes (Solver.cpp:961-1004)
__device__ __forceinline__ void aqss_rhs(const gpgmp_reaction* rt, int nreac, int S, const float* y, float* q,
                                         float* d, const CellReactions& on) {
    for (int i = 0; i < S; ++i) { q[i] = 0.0f; d[i] = 0.0f; }
    for (int k = 0; k < nreac; ++k) {
        if (!on(k)) continue;        // localised reaction, off in this cell
        const gpgmp_reaction& rc = rt[k];
        float law = rc.rate;
        for (int j = 0; j < rc.num_reactants; ++j)
            for (int m = 0; m < rc.reactant_stoich[j]; ++m) law *= y[rc.reactant_species[j]];
        // every species of the reaction once, in reactant-then-product order
        for (int pass = 0; pass < 2; ++pass) {
            const int cnt = pass == 0 ? rc.num_reactants : rc.num_products;
            for (int j = 0; j < cnt; ++j) {
                const int sp = pass == 0 ? rc.reactant_species[j] : rc.product_species[j];
                bool seen = false;
                for (int a = 0; a < rc.num_reactants && !seen; ++a)
                    if (rc.reactant_species[a] == sp && (pass == 1 || a < j)) seen = true;
                for (int a = 0; a < rc.num_products && !seen && pass == 1; ++a)
                    if (rc.product_species[a] == sp && a < j) seen = true;
                if (seen) continue;
                int net = 0;
                for (int a = 0; a < rc.num_products; ++a) if (rc.product_species[a] == sp) net += rc.product_stoich[a];
                for (int a = 0; a < rc.num_reactants; ++a) if (rc.reactant_species[a] == sp) net -= rc.reactant_stoich[a];
                if (net > 0) q[sp] += (float)net * law;
                else if (net < 0) d[sp] += (float)(-net) * law;
            }
        }
    }
}

__device__ __forceinline__ float aqss_alpha(float r) {
    return (180.0f + r * (60.0f + r * (11.0f + r))) / (360.0f + r * (60.0f + r * (12.0f + r)));
}

// One window of length dtg for the species x[0..S) of one cell.  A retried step
// restarts its predictor from the saved start state with the reduced step size
// (Mott & Oran's method).  literal: the reference's form instead -- the predictor
// takes the current production/destruction and the outer step's size
// (Deterministic.cl:381-387, which never shrinks on a retry, so a species growing
// from zero can be rejected forever) and the corrector coefficient as printed
// (`180.*+rtaub`, :424).  Returns GPGMP_SIM_EVENT_CAP if the step control did not
// finish within kAqssMaxIter passes.
__device__ int aqss_cell(const gpgmp_reaction* rt, int nreac, int S, float* y, float dtg, bool literal,
                         const CellReactions& on) {
    const float epsmin = 1e-2f, sqreps = 0.5f, epscl = 100.0f, epsmax = 10.0f, tfd = 1.000008f, dtmin = 1e-15f,
                ymin = 1e-20f;
    constexpr int itermax = 2;
    float q[kAqssMaxSpecies], d[kAqssMaxSpecies], ys[kAqssMaxSpecies], qs[kAqssMaxSpecies], ds[kAqssMaxSpecies],
        rtaus[kAqssMaxSpecies], scr[kAqssMaxSpecies], y1[kAqssMaxSpecies];
    float tn = 0.0f;
    for (int i = 0; i < S; ++i) y[i] = fmaxf(y[i], ymin);
    aqss_rhs(rt, nreac, S, y, q, d, on);
    float scrtch = 1e-25f;
    for (int i = 0; i < S; ++i) {
        const float ascr = fabsf(q[i]);
        const float scr2 = copysignf(1.0f / y[i], 0.1f * epsmin * ascr - d[i]);
        const float scr1 = scr2 * d[i];
        scrtch = fmaxf(fmaxf(scr1, -fabsf(ascr - d[i]) * scr2), scrtch);
    }
    float dt = fminf(sqreps / scrtch, dtg);
    int passes = 0;
    while (dtg > tn * tfd) {
        const float ts = tn;
        const float dtcurrent = dt;
        for (int i = 0; i < S; ++i) {
            ys[i] = y[i];
            qs[i] = q[i];
            ds[i] = d[i];
            rtaus[i] = dtcurrent * d[i] / y[i];
        }
        while (dtg > tn * tfd) {
            if (++passes > kAqssMaxIter) return GPGMP_SIM_EVENT_CAP;
            for (int i = 0; i < S; ++i) {
                if (literal) {
                    const float rtaui = dtcurrent * d[i] / y[i];
                    scr[i] = (q[i] - d[i]) / (1.0f + aqss_alpha(rtaui) * rtaui);
                } else {
                    const float rtaui = dt * ds[i] / ys[i];
                    scr[i] = (qs[i] - ds[i]) / (1.0f + aqss_alpha(rtaui) * rtaui);
                }
            }
            float eps = 1e-10f;
            for (int iteration = 0; iteration < itermax; ++iteration) {
                for (int i = 0; i < S; ++i) y[i] = fmaxf(ys[i] + dt * scr[i], ymin);
                if (iteration == 0) {
                    tn = ts + dt;
                    for (int i = 0; i < S; ++i) y1[i] = y[i];
                }
                aqss_rhs(rt, nreac, S, y, q, d, on);
                eps = 1e-10f;
                for (int i = 0; i < S; ++i) {
                    const float rtaub = 0.5f * (rtaus[i] + dt * d[i] / y[i]);
                    const float alpha =
                        literal ? (180.0f * rtaub * (60.0f + rtaub * (11.0f + rtaub))) /
                                      (360.0f + rtaub * (60.0f + rtaub * (12.0f + rtaub)))
                                : aqss_alpha(rtaub);
                    const float qt = qs[i] * (1.0f - alpha) + q[i] * alpha;
                    const float pb = rtaub / dt;
                    scr[i] = (qt - ys[i] * pb) / (1.0f + alpha * rtaub);
                }
            }
            for (int i = 0; i < S; ++i) {
                const float scr2 = fmaxf(ys[i] + dt * scr[i], 0.0f);
                float scr1 = fabsf(scr2 - y1[i]);
                y[i] = fmaxf(scr2, ymin);
                if (0.25f * (ys[i] + y[i]) > ymin) {
                    scr1 = scr1 / y[i];
                    eps = fmaxf(0.5f * (scr1 + fminf(fabsf(q[i] - d[i]) / (q[i] + d[i] + 1e-30f), scr1)), eps);
                }
            }
            eps = eps * epscl;
            if (dt <= dtmin + 1e-16f * tn) {
                dt = dtg - ts;
                dt = fminf(dtmin, fabsf(dt));
            }
            const float stab = 0.01f;     // the stability test needs itermax >= 3
            if (eps <= epsmax && stab <= 1.0f) {
                if (dtg <= tn * tfd) break;
            } else {
                tn = ts;
            }
            const float rteps = sqrtf(eps);
            float dto = dt;
            dt = fminf(fminf(dt * (1.0f / rteps + 0.005f), tfd * (dtg - tn)), dto / (stab + 0.001f));
            if (eps <= epsmax && stab <= 1.0f) break;
            dto = dt / dto;
            for (int i = 0; i < S; ++i) rtaus[i] *= dto;
        }
        aqss_rhs(rt, nreac, S, y, q, d, on);
    }
    return 0;
}

__global__ void k_aqss(float* state, int S, int area, int R, const gpgmp_reaction* __restrict__ reactions, int nreac,
                       float deltat, int literal, int32_t* status, const uint32_t* __restrict__ rmask,
                       int rmask_words) {
    extern __shared__ unsigned char smem[];
    gpgmp_reaction* rt = reinterpret_cast<gpgmp_reaction*>(smem);
    for (int i = threadIdx.x; i < nreac; i += blockDim.x) rt[i] = reactions[i];
    __syncthreads();
    const int64_t total = (int64_t)R * area;
    for (int64_t gi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; gi < total;
         gi += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(gi / area), c = (int)(gi % area);
        float* sp = state + (int64_t)r * S * area + c;
        float y[kAqssMaxSpecies];
        for (int s = 0; s < S; ++s) y[s] = sp[(int64_t)s * area];
        CellReactions on;
        on.load(rmask, rmask_words, area, c);
        const int e = aqss_cell(rt, nreac, S, y, deltat, literal != 0, on);
        for (int s = 0; s < S; ++s) sp[(int64_t)s * area] = y[s];
        if (e) atomicOr(&status[r], e);
    }
}

inline unsigned grid_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 64) b = 148 * 64;
    return (unsigned)b;
}

}  // namespace

cudaError_t launch_init_poisson(const GridDesc& g, Planes planes, uint32_t seed, const float* d_lambda,
                                cudaStream_t st) {
    const int area = g.W * g.H;
    k_init_poisson<<<grid_for((int64_t)g.R * area, 256), 256, 0, st>>>(planes, g.S, FastDiv(area), g.R, seed, d_lambda);
    return cudaGetLastError();
}

namespace {
template <class K>
cudaError_t allow_smem(K kernel, size_t smem) {
    return smem > 48 * 1024
               ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
               : cudaSuccess;
}
template <int NR, int NTH>
cudaError_t launch_ssa_small(const GridDesc& g, Planes planes, const gpgmp_reaction* d_reactions, const NetDesc& net,
                             uint32_t seed, uint32_t step_seed, float window, int32_t* d_status, cudaStream_t st) {
    const int area = g.W * g.H;
    const int64_t total = (int64_t)g.R * area;
    SmallNet<NR> sn;
    for (int q = 0; q < NR; ++q) {
        const PackedReaction& p = net.host[q];
        sn.rate[q] = p.rate;
        sn.sub[q] = p.sub;
        sn.o1[q] = p.s1 * NTH;
        sn.o2[q] = p.s2 * NTH;
        sn.net[q] = make_uint4(p.net[0], p.net[1], p.net[2], p.net[3]);
    }
    sn.nnet = net.nnet;
    const size_t smem = sizeof(float) * (g.S + 1) * NTH;
    k_ssa_small<NR, NTH><<<(unsigned)((total + NTH - 1) / NTH), NTH, smem, st>>>(
        planes, g.S, FastDiv(area), g.R, d_reactions, sn, seed, step_seed, window, d_status);
    return cudaGetLastError();
}
// The packed form where the network has one and every reaction is on everywhere; the
// table-driven form otherwise.  Up to kIncMinReactions reactions the running sums stay in
// registers, as in the table-driven form's own division: 47 us instead of its 78 for A + B
// <-> C on 1M cells; a larger network keeps them in shared memory, where the selection
// halves its range.
template <bool MASKED, int NTH>
cudaError_t launch_ssa_t(const GridDesc& g, Planes planes, const gpgmp_reaction* d_reactions, int nreac,
                         const NetDesc& net, uint32_t seed, uint32_t step_seed, float window, int32_t* d_status,
                         cudaStream_t st) {
    const int area = g.W * g.H;
    const int64_t total = (int64_t)g.R * area;
    const unsigned blocks = (unsigned)((total + NTH - 1) / NTH);
    if constexpr (!MASKED) {
        if (net.host) {
            switch (nreac) {
#define GPGMP_SMALL(N) \
    case N: return launch_ssa_small<N, NTH>(g, planes, d_reactions, net, seed, step_seed, window, d_status, st);
                GPGMP_SMALL(1)
                GPGMP_SMALL(2)
                GPGMP_SMALL(3)
                GPGMP_SMALL(4)
                GPGMP_SMALL(5)
                GPGMP_SMALL(6)
#undef GPGMP_SMALL
                default: break;
            }
            const size_t smem = (size_t)nreac * (sizeof(float4) + sizeof(uint4) + sizeof(float) * NTH) +
                                sizeof(float) * (g.S + 1) * NTH;
            cudaError_t e = allow_smem(k_ssa_packed<NTH>, smem);
            if (e != cudaSuccess) return e;
            k_ssa_packed<NTH><<<blocks, NTH, smem, st>>>(planes, g.S, FastDiv(area), g.R, d_reactions, nreac, net.dev, net.nnet,
                                                         seed, step_seed, window, d_status);
            return cudaGetLastError();
        }
    }
    const size_t smem = sizeof(gpgmp_reaction) * nreac + sizeof(uint32_t) * 4 * nreac +
                        sizeof(float) * (size_t)nreac * NTH + sizeof(int) * g.S * NTH;
    cudaError_t e = allow_smem(k_ssa<MASKED, NTH>, smem);
    if (e != cudaSuccess) return e;
    k_ssa<MASKED, NTH><<<blocks, NTH, smem, st>>>(planes, g.S, area, g.R, d_reactions, nreac, seed, step_seed, window,
                                                  d_status, g.rmask, g.rmask_words);
    return cudaGetLastError();
}
template <bool MASKED>
cudaError_t launch_ssa_m(const GridDesc& g, Planes planes, const gpgmp_reaction* d_reactions, int nreac,
                         const NetDesc& net, uint32_t seed, uint32_t step_seed, float window, int32_t* d_status,
                         cudaStream_t st) {
#define GPGMP_SSA(T) launch_ssa_t<MASKED, T>(g, planes, d_reactions, nreac, net, seed, step_seed, window, d_status, st)
    switch (kSsaThreadChoices[g.ssa_threads]) {
        case 64: return GPGMP_SSA(64);
        case 256: return GPGMP_SSA(256);
        default: return GPGMP_SSA(128);
    }
#undef GPGMP_SSA
}

template <int TW, int TH>
cudaError_t launch_tile_t(const GridDesc& g, const int32_t* in, int32_t* out, int species, uint32_t seed,
                          uint32_t step_seed, float pmove, cudaStream_t st) {
    dim3 grid((g.W + TW - 1) / TW, (g.H + TH - 1) / TH, g.R);
    const int4 bm = make_int4(g.bmask[0], g.bmask[1], g.bmask[2], g.bmask[3]);
    k_diffuse_tile<TW, TH><<<grid, NT, 0, st>>>(in, out, g.W, g.H, g.S, species, seed, step_seed, pmove, bm);
    return cudaGetLastError();
}

template <int DIR>
cudaError_t launch_sweep_t(const GridDesc& g, const int32_t* in, int32_t* out, int species, uint32_t seed,
                           uint32_t step_seed, const float* d_D, const float* d_r, float dt, float dx, int fpe,
                           cudaStream_t st) {
    constexpr int TW = DIR == 0 ? 32 : 8, TH = DIR == 0 ? 8 : 32;
    dim3 grid((g.W + TW - 1) / TW, (g.H + TH - 1) / TH, (g.R + kSweepReal - 1) / kSweepReal);
    const int tall = grid.y > 65535;      // then fewer than 2048 cells are a row: a grid has at most 2^30
    if (tall) std::swap(grid.x, grid.y);
    k_sweep<DIR><<<grid, NT, 0, st>>>(in, out, g.W, g.H, g.S, g.R, species, seed, step_seed, g.bmask[2 * DIR],
                                      g.bmask[2 * DIR + 1], d_D, d_r, dt, dx, fpe, tall);
    return cudaGetLastError();
}
}  // namespace

void diffusion_tile_shape(int index, int* w, int* h) {
    *w = kTileW[index];
    *h = kTileH[index];
}
int ssa_thread_choice(int index) { return kSsaThreadChoices[index]; }

cudaError_t launch_ssa(const GridDesc& g, Planes planes, const gpgmp_reaction* d_reactions, int nreac,
                       const NetDesc& net, uint32_t seed, uint32_t step_seed, float window, int32_t* d_status,
                       cudaStream_t st) {
    if (nreac <= 0) return cudaSuccess;
    return g.rmask ? launch_ssa_m<true>(g, planes, d_reactions, nreac, net, seed, step_seed, window, d_status, st)
                   : launch_ssa_m<false>(g, planes, d_reactions, nreac, net, seed, step_seed, window, d_status, st);
}

cudaError_t launch_homog_diffuse(const GridDesc& g, const int32_t* in, int32_t* out, int species, uint32_t seed,
                                 uint32_t step_seed, float pmove, cudaStream_t st) {
#define GPGMP_TILE(I)                                                                                         \
    case I:                                                                                                   \
        return launch_tile_t<kTileW[I], kTileH[I]>(g, in, out, species, seed, step_seed, pmove, st);
    switch (g.tile) {
        GPGMP_TILE(1)
        GPGMP_TILE(2)
        GPGMP_TILE(3)
        GPGMP_TILE(4)
        GPGMP_TILE(5)
        default: GPGMP_TILE(0)
    }
#undef GPGMP_TILE
}

cudaError_t launch_source(const GridDesc& g, int32_t* plane_base, int species, uint32_t seed, uint32_t step_seed,
                          int boundary, int count, float pi, cudaStream_t st) {
    k_source<<<grid_for((int64_t)g.R * g.W, 128), 128, 0, st>>>(plane_base, g.W, g.H, g.S, g.R, species, seed,
                                                                 step_seed, boundary, count, pi);
    return cudaGetLastError();
}

cudaError_t launch_sweep(const GridDesc& g, const int32_t* in, int32_t* out, int species, int sweep_y,
                         uint32_t seed, uint32_t step_seed, const float* d_D, const float* d_r, float dt, float dx,
                         cudaStream_t st, int fpe) {
    return sweep_y ? launch_sweep_t<1>(g, in, out, species, seed, step_seed, d_D, d_r, dt, dx, fpe, st)
                   : launch_sweep_t<0>(g, in, out, species, seed, step_seed, d_D, d_r, dt, dx, fpe, st);
}

cudaError_t launch_det_sweep(const GridDesc& g, const float* in, float* out, int species, int sweep_y,
                             const float* d_D, const float* d_r, float dt, float dx, cudaStream_t st) {
    const int64_t total = (int64_t)g.R * g.S * g.W * g.H;
    if (!sweep_y)
        k_det_sweep<0><<<grid_for(total, 256), 256, 0, st>>>(in, out, g.W, g.H, g.S, g.R, species, d_D, d_r, dt, dx);
    else
        k_det_sweep<1><<<grid_for(total, 256), 256, 0, st>>>(in, out, g.W, g.H, g.S, g.R, species, d_D, d_r, dt, dx);
    return cudaGetLastError();
}

cudaError_t launch_aqss(const GridDesc& g, float* state, const gpgmp_reaction* d_reactions, int nreac, float deltat,
                        int literal, int32_t* d_status, cudaStream_t st) {
    if (nreac <= 0) return cudaSuccess;
    const int area = g.W * g.H;
    const int64_t total = (int64_t)g.R * area;
    const int threads = 128;
    const size_t smem = sizeof(gpgmp_reaction) * nreac;
    k_aqss<<<grid_for(total, threads), threads, smem, st>>>(state, g.S, area, g.R, d_reactions, nreac, deltat, literal,
                                                             d_status, g.rmask, g.rmask_words);
    return cudaGetLastError();
}

cudaError_t launch_timestep(int area, const float* d_D, const float* d_r, float dx, uint32_t* d_min_key,
                            cudaStream_t st, int kind, float stay) {
    cudaError_t e = cudaMemsetAsync(d_min_key, 0xff, sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    k_timestep<<<grid_for(area, 256), 256, 0, st>>>(area, d_D, d_r, dx, d_min_key, kind, stay);
    return cudaGetLastError();
}

// inhomogeneous_computeMomentsX + reduceMomentsBlocks (StochasticInhomogeneousDriftDiffusion.cl:5-84)
// and getMeanX (helpers.cl:18-21): MeanX = L / W * (sum x n / sum n - W / 2) of one
// species plane, the sums taken exactly in 64-bit integers.
__global__ void k_moments_sum(const int32_t* __restrict__ plane, int W, int area, unsigned long long* sums) {
    unsigned long long mx = 0, n = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < area; c += gridDim.x * blockDim.x) {
        const long long v = plane[c] > 0 ? plane[c] : 0;
        mx += (unsigned long long)(v * (c % W));
        n += (unsigned long long)v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx += __shfl_xor_sync(0xffffffffu, mx, o);
        n += __shfl_xor_sync(0xffffffffu, n, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sums[0], mx);
        atomicAdd(&sums[1], n);
    }
}
__global__ void k_moments_finish(const unsigned long long* sums, int W, float L, float* meanx) {
    const float tmp = (float)sums[0] / (float)sums[1];
    *meanx = L / (float)W * (tmp - (float)W / 2.0f);
}

cudaError_t launch_moments(const int32_t* plane, int W, int H, float L, unsigned long long* d_sums, float* d_meanx,
                           cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(d_sums, 0, 2 * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    const int area = W * H;
    k_moments_sum<<<grid_for(area, 256), 256, 0, st>>>(plane, W, area, d_sums);
    k_moments_finish<<<1, 1, 0, st>>>(d_sums, W, L, d_meanx);
    return cudaGetLastError();
}

cudaError_t launch_diffusivity_drift(const GridDesc& g, int species, int method, const float* params, float L,
                                     float* dx, float* dy, float* rx, float* ry, cudaStream_t st) {
    DriftParams p;
    for (int i = 0; i < 8; ++i) p.p[i] = params[i];
    k_diffusivity_drift<<<grid_for((int64_t)g.W * g.H, 256), 256, 0, st>>>(g.W, g.H, species, method, p, L, dx, dy,
                                                                            rx, ry);
    return cudaGetLastError();
}

cudaError_t launch_det_diffuse(const GridDesc& g, const float* in, float* out, const float* d_D, float dt,
                               float dx2, cudaStream_t st) {
    const int64_t total = (int64_t)g.R * g.S * g.W * g.H;
    k_det_diffuse<<<grid_for(total, 256), 256, 0, st>>>(in, out, g.W, g.H, g.S, g.R, d_D, dt, dx2);
    return cudaGetLastError();
}

cudaError_t launch_rk4(const GridDesc& g, float* state, const gpgmp_reaction* d_reactions, int nreac, float deltat,
                       cudaStream_t st) {
    if (nreac <= 0) return cudaSuccess;
    const int threads = 64;
    const int area = g.W * g.H;
    const int64_t total = (int64_t)g.R * area;
    const size_t smem = sizeof(gpgmp_reaction) * nreac + sizeof(float) * 6 * g.S * threads;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_rk4, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k_rk4<<<(unsigned)((total + threads - 1) / threads), threads, smem, st>>>(state, g.S, area, g.R, d_reactions,
                                                                             nreac, deltat, g.rmask, g.rmask_words);
    return cudaGetLastError();
}

}  // namespace gpgmp
