// Tiled Gray-Scott forward kernel over the whole chip, any lattice side, float or double.
//
// The kernels that cut the lattice into row bands pay a hop between SMs in every step, and
// at most 64 SMs hold a 256^2 lattice.  Here the lattice is cut into tiles of at most 16 x
// 16 cells, one CTA each, and a CTA also keeps the 8 cells around its tile: 32 x 32 cells in
// the registers of four warps.  A cell that borders on what the CTA does not hold goes
// stale, one ring per step from the outside in, so after 8 steps exactly the tile is still
// right; then the CTAs swap the cells around their tiles through global memory.  Between
// swaps a step needs one barrier of four warps and no other SM.  The price is that 4 cells
// are computed for each one kept; what it buys is that a 256^2 lattice takes 256 CTAs, two
// per SM and more SMs than any cluster arrangement holds, and that one CTA computes while
// the other waits for its swap.
//
// A lane owns two adjacent columns of four rows (16 lanes a row, two row groups a warp):
// vertical neighbours inside the group are its own registers, the rows above and below come
// from shared memory, horizontal neighbours by shuffles inside the 16 lanes.  On even sides
// the two columns are one access where the caller's arrays are aligned for it.
//
// Swap: at every state 8 m each CTA writes its tile's values, packed with m into 64-bit words
// (a double as two words with half its bits each), to the exchange buffer and polls its
// neighbours' words until they carry m: no flag, no fence (a word is one single-copy atomic
// store).  The buffer alternates by the parity of m.  A CTA writes block m + 2 only after it
// has read the block m + 1 of every CTA within 8 cells, which those wrote after reading
// block m; as each reads exactly the cells within 8 of its tile, they are the ones that read
// its own words, and no word is overwritten before it has been read.  The host clears the
// buffer on the launching stream before each launch.  All CTAs must run at once: the launch
// is cooperative, and every wait is bounded (one that gives up writes NaN and sets
// g_gs_fwd_err).
//
// The update of a cell is that of the kernel it stands in for, bit for bit: gs_update's
// operations for the sides that have kernels of their own (FORM 0) and k_gs_forward's for
// the others (FORM 1).
//
// What bounds it is latency: a step takes 0.21 us with one CTA per SM and 0.31 with two, a
// swap 1.8 us (the words' way to L2 and back, twice), 0.23 a step.  us per step, before (one
// cell per iteration on one cluster) -> now, float32: 75^2 3.0 -> 0.69, 96^2 1.28 -> 0.46,
// 192^2 2.0 -> 0.50, 320^2 3.8 -> 0.75; float64: 96^2 1.43 -> 0.68, 256^2 2.0 -> 0.82.  At
// 256^2 float32 it takes 0.53, the four clusters of gs_mc.cuh 0.51: they keep that side.
//
// Included from gray_scott.cu after gs_mc.cuh.

constexpr int kTileGhost = 8, kTileCore = 16, kTileExt = kTileCore + 2 * kTileGhost;
constexpr int kTileWarps = 4;
constexpr uint32_t kTileWaitLimit = 1u << 22;

template <typename T>
struct TilePair;
template <>
struct TilePair<float> { using type = float2; };
template <>
struct TilePair<double> { using type = double2; };

// a value as exchange words: one for a float, two for a double
__device__ __forceinline__ uint64_t tile_pack(uint32_t bits, int m) { return ((uint64_t)(uint32_t)m << 32) | bits; }
__device__ __forceinline__ void tile_st(uint64_t* p, uint64_t w) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void tile_st(uint64_t* p, uint64_t a, uint64_t b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void tile_ld(const uint64_t* p, uint64_t* a) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(*a) : "l"(p) : "memory");
}
__device__ __forceinline__ void tile_ld(const uint64_t* p, uint64_t* a, uint64_t* b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(*a), "=l"(*b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool tile_is(uint64_t w, int m) { return (uint32_t)(w >> 32) == (uint32_t)m; }

// one value, and an aligned pair of values, to and from the words at p; reading tells
// whether all of them carry block m
__device__ __forceinline__ void tile_put(uint64_t* p, float v, int m) { tile_st(p, tile_pack(__float_as_uint(v), m)); }
__device__ __forceinline__ void tile_put(uint64_t* p, double v, int m) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    tile_st(p, tile_pack((uint32_t)b, m), tile_pack((uint32_t)(b >> 32), m));
}
__device__ __forceinline__ void tile_put(uint64_t* p, float2 v, int m) {
    tile_st(p, tile_pack(__float_as_uint(v.x), m), tile_pack(__float_as_uint(v.y), m));
}
__device__ __forceinline__ void tile_put(uint64_t* p, double2 v, int m) {
    tile_put(p, v.x, m);
    tile_put(p + 2, v.y, m);
}
__device__ __forceinline__ bool tile_get(const uint64_t* p, float* v, int m) {
    uint64_t w;
    tile_ld(p, &w);
    *v = __uint_as_float((uint32_t)w);
    return tile_is(w, m);
}
__device__ __forceinline__ bool tile_get(const uint64_t* p, double* v, int m) {
    uint64_t a, b;
    tile_ld(p, &a, &b);
    *v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
    return tile_is(a, m) && tile_is(b, m);
}
__device__ __forceinline__ bool tile_get(const uint64_t* p, float2* v, int m) {
    uint64_t a, b;
    tile_ld(p, &a, &b);
    *v = make_float2(__uint_as_float((uint32_t)a), __uint_as_float((uint32_t)b));
    return tile_is(a, m) && tile_is(b, m);
}
__device__ __forceinline__ bool tile_get(const uint64_t* p, double2* v, int m) {
    const bool x = tile_get(p, &v->x, m), y = tile_get(p + 2, &v->y, m);
    return x && y;
}

// first cell of tile i of p along a side of n cells (even for even n, so that a lane's two
// columns are an aligned pair in memory)
__device__ __forceinline__ int tile_first(int n, int i, int p) {
    return n % 2 == 0 ? 2 * (int)((int64_t)(n / 2) * i / p) : (int)((int64_t)n * i / p);
}

template <typename T>
struct TileCtx {
    using P = typename TilePair<T>::type;
    int n, lane, group;          // group: the row group (0..7), four rows each
    int gx[2], gy[4];            // lattice columns and rows of the lane's cells (periodic)
    bool cx[2], cy[4];           // whether they belong to the tile
    bool ex[2], ey[4];           // whether they are within 8 cells of it
    bool pair;                   // the two columns are an aligned pair in every array (the host's `pairs`)
    P* edges;                    // [parity][field][group][top / bottom][16 lanes]
    volatile int* failed;
    __device__ __forceinline__ P* edge(int par, int f, int g, int bottom) const {
        return edges + ((((par * 2 + f) * 8 + g) * 2 + bottom) * 16) + (lane & 15);
    }
    __device__ __forceinline__ void init(int side, int px, int py, int pairs, unsigned char* smem, volatile int* fail) {
        n = side;
        lane = threadIdx.x & 31;
        group = (int)(threadIdx.x >> 5) * 2 + (lane >> 4);
        const int bx = (int)blockIdx.x % px, by = (int)blockIdx.x / px;
        const int x0 = tile_first(n, bx, px), cw = tile_first(n, bx + 1, px) - x0;
        const int y0 = tile_first(n, by, py), ch = tile_first(n, by + 1, py) - y0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = 2 * (lane & 15) + i;
            gx[i] = ((x0 - kTileGhost + e) % n + n) % n;
            cx[i] = e >= kTileGhost && e < kTileGhost + cw;
            ex[i] = e < cw + 2 * kTileGhost;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e = group * 4 + r;
            gy[r] = ((y0 - kTileGhost + e) % n + n) % n;
            cy[r] = e >= kTileGhost && e < kTileGhost + ch;
            ey[r] = e < ch + 2 * kTileGhost;
        }
        pair = pairs != 0;
        edges = reinterpret_cast<P*>(smem);
        failed = fail;
        if (threadIdx.x == 0) *failed = 0;
    }
    __device__ __forceinline__ P load(const T* __restrict__ p, int r) const {
        const T* q = p + (size_t)gy[r] * n;
        if (pair) return *reinterpret_cast<const P*>(q + gx[0]);
        P v;
        v.x = q[gx[0]];
        v.y = q[gx[1]];
        return v;
    }
    __device__ __forceinline__ void store(T* __restrict__ p, int r, const P& v) const {
        if (!cy[r]) return;
        T* q = p + (size_t)gy[r] * n;
        if (pair) {
            if (cx[0]) *reinterpret_cast<P*>(q + gx[0]) = v;
            return;
        }
        if (cx[0]) q[gx[0]] = v.x;
        if (cx[1]) q[gx[1]] = v.y;
    }
    // the lane's edge rows into the shared copy of parity par, and the block's barrier.  The
    // copy's last readers are past: they read it before the barrier of the step before.  (A
    // barrier in two halves over mbarriers, with the rows that need no neighbour between
    // them, was slower: 0.59 us per step instead of 0.43 at 64^2.)
    __device__ __forceinline__ void put_edges(int par, const P (&u)[4], const P (&v)[4]) const {
        *edge(par, 0, group, 0) = u[0];
        *edge(par, 0, group, 1) = u[3];
        *edge(par, 1, group, 0) = v[0];
        *edge(par, 1, group, 1) = v[3];
        __syncthreads();
    }
    // swaps the cells around the tile at block m (see the file comment)
    __device__ __forceinline__ void swap(uint64_t* xbuf, int m, P (&u)[4], P (&v)[4]) const {
        constexpr int kWords = sizeof(T) / 4;
        const size_t plane = (size_t)n * n * kWords;
        uint64_t* base = xbuf + (size_t)(m & 1) * 2 * plane;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint64_t* q = base + ((size_t)gy[r] * n + gx[0]) * kWords;
            if (pair) {
                if (cy[r] && cx[0]) {
                    tile_put(q, u[r], m);
                    tile_put(q + plane, v[r], m);
                }
            } else {
                uint64_t* q1 = base + ((size_t)gy[r] * n + gx[1]) * kWords;
                if (cy[r] && cx[0]) {
                    tile_put(q, u[r].x, m);
                    tile_put(q + plane, v[r].x, m);
                }
                if (cy[r] && cx[1]) {
                    tile_put(q1, u[r].y, m);
                    tile_put(q1 + plane, v[r].y, m);
                }
            }
        }
        // rows still to come
        uint32_t want = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (ey[r] && ((ex[0] && !(cy[r] && cx[0])) || (ex[1] && !(cy[r] && cx[1])))) want |= 1u << r;
        uint32_t it = 0;
        while (want) {
            uint32_t next = want;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!(want & (1u << r))) continue;
                const uint64_t* q = base + ((size_t)gy[r] * n + gx[0]) * kWords;
                bool ok = true;
                if (pair) {
                    const bool a = tile_get(q, &u[r], m), b = tile_get(q + plane, &v[r], m);
                    ok = a && b;
                } else {
                    const uint64_t* q1 = base + ((size_t)gy[r] * n + gx[1]) * kWords;
                    if (ex[0] && !(cy[r] && cx[0])) {
                        const bool a = tile_get(q, &u[r].x, m), b = tile_get(q + plane, &v[r].x, m);
                        ok = a && b;
                    }
                    if (ex[1] && !(cy[r] && cx[1])) {
                        const bool a = tile_get(q1, &u[r].y, m), b = tile_get(q1 + plane, &v[r].y, m);
                        ok = ok && a && b;
                    }
                }
                if (ok) next &= ~(1u << r);
            }
            want = next;
            if (want && (*failed || ++it == kTileWaitLimit)) {
                *failed = 1;
                want = 0;
            }
        }
        __syncwarp();
    }
};

// k_gs_forward's update of one cell, expression for expression
template <typename T>
__device__ __forceinline__ void gs_update_plain(const GSArgs<T>& a, T uU, T uc, T uD, T uL, T uR, T vU, T vc, T vD, T vL,
                                                T vR, T* un, T* vn) {
    const T one = T(1), half = T(0.5), four = T(4);
    const T Fk = a.F + a.k;
    const T lu = uL + uR + uU + uD - four * uc;
    const T lv = vL + vR + vU + vD - four * vc;
    const T uvv = uc * vc * vc;
    const T adv_u = a.vx * (uR - uL) * half + a.vy * (uD - uU) * half;
    const T adv_v = a.vx * (vR - vL) * half + a.vy * (vD - vU) * half;
    *un = uc + a.dt * (a.Du * lu - adv_u - uvv + a.F * (one - uc));
    *vn = vc + a.dt * (a.Dv * lv - adv_v + uvv - Fk * vc);
}

template <typename T, int FORM>
struct TileCoef;
template <>
struct TileCoef<float, 0> : GSCoef2 {
    using GSCoef2::GSCoef2;
};
template <>
struct TileCoef<double, 0> : GSCoef<double> {
    using GSCoef<double>::GSCoef;
};
template <typename T>
struct TileCoef<T, 1> : GSArgs<T> {
    __device__ __forceinline__ explicit TileCoef(const GSArgs<T>& a) : GSArgs<T>(a) {}
};

// the next values of one pair of cells: the rows above, at and below, and the cells left of
// .x (l) and right of .y (r)
template <int DRIFT>
__device__ __forceinline__ void tile_update(const TileCoef<float, 0>& k, float2 uU, float2 uC, float2 uD, float ul,
                                            float ur, float2 vU, float2 vC, float2 vD, float vl, float vr, float2* un,
                                            float2* vn) {
    const float2 uh = make_float2(ul + uC.y, uC.x + ur), vh = make_float2(vl + vC.y, vC.x + vr);
    float2 ud = uh, vd = vh;
    if (DRIFT) {
        ud = make_float2(ul - uC.y, uC.x - ur);
        vd = make_float2(vl - vC.y, vC.x - vr);
    }
    gs_update2s<DRIFT>(k, uh, ud, uU, uC, uD, vh, vd, vU, vC, vD, un, vn);
}
template <int DRIFT>
__device__ __forceinline__ void tile_update(const TileCoef<double, 0>& k, double2 uU, double2 uC, double2 uD, double ul,
                                            double ur, double2 vU, double2 vC, double2 vD, double vl, double vr,
                                            double2* un, double2* vn) {
    gs_update<double>(k, uU.x, uC.x, uD.x, ul, uC.y, vU.x, vC.x, vD.x, vl, vC.y, &un->x, &vn->x);
    gs_update<double>(k, uU.y, uC.y, uD.y, uC.x, ur, vU.y, vC.y, vD.y, vC.x, vr, &un->y, &vn->y);
}
template <int DRIFT, typename T, typename P>
__device__ __forceinline__ void tile_update(const TileCoef<T, 1>& a, P uU, P uC, P uD, T ul, T ur, P vU, P vC, P vD, T vl,
                                            T vr, P* un, P* vn) {
    gs_update_plain<T>(a, uU.x, uC.x, uD.x, ul, uC.y, vU.x, vC.x, vD.x, vl, vC.y, &un->x, &vn->x);
    gs_update_plain<T>(a, uU.y, uC.y, uD.y, uC.x, ur, vU.y, vC.y, vD.y, vC.x, vr, &un->y, &vn->y);
}

// one step X -> Y of the lane's cells; the rows around the group are in the shared copy of
// parity par
template <int DRIFT, typename T, int FORM>
__device__ __forceinline__ void tile_step(const TileCtx<T>& c, const TileCoef<T, FORM>& k, int par,
                                          const typename TilePair<T>::type (&xu)[4],
                                          const typename TilePair<T>::type (&xv)[4],
                                          typename TilePair<T>::type (&yu)[4], typename TilePair<T>::type (&yv)[4]) {
    using P = typename TilePair<T>::type;
    const int up = (c.group + 7) & 7, dn = (c.group + 1) & 7;     // the outermost rows are stale anyway
    const P au = *c.edge(par, 0, up, 1), av = *c.edge(par, 1, up, 1);
    const P bu = *c.edge(par, 0, dn, 0), bv = *c.edge(par, 1, dn, 0);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const T ul = __shfl_up_sync(0xffffffffu, xu[r].y, 1, 16), ur = __shfl_down_sync(0xffffffffu, xu[r].x, 1, 16);
        const T vl = __shfl_up_sync(0xffffffffu, xv[r].y, 1, 16), vr = __shfl_down_sync(0xffffffffu, xv[r].x, 1, 16);
        tile_update<DRIFT>(k, r == 0 ? au : xu[r == 0 ? 0 : r - 1], xu[r], r == 3 ? bu : xu[r == 3 ? 3 : r + 1], ul, ur,
                           r == 0 ? av : xv[r == 0 ? 0 : r - 1], xv[r], r == 3 ? bv : xv[r == 3 ? 3 : r + 1], vl, vr,
                           &yu[r], &yv[r]);
    }
}

// (float: five CTAs per SM, so that the largest float32 sides fit at once)
template <typename T, int DRIFT, int FORM>
__global__ void __launch_bounds__(32 * kTileWarps, sizeof(T) == 4 ? 5 : 2)
    k_gs_forward_tile(GSArgs<T> a, const T* __restrict__ u0, const T* __restrict__ v0, T* __restrict__ uo,
                      T* __restrict__ vo, T* __restrict__ trace, int trace_every, uint64_t* __restrict__ xbuf, int px,
                      int py, int pairs) {
    using P = typename TilePair<T>::type;
    __shared__ __align__(16) unsigned char s_edges[2 * 2 * 8 * 2 * 16 * sizeof(P)];
    __shared__ int s_failed;
    TileCtx<T> c;
    c.init(a.n, px, py, pairs, s_edges, &s_failed);
    const TileCoef<T, FORM> k(a);
    const size_t nn = (size_t)a.n * a.n;
    P xu[4], xv[4], yu[4], yv[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        xu[r] = c.load(u0, r);
        xv[r] = c.load(v0, r);
    }
    c.put_edges(0, xu, xv);
    const int steps = a.steps;
    const int every = trace_every > 0 ? trace_every : 1;
    int until = 0;                 // steps to the next traced state
    T* tr = trace;
    const auto put_trace = [&](const P (&pu)[4], const P (&pv)[4]) {
        if (tr == nullptr) return;
        if (until == 0) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                c.store(tr, r, pu[r]);
                c.store(tr + nn, r, pv[r]);
            }
            tr += 2 * nn;
            until = every;
        }
        --until;
    };
    int s = 0;
    for (; s + 2 <= steps; s += 2) {      // X -> Y -> X
        put_trace(xu, xv);
        tile_step<DRIFT>(c, k, 0, xu, xv, yu, yv);
        c.put_edges(1, yu, yv);
        put_trace(yu, yv);
        tile_step<DRIFT>(c, k, 1, yu, yv, xu, xv);
        if ((s + 2) % kTileGhost == 0 && s + 2 < steps) c.swap(xbuf, (s + 2) / kTileGhost, xu, xv);
        c.put_edges(0, xu, xv);
    }
    if (s < steps) {
        put_trace(xu, xv);
        tile_step<DRIFT>(c, k, 0, xu, xv, yu, yv);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            xu[r] = yu[r];
            xv[r] = yv[r];
        }
    }
    __syncthreads();
    if (s_failed) {
        if (threadIdx.x == 0) atomicOr(&g_gs_fwd_err, 1);
        const T nan = (T)__int_as_float(0x7fc00000);
#pragma unroll
        for (int r = 0; r < 4; ++r) xu[r].x = xu[r].y = xv[r].x = xv[r].y = nan;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        c.store(uo, r, xu[r]);
        c.store(vo, r, xv[r]);
    }
}

// Adjoint of a segment on the same tiles, for the sides without a kernel of their own: the
// adjoint fields take the place of u and v in registers, edges and swaps, and the stored
// states of a step (the lane's four rows, the row above and the row below) come from L2 a
// step ahead.  Every cell of the window is updated, the parameter sums count the tile's own.
// The updates and the sums' terms are k_gs_adjoint's, expression for expression; the sums
// are in double, so their order over the tiles changes nothing that the result shows.
// A gradient of 2,000 steps, with k_gs_adjoint -> now: float32 75^2 16.6 -> 5.5 ms, 96^2 5.9 ->
// 4.8, 192^2 10.0 -> 5.2; float64 24^2 5.15 -> 4.9, 96^2 6.3 -> 5.1, 160^2 9.2 -> 5.6.
template <typename T>
__global__ void __launch_bounds__(32 * kTileWarps, sizeof(T) == 4 ? 3 : 2)
    k_gs_adjoint_tile(GSArgs<T> k, const T* __restrict__ states, int len, const T* __restrict__ lu_in,
                      const T* __restrict__ lv_in, T* __restrict__ lu_out, T* __restrict__ lv_out,
                      double* __restrict__ grad, int* __restrict__ err, uint64_t* __restrict__ xbuf, int px, int py,
                      int pairs) {
    using P = typename TilePair<T>::type;
    __shared__ __align__(16) unsigned char s_edges[2 * 2 * 8 * 2 * 16 * sizeof(P)];
    __shared__ int s_failed;
    __shared__ double s_red[6][kTileWarps];
    TileCtx<T> c;
    c.init(k.n, px, py, pairs, s_edges, &s_failed);
    const size_t nn = (size_t)k.n * k.n;
    const int above = c.gy[0] == 0 ? k.n - 1 : c.gy[0] - 1, below = c.gy[3] == k.n - 1 ? 0 : c.gy[3] + 1;
    const auto row = [&](const T* p, int y) {
        const T* q = p + (size_t)y * k.n;
        if (c.pair) return *reinterpret_cast<const P*>(q + c.gx[0]);
        P v;
        v.x = q[c.gx[0]];
        v.y = q[c.gx[1]];
        return v;
    };
    P nu[6], nv[6];                // the next step's states: rows above, the four, below
    const auto fetch = [&](int j) {
        if (j < 0) return;
        const T* us = states + (size_t)(2 * j) * nn;
        const T* vs = us + nn;
        nu[0] = row(us, above);
        nv[0] = row(vs, above);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            nu[r + 1] = c.load(us, r);
            nv[r + 1] = c.load(vs, r);
        }
        nu[5] = row(us, below);
        nv[5] = row(vs, below);
    };
    double gF = 0, gk = 0, gDu = 0, gDv = 0, gvx = 0, gvy = 0;
    const T two = T(2), half = T(0.5), four = T(4);
    const T Fk = k.F + k.k;
    const auto cell = [&](bool own, T uU, T uc, T uD, T uL, T uR, T vU, T vc, T vD, T vL, T vR, T aU, T ac, T aD, T aL,
                          T aR, T bU, T bc, T bD, T bL, T bR, T* an, T* bn) {
        const T lap_a = aL + aR + aU + aD - four * ac;
        const T lap_b = bL + bR + bU + bD - four * bc;
        const T dxa = (aR - aL) * half, dya = (aD - aU) * half;
        const T dxb = (bR - bL) * half, dyb = (bD - bU) * half;
        const T v2 = vc * vc, uv = uc * vc;
        *an = ac + k.dt * (k.Du * lap_a + k.vx * dxa + k.vy * dya + ac * (-v2 - k.F) + bc * v2);
        *bn = bc + k.dt * (k.Dv * lap_b + k.vx * dxb + k.vy * dyb + ac * (-two * uv) + bc * (two * uv - Fk));
        if (own) {
            const double lu = (double)(uL + uR + uU + uD - four * uc);
            const double lv = (double)(vL + vR + vU + vD - four * vc);
            gF += (double)ac * (1.0 - (double)uc) - (double)bc * (double)vc;
            gk += -(double)bc * (double)vc;
            gDu += (double)ac * lu;
            gDv += (double)bc * lv;
            gvx += -(double)ac * (double)((uR - uL) * half) - (double)bc * (double)((vR - vL) * half);
            gvy += -(double)ac * (double)((uD - uU) * half) - (double)bc * (double)((vD - vU) * half);
        }
    };
    const auto step = [&](int par, int j, const P (&xa)[4], const P (&xb)[4], P (&ya)[4], P (&yb)[4]) {
        P su[6], sv[6];
#pragma unroll
        for (int r = 0; r < 6; ++r) {
            su[r] = nu[r];
            sv[r] = nv[r];
        }
        fetch(j - 1);
        const int up = (c.group + 7) & 7, dn = (c.group + 1) & 7;     // the outermost rows are stale anyway
        const P ta = *c.edge(par, 0, up, 1), tb = *c.edge(par, 1, up, 1);
        const P ba = *c.edge(par, 0, dn, 0), bb = *c.edge(par, 1, dn, 0);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const auto left = [](T v) { return __shfl_up_sync(0xffffffffu, v, 1, 16); };
            const auto right = [](T v) { return __shfl_down_sync(0xffffffffu, v, 1, 16); };
            const P aU = r == 0 ? ta : xa[r == 0 ? 0 : r - 1], aD = r == 3 ? ba : xa[r == 3 ? 3 : r + 1];
            const P bU = r == 0 ? tb : xb[r == 0 ? 0 : r - 1], bD = r == 3 ? bb : xb[r == 3 ? 3 : r + 1];
            const P u = su[r + 1], v = sv[r + 1];
            const T al = left(xa[r].y), ar = right(xa[r].x), bl = left(xb[r].y), br = right(xb[r].x);
            const T ul = left(u.y), ur = right(u.x), vl = left(v.y), vr = right(v.x);
            cell(c.cy[r] && c.cx[0], su[r].x, u.x, su[r + 2].x, ul, u.y, sv[r].x, v.x, sv[r + 2].x, vl, v.y, aU.x, xa[r].x,
                 aD.x, al, xa[r].y, bU.x, xb[r].x, bD.x, bl, xb[r].y, &ya[r].x, &yb[r].x);
            cell(c.cy[r] && c.cx[1], su[r].y, u.y, su[r + 2].y, u.x, ur, sv[r].y, v.y, sv[r + 2].y, v.x, vr, aU.y, xa[r].y,
                 aD.y, xa[r].x, ar, bU.y, xb[r].y, bD.y, xb[r].x, br, &ya[r].y, &yb[r].y);
        }
    };
    P xa[4], xb[4], ya[4], yb[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        xa[r] = c.load(lu_in, r);
        xb[r] = c.load(lv_in, r);
    }
    fetch(len - 1);
    c.put_edges(0, xa, xb);
    int s = 0;
    for (; s + 2 <= len; s += 2) {
        step(0, len - 1 - s, xa, xb, ya, yb);
        c.put_edges(1, ya, yb);
        step(1, len - 2 - s, ya, yb, xa, xb);
        if ((s + 2) % kTileGhost == 0 && s + 2 < len) c.swap(xbuf, (s + 2) / kTileGhost, xa, xb);
        c.put_edges(0, xa, xb);
    }
    if (s < len) {
        step(0, len - 1 - s, xa, xb, ya, yb);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            xa[r] = ya[r];
            xb[r] = yb[r];
        }
    }
    double g[6] = {gF, gk, gDu, gDv, gvx, gvy};
    const double dtd = (double)k.dt;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        double v = g[q] * dtd;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (c.lane == 0) s_red[q][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (s_failed) {
        if (threadIdx.x == 0) atomicOr(err, 1);
        const T nan = (T)__int_as_float(0x7fc00000);
#pragma unroll
        for (int r = 0; r < 4; ++r) xa[r].x = xa[r].y = xb[r].x = xb[r].y = nan;
    }
    if (threadIdx.x < 6) {
        double v = 0;
        for (int w = 0; w < kTileWarps; ++w) v += s_red[threadIdx.x][w];
        atomicAdd(&grad[threadIdx.x], v);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        c.store(lu_out, r, xa[r]);
        c.store(lv_out, r, xb[r]);
    }
}
