// Batched float32 Gray-Scott forward kernel: row blocks on small clusters.
//
// One lattice per cluster of CL CTAs (1, 2, 4 or 8 instead of the 16 of gs_rr.cuh), so
// that a batch fills the chip with whole lattices: a CTA's warps own R = N / (CL WPC) rows
// each, kept in registers and updated in place, and with more rows per warp the arithmetic
// of a step outlasts its halo exchange (for a batch the exchange is overhead, not the
// step's length).  The exchange and its waits are those of gs_rr.cuh, but a producer warp
// arrives once on a neighbour's mbarrier instead of once per lane (the shared-memory pipe
// is shared by all the warps here).  Each cell's update is gs_update2f as everywhere: the
// bits are those of the single-lattice kernels.
//
// What bounds it: the FP32 pipe (18 packed operations per pair of cells, two cycles each: at
// most 7.1 cells per cycle and SM).  128^2 with 8 rows per warp runs at 5.2, 4 rows per warp
// 4.8 (the halo's loads, sends and waits); where the batch does not divide into the SMs the
// rest are idle.
//
// Included from gray_scott.cu after gs_rr.cuh.

template <int N, int CL, int WPC>
struct RBShape {
    static constexpr int R = N / (CL * WPC);           // rows per warp
    static constexpr int H = N / 64;                   // column pairs per lane
    static constexpr uint32_t kRow = 4u * N;           // bytes of one halo row of one field
    static constexpr uint32_t kHalo = (uint32_t)WPC * 8u * kRow;
    static constexpr uint32_t kSmem = kHalo + (uint32_t)WPC * 16u + 16u;
    static_assert(kSmem <= 227u * 1024u, "shared memory of a B200 CTA");
    static_assert(R >= 2 && R * CL * WPC == N && H >= 1 && 64 * H == N, "lattice split");
};

template <int N, int CL, int WPC>
struct RBCtx {
    using S = RBShape<N, CL, WPC>;
    uint32_t sbase;
    const unsigned char* smem;
    int lane, w;
    uint32_t up_rank, dn_rank;
    int up_w, dn_w;
    bool up_remote, dn_remote;
    uint32_t tx;             // bytes the producers in other CTAs deliver per phase
    volatile int* failed;
    __device__ __forceinline__ uint32_t slot(int ww, int par, int side, int f) const {
        return sbase + (uint32_t)(((ww * 2 + par) * 2 + side) * 2 + f) * S::kRow;
    }
    __device__ __forceinline__ uint32_t bar(int ww, int par) const { return sbase + S::kHalo + (uint32_t)(ww * 2 + par) * 8u; }
};

// one row into the neighbour's halo slot, as rr_send, with one arrive per warp
template <int H>
__device__ __forceinline__ void rb_send(const float2 (&pu)[H], const float2 (&pv)[H], uint32_t dst_u, uint32_t dst_v,
                                        uint32_t bar, bool remote, uint32_t rank, int lane) {
    if (remote) {
        rr_send<H>(pu, pv, dst_u, dst_v, bar, true, rank, lane);
        return;
    }
    constexpr uint32_t UB = RRUnit<H>::kBytes;
#pragma unroll
    for (int q = 0; q < RRUnit<H>::kCount; ++q) {
        const uint32_t off = (uint32_t)(q * 32 + lane) * UB;
        if constexpr (H >= 2) {
            rr_st_local(dst_u + off, make_float4(pu[2 * q].x, pu[2 * q].y, pu[2 * q + 1].x, pu[2 * q + 1].y));
            rr_st_local(dst_v + off, make_float4(pv[2 * q].x, pv[2 * q].y, pv[2 * q + 1].x, pv[2 * q + 1].y));
        } else {
            rr_st_local(dst_u + off, pu[0]);
            rr_st_local(dst_v + off, pv[0]);
        }
    }
    __syncwarp();             // the lanes' stores are before lane 0's releasing arrive
    if (lane == 0) rr_arrive(bar);
}

// sends the warp's edge rows of state s to its neighbours' halos of parity par
template <int N, int CL, int WPC>
__device__ __forceinline__ void rb_send_edges(const RBCtx<N, CL, WPC>& c, const float2 (&fu)[N / 64],
                                              const float2 (&fv)[N / 64], const float2 (&lu)[N / 64],
                                              const float2 (&lv)[N / 64], int par) {
    constexpr int H = N / 64;
    rb_send<H>(fu, fv, c.slot(c.up_w, par, 1, 0), c.slot(c.up_w, par, 1, 1), c.bar(c.up_w, par), c.up_remote,
               c.up_rank, c.lane);
    rb_send<H>(lu, lv, c.slot(c.dn_w, par, 0, 0), c.slot(c.dn_w, par, 0, 1), c.bar(c.dn_w, par), c.dn_remote,
               c.dn_rank, c.lane);
}

template <int N, int CL, int WPC, int DRIFT>
__global__ void __launch_bounds__(32 * WPC)
    k_gs_forward_rb(const GSArgs<float>* __restrict__ batch_args, const float* __restrict__ u0,
                    const float* __restrict__ v0, float* __restrict__ uo, float* __restrict__ vo) {
    using S = RBShape<N, CL, WPC>;
    constexpr int R = S::R, H = S::H;
    const int member = (int)blockIdx.x / CL;
    const size_t moff = (size_t)member * N * N;
    const GSArgs<float> a = batch_args[member];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RBCtx<N, CL, WPC> c;
    c.smem = smem_raw;
    c.sbase = smem_u32(smem_raw);
    c.lane = threadIdx.x & 31;
    c.w = threadIdx.x >> 5;
    const uint32_t rank = CL == 1 ? 0u : rr_ctarank();
    c.up_remote = CL > 1 && c.w == 0;
    c.dn_remote = CL > 1 && c.w == WPC - 1;
    c.up_rank = c.up_remote ? (rank + CL - 1) % CL : rank;
    c.dn_rank = c.dn_remote ? (rank + 1) % CL : rank;
    c.up_w = c.w == 0 ? WPC - 1 : c.w - 1;
    c.dn_w = c.w == WPC - 1 ? 0 : c.w + 1;
    c.failed = reinterpret_cast<volatile int*>(smem_raw + S::kHalo + WPC * 16);
    const int nremote = (int)c.up_remote + (int)c.dn_remote;
    c.tx = (uint32_t)nremote * 2u * S::kRow;
    const size_t first = moff + (size_t)(((int)rank * WPC + c.w) * R) * N + c.lane * 2 * H;
    const GSCoef2 k(a);
    if (c.lane == 0) {
        // arrivals per phase: the own arm and one per producer warp of this CTA
#pragma unroll
        for (int par = 0; par < 2; ++par)
            mbar_init(reinterpret_cast<uint64_t*>(smem_raw + (c.bar(c.w, par) - c.sbase)), 1 + 2 - nremote);
        fence_mbar_init();
    }
    if (threadIdx.x == 0) *c.failed = 0;
    float2 xu[R][H], xv[R][H];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        rr_load<H>(u0 + first + (size_t)r * N, xu[r]);
        rr_load<H>(v0 + first + (size_t)r * N, xv[r]);
    }
    __syncthreads();
    if (CL > 1) {
        cluster_arrive();     // every CTA's mbarriers exist before anyone sends
        cluster_wait();
    }
    const int steps = a.steps;
    if (steps > 0) {
        if (c.lane == 0) {
            rr_arm(c.bar(c.w, 0), c.tx);
            rr_arm(c.bar(c.w, 1), c.tx);
        }
        rb_send_edges<N, CL, WPC>(c, xu[0], xv[0], xu[R - 1], xv[R - 1], 0);
    }
    // two steps per iteration: the rows of the odd step live where the even step's old rows
    // were, so no row is moved at the end of a step
#pragma unroll 2
    for (int s = 0; s < steps; ++s) {
        const int par = s & 1;
        rr_wait(c.bar(c.w, par), (uint32_t)(s >> 1) & 1u, c.failed);
        __syncwarp();
        if (c.lane == 0) rr_arm(c.bar(c.w, par), c.tx);   // the phase of step s + 2
        // the edge rows first, sent while the interior rows are computed
        float2 fu[H], fv[H], lu[H], lv[H];
        {
            float2 hu[H], hv[H];
            rr_read_halo<H>(c.smem + (c.slot(c.w, par, 0, 0) - c.sbase), c.lane, hu);
            rr_read_halo<H>(c.smem + (c.slot(c.w, par, 0, 1) - c.sbase), c.lane, hv);
            rr_row<H, DRIFT>(k, hu, xu[0], xu[1], hv, xv[0], xv[1], fu, fv, c.lane);
            rr_read_halo<H>(c.smem + (c.slot(c.w, par, 1, 0) - c.sbase), c.lane, hu);
            rr_read_halo<H>(c.smem + (c.slot(c.w, par, 1, 1) - c.sbase), c.lane, hv);
            rr_row<H, DRIFT>(k, xu[R - 2], xu[R - 1], hu, xv[R - 2], xv[R - 1], hv, lu, lv, c.lane);
        }
        if (s + 1 < steps) rb_send_edges<N, CL, WPC>(c, fu, fv, lu, lv, par ^ 1);
        // the interior rows in place: pu, pv hold the old row above
        float2 pu[H], pv[H];
#pragma unroll
        for (int j = 0; j < H; ++j) {
            pu[j] = xu[0][j];
            pv[j] = xv[0][j];
            xu[0][j] = fu[j];
            xv[0][j] = fv[j];
        }
#pragma unroll
        for (int r = 1; r < R - 1; ++r) {
            float2 nu[H], nv[H];
            rr_row<H, DRIFT>(k, pu, xu[r], xu[r + 1], pv, xv[r], xv[r + 1], nu, nv, c.lane);
#pragma unroll
            for (int j = 0; j < H; ++j) {
                pu[j] = xu[r][j];
                pv[j] = xv[r][j];
                xu[r][j] = nu[j];
                xv[r][j] = nv[j];
            }
        }
#pragma unroll
        for (int j = 0; j < H; ++j) {
            xu[R - 1][j] = lu[j];
            xv[R - 1][j] = lv[j];
        }
    }
    __syncthreads();
    if (CL > 1) {
        cluster_arrive();     // no CTA leaves while a neighbour may still address its shared memory
        cluster_wait();
    }
    const bool bad = *c.failed != 0;
    if (bad && threadIdx.x == 0) atomicOr(&g_gs_fwd_err, 1);
    const float nan = __int_as_float(0x7fc00000);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (bad) {
#pragma unroll
            for (int j = 0; j < H; ++j) xu[r][j] = xv[r][j] = make_float2(nan, nan);
        }
        rr_store<H>(uo + first + (size_t)r * N, xu[r]);
        rr_store<H>(vo + first + (size_t)r * N, xv[r]);
    }
}
