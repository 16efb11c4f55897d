// Per-cell device routines of the stochastic solvers, shared by the wide kernels
// (one launch covers every realisation) and the persistent ensemble kernel.
//
// Reference semantics (paths inside the reference project):
//   ssa_cell      Gillespie.cl:58-99 direct method; hazards Reaction.cpp:119-138;
//                 reaction picked where the cumulative hazard first exceeds r2,
//                 which is what the isless/isgreaterequal masks of
//                 Solver.cpp:865-904 select; the event that crosses the window
//                 end is discarded (Gillespie.cl:80).
//   homog_lost    StochasticHomogeneousDiffusion.cl:56-92: each particle moves to
//                 one of four neighbours with probability (1-Stay)/6 each;
//                 reflecting walls keep it, absorbing walls lose it.  Here the
//                 four counts are one multinomial draw (binomial for "moved",
//                 then an equal four-way split) instead of one uniform per particle.
//   sweep_probs   StochasticInhomogeneousDriftDiffusion.cl:512-520 (X) and
//                 :642-650 (Y): ps, p1 (towards +), p2-p1 (towards -).
//   cell_timestep StochasticInhomogeneousDriftDiffusion.cl:124-151 (and the FPE
//                 and deterministic variants of the same kernel).
#pragma once
#include "common.cuh"
#include "../../include/gpgmp_c.h"

namespace gpgmp {

__device__ __forceinline__ float hazard(const gpgmp_reaction& rc, const int* x, int stride) {
    float v = rc.rate;
    for (int j = 0; j < rc.num_reactants; ++j) {
        const int a = x[rc.reactant_species[j] * stride];
        v = v * (float)a;
        for (int k = 1; k < rc.reactant_stoich[j]; ++k) v = v * (float)(a - k);
    }
    return v;
}

// The mass-action hazard as a functor; a model with custom propensity laws supplies
// its own (compiled at run time, csrc/jit.cpp).
struct MassActionHazard {
    __device__ __forceinline__ float operator()(const gpgmp_reaction* rt, int r, const int* x, int stride) const {
        return hazard(rt[r], x, stride);
    }
};

// Localised reactions: bit r of on[r / 32] says whether reaction r may fire in this
// cell (Reaction::reactionMask, Reaction.cpp:216-235).  The reference multiplies the
// law by the mask value 1 or 0 (Solver.cpp:852-854); a zero hazard is the same sum.
struct CellReactions {
    uint32_t on[4];
    // rmask: [words][area] bits of the cells (words = ceil(reactions / 32)); NULL: all on
    __device__ __forceinline__ void load(const uint32_t* __restrict__ rmask, int words, int area, int c) {
        on[0] = on[1] = on[2] = on[3] = 0xFFFFFFFFu;
        if (rmask)
            for (int w = 0; w < words; ++w) on[w] = rmask[(int64_t)w * area + c];
    }
    __device__ __forceinline__ bool operator()(int r) const { return (on[r >> 5] >> (r & 31)) & 1u; }
};
struct AllReactions {
    __device__ __forceinline__ bool operator()(int) const { return true; }
};
template <class HZ>
struct GatedHazard {
    HZ hz;
    CellReactions on;
    __device__ __forceinline__ float operator()(const gpgmp_reaction* rt, int r, const int* x, int stride) const {
        return on(r) ? hz(rt, r, x, stride) : 0.0f;
    }
};

// Runs one SSA window on the counts x[s * stride]; returns a GPGMP_SIM_* bit or 0.
// From time t and after `events` events where a window is continued.
template <class HZ>
__device__ __forceinline__ int ssa_cell_h(const gpgmp_reaction* rt, int R, int* x, int stride, Stream& st,
                                          float window, const HZ& hz, float t = 0.0f, int events = 0) {
    for (;;) {
        float h0 = 0.0f;
        for (int r = 0; r < R; ++r) h0 = h0 + hz(rt, r, x, stride);
        if (!(h0 > 0.0f)) return 0;
        const uint32_t a = st.next(), b = st.next();
        const float r1 = u01_open0(a);
        const float r2 = u01(b) * h0;
        const float dtev = -gp_logf(r1) / h0;
        t = t + dtev;
        if (!(t < window)) return 0;
        // second pass: same partial sums, stop at the first one above r2
        int j = -1;
        float hc = 0.0f;
        for (int r = 0; r < R; ++r) {
            hc = hc + hz(rt, r, x, stride);
            if (r2 < hc) { j = r; break; }
        }
        if (j >= 0) {
            const gpgmp_reaction& rc = rt[j];
            for (int q = 0; q < rc.num_products; ++q)
                if (x[rc.product_species[q] * stride] > INT32_MAX - rc.product_stoich[q]) return SIM_OVERFLOW;
            for (int q = 0; q < rc.num_reactants; ++q) x[rc.reactant_species[q] * stride] -= rc.reactant_stoich[q];
            for (int q = 0; q < rc.num_products; ++q) x[rc.product_species[q] * stride] += rc.product_stoich[q];
        }
        if (++events >= SSA_EVENT_CAP) return SIM_EVENT_CAP;
    }
}
__device__ __forceinline__ int ssa_cell(const gpgmp_reaction* rt, int R, int* x, int stride, Stream& st,
                                        float window) {
    return ssa_cell_h(rt, R, x, stride, st, window, MassActionHazard{});
}

// Dependency masks of the incremental SSA: bit q of deps[j * 4 + q / 32] is set when
// reaction j changes the count of a species that reaction q consumes, i.e. when q's
// hazard must be recomputed after j fires (Gibson & Bruck's dependency graph).  Built
// by all threads of a block; R <= 128.
__device__ __forceinline__ void build_deps(const gpgmp_reaction* rt, int R, uint32_t* deps) {
    for (int idx = threadIdx.x; idx < R * 4; idx += blockDim.x) deps[idx] = 0u;
    __syncthreads();
    for (int idx = threadIdx.x; idx < R * R; idx += blockDim.x) {
        const int j = idx / R, q = idx % R;
        const gpgmp_reaction& a = rt[j];
        const gpgmp_reaction& b = rt[q];
        bool dep = false;
        for (int u = 0; u < b.num_reactants && !dep; ++u) {
            const int sp = b.reactant_species[u];
            int net = 0;
            for (int v = 0; v < a.num_reactants; ++v) if (a.reactant_species[v] == sp) net -= a.reactant_stoich[v];
            for (int v = 0; v < a.num_products; ++v) if (a.product_species[v] == sp) net += a.product_stoich[v];
            dep = net != 0;
        }
        if (dep) atomicOr(&deps[j * 4 + (q >> 5)], 1u << (q & 31));
    }
    __syncthreads();
}

// The same SSA window as ssa_cell with per-reaction hazards kept in h[r * stride]
// and recomputed only where the fired reaction changed a reactant count.  The total
// and the selection sum the same values in the same order as the full recomputation,
// so the result is bit-identical.
// ON(r) gates the reactions of localised models (CellReactions), as in ssa_cell_h.
template <class ON = AllReactions>
__device__ __forceinline__ int ssa_cell_inc(const gpgmp_reaction* rt, const uint32_t* deps, int R, int* x, int stride,
                                            float* h, Stream& st, float window, const ON& on = ON{}) {
    for (int r = 0; r < R; ++r) h[r * stride] = on(r) ? hazard(rt[r], x, stride) : 0.0f;
    float t = 0.0f;
    int events = 0;
    for (;;) {
        float h0 = 0.0f;
        for (int r = 0; r < R; ++r) h0 = h0 + h[r * stride];
        if (!(h0 > 0.0f)) return 0;
        const uint32_t a = st.next(), b = st.next();
        const float r1 = u01_open0(a);
        const float r2 = u01(b) * h0;
        const float dtev = -gp_logf(r1) / h0;
        t = t + dtev;
        if (!(t < window)) return 0;
        int j = -1;
        float hc = 0.0f;
        for (int r = 0; r < R; ++r) {
            hc = hc + h[r * stride];
            if (r2 < hc) { j = r; break; }
        }
        if (j >= 0) {
            const gpgmp_reaction& rc = rt[j];
            for (int q = 0; q < rc.num_products; ++q)
                if (x[rc.product_species[q] * stride] > INT32_MAX - rc.product_stoich[q]) return SIM_OVERFLOW;
            for (int q = 0; q < rc.num_reactants; ++q) x[rc.reactant_species[q] * stride] -= rc.reactant_stoich[q];
            for (int q = 0; q < rc.num_products; ++q) x[rc.product_species[q] * stride] += rc.product_stoich[q];
            for (int w = 0; w * 32 < R; ++w) {
                uint32_t m = deps[j * 4 + w];
                while (m) {
                    const int q = w * 32 + __ffs(m) - 1;
                    m &= m - 1;
                    h[q * stride] = on(q) ? hazard(rt[q], x, stride) : 0.0f;
                }
            }
        }
        if (++events >= SSA_EVENT_CAP) return SIM_EVENT_CAP;
    }
}

// ---- packed networks -------------------------------------------------------------
// A network whose reactions have at most two reactant molecules and change at most four
// species (pack_network, netpack.h) runs its windows on float copies of the counts, which
// are exact up to 2^24.  Every hazard then is the same three operations, rate * x[s1] *
// (x[s2] - sub): an absent reactant is slot 0, which holds 1 (the
// products by 1 and the difference of 0 are exact; species s is slot s + 1), and 2A has s2 = s1, sub = 1, so the
// values and their running sums are those of ssa_cell bit for bit.  No table of the
// reaction structs is walked, nothing is converted per event and the sums are kept for the
// selection instead of formed twice: A + B <-> C on 1M cells, a window of 1.7 events per
// cell, 47 us instead of 78; predator and prey on 8.4M cells, 112 us instead of 171; 592
// random networks of 8 to 32 reactions, 75 ms instead of 238.
// A cell whose counts are negative or reach kPackedMax goes on in ssa_slow, which keeps the
// counts as integers in the same slots.  The limit is the largest change of a packed
// reaction below 2^24, so that the sum that passes it is still exact.
struct PackedReaction {
    float rate, sub;
    int32_t s1, s2;      // slots of the reactants
    uint32_t net[4];     // slot << 16 | upper half of the float change; unused: 0
};
constexpr int kPackedChange = 256;      // pack_network's largest change of a count
constexpr int kPackedMax = (1 << 24) - kPackedChange;

// Where a window stands: time, events, the last draws and how many of them are used.
struct SsaPos {
    float t;
    int events;
    uint32_t w[4];
    int used;
};

enum { SSA_SLOW = -1 };     // returned where the window has to go on in ssa_slow

// the time of an event from its draw and the total hazard (a draw's logarithm is 0 or
// between 2^-24 and 17 in size, so div_mid's range is the hazard's)
__device__ __forceinline__ float ssa_wait(uint32_t draw, float h0) {
    const float l = -log_draw(draw);
    return h0 > 8.6736174e-19f && h0 < 1.1529215e18f ? div_mid(l, h0) : l / h0;
}

// applies one event's changes; true while every changed count stays below kPackedMax
template <int STRIDE>
__device__ __forceinline__ bool packed_apply(const uint4& n, int nnet, float* x) {
    const uint32_t e[4] = {n.x, n.y, n.z, n.w};
    float top = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (i < nnet) {
            float* p = x + (e[i] >> 16) * STRIDE;
            const float v = *p + __uint_as_float(e[i] << 16);
            *p = v;
            top = fmaxf(top, v);
        }
    }
    return top < (float)kPackedMax;
}

// One window of a network of NR reactions given by value (kernel parameters): the running
// sums stay in registers.  nets: the changes of every reaction in shared memory.
template <int NR>
struct SmallNet {
    float rate[NR], sub[NR];
    int32_t o1[NR], o2[NR];  // slots of the reactants, times the threads of a block
    uint4 net[NR];
    int32_t nnet;            // most species that one reaction changes
};
template <int NR, int STRIDE>
__device__ __forceinline__ int ssa_small(const SmallNet<NR>& net, const uint4* nets, float* x, Stream& st,
                                         float window, SsaPos& pos) {
    pos.t = 0.0f;
    pos.events = 0;
    for (;;) {
        st.block(pos.w);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float c[NR], h0 = 0.0f;
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                h0 = h0 + net.rate[q] * x[net.o1[q]] * (x[net.o2[q]] - net.sub[q]);
                c[q] = h0;
            }
            if (!(h0 > 0.0f)) return 0;
            const float r2 = u01(pos.w[2 * half + 1]) * h0;
            pos.t = pos.t + ssa_wait(pos.w[2 * half], h0);
            if (!(pos.t < window)) return 0;
            int j = NR;
#pragma unroll
            for (int q = NR - 1; q >= 0; --q) j = r2 < c[q] ? q : j;
            bool small = true;
            if (j < NR) small = packed_apply<STRIDE>(nets[j], net.nnet, x);
            if (++pos.events >= SSA_EVENT_CAP) return SIM_EVENT_CAP;
            if (!small) {
                pos.used = 2 * half + 2;
                return SSA_SLOW;
            }
        }
    }
}

// The same for a network in shared memory (ent: rate, sub, s1 * STRIDE, s2 * STRIDE as
// bits), with the running sums in c[q * STRIDE]: they only grow, so the selection halves
// its range instead of walking it.
template <int STRIDE>
__device__ __forceinline__ int ssa_packed(const float4* ent, const uint4* nets, int nnet, int R, float* x, float* c,
                                          Stream& st, float window, SsaPos& pos) {
    int top = 1;
    while (2 * top <= R) top *= 2;
    pos.t = 0.0f;
    pos.events = 0;
    pos.used = 4;
    for (;;) {
        if (pos.used == 4) {
            st.block(pos.w);
            pos.used = 0;
        }
        float h0 = 0.0f;
#pragma unroll 4
        for (int q = 0; q < R; ++q) {
            const float4 e = ent[q];
            h0 = h0 + e.x * x[__float_as_int(e.z)] * (x[__float_as_int(e.w)] - e.y);
            c[q * STRIDE] = h0;
        }
        if (!(h0 > 0.0f)) return 0;
        const uint32_t a = pos.used ? pos.w[2] : pos.w[0], b = pos.used ? pos.w[3] : pos.w[1];
        pos.used += 2;
        const float r2 = u01(b) * h0;
        pos.t = pos.t + ssa_wait(a, h0);
        if (!(pos.t < window)) return 0;
        int j = 0;
        for (int s = top; s > 0; s >>= 1)
            if (j + s <= R && !(r2 < c[(j + s - 1) * STRIDE])) j += s;
        bool small = true;
        if (j < R) small = packed_apply<STRIDE>(nets[j], nnet, x);
        if (++pos.events >= SSA_EVENT_CAP) return SIM_EVENT_CAP;
        if (!small) return SSA_SLOW;
    }
}

// The tables of ssa_packed in shared memory, by all threads of a block (which then syncs).
template <int STRIDE>
__device__ __forceinline__ void packed_tables(const PackedReaction* __restrict__ p, int R, float4* ent, uint4* nets) {
    for (int q = threadIdx.x; q < R; q += blockDim.x) {
        ent[q] = make_float4(p[q].rate, p[q].sub, __int_as_float(p[q].s1 * STRIDE), __int_as_float(p[q].s2 * STRIDE));
        nets[q] = make_uint4(p[q].net[0], p[q].net[1], p[q].net[2], p[q].net[3]);
    }
}

// The counts of one cell from memory (at(s): species s) into the float slots; false where
// a count is negative or at least kPackedMax (the slots then hold the integers' bits).
template <int STRIDE, class AT>
__device__ __forceinline__ bool packed_load(const AT& at, int S, float* x) {
    bool fits = true;
    for (int s = 0; s < S; ++s) {
        const int v = at(s);
        fits = fits && (uint32_t)v < (uint32_t)kPackedMax;
        x[(s + 1) * STRIDE] = (float)v;
    }
    if (!fits)
        for (int s = 0; s < S; ++s) x[(s + 1) * STRIDE] = __int_as_float(at(s));
    x[0] = 1.0f;
    return fits;
}
// The rest of a window on integer counts (the slots hold their bits).
template <int STRIDE>
__device__ __noinline__ int ssa_slow(const gpgmp_reaction* rt, int R, float* x, const Stream& from, float window,
                                     const SsaPos& pos) {
    Stream st = from;
#pragma unroll
    for (int i = 0; i < 4; ++i) st.buf[i] = pos.w[i];
    st.idx = pos.used;
    return ssa_cell_h(rt, R, reinterpret_cast<int*>(x + STRIDE), STRIDE, st, window, MassActionHazard{}, pos.t, pos.events);
}
// One window of one cell: load, run (`run` is ssa_small or ssa_packed), store.  Returns a
// GPGMP_SIM_* bit or 0.
template <int STRIDE, class AT, class RUN>
__device__ __forceinline__ int packed_window(const gpgmp_reaction* rt, int R, const AT& at, int S, float* x,
                                             Stream& st, float window, const RUN& run) {
    SsaPos pos;
    int e = SSA_SLOW;
    if (packed_load<STRIDE>(at, S, x)) {
        e = run(x, st, pos);
        if (e != SSA_SLOW) {
            for (int s = 0; s < S; ++s) at(s) = (int)x[(s + 1) * STRIDE];
            return e;
        }
        for (int s = 1; s <= S; ++s) x[s * STRIDE] = __int_as_float((int)x[s * STRIDE]);
    } else {
        pos.t = 0.0f;
        pos.events = 0;
        pos.used = 4;
    }
    e = ssa_slow<STRIDE>(rt, R, x, st, window, pos);
    for (int s = 0; s < S; ++s) at(s) = __float_as_int(x[(s + 1) * STRIDE]);
    return e;
}

// Four lost counts (-x, +x, -y, +y) of one cell of n particles; jump: the draw of the moved
// ones (BinomialSetup or BinomialTable).
template <class JUMP>
__device__ __forceinline__ void homog_lost(int n, const JUMP& jump, Stream& st, int x, int y, int W, int H,
                                           const int* bmask, int l[4]) {
    l[0] = l[1] = l[2] = l[3] = 0;
    if (n <= 0 || jump.kind == 0) return;
    int moved;
    if (jump.single(n)) {          // one draw, the first of the block whose others serve the directions
        st.block(st.buf);
        st.idx = 1;
        moved = jump.count(st.buf[0], n);
    } else {
        moved = binomial(st, n, jump);
    }
    if (moved <= 64) {
        // sixteen 2-bit directions per draw, counted by their bits
        int c1 = 0, c2 = 0, c3 = 0;
        for (int left = moved; left > 0; left -= 16) {
            uint32_t w = st.next();
            if (left < 16) w &= (1u << (2 * left)) - 1u;
            const uint32_t lo = w & 0x55555555u, hi = (w >> 1) & 0x55555555u;
            const int both = __popc(lo & hi);
            c3 += both;
            c1 += __popc(lo) - both;
            c2 += __popc(hi) - both;
        }
        l[0] = moved - c1 - c2 - c3; l[1] = c1; l[2] = c2; l[3] = c3;
    } else {
        l[0] = binomial(st, moved, 0.25f);
        l[1] = binomial(st, moved - l[0], 1.0f / 3.0f);
        l[2] = binomial(st, moved - l[0] - l[1], 0.5f);
        l[3] = moved - l[0] - l[1] - l[2];
    }
    if (x == 0 && bmask[0] == 0) l[0] = 0;
    if (x == W - 1 && bmask[1] == 0) l[1] = 0;
    if (y == 0 && bmask[2] == 0) l[2] = 0;
    if (y == H - 1 && bmask[3] == 0) l[3] = 0;
}

__device__ __forceinline__ float clamp01(float v) { return v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v); }

__device__ __forceinline__ void sweep_probs(float D, float r, float dt, float dx, float* Pp, float* Pm) {
    const float denom = 2.0f * D + r * r * dt;
    const float ps = 1.0f - (dt * denom) / (dx * dx);
    const float q = 1.0f - ps;
    float p1 = 0.0f, pm = 0.0f;
    if (denom > 0.0f) {
        const float b = (dx * r) / denom;
        p1 = q * (1.0f + b) * 0.5f;
        pm = q * (1.0f - b) * 0.5f;
    }
    *Pp = clamp01(p1);
    const float rest = 1.0f - *Pp;
    *Pm = pm < 0.0f ? 0.0f : (pm > rest ? rest : pm);
}

// The FPE discretisation's jump probabilities (stochastic_inhomogeneous_fpe,
// StochasticInhomogeneousDriftDiffusion.cl:197-203 rates, :493-499 use): rate
// towards + is D/dx^2 + r/(2 dx), towards - is D/dx^2 - r/(2 dx), times dt.  A rate
// that comes out negative (|r| dx > 2 D) is clamped to 0.
__device__ __forceinline__ void sweep_probs_fpe(float D, float r, float dt, float dx, float* Pp, float* Pm) {
    const float a = D / (dx * dx), b = r / (2.0f * dx);
    *Pp = clamp01((a + b) * dt);
    const float pm = (a - b) * dt, rest = 1.0f - *Pp;
    *Pm = pm < 0.0f ? 0.0f : (pm > rest ? rest : pm);
}

// A directional sweep of one cell: the draw of the moved particles and of those among them
// that go towards +, set up once from the cell's fields; draw() takes one realisation's
// count.
struct SweepCell {
    BinomialSetup<7> moved;
    BinomialSetup<4> plus;
    bool stay_lo, stay_hi;      // a reflecting wall below / above
    __device__ __forceinline__ void init(float D, float r, float dt, float dx, bool lo, bool hi, bool fpe) {
        float Pp, Pm;
        if (fpe)
            sweep_probs_fpe(D, r, dt, dx, &Pp, &Pm);
        else
            sweep_probs(D, r, dt, dx, &Pp, &Pm);
        const float Pt = Pp + Pm;
        moved.init(Pt);
        plus.init(Pt > 0.0f ? Pp / Pt : 0.0f);
        stay_lo = lo;
        stay_hi = hi;
    }
    // (minus, plus) counts of n particles
    __device__ __forceinline__ void draw(int n, Stream& st, int* minus, int* plus_out) const {
        int k = 0, p = 0;
        if (n > 0 && moved.kind != 0) {
            Stream again = st;
            uint32_t w[4];
            st.block(w);
            if (moved.single(n) && plus.kind != 3) {     // one draw each, but for large counts
                k = moved.count(w[0], n);
                if (k > 0 && plus.kind != 0) {
                    if (k <= plus.chunk) {
                        p = plus.count(w[1], k);
                    } else {
                        again.next();
                        p = binomial(again, k, plus);
                    }
                }
            } else {
                k = binomial(again, n, moved);
                p = binomial(again, k, plus);
            }
        }
        *minus = stay_lo ? 0 : k - p;
        *plus_out = stay_hi ? 0 : p;
    }
};

// Evaluated in double; below |eps| = 1e-3 tanh and temp come from their series
// (tanh eps = eps - eps^3/3, temp = 1/3 + 4 eps^2/45) because the closed form
// cancels there (in float it gives NaN or 0 for small drift).
__device__ __forceinline__ double cell_timestep_d(float Df, float rf, float dxf) {
    const double D = Df, r = rf, dx = dxf;
    if (r == 0.0) return dx * dx / (2.0 * D) * (1.0 / 3.0);
    if (D == 0.0) return dx / fabs(r);
    const double eps = dx * r / (2.0 * D);
    const double a = fabs(eps);
    double th, temp;
    if (a < 1e-3) {
        th = eps - eps * eps * eps / 3.0;
        temp = 1.0 / 3.0 + 4.0 * eps * eps / 45.0;
    } else {
        const double t = gp_exp_d(-2.0 * a);
        const double tha = (1.0 - t) / (1.0 + t);
        th = eps < 0.0 ? -tha : tha;
        const double E = gp_exp_d(a);
        const double sha = (E - 1.0 / E) * 0.5;
        temp = 1.0 + (-1.0 / (th * eps) + 1.0 / (sha * sha));
        if (temp <= 0.0) temp = 1.0 / 3.0;
    }
    return dx / r * th * temp;
}
__device__ __forceinline__ float cell_timestep(float D, float r, float dx) { return (float)cell_timestep_d(D, r, dx); }

// Time step kinds of the per-cell minimum (StochasticInhomogeneousDriftDiffusion.cl:
// 124-151 stochastic, :124-129 FPE, :157-190 deterministic RK4 / alpha-QSS).
enum TimestepKind { kTsStochastic = 0, kTsFpe = 1, kTsDeterministic = 2 };

// FPE: StayProbability / 6 / (D / dx^2 + |r| / (2 dx)), in float.
__device__ __forceinline__ float fpe_timestep(float D, float r, float dx, float stay) {
    return stay / 6.0f / (D / (dx * dx) + fabsf(r) / (2.0f * dx));
}

// deterministic inhomogeneous solvers: the stochastic formula scaled by 0.1 where
// there is drift (the reference's r == 0 branch is not scaled); with D = 0 the
// reference divides by zero, here the step is 0.1 dx / |r|.
__device__ __forceinline__ float det_timestep(float D, float r, float dx) {
    if (r == 0.0f) return (float)cell_timestep_d(D, r, dx);
    return (float)(0.1 * cell_timestep_d(D, r, dx));
}

}  // namespace gpgmp
