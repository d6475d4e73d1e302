// sweep_march64.cuh -- FP64 LU-SGS sweeps as marching warps, the DeltaQ components over a CTA's warps.
//
// The tiles, their order and the words between them are those of sweep_march.cuh; the arithmetic
// is the reference's, operation by operation (bit-identical to the hyperplane launches).  An FP64
// warp instruction takes its sub-partition 63 cycles, dependent or not, and a step of 32 cells has
// ~205 of them (181 and 28 in the lower sweep, mean flow and k-omega; 176 and 28 in the upper), so a step's work is spread over the SM's four: a warp holds one component of the
// tile's 32 lines.  The share of a cell in its neighbour's sum of a component is a value of that
// component's warp, so it stays in the lane (i), or goes to lane a-1 or b-1 by shuffle (j, k); only
// the five mean-flow increments of the step cross warps, through shared memory and one barrier.
// The k and omega warps need none and run by themselves, in CTAs of their own.  The inputs of a
// step are contiguous in the records and come by bulk copies, three steps ahead: loaded into
// registers a step ahead they cost 90 registers, and loaded at the step's start their latency.
//
// The records hold each cell's own Jacobian terms (k_march64_jac: 656 bytes a cell), which serve its
// three neighbours in both sweeps; the hyperplane records keep the six neighbours' (1,280 bytes,
// each cell's terms formed twice).
//
// Bound by the FP64 pipe and the chain of a step: 46 FP64 instructions on the fullest sub-partition (1.4 us
// at 2,070 MHz) and a division on the integer pipe on the way from one step to the next, 2.16 us a step of a
// tile by itself.  Both sweeps with the records' preparation, hyperplane launches before and now: 24x16x5 cells
// 355 and 274 us, 96x48x8 1,213 and 779 us, a cascade of 352,256 cells 2,400 and 1,832 us, of 1,966,080 cells
// 8,047 and 4,838 us; k and omega alone (Runge-Kutta, annulus 70x38x26, three stages) 2,162 and 1,220 us.
#pragma once
#include "kernels.cuh"
#include "launch.h"
#include "march_words.cuh"

namespace tg {

// y + 0 * z without the FP64 instructions: y unless it is zero; the sum of two zeros is -0 only if both
// are; 0 times an infinity or NaN is NaN
__device__ __forceinline__ f64 add_zero_times(f64 y, f64 z) {
    const int yh = __double2hiint(y.v), yl = __double2loint(y.v), zh = __double2hiint(z.v);
    if ((zh & 0x7ff00000) == 0x7ff00000) return f64(__hiloint2double(0x7ff80000, 0));
    return ((yh << 1) | yl) ? y : f64(__hiloint2double(yh & zh & 0x80000000, 0));
}

// What the warps of a tile share: the place of the lane's cell, and the tag and bounds of the edge words.
template <bool LOWER>
struct March64Walk {
    static constexpr int side = LOWER ? 0 : 1, LJ = MARCH_J, LK = MARCH_K;
    static constexpr int REC = (LOWER ? 1 : -1) * M64_WIDTH * 32, DQS = (LOWER ? 1 : -1) * DQ_STRIDE * 32;   // a step on
    const MarchTile& T;
    const f64* rec;
    f64* dq;
    ulonglong2 *bufJ, *bufK;
    unsigned tag, limit;
    SweepSync* sy;
    int lane, a, b, cell, steps, lastJ, lastK;     // lastJ, lastK: steps with an edge word for this lane
    long long q0;
    bool in_jk, outJ, outK, lost;                  // lost: given up, the tile goes on without the words
    int stalled;                                   // the step whose inputs did not come, or -1
    __device__ March64Walk(const MarchTile& T_, const f64* rec_, f64* dq_, ulonglong2* bJ, ulonglong2* bK, unsigned tag_, SweepSync* sy_,
                           unsigned limit_)
        : T(T_), rec(rec_), dq(dq_), bufJ(bJ), bufK(bK), tag(tag_), limit(limit_), sy(sy_), lost(false), stalled(-1) {
        lane = threadIdx.x & 31;
        a = lane % LJ;
        b = lane / LJ;
        cell = LOWER ? lane : 31 - lane;
        steps = T.NI1 + (LJ - 1) + (LK - 1);
        in_jk = cell % LJ < T.nj && cell / LJ < T.nk;
        q0 = (long long)(T.s0 + (LOWER ? 0 : steps - 1)) * 32 + cell;
        lastK = T.sK[side] >= 0 && b == 0 ? steps - (LK - 1) : 0;
        lastJ = T.sJ[side] >= 0 && a == 0 ? steps - (LJ - 1) : 0;
        outK = T.sK[1 - side] >= 0 && b == LK - 1;
        outJ = T.sJ[1 - side] >= 0 && a == LJ - 1;
    }
    __device__ bool active(int t) const { return in_jk && (unsigned)(t - a - b) < (unsigned)T.NI1; }
    // the words of component L: those read (of the neighbouring tiles) and written, of step t
    __device__ const ulonglong2* inK(int L, int t) const { return bufK + ((size_t)(T.sK[side] + LK - 1 + t) * M64_EDGES + L) * LJ + a; }
    __device__ const ulonglong2* inJ(int L, int t) const { return bufJ + ((size_t)(T.sJ[side] + LJ - 1 + t) * M64_EDGES + L) * LK + b; }
    __device__ void put_j(int L, int t, f64 x) const {
        if (outJ) march_st(bufJ + ((size_t)(T.s0 + t) * M64_EDGES + L) * LK + b, __uint_as_float(__double2loint(x.v)), __uint_as_float(__double2hiint(x.v)), tag);
    }
    __device__ void put_k(int L, int t, f64 x) const {
        if (outK) march_st(bufK + ((size_t)(T.s0 + t) * M64_EDGES + L) * LJ + a, __uint_as_float(__double2loint(x.v)), __uint_as_float(__double2hiint(x.v)), tag);
    }
};

// Bulk copies of a step's inputs into a stage, complete on a transaction barrier; the wait for a phase
// is bounded like the others (and at M64_PHASE_LIMIT polls).  Four stages leave two mean-flow CTAs on an SM: at 1,966,080 cells 3.42 ms for both sweeps,
// against 3.71 with three stages and CTAs and 4.03 with two stages and four (the CTAs of one SM
// are on one diagonal, and the steps of each take longer); no difference at the smaller sizes.
constexpr int M64_STAGES = 4;
constexpr int M64_MEAN_IN = M64_MEAN_ROWS + 5, M64_TURB_IN = M64_WIDTH - M64_TURB_ROW0 + 1;     // rows of 32 values: records, then DeltaQ
constexpr unsigned M64_PHASE_LIMIT = 1u << 20;
__device__ __forceinline__ unsigned march64_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void march64_copy(f64* dst, const f64* src, unsigned rows, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(march64_smem(dst)),
                 "l"(src), "r"(rows * 256u), "r"(bar) : "memory");
}
__device__ __forceinline__ void march64_expect(unsigned bar, unsigned rows) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(rows * 256u) : "memory");
}
__device__ __forceinline__ bool march64_complete(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// a wait for the inputs of step t that the first look did not end: the step at which the tile gave up, or -1
static __device__ __noinline__ int march64_wait(unsigned bar, unsigned parity, int t, unsigned limit, SweepSync* sy) {
    for (unsigned n = 1; !march64_complete(bar, parity); ++n)
        if (n > min(limit, M64_PHASE_LIMIT) || (n % 1024u == 0 && *((volatile int*)&sy->err))) {
            atomicExch(&sy->err, 1);
            return t;
        }
    return -1;
}
// the inputs of step t are there; should the wait run out (or another have given up), the tile goes on without
// them, and without further waits and copies (w.stalled: the step)
template <class W>
__device__ __forceinline__ void march64_phase(W& w, unsigned bar, unsigned parity, int t) {
    if (!march64_complete(bar, parity) && w.stalled < 0) w.stalled = march64_wait(bar, parity, t, w.limit, w.sy);
}
// the lane that issued the copies, after a wait that ran out: those of steps before `issued` land before the CTA gives
// up its shared memory
__device__ __forceinline__ void march64_drain(unsigned full, int issued) {
    for (int st = 0; st < M64_STAGES && st < issued; ++st)
        for (unsigned n = 0; n < M64_PHASE_LIMIT && !march64_complete(full + 8 * st, (unsigned)((issued - 1 - st) / M64_STAGES) & 1u); ++n) {}
}

// The edge words of one component: read a step ahead, polled where they have not arrived.
template <bool LOWER>
struct March64Edge {
    ulonglong2 wJ, wK;
    __device__ void load(const March64Walk<LOWER>& w, const int L, int t) {
        if (t < w.lastK) wK = march_ld(w.inK(L, t));
        if (t < w.lastJ) wJ = march_ld(w.inJ(L, t));
    }
    // the terms of step t in xj, xk of the lanes that take them from a neighbouring tile (0: none there);
    // the wait is bounded, with the same answer for every lane
    __device__ void take(March64Walk<LOWER>& w, const int L, int t, f64& xj, f64& xk) {
        auto good = [&](const ulonglong2& x) { return (unsigned)(x.x >> 32) == w.tag && (unsigned)(x.y >> 32) == w.tag; };
        auto there = [&]() { return w.lost || ((t >= w.lastK || good(wK)) && (t >= w.lastJ || good(wJ))); };
        bool ok = there();
        unsigned polls = 0;
        while (!__all_sync(0xffffffffu, ok)) {
            ++polls;
            if (polls > w.limit || (polls % 1024u == 0 && __any_sync(0xffffffffu, *((volatile int*)&w.sy->err)))) {
                w.lost = true;
                if (w.lane == 0) atomicExch(&w.sy->err, 1);
            }
            if (!ok) {
                load(w, L, t);
                ok = there();
            }
        }
        if (w.a == 0) xj = t < w.lastJ ? f64(march_double(wJ)) : f64(0.0);
        if (w.b == 0) xk = t < w.lastK ? f64(march_double(wK)) : f64(0.0);
        load(w, L, t + 1);
    }
};

// the increment of step t of component L from its right-hand side and diagonal and the neighbours' terms
// (twice the reference's, which halves each: exact, so the half joins the last operation); stored
template <bool LOWER>
__device__ __forceinline__ f64 march64_step(const March64Walk<LOWER>& w, const int L, int t, bool act, f64 own, f64 stept, f64 cvs,
                                            f64 den, f64 xi, f64 xj, f64 xk) {
    const f64 c2 = (xi + xj + xk) * cvs;
    f64 v;
    if (LOWER) v = (act ? fma2(0.5, c2, own * stept) : f64(1.0)) / (act ? den : f64(1.0));
    else v = fma2(-0.5, (act ? c2 : f64(1.0)) / (act ? den : f64(1.0)), own);
    if (act) __stcg(reinterpret_cast<double*>(w.dq + m64_dq(w.q0, L) + (long long)t * w.DQS), v.v);
    return v;
}

// Mean flow.  Warp 0: energy; 1-3: a momentum component, and the density row along direction W - 1,
// whose shares go to warp 4 through shared memory; 4: the density increment, and the copies of the
// inputs.  (46 FP64 instructions a step on the fullest sub-partition; with a warp per
// component and its row, 64.)  in: the stages.
template <bool LOWER>
struct March64Mean {
    March64Walk<LOWER>& w;
    f64 (*in)[M64_MEAN_IN][32];
    f64 (*D)[5][32];
    f64 (*X0)[32];
    unsigned full;                                 // the stages' barriers
    __device__ void copy(int t) const {            // one lane
        if (t >= w.steps) return;
        const int st = t % M64_STAGES;
        const long long q = w.q0 & ~31ll;
        march64_expect(full + 8 * st, M64_MEAN_IN);
        march64_copy(in[st][0], w.rec + m64_rec(q, 0) + (long long)t * w.REC, M64_MEAN_ROWS, full + 8 * st);
        march64_copy(in[st][M64_MEAN_ROWS], w.dq + m64_dq(q, 0) + (long long)t * w.DQS, 5, full + 8 * st);
    }
    // ROLE 0: warp 0, 1: warps 1-3, 2: warp 4
    template <int ROLE>
    __device__ __forceinline__ void run(const int W) {
        constexpr int LJ = MARCH_J;
        const int L = ROLE == 0 ? 4 : ROLE == 1 ? W : 0, lane = w.lane, cell = w.cell;
        March64Edge<LOWER> edge;
        edge.load(w, L, 0);
        if (ROLE == 2 && lane == 0)
            for (int t = 0; t < M64_STAGES - 1; ++t) copy(t);
        f64 ci = f64(0.0), cj = f64(0.0), ck = f64(0.0);       // shares of this lane's last cell
        int st = 0;
        unsigned ph = 0;
        for (int t = 0; t < w.steps; ++t) {
            const f64(*const q)[32] = in[st];
            const bool act = w.active(t);
            f64 xi = ci, xj, xk;
            if constexpr (ROLE == 2) {
                if (t > 0) asm volatile("bar.sync 2, 128;" ::: "memory");      // the density shares of step t - 1
                xi = t > 0 ? X0[0][lane] : f64(0.0);
                xj = t > 0 && w.a > 0 ? X0[1][lane - 1] : f64(0.0);
                xk = t > 0 && w.b > 0 ? X0[2][lane - LJ] : f64(0.0);
            } else {
                xj = f64(__shfl_up_sync(0xffffffffu, cj.v, 1));
                xk = f64(__shfl_up_sync(0xffffffffu, ck.v, LJ));
            }
            march64_phase(w, full + 8 * st, ph, t);
            edge.take(w, L, t, xj, xk);
            const f64 v = march64_step<LOWER>(w, L, t, act, q[M64_MEAN_ROWS + L][cell], q[M64_STEPT][cell], q[M64_CVS][cell],
                                              q[M64_FM][cell], xi, xj, xk);
            D[t & 1][L][lane] = v;
            asm volatile("bar.sync 1, 160;" ::: "memory");
            if constexpr (ROLE == 2) {
                // every warp is past step t - 1: its stage takes the inputs of a later step
                if (lane == 0 && w.stalled < 0) copy(t + M64_STAGES - 1);
            } else {
                f64 A[5];                          // the step's increments of the lane's cell
#pragma unroll
                for (int m = 0; m < 5; ++m) A[m] = D[t & 1][m][lane];
                // rows of the cell's A(Q) DeltaQ with the radius term (TIME_LUSGS.F90:696-768)
                if constexpr (ROLE == 1) {
                    const f64(*const J)[32] = q + (W - 1) * M64_TERMS + JC_R0;
                    const f64 Dif = add_zero_times(add_zero_times(A[1] * J[0][cell], A[0]) + A[2] * J[1][cell] + A[3] * J[2][cell], A[4]);
                    const f64 rv = q[M64_RDS + W - 1][cell] * A[0];
                    const f64 x = act ? (LOWER ? Dif + rv : Dif - rv) : f64(0.0);
                    X0[W - 1][lane] = x;
                    asm volatile("bar.arrive 2, 128;" ::: "memory");
                    if (W == 2) w.put_j(0, t, x);
                    if (W == 3) w.put_k(0, t, x);
                }
                f64 x[3];
#pragma unroll
                for (int dir = 0; dir < 3; ++dir) {
                    const f64(*const J)[32] = q + dir * M64_TERMS + (ROLE == 0 ? 0 : JC_R1 + 5 * (L - 1));
                    auto k = [&](int m) { return J[m][cell]; };
                    f64 Dif;
                    if constexpr (ROLE == 0)
                        Dif = A[0] * k(JC_VP) * k(JC_GET1) + A[1] * k(JC_R4) + A[2] * k(JC_R4 + 1) + A[3] * k(JC_R4 + 2) + A[4] * k(JC_R4 + 3);
                    else
                        Dif = A[0] * k(0) + A[1] * k(1) + A[2] * k(2) + A[3] * k(3) + A[4] * k(4);
                    const f64 rv = q[M64_RDS + dir][cell] * v;
                    x[dir] = LOWER ? Dif + rv : Dif - rv;
                }
                ci = act ? x[0] : f64(0.0);
                cj = act ? x[1] : f64(0.0);
                ck = act ? x[2] : f64(0.0);
                w.put_j(L, t, cj);
                w.put_k(L, t, ck);
            }
            if (++st == M64_STAGES) { st = 0; ph ^= 1u; }
        }
        if constexpr (ROLE == 2) {
            asm volatile("bar.sync 2, 128;" ::: "memory");                         // the last step's arrivals
            if (lane == 0 && w.stalled >= 0) march64_drain(full, min(w.stalled + M64_STAGES - 1, w.steps));
        }
    }
};

// k and omega (L = 5, 6): a warp each, with stages of its own (TURBTWO_TIME_LUSGS_SST.F90:562-766).
template <bool LOWER>
__device__ __forceinline__ void march64_turb(const int L, March64Walk<LOWER>& w, f64 (*in)[M64_TURB_IN][32], unsigned full) {
    const int lane = w.lane, cell = w.cell;
    auto copy = [&](int t) {                       // one lane
        if (t >= w.steps) return;
        const int st = t % M64_STAGES;
        const long long q = w.q0 & ~31ll;
        march64_expect(full + 8 * st, M64_TURB_IN);
        march64_copy(in[st][0], w.rec + m64_rec(q, M64_TURB_ROW0) + (long long)t * w.REC, M64_TURB_IN - 1, full + 8 * st);
        march64_copy(in[st][M64_TURB_IN - 1], w.dq + m64_dq(q, L) + (long long)t * w.DQS, 1, full + 8 * st);
    };
    March64Edge<LOWER> edge;
    edge.load(w, L, 0);
    if (lane == 0)
        for (int t = 0; t < M64_STAGES; ++t) copy(t);
    f64 ci = f64(0.0), cj = f64(0.0), ck = f64(0.0);
    int st = 0;
    unsigned ph = 0;
    for (int t = 0; t < w.steps; ++t) {
        const f64(*const q)[32] = in[st];
        const bool act = w.active(t);
        f64 xj = f64(__shfl_up_sync(0xffffffffu, cj.v, 1)), xk = f64(__shfl_up_sync(0xffffffffu, ck.v, MARCH_J));
        march64_phase(w, full + 8 * st, ph, t);
        f64 vp[3], rds[3];
#pragma unroll
        for (int dir = 0; dir < 3; ++dir) {
            vp[dir] = q[M64_VPT - M64_TURB_ROW0 + dir][cell];
            rds[dir] = q[M64_RDS - M64_TURB_ROW0 + dir][cell];
        }
        const f64 own = q[M64_TURB_IN - 1][cell], stept = q[M64_STEPT - M64_TURB_ROW0][cell], cvs = q[M64_CVS - M64_TURB_ROW0][cell],
                  den = q[M64_FT - M64_TURB_ROW0][cell];
        __syncwarp();                              // the stage is read
        if (lane == 0 && w.stalled < 0) copy(t + M64_STAGES);
        edge.take(w, L, t, xj, xk);
        const f64 v = march64_step<LOWER>(w, L, t, act, own, stept, cvs, den, ci, xj, xk);
        f64 x[3];
#pragma unroll
        for (int dir = 0; dir < 3; ++dir) x[dir] = LOWER ? v * vp[dir] + rds[dir] * v : v * vp[dir] - rds[dir] * v;
        ci = act ? x[0] : f64(0.0);
        cj = act ? x[1] : f64(0.0);
        ck = act ? x[2] : f64(0.0);
        w.put_j(L, t, cj);
        w.put_k(L, t, ck);
        if (++st == M64_STAGES) { st = 0; ph ^= 1u; }
    }
    if (lane == 0 && w.stalled >= 0) march64_drain(full, min(w.stalled + M64_STAGES, w.steps));
}

// A CTA takes the mean flow of a tile, or k and omega of two.  TURB: the components swept, 0 mean flow,
// 1 all (per two tiles three CTAs), 2 k and omega only.
__host__ __device__ inline int march64_ctas(int ntiles, int turb) {
    const int pairs = (ntiles + 1) / 2;
    return turb == 0 ? ntiles : turb == 1 ? 3 * pairs : pairs;
}
constexpr size_t march64_bytes(int turb) { return (turb == 2 ? 4 * M64_TURB_IN : M64_MEAN_IN) * M64_STAGES * 32 * sizeof(f64); }
template <bool LOWER, int TURB>
__global__ void __launch_bounds__(160, 4)
k_march64(const MarchTile* __restrict__ tiles, int ntiles, const f64* __restrict__ rec, f64* dq, ulonglong2* bufJ, ulonglong2* bufK,
          MarchCtl* ctl, SweepSync* sy, unsigned limit) {
    constexpr int side = LOWER ? 0 : 1;
    extern __shared__ __align__(128) f64 inputs[];
    __shared__ f64 D[2][5][32], X0[3][32];
    __shared__ __align__(8) unsigned long long bars[4][M64_STAGES];       // of the mean flow, or of each k and omega warp
    __shared__ unsigned ticket_s;
    if (threadIdx.x == 0) {
        ticket_s = atomicAdd(&ctl->ticket[side], 1u);
        for (int n = 0; n < 4 * M64_STAGES; ++n) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(march64_smem(&bars[0][0] + n)) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    const int ticket = (int)ticket_s, W = threadIdx.x >> 5;
    const unsigned epoch = *((volatile unsigned*)&ctl->epoch);
    const unsigned tag = 2u * epoch + 1u + side;
    const bool turb = TURB == 2 || (TURB == 1 && ticket % 3 == 2);
    int n = TURB == 0 ? ticket : TURB == 1 ? ticket / 3 * 2 + ticket % 3 : 2 * ticket;
    if (turb) n = (TURB == 1 ? ticket / 3 * 2 : 2 * ticket) + (W >> 1);
    if (n < ntiles && !(turb && W == 4)) {
        const MarchTile T = tiles[LOWER ? n : ntiles - 1 - n];
        March64Walk<LOWER> w(T, rec, dq, bufJ, bufK, tag, sy, limit);
        if (TURB != 0 && turb) {
            march64_turb<LOWER>(5 + (W & 1), w, reinterpret_cast<f64(*)[M64_TURB_IN][32]>(inputs) + W * M64_STAGES,
                                march64_smem(bars[W]));
        } else if (TURB != 2) {
            March64Mean<LOWER> m{w, reinterpret_cast<f64(*)[M64_MEAN_IN][32]>(inputs), D, X0, march64_smem(bars[0])};
            if (W == 0) m.template run<0>(W);
            else if (W < 4) m.template run<1>(W);
            else m.template run<2>(W);
        }
    }
    __syncthreads();
    // the last CTA of the sweep makes the counters ready for the next one
    if (threadIdx.x == 0 && atomicAdd(&ctl->done[side], 1u) == (unsigned)gridDim.x - 1u) {
        ctl->ticket[side] = 0;
        ctl->done[side] = 0;
        if (!LOWER) ctl->epoch = epoch + 1u;
    }
}

// The cells' Jacobian terms and radii into the records, one warp per M64_JAC_STEPS steps of a tile: a step
// is 156 FP64 instructions, so warps of eight steps left the smallest blocks waiting (with prep, 24x16x5
// cells: 108 us, and 53 with two); consecutive steps of a lane read consecutive cells of its line
static __global__ void __launch_bounds__(128) k_march64_jac(const DevBlock* __restrict__ blks, const MarchTile* __restrict__ tiles,
                                                            const int2* __restrict__ runs, int nruns, f64* __restrict__ rec) {
    const int g = (blockIdx.x * 128 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (g >= nruns) return;
    const int2 run = runs[g];                      // tile, first step
    const MarchTile T = tiles[run.x];
    const DevBlock b = blks[T.blk];
    const int aj = lane % MARCH_J, ak = lane / MARCH_J;
    const int steps = T.NI1 + MARCH_J + MARCH_K - 2;
    const size_t nc = (size_t)b.ncell;
    for (int t = run.y; t < min(run.y + M64_JAC_STEPS, steps); ++t) {
        const int i = t - aj - ak;                 // 0-based
        if (aj >= T.nj || ak >= T.nk || (unsigned)i >= (unsigned)T.NI1) continue;
        const int c = cidx(b, i + 1, T.j0 + aj, T.k0 + ak);
        const f64* sv = rs<f64>(b, S_SVEL);
        const f64 u = sv[c], v = sv[c + nc], w = sv[c + 2 * nc], pp = rs<f64>(b, S_PP)[c], ri = rs<f64>(b, S_RINV)[c];
        f64* o = rec + m64_rec((long long)(T.s0 + t) * 32 + lane, 0);
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            const f64* asd = rs<f64>(b, S_ASD + 3 * d);
            f64 J[NJAC];
            jac_terms<f64>(u, v, w, asd[c], asd[c + nc], asd[c + 2 * nc], pp, ri, J);
#pragma unroll
            for (int m = 0; m < M64_TERMS; ++m) o[(d * M64_TERMS + m) * 32] = J[m];
            o[(M64_VPT + d) * 32] = J[JC_VPT];
            o[(M64_RDS + d) * 32] = rs<f64>(b, S_RDS + d)[c];
        }
    }
}

}  // namespace tg
