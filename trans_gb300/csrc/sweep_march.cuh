// sweep_march.cuh -- mixed-path LU-SGS sweeps as marching warps (schedule 6).
//
// The hyperplane launches pay a launch and a dependent L2 round trip per plane or two (2.4 us)
// for a few nanoseconds of arithmetic.  Here a warp owns a column of MARCH_J x MARCH_K lines in
// (j, k) and walks it along i, skewed by a + b for lane (a, b), so that at every step its lanes
// are on one i+j+k hyperplane: the i-neighbour is the lane's own previous result, the j- and
// k-neighbours are the previous results of lanes a-1 and b-1 (through shared memory), and only the
// first lane of a row or column needs a value from the neighbouring tile.  Those cross tiles
// through L2 as 64-bit words that carry a float and the tag of this sweep, so a reader polls the
// data itself: no flag, no fence, no launch and no grid barrier per plane.  A tile runs a few
// steps behind its neighbours and all of them stream.  Records and right-hand sides are stored in
// the order of the march, so a step's inputs are one contiguous range, copied MARCH_STAGES - 1
// steps ahead.
//
// What passes to a neighbour is this cell's share of the neighbour's sum (sweep_share), formed
// with the expressions of sweep_core, so every DeltaQ keeps its bits.
//
// Both sweeps of an iteration, against the best hyperplane schedule: benchmark cascade (1,966,080
// cells) 0.304 ms against 0.893; channel 97x49x9 0.097 against 0.246.  A lone tile takes 0.22 us a
// step, bound by the chain through shared memory, two barriers and ~12 dependent operations; a
// column of tiles adds ~1 us a tile (a store and a polled load through L2).
//
// Progress: tiles are numbered so that a tile only waits for lower numbers in the lower sweep
// (higher in the upper one), and a CTA takes its tile from a counter in that order, so every
// tile waited for is finished or running.  A wait for a tile is bounded: after `limit` polls the
// warp records the error and the tile goes on without the words.
#pragma once
#include "kernels.cuh"
#include "march_words.cuh"

namespace tg {

__device__ __forceinline__ void march_copy16(void* smem, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g) : "memory");
}

// The share of a cell with metric and radius g, velocity and enthalpy h and increment a in the
// sum of its neighbour along one direction: words 0-4 its mean-flow rows, word 5 the factor of
// the k and omega increments, words 6 and 7 (sweep_core's acc[] terms).
template <bool LOWER>
__device__ __forceinline__ void sweep_share(float4 g, float4 h, const float a[7], float c[8]) {
    const float sgn = LOWER ? 1.0f : -1.0f;
    const float Gm1 = 0.4f;
    const float sx = g.x, sy = g.y, sz = g.z, sr = sgn * g.w;
    const float u = h.x, v = h.y, w = h.z, H = h.w;
    const float vp = h.x * g.x + h.y * g.y + h.z * g.z;
    const float q2 = 0.5f * (h.x * h.x + h.y * h.y + h.z * h.z);
    const float sm = sx * a[1] + sy * a[2] + sz * a[3];
    const float th = sm - vp * a[0];
    const float ph = Gm1 * (q2 * a[0] - (u * a[1] + v * a[2] + w * a[3]) + a[4]);
    c[0] = sm + sr * a[0];
    c[1] = u * th + sx * ph + (vp + sr) * a[1];
    c[2] = v * th + sy * ph + (vp + sr) * a[2];
    c[3] = w * th + sz * ph + (vp + sr) * a[3];
    c[4] = H * th + vp * (ph + a[4]) + sr * a[4];
    c[5] = vp + sr;
    c[6] = a[5];
    c[7] = a[6];
}

// Named barriers between two warps of a tile: one arrives, the other waits for it (and for its
// accesses to shared memory before).  A wait costs ~25 cycles of a step; mbarrier waits took ~100,
// counters in shared memory a fence that waited for the global stores before it.
__device__ __forceinline__ void march_arrive(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void march_await(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
constexpr int MB_COPIED = 1, MB_SWEPT = 3, MB_FREE = 5, MB_EDGED = 7;    // 2, 2, 2 and MARCH_STAGES of them, in turn

// TURB as sweep_core's turb: 0 mean flow, 1 all, 2 k and omega only.
// Warp 0 sweeps.  Warp 1 copies its inputs ahead and hands its edge shares on to the next tiles.
// Warp 2 polls the neighbouring tiles' edge words and brings them to shared memory.  (In one warp a
// word loaded ahead of its use shared its scoreboard with the loads issued after it, so that every
// step waited a full L2 round trip for the newest of them.)
template <bool LOWER, int TURB>
__global__ void __launch_bounds__(96) k_sweep_march(const MarchTile* __restrict__ tiles, int ntiles, const float* __restrict__ rec,
                                                    float* dq, ulonglong2* bufJ, ulonglong2* bufK, MarchCtl* ctl, SweepSync* sy,
                                                    unsigned limit) {
    constexpr int S = MARCH_STAGES;                // stages of the inputs and of the edge words
    constexpr int side = LOWER ? 0 : 1;
    constexpr int LJ = MARCH_J, LK = MARCH_K;
    // records and right-hand sides of a step's cells, in the lower sweep's lane order
    __shared__ float4 ring[S][32][5], dring[S][32][2];
    // shares of a step for the next one, words 0-3 and 4-7: [parity][half][lane b, a + 1] for the
    // j-neighbour and [b + 1, a] for the k-neighbour; the first of a row comes from the edge words
    __shared__ float4 xj[2][2][LK][LJ + 1], xk[2][2][LK + 1][LJ];
    __shared__ float4 ej[S][2][LK], ek[S][2][LJ];
    __shared__ unsigned ticket_s;
    const int lane = threadIdx.x & 31, role = threadIdx.x >> 5;
    if (threadIdx.x == 0) ticket_s = atomicAdd(&ctl->ticket[side], 1u);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int n = threadIdx.x; n < 4 * LK * (LJ + 1); n += 96) (&xj[0][0][0][0])[n] = zero;
    for (int n = threadIdx.x; n < 4 * (LK + 1) * LJ; n += 96) (&xk[0][0][0][0])[n] = zero;
    for (int n = threadIdx.x; n < S * 2 * LK; n += 96) (&ej[0][0][0])[n] = zero;
    for (int n = threadIdx.x; n < S * 2 * LJ; n += 96) (&ek[0][0][0])[n] = zero;
    __syncthreads();
    const unsigned ticket = ticket_s;
    const unsigned epoch = *((volatile unsigned*)&ctl->epoch);
    const unsigned tag = 2u * epoch + 1u + side;
    const MarchTile T = tiles[LOWER ? ticket : ntiles - 1 - ticket];
    const int steps = T.NI1 + (LJ - 1) + (LK - 1);
    const int srcK = T.sK[side], srcJ = T.sJ[side];
    const int lastK = srcK >= 0 ? steps - (LK - 1) : 0, lastJ = srcJ >= 0 ? steps - (LJ - 1) : 0;   // steps with an edge
    const int edges = max(lastK, lastJ);
    // lane l carries word pair l / 8 of lane (l % 8, 0)'s k-share and, below 16, l / 4 of lane (0, l % 4)'s
    // j-share; a tile writes all its words at every step (zeros outside the block)
    const int mK = lane >> 3, mJ = (lane >> 2) & 3;
    // storage step of step t (the upper sweep walks backwards, with lane l at the lower one's lane 31 - l)
    auto stored = [&](int t) { return (size_t)(T.s0 + (LOWER ? t : steps - 1 - t)) * 32; };

    if (role == 0) {
        const int a = lane % LJ, b = lane / LJ, cell = LOWER ? lane : 31 - lane;
        const bool in_jk = cell % LJ < T.nj && cell / LJ < T.nk;
        float ci[8];                               // share of this lane's last cell for its i-neighbour
#pragma unroll
        for (int m = 0; m < 8; ++m) ci[m] = 0.0f;
        float4* W4 = reinterpret_cast<float4*>(dq) + (stored(0) + cell) * 2;
        for (int t = 0; t < steps; ++t) {
            const int st = t % S, par = t & 1;
            march_await(MB_COPIED + par);
            const float4 *const R = ring[st][cell], *const D = dring[st][cell];
            const float4 g0 = R[0], g1 = R[1], g2 = R[2], h = R[3], dg = R[4], o0 = D[0], o1 = D[1];
            if (t < edges) march_await(MB_EDGED + st);
            const float4* const pj = a == 0 ? &ej[st][0][b] : &xj[par][0][b][a];
            const float4* const pk = b == 0 ? &ek[st][0][a] : &xk[par][0][b][a];
            const float4 j0 = pj[0], j1 = pj[a == 0 ? LK : LK * (LJ + 1)];
            const float4 k0 = pk[0], k1 = pk[b == 0 ? LJ : (LK + 1) * LJ];
            const bool active = in_jk && (unsigned)(t - a - b) < (unsigned)T.NI1;
            float acc[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            auto add = [&](const float4& x, const float4& y) {
                acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w; acc[4] += y.x;
                acc[5] += y.y * y.z;
                acc[6] += y.y * y.w;
            };
            add(make_float4(ci[0], ci[1], ci[2], ci[3]), make_float4(ci[4], ci[5], ci[6], ci[7]));
            add(j0, j1);
            add(k0, k1);
            const float own[7] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z};
            const float stept = dg.x, hc = 0.5f * dg.y;
            float out[7];
#pragma unroll
            for (int L = 0; L < 7; ++L) {
                const float iden = L < 5 ? dg.z : dg.w;
                const bool act = TURB == 1 || (TURB == 0 ? L < 5 : L >= 5);
                const float nv = LOWER ? (own[L] * stept + acc[L] * hc) * iden : own[L] - acc[L] * hc * iden;
                out[L] = active ? (act ? nv : own[L]) : 0.0f;       // outside the block: no share
            }
            float cj[8], ck[8];
            sweep_share<LOWER>(g1, h, out, cj);
            sweep_share<LOWER>(g2, h, out, ck);
            xj[par ^ 1][0][b][a + 1] = make_float4(cj[0], cj[1], cj[2], cj[3]);
            xj[par ^ 1][1][b][a + 1] = make_float4(cj[4], cj[5], cj[6], cj[7]);
            xk[par ^ 1][0][b + 1][a] = make_float4(ck[0], ck[1], ck[2], ck[3]);
            xk[par ^ 1][1][b + 1][a] = make_float4(ck[4], ck[5], ck[6], ck[7]);
            march_arrive(MB_SWEPT + par);
            if ((t & 3) == 3 && t < edges) march_arrive(MB_FREE + ((t >> 2) & 1));   // the edge stages of these four steps
            __syncwarp();
            sweep_share<LOWER>(g0, h, out, ci);
            if (active) {
                __stcg(W4, make_float4(out[0], out[1], out[2], out[3]));
                __stcg(W4 + 1, make_float4(out[4], out[5], out[6], o1.w));
            }
            W4 += LOWER ? 64 : -64;
        }
    } else if (role == 1) {
        auto fetch = [&](int t) {
            if (t < steps) {
                const float4* const r = reinterpret_cast<const float4*>(rec) + stored(t) * (NCREC / 4) + lane;
                const float4* const d = reinterpret_cast<const float4*>(dq) + stored(t) * 2 + lane;
#pragma unroll
                for (int m = 0; m < 5; ++m) march_copy16(&ring[t % S][0][0] + m * 32 + lane, r + m * 32);
#pragma unroll
                for (int m = 0; m < 2; ++m) march_copy16(&dring[t % S][0][0] + m * 32 + lane, d + m * 32);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        const bool outK = T.sK[1 - side] >= 0, outJ = T.sJ[1 - side] >= 0 && lane < 16;
        const float2* const fK = reinterpret_cast<const float2*>(&xk[0][mK >> 1][LK][lane & 7]) + (mK & 1);
        const float2* const fJ = reinterpret_cast<const float2*>(&xj[0][mJ >> 1][lane & 3][LJ]) + (mJ & 1);
        ulonglong2* wrK = bufK + ((size_t)T.s0 * 4 + mK) * LJ + (lane & 7);
        ulonglong2* wrJ = bufJ + ((size_t)T.s0 * 4 + mJ) * LK + (lane & 3);
        // the shares of step t, before warp 0 can end step t + 2 (it then waits for MB_COPIED of step t + 2)
        auto hand_on = [&](int t) {
            march_await(MB_SWEPT + (t & 1));
            const int par = (t + 1) & 1;
            if (outK) {
                const float2 w = fK[par * (int)(sizeof(xk[0]) / sizeof(float2))];
                march_st(wrK, w.x, w.y, tag);
            }
            if (outJ) {
                const float2 w = fJ[par * (int)(sizeof(xj[0]) / sizeof(float2))];
                march_st(wrJ, w.x, w.y, tag);
            }
            wrK += 4 * LJ;
            wrJ += 4 * LK;
        };
        for (int t = 0; t < S - 1; ++t) fetch(t);
        for (int n = 0; n < steps; ++n) {
            asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
            march_arrive(MB_COPIED + (n & 1));
            if (n > 0) hand_on(n - 1);             // step n - 1 is swept: its stage is free
            fetch(n + S - 1);
        }
        hand_on(steps - 1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        const ulonglong2* const pK = bufK + ((size_t)(srcK + LK - 1) * 4 + mK) * LJ + (lane & 7);
        const ulonglong2* const pJ = bufJ + ((size_t)(srcJ + LJ - 1) * 4 + mJ) * LK + (lane & 3);
        bool lost = false;                         // given up: the remaining steps go on without the words
        for (int q = 0; q < edges; q += 4) {       // four steps polled at a time
            if (q >= S) march_await(MB_FREE + ((q >> 2) & 1));     // warp 0 has used the words of steps q - 8 .. q - 5
            unsigned polls = 0;
            int v = 0;                             // leading steps whose words are all there
            const int m = min(4, edges - q);
            while (v < m) {
                ulonglong2 wK[4], wJ[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    wK[u] = wJ[u] = make_ulonglong2(0, 0);
                    if (u >= v && q + u < lastK) wK[u] = march_ld(pK + (q + u) * 4 * LJ);
                    if (u >= v && q + u < lastJ && lane < 16) wJ[u] = march_ld(pJ + (q + u) * 4 * LK);
                }
                const int v0 = v;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    auto good = [&](const ulonglong2& w) { return (unsigned)(w.x >> 32) == tag && (unsigned)(w.y >> 32) == tag; };
                    const bool ok = lost || ((q + u >= lastK || good(wK[u])) && (q + u >= lastJ || lane >= 16 || good(wJ[u])));
                    if (v == u && u < m && __all_sync(0xffffffffu, ok)) {
                        v = u + 1;
                        const int st = (q + u) % S;
                        if (q + u < lastK)
                            (reinterpret_cast<float2*>(&ek[st][mK >> 1][lane & 7]))[mK & 1] = make_float2(__uint_as_float((unsigned)wK[u].x), __uint_as_float((unsigned)wK[u].y));
                        if (q + u < lastJ && lane < 16)
                            (reinterpret_cast<float2*>(&ej[st][mJ >> 1][lane & 3]))[mJ & 1] = make_float2(__uint_as_float((unsigned)wJ[u].x), __uint_as_float((unsigned)wJ[u].y));
                        march_arrive(MB_EDGED + st);
                    }
                }
                polls = v > v0 ? 0 : polls + 1;
                if (polls > limit || (polls && polls % 1024u == 0 && __any_sync(0xffffffffu, *((volatile int*)&sy->err)))) {
                    lost = true;                   // the same for every lane
                    if (lane == 0) atomicExch(&sy->err, 1);
                }
            }
        }
        // the arrivals of the last quads that nothing above waited for
        for (int q = max(S, (edges + 3) / 4 * 4); (q - S) + 3 < edges; q += 4) march_await(MB_FREE + ((q >> 2) & 1));
    }
    __syncthreads();
    // the last tile of the sweep makes the counters ready for the next one
    if (threadIdx.x == 0 && atomicAdd(&ctl->done[side], 1u) == (unsigned)ntiles - 1u) {
        ctl->ticket[side] = 0;
        ctl->done[side] = 0;
        if (!LOWER) ctl->epoch = epoch + 1u;
    }
}

}  // namespace tg
