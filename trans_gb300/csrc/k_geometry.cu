// k_geometry.cu -- GEOM_CalcDST (Geom/CalcDst.F90:28-719) on the device: the wall distance
// (:127-164) and the per-cell and per-face metrics of one block.
//
// Wall distance.
//
// The reference computes, for every interior cell centre, the squared distance
// DDD = Dx*Dx + Dy*Dy + Dz*Dz to the centre of every panel of every wall surface (panel centre =
// the average of its 4 nodes), keeps the minimum per surface (Dst_minN), combines the surfaces
// in order as  d = max(d, tiny); if (Dst_minN < d) d = Dst_minN  (starting from d = 1e20), and
// stores sqrt(d).  That is O(cells x panels): 8.8e11 pairs for a 5.7 M-cell cascade.
//
// Here each surface is scanned twice per cell in FP32 (the FP32 pipe is 58x the FP64 pipe on
// GB300): pass A finds the FP32 minimum m of the squared distances; pass B evaluates the
// reference's FP64 expression only for the panels whose FP32 squared distance is within
// (sqrt(m)(1 + 1e-5) + 2 Eabs)^2 (1 + 1e-5) of it, where Eabs = 1e-6 R bounds the error of an
// FP32 distance (coordinates rounded to FP32: 2^-24 |x| each, |x| <= R <= 1e18, three
// components; 1e-37 floor for subnormal FP32) and the relative slack covers the FP32 arithmetic.  The panel that minimises the FP64 DDD has an
// FP32 distance within 2 Eabs (+ the relative slack) of the FP32 minimum, so it is always
// evaluated, and the minimum of the evaluated FP64 values is the reference's Dst_minN exactly.
// Both passes leave out the chunks of panels (8 x 8 of a surface) that cannot matter: the FP32 distance to
// a chunk's bounding box, formed like the panels' with each coordinate's difference replaced by the
// gap to the box, is no larger than any of theirs (rounding is monotonic), so a chunk at or beyond the
// minimum so far, or beyond the candidates' limit, is passed over without a panel missed.
//
// Where panels are dense the limit of pass B lets dozens through, so a panel within it is measured again
// in FP32, on differences of coordinates split into two floats: sqrt(r) is within 5e-7 of the distance
// plus 2^-44 R (each difference within 2^-23 of itself and 2^-45 R, three products and sums).  Hence the
// panel of the FP64 minimum has sqrt(r) <= sqrt(rm)(1 + 1.1e-6) + 2.1 x 2^-44 R, with rm the smallest r,
// and only those within sqrt(rm)(1 + 1e-5) + 4e-13 R get the FP64 expression (all, should rm be below
// 1e-30, where FP32 squares near their smallest values).
// The FP64 arithmetic is compiled without contraction (-fmad=false), so the result is
// bit-identical to a sequential CPU evaluation of the reference's loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <memory>
#include <vector>

#include "../../include/trans_gpu.h"

namespace tg {

thread_local std::string g_stateless_err;
namespace eng {
const char* stateless_error() { return g_stateless_err.c_str(); }
}  // namespace eng

namespace {

constexpr int WD_THREADS = 256;
constexpr int WD_CHUNK = 8;               // panels of a chunk along each direction of its surface
struct WallChunk {                        // bounding box of panels first .. first + n - 1
    float lo[3];
    int n;
    float hi[3];
    int pad_;
    long long first, pad2_;
};

constexpr int WD_CAND = 8;                // candidates per surface held for the converged FP64 pass

// the reference's DDD (Geom/CalcDst.F90:150-155), in its order
__device__ __forceinline__ double ddd64(double px, double py, double pz, const double* __restrict__ q) {
    const double Dx = px - q[0], Dy = py - q[1], Dz = pz - q[2];
    return Dx * Dx + Dy * Dy + Dz * Dz;
}

__device__ __forceinline__ float d2f(float fx, float fy, float fz, float4 q) {
    const float dx = fx - q.x, dy = fy - q.y, dz = fz - q.z;
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
}

// the FP32 distance squared to a chunk's box: d2f of the nearest point
__device__ __forceinline__ float box2f(float fx, float fy, float fz, float4 lo, float4 hi) {
    const float gx = fmaxf(fmaxf(lo.x - fx, fx - hi.x), 0.0f), gy = fmaxf(fmaxf(lo.y - fy, fy - hi.y), 0.0f);
    const float gz = fmaxf(fmaxf(lo.z - fz, fz - hi.z), 0.0f);
    return __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, gx * gx));
}

// the FP32 distance squared from coordinates split into two floats
__device__ __forceinline__ float fine2f(float fx, float fy, float fz, float lx, float ly, float lz, float4 q, float4 ql) {
    const float dx = (fx - q.x) + (lx - ql.x), dy = (fy - q.y) + (ly - ql.y), dz = (fz - q.z) + (lz - ql.z);
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, dx * dx));
}

// and between two boxes, no larger than that of any two points in them
__device__ __forceinline__ float boxes2f(float3 a, float3 b, float4 lo, float4 hi) {
    const float gx = fmaxf(fmaxf(lo.x - b.x, a.x - hi.x), 0.0f), gy = fmaxf(fmaxf(lo.y - b.y, a.y - hi.y), 0.0f);
    const float gz = fmaxf(fmaxf(lo.z - b.z, a.z - hi.z), 0.0f);
    return __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, gx * gx));
}
template <bool MAX>
__device__ __forceinline__ float warp_extreme(float x) {
    for (int w = 16; w > 0; w >>= 1) {
        const float y = __shfl_xor_sync(0xffffffffu, x, w);
        x = MAX ? fmaxf(x, y) : fminf(x, y);
    }
    return x;
}

// Points in the caller's order may lie anywhere, and a warp whose points lie far apart meets most chunks and scans
// what any lane needs.  So they are grouped by the cell of a 2^b x 2^b x 2^b grid over their box, in
// Morton order: index idx[c] of the c-th (within a cell in any order: a point's result does not depend on its
// warp).
struct PointGrid { double lo[3], scale[3]; int bits; };
__device__ __forceinline__ unsigned point_bin(const PointGrid& g, const double* x) {
    unsigned key = 0;
    for (int m = 0; m < 3; ++m) {
        const double t = (x[m] - g.lo[m]) * g.scale[m];
        const unsigned q = (unsigned)fmin(fmax(t, 0.0), (double)((1 << g.bits) - 1));
        for (int b = 0; b < g.bits; ++b) key |= (q >> b & 1u) << (3 * b + m);
    }
    return key;
}
__global__ void k_point_count(unsigned n, const double* __restrict__ pts, PointGrid g, unsigned* __restrict__ bins) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < n) atomicAdd(bins + point_bin(g, pts + 3 * (size_t)c), 1u);
}
// counts into first places, one CTA of 1,024 threads, each with a run of bins in 16-byte words, many in flight
// (2^15 bins one by one took 51 us, as long as the search of 200,000 points on a small surface)
__global__ void __launch_bounds__(1024) k_point_scan(unsigned* __restrict__ bins, unsigned nbins) {
    __shared__ unsigned warp_sum[32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned words = nbins / 4, per = (words + 1023) / 1024, b0 = min(threadIdx.x * per, words), b1 = min(b0 + per, words);
    uint4* const v = reinterpret_cast<uint4*>(bins);
    unsigned sum = 0;
#pragma unroll 8
    for (unsigned b = b0; b < b1; ++b) {
        const uint4 c = v[b];
        sum += c.x + c.y + c.z + c.w;
    }
    unsigned at = sum;                             // inclusive over the warp, then over the warps
    for (int w = 1; w < 32; w <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, at, w);
        if (lane >= (unsigned)w) at += y;
    }
    if (lane == 31) warp_sum[warp] = at;
    __syncthreads();
    if (warp == 0) {
        unsigned x = warp_sum[lane];
        for (int w = 1; w < 32; w <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, w);
            if (lane >= (unsigned)w) x += y;
        }
        warp_sum[lane] = x;
    }
    __syncthreads();
    unsigned place = at - sum + (warp ? warp_sum[warp - 1] : 0u);
#pragma unroll 8
    for (unsigned b = b0; b < b1; ++b) {
        const uint4 c = v[b];
        const uint4 first = make_uint4(place, place + c.x, place + c.x + c.y, place + c.x + c.y + c.z);
        v[b] = first;
        place = first.w + c.w;
    }
}
__global__ void k_point_place(unsigned n, const double* __restrict__ pts, PointGrid g, unsigned* __restrict__ bins,
                              unsigned* __restrict__ idx) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < n) idx[atomicAdd(bins + point_bin(g, pts + 3 * (size_t)c), 1u)] = c;
}

// One thread per point, a warp's points together: its lanes first test 32 chunks at a time against the box
// of the warp's points, then each of those left against the points, and scan its panels where a lane
// needs them; panel loads have one address in all lanes.  Bound by the issue of FP32 instructions
// and the latency of the chunk loops (issue 55% busy): the coarse O-block, 208,896 cells and 26,368 panels,
// 5.65 ms with every panel scanned, 3.5 with the chunks but warps along lines, 0.69 with a warp's points a brick.
// ONE: a warp per point, its lanes over a chunk's panels; no points of its own to wait for, so a few points
// take the time of one (64 points on 26,368 panels 0.39 ms the whole call, 2.4 a lane per point).
template <bool ONE>
__global__ void __launch_bounds__(WD_THREADS)
k_wall_distance(long long n, const double* __restrict__ pts, const unsigned* __restrict__ idx, const float4* __restrict__ pan32, const float4* __restrict__ pan_lo,
                const double* __restrict__ pan64, const WallChunk* __restrict__ chunks, const int* __restrict__ coff, int nsurf, float eabs, double tiny,
                double* __restrict__ dst) {
    const unsigned full = 0xffffffffu;
    const long long place = ((long long)blockIdx.x * WD_THREADS + threadIdx.x) >> (ONE ? 5 : 0);
    const bool live = place < n;
    const long long c = idx && live ? idx[place] : place;
    const double px = live ? pts[3 * c] : 0.0, py = live ? pts[3 * c + 1] : 0.0, pz = live ? pts[3 * c + 2] : 0.0;
    const float fx = (float)px, fy = (float)py, fz = (float)pz;
    const float lx = (float)(px - (double)fx), ly = (float)(py - (double)fy), lz = (float)(pz - (double)fz);
    // the box of the warp's points, and one of them
    const int lane = threadIdx.x & 31;
    const float big = INFINITY;
    const float3 wlo = {warp_extreme<false>(live ? fx : big), warp_extreme<false>(live ? fy : big), warp_extreme<false>(live ? fz : big)};
    const float3 whi = {warp_extreme<true>(live ? fx : -big), warp_extreme<true>(live ? fy : -big), warp_extreme<true>(live ? fz : -big)};
    const unsigned alive = __ballot_sync(full, live);
    const int mid = (alive >> 16) & 1u ? 16 : 0;
    const float mx = __shfl_sync(full, fx, mid), my = __shfl_sync(full, fy, mid), mz = __shfl_sync(full, fz, mid);
    double d = 1.0e20;
    for (int s = 0; s < nsurf; ++s) {
        const int k0 = coff[s], k1 = coff[s + 1];
        auto box = [&](int k) {
            const float4* w = reinterpret_cast<const float4*>(chunks + k);
            return box2f(fx, fy, fz, __ldg(w), __ldg(w + 1));
        };
        // f(k) for the chunks whose distance to the warp's box is at most that of the farthest reach
        auto near_chunks = [&](auto&& reach, auto&& f) {
            for (int k = k0; k < k1; k += 32) {
                const float far2 = ONE ? reach() : warp_extreme<true>(live ? reach() : 0.0f);
                const float4* w = reinterpret_cast<const float4*>(chunks + min(k + lane, k1 - 1));
                unsigned left = __ballot_sync(full, k + lane < k1 && boxes2f(wlo, whi, __ldg(w), __ldg(w + 1)) <= far2);
                for (; left; left &= left - 1) f(k + __ffs(left) - 1);
            }
        };
        float m = INFINITY, m1 = INFINITY;     // two chains of minima
        auto scan = [&](int k) {
            const float4* q = pan32 + chunks[k].first;
            const int cnt = chunks[k].n;
            if constexpr (ONE) {
                for (int r = lane; r < cnt; r += 32) m = fminf(m, d2f(fx, fy, fz, __ldg(q + r)));
                m = warp_extreme<false>(m);
                return;
            }
            int r = 0;
#pragma unroll 4
            for (; r + 1 < cnt; r += 2) {
                m = fminf(m, d2f(fx, fy, fz, __ldg(q + r)));
                m1 = fminf(m1, d2f(fx, fy, fz, __ldg(q + r + 1)));
            }
            if (r < cnt) m = fminf(m, d2f(fx, fy, fz, __ldg(q + r)));
            m = fminf(m, m1);
        };
        // pass A: FP32 minimum over the surface, from the chunk nearest to one of the points on
        float near2 = INFINITY;
        int nearest = k0;
        for (int k = k0 + lane; k < k1; k += 32) {
            const float4* w = reinterpret_cast<const float4*>(chunks + k);
            const float b = box2f(mx, my, mz, __ldg(w), __ldg(w + 1));
            if (b < near2) { near2 = b; nearest = k; }
        }
        for (int w = 16; w > 0; w >>= 1) {
            const float b = __shfl_xor_sync(full, near2, w);
            const int k = __shfl_xor_sync(full, nearest, w);
            if (b < near2 || (b == near2 && k < nearest)) { near2 = b; nearest = k; }
        }
        if (k0 < k1) scan(nearest);
        near_chunks([&] { return m; }, [&](int k) {
            if (k != nearest && __any_sync(full, live && box(k) < m)) scan(k);
        });
        const float sm = sqrtf(m);
        const float bd = __fmaf_rn(sm, 1.0e-5f, sm) + 2.0f * eabs;
        const float thr = bd * bd * (1.0f + 1.0e-5f);
        // pass B: collect the candidates, then evaluate the reference's FP64 expression for them
        // with the warp's lanes together (a candidate found by one lane alone would otherwise
        // cost the whole warp's FP64 issue slots); a lane with more than WD_CAND candidates
        // evaluates the extra ones at once
        double a = 1.0e20;
        long long cand[WD_CAND];
        float cr[WD_CAND];
        int nc = 0;
        float rm = INFINITY, lim = INFINITY;
        auto take = [&](long long p) {
            const float r = fine2f(fx, fy, fz, lx, ly, lz, __ldg(pan32 + p), __ldg(pan_lo + p));
            if (!(r <= lim)) return;
            if (r < rm) {
                rm = r;
                const float sr = sqrtf(rm), br = __fmaf_rn(sr, 1.0e-5f, sr) + 4.0e-7f * eabs;      // eabs = 1e-6 R
                if (rm >= 1.0e-30f) lim = br * br * (1.0f + 1.0e-5f);
            }
            if (nc == WD_CAND) {               // drop those beyond the limit by now
                int kept = 0;
                for (int j = 0; j < WD_CAND; ++j)
                    if (cr[j] <= lim) { cand[kept] = cand[j]; cr[kept] = cr[j]; ++kept; }
                nc = kept;
            }
            if (nc < WD_CAND) {
                cand[nc] = p;
                cr[nc++] = r;
            } else {
                const double DDD = ddd64(px, py, pz, pan64 + 3 * p);
                if (DDD < a) a = DDD;
            }
        };
        near_chunks([&] { return thr; }, [&](int k) {
            if (!__any_sync(full, live && box(k) <= thr)) return;
            const long long p0 = chunks[k].first;
            const int cnt = chunks[k].n;
#pragma unroll 4
            for (int r = ONE ? lane : 0; r < cnt; r += ONE ? 32 : 1)
                if (d2f(fx, fy, fz, __ldg(pan32 + p0 + r)) <= thr) take(p0 + r);
        });
        // the candidates within the final limit, gathered to the front
        int kept = 0;
        for (int j = 0; j < nc; ++j)
            if (cr[j] <= lim) cand[kept++] = cand[j];
        __syncwarp();
        for (int j = 0; __any_sync(full, j < kept); ++j) {
            if (j < kept) {
                const double DDD = ddd64(px, py, pz, pan64 + 3 * cand[j]);
                if (DDD < a) a = DDD;
            }
        }
        if constexpr (ONE) {             // (values that are not negative, in the order of their bits)
            long long v = __double_as_longlong(a);
            for (int w = 16; w > 0; w >>= 1) v = min(v, __shfl_xor_sync(full, v, w));
            a = __longlong_as_double(v);
        }
        if (d < tiny) d = tiny;          // amax1(dst_minimum, tiny)
        if (a < d) d = a;
    }
    if (live && (!ONE || lane == 0)) dst[c] = sqrt(d);
}

// ---------------------------------------------------------------------------------------
// Block metrics (Geom/CalcDst.F90:95-521).  Arrays are ghost-padded (NI+5)(NJ+5)(NK+5), index
// -2..N+2 per direction; nodes are X, Y, Z of NI x NJ x NK, I fastest.  Every expression keeps
// the reference's operation order (no contraction), so the results equal a CPU evaluation.
// ---------------------------------------------------------------------------------------
struct Geo {
    int NI, NJ, NK, PI, PJ;
    const double* X;            // nodes: X, Y, Z planes
    double* out;                // GEO_NF padded fields
    size_t P;                   // padded cells per field
};
enum GeoField { G_XC = 0, G_YC, G_ZC, G_DST, G_ALENG, G_ASENG, G_VOL, G_RAD, G_THTC, G_SD = 9, G_GRAD = 18, G_ALAGM = 21,
                GEO_NF = 24 };

__device__ __forceinline__ size_t gp(const Geo& g, int i, int j, int k) {
    return (size_t)(i + 2) + (size_t)g.PI * ((size_t)(j + 2) + (size_t)g.PJ * (size_t)(k + 2));
}
__device__ __forceinline__ double nd(const Geo& g, int q, int I, int J, int K) {   // node (I,J,K), 1-based
    return g.X[(size_t)q * g.NI * g.NJ * g.NK + (size_t)(I - 1) + (size_t)g.NI * ((size_t)(J - 1) + (size_t)g.NJ * (K - 1))];
}
__device__ __forceinline__ double* gf(const Geo& g, int f) { return g.out + (size_t)f * g.P; }

// cell centre of cell (I,J,K) from its 8 nodes (:97-112)
__device__ __forceinline__ double cell_centre(const Geo& g, int q, int I, int J, int K) {
    const int I1 = I + 1, J1 = J + 1, K1 = K + 1;
    return (nd(g, q, I1, J1, K1) + nd(g, q, I1, J1, K) + nd(g, q, I1, J, K1) + nd(g, q, I1, J, K) + nd(g, q, I, J1, K1) +
            nd(g, q, I, J1, K) + nd(g, q, I, J, K1) + nd(g, q, I, J, K)) / 8.;
}

// atan over [0, 1]: two half-angle reductions atan t = 2 atan(t / (1 + sqrt(1 + t^2))), then the
// odd Taylor series to t^31 (the host set-up's own atan2, so the two agree bit for bit)
__device__ double atan01(double t) {
    for (int r = 0; r < 2; ++r) t = t / (1.0 + sqrt(1.0 + t * t));
    const double t2 = t * t;
    double p = 0.0;
    for (int n = 31; n > 1; n -= 2) p = (1.0 / n - p) * t2;
    return 4.0 * (t - t * p);
}
__device__ double det_atan2(double y, double x) {
    const double PI = 3.141592653589793115997963468544185161590576171875;     // RN(pi)
    const double PIO2 = 1.5707963267948965579989817342720925807952880859375;  // RN(pi/2)
    const double ay = fabs(y), ax = fabs(x);
    const bool big = ay > ax;
    const double num = big ? ax : ay, den = big ? ay : ax;
    const double t = den > 0 ? num / den : 0.0;
    double a = atan01(t);
    if (big) a = PIO2 - a;
    if (x < 0) a = PI - a;
    if (y < 0) a = -a;
    return a;
}

// interior cells: centres, thtc, rad, and the points of the wall distance
__global__ void k_geo_cells(Geo g) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int NI1 = g.NI - 1, NJ1 = g.NJ - 1, NK1 = g.NK - 1;
    if (n >= (long long)NI1 * NJ1 * NK1) return;
    const int I = (int)(n % NI1) + 1, J = (int)((n / NI1) % NJ1) + 1, K = (int)(n / ((long long)NI1 * NJ1)) + 1;
    const size_t c = gp(g, I, J, K);
    const double zc = cell_centre(g, 2, I, J, K), yc = cell_centre(g, 1, I, J, K), xc = cell_centre(g, 0, I, J, K);
    gf(g, G_XC)[c] = xc; gf(g, G_YC)[c] = yc; gf(g, G_ZC)[c] = zc;
    gf(g, G_THTC)[c] = det_atan2(zc, yc);
    gf(g, G_RAD)[c] = sqrt(yc * yc + zc * zc);
}

// The cell centres for the wall distance, a warp's points a brick of cells: at the coarse O-block the chunks
// near a brick of 4 x 4 x 2 are 24 and its candidates 170, near 32 cells of a line 58 and 880.  Places past
// the block repeat its last cells.
constexpr int WD_BI = 4, WD_BJ = 4, WD_BK = 2;
__host__ __device__ inline long long brick_places(int NI1, int NJ1, int NK1) {
    return 32LL * ((NI1 + WD_BI - 1) / WD_BI) * ((NJ1 + WD_BJ - 1) / WD_BJ) * ((NK1 + WD_BK - 1) / WD_BK);
}
struct BrickCell { int I, J, K; bool in; };
__device__ __forceinline__ BrickCell brick_cell(const Geo& g, long long n) {
    const int NI1 = g.NI - 1, NJ1 = g.NJ - 1, NK1 = g.NK - 1, l = (int)(n & 31);
    const int bi = (NI1 + WD_BI - 1) / WD_BI, bj = (NJ1 + WD_BJ - 1) / WD_BJ;
    const long long b = n >> 5;
    const int i = (int)(b % bi) * WD_BI + l % WD_BI, j = (int)(b / bi % bj) * WD_BJ + l / WD_BI % WD_BJ;
    const int k = (int)(b / bi / bj) * WD_BK + l / (WD_BI * WD_BJ);
    return {min(i, NI1 - 1) + 1, min(j, NJ1 - 1) + 1, min(k, NK1 - 1) + 1, i < NI1 && j < NJ1 && k < NK1};
}
__global__ void k_geo_points(Geo g, double* __restrict__ pts) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= brick_places(g.NI - 1, g.NJ - 1, g.NK - 1)) return;
    const BrickCell b = brick_cell(g, n);
    const size_t c = gp(g, b.I, b.J, b.K);
    for (int q = 0; q < 3; ++q) pts[3 * n + q] = gf(g, G_XC + q)[c];
}

__global__ void k_geo_dst(Geo g, const double* __restrict__ dst) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= brick_places(g.NI - 1, g.NJ - 1, g.NK - 1)) return;
    const BrickCell b = brick_cell(g, n);
    if (b.in) gf(g, G_DST)[gp(g, b.I, b.J, b.K)] = dst[n];
}

// half cross product of the two face diagonals of face (I,J,K) of direction d (:180-300)
__device__ void face_cross(const Geo& g, int d, int I, int J, int K, double* xs) {
    double R1[3], R2[3];
    for (int q = 0; q < 3; ++q) {
        if (d == 0) {
            R1[q] = nd(g, q, I, J + 1, K + 1) - nd(g, q, I, J, K);
            R2[q] = nd(g, q, I, J, K + 1) - nd(g, q, I, J + 1, K);
        } else if (d == 1) {
            R1[q] = nd(g, q, I, J, K + 1) - nd(g, q, I + 1, J, K);
            R2[q] = nd(g, q, I + 1, J, K + 1) - nd(g, q, I, J, K);
        } else {
            R1[q] = nd(g, q, I + 1, J, K) - nd(g, q, I, J + 1, K);
            R2[q] = nd(g, q, I + 1, J + 1, K) - nd(g, q, I, J, K);
        }
    }
    xs[0] = (R1[1] * R2[2] - R1[2] * R2[1]) * 0.5;
    xs[1] = (R1[2] * R2[0] - R1[0] * R2[2]) * 0.5;
    xs[2] = (R1[0] * R2[1] - R1[1] * R2[0]) * 0.5;
}

// faces of direction d: SD = the half cross product oriented by the block's handedness (dl),
// Grad = |SD| (+ tiny under the root); face 0 copies face 1
__global__ void k_geo_faces(Geo g, int d, double tiny) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nI = d == 0 ? g.NI : g.NI - 1, nJ = d == 1 ? g.NJ : g.NJ - 1, nK = d == 2 ? g.NK : g.NK - 1;
    if (n >= (long long)nI * nJ * nK) return;
    const int I = (int)(n % nI) + 1, J = (int)((n / nI) % nJ) + 1, K = (int)(n / ((long long)nI * nJ)) + 1;
    // handedness: the first i-face normal against the direction from cell (1,1,1) to (2,1,1)
    double x0[3];
    face_cross(g, 0, 1, 1, 1, x0);
    const double xv = cell_centre(g, 0, 2, 1, 1) - cell_centre(g, 0, 1, 1, 1);
    const double yv = cell_centre(g, 1, 2, 1, 1) - cell_centre(g, 1, 1, 1, 1);
    const double zv = cell_centre(g, 2, 2, 1, 1) - cell_centre(g, 2, 1, 1, 1);
    const double dl = (xv * x0[0] + yv * x0[1] + zv * x0[2] < 0) ? -1.0 : 1.0;
    double xs[3];
    face_cross(g, d, I, J, K, xs);
    const size_t c = gp(g, I, J, K);
    double sd[3];
    for (int q = 0; q < 3; ++q) { sd[q] = xs[q] * dl; gf(g, G_SD + 3 * d + q)[c] = sd[q]; }
    const double gr = sqrt(sd[0] * sd[0] + sd[1] * sd[1] + sd[2] * sd[2] + tiny);
    gf(g, G_GRAD + d)[c] = gr;
    const int e1 = d == 0 ? I : (d == 1 ? J : K);
    if (e1 == 1) {
        const size_t c0 = gp(g, I - (d == 0), J - (d == 1), K - (d == 2));
        for (int q = 0; q < 3; ++q) gf(g, G_SD + 3 * d + q)[c0] = sd[q];
        gf(g, G_GRAD + d)[c0] = gr;
    }
}

// face centre (0.25 of the sum of 4 nodes) of face `f` (w e s n b t) of cell (I,J,K), component q
__device__ double face_centre(const Geo& g, int q, int f, int I, int J, int K) {
    int a[4][3];
    switch (f) {
        case 0: { int t[4][3] = {{0, 0, 0}, {0, 1, 0}, {0, 0, 1}, {0, 1, 1}}; memcpy(a, t, sizeof(a)); break; }
        case 1: { int t[4][3] = {{1, 0, 0}, {1, 1, 0}, {1, 0, 1}, {1, 1, 1}}; memcpy(a, t, sizeof(a)); break; }
        case 2: { int t[4][3] = {{0, 0, 0}, {1, 0, 0}, {0, 0, 1}, {1, 0, 1}}; memcpy(a, t, sizeof(a)); break; }
        case 3: { int t[4][3] = {{0, 1, 0}, {1, 1, 0}, {0, 1, 1}, {1, 1, 1}}; memcpy(a, t, sizeof(a)); break; }
        case 4: { int t[4][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {1, 1, 0}}; memcpy(a, t, sizeof(a)); break; }
        default: { int t[4][3] = {{0, 0, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}}; memcpy(a, t, sizeof(a)); break; }
    }
    double s = nd(g, q, I + a[0][0], J + a[0][1], K + a[0][2]) + nd(g, q, I + a[1][0], J + a[1][1], K + a[1][2]);
    s = s + nd(g, q, I + a[2][0], J + a[2][1], K + a[2][2]);
    s = s + nd(g, q, I + a[3][0], J + a[3][1], K + a[3][2]);
    return 0.25 * s;
}

// Alagm (:322-358): distance between the two opposite face centres of a cell, per direction
__global__ void k_geo_alagm(Geo g) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int NI1 = g.NI - 1, NJ1 = g.NJ - 1, NK1 = g.NK - 1;
    if (n >= (long long)NI1 * NJ1 * NK1) return;
    const int I = (int)(n % NI1) + 1, J = (int)((n / NI1) % NJ1) + 1, K = (int)(n / ((long long)NI1 * NJ1)) + 1;
    const size_t c = gp(g, I, J, K);
    for (int d = 0; d < 3; ++d) {
        const double dx = face_centre(g, 0, 2 * d, I, J, K) - face_centre(g, 0, 2 * d + 1, I, J, K);
        const double dy = face_centre(g, 1, 2 * d, I, J, K) - face_centre(g, 1, 2 * d + 1, I, J, K);
        const double dz = face_centre(g, 2, 2 * d, I, J, K) - face_centre(g, 2, 2 * d + 1, I, J, K);
        gf(g, G_ALAGM + d)[c] = sqrt(dx * dx + dy * dy + dz * dz);
    }
}

// centres of the boundary faces stored in the first ghost layer (:370-422): one thread per
// face cell of the six block faces
__global__ void k_geo_bface(Geo g) {
    const int NI1 = g.NI - 1, NJ1 = g.NJ - 1, NK1 = g.NK - 1;
    const long long nI = (long long)NJ1 * NK1, nJ = (long long)NI1 * NK1, nK = (long long)NI1 * NJ1;
    long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= 2 * (nI + nJ + nK)) return;
    int d, side, a, b;
    if (n < 2 * nI) { d = 0; side = (int)(n / nI); n %= nI; a = (int)(n % NJ1) + 1; b = (int)(n / NJ1) + 1; }
    else if ((n -= 2 * nI) < 2 * nJ) { d = 1; side = (int)(n / nJ); n %= nJ; a = (int)(n % NI1) + 1; b = (int)(n / NI1) + 1; }
    else { n -= 2 * nJ; d = 2; side = (int)(n / nK); n %= nK; a = (int)(n % NI1) + 1; b = (int)(n / NI1) + 1; }
    for (int q = 0; q < 3; ++q) {
        double v;
        size_t c;
        if (d == 0) {
            const int ii = side ? g.NI : 1;
            v = (nd(g, q, ii, a, b) + nd(g, q, ii, a + 1, b) + nd(g, q, ii, a, b + 1) + nd(g, q, ii, a + 1, b + 1)) / 4.0;
            c = gp(g, side ? g.NI : 0, a, b);
        } else if (d == 1) {
            const int jj = side ? g.NJ : 1;
            v = (nd(g, q, a, jj, b) + nd(g, q, a + 1, jj, b) + nd(g, q, a, jj, b + 1) + nd(g, q, a + 1, jj, b + 1)) / 4.0;
            c = gp(g, a, side ? g.NJ : 0, b);
        } else {
            const int kk = side ? g.NK : 1;
            v = (nd(g, q, a, b, kk) + nd(g, q, a + 1, b, kk) + nd(g, q, a, b + 1, kk) + nd(g, q, a + 1, b + 1, kk)) / 4.0;
            c = gp(g, a, b, side ? g.NK : 0);
        }
        gf(g, G_XC + q)[c] = v;
    }
}

// aLeng / aSeng (:430-480): largest and smallest distance to the six neighbouring centres
// (boundary face centres at the block faces), directions of 2 cells left out; Vol (:488-521)
__global__ void k_geo_len_vol(Geo g, double tiny, int* __restrict__ bad) {
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int NI1 = g.NI - 1, NJ1 = g.NJ - 1, NK1 = g.NK - 1;
    if (n >= (long long)NI1 * NJ1 * NK1) return;
    const int I = (int)(n % NI1) + 1, J = (int)((n / NI1) % NJ1) + 1, K = (int)(n / ((long long)NI1 * NJ1)) + 1;
    const size_t c = gp(g, I, J, K);
    const double* Xc = gf(g, G_XC);
    const double* Yc = gf(g, G_YC);
    const double* Zc = gf(g, G_ZC);
    const int off[6][3] = {{-1, 0, 0}, {1, 0, 0}, {0, -1, 0}, {0, 1, 0}, {0, 0, -1}, {0, 0, 1}};
    double dd[6];
    for (int m = 0; m < 6; ++m) {
        const size_t o = gp(g, I + off[m][0], J + off[m][1], K + off[m][2]);
        const double dx = Xc[o] - Xc[c], dy = Yc[o] - Yc[c], dz = Zc[o] - Zc[c];
        dd[m] = sqrt(dx * dx + dy * dy + dz * dz);
    }
    int use[6] = {1, 1, 1, 1, 1, 1};
    if (NI1 == 2) { use[0] = 0; use[1] = 0; use[2] = 1; use[3] = 1; use[4] = 1; use[5] = 1; }
    if (NJ1 == 2) { use[0] = 1; use[1] = 1; use[2] = 0; use[3] = 0; use[4] = 1; use[5] = 1; }
    if (NK1 == 2) { use[0] = 1; use[1] = 1; use[2] = 1; use[3] = 1; use[4] = 0; use[5] = 0; }
    double mx = -INFINITY, mn = INFINITY;
    for (int m = 0; m < 6; ++m)
        if (use[m]) { mx = fmax(mx, dd[m]); mn = fmin(mn, dd[m]); }
    gf(g, G_ALENG)[c] = mx;
    gf(g, G_ASENG)[c] = mn;
    // Vol = (1/3) sum over the three min faces of (diagonal node difference) . SD
    const double* SD = gf(g, G_SD);
    auto sd = [&](int d, int q) { return SD[(size_t)(3 * d + q) * g.P + c]; };
    double XR = nd(g, 0, I + 1, J + 1, K + 1) - nd(g, 0, I, J + 1, K + 1);
    double YR = nd(g, 1, I + 1, J + 1, K + 1) - nd(g, 1, I, J + 1, K + 1);
    double ZR = nd(g, 2, I + 1, J + 1, K + 1) - nd(g, 2, I, J + 1, K + 1);
    double OMG = XR * sd(0, 0) + YR * sd(0, 1) + ZR * sd(0, 2);
    XR = nd(g, 0, I + 1, J + 1, K + 1) - nd(g, 0, I + 1, J, K + 1);
    YR = nd(g, 1, I + 1, J + 1, K + 1) - nd(g, 1, I + 1, J, K + 1);
    ZR = nd(g, 2, I + 1, J + 1, K + 1) - nd(g, 2, I + 1, J, K + 1);
    OMG = OMG + XR * sd(1, 0) + YR * sd(1, 1) + ZR * sd(1, 2);
    XR = nd(g, 0, I + 1, J + 1, K + 1) - nd(g, 0, I + 1, J + 1, K);
    YR = nd(g, 1, I + 1, J + 1, K + 1) - nd(g, 1, I + 1, J + 1, K);
    ZR = nd(g, 2, I + 1, J + 1, K + 1) - nd(g, 2, I + 1, J + 1, K);
    OMG = OMG + XR * sd(2, 0) + YR * sd(2, 1) + ZR * sd(2, 2);
    const double vol = (1.0 / 3.0) * OMG;
    gf(g, G_VOL)[c] = vol;
    if (vol < tiny) atomicExch(bad, 1);
}

int wd_fail(int code, const std::string& msg) {
    g_stateless_err = msg;
    return code;
}

}  // namespace
}  // namespace tg

namespace tg {
namespace {

// panel centres of the wall surfaces (the reference's expression), their FP32 copies, chunk by chunk, the
// chunks and each surface's first one, and the largest coordinate magnitude; all of it one buffer, which
// goes to the device as one allocation and one copy (on small surfaces the call is mostly those)
struct Panels {
    std::unique_ptr<char[]> buf;
    size_t bytes = 0, at32 = 0, at_lo = 0, at64 = 0, at_chunk = 0, at_first = 0;
    int nchunk = 0;
    double R = 0.0;
};

int make_panels(int nsurf, const int* dims, const double* nodes, Panels& P) {
    size_t np = 0, nc = 0;
    for (int s = 0; s < nsurf; ++s) {
        const int ni = dims[2 * s], nj = dims[2 * s + 1];
        if (ni < 1 || nj < 1) return wd_fail(TRANS_E_ARG, "bad surface dimensions");
        np += (size_t)(ni - 1) * (nj - 1);
        nc += (size_t)((ni - 1 + WD_CHUNK - 1) / WD_CHUNK) * ((nj - 1 + WD_CHUNK - 1) / WD_CHUNK);
    }
    auto take = [&](size_t bytes) {
        const size_t at = P.bytes;
        P.bytes += (bytes + 255) / 256 * 256;
        return at;
    };
    P.at32 = take(sizeof(float) * 4 * np);         // rounded to FP32,
    P.at_lo = take(sizeof(float) * 4 * np);        // and what the rounding left
    P.at64 = take(sizeof(double) * 3 * np);
    P.at_chunk = take(sizeof(WallChunk) * nc);
    P.at_first = take(sizeof(int) * ((size_t)nsurf + 1));
    P.buf.reset(new char[P.bytes]);
    float* const p32 = reinterpret_cast<float*>(P.buf.get() + P.at32);
    float* const plo = reinterpret_cast<float*>(P.buf.get() + P.at_lo);
    double* const p64 = reinterpret_cast<double*>(P.buf.get() + P.at64);
    WallChunk* const chunks = reinterpret_cast<WallChunk*>(P.buf.get() + P.at_chunk);
    int* const first = reinterpret_cast<int*>(P.buf.get() + P.at_first);
    first[0] = 0;
    size_t base = 0;
    long long p = 0;
    for (int s = 0; s < nsurf; ++s) {
        const int ni = dims[2 * s], nj = dims[2 * s + 1];
        const size_t plane = (size_t)ni * nj;
        const double* X = nodes + base;
        const double* Y = X + plane;
        const double* Z = Y + plane;
        for (int J0 = 0; J0 < nj - 1; J0 += WD_CHUNK)
            for (int I0 = 0; I0 < ni - 1; I0 += WD_CHUNK) {
                const int I1 = std::min(I0 + WD_CHUNK, ni - 1), J1 = std::min(J0 + WD_CHUNK, nj - 1);
                WallChunk k{{INFINITY, INFINITY, INFINITY}, (I1 - I0) * (J1 - J0), {-INFINITY, -INFINITY, -INFINITY}, 0, p, 0};
                for (int J = J0; J < J1; ++J)
                    for (int I = I0; I < I1; ++I, ++p) {
                        const size_t a = (size_t)I + (size_t)ni * J, b = a + 1, cc = a + ni, dd = cc + 1;
                        const double x[3] = {(X[a] + X[b] + X[cc] + X[dd]) / 4.0, (Y[a] + Y[b] + Y[cc] + Y[dd]) / 4.0,
                                             (Z[a] + Z[b] + Z[cc] + Z[dd]) / 4.0};
                        for (int m = 0; m < 3; ++m) {
                            if (!std::isfinite(x[m])) return wd_fail(TRANS_E_ARG, "surface coordinates not finite");
                            const float f = (float)x[m];
                            p64[3 * p + m] = x[m];
                            p32[4 * p + m] = f;
                            plo[4 * p + m] = (float)(x[m] - (double)f);
                            k.lo[m] = std::min(k.lo[m], f);
                            k.hi[m] = std::max(k.hi[m], f);
                            P.R = std::max(P.R, std::fabs(x[m]));
                        }
                        p32[4 * p + 3] = plo[4 * p + 3] = 0.0f;
                    }
                chunks[P.nchunk++] = k;
            }
        first[s + 1] = P.nchunk;
        base += 3 * plane;
    }
    return TRANS_OK;
}

struct DevBufs {
    std::vector<void*> v;
    ~DevBufs() { for (void* p : v) cudaFree(p); }
    template <typename T> cudaError_t get(T** p, size_t bytes) {
        cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(bytes, 16));
        if (e == cudaSuccess) v.push_back((void*)*p);
        return e;
    }
};

// Which warps take which points: a warp a point while these warps are few, the points grouped where there is
// enough to pass over, otherwise as they come.  Whole calls on points in no order, ms (a lane per point as
// they come, grouped, a warp per point; before, with every panel scanned from shared memory): 208,896 points on
// 64 panels 0.70, 0.74, 1.09 (0.70), on 1,024 panels 0.95, 0.80, 1.11 (0.85), on 26,368 panels 6.28, 1.85, 3.42
// (6.25); 32,768 points on 64 panels 0.23, 0.26, 0.28 (0.22), on 1,024 panels 0.33, 0.31, 0.29 (0.29), on 26,368
// panels 2.71, 1.30, 0.92 (2.42); 64 points on 64 panels 0.13, 0.16, 0.12 (0.13), on 26,368 panels 2.37, 2.32, 0.39
// (2.09).
bool one_point_a_warp(long long n, const Panels& P) {
    return n <= std::min(32768LL, std::max(4096LL, 2048LL * P.nchunk));
}
bool group_by_place(long long n, const Panels& P) {
    return !one_point_a_warp(n, P) && P.nchunk >= 16 && n <= 0x7fffffffLL;
}

// the wall distance of n device points (x y z interleaved) into d_dst, on stream st
int run_wall_distance(cudaStream_t st, long long n, const double* d_pts, const unsigned* d_idx, int nsurf, const Panels& P,
                      double R, double tiny, double* d_dst, DevBufs& bufs) {
    if (R > 1.0e18) return wd_fail(TRANS_E_ARG, "coordinates beyond 1e18");   // FP32 squares stay finite
    const float eabs = std::max((float)(1.0e-6 * R), 1.0e-37f);
    char* d = nullptr;
    cudaError_t e;
    if ((e = bufs.get(&d, P.bytes)) != cudaSuccess ||
        (e = cudaMemcpyAsync(d, P.buf.get(), P.bytes, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return wd_fail(TRANS_E_CUDA, std::string("wall distance set-up: ") + cudaGetErrorString(e));
    auto run = [&](auto kernel, long long threads) {
        kernel<<<(unsigned)((threads + WD_THREADS - 1) / WD_THREADS), WD_THREADS, 0, st>>>(
            n, d_pts, d_idx, reinterpret_cast<const float4*>(d + P.at32), reinterpret_cast<const float4*>(d + P.at_lo),
            reinterpret_cast<const double*>(d + P.at64), reinterpret_cast<const WallChunk*>(d + P.at_chunk),
            reinterpret_cast<const int*>(d + P.at_first), nsurf, eabs, tiny, d_dst);
    };
    if (one_point_a_warp(n, P)) run(k_wall_distance<true>, 32 * n);
    else run(k_wall_distance<false>, n);
    if ((e = cudaGetLastError()) != cudaSuccess) return wd_fail(TRANS_E_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    return TRANS_OK;
}

// The points' grouping (k_point_count): where there is one, its grid; bits 0: as they come
PointGrid group_grid(long long n, const double* xyz, const Panels& P) {
    constexpr int SAMPLE = 1024;                   // points whose box stands for all (others: the outermost cells)
    PointGrid g{};
    if (!group_by_place(n, P)) return g;
    g.bits = 2;
    while (g.bits < 6 && (16LL << (3 * g.bits)) < n) ++g.bits;     // 2 to 16 points a cell; at most 2^18 cells
    for (int m = 0; m < 3; ++m) {
        double lo = xyz[m], hi = lo;
        for (long long k = 1; k < SAMPLE; ++k) {
            const double x = xyz[3 * (n / SAMPLE * k + n % SAMPLE * k / SAMPLE) + m];
            lo = std::min(lo, x);
            hi = std::max(hi, x);
        }
        g.lo[m] = lo;
        g.scale[m] = hi > lo ? (1 << g.bits) / (hi - lo) : 0.0;
        if (!std::isfinite(g.scale[m])) g.scale[m] = 0.0;
    }
    return g;
}
// the points' order, in bins[0 .. cells - 1] and behind them n indexes
const unsigned* group_points(cudaStream_t st, long long n, const double* d_pts, const PointGrid& g, unsigned* bins) {
    const unsigned nbins = 1u << (3 * g.bits), grid = (unsigned)((n + 255) / 256);
    cudaMemsetAsync(bins, 0, sizeof(unsigned) * nbins, st);
    k_point_count<<<grid, 256, 0, st>>>((unsigned)n, d_pts, g, bins);
    k_point_scan<<<1, 1024, 0, st>>>(bins, nbins);
    k_point_place<<<grid, 256, 0, st>>>((unsigned)n, d_pts, g, bins, bins + nbins);
    return bins + nbins;
}

struct StreamGuard {
    cudaStream_t s = nullptr;
    ~StreamGuard() { if (s) cudaStreamDestroy(s); }
};

}  // namespace
}  // namespace tg

using namespace tg;

extern "C" int trans_wall_distance(long long n, const double* xyz, int nsurf, const int* dims, const double* nodes,
                                   double tiny, double* dst) {
    g_stateless_err.clear();
    if (n < 0 || nsurf < 0 || (n > 0 && (!xyz || !dst)) || (nsurf > 0 && (!dims || !nodes)))
        return wd_fail(TRANS_E_ARG, "bad argument");
    if (n == 0) return TRANS_OK;
    if (n > (long long)2147483647 * WD_THREADS) return wd_fail(TRANS_E_ARG, "too many points");
    Panels P;
    int rc = make_panels(nsurf, dims, nodes, P);
    if (rc) return rc;
    double R = P.R;
    for (long long q = 0; q < 3 * n; ++q) {
        if (!std::isfinite(xyz[q])) return wd_fail(TRANS_E_ARG, "point coordinates not finite");
        R = std::max(R, std::fabs(xyz[q]));
    }
    StreamGuard sg;
    DevBufs bufs;
    double* d_pts = nullptr;                       // points, distances and, where they are grouped, cells and order
    PointGrid g = group_grid(n, xyz, P);
    const size_t words = sizeof(double) * 4 * (size_t)n;
    auto room = [&]() { return bufs.get(&d_pts, words + (g.bits ? sizeof(unsigned) * (((size_t)1 << (3 * g.bits)) + (size_t)n) : 0)); };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&sg.s, cudaStreamNonBlocking)) == cudaSuccess && (e = room()) != cudaSuccess && g.bits) {
        cudaGetLastError();
        g.bits = 0;
        e = room();
    }
    if (e != cudaSuccess ||
        (e = cudaMemcpyAsync(d_pts, xyz, sizeof(double) * 3 * (size_t)n, cudaMemcpyHostToDevice, sg.s)) != cudaSuccess)
        return wd_fail(TRANS_E_CUDA, std::string("set-up: ") + cudaGetErrorString(e));
    double* const d_dst = d_pts + 3 * (size_t)n;
    const unsigned* d_idx = g.bits ? group_points(sg.s, n, d_pts, g, reinterpret_cast<unsigned*>(d_dst + n)) : nullptr;
    if ((rc = run_wall_distance(sg.s, n, d_pts, d_idx, nsurf, P, R, tiny, d_dst, bufs))) { cudaStreamSynchronize(sg.s); return rc; }
    if ((e = cudaMemcpyAsync(dst, d_dst, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost, sg.s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(sg.s)) != cudaSuccess)
        return wd_fail(TRANS_E_CUDA, std::string("wall distance: ") + cudaGetErrorString(e));
    return TRANS_OK;
}

extern "C" int trans_block_metrics(int ni, int nj, int nk, const double* xyz, int nsurf, const int* dims,
                                   const double* nodes, double tiny, double* out) {
    g_stateless_err.clear();
    if (ni < 3 || nj < 3 || nk < 3 || !xyz || !out || nsurf < 0 || (nsurf > 0 && (!dims || !nodes)))
        return wd_fail(TRANS_E_ARG, "bad argument");
    const size_t nn = (size_t)ni * nj * nk;
    const size_t P = (size_t)(ni + 5) * (nj + 5) * (nk + 5);
    if (P * GEO_NF > ((size_t)1 << 33)) return wd_fail(TRANS_E_ARG, "block too large");
    Panels pan;
    int rc = make_panels(nsurf, dims, nodes, pan);
    if (rc) return rc;
    double R = pan.R;
    for (size_t q = 0; q < 3 * nn; ++q) {
        if (!std::isfinite(xyz[q])) return wd_fail(TRANS_E_ARG, "node coordinates not finite");
        R = std::max(R, std::fabs(xyz[q]));          // cell centres lie within the nodes' bound
    }
    const long long ncell = (long long)(ni - 1) * (nj - 1) * (nk - 1), nplace = brick_places(ni - 1, nj - 1, nk - 1);
    StreamGuard sg;
    DevBufs bufs;
    double *d_x = nullptr, *d_out = nullptr, *d_pts = nullptr, *d_dst = nullptr;
    int* d_bad = nullptr;
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&sg.s, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = bufs.get(&d_x, sizeof(double) * 3 * nn)) != cudaSuccess ||
        (e = bufs.get(&d_out, sizeof(double) * GEO_NF * P)) != cudaSuccess ||
        (e = bufs.get(&d_pts, sizeof(double) * 3 * (size_t)nplace)) != cudaSuccess ||
        (e = bufs.get(&d_dst, sizeof(double) * (size_t)nplace)) != cudaSuccess ||
        (e = bufs.get(&d_bad, sizeof(int))) != cudaSuccess ||
        (e = cudaMemcpyAsync(d_x, xyz, sizeof(double) * 3 * nn, cudaMemcpyHostToDevice, sg.s)) != cudaSuccess ||
        (e = cudaMemsetAsync(d_out, 0, sizeof(double) * GEO_NF * P, sg.s)) != cudaSuccess ||
        (e = cudaMemsetAsync(d_bad, 0, sizeof(int), sg.s)) != cudaSuccess)
        return wd_fail(TRANS_E_CUDA, std::string("set-up: ") + cudaGetErrorString(e));
    Geo g{ni, nj, nk, ni + 5, nj + 5, d_x, d_out, P};
    const unsigned T = 256;
    auto blocks = [&](long long n) { return (unsigned)((n + T - 1) / T); };
    k_geo_cells<<<blocks(ncell), T, 0, sg.s>>>(g);
    k_geo_points<<<blocks(nplace), T, 0, sg.s>>>(g, d_pts);
    for (int d = 0; d < 3; ++d) {
        const long long nf = (long long)(d == 0 ? ni : ni - 1) * (d == 1 ? nj : nj - 1) * (d == 2 ? nk : nk - 1);
        k_geo_faces<<<blocks(nf), T, 0, sg.s>>>(g, d, tiny);
    }
    k_geo_alagm<<<blocks(ncell), T, 0, sg.s>>>(g);
    const long long nb = 2LL * ((long long)(nj - 1) * (nk - 1) + (long long)(ni - 1) * (nk - 1) + (long long)(ni - 1) * (nj - 1));
    k_geo_bface<<<blocks(nb), T, 0, sg.s>>>(g);
    k_geo_len_vol<<<blocks(ncell), T, 0, sg.s>>>(g, tiny, d_bad);
    if ((e = cudaGetLastError()) != cudaSuccess) return wd_fail(TRANS_E_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    if ((rc = run_wall_distance(sg.s, nplace, d_pts, nullptr, nsurf, pan, R, tiny, d_dst, bufs))) { cudaStreamSynchronize(sg.s); return rc; }
    k_geo_dst<<<blocks(nplace), T, 0, sg.s>>>(g, d_dst);
    int bad = 0;
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(out, d_out, sizeof(double) * GEO_NF * P, cudaMemcpyDeviceToHost, sg.s)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, sg.s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(sg.s)) != cudaSuccess)
        return wd_fail(TRANS_E_CUDA, std::string("metrics: ") + cudaGetErrorString(e));
    if (bad) return wd_fail(TRANS_E_ARG, "negative volume");
    return TRANS_OK;
}
