// Anisotropic particle kernels for surface reconstruction: the reference's
// AnisotropicKernelGenerator<3, float>::computeAniKernels
// (Simulation/SurfaceReconstruction/AniKernelGenerator.cpp:53-101), which
// PIC_Solver::saveFrameData runs when "AniKernel" is among the saved data
// (Simulation/ParticleSolvers/PICFluid/PIC_Solver.cpp:248-252).
//
// Per particle p, over its neighbours q (|p - q|^2 < r^2, q != p; r = kernelRatio x
// particleRadius) and with W(d) = 1 - (|d| / r)^3:
//   weighted mean m = (p + sum W(p-q) q) / (1 + sum W(p-q)), centre = lerp(p, m, blend);
//   fewer than `threshold` neighbours: kernel = defaultSpraySize x identity;
//   else C = sum W(q-m) (q-m)(q-m)^T / (1 + sum W(q-m)), C = Q diag(S) Q^T with S sorted
//   descending, S[1,2] = max(S[1,2], S[0] / axisRatio), S *= cbrt(1 / prod S),
//   kernel = Q diag(S) Q^T (column-major, glm::mat3 memory order).
//
// One thread per particle in cell-sorted order.  Both passes walk the cell rows around the
// particle (z outer, y inner) and, in each row, the sorted particles of the cells its
// kernel sphere can reach, so every thread sums its neighbours in the canonical order
// (rows, then cell-sorted order).  Candidates are taken two at a time: of points
// 2i and 2i + 1, {x pair, y pair} is one 16-byte load and {z pair} one of 8, and distances,
// weights and products are formed in packed FP32 (each half rounded as the scalar operation); the sums stay serial and
// take a neighbour's terms alone (add_hits).  Rows and cells that provably hold no neighbour are
// skipped; the margins cover the float rounding of the cell index (see row_range).  The
// covariance is symmetric positive semi-definite, so its SVD is its
// eigen-decomposition; a cyclic Jacobi iteration gives it, and the cube root is Newton's
// iteration in double precision, so the whole pass uses only correctly rounded
// operations and matches the CPU restatement bit for bit.
#include "bnn_internal.cuh"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

namespace bnn {

namespace {

struct AnisoArgs {
    float r2;         // kernel radius squared (float product, as the reference)
    float r2m;        // r2 (1 + 1e-4): the pruning radius squared
    float rinv;       // 1 / r
    float blend, axisRatio, spray;
    uint32_t threshold;
    int R;            // cell rows / columns a neighbour can lie away
    float margin;     // 0.01 cell: bound on how far a point's cell index can be off its position
};

// Packed FP32 pairs.  A packed product followed by a packed sum would be fused by the assembler
// and round once, so products are a * b + (-0) with the -0 pair a kernel argument, unknown to it.
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float lo, float hi) {
    return (F2)__float_as_uint(lo) | (F2)__float_as_uint(hi) << 32;
}
__device__ __forceinline__ float lo2(F2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(F2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
struct Packed {
    F2 minus0, minus1, one;
};
__device__ __forceinline__ F2 mul2(F2 a, F2 b, const Packed& k) { return fma2(a, b, k.minus0); }
// (a a + b b) + c c
__device__ __forceinline__ F2 len2(F2 a, F2 b, F2 c, const Packed& k) {
    return add2(add2(mul2(a, a, k), mul2(b, b, k)), mul2(c, c, k));
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Correctly rounded square roots of a pair: g = x y with y near x^(-1/2), then one Newton step
// on the residual, g + (x - g g) y / 2 with the residual fused (P. Markstein, IBM J. Res. Dev.
// 34, 1990); y / 2 is y with its exponent lowered.  Equal to sqrtf for every float in [2^-100,
// 2^100] (all of them tried).  x is raised to 2^-100 first, which keeps 0 out of the
// reciprocal: below 2^-75 kernel_w2 gives 1 either way while r >= 2^-24.  bnn_aniso_sqrt_probe tries
// them again.
__device__ __forceinline__ F2 sqrt2(F2 v, const Packed& k) {
    const float x0 = fmaxf(lo2(v), 0x1p-100f), x1 = fmaxf(hi2(v), 0x1p-100f);
    const float y0 = rsqrt_approx(x0), y1 = rsqrt_approx(x1);
    const F2 g = mul2(pack2(x0, x1), pack2(y0, y1), k);
    const F2 e = pack2(fmaf(-lo2(g), lo2(g), x0), fmaf(-hi2(g), hi2(g), x1));
    const F2 h = pack2(__uint_as_float(__float_as_uint(y0) - 0x00800000u), __uint_as_float(__float_as_uint(y1) - 0x00800000u));
    return fma2(e, h, g);
}
// W = 1 - (|d| / r)^3 of a pair of squared distances.  FAST: 2^-24 <= r <= 2^24, the range in
// which sqrt2 is exact (or the weight does not depend on it)
template<bool FAST> __device__ __forceinline__ F2 kernel_w2(F2 d2, F2 rinv, const Packed& k) {
    const F2 root = FAST ? sqrt2(d2, k) : pack2(sqrtf(lo2(d2)), sqrtf(hi2(d2)));
    const F2 t = mul2(root, rinv, k);
    return fma2(mul2(mul2(t, t, k), t, k), k.minus1, k.one);
}

// a + v.lo + v.hi, each only where it is a neighbour's, as predicated sums: a candidate that is none
// leaves a as it is, whatever its coordinates (not finite, the pair mate of another row).  A sum of
// 0 instead would make a running -0 to 0, and 0 times a NaN coordinate is NaN.
__device__ __forceinline__ float add_hits(float a, F2 v, bool h0, bool h1) {
    asm("{ .reg .pred p, q; setp.ne.s32 p, %3, 0; setp.ne.s32 q, %4, 0; @p add.rn.f32 %0, %0, %1; @q add.rn.f32 %0, %0, %2; }"
        : "+f"(a) : "f"(lo2(v)), "f"(hi2(v)), "r"((int)h0), "r"((int)h1));
    return a;
}

// The sorted-index range [s, e) of cell row (j, k) that may hold neighbours of p.  A
// point stored in interior cell c lies within c * dx - margin .. (c + 1) * dx + margin
// of bmin (the truncated cell index is off by at most ~1e-4 cell for grids up to 1024
// cells); the border rows and columns also hold any point clamped onto them.  Rows whose
// distance from p exceeds the pruning radius hold no neighbour, and within a row only the
// cells within the chord (plus the margin) can.
__device__ __forceinline__ bool row_range(const AnisoGrid& g, const AnisoArgs& a, const uint32_t* __restrict__ cellStart,
                                          float px, float py, float pz, int j, int k, uint32_t& s, uint32_t& e) {
    if(j < 0 || j >= g.G[1] || k < 0 || k >= g.G[2]) return false;
    const float ylo = j == 0 ? -INFINITY : g.bmin[1] + (float)j * g.dx - a.margin;
    const float yhi = j == g.G[1] - 1 ? INFINITY : g.bmin[1] + (float)(j + 1) * g.dx + a.margin;
    const float zlo = k == 0 ? -INFINITY : g.bmin[2] + (float)k * g.dx - a.margin;
    const float zhi = k == g.G[2] - 1 ? INFINITY : g.bmin[2] + (float)(k + 1) * g.dx + a.margin;
    const float dy = fmaxf(0.0f, fmaxf(ylo - py, py - yhi));
    const float dz = fmaxf(0.0f, fmaxf(zlo - pz, pz - zhi));
    const float dyz = dy * dy + dz * dz;
    if(!(dyz < a.r2m)) return false;
    const float ext = sqrtf(a.r2m - dyz) + a.margin;
    int i0 = (int)floorf((px - ext - g.bmin[0]) / g.dx);
    int i1 = (int)floorf((px + ext - g.bmin[0]) / g.dx);
    i0 = i0 < 0 ? 0 : i0;
    i1 = i1 > g.G[0] - 1 ? g.G[0] - 1 : i1;
    if(i0 > i1) return false;
    const size_t row = ((size_t)k * g.G[1] + j) * g.G[0];
    s = cellStart[row + i0];
    e = cellStart[row + i1 + 1];
    return s < e;
}

// Newton's iteration for the cube root, x <- (2x + m / x^2) / 3, on the mantissa in
// [0.5, 4) with the exponent split off exactly; 0, inf and NaN map to themselves.
__device__ __forceinline__ double cbrt_newton(double y) {
    if(!(y == y) || y == 0.0 || isinf(y)) return y;
    const bool neg = y < 0.0;
    int e;
    double m = frexp(neg ? -y : y, &e);
    int q = e / 3, r = e % 3;
    if(r < 0) { r += 3; --q; }
    m = ldexp(m, r);
    double x = 1.0;
#pragma unroll 1
    for(int it = 0; it < 8; ++it) x = (2.0 * x + m / (x * x)) / 3.0;
    x = ldexp(x, q);
    return neg ? -x : x;
}

// One Jacobi rotation annihilating a[P][Q] (symmetric a, eigenvectors in v's columns)
template<int P, int Q>
__device__ __forceinline__ void jacobi_rotate(float a[3][3], float v[3][3]) {
    constexpr int R = 3 - P - Q;
    const float apq = a[P][Q];
    if(apq == 0.0f) return;
    const float app = a[P][P], aqq = a[Q][Q];
    if(fabsf(apq) < 1e-9f * (fabsf(app) + fabsf(aqq))) {
        a[P][Q] = a[Q][P] = 0.0f;
        return;
    }
    const float tau = (aqq - app) / (2.0f * apq);
    float t;
    if(fabsf(tau) > 1e15f) t = 0.5f / tau;
    else {
        t = 1.0f / (fabsf(tau) + sqrtf(1.0f + tau * tau));
        if(tau < 0.0f) t = -t;
    }
    const float c = 1.0f / sqrtf(1.0f + t * t);
    const float s = t * c;
    a[P][P] = app - t * apq;
    a[Q][Q] = aqq + t * apq;
    a[P][Q] = a[Q][P] = 0.0f;
    const float arp = a[R][P], arq = a[R][Q];
    a[R][P] = a[P][R] = c * arp - s * arq;
    a[R][Q] = a[Q][R] = s * arp + c * arq;
#pragma unroll
    for(int k = 0; k < 3; ++k) {
        const float vkp = v[k][P], vkq = v[k][Q];
        v[k][P] = c * vkp - s * vkq;
        v[k][Q] = s * vkp + c * vkq;
    }
}

template<int I, int J>
__device__ __forceinline__ void sort_pair(float lam[3], float v[3][3]) {
    if(lam[I] < lam[J]) {
        const float t = lam[I]; lam[I] = lam[J]; lam[J] = t;
#pragma unroll
        for(int k = 0; k < 3; ++k) { const float u = v[k][I]; v[k][I] = v[k][J]; v[k][J] = u; }
    }
}

// AniKernelGenerator.cpp:91-98 on the covariance a (destroyed); out column-major
__device__ __forceinline__ void kernel_matrix(float a[3][3], float axisRatio, float out[9]) {
    float v[3][3] = {{1.0f, 0.0f, 0.0f}, {0.0f, 1.0f, 0.0f}, {0.0f, 0.0f, 1.0f}};
#pragma unroll 1
    for(int sweep = 0; sweep < 10; ++sweep) {
        if(a[0][1] == 0.0f && a[0][2] == 0.0f && a[1][2] == 0.0f) break;
        jacobi_rotate<0, 1>(a, v);
        jacobi_rotate<0, 2>(a, v);
        jacobi_rotate<1, 2>(a, v);
    }
    float S[3] = {a[0][0], a[1][1], a[2][2]};
    sort_pair<0, 1>(S, v);
    sort_pair<1, 2>(S, v);
    sort_pair<0, 1>(S, v);
    const float lo = S[0] / axisRatio;
    S[1] = S[1] < lo ? lo : S[1];
    S[2] = S[2] < lo ? lo : S[2];
    const float prod = S[0] * S[1] * S[2];
    const float sc = (float)cbrt_newton((double)(1.0f / prod));
#pragma unroll
    for(int i = 0; i < 3; ++i) S[i] = S[i] * sc;
#pragma unroll
    for(int c = 0; c < 3; ++c)
#pragma unroll
        for(int r = 0; r < 3; ++r)
            out[c * 3 + r] = v[r][0] * S[0] * v[c][0] + v[r][1] * S[1] * v[c][1] + v[r][2] * S[2] * v[c][2];
}

// Bound by the FP32 pipe (a packed operation takes it for two cycles, so packing saves issue
// slots, not pipe cycles; 1.58 M points: pipe busy 67 % of the cycles, ALU 50 %, issue 76 %, 25.5 of 32
// lanes, stalls math_pipe_throttle 3.6 and not_selected 3.3) and, below a few hundred thousand points, by the serial chain of a particle's candidates.  ms against one candidate at a
// time with sqrtf and a 16-byte record: 5,000 points 0.467 (0.947), 50,000 0.766 (1.28), 200,003
// 2.51 (2.75), 600,001 7.18 (7.63), 1,000,000 11.86 (12.45), 3,000,000 36.3 (38.1); the pass over a
// 256^3 scene with its layout 155.7 (163.5).  Coordinates in three planes, three loads a pair:
// 0.456, 0.798, 2.62, 7.58, 12.55, 38.5.  Sums of selected terms instead of predicated ones:
// 0.498, 0.867, 2.77 and 13.2 at a million.  Nine blocks per SM: 200,003 points 2.62 ms against
// 2.75 at ten (planes).
template<bool FAST>
__global__ void __launch_bounds__(128, 9) k_aniso(int n, const ulonglong2* __restrict__ xy, const F2* __restrict__ zz,
                                               const uint32_t* __restrict__ ids,
                                               const uint32_t* __restrict__ cellStart, AnisoGrid g, AnisoArgs a, Packed k2,
                                               float* __restrict__ outC, float* __restrict__ outM,
                                               unsigned* __restrict__ counters) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = p < n;
    float Px = 0.f, Py = 0.f, Pz = 0.f;
    if(active) {
        const float* own = reinterpret_cast<const float*>(xy + (p >> 1)) + (p & 1);
        Px = own[0];
        Py = own[2];
        Pz = reinterpret_cast<const float*>(zz)[p];
    }
    int cj, ck;
    {
        int c[3] = {(int)((Px - g.bmin[0]) / g.dx), (int)((Py - g.bmin[1]) / g.dx), (int)((Pz - g.bmin[2]) / g.dx)};
        bool out = false;
#pragma unroll
        for(int d = 0; d < 3; ++d) {
            if(c[d] < 0) { c[d] = 0; out = true; }
            if(c[d] > g.G[d] - 1) { c[d] = g.G[d] - 1; out = true; }
        }
        // the pruning assumes every point lies in the grid it was sorted on
        if(active && out) atomicAdd(counters + 1, 1u);
        cj = c[1];
        ck = c[2];
    }
    const int R = a.R;
    const uint32_t self = (uint32_t)p;
    const F2 Px2 = pack2(Px, Px), Py2 = pack2(Py, Py), Pz2 = pack2(Pz, Pz), rinv = pack2(a.rinv, a.rinv);

    // pass 1: neighbour count and weighted mean (AniKernelGenerator.cpp:65-75)
    float sw = 1.0f, mx = Px, my = Py, mz = Pz;
    uint32_t cnt = 0;
    for(int dz = -R; dz <= R; ++dz)
        for(int dy = -R; dy <= R; ++dy) {
            uint32_t s = 0, e = 0;
            if(active) row_range(g, a, cellStart, Px, Py, Pz, cj + dy, ck + dz, s, e);
            const uint32_t len = e - s;
#pragma unroll 2
            for(uint32_t i = s >> 1; 2 * i < e; ++i) {
                const uint32_t q = 2 * i;
                const ulonglong2 Qxy = __ldg(xy + i);
                const F2 Qx = Qxy.x, Qy = Qxy.y, Qz = __ldg(zz + i);
                const F2 ex = fma2(Qx, k2.minus1, Px2), ey = fma2(Qy, k2.minus1, Py2), ez = fma2(Qz, k2.minus1, Pz2);
                const F2 d2 = len2(ex, ey, ez, k2);
                const bool h0 = lo2(d2) < a.r2 && q - s < len && q != self;
                const bool h1 = hi2(d2) < a.r2 && q + 1 - s < len && q + 1 != self;
                const F2 w = kernel_w2<FAST>(d2, rinv, k2);
                cnt += (h0 ? 1u : 0u) + (h1 ? 1u : 0u);
                sw = add_hits(sw, w, h0, h1);
                mx = add_hits(mx, mul2(w, Qx, k2), h0, h1);
                my = add_hits(my, mul2(w, Qy, k2), h0, h1);
                mz = add_hits(mz, mul2(w, Qz, k2), h0, h1);
            }
        }
    const float wx = mx / sw, wy = my / sw, wz = mz / sw;
    const uint32_t id = active ? ids[p] : 0u;
    if(active) {
        // MathHelpers::lerp (MathHelpers.h:549-551)
        const float f = a.blend, omf = 1.0f - f;
        outC[3 * (size_t)id] = omf * Px + f * wx;
        outC[3 * (size_t)id + 1] = omf * Py + f * wy;
        outC[3 * (size_t)id + 2] = omf * Pz + f * wz;
    }
    const bool need = active && cnt >= a.threshold;
    const unsigned sprayMask = __ballot_sync(0xffffffffu, active && !need);
    if((threadIdx.x & 31) == 0 && sprayMask) atomicAdd(counters, (unsigned)__popc(sprayMask));
    if(active && !need) {
        float* M = outM + 9 * (size_t)id;
#pragma unroll
        for(int e = 0; e < 9; ++e) M[e] = (e % 4 == 0) ? a.spray : 0.0f;
    }
    if(!__any_sync(0xffffffffu, need)) return;

    // pass 2: covariance about the weighted mean (AniKernelGenerator.cpp:80-89)
    float sw2 = 1.0f, c00 = 0.f, c01 = 0.f, c02 = 0.f, c11 = 0.f, c12 = 0.f, c22 = 0.f;
    const F2 Wx2 = pack2(-wx, -wx), Wy2 = pack2(-wy, -wy), Wz2 = pack2(-wz, -wz);
    for(int dz = -R; dz <= R; ++dz)
        for(int dy = -R; dy <= R; ++dy) {
            uint32_t s = 0, e = 0;
            if(need) row_range(g, a, cellStart, Px, Py, Pz, cj + dy, ck + dz, s, e);
            const uint32_t len = e - s;
#pragma unroll 2
            for(uint32_t i = s >> 1; 2 * i < e; ++i) {
                const uint32_t q = 2 * i;
                const ulonglong2 Qxy = __ldg(xy + i);
                const F2 Qx = Qxy.x, Qy = Qxy.y, Qz = __ldg(zz + i);
                const F2 ex = fma2(Qx, k2.minus1, Px2), ey = fma2(Qy, k2.minus1, Py2), ez = fma2(Qz, k2.minus1, Pz2);
                const F2 d2 = len2(ex, ey, ez, k2);
                const F2 x0 = add2(Qx, Wx2), x1 = add2(Qy, Wy2), x2 = add2(Qz, Wz2);
                const F2 q00 = mul2(x0, x0, k2), q11 = mul2(x1, x1, k2), q22 = mul2(x2, x2, k2);
                const F2 dm = add2(add2(q00, q11), q22);
                const bool h0 = lo2(d2) < a.r2 && q - s < len && q != self && lo2(dm) < a.r2;
                const bool h1 = hi2(d2) < a.r2 && q + 1 - s < len && q + 1 != self && hi2(dm) < a.r2;
                const F2 w = kernel_w2<FAST>(dm, rinv, k2);
                auto acc = [&](float c, F2 v) { return add_hits(c, mul2(w, v, k2), h0, h1); };
                sw2 = add_hits(sw2, w, h0, h1);
                c00 = acc(c00, q00);
                c01 = acc(c01, mul2(x0, x1, k2));
                c02 = acc(c02, mul2(x0, x2, k2));
                c11 = acc(c11, q11);
                c12 = acc(c12, mul2(x1, x2, k2));
                c22 = acc(c22, q22);
            }
        }
    if(!need) return;
    float C[3][3];
    C[0][0] = c00 / sw2; C[0][1] = c01 / sw2; C[0][2] = c02 / sw2;
    C[1][1] = c11 / sw2; C[1][2] = c12 / sw2; C[2][2] = c22 / sw2;
    C[1][0] = C[0][1]; C[2][0] = C[0][2]; C[2][1] = C[1][2];
    float M[9];
    kernel_matrix(C, a.axisRatio, M);
    float* out = outM + 9 * (size_t)id;
#pragma unroll
    for(int e = 0; e < 9; ++e) out[e] = M[e];
}

// Sorted points as pairs (PairPoints): point i is order[i] of the AoS positions, or i of the
// coordinate planes of stride `stride`; the last point of an odd number gets a mate at 0
template<bool PLANES>
__global__ void k_pack_pairs(const float* __restrict__ pos, size_t stride, const uint32_t* __restrict__ order, uint32_t n,
                             float4* __restrict__ xy, float2* __restrict__ z) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= (((size_t)n + 1) & ~(size_t)1)) return;
    float v[3] = {0.f, 0.f, 0.f};
    if(i < n) {
        const size_t p = PLANES ? i : order[i];
#pragma unroll
        for(int d = 0; d < 3; ++d) v[d] = PLANES ? pos[d * stride + p] : pos[3 * p + d];
    }
    float* at = reinterpret_cast<float*>(xy + (i >> 1)) + (i & 1);
    at[0] = v[0];
    at[2] = v[1];
    reinterpret_cast<float*>(z)[i] = v[2];
}

// order-preserving float <-> uint keys for atomic min / max
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
float fkey_inv(unsigned k) {
    const unsigned b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    std::memcpy(&f, &b, 4);
    return f;
}

// Bounding box of the points (keys[0..2] min, keys[3..5] max) and a count of non-finite
// coordinates (keys[6])
__global__ void __launch_bounds__(256) k_bounds(const float* __restrict__ pos, uint32_t n, unsigned* keys) {
    unsigned mn[3] = {~0u, ~0u, ~0u}, mx[3] = {0u, 0u, 0u}, bad = 0;
    for(size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x)
#pragma unroll
        for(int d = 0; d < 3; ++d) {
            const float v = pos[3 * p + d];
            if(!isfinite(v)) { ++bad; continue; }
            const unsigned k = fkey(v);
            mn[d] = min(mn[d], k);
            mx[d] = max(mx[d], k);
        }
#pragma unroll
    for(int d = 0; d < 3; ++d)
        for(int off = 16; off > 0; off >>= 1) {
            mn[d] = min(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], off));
            mx[d] = max(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], off));
        }
    for(int off = 16; off > 0; off >>= 1) bad += __shfl_xor_sync(0xffffffffu, bad, off);
    if((threadIdx.x & 31) == 0) {
        for(int d = 0; d < 3; ++d) { atomicMin(keys + d, mn[d]); atomicMax(keys + 3 + d, mx[d]); }
        if(bad) atomicAdd(keys + 6, bad);
    }
}

AnisoArgs make_args(const bnn_aniso_params& prm, float dx) {
    AnisoArgs a;
    // AnisotropicKernelGenerator constructor (AniKernelGenerator.cpp:30-42)
    const float r = prm.kernel_ratio * prm.particle_radius;
    a.r2 = r * r;
    a.r2m = a.r2 * (1.0f + 1e-4f);
    a.rinv = 1.0f / r;
    a.blend = prm.position_blending;
    a.axisRatio = prm.axis_ratio;
    a.spray = prm.default_spray_size;
    a.threshold = prm.neighbor_threshold;
    a.R = (int)(r / dx) + 2;
    a.margin = 0.01f * dx;
    return a;
}

// sqrt2 against sqrtf for the floats with bits [first, first + count), each in both halves beside
// another value of the range
__global__ void __launch_bounds__(256) k_sqrt_probe(unsigned first, unsigned count, Packed k, unsigned long long* bad) {
    unsigned wrong = 0;
    for(size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        const float a = __uint_as_float(first + (unsigned)i), b = __uint_as_float(first + (count - 1u - (unsigned)i));
        const F2 r = sqrt2(pack2(a, b), k);
        wrong += (__float_as_uint(lo2(r)) != __float_as_uint(sqrtf(a)) ? 1u : 0u) +
                 (__float_as_uint(hi2(r)) != __float_as_uint(sqrtf(b)) ? 1u : 0u);
    }
    if(wrong) atomicAdd(bad, (unsigned long long)wrong);
}
Packed packed_constants() {
    auto both = [](unsigned bits) { return (F2)bits << 32 | bits; };
    return Packed{both(0x80000000u), both(0xbf800000u), both(0x3f800000u)};
}

} // namespace

bnn_aniso_params aniso_defaults(float particleRadius) {
    // AniKernelGenerator.h:41-45 (constructor defaults) and :51 (setParameters defaults)
    bnn_aniso_params p;
    p.particle_radius = particleRadius;
    p.kernel_ratio = 8.0f;
    p.default_spray_size = 0.75f;
    p.position_blending = 0.5f;
    p.axis_ratio = 8.0f;
    p.neighbor_threshold = 25u;
    return p;
}

int aniso_check_params(const bnn_aniso_params& p) {
    const float r = p.kernel_ratio * p.particle_radius;
    if(!(r > 0.0f) || !std::isfinite(r) || !(p.axis_ratio > 0.0f)) return BNN_ERR_INVALID_ARGUMENT;
    return BNN_OK;
}

// Lays n sorted points out for launch_aniso
PairPoints aniso_pairs(void* mem, int n) {
    PairPoints q;
    q.xy = (float4*)mem;
    q.z = (float2*)(q.xy + ((size_t)n + 1) / 2);
    return q;
}
static void launch_pack(const PairPoints& q, const float* pos, size_t stride, const uint32_t* order, int n, cudaStream_t s) {
    const unsigned blocks = (unsigned)(((size_t)n + 256) / 256);
    if(order) k_pack_pairs<false><<<blocks, 256, 0, s>>>(pos, stride, order, (uint32_t)n, q.xy, q.z);
    else k_pack_pairs<true><<<blocks, 256, 0, s>>>(pos, stride, order, (uint32_t)n, q.xy, q.z);
    bnn_note_launch();
}
void launch_aniso_pack(const PairPoints& q, const float* planes, size_t stride, int n, cudaStream_t s) {
    if(n > 0) launch_pack(q, planes, stride, nullptr, n, s);
}

// The pass over cell-sorted points q (laid out by launch_aniso_pack), ids = input index of each
// sorted point, cellStart = C + 1 offsets of grid g.  counters[0] receives the spray points,
// counters[1] the points outside g (both must be zeroed by the caller).
cudaError_t launch_aniso(int n, const PairPoints& q, const uint32_t* ids, const uint32_t* cellStart, const AnisoGrid& g,
                         const bnn_aniso_params& prm, float* outC, float* outM, unsigned* counters, cudaStream_t s) {
    if(n <= 0) return cudaSuccess;
    const AnisoArgs a = make_args(prm, g.dx);
    const Packed k = packed_constants();
    const float r = prm.kernel_ratio * prm.particle_radius;
    const bool fast = r >= 0x1p-24f && r <= 0x1p24f;
    const unsigned blocks = (unsigned)((n + 127) / 128);
    const ulonglong2* xy = reinterpret_cast<const ulonglong2*>(q.xy);
    const F2* zz = reinterpret_cast<const F2*>(q.z);
    if(fast) k_aniso<true><<<blocks, 128, 0, s>>>(n, xy, zz, ids, cellStart, g, a, k, outC, outM, counters);
    else k_aniso<false><<<blocks, 128, 0, s>>>(n, xy, zz, ids, cellStart, g, a, k, outC, outM, counters);
    bnn_note_launch();
    return cudaGetLastError();
}

} // namespace bnn

using namespace bnn;

namespace {
// Temporary memory of the device's pool, in order on the caller's stream
struct DevMem {
    void* p = nullptr;
    cudaStream_t s = nullptr;
    ~DevMem() { if(p) cudaFreeAsync(p, s); }
    cudaError_t alloc(size_t b, cudaStream_t st) {
        const cudaError_t e = mem_pool_setup();
        if(e != cudaSuccess) return e;
        s = st;
        return cudaMallocAsync(&p, b ? b : 1, st);
    }
    template<class T> T* as() { return (T*)p; }
};
} // namespace

extern "C" int bnn_aniso_default_params(float particle_radius, bnn_aniso_params* out) {
    if(!out) return BNN_ERR_INVALID_ARGUMENT;
    *out = aniso_defaults(particle_radius);
    return BNN_OK;
}

extern "C" int bnn_aniso_sqrt_probe(uint64_t* tested, uint64_t* mismatches) {
    if(!tested || !mismatches) return BNN_ERR_INVALID_ARGUMENT;
    constexpr unsigned first = (127u - 100u) << 23, last = (127u + 100u) << 23;  // 2^-100 .. 2^100
    DevMem bad;
    BNN_CUDA_CHECK(bad.alloc(sizeof(unsigned long long), cudaStreamPerThread));
    BNN_CUDA_CHECK(cudaMemsetAsync(bad.p, 0, sizeof(unsigned long long), cudaStreamPerThread));
    k_sqrt_probe<<<2048, 256, 0, cudaStreamPerThread>>>(first, last - first + 1u, packed_constants(), bad.as<unsigned long long>());
    bnn_note_launch();
    BNN_CUDA_CHECK(cudaGetLastError());
    unsigned long long h = 0;
    BNN_CUDA_CHECK(cudaMemcpyAsync(&h, bad.p, sizeof(h), cudaMemcpyDeviceToHost, cudaStreamPerThread));
    BNN_CUDA_CHECK(cudaStreamSynchronize(cudaStreamPerThread));
    *tested = last - first + 1u;
    *mismatches = h;
    return BNN_OK;
}

extern "C" int bnn_anisotropic_kernels(const float* pos_dev, uint32_t n, const bnn_aniso_params* params,
                                       float* centers_dev, float* matrices_dev, bnn_aniso_stats* stats, void* stream) {
    if(!params || (n && (!pos_dev || !centers_dev || !matrices_dev))) return BNN_ERR_INVALID_ARGUMENT;
    int rc = aniso_check_params(*params);
    if(rc != BNN_OK) return rc;
    if(stats) std::memset(stats, 0, sizeof(*stats));
    if(n == 0) return BNN_OK;
    cudaStream_t s = (cudaStream_t)stream;
    // bounding box of the points -> the cell grid (cells of a quarter kernel radius)
    DevMem keys;
    BNN_CUDA_CHECK(keys.alloc(8 * sizeof(unsigned), s));
    const unsigned init[8] = {~0u, ~0u, ~0u, 0u, 0u, 0u, 0u, 0u};
    BNN_CUDA_CHECK(cudaMemcpyAsync(keys.p, init, sizeof(init), cudaMemcpyHostToDevice, s));
    { k_bounds<<<(unsigned)std::min<size_t>(((size_t)n + 255) / 256, 4 * 148), 256, 0, s>>>(pos_dev, n, keys.as<unsigned>()); bnn_note_launch(); }
    unsigned hk[8];
    BNN_CUDA_CHECK(cudaMemcpyAsync(hk, keys.p, sizeof(hk), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    if(hk[6]) {
        bnn_set_error("bnn_anisotropic_kernels: non-finite coordinates");
        return BNN_ERR_INVALID_ARGUMENT;
    }
    const float r = params->kernel_ratio * params->particle_radius;
    AnisoGrid g;
    float lo[3], hi[3];
    for(int d = 0; d < 3; ++d) { lo[d] = fkey_inv(hk[d]); hi[d] = fkey_inv(hk[3 + d]); g.bmin[d] = lo[d]; }
    float cell = 0.25f * r;
    for(;;) {
        size_t C = 1;
        for(int d = 0; d < 3; ++d) {
            const float t = (hi[d] - lo[d]) / cell;
            g.G[d] = (int)t + 1;
            C *= (size_t)g.G[d];
        }
        if(C <= ((size_t)1 << 27)) break;
        cell = cell * std::cbrt((float)C / (float)((size_t)1 << 27)) * 1.01f;
    }
    g.dx = cell;
    const size_t C = (size_t)g.G[0] * g.G[1] * g.G[2];
    DevMem cid, order, start, pairs, cnt;
    BNN_CUDA_CHECK(cid.alloc((size_t)n * 4, s));
    BNN_CUDA_CHECK(order.alloc((size_t)n * 4, s));
    BNN_CUDA_CHECK(start.alloc((C + 1) * 4, s));
    BNN_CUDA_CHECK(pairs.alloc(pair_bytes(n), s));
    BNN_CUDA_CHECK(cnt.alloc(2 * sizeof(unsigned), s));
    uint32_t oor = 0;
    rc = bnn_cell_sort(pos_dev, n, g.bmin, g.dx, g.G, cid.as<uint32_t>(), order.as<uint32_t>(), start.as<uint32_t>(),
                       &oor, stream);
    if(rc != BNN_OK) return rc;
    const PairPoints q = aniso_pairs(pairs.p, (int)n);
    launch_pack(q, pos_dev, 0, order.as<uint32_t>(), (int)n, s);
    BNN_CUDA_CHECK(cudaMemsetAsync(cnt.p, 0, 2 * sizeof(unsigned), s));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    BNN_CUDA_CHECK(launch_aniso((int)n, q, order.as<uint32_t>(), start.as<uint32_t>(), g, *params, centers_dev, matrices_dev,
                                cnt.as<unsigned>(), s));
    cudaEventRecord(e1, s);
    unsigned hc[2];
    BNN_CUDA_CHECK(cudaMemcpyAsync(hc, cnt.p, sizeof(hc), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    BNN_CUDA_CHECK(cudaGetLastError());
    if(stats) {
        for(int d = 0; d < 3; ++d) { stats->grid_bmin[d] = g.bmin[d]; stats->grid_dims[d] = g.G[d]; }
        stats->grid_cell_size = g.dx;
        stats->sprays = hc[0];
        stats->ms = ms;
    }
    if(oor || hc[1]) {
        bnn_set_error("bnn_anisotropic_kernels: a point fell outside its cell grid");
        return BNN_ERR_DEVICE_CHECK;
    }
    return BNN_OK;
}
