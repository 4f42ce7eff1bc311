// Matrix-free Jacobi PCG for the 7-point pressure system (PCGSolver::solve_precond,
// BananaCore/Banana/LinearAlgebra/LinearSolvers/PCGSolver.cpp:143-199).
//
// Rows are the fluid cells in linear-cell order.  Per row: diag (float), 1/diag, and six
// neighbour row indices in ascending column order (-z,-y,-x,+x,+y,+z; -1 = none), stored
// as six planes nbr[q*n + r].  With face weights 1 every off-diagonal equals -dt, so the
// matrix is never materialised; with solid boundaries (weights below 1) the off-diagonal
// values ride along: six planes coef[q*n + r] with the compact rows, or two float4 per
// row (k_pack_coef) with the packed ones.
//
// Rows of a grid (rows numbered in cell order) are also packed into one 16-byte record
// each: the x neighbours are always rows r-1 / r+1, so they become two flag bits, the y
// and z neighbours become row distances, and the diagonal rides along.  One load then
// replaces seven, and the x neighbours' values come from the adjacent lanes by warp
// shuffles instead of loads.  Record {y, zm, zp, diag}: y = dy- | dy+ << 16 (row distances
// of the -y / +y neighbours, 0 = none), zm = dz- | (has -x) << 31, zp = dz+ | (has +x) << 31.
//
// A system whose chunks fit on the chip is solved by k_pcg_cluster or k_pcg_chunk (below), from
// the compact rows.  Beyond that the solve is k_pcg_persistent, one persistent cooperative
// kernel on the packed ones.  In all of them every iteration works in the canonical
// 2048-row chunk layout so the FP64 dot products are bit-reproducible:
//   phase A: s = z + beta*s_old formed on the fly (double buffered), q = A s, partial s.q;
//   grid barrier; every block reduces the partials to the same alpha;
//   phase B: x += alpha s, r -= alpha q, max|r|, z = D^-1 r, partial z.r;
//   grid barrier; every block reduces to the same rho, max|r| and beta.
#include "bnn_internal.cuh"
#include "coop_share.cuh"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

namespace bnn {

template<class VT> struct Sc;
template<> struct Sc<float> {
    __device__ static float alpha(const DevState* s) { return s->alpha; }
    __device__ static float beta(const DevState* s) { return s->beta; }
    __device__ static void set_alpha(DevState* s, double a) { s->alpha = (float)a; }
    __device__ static void set_beta(DevState* s, double b) { s->beta = (float)b; }
    __device__ static float tol(const DevState* s) { return s->tol; }
    __device__ static void set_tol(DevState* s, float t) { s->tol = t; }
    __device__ static void set_resid(DevState* s, float r) { s->resid = r; s->resid64 = r; }
};
template<> struct Sc<double> {
    __device__ static double alpha(const DevState* s) { return s->alpha64; }
    __device__ static double beta(const DevState* s) { return s->beta64; }
    __device__ static void set_alpha(DevState* s, double a) { s->alpha64 = a; }
    __device__ static void set_beta(DevState* s, double b) { s->beta64 = b; }
    __device__ static double tol(const DevState* s) { return s->tol64; }
    __device__ static void set_tol(DevState* s, double t) { s->tol64 = t; }
    __device__ static void set_resid(DevState* s, double r) { s->resid64 = r; s->resid = (float)r; }
};

template<class VT> __device__ __forceinline__ VT vabs(VT x) { return x < VT(0) ? -x : x; }

template<class VT> __device__ __forceinline__ VT block_max_t(VT v, VT* sm) {
    const int t = threadIdx.x;
    sm[t] = v;
    __syncthreads();
    for(int off = 128; off > 0; off >>= 1) {
        if(t < off) { VT o = sm[t + off]; sm[t] = sm[t] > o ? sm[t] : o; }
        __syncthreads();
    }
    VT r = sm[0];
    __syncthreads();
    return r;
}
template<class VT> __device__ __forceinline__ VT reduce_max_t(const VT* part, int nch, VT* sm) {
    VT acc = VT(0);
    for(int c = threadIdx.x; c < nch; c += kLanes) { VT o = __ldcg(part + c); acc = acc > o ? acc : o; }
    return block_max_t(acc, sm);
}

// ---------------------------------------------------------------------------------
// Persistent PCG: one cooperative launch per solve.  Blocks own fixed 2048-row chunks
// (c = blockIdx.x, +gridDim.x, ...), every phase writes one FP64 partial per chunk, and
// after each grid barrier EVERY block reduces the partials in the canonical order, so all
// blocks hold bit-identical scalars and take the same branch without a broadcast.  Data
// written by other blocks is read with ld.global.cg (L2), never through a stale L1 line.
// ---------------------------------------------------------------------------------
// A barrier wait gives up once it has polled minSpins times and ns more of wall time
// (%globaltimer) have passed, or after maxSpins polls whatever the clock says.  Counting
// polls as well as time keeps a solve that the GPU time-slices away from giving up early.
struct BarrierLimit {
    unsigned long long ns;
    unsigned minSpins, maxSpins;
};
__host__ __device__ constexpr BarrierLimit solve_barrier_limit() { return {1000000000ull, 1u << 20, 1u << 26}; }
// Pause between polls of the barrier word: fewer acquire loads queue at the word's L2
// slice behind the arrivals (1.59M-row solve, us per iteration: 22.59 without a pause,
// 22.42-22.46 at 32 or 100 ns, 22.74 at 256, 22.83-22.92 at 1000; a relaxed poll followed
// by one acquire fence: 23.24)
#ifndef BNN_BARRIER_SLEEP_NS
#define BNN_BARRIER_SLEEP_NS 100
#endif

// Canonical 256-lane tree (lane t of the chunk owns v; levels 128, 64, 32 then a warp
// shuffle tree), with one shared-memory staging step: warp 0 forms the three upper
// levels in registers in the same association as the level-by-level tree.  The sum is
// valid in thread 0.  `m` (optional) is max-reduced alongside.
template<class VT>
__device__ __forceinline__ void block_sum_max_256(double v, VT m, double* sm, VT* smm, double& sum, VT& mx,
                                                  bool withMax) {
    const int t = threadIdx.x;
    sm[t] = v;
    if(withMax) smm[t] = m;
    __syncthreads();
    if(t < 32) {
        const double a0 = sm[t] + sm[t + 128];
        const double a1 = sm[t + 64] + sm[t + 192];
        const double a2 = sm[t + 32] + sm[t + 160];
        const double a3 = sm[t + 96] + sm[t + 224];
        double c = (a0 + a1) + (a2 + a3);
#pragma unroll
        for(int off = 16; off > 0; off >>= 1) c = c + __shfl_down_sync(0xffffffffu, c, off);
        sum = c;
        if(withMax) {
            VT x = smm[t];
#pragma unroll
            for(int q = 1; q < 8; ++q) { const VT o = smm[t + 32 * q]; x = x > o ? x : o; }
#pragma unroll
            for(int off = 16; off > 0; off >>= 1) { const VT o = __shfl_down_sync(0xffffffffu, x, off); x = x > o ? x : o; }
            mx = x;
        }
    }
    __syncthreads();
}

// Reduce the chunk partials (sum in canonical order, and max) and give the result to
// every thread of the block.  A thread's partials (chunks t, t + 256, ...) are loaded four
// at a time before they are added in chunk order; warp 0 forms the block result and lane 0
// publishes it in its own shared slot, so one block barrier separates it from the readers
// (the next write of the slot comes after the next reduction's first barrier, which every
// reader reaches only after reading).
template<class VT>
__device__ __forceinline__ void reduce_partials_bcast(const double* part, const VT* pmax, int nch, double* sm, VT* smm,
                                                      double& sum, VT& mx) {
    __shared__ double sSum;
    __shared__ VT sMax;
    constexpr int U = 4;
    double acc = 0.0;
    VT m = VT(0);
    for(int c0 = threadIdx.x; c0 < nch; c0 += U * kLanes) {
        double p[U];
        VT o[U];
#pragma unroll
        for(int u = 0; u < U; ++u) {
            const int c = c0 + u * kLanes;
            p[u] = c < nch ? __ldcg(part + c) : 0.0;
            o[u] = (pmax && c < nch) ? __ldcg(pmax + c) : VT(0);
        }
#pragma unroll
        for(int u = 0; u < U; ++u)
            if(c0 + u * kLanes < nch) {
                acc = acc + p[u];
                if(pmax) m = m > o[u] ? m : o[u];
            }
    }
    const int t = threadIdx.x;
    sm[t] = acc;
    if(pmax) smm[t] = m;
    __syncthreads();
    if(t < 32) {
        // the association of block_sum_max_256
        const double a0 = sm[t] + sm[t + 128];
        const double a1 = sm[t + 64] + sm[t + 192];
        const double a2 = sm[t + 32] + sm[t + 160];
        const double a3 = sm[t + 96] + sm[t + 224];
        double c = (a0 + a1) + (a2 + a3);
#pragma unroll
        for(int off = 16; off > 0; off >>= 1) c = c + __shfl_down_sync(0xffffffffu, c, off);
        VT x = VT(0);
        if(pmax) {
            x = smm[t];
#pragma unroll
            for(int q = 1; q < 8; ++q) { const VT o = smm[t + 32 * q]; x = x > o ? x : o; }
#pragma unroll
            for(int off = 16; off > 0; off >>= 1) { const VT o = __shfl_down_sync(0xffffffffu, x, off); x = x > o ? x : o; }
        }
        if(t == 0) { sSum = c; sMax = x; }
    }
    __syncthreads();
    sum = sSum;
    mx = sMax;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_add_release_u32(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" : : "l"(p), "r"(v) : "memory");
}

// Grid-wide barrier with a bounded wait (sense reversal on one word, zeroed before the
// launch): block 0 adds 2^31 - (nblocks - 1), every other block adds 1, so the word's top
// bit flips exactly when the last block arrives and its low bits return to where they
// were.  After the b-th barrier the top bit is b & 1; each block counts its barriers in
// `sense`, so the arrival is a fire-and-forget reduction (release) and the poll (acquire)
// starts at once.  Each block's writes before the barrier are visible to every block
// after it.  Returns false (and sets the timeout flag) when the wait gave up.
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool grid_barrier(GridSync* gs, unsigned nblocks, unsigned& sense, unsigned* flags,
                                             BarrierLimit lim) {
    __shared__ int sOk;
    sense ^= 1u;
    __syncthreads();
    if(threadIdx.x == 0) {
        int ok = 1;
        const unsigned add = blockIdx.x == 0 ? 0x80000000u - (nblocks - 1u) : 1u;
        red_add_release_u32(&gs->count, add);
        unsigned spins = 0;
        unsigned long long t0 = 0;
        while((ld_acquire_u32(&gs->count) >> 31) != sense) {
            ++spins;
            if(spins == lim.minSpins) t0 = global_ns();
            if(spins >= lim.maxSpins || (spins > lim.minSpins && (spins & 255u) == 0u && global_ns() - t0 >= lim.ns)) {
                ok = 0;
                atomicOr(flags, BNN_FLAG_TIMEOUT);
                break;
            }
            if(BNN_BARRIER_SLEEP_NS) __nanosleep(BNN_BARRIER_SLEEP_NS);
        }
        sOk = ok;
    }
    __syncthreads();
    return sOk != 0;
}

template<class VT> struct PcgArgs {
    int n;
    const float* rhsF;
    const float* diag;
    const VT* invd;
    const int32_t* nbr;
    const int4* rec;
    const float* coef;  // compact rows: off-diagonal planes (nullptr: all negoff)
    const float4* coefRow;  // packed rows with coefficients: 2 float4 per row (6 used)
    VT negoff;
    VT tolFactor;
    unsigned maxIter;
    VT *x, *r, *z, *s0, *s1, *q;
    double *part0, *part1, *part2;
    VT* partMax;
    DevState* st;
    GridSync* gs;
};

template<class VT>
__device__ __forceinline__ VT s_val(const VT* z, const VT* sOld, VT beta, bool first, size_t e) {
    return first ? __ldcg(z + e) : __ldcg(z + e) + beta * __ldcg(sOld + e);
}

// Resident blocks per SM the register budget is sized for, and rows per lane whose loads
// are in flight together in the SpMV phase (a divisor of kPerLane).  With the chunk's row
// records loaded before its neighbour loads, three blocks of two rows run best for every
// vector type (1.59M rows, us per iteration: FP32 22.9 against 23.5 at two blocks of four
// rows and 23.9 at two blocks of two; FP64 42.1 against 44.5 and 46.8; rows with
// off-diagonal values 38.5 against 42.6 at two blocks of four rows, which spill).
#ifndef BNN_PCG_MIN_BLOCKS
#define BNN_PCG_MIN_BLOCKS 3
#endif
#ifndef BNN_PCG_ROW_GROUP
#define BNN_PCG_ROW_GROUP 2
#endif
#ifndef BNN_PCG_MIN_BLOCKS_F64
#define BNN_PCG_MIN_BLOCKS_F64 3
#endif
#ifndef BNN_PCG_ROW_GROUP_F64
#define BNN_PCG_ROW_GROUP_F64 2
#endif
#ifndef BNN_PCG_MIN_BLOCKS_COEF
#define BNN_PCG_MIN_BLOCKS_COEF 3
#endif
#ifndef BNN_PCG_ROW_GROUP_COEF
#define BNN_PCG_ROW_GROUP_COEF 2
#endif
template<class VT, bool COEF> constexpr int pcg_min_blocks() {
    return sizeof(VT) == 8 ? BNN_PCG_MIN_BLOCKS_F64 : (COEF ? BNN_PCG_MIN_BLOCKS_COEF : BNN_PCG_MIN_BLOCKS);
}
template<class VT, bool COEF> constexpr int pcg_row_group() {
    return sizeof(VT) == 8 ? BNN_PCG_ROW_GROUP_F64 : (COEF ? BNN_PCG_ROW_GROUP_COEF : BNN_PCG_ROW_GROUP);
}
template<class VT, bool PACKED, bool COEF = false>
__global__ void __launch_bounds__(kLanes, pcg_min_blocks<VT, COEF>()) k_pcg_persistent(PcgArgs<VT> a) {
    constexpr int kRowGroup = pcg_row_group<VT, COEF>();
    static_assert(kPerLane % kRowGroup == 0, "row groups must tile a lane's rows");
    __shared__ double smd[kLanes];
    __shared__ VT smv[kLanes];
    const int n = a.n;
    const int nch = (n + kChunk - 1) / kChunk;
    const unsigned nb = gridDim.x;
    unsigned sense = 0;  // barriers passed, mod 2
    unsigned* flags = &a.st->flags;
    VT* __restrict__ xR = a.x;
    VT* __restrict__ rR = a.r;
    VT* __restrict__ zR = a.z;
    VT* __restrict__ qR = a.q;
    const VT* __restrict__ invdR = a.invd;
    const float* __restrict__ diagR = a.diag;
    const int32_t* __restrict__ nbrR = a.nbr;
    const int4* __restrict__ recR = a.rec;
    const float* __restrict__ coefR = a.coef;
    const VT negoff = a.negoff;
    const int lane = threadIdx.x & 31;

    // ---- init: r = rhs, x = 0, z = D^-1 r; partial z.r and max|r| (PCGSolver.cpp:151-168)
    for(int c = blockIdx.x; c < nch; c += nb) {
        double acc = 0.0;
        VT m = VT(0);
        const size_t base = (size_t)c * kChunk + threadIdx.x;
#pragma unroll
        for(int j = 0; j < kPerLane; ++j) {
            const size_t e = base + (size_t)j * kLanes;
            if(e < (size_t)n) {
                const VT rv = (VT)a.rhsF[e];
                a.r[e] = rv;
                a.x[e] = VT(0);
                const VT ab = vabs(rv);
                m = m > ab ? m : ab;
                const VT zv = __ldg(a.invd + e) * rv;
                a.z[e] = zv;
                acc = acc + (double)zv * (double)rv;
            }
        }
        double bs;
        VT bm;
        block_sum_max_256<VT>(acc, m, smd, smv, bs, bm, true);
        if(threadIdx.x == 0) { a.part0[c] = bs; a.partMax[c] = bm; }
    }
    if(!grid_barrier(a.gs, nb, sense, flags, solve_barrier_limit())) return;
    double rho;
    VT resid;
    reduce_partials_bcast<VT>(a.part0, a.partMax, nch, smd, smv, rho, resid);
    const VT tolFactor = fmax(a.tolFactor, VT(1e-30));
    unsigned iter = 0, success = 0;
    bool done = false;
    VT tol = VT(0);
    if(resid < (VT)FLT_MIN) {
        done = true;
        success = 1;
    } else {
        tol = tolFactor * resid;
        if(rho < (double)FLT_MIN || isnan(rho)) done = true;
    }
    if(a.maxIter == 0) done = true;

    VT beta = VT(0);
    bool first = true;
#ifdef BNN_PCG_TIMING
    unsigned long long tc[6] = {0, 0, 0, 0, 0, 0};
    long long t0_ = clock64();
#define TMARK(k) do { long long t1_ = clock64(); tc[k] += (unsigned long long)(t1_ - t0_); t0_ = t1_; } while(0)
#else
#define TMARK(k) do {} while(0)
#endif
    VT* sOld = a.s1;
    VT* sNew = a.s0;
    while(!done) {
        // ---- phase A: s = z + beta s_old, q = A s, partial s.q (PCGSolver.cpp:173-174,192-193)
        // Every load of a chunk is issued before any store (missing neighbours read the
        // row itself and are masked afterwards), so the chunk costs a few L2 round trips
        // instead of one per row and neighbour.
        for(int c = blockIdx.x; c < nch; c += nb) {
            const size_t base = (size_t)c * kChunk + threadIdx.x;
            VT sOut[kPerLane], qOut[kPerLane];
            // the row records of the whole chunk first: one round trip for all of them
            int4 recAll[PACKED ? kPerLane : 1];
            if constexpr(PACKED) {
#pragma unroll
                for(int j = 0; j < kPerLane; ++j) {
                    const size_t e = base + (size_t)j * kLanes;
                    recAll[j] = __ldg(recR + (e < (size_t)n ? e : 0));
                }
            }
#pragma unroll
            for(int g0 = 0; g0 < kPerLane; g0 += kRowGroup) {
                int32_t id[kRowGroup][7];
                bool has[kRowGroup][7];
                float dg[kRowGroup];
                size_t rowE[kRowGroup];
#pragma unroll
                for(int u = 0; u < kRowGroup; ++u) {
                    const size_t e = base + (size_t)(g0 + u) * kLanes;
                    const size_t ee = e < (size_t)n ? e : 0;
                    if constexpr(PACKED) {
                        // a row past n reads row 0, whose neighbours are all valid rows
                        const int4 rr = recAll[g0 + u];
                        const int dyM = rr.x & 0xffff, dyP = (int)((unsigned)rr.x >> 16);
                        const int dzM = rr.y & 0x7fffffff, dzP = rr.z & 0x7fffffff;
                        const int32_t r0 = (int32_t)ee;
                        has[u][0] = dzM != 0; id[u][0] = r0 - dzM;
                        has[u][1] = dyM != 0; id[u][1] = r0 - dyM;
                        // x neighbours: lanes 0 / 31 load them, the others take a shuffle
                        has[u][2] = rr.y < 0; id[u][2] = (lane == 0 && rr.y < 0) ? r0 - 1 : r0;
                        has[u][3] = true; id[u][3] = r0;
                        has[u][4] = rr.z < 0; id[u][4] = (lane == 31 && rr.z < 0) ? r0 + 1 : r0;
                        has[u][5] = dyP != 0; id[u][5] = r0 + dyP;
                        has[u][6] = dzP != 0; id[u][6] = r0 + dzP;
                        dg[u] = __int_as_float(rr.w);
                    } else {
#pragma unroll
                        for(int q = 0; q < 6; ++q) {
                            const int32_t v = __ldg(nbrR + (size_t)q * n + ee);
                            const int slot = q < 3 ? q : q + 1;
                            has[u][slot] = v >= 0;
                            id[u][slot] = v >= 0 ? v : (int32_t)ee;
                        }
                        rowE[u] = ee;
                        id[u][3] = (int32_t)ee;
                        has[u][3] = true;
                        dg[u] = __ldg(diagR + ee);
                    }
                }
                VT zv[kRowGroup][7], sv[kRowGroup][7];
#pragma unroll
                for(int u = 0; u < kRowGroup; ++u)
#pragma unroll
                    for(int q = 0; q < 7; ++q) {
                        const bool load = !PACKED || (q != 2 && q != 4) || (q == 2 && lane == 0) || (q == 4 && lane == 31);
                        zv[u][q] = load ? __ldcg(zR + id[u][q]) : VT(0);
                        sv[u][q] = (first || !load) ? VT(0) : __ldcg(sOld + id[u][q]);
                    }
#pragma unroll
                for(int u = 0; u < kRowGroup; ++u) {
                    VT s7[7];
#pragma unroll
                    for(int q = 0; q < 7; ++q) s7[q] = first ? zv[u][q] : zv[u][q] + beta * sv[u][q];
                    if constexpr(PACKED) {
                        // rows e-1 / e+1 belong to the neighbouring lanes of this warp
                        const VT up = __shfl_up_sync(0xffffffffu, s7[3], 1);
                        const VT dn = __shfl_down_sync(0xffffffffu, s7[3], 1);
                        if(lane != 0) s7[2] = up;
                        if(lane != 31) s7[4] = dn;
                    }
                    VT t = VT(0);
                    if constexpr(PACKED && COEF) {
                        // the row's off-diagonals in slot order (-z, -y, -x | +x, +y, +z)
                        const size_t e = base + (size_t)(g0 + u) * kLanes;
                        const size_t ee = e < (size_t)n ? e : 0;
                        const float4 c0 = __ldg(a.coefRow + 2 * ee), c1 = __ldg(a.coefRow + 2 * ee + 1);
                        const VT co[7] = {(VT)c0.x, (VT)c0.y, (VT)c0.z, VT(0), (VT)c0.w, (VT)c1.x, (VT)c1.y};
#pragma unroll
                        for(int q = 0; q < 3; ++q) if(has[u][q]) t += co[q] * s7[q];
                        if(dg[u] != 0.f) t += (VT)dg[u] * s7[3];
#pragma unroll
                        for(int q = 4; q < 7; ++q) if(has[u][q]) t += co[q] * s7[q];
                    } else if constexpr(PACKED) {
#pragma unroll
                        for(int q = 0; q < 3; ++q) if(has[u][q]) t += negoff * s7[q];
                        if(dg[u] != 0.f) t += (VT)dg[u] * s7[3];
#pragma unroll
                        for(int q = 4; q < 7; ++q) if(has[u][q]) t += negoff * s7[q];
                    } else {
                        // off-diagonal of slot q (plane q, or q - 1 above the diagonal)
                        auto cf = [&](int q) {
                            return coefR ? (VT)__ldg(coefR + (size_t)(q < 3 ? q : q - 1) * n + rowE[u]) : negoff;
                        };
#pragma unroll
                        for(int q = 0; q < 3; ++q) if(has[u][q]) t += cf(q) * s7[q];
                        if(dg[u] != 0.f) t += (VT)dg[u] * s7[3];
#pragma unroll
                        for(int q = 4; q < 7; ++q) if(has[u][q]) t += cf(q) * s7[q];
                    }
                    sOut[g0 + u] = s7[3];
                    qOut[g0 + u] = t;
                }
            }
            double acc = 0.0;
#pragma unroll
            for(int j = 0; j < kPerLane; ++j) {
                const size_t e = base + (size_t)j * kLanes;
                if(e < (size_t)n) {
                    sNew[e] = sOut[j];
                    qR[e] = qOut[j];
                    acc = acc + (double)sOut[j] * (double)qOut[j];
                }
            }
            double bs;
            VT unused;
            block_sum_max_256<VT>(acc, VT(0), smd, smv, bs, unused, false);
            if(threadIdx.x == 0) a.part1[c] = bs;
        }
        TMARK(0);
        if(!grid_barrier(a.gs, nb, sense, flags, solve_barrier_limit())) return;
        TMARK(1);
        double tmp;
        VT unused2;
        reduce_partials_bcast<VT>(a.part1, (const VT*)nullptr, nch, smd, smv, tmp, unused2);
        if(tmp < (double)FLT_MIN) {
            ++iter;
            success = 1;
            break;
        }
        const VT alpha = (VT)(rho / tmp);
        TMARK(2);
        // ---- phase B: x += alpha s, r -= alpha q, max|r|, z = D^-1 r, partial z.r
        for(int c = blockIdx.x; c < nch; c += nb) {
            const size_t base = (size_t)c * kChunk + threadIdx.x;
            VT xs[kPerLane], ss[kPerLane], rs[kPerLane], qs[kPerLane], is[kPerLane];
#pragma unroll
            for(int j = 0; j < kPerLane; ++j) {
                const size_t e = base + (size_t)j * kLanes;
                const size_t ee = e < (size_t)n ? e : 0;
                xs[j] = __ldcg(xR + ee);
                ss[j] = __ldcg(sNew + ee);
                rs[j] = __ldcg(rR + ee);
                qs[j] = __ldcg(qR + ee);
                is[j] = __ldg(invdR + ee);
            }
            double acc = 0.0;
            VT m = VT(0);
#pragma unroll
            for(int j = 0; j < kPerLane; ++j) {
                const size_t e = base + (size_t)j * kLanes;
                if(e < (size_t)n) {
                    xR[e] = xs[j] + alpha * ss[j];
                    const VT rv = rs[j] + (-alpha) * qs[j];
                    rR[e] = rv;
                    const VT ab = vabs(rv);
                    m = m > ab ? m : ab;
                    const VT zv = is[j] * rv;
                    zR[e] = zv;
                    acc = acc + (double)zv * (double)rv;
                }
            }
            double bs;
            VT bm;
            block_sum_max_256<VT>(acc, m, smd, smv, bs, bm, true);
            if(threadIdx.x == 0) { a.part2[c] = bs; a.partMax[c] = bm; }
        }
        TMARK(3);
        if(!grid_barrier(a.gs, nb, sense, flags, solve_barrier_limit())) return;
        TMARK(4);
        double rhoNew;
        reduce_partials_bcast<VT>(a.part2, a.partMax, nch, smd, smv, rhoNew, resid);
        TMARK(5);
        ++iter;
        if(resid < tol) {
            success = 1;
            break;
        }
        beta = (VT)(rhoNew / rho);
        rho = rhoNew;
        if(iter >= a.maxIter) {
            if(blockIdx.x == 0 && threadIdx.x == 0) atomicOr(flags, BNN_FLAG_PCG_MAXITER);
            break;
        }
        VT* t = sOld;
        sOld = sNew;
        sNew = t;
        first = false;
    }
#ifdef BNN_PCG_TIMING
    if(threadIdx.x == 0) {
        unsigned smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        printf("blk %d sm %u iters %u  cycles/iter: phaseA %.0f bar1 %.0f red1 %.0f phaseB %.0f bar2 %.0f red2 %.0f\n",
               (int)blockIdx.x, smid, iter, tc[0] / (double)iter, tc[1] / (double)iter, tc[2] / (double)iter,
               tc[3] / (double)iter, tc[4] / (double)iter, tc[5] / (double)iter);
    }
#endif
    if(blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->iter = iter;
        a.st->success = success;
        a.st->done = 1;
        Sc<VT>::set_resid(a.st, resid);
    }
}

// The 16-byte record of row r (layout at the top of this file).  The caller guarantees the
// x neighbours are rows r-1 / r+1 and the y distances fit 16 bits.
__device__ __forceinline__ int4 pack_row(int r, const int32_t nb[6], float diag) {
    const unsigned dyM = nb[1] >= 0 ? (unsigned)(r - nb[1]) : 0u, dyP = nb[4] >= 0 ? (unsigned)(nb[4] - r) : 0u;
    const unsigned dzM = nb[0] >= 0 ? (unsigned)(r - nb[0]) : 0u, dzP = nb[5] >= 0 ? (unsigned)(nb[5] - r) : 0u;
    int4 v;
    v.x = (int)(dyM | (dyP << 16));
    v.y = (int)(dzM | (nb[2] >= 0 ? 0x80000000u : 0u));
    v.z = (int)(dzP | (nb[3] >= 0 ? 0x80000000u : 0u));
    v.w = __float_as_int(diag);
    return v;
}

// ---------------------------------------------------------------------------------
// Chunk-resident PCG: the same iteration for systems whose 2048-row chunks are all on the
// chip at once.  One block per SM, of G groups of 256 threads; a group owns K chunks for the
// whole solve and keeps what its own rows need on the chip: r and z / q in registers, s and
// the row records in shared memory.  Only what other blocks read crosses L2 on the critical
// path: a pair {z, s} per row, written once per iteration (phase B) and read by its z
// neighbours and across chunk ends (phase A).  The pairs are double-buffered by the exchange's
// parity: the second exchange, which passes them on, releases and acquires, the first does not,
// so a buffer is written again only after a second exchange that followed its reads.  The x and
// y neighbours inside a chunk are read from shared memory.
//
// The grid barriers are merged with the reductions: a group publishes a chunk's partial sum
// and max as one 16-byte packet, and every block polls the packets of all chunks and adds them
// in the canonical order; a block has passed when it has seen all of them.  A packet's max
// carries the parity of its exchange in the top bit (a block is at most one exchange ahead of
// the slowest, so one bit tells old from new; the packets start zeroed).  Packets lie 128
// bytes apart so that the polls of all blocks spread over the L2 slices; the word behind a
// packet says that its chunk's pairs can be read (kSplit).  The x update overlaps the second
// wait.
//
// What bounds it: up to a chunk per SM the latency of the two exchanges (a packet's way through
// L2, the FP64 trees on both sides, the pairs' way to L2) and of one round of neighbour loads; at
// six chunks per SM the instructions of phase A, the pair stores of phase B and the
// FP32-to-FP64 conversions of the products (16 a clock and SM).  One block per SM instead of
// three: one poller per SM, and a group's registers can hold a whole chunk's loads.
// Measured, us per iteration with everything around it (k_pcg_persistent before): FP32 161,057
// rows 5.0 (9.63), 315,698 6.25 (10.96), 705,846 8.3 (13.81), 1,283,026 15.1 (22.1), 1,736,304
// 17.3 (22.9); FP64 315,698 7.4 (15.2), 705,846 13.9 (19.8).  One buffer of pairs, whose rewriting
// only the order of loads and dependent stores keeps off its readers: 0 to 3 % less (705,846 rows
// 8.15, 1,736,304 16.8); one buffer and a first exchange that releases and acquires: 8.95, 17.95.
// ---------------------------------------------------------------------------------
template<class VT> struct alignas(2 * sizeof(VT)) RowPair {
    VT z, s;
};
// A pair where `on`, zeros elsewhere, as one predicated load (a branch around each of a
// row's loads costs more than the load)
template<class VT> __device__ __forceinline__ RowPair<VT> ld_pair_if(const RowPair<VT>* p, bool on) {
    RowPair<VT> v{VT(0), VT(0)};
    if constexpr(sizeof(VT) == 4)
        asm volatile("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p ld.global.cg.v2.f32 {%0, %1}, [%2]; }"
                     : "+f"(v.z), "+f"(v.s) : "l"(p), "r"((int)on) : "memory");
    else
        asm volatile("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p ld.global.cg.v2.f64 {%0, %1}, [%2]; }"
                     : "+d"(v.z), "+d"(v.s) : "l"(p), "r"((int)on) : "memory");
    return v;
}
// volatile: issued where it stands, ahead of a wait
__device__ __forceinline__ float ld_const_if(const float* p, bool on) {
    float v = 0.f;
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %2, 0; @p ld.global.nc.f32 %0, [%1]; }" : "+f"(v) : "l"(p), "r"((int)on));
    return v;
}
__device__ __forceinline__ double ld_const_if(const double* p, bool on) {
    double v = 0.0;
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %2, 0; @p ld.global.nc.f64 %0, [%1]; }" : "+d"(v) : "l"(p), "r"((int)on));
    return v;
}
// A chunk's partial of one exchange: the bits of the FP64 sum, and of the max in its vector
// type, the exchange's parity in the top bit
struct alignas(16) PcgPacket {
    unsigned long long sum, max;
};
constexpr int kPacketStride = 8;  // packets apart
__device__ __forceinline__ unsigned long long max_bits(float m) { return __float_as_uint(m) & 0x7fffffffu; }
// The mask is written out: in C it is the absolute value to the compiler, whose result for a NaN may
// have either sign (abs.f64), and the sign's place is the parity's
__device__ __forceinline__ unsigned long long max_bits(double m) {
    unsigned long long b = (unsigned long long)__double_as_longlong(m);
    asm("and.b64 %0, %0, 0x7fffffffffffffff;" : "+l"(b));
    return b;
}
template<class VT> __device__ __forceinline__ VT max_of(unsigned long long b) {
    if constexpr(sizeof(VT) == 4) return __uint_as_float((unsigned)b);
    else return __longlong_as_double((long long)(b & 0x7fffffffffffffffull));
}
// 16-byte accesses are single (PTX .b128), so a packet is never seen half written
__device__ __forceinline__ void st_relaxed_packet(PcgPacket* p, PcgPacket v) {
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
                 : : "l"(p), "l"(v.sum), "l"(v.max) : "memory");
}
__device__ __forceinline__ PcgPacket ld_relaxed_packet(const PcgPacket* p) {
    PcgPacket v;
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(v.sum), "=l"(v.max) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_packet(PcgPacket* p, PcgPacket v) {
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.release.gpu.global.b128 [%0], t; }"
                 : : "l"(p), "l"(v.sum), "l"(v.max) : "memory");
}
__device__ __forceinline__ PcgPacket ld_acquire_packet(const PcgPacket* p) {
    PcgPacket v;
    asm volatile("{ .reg .b128 t; ld.acquire.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(v.sum), "=l"(v.max) : "l"(p) : "memory");
    return v;
}
// The word behind a packet: its chunk's pairs of an exchange of this parity are visible
__device__ __forceinline__ void st_ready(PcgPacket* slot, unsigned parity) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" : : "l"(slot + 1), "r"(parity) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_ready(const PcgPacket* slot) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(slot + 1) : "memory");
    return v;
}

struct Yes { static constexpr bool value = true; };
struct No { static constexpr bool value = false; };

// Barrier over one group of 256 threads (hardware barriers 1 .. G; 0 is the whole block's)
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 256;" : : "r"(g + 1) : "memory"); }

// One warp: sum and max (MAX) of 256 lanes' values in the canonical order (as
// block_sum_max_256); valid in lane 0
template<class VT, bool MAX>
__device__ __forceinline__ void lane_tree(const double* smd, const VT* smv, double& sum, VT& mx) {
    const int t = threadIdx.x & 31;
    const double a0 = smd[t] + smd[t + 128];
    const double a1 = smd[t + 64] + smd[t + 192];
    const double a2 = smd[t + 32] + smd[t + 160];
    const double a3 = smd[t + 96] + smd[t + 224];
    double c = (a0 + a1) + (a2 + a3);
    VT x = VT(0);
    if(MAX) {
        x = smv[t];
#pragma unroll
        for(int q = 1; q < 8; ++q) { const VT o = smv[t + 32 * q]; x = x > o ? x : o; }
    }
#pragma unroll
    for(int off = 16; off > 0; off >>= 1) {
        c = c + __shfl_down_sync(0xffffffffu, c, off);
        if(MAX) { const VT o = __shfl_down_sync(0xffffffffu, x, off); x = x > o ? x : o; }
    }
    sum = c;
    mx = x;
}

// One warp: a chunk's sum and max from its 256 lanes' values out to its packet.  RELEASE:
// everything the group wrote before its last barrier is visible to whoever acquires the packet.
template<class VT, bool MAX, bool RELEASE>
__device__ __forceinline__ void packet_publish(const double* smd, const VT* smv, PcgPacket* slot, unsigned parity) {
    double c;
    VT x;
    lane_tree<VT, MAX>(smd, smv, c, x);
    if((threadIdx.x & 31) == 0) {
        PcgPacket v;
        v.sum = (unsigned long long)__double_as_longlong(c);
        v.max = max_bits(x) | ((unsigned long long)parity << 63);
        if(RELEASE) st_release_packet(slot, v);
        else st_relaxed_packet(slot, v);
    }
}

// Tries until `got` is true in every lane of the warp; false when the bounded wait gave up
template<class F> __device__ __forceinline__ bool warp_poll(F got, BarrierLimit lim) {
    unsigned spins = 0;
    unsigned long long t0 = 0;
    while(true) {
        if(__all_sync(0xffffffffu, got())) return true;
        ++spins;
        if(spins == lim.minSpins) t0 = global_ns();
        const bool late = spins >= lim.maxSpins ||
                          (spins > lim.minSpins && (spins & 255u) == 0u && global_ns() - t0 >= lim.ns);
        if(__any_sync(0xffffffffu, late)) return false;
    }
}
// One packet per lane (where `on`), until all carry `parity`
template<bool ACQUIRE>
__device__ __forceinline__ bool packet_poll(const PcgPacket* slot, bool on, unsigned parity, PcgPacket& pk, BarrierLimit lim) {
    return warp_poll([&] {
        if(on) {
            pk = ACQUIRE ? ld_acquire_packet(slot) : ld_relaxed_packet(slot);
            on = (unsigned)(pk.max >> 63) != parity;
        }
        return !on;
    }, lim);
}

// One warp: the packets of up to 32 chunks, their canonical sum and max (valid in lane 0);
// false when the wait gave up
template<class VT, bool MAX, bool ACQUIRE>
__device__ __forceinline__ bool warp_packets(const PcgPacket* slots, int nch, unsigned parity, double& sum, VT& mx,
                                             BarrierLimit lim) {
    const int t = threadIdx.x & 31;
    PcgPacket pk;
    const bool ok = packet_poll<ACQUIRE>(slots + (size_t)t * kPacketStride, t < nch, parity, pk, lim);
    double c = 0.0;
    VT m = VT(0);
    if(t < nch) {
        c = c + __longlong_as_double((long long)pk.sum);
        if(MAX) { const VT o = max_of<VT>(pk.max); m = m > o ? m : o; }
    }
#pragma unroll
    for(int off = 16; off > 0; off >>= 1) {
        if(off >= nch) continue;  // the tree's other half holds no chunk: +0
        c = c + __shfl_down_sync(0xffffffffu, c, off);
        if(MAX) { const VT o = __shfl_down_sync(0xffffffffu, m, off); m = m > o ? m : o; }
    }
    sum = c;
    mx = m;
    return ok;
}

// Second half of an exchange: waits for every chunk's packet of this parity and gives the
// canonical sum and max (as reduce_partials_bcast) to every thread of the block: all
// threads poll, the sums go through the W's arrays.  ACQUIRE: what the other blocks released is
// visible.  False when the bounded wait gave up (the timeout flag is set).
constexpr int kMostSM = 160;  // SMs a chunk-resident solve is spread over at most
template<class VT, int CH> struct WaitSmem {
    double part[CH * kMostSM];  // the chunks' sums and maxima as polled
    VT partMax[CH * kMostSM];
    double lanes[kLanes];       // ... of the 256 lanes of the canonical tree
    VT lanesMax[kLanes];
    // The result, and whether the wait gave up: a slot for each of an iteration's two exchanges
    // (MAX: the second).  A group without a chunk publishes nothing, so no packet says that its
    // warps have read a wait's result before the next wait writes its own; a slot is written again
    // only after the other exchange's closing barrier, which every reader has reached by then.
    double sum[2];
    VT max[2];
    int bad[2];
};
template<class VT, bool MAX, bool ACQUIRE, int CH>
__device__ __forceinline__ bool packet_wait(const PcgPacket* slots, int nch, unsigned parity, unsigned* flags,
                                            WaitSmem<VT, CH>& W, double& sum, VT& mx,
                                            BarrierLimit lim = solve_barrier_limit()) {
    constexpr int X = MAX ? 1 : 0;
    const int t = threadIdx.x;
    // whole warps stay in the loop (the poll votes)
    for(int c = t; c < ((nch + 31) & ~31); c += (int)blockDim.x) {
        PcgPacket pk;
        if(!packet_poll<ACQUIRE>(slots + (size_t)c * kPacketStride, c < nch, parity, pk, lim)) { W.bad[X] = 1; break; }
        if(c < nch) {
            W.part[c] = __longlong_as_double((long long)pk.sum);
            if(MAX) W.partMax[c] = max_of<VT>(pk.max);
        }
    }
    __syncthreads();
    if(t < kLanes) {
        double acc = 0.0;
        VT m = VT(0);
        for(int c = t; c < nch; c += kLanes) {
            acc = acc + W.part[c];
            if(MAX) { const VT o = W.partMax[c]; m = m > o ? m : o; }
        }
        W.lanes[t] = acc;
        if(MAX) W.lanesMax[t] = m;
        group_sync(0);
    }
    if(t < 32) {
        double c;
        VT x;
        lane_tree<VT, MAX>(W.lanes, W.lanesMax, c, x);
        if(t == 0) { W.sum[X] = c; W.max[X] = x; }
    }
    __syncthreads();
    sum = W.sum[X];
    mx = W.max[X];
    if(W.bad[X] == 0) return true;
    if(t == 0) atomicOr(flags, BNN_FLAG_TIMEOUT);
    return false;
}

// packet_wait where the sums come ahead of the pairs (kSplit): the first 256 threads poll the
// packets, chunk c the lane c mod 256 of the canonical tree; with PAIRS the warps that have no
// packets wait for the words that say the pairs are visible.  kPer: packets of a lane.
__device__ __forceinline__ void front_sync(int threads) { asm volatile("bar.sync 15, %0;" : : "r"(threads) : "memory"); }
template<class VT, bool MAX, bool PAIRS, int kPer, int CH>
__device__ __forceinline__ bool packet_wait_split(const PcgPacket* slots, int nch, unsigned parity, unsigned* flags,
                                                  WaitSmem<VT, CH>& W, double& sum, VT& mx,
                                                  BarrierLimit lim = solve_barrier_limit()) {
    constexpr int X = MAX ? 1 : 0;
    const int t = threadIdx.x, front = min((nch + 31) & ~31, kLanes);
    if(t < front) {
        PcgPacket pk[kPer];
        unsigned late = (1u << kPer) - 1u;
#pragma unroll
        for(int i = 0; i < kPer; ++i)
            if(t + i * kLanes >= nch) late &= ~(1u << i);
        if(!warp_poll([&] {
#pragma unroll
               for(int i = 0; i < kPer; ++i)
                   if(late >> i & 1u) pk[i] = ld_relaxed_packet(slots + (size_t)(t + i * kLanes) * kPacketStride);
#pragma unroll
               for(int i = 0; i < kPer; ++i)
                   if((late >> i & 1u) && (unsigned)(pk[i].max >> 63) == parity) late &= ~(1u << i);
               return late == 0u;
           }, lim)) W.bad[X] = 1;
        double c = 0.0;
        VT m = VT(0);
#pragma unroll
        for(int i = 0; i < kPer; ++i)
            if(t + i * kLanes < nch) {
                c = c + __longlong_as_double((long long)pk[i].sum);
                if(MAX) { const VT o = max_of<VT>(pk[i].max); m = m > o ? m : o; }
            }
        W.lanes[t] = c;
        if(MAX) W.lanesMax[t] = m;
        front_sync(front);  // past it the lanes are 0
        if(t < 32) {
            lane_tree<VT, MAX>(W.lanes, W.lanesMax, c, m);
            if(t == 0) { W.sum[X] = c; W.max[X] = m; }
        }
    } else if constexpr(PAIRS) {
        for(int c = t - front; c < ((nch + 31) & ~31); c += (int)blockDim.x - front) {
            bool on = c < nch;
            if(!warp_poll([&] {
                   if(on) on = ld_acquire_ready(slots + (size_t)c * kPacketStride) != parity;
                   return !on;
               }, lim)) { W.bad[X] = 1; break; }
        }
    }
    __syncthreads();
    sum = W.sum[X];
    mx = W.max[X];
    if(W.bad[X] == 0) return true;
    if(t == 0) atomicOr(flags, BNN_FLAG_TIMEOUT);
    return false;
}

// packet_wait for one group on its own (a scene of a batch): the group polls its scene's
// packets, and no other group waits for it.  Up to 32 chunks are polled by its first warp, which
// then needs no shared memory for their sum.
constexpr int kWarpPackets = 32;
template<class VT> struct GroupWaitSmem {
    double lanes[kLanes];
    VT lanesMax[kLanes];
    double sum;
    VT max;
    int bad;
};
template<class VT, bool MAX, bool ACQUIRE>
__device__ __forceinline__ bool group_wait(const PcgPacket* slots, int nch, unsigned parity, unsigned* flags,
                                           GroupWaitSmem<VT>& W, int grp, int t, double& sum, VT& mx,
                                           BarrierLimit lim = solve_barrier_limit()) {
    if(nch > kWarpPackets) {
        double acc = 0.0;
        VT m = VT(0);
        for(int c = t; c < ((nch + 31) & ~31); c += kLanes) {
            PcgPacket pk;
            if(!packet_poll<ACQUIRE>(slots + (size_t)c * kPacketStride, c < nch, parity, pk, lim)) { W.bad = 1; break; }
            if(c < nch) {
                acc = acc + __longlong_as_double((long long)pk.sum);
                if(MAX) { const VT o = max_of<VT>(pk.max); m = m > o ? m : o; }
            }
        }
        W.lanes[t] = acc;
        if(MAX) W.lanesMax[t] = m;
        group_sync(grp);
        if(t < 32) {
            double c;
            VT x;
            lane_tree<VT, MAX>(W.lanes, W.lanesMax, c, x);
            if(t == 0) { W.sum = c; W.max = x; }
        }
    } else if(t < 32) {
        double c;
        VT m;
        if(!warp_packets<VT, MAX, ACQUIRE>(slots, nch, parity, c, m, lim)) W.bad = 1;
        if(t == 0) { W.sum = c; W.max = m; }
    }
    group_sync(grp);
    sum = W.sum;
    mx = W.max;
    if(W.bad == 0) return true;
    if(t == 0) atomicOr(flags, BNN_FLAG_TIMEOUT);
    return false;
}

template<class VT> struct ChunkArgs {
    int n;
    int nch;
    const float* rhsF;
    const float* diag;
    const VT* invd;
    const int32_t* nbr;
    const float* coef;  // off-diagonal planes (COEF)
    VT negoff;
    VT tolFactor;
    unsigned maxIter;
    VT* x;
    RowPair<VT>* pair;  // two buffers of pairStride rows
    int pairStride;
    PcgPacket *pkA, *pkB;  // nch packets each, zeroed
    DevState* st;
};
// A row's neighbours in 8 bytes: .x = dz- | y- << 18 | (has -x) << 31, .y = dz+ | y+ << 18 |
// (has +x) << 31.  dz is a row distance (0 = none); y is the neighbour's place in the chunk,
// kNoRow for none, kNoRow + 1 + its distance when it lies in another chunk.  Grids of up to
// kCompactDy cells along x and kCompactDz cells per z plane fit (kRowsCompact).  With y
// neighbours within two of the chunk's eight 256-row strips, only its first and last two
// strips reach across its ends.
constexpr unsigned kNoRow = kChunk;
static_assert(kCompactDy <= 2 * kLanes && kNoRow + 1 + kCompactDy < (1 << 12) && kCompactDz < (1 << 18),
              "the records' fields");
__device__ __forceinline__ unsigned row_code(int dz, int l, int dy, int sign, bool x) {
    const int to = l + sign * dy;
    const unsigned y = dy == 0 ? kNoRow : ((unsigned)to < (unsigned)kChunk ? (unsigned)to : kNoRow + 1u + (unsigned)dy);
    return (unsigned)dz | y << 18 | (x ? 0x80000000u : 0u);
}
// Shared memory of a block: CH chunks.  x and 1/diag are kept there too where they fit (else
// x stays in global memory and 1/diag is loaded ahead of every iteration's first exchange).
template<class VT> constexpr int kRoomy = sizeof(VT) == 4 ? 3 : 2;
template<class VT, bool COEF, int CH, bool HERE = (CH <= kRoomy<VT>)> struct ChunkRowsSmem {
    static constexpr bool kHere = HERE;
    static constexpr int kX = HERE ? CH : 1, kXRows = HERE ? kChunk : 1;
    VT s[CH][kChunk + 16 / sizeof(VT)];  // s[kNoRow] = 0: what a missing neighbour adds
    uint2 nb[CH][kChunk];
    float diag[CH][kChunk];
    VT inv[kX][kXRows], x[kX][kXRows];
    float co[COEF ? CH : 1][COEF ? 6 : 1][COEF ? kChunk : 1];
    double sum[CH][kLanes];
    VT max[CH][kLanes];
};
template<class VT, bool COEF, int G, int K> struct ChunkSmem : ChunkRowsSmem<VT, COEF, G * K> {
    WaitSmem<VT, G * K> wait;
};
// A cluster's block: the pairs live in shared memory, and every block holds all packets
constexpr int kMostCluster = 16;
template<class VT, bool COEF> struct ClusterSmem : ChunkRowsSmem<VT, COEF, 1, true> {
    RowPair<VT> pair[kChunk];
    PcgPacket packets[2][kMostCluster];
};
// A batch's block: every group solves for a scene of its own
template<class VT, int G, int K> struct BatchChunkSmem : ChunkRowsSmem<VT, false, G * K> {
    GroupWaitSmem<VT> wait[G];
    ChunkArgs<VT> args[G];
};

// Who waits for whom in chunk_solve.  kGrid: all groups of the launch belong to one system, a
// block waits as a whole.  kScene: a group is one of a scene's groups, and waits and returns by
// itself.  kCluster: the launch is one thread-block cluster and holds one system; pairs and
// packets are exchanged through distributed shared memory, and the waits are cluster barriers.
enum ChunkMode { kGrid, kScene, kCluster };

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_to_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" : : : "memory");
}
// ld_pair_if from another block's (or the own) shared memory
template<class VT> __device__ __forceinline__ RowPair<VT> ld_cluster_pair_if(unsigned addr, bool on) {
    RowPair<VT> v{VT(0), VT(0)};
    if constexpr(sizeof(VT) == 4)
        asm volatile("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p ld.shared::cluster.v2.f32 {%0, %1}, [%2]; }"
                     : "+f"(v.z), "+f"(v.s) : "r"(addr), "r"((int)on) : "memory");
    else
        asm volatile("{ .reg .pred p; setp.ne.s32 p, %3, 0; @p ld.shared::cluster.v2.f64 {%0, %1}, [%2]; }"
                     : "+d"(v.z), "+d"(v.s) : "r"(addr), "r"((int)on) : "memory");
    return v;
}

// One warp: a chunk's packet to every block of the cluster
template<class VT, bool MAX>
__device__ __forceinline__ void cluster_publish(const double* smd, const VT* smv, PcgPacket* slot, unsigned blocks) {
    double c;
    VT x;
    lane_tree<VT, MAX>(smd, smv, c, x);
    c = __shfl_sync(0xffffffffu, c, 0);
    if(MAX) x = __shfl_sync(0xffffffffu, x, 0);
    const unsigned lane = threadIdx.x & 31;
    if(lane < blocks) {
        const unsigned to = map_to_rank(smem_addr(slot), lane);
        asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" : : "r"(to), "l"(__double_as_longlong(c)),
                     "l"((long long)max_bits(x)) : "memory");
    }
}
// After the cluster's barrier every warp forms the sum and max of its block's copy of the
// packets (canonical tree; the part of it past 16 chunks is 0)
template<class VT, bool MAX>
__device__ __forceinline__ void cluster_sum(const PcgPacket* packets, int nch, double& sum, VT& mx) {
    const int t = threadIdx.x & 31;
    double c = 0.0;
    VT m = VT(0);
    if(t < nch) {
        c = c + __longlong_as_double((long long)packets[t].sum);
        if(MAX) { const VT o = max_of<VT>(packets[t].max); m = m > o ? m : o; }
    }
#pragma unroll
    for(int off = kMostCluster / 2; off > 0; off >>= 1) {
        c = c + __shfl_down_sync(0xffffffffu, c, off);
        if(MAX) { const VT o = __shfl_down_sync(0xffffffffu, m, off); m = m > o ? m : o; }
    }
    sum = __shfl_sync(0xffffffffu, c, 0);
    mx = MAX ? __shfl_sync(0xffffffffu, m, 0) : m;
}

// The solve of the K chunks c0, c0 + cStep, ... by group grp of a block of G groups (kCluster:
// one chunk a block, cStep blocks).
template<class VT, bool COEF, int G, int K, ChunkMode MODE, class Smem>
__device__ __forceinline__ void chunk_solve(const ChunkArgs<VT>& a, Smem& S, const int grp, const int t, const int c0,
                                            const int cStep) {
    // rows whose neighbour loads are in flight together
    constexpr int kGroup = sizeof(VT) == 4 ? (G == 1 ? 8 : 4) : (G == 1 ? 4 : 2);
    constexpr int R = K * kPerLane;
    constexpr bool kHere = Smem::kHere;  // x and 1/diag in shared memory
    const int n = a.n, nch = a.nch;
    unsigned* flags = &a.st->flags;
    RowPair<VT>* __restrict__ pair = a.pair;
    int buf = 0;  // where the buffer of the last second exchange starts
    const VT negoff = a.negoff;
    auto chunk_of = [&](int k) { return c0 + k * cStep; };
    auto rows_of = [&](int k) { return max(min(n - chunk_of(k) * kChunk, kChunk), 0); };
    // the pair of another row of the system, and of an own one
    auto other_pair = [&](int row, bool on) {
        if constexpr(MODE == kCluster) {
            const unsigned block = (unsigned)row / kChunk % kMostCluster, l = (unsigned)row % kChunk;
            return ld_cluster_pair_if<VT>(map_to_rank(smem_addr(S.pair) + l * (unsigned)sizeof(RowPair<VT>), on ? block : 0u), on);
        } else return ld_pair_if(pair + (row + buf), on);
    };
    auto own_pair = [&](int k, int l) -> RowPair<VT>& {
        if constexpr(MODE == kCluster) return S.pair[l];
        else return pair[chunk_of(k) * kChunk + l + buf];
    };
    // Split: an iteration's second exchange passes sums and pairs.  The sums go out at once, and
    // another warp waits for the pairs to reach L2 and says so in a word of its own: both ways
    // are taken at the same time, where a released packet takes them in turn.  Measured, us per
    // iteration with everything around it (without): FP32 79 chunks 5.0 (5.45), 226 6.8 (7.36),
    // 345 8.3 (8.8); FP64 79 5.86 (6.45), 226 8.2 (8.9).  With two chunks per group the longer
    // wait costs registers that spill (627 chunks 18.0 against 15.4): those release the packets.
    // A scene of a batch shares its SM with others that fill the wait (no difference).
    constexpr bool kSplit = MODE == kGrid && K == 1;
    auto wait = [&](auto withMax, auto acquire, const PcgPacket* slots, unsigned parity, double& sum, VT& mx) {
        constexpr bool MAX = decltype(withMax)::value;
        [[maybe_unused]] constexpr bool ACQUIRE = decltype(acquire)::value;
        if constexpr(MODE == kCluster) {
            cluster_barrier();
            cluster_sum<VT, MAX>(S.packets[MAX ? 1 : 0], nch, sum, mx);
            return true;
        } else if constexpr(MODE == kScene)
            return group_wait<VT, MAX, ACQUIRE>(slots, nch, parity, flags, S.wait[grp], grp, t, sum, mx);
        else {
            if constexpr(kSplit) {
                static_assert(G * kMostSM <= 2 * kLanes, "packets of a lane");
                if(G == 1 || (G == 2 && nch <= kLanes))
                    return packet_wait_split<VT, MAX, ACQUIRE, 1>(slots, nch, parity, flags, S.wait, sum, mx);
                return packet_wait_split<VT, MAX, ACQUIRE, 2>(slots, nch, parity, flags, S.wait, sum, mx);
            } else return packet_wait<VT, MAX, ACQUIRE, G * K>(slots, nch, parity, flags, S.wait, sum, mx);
        }
    };

    // ---- init: r = rhs, x = 0, z = D^-1 r; partial z.r and max|r| (PCGSolver.cpp:151-168)
    if constexpr(MODE == kScene) {
        if(t == 0) S.wait[grp].bad = 0;
    } else if constexpr(MODE == kGrid) {
        if(threadIdx.x == 0) S.wait.bad[0] = S.wait.bad[1] = 0;
        if(threadIdx.x < kLanes) {  // the lanes that no chunk fills
            S.wait.lanes[threadIdx.x] = 0.0;
            S.wait.lanesMax[threadIdx.x] = VT(0);
        }
    }
    VT r[R], q[R];  // q holds z from phase B to the next phase A
#pragma unroll
    for(int k = 0; k < K; ++k) {
        const int slot = grp * K + k, base = chunk_of(k) * kChunk, rows = rows_of(k);
        double acc = 0.0;
        VT m = VT(0);
#pragma unroll
        for(int j = 0; j < kPerLane; ++j) {
            const int l = t + j * kLanes;
            uint2 nbv = make_uint2(kNoRow << 18, kNoRow << 18);
            float dg = 0.f;
            VT rv = VT(0), zv = VT(0), iv = VT(0);
            asm volatile("" : : : "memory");  // a row's loads at a time: registers
            if(l < rows) {
                const int e = base + l;
                int32_t nb[6];
#pragma unroll
                for(int p = 0; p < 6; ++p) nb[p] = __ldg(a.nbr + (size_t)p * n + e);
                nbv.x = row_code(nb[0] >= 0 ? e - nb[0] : 0, l, nb[1] >= 0 ? e - nb[1] : 0, -1, nb[2] >= 0);
                nbv.y = row_code(nb[5] >= 0 ? nb[5] - e : 0, l, nb[4] >= 0 ? nb[4] - e : 0, 1, nb[3] >= 0);
                dg = __ldg(a.diag + e);
                if constexpr(COEF)
#pragma unroll
                    for(int p = 0; p < 6; ++p) S.co[slot][p][l] = __ldg(a.coef + (size_t)p * n + e);
                rv = (VT)__ldg(a.rhsF + e);
                const VT ab = vabs(rv);
                m = m > ab ? m : ab;
                iv = __ldg(a.invd + e);
                zv = iv * rv;
                own_pair(k, l) = {zv, VT(0)};
                acc = acc + (double)zv * (double)rv;
            }
            if constexpr(kHere) {
                S.inv[slot][l] = iv;
                S.x[slot][l] = VT(0);
            } else if(rows > 0) a.x[base + l] = VT(0);
            S.nb[slot][l] = nbv;
            S.diag[slot][l] = dg;
            S.s[slot][l] = VT(0);
            r[k * kPerLane + j] = rv;
            q[k * kPerLane + j] = zv;
        }
        if(t == 0) S.s[slot][kNoRow] = VT(0);
        if constexpr(COEF) if(rows < kChunk)
            for(int l = rows + t; l < kChunk; l += kLanes)
#pragma unroll
                for(int p = 0; p < 6; ++p) S.co[slot][p][l] = 0.f;
        S.sum[slot][t] = acc;
        S.max[slot][t] = m;
    }
    if constexpr(MODE == kScene) group_sync(grp);
    else __syncthreads();
    double rho;
    VT resid;
    unsigned parity = 1;  // of this iteration's exchanges
    auto publish = [&](auto withMax, auto release, PcgPacket* slots) {
        // a warp of the group for each of its chunks, and one for their pairs (split)
        constexpr bool MAX = decltype(withMax)::value, RELEASE = decltype(release)::value;
        if(t < 32 * K) {
            const int k = t >> 5, slot = grp * K + k, c = chunk_of(k);
            if(c >= nch) return;
            [[maybe_unused]] PcgPacket* to = slots + (size_t)c * kPacketStride;
            if constexpr(MODE == kCluster)
                cluster_publish<VT, MAX>(S.sum[slot], S.max[slot], &S.packets[MAX ? 1 : 0][c], (unsigned)cStep);
            else packet_publish<VT, MAX, RELEASE && !kSplit>(S.sum[slot], S.max[slot], to, parity);
        } else if(kSplit && RELEASE && t == 32 * K) {
            __threadfence();
#pragma unroll
            for(int k = 0; k < K; ++k)
                if(chunk_of(k) < nch) st_ready(slots + (size_t)chunk_of(k) * kPacketStride, parity);
        }
    };
    publish(Yes(), Yes(), a.pkB);
    if(!wait(Yes(), Yes(), a.pkB, parity, rho, resid)) return;
    const VT tolFactor = fmax(a.tolFactor, VT(1e-30));
    unsigned iter = 0, success = 0;
    bool done = false;
    VT tol = VT(0);
    if(resid < (VT)FLT_MIN) {
        done = true;
        success = 1;
    } else {
        tol = tolFactor * resid;
        if(rho < (double)FLT_MIN || isnan(rho)) done = true;
    }
    if(a.maxIter == 0) done = true;

    // beta and every s are 0 in the first iteration, where s = z: z + 0 * 0 differs from z in
    // the sign of a zero at most, which no sum or product keeps
    VT beta = VT(0);
    while(!done) {
        // ---- phase A: s = z + beta s_old, q = A s, partial s.q (PCGSolver.cpp:173-174,192-193)
        RowPair<VT> zn[kGroup][2], ye[kGroup];
        uint2 nb[kGroup];
        // what rows g0 .. of chunk k read from the pairs: their z neighbours, and the y
        // neighbours across the chunk's ends
        auto load_pairs = [&](int k, int g0) {
            const int base = chunk_of(k) * kChunk;
#pragma unroll
            for(int u = 0; u < kGroup; ++u) {
                const int j = g0 + u, l = t + j * kLanes;
                nb[u] = S.nb[grp * K + k][l];
                const int dM = (int)(nb[u].x & 0x3ffffu), dP = (int)(nb[u].y & 0x3ffffu);
                zn[u][0] = other_pair(base + l - dM, dM != 0);
                zn[u][1] = other_pair(base + l + dP, dP != 0);
                if(j < 2) {
                    const unsigned y = nb[u].x >> 18 & 0xfffu;
                    ye[u] = other_pair(base + l - (int)(y - kNoRow - 1u), y > kNoRow);
                }
                if(j >= kPerLane - 2) {
                    const unsigned y = nb[u].y >> 18 & 0xfffu;
                    ye[u] = other_pair(base + l + (int)(y - kNoRow - 1u), y > kNoRow);
                }
            }
        };
        // the x neighbours across the chunk's ends: of its first and its last row
        RowPair<VT> xe[K];
#pragma unroll
        for(int k = 0; k < K; ++k) {
            const uint2 e = S.nb[grp * K + k][t == 0 ? 0 : kChunk - 1];
            xe[k] = other_pair(t == 0 ? chunk_of(k) * kChunk - 1 : (chunk_of(k) + 1) * kChunk,
                               (t == 0 && (int)e.x < 0) || (t == kLanes - 1 && (int)e.y < 0));
        }
        load_pairs(0, 0);
#pragma unroll
        for(int k = 0; k < K; ++k)
#pragma unroll
            for(int j = 0; j < kPerLane; ++j) {
                VT* ps = &S.s[grp * K + k][t + j * kLanes];
                *ps = q[k * kPerLane + j] + beta * *ps;
            }
        group_sync(grp);
        auto s_of = [&](const RowPair<VT>& p) { return p.z + beta * p.s; };
#pragma unroll
        for(int k = 0; k < K; ++k) {
            const int slot = grp * K + k;
            const VT* __restrict__ sS = S.s[slot];
            double acc = 0.0;
#pragma unroll
            for(int g0 = 0; g0 < kPerLane; g0 += kGroup) {
                if(k + g0 > 0) load_pairs(k, g0);
#pragma unroll
                for(int u = 0; u < kGroup; ++u) {
                    const int j = g0 + u, l = t + j * kLanes;
                    const unsigned yM = nb[u].x >> 18 & 0xfffu, yP = nb[u].y >> 18 & 0xfffu;
                    // a missing neighbour's value is 0: its term -0 (or 0) changes no sum
                    VT vyM = sS[j < 2 ? min(yM, kNoRow) : yM], vyP = sS[j >= kPerLane - 2 ? min(yP, kNoRow) : yP];
                    if(j < 2) vyM = yM > kNoRow ? s_of(ye[u]) : vyM;
                    if(j >= kPerLane - 2) vyP = yP > kNoRow ? s_of(ye[u]) : vyP;
                    VT vxM = sS[j == 0 ? max(l - 1, 0) : l - 1], vxP = sS[l + 1];
                    if(j == 0) vxM = t == 0 ? s_of(xe[k]) : vxM;
                    if(j == kPerLane - 1) vxP = t == kLanes - 1 ? s_of(xe[k]) : vxP;
                    vxM = (int)nb[u].x < 0 ? vxM : VT(0);
                    vxP = (int)nb[u].y < 0 ? vxP : VT(0);
                    auto cf = [&](int p) { return COEF ? (VT)S.co[slot][p][l] : negoff; };
                    const VT sv = sS[l];
                    VT tq = VT(0) + cf(0) * s_of(zn[u][0]);
                    tq = tq + cf(1) * vyM;
                    tq = tq + cf(2) * vxM;
                    tq = tq + (VT)S.diag[slot][l] * sv;
                    tq = tq + cf(3) * vxP;
                    tq = tq + cf(4) * vyP;
                    tq = tq + cf(5) * s_of(zn[u][1]);
                    q[k * kPerLane + j] = tq;
                    acc = acc + (double)sv * (double)tq;
                }
            }
            S.sum[slot][t] = acc;
        }
        group_sync(grp);
        // relaxed: phase A writes nothing that other blocks read, and the pairs it read are not
        // written again before the exchange after this one's second
        publish(No(), No(), a.pkA);
        VT inv[kHere ? 1 : R];
        if constexpr(!kHere)
#pragma unroll
            for(int k = 0; k < K; ++k)
#pragma unroll
                for(int j = 0; j < kPerLane; ++j) {
                    const int l = t + j * kLanes;
                    inv[k * kPerLane + j] = ld_const_if(a.invd + (size_t)chunk_of(k) * kChunk + l, l < rows_of(k));
                }
        double tmp;
        VT unused;
        if(!wait(No(), No(), a.pkA, parity, tmp, unused)) return;
        if(tmp < (double)FLT_MIN) {
            ++iter;
            success = 1;
            break;
        }
        const VT alpha = (VT)(rho / tmp);
        parity ^= 1u;
        if constexpr(MODE != kCluster) buf = a.pairStride - buf;
        // ---- phase B: r -= alpha q, max|r|, z = D^-1 r, partial z.r; then x += alpha s
#pragma unroll
        for(int k = 0; k < K; ++k) {
            const int slot = grp * K + k;
            const bool live = chunk_of(k) < nch;
            double acc = 0.0;
            VT m = VT(0);
#pragma unroll
            for(int j = 0; j < kPerLane; ++j) {
                const int l = t + j * kLanes, i = k * kPerLane + j;
                const VT rv = r[i] + (-alpha) * q[i];
                r[i] = rv;
                const VT ab = vabs(rv);
                m = m > ab ? m : ab;
                VT iv;
                if constexpr(kHere) iv = S.inv[slot][l];
                else iv = inv[i];
                const VT zv = iv * rv;
                q[i] = zv;
                if(live) own_pair(k, l) = {zv, S.s[slot][l]};
                acc = acc + (double)zv * (double)rv;
            }
            S.sum[slot][t] = acc;
            S.max[slot][t] = m;
        }
        group_sync(grp);
        publish(Yes(), Yes(), a.pkB);
#pragma unroll
        for(int k = 0; k < K; ++k) {
            const int slot = grp * K + k;
            if constexpr(kHere) {
#pragma unroll
                for(int j = 0; j < kPerLane; ++j)
                    S.x[slot][t + j * kLanes] = S.x[slot][t + j * kLanes] + alpha * S.s[slot][t + j * kLanes];
            } else if(chunk_of(k) < nch) {
                VT* xp = a.x + (size_t)chunk_of(k) * kChunk + t;
                VT xv[kPerLane];
#pragma unroll
                for(int j = 0; j < kPerLane; ++j) xv[j] = __ldcg(xp + j * kLanes);
#pragma unroll
                for(int j = 0; j < kPerLane; ++j) xp[j * kLanes] = xv[j] + alpha * S.s[slot][t + j * kLanes];
            }
        }
        double rhoNew;
        if(!wait(Yes(), Yes(), a.pkB, parity, rhoNew, resid)) return;
        ++iter;
        if(resid < tol) {
            success = 1;
            break;
        }
        beta = (VT)(rhoNew / rho);
        rho = rhoNew;
        if(iter >= a.maxIter) {
            if(chunk_of(0) == 0 && t == 0) atomicOr(flags, BNN_FLAG_PCG_MAXITER);
            break;
        }
    }
    if constexpr(kHere)
#pragma unroll
        for(int k = 0; k < K; ++k)
#pragma unroll
            for(int j = 0; j < kPerLane; ++j) {
                const int l = t + j * kLanes;
                if(l < rows_of(k)) a.x[(size_t)chunk_of(k) * kChunk + l] = S.x[grp * K + k][l];
            }
    if(chunk_of(0) == 0 && t == 0) {
        a.st->iter = iter;
        a.st->success = success;
        a.st->done = 1;
        Sc<VT>::set_resid(a.st, resid);
    }
}

// A lone system: the chunks are striped over the grid's groups, so that the blocks' counts
// differ by one at most
template<class VT, bool COEF, int G, int K>
__global__ void __launch_bounds__(G * kLanes, 1) k_pcg_chunk(ChunkArgs<VT> a) {
    extern __shared__ __align__(16) unsigned char dynSm[];
    auto& S = *reinterpret_cast<ChunkSmem<VT, COEF, G, K>*>(dynSm);
    const int grp = (int)threadIdx.x / kLanes, t = (int)threadIdx.x % kLanes;
    chunk_solve<VT, COEF, G, K, kGrid>(a, S, grp, t, (int)(blockIdx.x + grp * K * gridDim.x), (int)gridDim.x);
}

// A system of up to 16 chunks in one cluster, a chunk per block: an exchange is a write to the
// other blocks' shared memory and a hardware barrier, a neighbour's pair a load from their
// shared memory, against a trip through L2 each.  us per iteration with everything around it
// (k_pcg_chunk): FP32 2,048 rows 3.5 (4.3), 26,652 rows 3.4 (4.9); FP64 26,652 rows 4.0 (5.9);
// the solve of a 64^3 scene 0.34 ms (0.48).  What is left is the chain of one iteration: two
// barriers with a reduction before each, two rounds of loads.  Two or three chunks per block,
// for up to 48, took longer than k_pcg_chunk on as many SMs as there are chunks (solve of a
// 121 x 77 x 95 scene 0.97 ms against 0.68).
template<class VT, bool COEF>
__global__ void __launch_bounds__(kLanes, 1) k_pcg_cluster(ChunkArgs<VT> a) {
    extern __shared__ __align__(16) unsigned char dynSm[];
    auto& S = *reinterpret_cast<ClusterSmem<VT, COEF>*>(dynSm);
    cluster_barrier();  // every block has started: its shared memory may be written
    chunk_solve<VT, COEF, 1, 1, kCluster>(a, S, 0, (int)threadIdx.x, (int)blockIdx.x, (int)gridDim.x);
    cluster_barrier();  // no block ends while another may still reach into it
}

// The FP32 systems of many scenes in one launch (BatchGroup: which chunks a group of 256
// threads owns).  A scene's groups exchange with one another alone, so a scene iterates at the
// pace of its own chunks and its groups end when it has converged; all groups of the launch
// are resident.  Every scene gets the scalars, iterates and iteration count of a lone solve.
struct BatchGroup {
    int scene;   // -1: no work
    int chunk0;  // its first chunk; the K of a group follow one another
};
template<int G, int K>
__global__ void __launch_bounds__(G * kLanes, 1) k_pcg_chunk_batch(const ChunkArgs<float>* __restrict__ scenes,
                                                                   const BatchGroup* __restrict__ groups) {
    extern __shared__ __align__(16) unsigned char dynSm[];
    auto& S = *reinterpret_cast<BatchChunkSmem<float, G, K>*>(dynSm);
    const int grp = (int)threadIdx.x / kLanes, t = (int)threadIdx.x % kLanes;
    const BatchGroup g = groups[blockIdx.x * G + grp];
    if(g.scene < 0) return;
    if(t == 0) S.args[grp] = scenes[g.scene];
    group_sync(grp);
    chunk_solve<float, false, G, K, kScene>(S.args[grp], S, grp, t, g.chunk0, 1);
}

// ---------------------------------------------------------------------------------
// Single-reduction PCG (Chronopoulos & Gear, 1989): the same Krylov iterates as
// PCGSolver::solve_precond (PCGSolver.cpp:143-199) in exact arithmetic, with both inner
// products of an iteration formed in one reduction, so one grid barrier per iteration
// instead of two.  With u = D^-1 r and w = A u:
//   gamma_i = (r_i, u_i), delta_i = (w_i, u_i)
//   beta_i  = gamma_i / gamma_{i-1},  alpha_i = gamma_i / (delta_i - beta_i gamma_i / alpha_{i-1})
//   p_i = u_i + beta_i p_{i-1},  s_i = w_i + beta_i s_{i-1}   (s_i = A p_i)
//   x_{i+1} = x_i + alpha_i p_i,  r_{i+1} = r_i - alpha_i s_i,  then u_{i+1}, w_{i+1}
// (the denominator is (p_i, A p_i); the first iteration takes beta = 0, alpha = gamma/delta).
// w_{i+1} = A u_{i+1} needs the neighbours' new u.  Instead of a second barrier, a row
// recomputes each neighbour's new u from the neighbour's old record {r, w, s, 1/diag}
// with the exact operations the neighbour uses for itself, so both agree bit for bit.  The
// records are double-buffered (read one, write the other), and so are the chunk partials
// (a block may start the next iteration while another still reads this one's partials).
// Per row and iteration: its own record, p and x, one record per y / z neighbour; the x
// neighbours' u come from the adjacent lanes by shuffles (packed rows).  Scalars are
// formed in FP64 from the canonical FP64 sums and rounded to the vector type.
// ---------------------------------------------------------------------------------
template<class VT> struct alignas(4 * sizeof(VT)) RowState {
    VT r, w, s, inv;
};
template<class VT> __device__ __forceinline__ RowState<VT> ld_state(const RowState<VT>* p) {
    RowState<VT> o;
    if constexpr(sizeof(VT) == 4) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
        o.r = v.x; o.w = v.y; o.s = v.z; o.inv = v.w;
    } else {
        const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
        const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
        o.r = a.x; o.w = a.y; o.s = b.x; o.inv = b.y;
    }
    return o;
}
template<class VT> __device__ __forceinline__ void st_state(RowState<VT>* p, VT r, VT w, VT s, VT inv) {
    if constexpr(sizeof(VT) == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(r, w, s, inv);
    } else {
        reinterpret_cast<double2*>(p)[0] = make_double2(r, w);
        reinterpret_cast<double2*>(p)[1] = make_double2(s, inv);
    }
}
// The new preconditioned residual of a row from its old record: the row's own update
// written out (s_i = w_i + beta s_{i-1}, r_{i+1} = r_i - alpha s_i, u_{i+1} = r_{i+1} / diag).
template<class VT> __device__ __forceinline__ VT u_next(const RowState<VT>& o, VT alpha, VT beta, bool first) {
    const VT s = first ? o.w : o.w + beta * o.s;
    const VT r = o.r + (-alpha) * s;
    return o.inv * r;
}

template<class VT> struct Cg1Args {
    int n;
    const float* rhsF;
    const float* diag;
    const VT* invd;
    const int32_t* nbr;
    const int4* rec;
    const float* coef;
    const float4* coefRow;
    VT negoff;
    VT tolFactor;
    unsigned maxIter;
    VT *x, *p;
    RowState<VT>* st[2];
    double* part;  // [set 0/1][gamma, delta][nchCap]
    double* pmax;  // [set 0/1][nchCap]
    int nchCap;
    DevState* dst;
    GridSync* gs;
};

// Two canonical 256-lane sums and a max in one block pass (association of
// block_sum_max_256); valid in thread 0.
__device__ __forceinline__ void block_sum2_max_256(double a, double b, double m, double* sa, double* sb, double* sm,
                                                   double& ra, double& rb, double& rm) {
    const int t = threadIdx.x;
    sa[t] = a; sb[t] = b; sm[t] = m;
    __syncthreads();
    if(t < 32) {
        double c[2];
#pragma unroll
        for(int k = 0; k < 2; ++k) {
            const double* sx = k == 0 ? sa : sb;
            const double a0 = sx[t] + sx[t + 128];
            const double a1 = sx[t + 64] + sx[t + 192];
            const double a2 = sx[t + 32] + sx[t + 160];
            const double a3 = sx[t + 96] + sx[t + 224];
            double v = (a0 + a1) + (a2 + a3);
#pragma unroll
            for(int off = 16; off > 0; off >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, off);
            c[k] = v;
        }
        double x = sm[t];
#pragma unroll
        for(int q = 1; q < 8; ++q) { const double o = sm[t + 32 * q]; x = x > o ? x : o; }
#pragma unroll
        for(int off = 16; off > 0; off >>= 1) { const double o = __shfl_down_sync(0xffffffffu, x, off); x = x > o ? x : o; }
        ra = c[0]; rb = c[1]; rm = x;
    }
    __syncthreads();
}

// The chunk partials of both sums (canonical order) and their max, to every thread.
__device__ __forceinline__ void reduce_partials2_bcast(const double* pa, const double* pb, const double* pm, int nch,
                                                       double* sa, double* sb, double* sm, double& ra, double& rb,
                                                       double& rm) {
    __shared__ double sRes[3];
    constexpr int U = 4;
    double acc0 = 0.0, acc1 = 0.0, m = 0.0;
    for(int c0 = threadIdx.x; c0 < nch; c0 += U * kLanes) {
        double x0[U], x1[U], xm[U];
#pragma unroll
        for(int u = 0; u < U; ++u) {
            const int c = c0 + u * kLanes;
            x0[u] = c < nch ? __ldcg(pa + c) : 0.0;
            x1[u] = c < nch ? __ldcg(pb + c) : 0.0;
            xm[u] = c < nch ? __ldcg(pm + c) : 0.0;
        }
#pragma unroll
        for(int u = 0; u < U; ++u)
            if(c0 + u * kLanes < nch) {
                acc0 = acc0 + x0[u];
                acc1 = acc1 + x1[u];
                m = m > xm[u] ? m : xm[u];
            }
    }
    double r0 = 0.0, r1 = 0.0, r2 = 0.0;
    block_sum2_max_256(acc0, acc1, m, sa, sb, sm, r0, r1, r2);
    if(threadIdx.x == 0) { sRes[0] = r0; sRes[1] = r1; sRes[2] = r2; }
    __syncthreads();
    ra = sRes[0]; rb = sRes[1]; rm = sRes[2];
    __syncthreads();
}

// Rows whose loads a lane keeps in flight together in the single-reduction kernel (each
// row holds seven 4-value records)
#ifndef BNN_CG1_ROW_GROUP
#define BNN_CG1_ROW_GROUP 1
#endif
#ifndef BNN_CG1_MIN_BLOCKS
#define BNN_CG1_MIN_BLOCKS 3
#endif
#ifndef BNN_CG1_MIN_BLOCKS_F64
#define BNN_CG1_MIN_BLOCKS_F64 2
#endif
template<class VT> constexpr int cg1_row_group() { return sizeof(VT) == 8 ? 1 : BNN_CG1_ROW_GROUP; }
template<class VT> constexpr int cg1_min_blocks() { return sizeof(VT) == 8 ? BNN_CG1_MIN_BLOCKS_F64 : BNN_CG1_MIN_BLOCKS; }

template<class VT, bool PACKED, bool COEF>
__global__ void __launch_bounds__(kLanes, cg1_min_blocks<VT>()) k_pcg_cg1(Cg1Args<VT> a) {
    constexpr int kRowGroup = cg1_row_group<VT>();
    __shared__ double sa[kLanes], sb[kLanes], smx[kLanes];
    const int n = a.n;
    const int nch = (n + kChunk - 1) / kChunk;
    const unsigned nb = gridDim.x;
    unsigned sense = 0;
    unsigned* flags = &a.dst->flags;
    const int lane = threadIdx.x & 31;
    const VT negoff = a.negoff;

    // neighbour rows of row ee in slot order (-z,-y,-x,self,+x,+y,+z); a missing one reads
    // the row itself (masked by has)
    auto neighbours = [&](size_t ee, const int4& rr, int32_t id[7], bool has[7], float& dg) {
        if constexpr(PACKED) {
            const int dyM = rr.x & 0xffff, dyP = (int)((unsigned)rr.x >> 16);
            const int dzM = rr.y & 0x7fffffff, dzP = rr.z & 0x7fffffff;
            const int32_t r0 = (int32_t)ee;
            has[0] = dzM != 0; id[0] = r0 - dzM;
            has[1] = dyM != 0; id[1] = r0 - dyM;
            has[2] = rr.y < 0; id[2] = (lane == 0 && rr.y < 0) ? r0 - 1 : r0;
            has[3] = true; id[3] = r0;
            has[4] = rr.z < 0; id[4] = (lane == 31 && rr.z < 0) ? r0 + 1 : r0;
            has[5] = dyP != 0; id[5] = r0 + dyP;
            has[6] = dzP != 0; id[6] = r0 + dzP;
            dg = __int_as_float(rr.w);
        } else {
#pragma unroll
            for(int q = 0; q < 6; ++q) {
                const int32_t v = __ldg(a.nbr + (size_t)q * n + ee);
                const int slot = q < 3 ? q : q + 1;
                has[slot] = v >= 0;
                id[slot] = v >= 0 ? v : (int32_t)ee;
            }
            id[3] = (int32_t)ee;
            has[3] = true;
            dg = __ldg(a.diag + ee);
        }
    };
    // (A v) of a row from its seven slot values, summed in slot order (FixedSparseMatrix::
    // multiply, SparseMatrix.cpp:222-235: column-sorted)
    auto apply_row = [&](size_t ee, const bool has[7], float dg, const VT v7[7]) {
        VT t = VT(0);
        if constexpr(COEF) {
            VT co[7];
            if constexpr(PACKED) {
                const float4 c0 = __ldg(a.coefRow + 2 * ee), c1 = __ldg(a.coefRow + 2 * ee + 1);
                co[0] = (VT)c0.x; co[1] = (VT)c0.y; co[2] = (VT)c0.z; co[3] = VT(0);
                co[4] = (VT)c0.w; co[5] = (VT)c1.x; co[6] = (VT)c1.y;
            } else {
#pragma unroll
                for(int q = 0; q < 7; ++q) co[q] = q == 3 ? VT(0) : (VT)__ldg(a.coef + (size_t)(q < 3 ? q : q - 1) * n + ee);
            }
#pragma unroll
            for(int q = 0; q < 3; ++q) if(has[q]) t += co[q] * v7[q];
            if(dg != 0.f) t += (VT)dg * v7[3];
#pragma unroll
            for(int q = 4; q < 7; ++q) if(has[q]) t += co[q] * v7[q];
        } else {
#pragma unroll
            for(int q = 0; q < 3; ++q) if(has[q]) t += negoff * v7[q];
            if(dg != 0.f) t += (VT)dg * v7[3];
#pragma unroll
            for(int q = 4; q < 7; ++q) if(has[q]) t += negoff * v7[q];
        }
        return t;
    };

    // ---- init: r = b, x = 0, u = D^-1 b, w = A u; gamma, delta, max|r| (set 0)
    for(int c = blockIdx.x; c < nch; c += nb) {
        const size_t base = (size_t)c * kChunk + threadIdx.x;
        double g = 0.0, d = 0.0, m = 0.0;
#pragma unroll 2
        for(int j = 0; j < kPerLane; ++j) {
            const size_t e = base + (size_t)j * kLanes;
            const size_t ee = e < (size_t)n ? e : 0;
            int32_t id[7];
            bool has[7];
            float dg;
            int4 rr = make_int4(0, 0, 0, 0);
            if constexpr(PACKED) rr = __ldg(a.rec + ee);
            neighbours(ee, rr, id, has, dg);
            VT u7[7];
#pragma unroll
            for(int q = 0; q < 7; ++q) {
                const bool load = !PACKED || (q != 2 && q != 4) || (q == 2 && lane == 0) || (q == 4 && lane == 31);
                u7[q] = load ? __ldg(a.invd + id[q]) * (VT)__ldg(a.rhsF + id[q]) : VT(0);
            }
            if constexpr(PACKED) {
                const VT up = __shfl_up_sync(0xffffffffu, u7[3], 1);
                const VT dn = __shfl_down_sync(0xffffffffu, u7[3], 1);
                if(lane != 0) u7[2] = up;
                if(lane != 31) u7[4] = dn;
            }
            const VT wv = apply_row(ee, has, dg, u7);
            if(e < (size_t)n) {
                const VT rv = (VT)a.rhsF[e];
                a.x[e] = VT(0);
                st_state(a.st[0] + e, rv, wv, VT(0), __ldg(a.invd + e));
                g = g + (double)u7[3] * (double)rv;
                d = d + (double)wv * (double)u7[3];
                const double ab = (double)vabs(rv);
                m = m > ab ? m : ab;
            }
        }
        double bg, bd, bm;
        block_sum2_max_256(g, d, m, sa, sb, smx, bg, bd, bm);
        if(threadIdx.x == 0) { a.part[c] = bg; a.part[(size_t)a.nchCap + c] = bd; a.pmax[c] = bm; }
    }
    if(!grid_barrier(a.gs, nb, sense, flags, solve_barrier_limit())) return;
    double gamma, delta, rmax;
    reduce_partials2_bcast(a.part, a.part + a.nchCap, a.pmax, nch, sa, sb, smx, gamma, delta, rmax);
    VT resid = (VT)rmax;
    const VT tolFactor = fmax(a.tolFactor, VT(1e-30));
    unsigned iter = 0, success = 0;
    bool done = false;
    VT tol = VT(0);
    if(resid < (VT)FLT_MIN) {
        done = true;
        success = 1;
    } else {
        tol = tolFactor * resid;
        if(gamma < (double)FLT_MIN || isnan(gamma)) done = true;
    }
    if(a.maxIter == 0) done = true;
    bool first = true;
    double gammaOld = 0.0, a64Old = 0.0;
    int cur = 0, set = 1;
    while(!done) {
        // alpha_i, beta_i; a denominator (p, A p) below FLT_MIN ends the solve as
        // PCGSolver's (p, s) check does (PCGSolver.cpp:173-176)
        double b64 = 0.0, den = delta;
        if(!first) {
            b64 = gamma / gammaOld;
            den = delta - (b64 * gamma) / a64Old;
        }
        if(den < (double)FLT_MIN) {
            ++iter;
            success = 1;
            break;
        }
        const double a64 = gamma / den;
        const VT alpha = (VT)a64, beta = (VT)b64;
        const RowState<VT>* __restrict__ sIn = a.st[cur];
        RowState<VT>* __restrict__ sOut = a.st[1 - cur];
        double* __restrict__ pg = a.part + (size_t)set * 2 * a.nchCap;
        double* __restrict__ pd = pg + a.nchCap;
        double* __restrict__ pm = a.pmax + (size_t)set * a.nchCap;
        for(int c = blockIdx.x; c < nch; c += nb) {
            const size_t base = (size_t)c * kChunk + threadIdx.x;
            int4 recAll[PACKED ? kPerLane : 1];
            if constexpr(PACKED) {
#pragma unroll
                for(int j = 0; j < kPerLane; ++j) {
                    const size_t e = base + (size_t)j * kLanes;
                    recAll[j] = __ldg(a.rec + (e < (size_t)n ? e : 0));
                }
            }
            double g = 0.0, d = 0.0, m = 0.0;
#pragma unroll
            for(int g0 = 0; g0 < kPerLane; g0 += kRowGroup) {
                int32_t id[kRowGroup][7];
                bool has[kRowGroup][7];
                float dg[kRowGroup];
                size_t rowE[kRowGroup];
#pragma unroll
                for(int u = 0; u < kRowGroup; ++u) {
                    const size_t e = base + (size_t)(g0 + u) * kLanes;
                    rowE[u] = e < (size_t)n ? e : 0;
                    neighbours(rowE[u], PACKED ? recAll[g0 + u] : make_int4(0, 0, 0, 0), id[u], has[u], dg[u]);
                }
                RowState<VT> S[kRowGroup][7];
                VT pOld[kRowGroup], xOld[kRowGroup];
#pragma unroll
                for(int u = 0; u < kRowGroup; ++u) {
#pragma unroll
                    for(int q = 0; q < 7; ++q) {
                        const bool load = !PACKED || (q != 2 && q != 4) || (q == 2 && lane == 0) || (q == 4 && lane == 31);
                        if(load) S[u][q] = ld_state(sIn + id[u][q]);
                        else S[u][q] = RowState<VT>{VT(0), VT(0), VT(0), VT(0)};
                    }
                    pOld[u] = first ? VT(0) : __ldcg(a.p + rowE[u]);
                    xOld[u] = __ldcg(a.x + rowE[u]);
                }
#pragma unroll
                for(int u = 0; u < kRowGroup; ++u) {
                    const RowState<VT>& o = S[u][3];
                    const VT uOld = o.inv * o.r;
                    const VT pNew = first ? uOld : uOld + beta * pOld[u];
                    const VT sNew = first ? o.w : o.w + beta * o.s;
                    const VT xNew = xOld[u] + alpha * pNew;
                    const VT rNew = o.r + (-alpha) * sNew;
                    VT u7[7];
#pragma unroll
                    for(int q = 0; q < 7; ++q) u7[q] = q == 3 ? o.inv * rNew : u_next(S[u][q], alpha, beta, first);
                    if constexpr(PACKED) {
                        const VT up = __shfl_up_sync(0xffffffffu, u7[3], 1);
                        const VT dn = __shfl_down_sync(0xffffffffu, u7[3], 1);
                        if(lane != 0) u7[2] = up;
                        if(lane != 31) u7[4] = dn;
                    }
                    const VT wNew = apply_row(rowE[u], has[u], dg[u], u7);
                    const size_t e = base + (size_t)(g0 + u) * kLanes;
                    if(e < (size_t)n) {
                        st_state(sOut + e, rNew, wNew, sNew, o.inv);
                        a.p[e] = pNew;
                        a.x[e] = xNew;
                        g = g + (double)u7[3] * (double)rNew;
                        d = d + (double)wNew * (double)u7[3];
                        const double ab = (double)vabs(rNew);
                        m = m > ab ? m : ab;
                    }
                }
            }
            double bg, bd, bm;
            block_sum2_max_256(g, d, m, sa, sb, smx, bg, bd, bm);
            if(threadIdx.x == 0) { pg[c] = bg; pd[c] = bd; pm[c] = bm; }
        }
        if(!grid_barrier(a.gs, nb, sense, flags, solve_barrier_limit())) return;
        double gNew, dNew, mNew;
        reduce_partials2_bcast(pg, pd, pm, nch, sa, sb, smx, gNew, dNew, mNew);
        resid = (VT)mNew;
        ++iter;
        if(resid < tol) {
            success = 1;
            break;
        }
        if(iter >= a.maxIter) {
            if(blockIdx.x == 0 && threadIdx.x == 0) atomicOr(flags, BNN_FLAG_PCG_MAXITER);
            break;
        }
        gammaOld = gamma;
        gamma = gNew;
        delta = dNew;
        a64Old = a64;
        cur = 1 - cur;
        set = 1 - set;
        first = false;
    }
    if(blockIdx.x == 0 && threadIdx.x == 0) {
        a.dst->iter = iter;
        a.dst->success = success;
        a.dst->done = 1;
        Sc<VT>::set_resid(a.dst, resid);
    }
}

// ---- iterative refinement helpers -------------------------------------------------
// Last-block-done over a block's share `blk` of a launch (the batched launches give every
// scene its own share, so the count to reach is the share's, not gridDim.x)
__device__ __forceinline__ bool last_block_of(unsigned* counter, unsigned nblocks) {
    __shared__ bool amLast;
    __threadfence();
    __syncthreads();
    if(threadIdx.x == 0) amLast = atomicAdd(counter, 1u) == nblocks - 1;
    __syncthreads();
    return amLast;
}
// x64 = 0, r64 = b, outer_bmax = outer_res = max|b|
__device__ __forceinline__ void ir_init_body(Blk blk, int n, const float* __restrict__ b, double* __restrict__ x64,
                                             double* __restrict__ r64, double* __restrict__ partMax, DevState* st) {
    __shared__ double sm[kLanes];
    const size_t base = (size_t)blk.x * kChunk + threadIdx.x;
    double m = 0.0;
    for(int j = 0; j < kPerLane; ++j) {
        const size_t e = base + (size_t)j * kLanes;
        if(e < (size_t)n) {
            const double bv = (double)b[e];
            x64[e] = 0.0;
            r64[e] = bv;
            const double a = vabs(bv);
            m = m > a ? m : a;
        }
    }
    const double bm = block_max_t(m, sm);
    if(threadIdx.x == 0) partMax[blk.x] = bm;
    if(last_block_of(&st->counter3, blk.n)) {
        const double mx = reduce_max_t(partMax, (int)blk.n, sm);
        if(threadIdx.x == 0) { st->counter3 = 0; st->outer_bmax = mx; st->outer_res = mx; }
    }
}
__global__ void __launch_bounds__(kLanes) k_ir_init(int n, const float* __restrict__ b, double* __restrict__ x64,
                                                    double* __restrict__ r64, double* __restrict__ partMax,
                                                    DevState* st) {
    ir_init_body(own_blk(), n, b, x64, r64, partMax, st);
}
// r32 = (float) r64
__global__ void k_ir_to_f32(int n, const double* __restrict__ r64, float* __restrict__ r32) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(e < (size_t)n) r32[e] = (float)r64[e];
}
__global__ void k_ir_accumulate(int n, double* __restrict__ x64, const float* __restrict__ d) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(e < (size_t)n) x64[e] = x64[e] + (double)d[e];
}
// r64 = b - A x64 in FP64, outer_res = max|r64|
__device__ __forceinline__ void ir_residual_body(Blk blk, int n, const float* __restrict__ b,
                                                 const double* __restrict__ x64, double* __restrict__ r64,
                                                 const float* __restrict__ diag, const int32_t* __restrict__ nbr,
                                                 const float* __restrict__ coef, double negoff,
                                                 double* __restrict__ partMax, DevState* st) {
    __shared__ double sm[kLanes];
    const size_t base = (size_t)blk.x * kChunk + threadIdx.x;
    double m = 0.0;
    for(int j = 0; j < kPerLane; ++j) {
        const size_t e = base + (size_t)j * kLanes;
        if(e < (size_t)n) {
            const int32_t nn[6] = {nbr[e], nbr[(size_t)n + e], nbr[2 * (size_t)n + e], nbr[3 * (size_t)n + e],
                                   nbr[4 * (size_t)n + e], nbr[5 * (size_t)n + e]};
            double co[6];
#pragma unroll
            for(int q = 0; q < 6; ++q) co[q] = coef ? (double)coef[(size_t)q * n + e] : negoff;
            double t = 0.0;
            if(nn[0] >= 0) t += co[0] * x64[nn[0]];
            if(nn[1] >= 0) t += co[1] * x64[nn[1]];
            if(nn[2] >= 0) t += co[2] * x64[nn[2]];
            if(diag[e] != 0.f) t += (double)diag[e] * x64[e];
            if(nn[3] >= 0) t += co[3] * x64[nn[3]];
            if(nn[4] >= 0) t += co[4] * x64[nn[4]];
            if(nn[5] >= 0) t += co[5] * x64[nn[5]];
            const double rv = (double)b[e] - t;
            r64[e] = rv;
            const double a = vabs(rv);
            m = m > a ? m : a;
        }
    }
    const double bm = block_max_t(m, sm);
    if(threadIdx.x == 0) partMax[blk.x] = bm;
    if(last_block_of(&st->counter3, blk.n)) {
        const double mx = reduce_max_t(partMax, (int)blk.n, sm);
        if(threadIdx.x == 0) { st->counter3 = 0; st->outer_res = mx; }
    }
}
__global__ void __launch_bounds__(kLanes) k_ir_residual(int n, const float* __restrict__ b,
                                                        const double* __restrict__ x64, double* __restrict__ r64,
                                                        const float* __restrict__ diag,
                                                        const int32_t* __restrict__ nbr,
                                                        const float* __restrict__ coef, double negoff,
                                                        double* __restrict__ partMax, DevState* st) {
    ir_residual_body(own_blk(), n, b, x64, r64, diag, nbr, coef, negoff, partMax, st);
}
__global__ void k_inv_diag64(int n, const float* __restrict__ diag, double* __restrict__ inv) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(e < (size_t)n) inv[e] = diag[e] != 0.f ? 1.0 / (double)diag[e] : 0.0;
}
__global__ void k_f32_to_f64(int n, const float* __restrict__ a, double* __restrict__ b) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(e < (size_t)n) b[e] = (double)a[e];
}
__global__ void k_d64_to_f32(int n, const double* __restrict__ a, float* __restrict__ b) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(e < (size_t)n) b[e] = (float)a[e];
}

// A block stages its 256 rows of the table through shared memory, so that both the table's
// reads and the planes' writes are coalesced (161,057 rows: 12 us; with one allocation instead of
// eight the whole bnn_pcg_solve_7pt call went from 5.7 to 1.7 ms).
// Indices are only compared here, never followed; the caller reads `bad` before any solve.
__global__ void __launch_bounds__(256) k_rows_from_table(int n, const int32_t* __restrict__ table,
                                                         const float* __restrict__ diag, int32_t* __restrict__ planes,
                                                         float* __restrict__ invd, RowsInfo* info) {
    __shared__ int32_t sm[6 * 256];
    const int r0 = blockIdx.x * 256, rows = min(256, n - r0), r = r0 + (int)threadIdx.x;
    for(int i = threadIdx.x; i < 6 * rows; i += 256) sm[i] = __ldg(table + 6 * (size_t)r0 + i);
    __syncthreads();
    unsigned bad = 0, notGrid = 0;
    int dy = 0, dz = 0;
    if(r < n) {
        int32_t nb[6];
#pragma unroll
        for(int q = 0; q < 6; ++q) {
            nb[q] = sm[6 * threadIdx.x + q];
            bad |= nb[q] < -1 || nb[q] >= n;
            planes[(size_t)q * n + r] = nb[q];
        }
        const float d = __ldg(diag + r);
        invd[r] = d != 0.f ? 1.0f / d : 0.f;
        if(nb[2] >= 0 && nb[2] != r - 1) notGrid = 1;
        if(nb[3] >= 0 && nb[3] != r + 1) notGrid = 1;
        if(nb[1] >= 0) { if(nb[1] >= r || r - nb[1] > 65535) notGrid = 1; else dy = max(dy, r - nb[1]); }
        if(nb[4] >= 0) { if(nb[4] <= r || nb[4] - r > 65535) notGrid = 1; else dy = max(dy, nb[4] - r); }
        if(nb[0] >= 0) { if(nb[0] >= r) notGrid = 1; else dz = max(dz, r - nb[0]); }
        if(nb[5] >= 0) { if(nb[5] <= r) notGrid = 1; else dz = max(dz, nb[5] - r); }
    }
    bad = __syncthreads_or((int)bad);
    notGrid = __syncthreads_or((int)notGrid);
    dy = __reduce_max_sync(0xffffffffu, dy);
    dz = __reduce_max_sync(0xffffffffu, dz);
    if((threadIdx.x & 31) == 0) {
        if(dy > *(volatile int*)&info->maxDy) atomicMax(&info->maxDy, dy);
        if(dz > *(volatile int*)&info->maxDz) atomicMax(&info->maxDz, dz);
    }
    if(threadIdx.x == 0) {
        if(bad) atomicOr(&info->bad, 1u);
        if(notGrid) atomicOr(&info->notGrid, 1u);
    }
}
void launch_rows_from_table(int n, const int32_t* table, const float* diag, int32_t* planes, float* invd, RowsInfo* info,
                            cudaStream_t s) {
    k_rows_from_table<<<(n + 255) / 256, 256, 0, s>>>(n, table, diag, planes, invd, info);
    bnn_note_launch();
}

// Packs rows of a grid into the 16-byte records
__global__ void k_pack_rows(int n, const float* __restrict__ diag, const int32_t* __restrict__ nbr,
                            int4* __restrict__ rec) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if(r >= n) return;
    int32_t nb[6];
#pragma unroll
    for(int q = 0; q < 6; ++q) nb[q] = nbr[(size_t)q * n + r];
    rec[r] = pack_row(r, nb, diag[r]);
}
// The off-diagonal planes of the rows as 2 float4 per row (6 values, plane order)
__global__ void k_pack_coef(int n, const float* __restrict__ coef, float4* __restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if(r >= n) return;
    float c[6];
#pragma unroll
    for(int q = 0; q < 6; ++q) c[q] = coef[(size_t)q * n + r];
    out[2 * (size_t)r] = make_float4(c[0], c[1], c[2], c[3]);
    out[2 * (size_t)r + 1] = make_float4(c[4], c[5], 0.f, 0.f);
}

// ---------------------------------------------------------------------------------
// Host driver
// ---------------------------------------------------------------------------------

// Process-wide record of the cooperative PCG kernels: SM count, resident blocks per SM of
// each variant, and what the solves in flight hold of the GPU (coop_share.cuh).
struct CoopState {
    std::mutex mu;
    std::condition_variable cv;
    int numSM = 0;
    int perSM[16] = {};
    CoopLoad held;
};
static CoopState g_coop;

static int coop_sm_count(int& numSM) {
    std::lock_guard<std::mutex> lk(g_coop.mu);
    if(!g_coop.numSM) {
        int dev = 0;
        BNN_CUDA_CHECK(cudaGetDevice(&dev));
        BNN_CUDA_CHECK(cudaDeviceGetAttribute(&g_coop.numSM, cudaDevAttrMultiProcessorCount, dev));
    }
    numSM = g_coop.numSM;
    return BNN_OK;
}

// Holds a launch's part of the GPU for the lifetime of the object; waits while other solves
// hold so much that it would not fit beside them.  A launch fits an empty GPU.
struct CoopShare {
    const CoopLoad load;
    CoopShare(const CoopLoad& l, int numSM) : load(l) {
        std::unique_lock<std::mutex> lk(g_coop.mu);
        g_coop.cv.wait(lk, [&] { return coop_fits(g_coop.held + load, numSM); });
        g_coop.held = g_coop.held + load;
    }
    CoopShare(const CoopShare&) = delete;
    ~CoopShare() {
        {
            std::lock_guard<std::mutex> lk(g_coop.mu);
            g_coop.held = g_coop.held - load;
        }
        g_coop.cv.notify_all();
    }
};

int pcg_reserve(PcgWork& w, int n, bool fp64) {
    if(n <= w.cap && (!fp64 || w.x64)) return BNN_OK;
    if(n > w.cap) {
        pcg_release(w);
        // whole chunks: the chunk-resident solve writes its last chunk's rows past n too
        const int cap = ((int)(n * 1.25) + 4096 + kChunk - 1) / kChunk * kChunk;
        const size_t nch = ((size_t)cap + kChunk - 1) / kChunk + 1;
        w.nchCap = (int)nch;
        BNN_CUDA_CHECK(dev_alloc(&w.x, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.r, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.z, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.s0, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.s1, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.q, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.d32, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.r32, cap * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.rec, cap * sizeof(int4)));
        BNN_CUDA_CHECK(dev_alloc(&w.part, 3 * nch * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.packets, 2 * nch * kPacketStride * sizeof(PcgPacket)));
        BNN_CUDA_CHECK(dev_alloc(&w.gs, sizeof(GridSync)));
        BNN_CUDA_CHECK(cudaMemset(w.gs, 0, sizeof(GridSync)));
        BNN_CUDA_CHECK(dev_alloc(&w.partMaxF, nch * sizeof(float)));
        BNN_CUDA_CHECK(dev_alloc(&w.partMaxD, nch * sizeof(double)));
        w.cap = cap;
    }
    for(auto& e : w.ev)
        if(!e) BNN_CUDA_CHECK(cudaEventCreate(&e));
    if(!w.st32[0]) {
        // single-reduction solve: double-buffered row records and partials
        for(int b = 0; b < 2; ++b) BNN_CUDA_CHECK(dev_alloc(&w.st32[b], w.cap * sizeof(float4)));
        BNN_CUDA_CHECK(dev_alloc(&w.cgPart, 4 * (size_t)w.nchCap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.cgMax, 2 * (size_t)w.nchCap * sizeof(double)));
    }
    if(fp64 && !w.st64[0])
        for(int b = 0; b < 2; ++b) BNN_CUDA_CHECK(dev_alloc(&w.st64[b], w.cap * 4 * sizeof(double)));
    if(fp64 && !w.x64) {
        BNN_CUDA_CHECK(dev_alloc(&w.x64, w.cap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.r64, w.cap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.z64, w.cap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.s064, w.cap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.s164, w.cap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.q64, w.cap * sizeof(double)));
        BNN_CUDA_CHECK(dev_alloc(&w.inv64, w.cap * sizeof(double)));
    }
    return BNN_OK;
}

void pcg_release(PcgWork& w) {
    for(auto& e : w.ev)
        if(e) cudaEventDestroy(e);
    for(void* p : {(void*)w.rec, (void*)w.coefRow, (void*)w.x, (void*)w.r, (void*)w.z, (void*)w.s0, (void*)w.s1, (void*)w.q, (void*)w.d32, (void*)w.r32,
                   (void*)w.part, (void*)w.partMaxF, (void*)w.partMaxD, (void*)w.x64, (void*)w.r64, (void*)w.z64,
                   (void*)w.s064, (void*)w.s164, (void*)w.q64, (void*)w.inv64, (void*)w.gs, (void*)w.packets, (void*)w.st32[0],
                   (void*)w.st32[1], (void*)w.st64[0], (void*)w.st64[1], (void*)w.cgPart, (void*)w.cgMax})
        if(p) dev_free(p);
    w = PcgWork();
}

struct ChunkKernel {
    const void* fn = nullptr;
    size_t smem = 0;
};
template<class VT> static ChunkKernel cluster_kernel(bool coef) {
    if(coef) return {(const void*)k_pcg_cluster<VT, true>, sizeof(ClusterSmem<VT, true>)};
    return {(const void*)k_pcg_cluster<VT, false>, sizeof(ClusterSmem<VT, false>)};
}
static cudaLaunchConfig_t cluster_config(const ChunkKernel& k, int blocks, cudaLaunchAttribute* attr, cudaStream_t s) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)blocks;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3(kLanes);
    c.dynamicSmemBytes = k.smem;
    c.stream = s;
    c.attrs = attr;
    c.numAttrs = 1;
    return c;
}
static cudaError_t cluster_opt_in(const ChunkKernel& k) {
    const cudaError_t e = cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    if(e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
// Whether the current device can hold such a cluster (blocks of a whole SM each within one
// GPC); asked once per device and size
template<class VT> static bool cluster_fits(bool coef, int blocks) {
    static std::atomic<uint32_t> known[64];  // per device: bit 2i asked, 2i + 1 the answer
    int dev = 0;
    if(cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int i = coef ? 5 : 0;  // + log2 of the blocks, 0 .. 4
    for(int b = 1; b < blocks; b *= 2) ++i;
    const uint32_t k = known[dev].load(std::memory_order_acquire);
    if(k >> (2 * i) & 1u) return (k >> (2 * i + 1) & 1u) != 0u;
    const ChunkKernel kern = cluster_kernel<VT>(coef);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cluster_config(kern, blocks, &attr, nullptr);
    int clusters = 0;
    const bool ok = cluster_opt_in(kern) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, kern.fn, &cfg) == cudaSuccess && clusters > 0;
    if(!ok) cudaGetLastError();
    known[dev].fetch_or(1u << (2 * i) | (uint32_t)ok << (2 * i + 1), std::memory_order_acq_rel);
    return ok;
}

// The shape of a chunk-resident solve of n rows: groups per block and chunks per group (0:
// more chunks than it holds, they take turns in k_pcg_persistent).  One block per SM; as few
// groups as hold the chunks (more registers and loads in flight for each), then two chunks per
// group.  The line lies where registers and shared memory end: 6 FP32 chunks per SM are 210 KB
// of records, s and partials (1.82 M rows on 148 SMs), 4 FP64 chunks 186 KB; with off-diagonal
// values 2 and 1.  Up to that line it is faster than k_pcg_persistent at every size (figures
// above).
struct ChunkShape {
    int G = 0, K = 0;
    int cluster = 0;  // blocks of the one cluster (k_pcg_cluster); 0: k_pcg_chunk over the grid
};
template<class VT> static ChunkShape chunk_shape(int n, bool coef, int numSM) {
    const int nch = (n + kChunk - 1) / kChunk;
    // up to 16 chunks, the most blocks of a cluster: k_pcg_cluster, a power of two of blocks
    if(nch <= kMostCluster) {
        int blocks = 1;
        while(blocks < nch) blocks *= 2;
        if(cluster_fits<VT>(coef, blocks)) return ChunkShape{1, 1, blocks};
    }
    const int per = (nch + numSM - 1) / numSM;
    if(coef) return per <= (sizeof(VT) == 4 ? 2 : 1) ? ChunkShape{per, 1} : ChunkShape{};
    const int most = sizeof(VT) == 4 ? 3 : 2;
    if(per <= most) return {per, 1};
    return per <= 2 * most ? ChunkShape{most, 2} : ChunkShape{};
}
template<class VT, bool COEF, int G, int K> static ChunkKernel chunk_kernel_of() {
    return {(const void*)k_pcg_chunk<VT, COEF, G, K>, sizeof(ChunkSmem<VT, COEF, G, K>)};
}
template<class VT> static ChunkKernel chunk_kernel(bool coef, ChunkShape c) {
    if(coef) {
        if constexpr(sizeof(VT) == 4) if(c.G == 2) return chunk_kernel_of<VT, true, 2, 1>();
        return chunk_kernel_of<VT, true, 1, 1>();
    }
    if(c.G == 1) return chunk_kernel_of<VT, false, 1, 1>();
    if constexpr(sizeof(VT) == 4) {
        if(c.G == 2) return chunk_kernel_of<VT, false, 2, 1>();
        return c.K == 1 ? chunk_kernel_of<VT, false, 3, 1>() : chunk_kernel_of<VT, false, 3, 2>();
    } else {
        return c.K == 1 ? chunk_kernel_of<VT, false, 2, 1>() : chunk_kernel_of<VT, false, 2, 2>();
    }
}

// What the host waits for after a solve's launch: the state record, and the launch's time
template<class VT> static int pcg_read_outcome(PcgWork& w, DevState* dst, DevState* hst, cudaStream_t s, PcgOutcome& out) {
    BNN_CUDA_CHECK(cudaMemcpyAsync(hst, dst, sizeof(DevState), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    if(w.ev[0] && w.ev[1]) {
        float ms = 0.f;
        if(cudaEventElapsedTime(&ms, w.ev[0], w.ev[1]) == cudaSuccess) out.kernelMs = ms;
    }
    if(hst->flags & BNN_FLAG_TIMEOUT) { bnn_set_error("PCG grid barrier timed out"); return BNN_ERR_TIMEOUT; }
    out.iterations = hst->iter;
    out.success = hst->success;
    out.residual = sizeof(VT) == 8 ? hst->resid64 : (double)hst->resid;
    return BNN_OK;
}

// One PCG solve by k_pcg_chunk in the shape chunk_shape gave
template<class VT>
static int pcg_solve_chunk(PcgWork& w, int n, ChunkShape shape, int numSM, const float* rhsF, const float* diag,
                           const VT* invd, const int32_t* nbr, const float* coef, VT negoff, VT tolFactor,
                           unsigned maxIter, VT* x, DevState* dst, DevState* hst, cudaStream_t s, PcgOutcome& out) {
    out = PcgOutcome();
    ChunkArgs<VT> a;
    a.n = n; a.nch = (n + kChunk - 1) / kChunk;
    a.rhsF = rhsF; a.diag = diag; a.invd = invd; a.nbr = nbr; a.coef = coef; a.negoff = negoff;
    a.tolFactor = tolFactor; a.maxIter = maxIter; a.x = x;
    a.pair = sizeof(VT) == 8 ? (RowPair<VT>*)(void*)w.st64[0] : (RowPair<VT>*)(void*)w.st32[0];
    a.pairStride = w.cap;
    a.pkA = w.packets;
    a.pkB = a.pkA + (size_t)w.nchCap * kPacketStride;
    a.st = dst;
    void* args[] = {(void*)&a};
    if(shape.cluster > 0) {
        // blocks of a cluster start together and wait for no other launch: no share to hold
        const ChunkKernel kern = cluster_kernel<VT>(coef != nullptr);
        BNN_CUDA_CHECK(cluster_opt_in(kern));
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = cluster_config(kern, shape.cluster, &attr, s);
        if(w.ev[0]) BNN_CUDA_CHECK(cudaEventRecord(w.ev[0], s));
        BNN_CUDA_CHECK(cudaLaunchKernelExC(&cfg, kern.fn, args));
        bnn_note_launch();
        if(w.ev[1]) BNN_CUDA_CHECK(cudaEventRecord(w.ev[1], s));
        return pcg_read_outcome<VT>(w, dst, hst, s, out);
    }
    const ChunkKernel kern = chunk_kernel<VT>(coef != nullptr, shape);
    BNN_CUDA_CHECK(cudaFuncSetAttribute(kern.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kern.smem));
    BNN_CUDA_CHECK(cudaMemsetAsync(w.packets, 0, 2 * (size_t)w.nchCap * kPacketStride * sizeof(PcgPacket), s));
    const int most = numSM < kMostSM ? numSM : kMostSM, grid = a.nch < most ? a.nch : most;
    CoopShare share(CoopLoad{grid, 0, 0}, numSM);
    if(w.ev[0]) BNN_CUDA_CHECK(cudaEventRecord(w.ev[0], s));
    BNN_CUDA_CHECK(cudaLaunchCooperativeKernel(kern.fn, dim3(grid), dim3(shape.G * kLanes), args, kern.smem, s));
    bnn_note_launch();
    if(w.ev[1]) BNN_CUDA_CHECK(cudaEventRecord(w.ev[1], s));
    return pcg_read_outcome<VT>(w, dst, hst, s, out);
}

// Runs one PCG solve (VT vectors) as a single cooperative launch.  Returns BNN status;
// the solution is left in x.
template<class VT>
static int pcg_solve_t(PcgWork& w, int n, ChunkShape shape, int numSM, const float* rhsF, const float* diag, const VT* invd, const int32_t* nbr,
                       const int4* rec, const float* coef, const float4* coefRow, VT negoff, VT tolFactor, unsigned maxIter, VT* x, VT* r, VT* z, VT* s0, VT* s1, VT* q,
                       VT* partMax, bool twoReductions, DevState* dst, DevState* hst, cudaStream_t s, PcgOutcome& out) {
    out = PcgOutcome();
    if(n == 0) { out.success = 1; return BNN_OK; }
    if(shape.G > 0)
        return pcg_solve_chunk<VT>(w, n, shape, numSM, rhsF, diag, invd, nbr, coef, negoff, tolFactor, maxIter, x, dst, hst,
                                   s, out);
    const int nch = (n + kChunk - 1) / kChunk;
    const bool packedCoef = rec && coefRow;
    // kernel variant: bit 0 FP64, bit 1 packed rows, bit 2 coefficients, bit 3 single reduction
    const int ti = (sizeof(VT) == 8 ? 1 : 0) + (rec ? 2 : 0) + ((coef || coefRow) ? 4 : 0) + (twoReductions ? 0 : 8);
    const void* kern;
    if(twoReductions)
        kern = packedCoef ? (const void*)k_pcg_persistent<VT, true, true>
                          : (rec ? (const void*)k_pcg_persistent<VT, true> : (const void*)k_pcg_persistent<VT, false>);
    else if(rec)
        kern = coefRow ? (const void*)k_pcg_cg1<VT, true, true> : (const void*)k_pcg_cg1<VT, true, false>;
    else
        kern = coef ? (const void*)k_pcg_cg1<VT, false, true> : (const void*)k_pcg_cg1<VT, false, false>;
    int perSMv = 0;
    {
        std::lock_guard<std::mutex> lk(g_coop.mu);
        if(!g_coop.perSM[ti]) {
            BNN_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_coop.perSM[ti], kern, kLanes, 0));
            if(g_coop.perSM[ti] < 1) { bnn_set_error("persistent PCG kernel cannot be resident"); return BNN_ERR_CUDA; }
        }
        perSMv = g_coop.perSM[ti];
    }
    const int cap = numSM * perSMv;
    const int perBlock = (nch + cap - 1) / cap;           // chunks per block
    const int grid = (nch + perBlock - 1) / perBlock;     // balanced: every block the same count
    PcgArgs<VT> a;
    a.n = n; a.rhsF = rhsF; a.diag = diag; a.invd = invd; a.nbr = nbr; a.rec = rec; a.coef = coef; a.coefRow = coefRow; a.negoff = negoff; a.tolFactor = tolFactor;
    a.maxIter = maxIter; a.x = x; a.r = r; a.z = z; a.s0 = s0; a.s1 = s1; a.q = q;
    a.part0 = w.part; a.part1 = w.part + w.nchCap; a.part2 = w.part + 2 * (size_t)w.nchCap; a.partMax = partMax;
    a.st = dst; a.gs = w.gs;
    Cg1Args<VT> c;
    c.n = n; c.rhsF = rhsF; c.diag = diag; c.invd = invd; c.nbr = nbr; c.rec = rec; c.coef = coef; c.coefRow = coefRow;
    c.negoff = negoff; c.tolFactor = tolFactor; c.maxIter = maxIter; c.x = x; c.p = s0;
    for(int b = 0; b < 2; ++b)
        c.st[b] = sizeof(VT) == 8 ? (RowState<VT>*)(void*)w.st64[b] : (RowState<VT>*)(void*)w.st32[b];
    c.part = w.cgPart; c.pmax = w.cgMax; c.nchCap = w.nchCap; c.dst = dst; c.gs = w.gs;
    BNN_CUDA_CHECK(cudaMemsetAsync(&w.gs->count, 0, sizeof(unsigned), s));
    void* args[] = {twoReductions ? (void*)&a : (void*)&c};
    // grids of concurrent solves (several solver handles on several host threads) must
    // fit the GPU together, or blocks of one could wait for SMs held by another's barrier
    CoopShare share(CoopLoad{0, grid, grid * (kShareUnits / perSMv)}, numSM);
    if(w.ev[0]) BNN_CUDA_CHECK(cudaEventRecord(w.ev[0], s));
    BNN_CUDA_CHECK(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kLanes), args, 0, s));
    bnn_note_launch();
    if(w.ev[1]) BNN_CUDA_CHECK(cudaEventRecord(w.ev[1], s));
    return pcg_read_outcome<VT>(w, dst, hst, s, out);
}

// mode: BNN_PCG_FP32 / FP64 / REFINED, optionally with BNN_PCG_SINGLE_REDUCTION.  Pressure
// written to `pressure` (float, n).
int pcg_solve(PcgWork& w, int n, const float* rhs, const float* diag, const float* invd, const int32_t* nbr,
              const float* coef, RowLayout layout, float dt, int modeFlags, float tol, unsigned maxIter, float innerTol,
              float outerTol, float* pressure, double* x64out, DevState* dst, DevState* hst, cudaStream_t s,
              PcgOutcome& out) {
    const int mode = modeFlags & BNN_PCG_MODE_MASK;
    const bool two = (modeFlags & BNN_PCG_SINGLE_REDUCTION) == 0;
    int rc = pcg_reserve(w, n, mode != BNN_PCG_FP32);
    if(rc != BNN_OK) return rc;
    const unsigned nb = (unsigned)((n + 255) / 256);
    const unsigned nch = (unsigned)((n + kChunk - 1) / kChunk);
    out = PcgOutcome();
    const int4* rec = nullptr;
    const float4* coefRow = nullptr;
    int numSM = 0;
    rc = coop_sm_count(numSM);
    if(rc != BNN_OK) return rc;
    const int chunkSM = numSM < kMostSM ? numSM : kMostSM;
    const bool gridRows = layout != kRowsAny;
    ChunkShape shape;
    if(layout == kRowsCompact && two && n > 0)
        shape = mode == BNN_PCG_FP64 ? chunk_shape<double>(n, coef != nullptr, chunkSM)
                                     : chunk_shape<float>(n, coef != nullptr, chunkSM);
    if(gridRows && n > 0 && shape.G == 0) {
        { k_pack_rows<<<nb, 256, 0, s>>>(n, diag, nbr, w.rec); bnn_note_launch(); }
        rec = w.rec;
        if(coef) {
            // off-diagonal values ride along as 2 float4 per row
            if(!w.coefRow) BNN_CUDA_CHECK(dev_alloc(&w.coefRow, 2 * (size_t)w.cap * sizeof(float4)));
            { k_pack_coef<<<nb, 256, 0, s>>>(n, coef, w.coefRow); bnn_note_launch(); }
            coefRow = w.coefRow;
        }
    }
    if(mode == BNN_PCG_FP32) {
        rc = pcg_solve_t<float>(w, n, shape, numSM, rhs, diag, invd, nbr, rec, coef, coefRow, -(1.0f * dt), tol, maxIter, w.x, w.r, w.z, w.s0, w.s1,
                                w.q, w.partMaxF, two, dst, hst, s, out);
        if(rc != BNN_OK) return rc;
        if(n > 0) BNN_CUDA_CHECK(cudaMemcpyAsync(pressure, w.x, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
        if(x64out && n > 0) { k_f32_to_f64<<<nb, 256, 0, s>>>(n, w.x, x64out); bnn_note_launch(); }
        return BNN_OK;
    }
    if(mode == BNN_PCG_FP64) {
        if(n > 0) { k_inv_diag64<<<nb, 256, 0, s>>>(n, diag, w.inv64); bnn_note_launch(); }
        rc = pcg_solve_t<double>(w, n, shape, numSM, rhs, diag, w.inv64, nbr, rec, coef, coefRow, -(double)(1.0f * dt), (double)tol, maxIter, w.x64,
                                 w.r64, w.z64, w.s064, w.s164, w.q64, w.partMaxD, two, dst, hst, s, out);
        if(rc != BNN_OK) return rc;
        if(n > 0) { k_d64_to_f32<<<nb, 256, 0, s>>>(n, w.x64, pressure); bnn_note_launch(); }
        if(x64out && n > 0)
            BNN_CUDA_CHECK(cudaMemcpyAsync(x64out, w.x64, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
        return BNN_OK;
    }
    // refined: FP64 outer residual and solution, FP32 inner solves
    if(n == 0) { out.success = 1; return BNN_OK; }
    { k_ir_init<<<nch, kLanes, 0, s>>>(n, rhs, w.x64, w.r64, w.partMaxD, dst); bnn_note_launch(); }
    BNN_CUDA_CHECK(cudaMemcpyAsync(hst, dst, sizeof(DevState), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    const double bmax = hst->outer_bmax;
    unsigned total = 0, outer = 0;
    float kernelMs = 0.f;
    const unsigned maxOuter = 60;
    double res = bmax;
    bool ok = bmax < (double)FLT_MIN;
    while(!ok && outer < maxOuter) {
        if(res < (double)outerTol * bmax) { ok = true; break; }
        { k_ir_to_f32<<<nb, 256, 0, s>>>(n, w.r64, w.r32); bnn_note_launch(); }
        PcgOutcome inner;
        rc = pcg_solve_t<float>(w, n, shape, numSM, w.r32, diag, invd, nbr, rec, coef, coefRow, -(1.0f * dt), innerTol, maxIter, w.d32, w.r, w.z, w.s0,
                                w.s1, w.q, w.partMaxF, two, dst, hst, s, inner);
        if(rc != BNN_OK) return rc;
        total += inner.iterations;
        kernelMs += inner.kernelMs;
        { k_ir_accumulate<<<nb, 256, 0, s>>>(n, w.x64, w.d32); bnn_note_launch(); }
        { k_ir_residual<<<nch, kLanes, 0, s>>>(n, rhs, w.x64, w.r64, diag, nbr, coef, (double)(-(1.0f * dt)), w.partMaxD, dst); bnn_note_launch(); }
        BNN_CUDA_CHECK(cudaMemcpyAsync(hst, dst, sizeof(DevState), cudaMemcpyDeviceToHost, s));
        BNN_CUDA_CHECK(cudaStreamSynchronize(s));
        res = hst->outer_res;
        ++outer;
        if(total >= maxIter) break;
    }
    if(!ok && res < (double)outerTol * bmax) ok = true;
    out.iterations = total;
    out.outer = outer;
    out.kernelMs = kernelMs;
    out.residual = res;
    out.success = ok ? 1 : 0;
    { k_d64_to_f32<<<nb, 256, 0, s>>>(n, w.x64, pressure); bnn_note_launch(); }
    if(x64out) BNN_CUDA_CHECK(cudaMemcpyAsync(x64out, w.x64, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    return BNN_OK;
}

// ---------------------------------------------------------------------------------
// Batched refinement: pcg_solve's BNN_PCG_REFINED loop for many scenes at once.  Every
// stage is one launch over the scenes still refining (each scene's blocks found through a
// per-scene block prefix, as the batched step kernels do); their inner FP32 solves are
// k_pcg_chunk_batch launches of as many scenes as are resident together.  A scene that does
// not fit the chunk-resident solve is solved alone, between them.  The host keeps each scene's
// outer loop state and takes exactly the decisions the lone loop takes, from the same device
// values.
// ---------------------------------------------------------------------------------
struct IrScene {
    int n;
    const float* b;            // right-hand side
    double *x64, *r64;
    float *r32, *d32;
    const float* diag;
    const int32_t* nbr;
    double negoff;             // (double)(-(1 * dt))
    double* partMax;
    DevState* st;
    float* pressure;
    PcgPacket *pkA, *pkB;      // of the chunk-resident solve, zeroed before it
};
struct IrReport {
    double res, bmax;
    unsigned iter, flags, done, pad;
};

__global__ void __launch_bounds__(kLanes) kb_ir_init(const IrScene* __restrict__ S, const unsigned* __restrict__ P,
                                                     int ns) {
    int q;
    const Blk b = seg_blk(P, ns, q);
    const IrScene& c = S[q];
    ir_init_body(b, c.n, c.b, c.x64, c.r64, c.partMax, c.st);
}
// r32 = (float) r64, and the packets of the solve that follows zeroed (a block of 256 rows in
// every chunk does its chunk's)
__global__ void kb_ir_to_f32(const IrScene* __restrict__ S, const unsigned* __restrict__ P, int ns) {
    int q;
    const Blk b = seg_blk(P, ns, q);
    const IrScene& c = S[q];
    const size_t e = (size_t)b.x * blockDim.x + threadIdx.x;
    if(e < (size_t)c.n) c.r32[e] = (float)c.r64[e];
    if(b.x % kPerLane == 0 && threadIdx.x < 2) {
        PcgPacket* p = threadIdx.x == 0 ? c.pkA : c.pkB;
        p[(size_t)(b.x / kPerLane) * kPacketStride] = PcgPacket{0ull, 0ull};
    }
}
__global__ void kb_ir_accumulate(const IrScene* __restrict__ S, const unsigned* __restrict__ P, int ns) {
    int q;
    const Blk b = seg_blk(P, ns, q);
    const IrScene& c = S[q];
    const size_t e = (size_t)b.x * blockDim.x + threadIdx.x;
    if(e < (size_t)c.n) c.x64[e] = c.x64[e] + (double)c.d32[e];
}
__global__ void __launch_bounds__(kLanes) kb_ir_residual(const IrScene* __restrict__ S,
                                                         const unsigned* __restrict__ P, int ns) {
    int q;
    const Blk b = seg_blk(P, ns, q);
    const IrScene& c = S[q];
    ir_residual_body(b, c.n, c.b, c.x64, c.r64, c.diag, c.nbr, nullptr, c.negoff, c.partMax, c.st);
}
__global__ void kb_ir_finish(const IrScene* __restrict__ S, const unsigned* __restrict__ P, int ns) {
    int q;
    const Blk b = seg_blk(P, ns, q);
    const IrScene& c = S[q];
    const size_t e = (size_t)b.x * blockDim.x + threadIdx.x;
    if(e < (size_t)c.n) c.pressure[e] = (float)c.x64[e];
}
// one thread per scene: what the host's outer loop reads
__global__ void kb_ir_report(const IrScene* __restrict__ S, int ns, IrReport* __restrict__ out) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if(q < ns) {
        const DevState* st = S[q].st;
        out[q] = IrReport{st->outer_res, st->outer_bmax, st->iter, st->flags, st->done, 0u};
    }
}

namespace {
// Layout of the context's device blob (the same offsets in the pinned host mirror):
// IrScene[cap], ChunkArgs[cap], the prefixes of 256-row blocks and of 2048-row chunks (cap + 1
// each), BatchGroup[capGroups], then IrReport[cap] (read back, not uploaded).
struct BatchLayout {
    size_t irs, args, p256, pch, grp, rep, up, total;
    BatchLayout(int cap, int capGroups) {
        auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
        const size_t pre = (size_t)(cap + 1) * sizeof(unsigned);
        irs = 0;
        args = irs + al((size_t)cap * sizeof(IrScene));
        p256 = args + al((size_t)cap * sizeof(ChunkArgs<float>));
        pch = p256 + al(pre);
        grp = pch + al(pre);
        up = grp + al((size_t)capGroups * sizeof(BatchGroup));
        rep = up;
        total = rep + al((size_t)cap * sizeof(IrReport));
    }
};
// One launch of a round's inner solves: its shape, first group and blocks
struct BatchLaunch {
    ChunkShape shape;
    int group0 = 0, blocks = 0;
};
ChunkKernel batch_chunk_kernel(ChunkShape c) {
    if(c.K == 2) return {(const void*)k_pcg_chunk_batch<3, 2>, sizeof(BatchChunkSmem<float, 3, 2>)};
    if(c.G == 3) return {(const void*)k_pcg_chunk_batch<3, 1>, sizeof(BatchChunkSmem<float, 3, 1>)};
    if(c.G == 2) return {(const void*)k_pcg_chunk_batch<2, 1>, sizeof(BatchChunkSmem<float, 2, 1>)};
    return {(const void*)k_pcg_chunk_batch<1, 1>, sizeof(BatchChunkSmem<float, 1, 1>)};
}
// The groups of the scenes with these chunk counts, cut into launches whose groups are all
// resident.  Scenes go in descending size: those of a launch then take about as many
// iterations.  K = 1 while one launch holds all chunks that way, else 2 chunks per group.
// No scene may have more chunks than a launch holds (batch_most_chunks).
int batch_most_chunks(int numSM) { return numSM * 3 * 2; }
void batch_groups(const std::vector<int>& nch, int numSM, std::vector<BatchGroup>& groups, std::vector<BatchLaunch>& launches) {
    groups.clear();
    launches.clear();
    std::vector<int> order(nch.size());
    long long total = 0;
    for(size_t i = 0; i < nch.size(); ++i) { order[i] = (int)i; total += nch[i]; }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return nch[a] > nch[b]; });
    ChunkShape shape{3, 2};
    if(total <= (long long)numSM * 3) shape = ChunkShape{(int)((total + numSM - 1) / numSM), 1};
    const int most = numSM * shape.G;  // groups of a launch
    for(size_t i = 0; i < order.size();) {
        BatchLaunch l;
        l.shape = shape;
        l.group0 = (int)groups.size();
        int used = 0;
        for(; i < order.size(); ++i) {
            const int need = (nch[order[i]] + shape.K - 1) / shape.K;
            if(used + need > most) break;
            for(int c = 0; c < nch[order[i]]; c += shape.K) groups.push_back(BatchGroup{order[i], c});
            used += need;
        }
        l.blocks = (used + shape.G - 1) / shape.G;
        groups.resize((size_t)l.group0 + (size_t)l.blocks * shape.G, BatchGroup{-1, 0});
        launches.push_back(l);
    }
}
} // namespace

static int batch_reserve(BatchPcgCtx& ctx, int count, int groups) {
    if(count <= ctx.cap && groups <= ctx.capGroups && ctx.dev) return BNN_OK;
    const int cap = std::max(ctx.cap, count < 64 ? 64 : count + count / 4);
    const int capGroups = std::max(ctx.capGroups, groups + groups / 4 + 256);
    pcg_batch_release(ctx);
    const BatchLayout L(cap, capGroups);
    BNN_CUDA_CHECK(cudaMalloc(&ctx.dev, L.total));
    BNN_CUDA_CHECK(cudaMallocHost(&ctx.host, L.total));
    std::memset(ctx.host, 0, L.total);
    for(auto& e : ctx.ev) BNN_CUDA_CHECK(cudaEventCreate(&e));
    ctx.cap = cap;
    ctx.capGroups = capGroups;
    return BNN_OK;
}

void pcg_batch_release(BatchPcgCtx& ctx) {
    if(ctx.dev) cudaFree(ctx.dev);
    if(ctx.host) cudaFreeHost(ctx.host);
    for(auto& e : ctx.ev)
        if(e) cudaEventDestroy(e);
    ctx = BatchPcgCtx();
}

int pcg_solve_batch_refined(BatchPcgCtx& ctx, BatchSolveItem* items, int count, cudaStream_t s) {
    constexpr unsigned kMaxOuter = 60;  // pcg_solve's outer limit
    struct Outer {
        double bmax = 0, res = 0;
        unsigned outer = 0, total = 0;
        bool ok = false, stopped = false;
        float kernelMs = 0.f;
    };
    int numSM = 0;
    int rc = coop_sm_count(numSM);
    if(rc != BNN_OK) return rc;
    const int chunkSM = numSM < kMostSM ? numSM : kMostSM;
    auto chunks_of = [&](int i) { return (items[i].n + kChunk - 1) / kChunk; };
    std::vector<char> alone(count, 0);  // scenes the chunk-resident solve does not take
    std::vector<int> live;
    int groupsMost = 0;
    for(int i = 0; i < count; ++i) {
        items[i].out = PcgOutcome();
        if(items[i].n == 0) { items[i].out.success = 1; continue; }
        rc = pcg_reserve(*items[i].w, items[i].n, true);
        if(rc != BNN_OK) return rc;
        alone[i] = items[i].layout != kRowsCompact || chunks_of(i) > batch_most_chunks(chunkSM);
        live.push_back(i);
        groupsMost += chunks_of(i) + 1;
    }
    if(live.empty()) return BNN_OK;
    // a launch's last block may hold up to 2 empty groups, and there are no more launches than scenes
    rc = batch_reserve(ctx, (int)live.size(), groupsMost + 2 * (int)live.size());
    if(rc != BNN_OK) return rc;
    const BatchLayout L(ctx.cap, ctx.capGroups);
    char* H = (char*)ctx.host;
    char* D = (char*)ctx.dev;
    IrScene* hirs = (IrScene*)(H + L.irs);
    ChunkArgs<float>* hargs = (ChunkArgs<float>*)(H + L.args);
    unsigned* hp256 = (unsigned*)(H + L.p256);
    unsigned* hpch = (unsigned*)(H + L.pch);
    const IrReport* hrep = (const IrReport*)(H + L.rep);
    const IrScene* dirs = (const IrScene*)(D + L.irs);
    const unsigned* dp256 = (const unsigned*)(D + L.p256);
    const unsigned* dpch = (const unsigned*)(D + L.pch);
    IrReport* drep = (IrReport*)(D + L.rep);
    std::vector<BatchGroup> groups;
    std::vector<BatchLaunch> launches;

    // tables for the scenes `set` (positions in items), uploaded in one copy; solve: with the
    // groups of their inner solves
    auto upload = [&](const std::vector<int>& set, bool solve) -> cudaError_t {
        hp256[0] = hpch[0] = 0;
        std::vector<int> nch, at;
        for(size_t k = 0; k < set.size(); ++k) {
            const BatchSolveItem& it = items[set[k]];
            PcgWork& w = *it.w;
            const int n = it.n;
            PcgPacket *pkA = w.packets, *pkB = w.packets + (size_t)w.nchCap * kPacketStride;
            hirs[k] = IrScene{n, it.rhs, w.x64, w.r64, w.r32, w.d32, it.diag, it.nbr, (double)(-(1.0f * it.dt)),
                              w.partMaxD, it.dst, it.pressure, pkA, pkB};
            hp256[k + 1] = hp256[k] + (unsigned)((n + 255) / 256);
            hpch[k + 1] = hpch[k] + (unsigned)((n + kChunk - 1) / kChunk);
            ChunkArgs<float>& c = hargs[k];
            c.n = n; c.nch = chunks_of(set[k]); c.rhsF = w.r32; c.diag = it.diag; c.invd = it.invd; c.nbr = it.nbr;
            c.coef = nullptr; c.negoff = -(1.0f * it.dt); c.tolFactor = it.innerTol; c.maxIter = it.maxIter; c.x = w.d32;
            c.pair = (RowPair<float>*)(void*)w.st32[0]; c.pairStride = w.cap; c.pkA = pkA; c.pkB = pkB; c.st = it.dst;
            if(!alone[set[k]]) { nch.push_back(c.nch); at.push_back((int)k); }
        }
        if(solve) {
            batch_groups(nch, chunkSM, groups, launches);
            BatchGroup* hg = (BatchGroup*)(H + L.grp);
            for(size_t q = 0; q < groups.size(); ++q)
                hg[q] = BatchGroup{groups[q].scene < 0 ? -1 : at[groups[q].scene], groups[q].chunk0};
        }
        return cudaMemcpyAsync(D, H, solve ? L.up : L.grp, cudaMemcpyHostToDevice, s);
    };
    auto report = [&](int ns) -> int {
        { kb_ir_report<<<(ns + 127) / 128, 128, 0, s>>>(dirs, ns, drep); bnn_note_launch(); }
        BNN_CUDA_CHECK(cudaMemcpyAsync(H + L.rep, drep, (size_t)ns * sizeof(IrReport), cudaMemcpyDeviceToHost, s));
        BNN_CUDA_CHECK(cudaStreamSynchronize(s));
        for(int k = 0; k < ns; ++k)
            if(hrep[k].flags & BNN_FLAG_TIMEOUT) { bnn_set_error("batched PCG grid barrier timed out"); return BNN_ERR_TIMEOUT; }
        return BNN_OK;
    };

    // outer loop start of every scene: x64 = 0, r64 = b, bmax
    std::vector<Outer> o(count);
    const int nl = (int)live.size();
    BNN_CUDA_CHECK(upload(live, false));
    { kb_ir_init<<<hpch[nl], kLanes, 0, s>>>(dirs, dpch, nl); bnn_note_launch(); }
    for(int i : live)
        if(alone[i]) {
            k_pack_rows<<<(items[i].n + 255) / 256, 256, 0, s>>>(items[i].n, items[i].diag, items[i].nbr, items[i].w->rec);
            bnn_note_launch();
        }
    rc = report(nl);
    if(rc != BNN_OK) return rc;
    for(int k = 0; k < nl; ++k) {
        Outer& e = o[live[k]];
        e.bmax = hrep[k].bmax;
        e.res = hrep[k].res;
        e.ok = e.bmax < (double)FLT_MIN;
    }

    std::vector<int> set;
    for(;;) {
        // the lone loop's decisions, scene by scene
        set.clear();
        for(int i : live) {
            Outer& e = o[i];
            if(e.ok || e.stopped || e.outer >= kMaxOuter) continue;
            if(e.res < (double)items[i].outerTol * e.bmax) { e.ok = true; continue; }
            set.push_back(i);
        }
        if(set.empty()) break;
        const int ns = (int)set.size();
        BNN_CUDA_CHECK(upload(set, true));
        { kb_ir_to_f32<<<hp256[ns], 256, 0, s>>>(dirs, dp256, ns); bnn_note_launch(); }
        float ms = 0.f;
        for(const BatchLaunch& l : launches) {
            const ChunkKernel kern = batch_chunk_kernel(l.shape);
            BNN_CUDA_CHECK(cudaFuncSetAttribute(kern.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kern.smem));
            const ChunkArgs<float>* dargs = (const ChunkArgs<float>*)(D + L.args);
            const BatchGroup* dgrp = (const BatchGroup*)(D + L.grp) + l.group0;
            void* args[] = {(void*)&dargs, (void*)&dgrp};
            // the share is held until the launch has ended
            CoopShare share(CoopLoad{l.blocks, 0, 0}, numSM);
            BNN_CUDA_CHECK(cudaEventRecord(ctx.ev[0], s));
            BNN_CUDA_CHECK(cudaLaunchCooperativeKernel(kern.fn, dim3(l.blocks), dim3(l.shape.G * kLanes), args, kern.smem, s));
            bnn_note_launch();
            BNN_CUDA_CHECK(cudaEventRecord(ctx.ev[1], s));
            BNN_CUDA_CHECK(cudaEventSynchronize(ctx.ev[1]));
            float lm = 0.f;
            cudaEventElapsedTime(&lm, ctx.ev[0], ctx.ev[1]);
            ms += lm;
        }
        for(int i : set) {
            if(!alone[i]) continue;
            const BatchSolveItem& it = items[i];
            PcgWork& w = *it.w;
            const bool grid = it.layout != kRowsAny;
            PcgOutcome inner;
            rc = pcg_solve_t<float>(w, it.n, ChunkShape{}, numSM, w.r32, it.diag, it.invd, it.nbr, grid ? w.rec : nullptr, nullptr,
                                    nullptr, -(1.0f * it.dt), it.innerTol, it.maxIter, w.d32, w.r, w.z, w.s0, w.s1, w.q,
                                    w.partMaxF, true, it.dst, it.hst, s, inner);
            if(rc != BNN_OK) return rc;
            ms += inner.kernelMs;
        }
        { kb_ir_accumulate<<<hp256[ns], 256, 0, s>>>(dirs, dp256, ns); bnn_note_launch(); }
        { kb_ir_residual<<<hpch[ns], kLanes, 0, s>>>(dirs, dpch, ns); bnn_note_launch(); }
        rc = report(ns);
        if(rc != BNN_OK) return rc;
        for(int k = 0; k < ns; ++k) {
            Outer& e = o[set[k]];
            e.total += hrep[k].iter;
            e.kernelMs += ms;
            e.res = hrep[k].res;
            ++e.outer;
            if(e.total >= items[set[k]].maxIter) e.stopped = true;
        }
    }
    for(int i : live) {
        Outer& e = o[i];
        if(!e.ok && e.res < (double)items[i].outerTol * e.bmax) e.ok = true;
        PcgOutcome& out = items[i].out;
        out.iterations = e.total;
        out.outer = e.outer;
        out.kernelMs = e.kernelMs;
        out.residual = e.res;
        out.success = e.ok ? 1 : 0;
    }
    // pressure = (float) x64
    BNN_CUDA_CHECK(upload(live, false));
    { kb_ir_finish<<<hp256[nl], 256, 0, s>>>(dirs, dp256, nl); bnn_note_launch(); }
    BNN_CUDA_CHECK(cudaGetLastError());
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    return BNN_OK;
}

// ---- self-test of the bounded barrier wait -------------------------------------------
// One block arrives at a barrier sized for two blocks, so the wait can only end by giving
// up; out[0] = 1 when it gave up, out[1] = the block's polling time in ns.
__global__ void k_barrier_probe(GridSync* gs, unsigned* flags, BarrierLimit lim, unsigned long long* out) {
    unsigned sense = 0;
    const unsigned long long t0 = global_ns();
    const bool passed = grid_barrier(gs, 2u, sense, flags, lim);
    if(threadIdx.x == 0) {
        out[0] = passed ? 0ull : 1ull;
        out[1] = global_ns() - t0;
    }
}

// The packet waits in turn, each with a packet that nobody publishes: a block of two groups as one
// (both forms), then the groups apart, the first of them with all its packets there.  passed[k] and
// flags[k] of wait k; what is left to do after a wait is what a solve does: return.
constexpr int kProbeWaits = 7, kProbeChunks = 40;
__global__ void __launch_bounds__(2 * kLanes) k_wait_probe(PcgPacket* slots, unsigned* passed, unsigned* flags, BarrierLimit lim) {
    __shared__ WaitSmem<float, 2> split;
    __shared__ WaitSmem<float, 6> whole;
    __shared__ GroupWaitSmem<float> group[2];
    const int grp = (int)threadIdx.x / kLanes, t = (int)threadIdx.x % kLanes;
    double sum;
    float mx;
    if(threadIdx.x == 0) {
        for(int x = 0; x < 2; ++x) split.bad[x] = whole.bad[x] = 0;
        // chunk 0 is there, the others are not
        st_release_packet(slots, PcgPacket{(unsigned long long)__double_as_longlong(2.0), max_bits(3.0f) | 1ull << 63});
        st_ready(slots, 1u);
    }
    if(t == 0) group[grp].bad = 0;
    __syncthreads();
    auto note = [&](int k, bool ok, bool writer) { if(writer) passed[k] = ok ? 1u : 0u; };
    note(0, packet_wait_split<float, false, false, 1, 2>(slots, 2, 1u, flags + 0, split, sum, mx, lim), threadIdx.x == 0);
    note(1, packet_wait_split<float, true, true, 1, 2>(slots, 2, 1u, flags + 1, split, sum, mx, lim), threadIdx.x == 0);
    note(2, packet_wait<float, false, false, 6>(slots, 2, 1u, flags + 2, whole, sum, mx, lim), threadIdx.x == 0);
    note(3, packet_wait<float, true, true, 6>(slots, kProbeChunks, 1u, flags + 3, whole, sum, mx, lim), threadIdx.x == 0);
    if(grp == 0) {
        const bool ok = group_wait<float, true, true>(slots, 1, 1u, flags + 4, group[0], 0, t, sum, mx, lim);
        note(4, ok && sum == 2.0 && mx == 3.0f, t == 0);
    } else {
        note(5, group_wait<float, true, true>(slots, 2, 1u, flags + 5, group[1], 1, t, sum, mx, lim), t == 0);
        note(6, group_wait<float, true, true>(slots, kProbeChunks, 1u, flags + 6, group[1], 1, t, sum, mx, lim), t == 0);
    }
}

int pcg_barrier_probe(float limitSeconds, int* barrierStatus, float* elapsedMs) {
    GridSync* gs = nullptr;
    unsigned* flags = nullptr;
    unsigned long long* out = nullptr;
    int rc = BNN_OK;
    auto chk = [&](cudaError_t e) { if(e != cudaSuccess && rc == BNN_OK) { bnn_set_error(cudaGetErrorString(e)); rc = e == cudaErrorMemoryAllocation ? BNN_ERR_OUT_OF_MEMORY : BNN_ERR_CUDA; } };
    chk(cudaMalloc(&gs, sizeof(GridSync)));
    chk(cudaMalloc(&flags, sizeof(unsigned)));
    chk(cudaMalloc(&out, 2 * sizeof(unsigned long long)));
    constexpr size_t slotBytes = (size_t)kProbeChunks * kPacketStride * sizeof(PcgPacket), waitBytes = 2 * kProbeWaits * sizeof(unsigned);
    PcgPacket* slots = nullptr;
    chk(cudaMalloc(&slots, slotBytes + waitBytes));
    unsigned long long h[2] = {0, 0};
    unsigned hf = 0, hw[2 * kProbeWaits] = {};
    if(rc == BNN_OK) {
        chk(cudaMemset(gs, 0, sizeof(GridSync)));
        chk(cudaMemset(flags, 0, sizeof(unsigned)));
        chk(cudaMemset(slots, 0, slotBytes + waitBytes));
    }
    if(rc == BNN_OK) {
        // 4096 polls, then limitSeconds of time; 2^26 polls at most whatever the clock says
        const BarrierLimit lim = {(unsigned long long)((double)limitSeconds * 1e9), 1u << 12, 1u << 26};
        k_barrier_probe<<<1, kLanes>>>(gs, flags, lim, out);
        bnn_note_launch();
        chk(cudaGetLastError());
        unsigned* waits = (unsigned*)((char*)slots + slotBytes);
        // six waits in turn: at most 50 ms each
        const BarrierLimit each = {std::min(lim.ns, 50000000ull), lim.minSpins, lim.maxSpins};
        k_wait_probe<<<1, 2 * kLanes>>>(slots, waits, waits + kProbeWaits, each);
        bnn_note_launch();
        chk(cudaGetLastError());
        chk(cudaDeviceSynchronize());
        chk(cudaMemcpy(hw, waits, waitBytes, cudaMemcpyDeviceToHost));
        chk(cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost));
        chk(cudaMemcpy(&hf, flags, sizeof(hf), cudaMemcpyDeviceToHost));
    }
    cudaFree(gs);
    cudaFree(flags);
    cudaFree(out);
    cudaFree(slots);
    if(rc != BNN_OK) return rc;
    bool gaveUp = h[0] == 1ull && (hf & BNN_FLAG_TIMEOUT);
    for(int k = 0; k < kProbeWaits; ++k)  // wait 4 has its packet
        gaveUp = gaveUp && hw[k] == (k == 4 ? 1u : 0u) && hw[kProbeWaits + k] == (k == 4 ? 0u : (unsigned)BNN_FLAG_TIMEOUT);
    *barrierStatus = gaveUp ? BNN_ERR_TIMEOUT : BNN_OK;
    *elapsedMs = (float)((double)h[1] * 1e-6);
    return BNN_OK;
}

} // namespace bnn
