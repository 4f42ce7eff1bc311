// Uniform-grid cell sort, Morton z-sort and neighbour search (BananaCore/Banana/Grid,
// BananaCore/Banana/NeighborSearch) as standalone device entry points.
//
// Sorting is a stable LSD radix sort (8-bit digits, passes only over the bits a key can have): per
// 2048-item tile a 256-bin histogram, per digit an exclusive scan over the tiles, then a scatter
// that ranks equal digits in input order with warp match masks.  Stability gives the canonical
// order of equal keys (input order), which is what the reference's one-thread bucket fill
// produces.
#include "bnn_internal.cuh"

#include <algorithm>
#include <mutex>

namespace bnn {
cudaError_t exclusive_scan_u32_to_u64(const uint32_t* in, unsigned long long* out, size_t n, void* ws, cudaStream_t s);
size_t scan_workspace_bytes_u64(size_t n);

namespace {
constexpr int kRT = 256;           // threads per radix tile
constexpr int kRPer = 8;           // rounds per tile
constexpr int kRTile = kRT * kRPer;
constexpr int kWarps = kRT / 32;

// Tile histograms of one digit: hist[digit * ntiles + tile]
template<class K> __global__ void __launch_bounds__(kRT) k_radix_hist(const K* __restrict__ keys, size_t n, int shift,
                                                                      uint32_t* __restrict__ hist, unsigned ntiles) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kRTile;
#pragma unroll
    for(int r = 0; r < kRPer; ++r) {
        size_t e = base + (size_t)r * kRT + threadIdx.x;
        if(e < n) atomicAdd(&h[(unsigned)((keys[e] >> shift) & 0xFF)], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// A block per digit: its row of tile counts becomes their exclusive scan, the row's total goes to
// totals[digit]
__global__ void __launch_bounds__(kRT) k_radix_rows(uint32_t* __restrict__ hist, unsigned ntiles, uint32_t* __restrict__ totals) {
    __shared__ uint32_t warpSum[kWarps];
    uint32_t* row = hist + (size_t)blockIdx.x * ntiles;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t run = 0;
    for(unsigned t0 = 0; t0 < ntiles; t0 += kRT) {
        const unsigned i = t0 + threadIdx.x;
        const uint32_t v = i < ntiles ? row[i] : 0u;
        uint32_t x = v;
#pragma unroll
        for(int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, x, off);
            if(lane >= off) x += o;
        }
        if(lane == 31) warpSum[w] = x;
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for(int q = 0; q < kWarps; ++q) {
            const uint32_t o = warpSum[q];
            before += q < w ? o : 0u;
            all += o;
        }
        if(i < ntiles) row[i] = run + before + x - v;
        run += all;
        __syncthreads();
    }
    if(threadIdx.x == 0) totals[blockIdx.x] = run;
}

// Each warp owns 256 consecutive items of its tile and ranks them among its own; after a prefix
// over the tile's warps and digits the tile is sorted in shared memory and written out in order,
// so that a digit's items leave as a run of consecutive addresses.
template<class K> __global__ void __launch_bounds__(kRT) k_radix_scatter(const K* __restrict__ kin,
                                                                         const uint32_t* __restrict__ vin,
                                                                         K* __restrict__ kout, uint32_t* __restrict__ vout,
                                                                         size_t n, int shift,
                                                                         const uint32_t* __restrict__ rows,
                                                                         const uint32_t* __restrict__ totals,
                                                                         unsigned ntiles) {
    __shared__ uint32_t cnt[kWarps][256];
    __shared__ uint32_t toOut[256];  // a digit's place in the output minus its place in the tile
    __shared__ uint32_t warpSum[2][kWarps];
    __shared__ K sKey[kRTile];
    __shared__ uint32_t sVal[kRTile];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const size_t base = (size_t)blockIdx.x * kRTile + (size_t)w * (32 * kRPer) + lane;
    const unsigned lt = (1u << lane) - 1u;
    auto warp_exclusive = [&](uint32_t v, uint32_t* sum) {
        uint32_t x = v;
#pragma unroll
        for(int off = 1; off < 32; off <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, x, off);
            if(lane >= off) x += o;
        }
        if(lane == 31) sum[w] = x;
        return x - v;
    };
    K key[kRPer];
    uint32_t val[kRPer];
#pragma unroll
    for(int r = 0; r < kRPer; ++r) {
        const size_t e = base + 32 * r;
        key[r] = e < n ? kin[e] : K(0);
        val[r] = e < n ? (vin ? vin[e] : (uint32_t)e) : 0u;
    }
    // where digit t's items of this tile start: the digits before it and the tiles before this one
    uint32_t start = warp_exclusive(totals[t], warpSum[0]) + rows[(size_t)t * ntiles + blockIdx.x];
#pragma unroll
    for(int q = lane; q < 256; q += 32) cnt[w][q] = 0;
    __syncwarp();
    // rank of an item among the warp's items of its digit so far
    uint32_t rank[kRPer];
#pragma unroll
    for(int r = 0; r < kRPer; ++r) {
        const bool valid = base + 32 * r < n;
        const unsigned d = valid ? (unsigned)((key[r] >> shift) & 0xFF) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned before = __popc(peers & lt);
        rank[r] = valid ? cnt[w][d] + before : 0u;
        __syncwarp();
        if(valid && before == 0) cnt[w][d] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    uint32_t mine = 0;  // digit t's items in the tile, then their place in it
#pragma unroll
    for(int q = 0; q < kWarps; ++q) mine += cnt[q][t];
    const uint32_t within = warp_exclusive(mine, warpSum[1]);
    __syncthreads();
    {
        uint32_t run = within;
        for(int q = 0; q < w; ++q) { start += warpSum[0][q]; run += warpSum[1][q]; }
        toOut[t] = start - run;
#pragma unroll
        for(int q = 0; q < kWarps; ++q) {
            const uint32_t c = cnt[q][t];
            cnt[q][t] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for(int r = 0; r < kRPer; ++r)
        if(base + 32 * r < n) {
            const uint32_t at = cnt[w][(unsigned)((key[r] >> shift) & 0xFF)] + rank[r];
            sKey[at] = key[r];
            sVal[at] = val[r];
        }
    __syncthreads();
    const uint32_t items = (uint32_t)min((size_t)kRTile, n - (size_t)blockIdx.x * kRTile);
#pragma unroll
    for(int r = 0; r < kRPer; ++r) {
        const uint32_t i = r * kRT + t;
        if(i < items) {
            const K k = sKey[i];
            const uint32_t dst = toOut[(unsigned)((k >> shift) & 0xFF)] + i;
            kout[dst] = k;
            vout[dst] = sVal[i];
        }
    }
}

// OR and AND of all keys, reduced over the block before the two atomics
template<class K> __global__ void __launch_bounds__(256) k_key_bits(const K* __restrict__ keys, size_t n, unsigned long long* orv,
                                                                    unsigned long long* andv) {
    __shared__ unsigned long long so[8], sa[8];
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long o = 0, a = ~0ull;
    for(; i < n; i += (size_t)gridDim.x * blockDim.x) {
        unsigned long long k = (unsigned long long)keys[i];
        o |= k;
        a &= k;
    }
    for(int off = 16; off > 0; off >>= 1) {
        o |= __shfl_xor_sync(0xffffffffu, o, off);
        a &= __shfl_xor_sync(0xffffffffu, a, off);
    }
    if((threadIdx.x & 31) == 0) { so[threadIdx.x >> 5] = o; sa[threadIdx.x >> 5] = a; }
    __syncthreads();
    if(threadIdx.x == 0) {
        for(int q = 1; q < 8; ++q) { o |= so[q]; a &= sa[q]; }
        atomicOr(orv, o);
        atomicAnd(andv, a);
    }
}

__global__ void k_iota(uint32_t* v, size_t n) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i < n) v[i] = (uint32_t)i;
}

// Grid::getCellIdx + getCellLinearizedIndex (Grid.h:108-111,156-162), clamped to the grid; on
// the way the tile histogram of the sort's first digit (hist, a block per tile) and the count
// of every cell (count, optional)
__global__ void __launch_bounds__(kRT) k_grid_cell_ids(const float* __restrict__ pos, uint32_t n, float b0, float b1, float b2,
                                                       float cs, int n0, int n1, int n2, uint32_t* __restrict__ cid,
                                                       unsigned* oor, uint32_t* __restrict__ hist, unsigned ntiles,
                                                       uint32_t* __restrict__ count) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int nn[3] = {n0, n1, n2};
    const float bb[3] = {b0, b1, b2};
    int left = 0;  // points outside the grid
#pragma unroll 4
    for(int r = 0; r < kRPer; ++r) {
        const size_t p = (size_t)blockIdx.x * kRTile + (size_t)r * kRT + threadIdx.x;
        if(p >= n) break;
        int c[3];
        bool out = false;
#pragma unroll
        for(int d = 0; d < 3; ++d) {
            c[d] = (int)((pos[3 * p + d] - bb[d]) / cs);
            if(c[d] < 0) { c[d] = 0; out = true; }
            if(c[d] >= nn[d]) { c[d] = nn[d] - 1; out = true; }
        }
        left += out ? 1 : 0;
        const uint32_t id = (uint32_t)(((size_t)c[2] * n1 + c[1]) * n0 + c[0]);
        cid[p] = id;
        atomicAdd(&h[id & 0xFF], 1u);
        if(count) atomicAdd(count + id, 1u);
    }
    if(left) atomicAdd(oor, (unsigned)left);
    __syncthreads();
    hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

__global__ void k_histogram(const uint32_t* __restrict__ keys, size_t n, uint32_t* __restrict__ count) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i < n) atomicAdd(count + keys[i], 1u);
}

// NeighborSearch::cell_index (NeighborSearch.cpp:44-52) with SHIFT_POSITION 1.2345
// (DataStructures.h:32) and inv_cell_size = float(1.0 / r)
__device__ __forceinline__ void ns_key(float x, float y, float z, float inv, int k[3]) {
    const float sh = 1.2345f;
    const float t[3] = {x - sh, y - sh, z - sh};
#pragma unroll
    for(int d = 0; d < 3; ++d) k[d] = t[d] >= 0.f ? (int)(inv * t[d]) : (int)(inv * t[d]) - 1;
}

// Morton code as m3D_e_sLUT<uint_fast64_t, uint_fast32_t> (Morton/Morton3D.h:54-66):
// 8 byte groups, each x/y/z byte bit-interleaved and shifted in by 24 bits, so only the
// three low bytes of each coordinate survive in the 64-bit code.
__device__ __forceinline__ unsigned long long spread8(unsigned b) {
    unsigned long long r = 0;
#pragma unroll
    for(int i = 0; i < 8; ++i) r |= (unsigned long long)((b >> i) & 1u) << (3 * i);
    return r;
}
__device__ __forceinline__ unsigned long long morton3d(unsigned long long x, unsigned long long y,
                                                       unsigned long long z) {
    unsigned long long ans = 0;
#pragma unroll
    for(int i = 8; i > 0; --i) {
        const unsigned sh = (unsigned)(i - 1) * 8;
        ans = (ans << 24) | (spread8((unsigned)((z >> sh) & 0xFF)) << 2) | (spread8((unsigned)((y >> sh) & 0xFF)) << 1) |
              spread8((unsigned)((x >> sh) & 0xFF));
    }
    return ans;
}

// NeighborSearch::z_value (NeighborSearch.cpp:57-67)
__global__ void k_zvalues(const float* __restrict__ pos, uint32_t n, float inv, unsigned long long* __restrict__ z) {
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= n) return;
    int k[3];
    ns_key(pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], inv, k);
    unsigned long long c[3];
#pragma unroll
    for(int d = 0; d < 3; ++d) c[d] = (unsigned long long)((long long)k[d] - ((long long)INT_MIN + 1));
    z[p] = morton3d(c[0], c[1], c[2]);
}

// Hash keys of the points and their box: reduced over the block first, so the six
// words of the box see one atomic per block instead of one per warp
__global__ void __launch_bounds__(256) k_ns_keys(const float* __restrict__ pos, uint32_t n, float inv,
                                                 int* __restrict__ keys3, int* __restrict__ kmin,
                                                 int* __restrict__ kmax) {
    __shared__ int sMin[3][8], sMax[3][8];
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int k[3] = {INT_MAX, INT_MAX, INT_MAX}, km[3] = {INT_MIN, INT_MIN, INT_MIN};
    if(p < n) {
        ns_key(pos[3 * p], pos[3 * p + 1], pos[3 * p + 2], inv, k);
#pragma unroll
        for(int d = 0; d < 3; ++d) { keys3[3 * p + d] = k[d]; km[d] = k[d]; }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for(int d = 0; d < 3; ++d) {
        int a = k[d], b = km[d];
        for(int off = 16; off > 0; off >>= 1) {
            a = min(a, __shfl_xor_sync(0xffffffffu, a, off));
            b = max(b, __shfl_xor_sync(0xffffffffu, b, off));
        }
        if(lane == 0) { sMin[d][w] = a; sMax[d][w] = b; }
    }
    __syncthreads();
    if(threadIdx.x < 3) {
        const int d = threadIdx.x;
        int a = INT_MAX, b = INT_MIN;
        for(int q = 0; q < (int)(blockDim.x >> 5); ++q) { a = min(a, sMin[d][q]); b = max(b, sMax[d][q]); }
        if(a != INT_MAX) atomicMin(kmin + d, a);
        if(b != INT_MIN) atomicMax(kmax + d, b);
    }
}

__global__ void k_dense_cell(const int* __restrict__ keys3, uint32_t n, const int* __restrict__ kmin, int d0, int d1,
                             uint32_t* __restrict__ cid) {
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= n) return;
    const int x = keys3[3 * p] - kmin[0] + 1, y = keys3[3 * p + 1] - kmin[1] + 1, z = keys3[3 * p + 2] - kmin[2] + 1;
    cid[p] = (uint32_t)(((size_t)z * d1 + y) * d0 + x);
}

__global__ void k_gather_pos(const float* __restrict__ pos, const uint32_t* __restrict__ order, uint32_t n,
                             float4* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const uint32_t p = order[i];
    out[i] = make_float4(pos[3 * (size_t)p], pos[3 * (size_t)p + 1], pos[3 * (size_t)p + 2], __uint_as_float(p));
}

// Packed FP32: two lanes of a 64-bit register, each operation rounded as the scalar one
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    return (unsigned long long)__float_as_uint(lo) | (unsigned long long)__float_as_uint(hi) << 32;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// a * b as a * b + (-0), which rounds to the product.  The -0 pair comes in as a kernel
// argument: of a plain packed product and sum the assembler makes one fused operation, which
// rounds once (20 of 4M points' lists changed).
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b, unsigned long long minus0) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(minus0));
    return d;
}
constexpr unsigned long long kMinusZero2 = 0x8000000080000000ull;

// NeighborSearch::query3D (NeighborSearch.cpp:530-692): every other point of the 27 hash cells
// around a point with (dx*dx + dy*dy) + dz*dz < r^2, in the order of the cells (z, y, x major)
// and of the sorted points inside them.
//
// A warp owns P consecutive sorted points.  Points of one cell share their candidates, the 9
// rows of 3 cells around it laid end to end: a lane holds one candidate of a group of 32 and
// tests it against the cell's points one pair at a time (packed FP32, the points broadcast from
// shared memory), a vote makes each point's hits in the group one word, kept by the point's
// lane.  Counting is then one population count per lane and group; in the writing pass
// (WRITE) the warp writes each point's hits as consecutive entries.  A point is tested against
// itself too; that bit is cleared in its word.
//
// Bound by instruction issue: about 9 per point and 32 candidates, 20 when writing, against 15
// per point and candidate (and its store through a shared buffer) with a thread per point that
// walks the candidates alone.  Measured, whole bnn_neighbors call: 4M points and 933 M entries
// 8.45 ms (11.45 with a thread per point), 20,011 points 0.305 ms (0.602).
//
// That takes turns over the cells of a warp's points.  In sparse sets a cell holds a few points and
// a turn is nearly all waiting, so a warp of 32 points whose points lie in many cells has a thread
// walk each point's rows alone (ns_alone).  Lines at more than 4 cells when counting and 8 when
// writing, where one thread's short runs of stores cost more.  Whole call, ms, thread per point for
// all (this warp form for all) -> by the lines: 1M points of 0.5 a cell 0.445 (0.578) -> 0.320, of 5
// 0.650 (0.655) -> 0.578, of 20 1.247 (1.069) -> 1.080; 4M points of 0.5 a cell 1.04 (1.87) -> 0.89,
// of 3 1.51 (1.97) -> 1.40, of 6 2.04 (2.22) -> 2.04, of 20 4.30 (3.87) -> 3.91.
constexpr int kNsWarps = 4;  // warps per block: they end at different times
template<bool WRITE> constexpr int kNsCells = WRITE ? 8 : 4;
// One point's hits, counted or written to `to`
template<bool WRITE>
__device__ __forceinline__ uint32_t ns_alone(const float4* __restrict__ sp, const float4& a, uint32_t at, uint32_t cell,
                                             const uint32_t* __restrict__ cellStart, int d0, int d1, float r2,
                                             uint32_t* __restrict__ to) {
    uint32_t cnt = 0;
#pragma unroll 1
    for(int dz = -1; dz <= 1; ++dz) {
        uint32_t b[3], e[3];
#pragma unroll
        for(int dy = 0; dy < 3; ++dy) {
            const long long row = (long long)cell + dz * ((long long)d0 * d1) + (dy - 1) * (long long)d0;
            b[dy] = cellStart[row - 1];
            e[dy] = cellStart[row + 2];
        }
#pragma unroll
        for(int dy = 0; dy < 3; ++dy)
            for(uint32_t j = b[dy]; j < e[dy]; ++j) {
                const float4 q = sp[j];
                const float t0 = a.x - q.x, t1 = a.y - q.y, t2 = a.z - q.z;
                const float l2 = t0 * t0 + t1 * t1 + t2 * t2;
                if(l2 < r2 && j != at) {
                    if(WRITE) to[cnt] = __float_as_uint(q.w);
                    ++cnt;
                }
            }
    }
    return cnt;
}
template<int P, bool WRITE>
__global__ void __launch_bounds__(kNsWarps * 32) k_ns_pairs(const float4* __restrict__ sp, const uint32_t* __restrict__ scid,
                                                            uint32_t n, const uint32_t* __restrict__ cellStart, int d0,
                                                            int d1, float r2, unsigned long long minus0,
                                                            uint32_t* __restrict__ counts,
                                                            const unsigned long long* __restrict__ offsets,
                                                            uint32_t* __restrict__ idx) {
    constexpr unsigned full = 0xffffffffu;
    __shared__ __align__(16) float2 sXY[kNsWarps][P], sZ[kNsWarps][P / 2];  // {x pair, y pair} per pair, {z pair}
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = (blockIdx.x * kNsWarps + warp) * (uint32_t)P;
    if(first >= n) return;
    const int mine = (int)min((uint32_t)P, n - first);  // points of this warp
    const bool live = lane < mine;
    const float4 a = live ? sp[first + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t self = __float_as_uint(a.w);
    const uint32_t cell = live ? scid[first + lane] : full;
    if constexpr(P == 32) {
        const uint32_t before = __shfl_up_sync(full, cell, 1);
        if(__popc(__ballot_sync(full, live && (lane == 0 || cell != before))) > kNsCells<WRITE>) {
            if(live) {
                const uint32_t cnt = ns_alone<WRITE>(sp, a, first + lane, cell, cellStart, d0, d1, r2,
                                                     WRITE ? idx + offsets[self] : nullptr);
                if(!WRITE) counts[self] = cnt;
            }
            return;
        }
    }
    if(lane < P) {
        float* xy = reinterpret_cast<float*>(&sXY[warp][lane & ~1]);
        xy[lane & 1] = a.x;
        xy[2 + (lane & 1)] = a.y;
        reinterpret_cast<float*>(sZ[warp])[lane] = a.z;
    }
    __syncwarp();
    unsigned long long o = WRITE && live ? offsets[self] : 0ull;
    uint32_t cnt = 0;
    for(int s0 = 0; s0 < mine;) {
        // the points s0 .. s1 - 1 of one cell
        const uint32_t c = __shfl_sync(full, cell, s0);
        const int s1 = s0 + __popc(__ballot_sync(full, cell == c && live));
        // its candidate rows: lane q the q-th one, at places before .. before + len - 1 of the list
        uint32_t b = 0, len = 0;
        if(lane < 9) {
            const long long row = (long long)c + (lane / 3 - 1) * ((long long)d0 * d1) + (lane % 3 - 1) * (long long)d0;
            b = cellStart[row - 1];
            len = cellStart[row + 2] - b;
        }
        uint32_t before = len;
#pragma unroll
        for(int off = 1; off < 16; off <<= 1) {
            const uint32_t v = __shfl_up_sync(full, before, off);
            if(lane >= off) before += v;
        }
        const uint32_t total = __shfl_sync(full, before, 8);
        before -= len;
        const uint32_t shift = b - before;  // place in the list + shift = sorted index
        uint32_t rowAt[9], rowShift[9];
#pragma unroll
        for(int q = 0; q < 9; ++q) {
            rowAt[q] = __shfl_sync(full, before, q);
            rowShift[q] = __shfl_sync(full, shift, q);
        }
        // this lane's point stands at this place of the list (the middle row holds its cell)
        const uint32_t selfAt = first + lane - rowShift[4];
        for(uint32_t g = 0; g < total; g += 32) {
            const uint32_t at = g + lane;
            uint32_t sh = rowShift[0];
#pragma unroll
            for(int q = 1; q < 9; ++q) sh = at >= rowAt[q] ? rowShift[q] : sh;
            const float4 q = at < total ? sp[at + sh] : make_float4(INFINITY, 0.f, 0.f, 0.f);
            const unsigned long long nx = pack2(-q.x, -q.x), ny = pack2(-q.y, -q.y), nz = pack2(-q.z, -q.z);
            unsigned hits = 0;
            for(int k = s0 & ~1; k < s1; k += 2) {
                const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(&sXY[warp][k]);
                const unsigned long long z = *reinterpret_cast<const unsigned long long*>(&sZ[warp][k >> 1]);
                const unsigned long long t0 = add2(xy.x, nx), t1 = add2(xy.y, ny), t2 = add2(z, nz);
                const unsigned long long l2 = add2(add2(mul2(t0, t0, minus0), mul2(t1, t1, minus0)), mul2(t2, t2, minus0));
                const unsigned h0 = __ballot_sync(full, __uint_as_float((unsigned)l2) < r2);
                const unsigned h1 = __ballot_sync(full, __uint_as_float((unsigned)(l2 >> 32)) < r2);
                if(lane == k) hits = h0;
                if(lane == k + 1) hits = h1;
            }
            if(lane < s0 || lane >= s1) hits = 0;
            if(selfAt - g < 32u) hits &= ~(1u << (selfAt - g));
            if constexpr(!WRITE) cnt += __popc(hits);
            else {
                const uint32_t other = __float_as_uint(q.w);
                const unsigned lt = (1u << lane) - 1u;
                for(unsigned todo = __ballot_sync(full, hits != 0u); todo; todo &= todo - 1) {
                    const int k = __ffs(todo) - 1;
                    const unsigned h = __shfl_sync(full, hits, k);
                    const unsigned long long to = __shfl_sync(full, o, k);
                    if(h >> lane & 1u) idx[to + __popc(h & lt)] = other;
                }
                o += __popc(hits);
            }
        }
        s0 = s1;
    }
    if(!WRITE && live) counts[self] = cnt;
}
// Points per warp: 32 share their candidates' loads best; below kNsFew points, 8 give the GPU
// four times the warps.  Whole call, ms with 8 (with 32) on 148 SMs: 20,000 points of 20 a cell 0.190
// (0.243), of 0.5 0.157 (0.159); 80,000 0.249 (0.259), 0.202 (0.182); 160,000 0.337 (0.324), 0.231
// (0.187); 400,000 0.612 (0.548), 0.340 (0.226).  The two are within 4 % from 80,000 to 160,000
// points of 20 a cell.
constexpr uint32_t kNsFew = 150000;
template<bool WRITE>
void launch_ns_pairs(const float4* sp, const uint32_t* scid, uint32_t n, const uint32_t* cellStart, int d0, int d1, float r2,
                     uint32_t* counts, const unsigned long long* offsets, uint32_t* idx, cudaStream_t s) {
    const uint32_t per = (n < kNsFew ? 8u : 32u) * kNsWarps;
    const unsigned blocks = (n + per - 1) / per;
    if(n < kNsFew) k_ns_pairs<8, WRITE><<<blocks, kNsWarps * 32, 0, s>>>(sp, scid, n, cellStart, d0, d1, r2, kMinusZero2, counts, offsets, idx);
    else k_ns_pairs<32, WRITE><<<blocks, kNsWarps * 32, 0, s>>>(sp, scid, n, cellStart, d0, d1, r2, kMinusZero2, counts, offsets, idx);
    bnn_note_launch();
}
} // namespace

// ---- host helpers -------------------------------------------------------------------
namespace {
// Temporary device memory from the device's memory pool, allocated and freed in order on
// the stream that uses it (no device-wide synchronisation, freed memory reused by the next
// call)
struct DevBuf {
    void* p = nullptr;
    cudaStream_t s = nullptr;
    ~DevBuf() { if(p) cudaFreeAsync(p, s); }
    cudaError_t alloc(size_t b, cudaStream_t st) {
        const cudaError_t e = mem_pool_setup();
        if(e != cudaSuccess) return e;
        s = st;
        return cudaMallocAsync(&p, b ? b : 1, st);
    }
    template<class T> T* as() { return (T*)p; }
};

// uint32 words a sort of n keys needs for its tile histograms and digit totals
size_t radix_scratch_words(size_t n) { return 256 * ((n + kRTile - 1) / kRTile) + 256; }

// Stable sort (input order for ties) of the key bits [lo, hi): the permutation in permOut, the
// sorted keys in keysOut; k2 / v2 hold n keys / values, scratch radix_scratch_words(n).  firstHist:
// scratch already holds the tile histograms of the first digit.
template<class K>
cudaError_t radix_passes(const K* keys, size_t n, int lo, int hi, K* keysOut, uint32_t* permOut, K* k2, uint32_t* v2,
                         uint32_t* scratch, bool firstHist, cudaStream_t s) {
    const unsigned ntiles = (unsigned)((n + kRTile - 1) / kRTile);
    uint32_t* totals = scratch + (size_t)256 * ntiles;
    const K* kin = keys;
    const uint32_t* vin = nullptr;
    const int np = (hi - lo + 7) / 8;
    if(np <= 0) {
        if(keysOut) {
            const cudaError_t e = cudaMemcpyAsync(keysOut, keys, n * sizeof(K), cudaMemcpyDeviceToDevice, s);
            if(e != cudaSuccess) return e;
        }
        { k_iota<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(permOut, n); bnn_note_launch(); }
        return cudaGetLastError();
    }
    for(int pi = 0; pi < np; ++pi) {
        // ping-pong so that the last pass lands in keysOut / permOut
        const bool toOut = ((np - 1 - pi) % 2) == 0;
        K* kout = toOut ? keysOut : k2;
        uint32_t* vout = toOut ? permOut : v2;
        const int shift = lo + 8 * pi;
        if(pi > 0 || !firstHist) { k_radix_hist<K><<<ntiles, kRT, 0, s>>>(kin, n, shift, scratch, ntiles); bnn_note_launch(); }
        { k_radix_rows<<<256, kRT, 0, s>>>(scratch, ntiles, totals); bnn_note_launch(); }
        { k_radix_scatter<K><<<ntiles, kRT, 0, s>>>(kin, vin, kout, vout, n, shift, scratch, totals, ntiles); bnn_note_launch(); }
        kin = kout;
        vin = vout;
    }
    return cudaGetLastError();
}
// bits of the values below `bound`
int bits_below(size_t bound) {
    int b = 0;
    while(b < 63 && ((size_t)1 << b) < bound) ++b;
    return b;
}

// radix_passes with its temporaries from the pool, in order on s
template<class K>
int radix_sort(const K* keys, size_t n, int lo, int hi, K* keysOut, uint32_t* permOut, cudaStream_t s) {
    if(n == 0) return BNN_OK;
    DevBuf k2, v2, scratch;
    BNN_CUDA_CHECK(k2.alloc(n * sizeof(K), s));
    BNN_CUDA_CHECK(v2.alloc(n * sizeof(uint32_t), s));
    BNN_CUDA_CHECK(scratch.alloc(radix_scratch_words(n) * sizeof(uint32_t), s));
    BNN_CUDA_CHECK(radix_passes<K>(keys, n, lo, hi, keysOut, permOut, k2.as<K>(), v2.as<uint32_t>(), scratch.as<uint32_t>(),
                                   false, s));
    return BNN_OK;
}
} // namespace
} // namespace bnn

using namespace bnn;

extern "C" int bnn_cell_sort(const float* pos_dev, uint32_t n, const float bmin[3], float cell_size,
                             const int32_t ncells[3], uint32_t* cell_id_dev, uint32_t* sorted_idx_dev,
                             uint32_t* cell_start_dev, uint32_t* out_of_range, void* stream) {
    if((n && (!pos_dev || !cell_id_dev || !sorted_idx_dev)) || !bmin || !ncells || !(cell_size > 0.f))
        return BNN_ERR_INVALID_ARGUMENT;
    for(int d = 0; d < 3; ++d) if(ncells[d] <= 0) return BNN_ERR_INVALID_ARGUMENT;
    const size_t C = (size_t)ncells[0] * ncells[1] * ncells[2];
    if(C >= 0xffffffffull) return BNN_ERR_NOT_SUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    // one allocation: the out-of-grid counter and the cell counts (zeroed together), the sort's
    // key and value arrays, its histograms, the scan's workspace
    size_t bytes = 0;
    auto take = [&](size_t b) { const size_t at = bytes; bytes += (b + 255) & ~(size_t)255; return at; };
    const size_t aOor = take(sizeof(unsigned)), aCells = take(cell_start_dev ? C * sizeof(uint32_t) : 0), zeroed = bytes;
    const size_t aKeys = take((size_t)n * 4), aK2 = take((size_t)n * 4), aV2 = take((size_t)n * 4);
    const size_t aScratch = take(radix_scratch_words(n) * 4), aWs = take(cell_start_dev ? scan_workspace_bytes(C) : 0);
    DevBuf buf;
    BNN_CUDA_CHECK(buf.alloc(bytes, s));
    char* D = buf.as<char>();
    unsigned* oor = (unsigned*)(D + aOor);
    uint32_t* count = cell_start_dev ? (uint32_t*)(D + aCells) : nullptr;
    BNN_CUDA_CHECK(cudaMemsetAsync(D, 0, zeroed, s));
    if(n) {
        uint32_t* scratch = (uint32_t*)(D + aScratch);
        const unsigned ntiles = (unsigned)(((size_t)n + kRTile - 1) / kRTile);
        { k_grid_cell_ids<<<ntiles, kRT, 0, s>>>(pos_dev, n, bmin[0], bmin[1], bmin[2], cell_size, ncells[0], ncells[1], ncells[2],
                                                 cell_id_dev, oor, scratch, ntiles, count); bnn_note_launch(); }
        // the ids' bits are known from the cell count: no pass over the keys to find them
        BNN_CUDA_CHECK(radix_passes<uint32_t>(cell_id_dev, n, 0, bits_below(C), (uint32_t*)(D + aKeys), sorted_idx_dev,
                                              (uint32_t*)(D + aK2), (uint32_t*)(D + aV2), scratch, true, s));
    }
    if(cell_start_dev) BNN_CUDA_CHECK(exclusive_scan_u32(count, cell_start_dev, C, D + aWs, s));
    unsigned h = 0;
    BNN_CUDA_CHECK(cudaMemcpyAsync(&h, oor, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    if(out_of_range) *out_of_range = h;
    return BNN_OK;
}

extern "C" int bnn_z_sort(const float* pos_dev, uint32_t n, float radius, uint64_t* zvalue_dev, uint32_t* perm_dev,
                          void* stream) {
    if((n && (!pos_dev || !zvalue_dev || !perm_dev)) || !(radius > 0.f)) return BNN_ERR_INVALID_ARGUMENT;
    if(n == 0) return BNN_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const float inv = (float)(1.0 / (double)radius);
    { k_zvalues<<<(n + 255) / 256, 256, 0, s>>>(pos_dev, n, inv, (unsigned long long*)zvalue_dev); bnn_note_launch(); }
    // the codes' top bits are the same for all points: sort only the bits that vary
    DevBuf sorted, bits;
    BNN_CUDA_CHECK(bits.alloc(2 * sizeof(unsigned long long), s));
    BNN_CUDA_CHECK(cudaMemsetAsync(bits.p, 0, sizeof(unsigned long long), s));
    BNN_CUDA_CHECK(cudaMemsetAsync(bits.as<unsigned long long>() + 1, 0xff, sizeof(unsigned long long), s));
    { k_key_bits<unsigned long long><<<(unsigned)std::min<size_t>(((size_t)n + 255) / 256, 592), 256, 0, s>>>(
          (const unsigned long long*)zvalue_dev, n, bits.as<unsigned long long>(), bits.as<unsigned long long>() + 1); bnn_note_launch(); }
    unsigned long long hb[2];
    BNN_CUDA_CHECK(cudaMemcpyAsync(hb, bits.p, sizeof(hb), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    const unsigned long long vary = hb[0] ^ hb[1];
    const int lo = vary ? __builtin_ctzll(vary) & ~7 : 0, hi = vary ? 64 - __builtin_clzll(vary) : 0;
    BNN_CUDA_CHECK(sorted.alloc((size_t)n * sizeof(unsigned long long), s));
    int rc = radix_sort<unsigned long long>((const unsigned long long*)zvalue_dev, n, lo, hi, sorted.as<unsigned long long>(),
                                            perm_dev, s);
    if(rc != BNN_OK) return rc;
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    return BNN_OK;
}

extern "C" int bnn_neighbors(const float* pos_dev, uint32_t n, float radius, uint64_t* offsets_dev, uint32_t* idx_dev,
                             uint64_t capacity, uint64_t* total, void* stream) {
    if((n && (!pos_dev || !offsets_dev)) || !(radius > 0.f)) return BNN_ERR_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    if(n == 0) {
        BNN_CUDA_CHECK(cudaMemsetAsync(offsets_dev, 0, sizeof(uint64_t), s));
        if(total) *total = 0;
        return BNN_OK;
    }
    const float inv = (float)(1.0 / (double)radius);
    const float r2 = radius * radius;
    DevBuf keys3, kmm, cid, cidSorted, order, sp, cnt, start, ws, counts, ws64;
    BNN_CUDA_CHECK(keys3.alloc((size_t)n * 3 * sizeof(int), s));
    BNN_CUDA_CHECK(kmm.alloc(6 * sizeof(int), s));
    int init[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};
    BNN_CUDA_CHECK(cudaMemcpyAsync(kmm.p, init, sizeof(init), cudaMemcpyHostToDevice, s));
    { k_ns_keys<<<(n + 255) / 256, 256, 0, s>>>(pos_dev, n, inv, keys3.as<int>(), kmm.as<int>(), kmm.as<int>() + 3); bnn_note_launch(); }
    int hk[6];
    BNN_CUDA_CHECK(cudaMemcpyAsync(hk, kmm.p, sizeof(hk), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    // dense key box with one empty cell of padding on every side
    const long long d0 = (long long)hk[3] - hk[0] + 3, d1 = (long long)hk[4] - hk[1] + 3, d2 = (long long)hk[5] - hk[2] + 3;
    const long long V = d0 * d1 * d2;
    if(V > (1ll << 30)) return BNN_ERR_NOT_SUPPORTED;
    BNN_CUDA_CHECK(cid.alloc((size_t)n * sizeof(uint32_t), s));
    { k_dense_cell<<<(n + 255) / 256, 256, 0, s>>>(keys3.as<int>(), n, kmm.as<int>(), (int)d0, (int)d1, cid.as<uint32_t>()); bnn_note_launch(); }
    BNN_CUDA_CHECK(cidSorted.alloc((size_t)n * sizeof(uint32_t), s));
    BNN_CUDA_CHECK(order.alloc((size_t)n * sizeof(uint32_t), s));
    int rc = radix_sort<uint32_t>(cid.as<uint32_t>(), n, 0, bits_below((size_t)V), cidSorted.as<uint32_t>(), order.as<uint32_t>(), s);
    if(rc != BNN_OK) return rc;
    BNN_CUDA_CHECK(sp.alloc((size_t)n * sizeof(float4), s));
    { k_gather_pos<<<(n + 255) / 256, 256, 0, s>>>(pos_dev, order.as<uint32_t>(), n, sp.as<float4>()); bnn_note_launch(); }
    BNN_CUDA_CHECK(cnt.alloc((size_t)V * sizeof(uint32_t), s));
    BNN_CUDA_CHECK(start.alloc(((size_t)V + 1) * sizeof(uint32_t), s));
    BNN_CUDA_CHECK(cudaMemsetAsync(cnt.p, 0, (size_t)V * sizeof(uint32_t), s));
    { k_histogram<<<(n + 255) / 256, 256, 0, s>>>(cid.as<uint32_t>(), n, cnt.as<uint32_t>()); bnn_note_launch(); }
    size_t wsb = scan_workspace_bytes((size_t)V);
    if(wsb) BNN_CUDA_CHECK(ws.alloc(wsb, s));
    BNN_CUDA_CHECK(exclusive_scan_u32(cnt.as<uint32_t>(), start.as<uint32_t>(), (size_t)V, ws.p, s));
    BNN_CUDA_CHECK(counts.alloc((size_t)n * sizeof(uint32_t), s));
    launch_ns_pairs<false>(sp.as<float4>(), cidSorted.as<uint32_t>(), n, start.as<uint32_t>(), (int)d0, (int)d1, r2,
                           counts.as<uint32_t>(), nullptr, nullptr, s);
    size_t wsb64 = scan_workspace_bytes_u64(n);
    if(wsb64) BNN_CUDA_CHECK(ws64.alloc(wsb64, s));
    BNN_CUDA_CHECK(exclusive_scan_u32_to_u64(counts.as<uint32_t>(), (unsigned long long*)offsets_dev, n, ws64.p, s));
    uint64_t tot = 0;
    BNN_CUDA_CHECK(cudaMemcpyAsync(&tot, offsets_dev + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    if(total) *total = tot;
    if(tot > capacity) return BNN_ERR_CAPACITY;
    if(tot && !idx_dev) return BNN_ERR_INVALID_ARGUMENT;
    launch_ns_pairs<true>(sp.as<float4>(), cidSorted.as<uint32_t>(), n, start.as<uint32_t>(), (int)d0, (int)d1, r2, nullptr,
                          (const unsigned long long*)offsets_dev, idx_dev, s);
    BNN_CUDA_CHECK(cudaGetLastError());
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    return BNN_OK;
}

// ---------------------------------------------------------------------------------
// Cell sort without any device allocation.
//
// Some callers cannot allocate device memory at the moment they need a sort: an
// application whose own pool allocator has already reserved all device memory, or a loop
// on a latency budget in which cudaMalloc / cudaFree would synchronise the device and
// stall the work queued on other streams.  For them this entry point works entirely in a
// fixed scratch array compiled into the library: every GPU that loads the library holds
// kNoAllocScratchBytes (about 21 MiB) until the process exits.  Limits: at most
// kNoAllocMaxPoints points and kNoAllocMaxCells grid cells.
// ---------------------------------------------------------------------------------
namespace {
constexpr uint32_t kNoAllocMaxPoints = 1u << 20;  // 1,048,576 points
constexpr uint32_t kNoAllocMaxCells = 1u << 21;   // 2,097,152 cells (e.g. 128^3)
constexpr uint32_t kNoAllocTiles = (kNoAllocMaxPoints + kRTile - 1) / kRTile;
constexpr size_t kAlign = 256;
constexpr size_t alignUp(size_t b) { return (b + kAlign - 1) / kAlign * kAlign; }
constexpr size_t kOffCounter = 0;                                                     // out-of-range count
constexpr size_t kOffKeys0 = alignUp(kOffCounter + 16);                               // sorted keys
constexpr size_t kOffKeys1 = alignUp(kOffKeys0 + sizeof(uint32_t) * kNoAllocMaxPoints);  // ping-pong keys
constexpr size_t kOffVals1 = alignUp(kOffKeys1 + sizeof(uint32_t) * kNoAllocMaxPoints);  // ping-pong payload
constexpr size_t kOffHist = alignUp(kOffVals1 + sizeof(uint32_t) * kNoAllocMaxPoints);   // radix histograms, digit totals
constexpr size_t kOffCells = alignUp(kOffHist + sizeof(uint32_t) * (256u * kNoAllocTiles + 256));  // cell counts
constexpr size_t kOffScanWs = alignUp(kOffCells + sizeof(uint32_t) * kNoAllocMaxCells);  // scan workspace
constexpr size_t kScanWsBytes = 64u * 1024u;  // >= scan_workspace_bytes of either scan, checked at run time
constexpr size_t kNoAllocScratchBytes = alignUp(kOffScanWs + kScanWsBytes);
} // namespace

static __device__ __align__(256) unsigned char g_cellSortScratch[kNoAllocScratchBytes];

namespace {
std::mutex g_noallocMutex;
// device address of g_cellSortScratch per device ordinal, and the id of the context it
// was resolved in (a reset device gets a new context, in which the module -- and so the
// array -- can sit at another address)
void* g_noallocPtr[64] = {};
unsigned long long g_noallocCtx[64] = {};

// Id of the current context (cuCtxGetId through the runtime's driver entry point, so the
// library does not link libcuda); 0 when the driver cannot tell.
unsigned long long current_context_id() {
    using GetId = int (*)(void*, unsigned long long*);  // CUresult cuCtxGetId(CUcontext, unsigned long long*)
    static GetId fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if(cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess ||
           q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (GetId)f;
    }();
    unsigned long long id = 0;
    if(fn && fn(nullptr, &id) != 0) id = 0;
    return id;
}

// First call on a device (or in a new context of it): resolve the scratch array's device
// address with that device current.  The host-side symbol is only a stand-in and must
// never reach a kernel.
int noalloc_scratch(unsigned char** out) {
    int dev = 0;
    BNN_CUDA_CHECK(cudaGetDevice(&dev));
    if(dev < 0 || dev >= 64) return BNN_ERR_NOT_SUPPORTED;
    // 0 before the runtime made a context current: resolve (which makes it current)
    const unsigned long long ctx = current_context_id();
    std::lock_guard<std::mutex> lock(g_noallocMutex);
    if(!g_noallocPtr[dev] || ctx == 0 || g_noallocCtx[dev] != ctx) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_cellSortScratch);
        if(e != cudaSuccess || !p) {
            bnn_set_error(e != cudaSuccess ? cudaGetErrorString(e) : "scratch symbol has no device address");
            return BNN_ERR_CUDA;
        }
        g_noallocPtr[dev] = p;
        g_noallocCtx[dev] = current_context_id();
    }
    *out = (unsigned char*)g_noallocPtr[dev];
    return BNN_OK;
}
} // namespace

extern "C" int bnn_cell_sort_noalloc(const float* pos_dev, uint32_t n, const float bmin[3], float cell_size,
                                     const int32_t ncells[3], uint32_t* cell_id_dev, uint32_t* sorted_idx_dev,
                                     uint32_t* cell_start_dev, uint32_t* out_of_range, void* stream) {
    if((n && (!pos_dev || !cell_id_dev || !sorted_idx_dev)) || !bmin || !ncells || !(cell_size > 0.f))
        return BNN_ERR_INVALID_ARGUMENT;
    for(int d = 0; d < 3; ++d) if(ncells[d] <= 0) return BNN_ERR_INVALID_ARGUMENT;
    const size_t C = (size_t)ncells[0] * ncells[1] * ncells[2];
    if(n > kNoAllocMaxPoints || C > kNoAllocMaxCells) {
        bnn_set_error("bnn_cell_sort_noalloc: more than 1,048,576 points or 2,097,152 cells does not fit the "
                      "fixed scratch array; use bnn_cell_sort");
        return BNN_ERR_CAPACITY;
    }
    if(scan_workspace_bytes(C) > kScanWsBytes) return BNN_ERR_CAPACITY;
    unsigned char* scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if(rc != BNN_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    unsigned* oor = (unsigned*)(scratch + kOffCounter);
    uint32_t* keys0 = (uint32_t*)(scratch + kOffKeys0);
    uint32_t* keys1 = (uint32_t*)(scratch + kOffKeys1);
    uint32_t* vals1 = (uint32_t*)(scratch + kOffVals1);
    uint32_t* hist = (uint32_t*)(scratch + kOffHist);
    uint32_t* cells = (uint32_t*)(scratch + kOffCells);
    void* scanWs = scratch + kOffScanWs;
    // the array keeps the previous call's contents: zero what is accumulated into
    BNN_CUDA_CHECK(cudaMemsetAsync(oor, 0, sizeof(unsigned), s));
    if(cell_start_dev) BNN_CUDA_CHECK(cudaMemsetAsync(cells, 0, C * sizeof(uint32_t), s));
    if(n) {
        const unsigned ntiles = (n + kRTile - 1) / kRTile;
        { k_grid_cell_ids<<<ntiles, kRT, 0, s>>>(pos_dev, n, bmin[0], bmin[1], bmin[2], cell_size, ncells[0], ncells[1], ncells[2],
                                                 cell_id_dev, oor, hist, ntiles, cell_start_dev ? cells : nullptr); bnn_note_launch(); }
        BNN_CUDA_CHECK(radix_passes<uint32_t>(cell_id_dev, n, 0, bits_below(C), keys0, sorted_idx_dev, keys1, vals1, hist, true, s));
    }
    if(cell_start_dev) BNN_CUDA_CHECK(exclusive_scan_u32(cells, cell_start_dev, C, scanWs, s));
    BNN_CUDA_CHECK(cudaGetLastError());
    unsigned h = 0;
    BNN_CUDA_CHECK(cudaMemcpyAsync(&h, oor, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    BNN_CUDA_CHECK(cudaStreamSynchronize(s));
    if(out_of_range) *out_of_range = h;
    return BNN_OK;
}
